// twogrid_fx2a.cu -- x transfers of 48- to 128-point rows (see twogrid_fx2.cuh).
#include "twogrid_fx2_impl.cuh"

namespace rism {
RISM_INST_FX2(24) RISM_INST_FX2(27) RISM_INST_FX2(32) RISM_INST_FX2(36) RISM_INST_FX2(48) RISM_INST_FX2(54)
RISM_INST_FX2(64)
}  // namespace rism
