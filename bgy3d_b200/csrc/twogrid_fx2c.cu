// twogrid_fx2c.cu -- x transfers of 256- to 512-point rows (see twogrid_fx2.cuh).
#include "twogrid_fx2_impl.cuh"

namespace rism {
RISM_INST_FX2(128) RISM_INST_FX2(144) RISM_INST_FX2(162) RISM_INST_FX2(192) RISM_INST_FX2(216) RISM_INST_FX2(243)
RISM_INST_FX2(256)
}  // namespace rism
