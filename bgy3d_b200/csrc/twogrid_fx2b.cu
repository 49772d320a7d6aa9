// twogrid_fx2b.cu -- x transfers of 144- to 216-point rows (see twogrid_fx2.cuh).
#include "twogrid_fx2_impl.cuh"

namespace rism {
RISM_INST_FX2(72) RISM_INST_FX2(81) RISM_INST_FX2(96) RISM_INST_FX2(108)
}  // namespace rism
