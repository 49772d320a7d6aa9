// passes_z2.cu -- z passes of 108- to 256-point columns (see passes.cuh).
#include "passes_impl.cuh"

namespace rism {
RISM_INST_Z(108) RISM_INST_Z(128) RISM_INST_Z(144) RISM_INST_Z(162) RISM_INST_Z(192) RISM_INST_Z(216) RISM_INST_Z(256)
}  // namespace rism
