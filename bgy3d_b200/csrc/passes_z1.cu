// passes_z1.cu -- z passes of 32- to 96-point columns (see passes.cuh).
#include "passes_impl.cuh"

namespace rism {
RISM_INST_Z(32) RISM_INST_Z(36) RISM_INST_Z(48) RISM_INST_Z(54) RISM_INST_Z(64) RISM_INST_Z(72) RISM_INST_Z(96)
}  // namespace rism
