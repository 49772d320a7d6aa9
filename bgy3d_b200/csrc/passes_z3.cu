// passes_z3.cu -- z passes of 288- to 512-point columns (see passes.cuh).
#include "passes_impl.cuh"

namespace rism {
RISM_INST_Z(288) RISM_INST_Z(324) RISM_INST_Z(384) RISM_INST_Z(432) RISM_INST_Z(486) RISM_INST_Z(512)
}  // namespace rism
