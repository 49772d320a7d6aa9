// passes_y.cu -- y passes (see passes.cuh).
#include "passes_impl.cuh"

namespace rism {
RISM_YZ_LENS(RISM_INST_Y)
}  // namespace rism
