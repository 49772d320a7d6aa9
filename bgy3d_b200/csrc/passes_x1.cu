// passes_x1.cu -- x passes of 32- to 162-point rows (see passes.cuh).
#include "passes_impl.cuh"

namespace rism {
RISM_INST_X(16) RISM_INST_X(18) RISM_INST_X(24) RISM_INST_X(27) RISM_INST_X(32) RISM_INST_X(36) RISM_INST_X(48)
RISM_INST_X(54) RISM_INST_X(64) RISM_INST_X(72) RISM_INST_X(81)
}  // namespace rism
