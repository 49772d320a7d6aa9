// passes_x2.cu -- x passes of 192- to 512-point rows (see passes.cuh).
#include "passes_impl.cuh"

namespace rism {
RISM_INST_X(96) RISM_INST_X(108) RISM_INST_X(128) RISM_INST_X(144) RISM_INST_X(162) RISM_INST_X(192) RISM_INST_X(216)
RISM_INST_X(243) RISM_INST_X(256)
}  // namespace rism
