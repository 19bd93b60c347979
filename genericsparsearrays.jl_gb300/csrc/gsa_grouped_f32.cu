// Grouped products of Float32 values (gsa_grouped.cuh).
#include "gsa_grouped.cuh"

namespace gsa {
GSA_INST_GROUPED(float, int32_t)
GSA_INST_GROUPED(float, int64_t)
}  // namespace gsa
