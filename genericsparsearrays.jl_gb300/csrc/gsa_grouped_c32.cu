// Grouped products of ComplexF32 values (gsa_grouped.cuh).
#include "gsa_grouped.cuh"

namespace gsa {
GSA_INST_GROUPED(cf32, int32_t)
GSA_INST_GROUPED(cf32, int64_t)
}  // namespace gsa
