// Grouped products of ComplexF64 values, Int64 indices (gsa_grouped.cuh).
#include "gsa_grouped.cuh"

namespace gsa {
GSA_INST_GROUPED(cf64, int64_t)
}  // namespace gsa
