// Grouped products of ComplexF64 values, Int32 indices (gsa_grouped.cuh).
#include "gsa_grouped.cuh"

namespace gsa {
GSA_INST_GROUPED(cf64, int32_t)
}  // namespace gsa
