// Grouped products of Int64 values (gsa_grouped.cuh).
#include "gsa_grouped.cuh"

namespace gsa {
GSA_INST_GROUPED(int64_t, int32_t)
GSA_INST_GROUPED(int64_t, int64_t)
}  // namespace gsa
