// Grouped products of Int32 values (gsa_grouped.cuh).
#include "gsa_grouped.cuh"

namespace gsa {
GSA_INST_GROUPED(int32_t, int32_t)
GSA_INST_GROUPED(int32_t, int64_t)
}  // namespace gsa
