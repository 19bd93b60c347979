// Grouped products of Float64 values (gsa_grouped.cuh).
#include "gsa_grouped.cuh"

namespace gsa {
GSA_INST_GROUPED(double, int32_t)
GSA_INST_GROUPED(double, int64_t)
}  // namespace gsa
