// Row-block gather of Float64 values (gsa_rowblock.cuh).
#include "gsa_rowblock.cuh"

namespace gsa {
GSA_INST_RB(double)
}  // namespace gsa
