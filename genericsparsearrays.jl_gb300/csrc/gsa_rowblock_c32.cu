// Row-block gather of ComplexF32 values (gsa_rowblock.cuh).
#include "gsa_rowblock.cuh"

namespace gsa {
GSA_INST_RB(cf32)
}  // namespace gsa
