// Row-block gather of ComplexF64 values (gsa_rowblock.cuh).
#include "gsa_rowblock.cuh"

namespace gsa {
GSA_INST_RB(cf64)
}  // namespace gsa
