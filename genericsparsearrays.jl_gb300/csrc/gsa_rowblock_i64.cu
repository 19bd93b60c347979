// Row-block gather of Int64 values (gsa_rowblock.cuh).
#include "gsa_rowblock.cuh"

namespace gsa {
GSA_INST_RB(int64_t)
}  // namespace gsa
