// Row-block gather of Int32 values (gsa_rowblock.cuh).
#include "gsa_rowblock.cuh"

namespace gsa {
GSA_INST_RB(int32_t)
}  // namespace gsa
