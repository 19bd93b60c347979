// Row-block gather of Float32 values (gsa_rowblock.cuh).
#include "gsa_rowblock.cuh"

namespace gsa {
GSA_INST_RB(float)
}  // namespace gsa
