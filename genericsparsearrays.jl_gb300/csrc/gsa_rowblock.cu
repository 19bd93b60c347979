// Row-block gather: the parts that no value type has of its own -- tuning knobs and workspace
// sizes (kernels: gsa_rowblock.cuh).
#include <atomic>

#include "gsa_rows.cuh"

namespace gsa {

// Process-wide tuning knobs: atomics, since any host thread may set them while others launch.
static std::atomic<int> g_spmm_columns{0};  // 0: by value size
void set_spmm_columns(int c) { g_spmm_columns.store(c, std::memory_order_relaxed); }
int get_spmm_columns() { return g_spmm_columns.load(std::memory_order_relaxed); }
static std::atomic<int> g_plan_order{0};    // 0: the plan's choice, 1: natural order always
void set_plan_natural(int v) { g_plan_order.store(v, std::memory_order_relaxed); }
int get_plan_natural() { return g_plan_order.load(std::memory_order_relaxed); }

static std::atomic<int> g_x_pairs{1};
void set_x_pairs(int v) { g_x_pairs.store(v, std::memory_order_relaxed); }
int get_x_pairs() { return g_x_pairs.load(std::memory_order_relaxed); }

static std::atomic<int> g_stage_rows{0};
void set_stage_rows(int v) { g_stage_rows.store(v, std::memory_order_relaxed); }
int get_stage_rows() { return g_stage_rows.load(std::memory_order_relaxed); }

size_t rowblock_workspace_size(const Plan *plan, size_t vsize, int64_t k) {
    if (!plan || k == 0) return 0;
    // enough for either chunk set; ncg <= k for any KC
    const int64_t nlong = plan->nat.nlong > plan->bin.nlong ? plan->nat.nlong : plan->bin.nlong;
    const int64_t nchunks = plan->nat.nchunks > plan->bin.nchunks ? plan->nat.nchunks : plan->bin.nchunks;
    if (nlong == 0) return 0;
    Carver cv(nullptr);
    cv.take<int>((size_t)(nlong * k));
    cv.take<unsigned char>((size_t)(nchunks * k) * vsize + 16);
    return align_up(cv.off, 256);
}

}  // namespace gsa
