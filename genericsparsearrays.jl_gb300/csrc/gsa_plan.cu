// Plans (gsa_plan_create): the inspector over one compressed structure, run on the GPU.
//
// What a plan holds is described at gsa_plan (gsa_internal.cuh).  Making it is three passes over
// the row pointers, which they are bound by (8 B per row at most; 10^6 rows: tens of
// microseconds), with the few numbers per 2048 rows that set the sizes worked out on the host in
// between:
//   1. plan_stats_kernel: per 2048 rows the chunked rows and chunks of both sets; over all rows the
//      longest row and how much of the natural order's lanes would be busy; per segment the rows
//      of each bin.
//   2. the host sums the 2048-row counts into offsets and lays out groups and warps.
//   3. chunk_set_kernel writes a set's rows, chunks and mask; bin_order_kernel a segment's rows by
//      bin, stable, and its warps' groups.
// The same work on the host, one thread over a copy of the pointers, took 7.2 ms for 10^6 rows of
// power-law lengths (now 0.14) and 12.0 ms for the 4.2M rows of the 2048^2 grid (now 0.09) -- some
// hundred products of the matrix -- before the first product of every new matrix.
#include <algorithm>
#include <mutex>
#include <vector>

#include "gsa_rows.cuh"

namespace gsa {
namespace {

constexpr int PL_THREADS = 256;
constexpr int PL_WARPS = PL_THREADS / 32;
constexpr int64_t PL_ROWS = 2048;       // rows per CTA of the counting and chunk passes
constexpr int64_t PL_ALONE = 8192;      // up to as many rows one CTA takes them all
constexpr int64_t BIN_SEGMENT = 32768;  // rows per segment of the bin order
constexpr int BO_THREADS = 1024;
constexpr int BO_WARPS = BO_THREADS / 32;
static_assert(BIN_SEGMENT % PL_ROWS == 0 && PL_ALONE <= BIN_SEGMENT, "a counting CTA lies in one segment");
static_assert(BIN_SEGMENT % (32 * BO_WARPS) == 0, "a segment's warps take whole groups of 32 rows");

// Bin of a row of len <= CHUNK entries and its lanes per row: rows of equal length up to
// 32 (a lane each), then for 32 < len <= 512 the G = 2, 4, 8 or 16 lanes with 16 <
// ceil(len / G) <= 32 and one bin per value of ceil(len / G): every lane of a warp does
// the same number of multiply-adds, 17 to 32, before the width-G reduction.
constexpr int NBINS = 97;
__device__ __forceinline__ int bin_of(int len) {
    if (len <= 32) return len;
    const int lg = 27 - __clz(len - 1);  // G = 2^lg lanes, the fewest with 32 * G >= len
    const int q = (len + (1 << lg) - 1) >> lg;  // 17 .. 32
    return 33 + (lg - 1) * 16 + (q - 17);
}
int bin_lanes(int b) { return b <= 32 ? 1 : 1 << (1 + (b - 33) / 16); }

// Length of row r, its extent clamped to [0, nnz] (0 past the last row).
template <typename I>
__device__ __forceinline__ int64_t row_length(const I *__restrict__ ptr, int base, int64_t outer_n, int64_t nnz,
                                              int64_t r) {
    if (r >= outer_n) return 0;
    int64_t b = (int64_t)__ldg(ptr + r) - base, e = (int64_t)__ldg(ptr + r + 1) - base;
    b = b < 0 ? 0 : (b > nnz ? nnz : b);
    e = e < b ? b : (e > nnz ? nnz : e);
    return e - b;
}

// Whether set t (0 natural, 1 bin) cuts a row into chunks, the lengths of the warp's 32 rows
// known.  Natural order: longer than CHUNK, or longer than PLAN_LEN and more than 4x the average
// of its 32 rows (it would hold the warp's other rows back).  Bin order: longer than CHUNK.
__device__ __forceinline__ bool chunked(int t, int64_t len, int64_t sum32) {
    return len > (int64_t)CHUNK || (t == 0 && len > (int64_t)PLAN_LEN && 8 * len > sum32);
}

__device__ __forceinline__ int64_t warp_sum(int64_t v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

// Totals over all rows, zero before the pass.
struct PlanTotals {
    unsigned long long max_len, busy, held;
};
// Chunked rows and their chunks of one CTA's 2048 rows, per set.
struct PlanCount {
    unsigned long long rows[2], chunks[2];
};

// busy: entries the natural order's lanes sum; held: 32 x the iterations its warps make (G lanes
// per row from the average of the warp's unchunked rows, as warp_extent and dispatch_lanes pick
// it; each of the G passes lasts as long as its longest row).  hist: rows of each bin per segment.
template <typename I>
__global__ void __launch_bounds__(PL_THREADS)
plan_stats_kernel(int64_t outer_n, int64_t nnz, const I *__restrict__ ptr, int base, int64_t rows,
                  PlanTotals *__restrict__ totals,
                  PlanCount *__restrict__ counts, uint32_t *__restrict__ hist) {
    __shared__ uint32_t s_hist[NBINS];
    __shared__ unsigned long long s_sum[7];  // max_len, busy, held, rows[2], chunks[2]
    for (int b = threadIdx.x; b < NBINS; b += PL_THREADS) s_hist[b] = 0;
    if (threadIdx.x < 7) s_sum[threadIdx.x] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    int64_t longest = 0, busy = 0, held = 0, nrows[2] = {0, 0}, nchunks[2] = {0, 0};
    const int64_t r0 = (int64_t)blockIdx.x * rows;
#pragma unroll 4
    for (int64_t w0 = r0 + (threadIdx.x & ~31); w0 < r0 + rows; w0 += PL_THREADS) {
        if (w0 >= outer_n) break;  // the whole warp
        const int64_t len = row_length(ptr, base, outer_n, nnz, w0 + lane);
        longest = len > longest ? len : longest;
        const int64_t sum32 = warp_sum(len);
#pragma unroll
        for (int t = 0; t < 2; ++t)
            if (chunked(t, len, sum32)) {
                ++nrows[t];
                nchunks[t] += (len + CHUNK - 1) / CHUNK;
            }
        const unsigned l = chunked(0, len, sum32) ? 0u : (unsigned)len;
        const unsigned total = __reduce_add_sync(0xffffffffu, l);
        const unsigned avg = total >> 5;
        unsigned G = 1;
        while (G < 32u && avg > G * (unsigned)G1_AVG) G <<= 1;
        unsigned pass = l;  // the longest row of the pass this lane's row is in
        for (unsigned d = 1; d < 32u / G; d <<= 1) {
            const unsigned o = __shfl_xor_sync(0xffffffffu, pass, d);
            pass = o > pass ? o : pass;
        }
        const unsigned steps = (lane & (32u / G - 1)) == 0 ? (pass + G - 1) / G : 0u;
        held += __reduce_add_sync(0xffffffffu, steps);
        busy += total;
        if (w0 + lane < outer_n && len <= (int64_t)CHUNK) atomicAdd(&s_hist[bin_of((int)len)], 1u);
    }
    const int64_t all[4] = {warp_sum(nrows[0]), warp_sum(nrows[1]), warp_sum(nchunks[0]), warp_sum(nchunks[1])};
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        const int64_t o = __shfl_xor_sync(0xffffffffu, longest, d);
        longest = o > longest ? o : longest;
    }
    if (lane == 0) {
        atomicMax(&s_sum[0], (unsigned long long)longest);
        atomicAdd(&s_sum[1], (unsigned long long)busy);
        atomicAdd(&s_sum[2], 32ull * (unsigned long long)held);
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (all[t]) atomicAdd(&s_sum[3 + t], (unsigned long long)all[t]);
    }
    __syncthreads();
    // the only CTA writes its sums as they are: no clearing before it
    const bool alone = gridDim.x == 1;
    if (threadIdx.x == 0) {
        if (alone) {
            *totals = PlanTotals{s_sum[0], s_sum[1], s_sum[2]};
        } else {
            atomicMax(&totals->max_len, s_sum[0]);
            atomicAdd(&totals->busy, s_sum[1]);
            atomicAdd(&totals->held, s_sum[2]);
        }
        counts[blockIdx.x] = PlanCount{{s_sum[3], s_sum[4]}, {s_sum[5], s_sum[6]}};
    }
    uint32_t *h = hist + (r0 / BIN_SEGMENT) * NBINS;
    for (int b = threadIdx.x; b < NBINS; b += PL_THREADS) {
        if (alone) h[b] = s_hist[b];
        else if (s_hist[b]) atomicAdd(&h[b], s_hist[b]);
    }
}

// First chunked row and first chunk of each CTA's 2048 rows.
struct PlanFirst {
    int64_t row, chunk;
};

// One set's arrays as chunk_set_kernel writes them.
struct PlanSet {
    const PlanFirst *firsts;
    int64_t *row;
    int32_t *first, *count, *chunk_slot;
    uint32_t *mask;
};

// Rows, chunks and mask of set t = blockIdx.y, in row order: a CTA's 2048 rows in steps of 256, each
// step's places from a scan over the CTA's warps.
template <typename I>
__global__ void __launch_bounds__(PL_THREADS)
chunk_set_kernel(int64_t outer_n, int64_t nnz, const I *__restrict__ ptr, int base, int64_t rows, PlanSet natural,
                 PlanSet binned) {
    const int t = blockIdx.y;
    const PlanSet &set = t == 0 ? natural : binned;
    const PlanFirst *__restrict__ firsts = set.firsts;
    int64_t *__restrict__ row = set.row;
    int32_t *__restrict__ first = set.first, *__restrict__ count = set.count;
    int32_t *__restrict__ chunk_slot = set.chunk_slot;
    uint32_t *__restrict__ mask = set.mask;
    __shared__ int64_t s_rows[PL_WARPS], s_chunks[PL_WARPS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int64_t at_row = firsts[blockIdx.x].row, at_chunk = firsts[blockIdx.x].chunk;
    for (int64_t b0 = (int64_t)blockIdx.x * rows; b0 < (int64_t)(blockIdx.x + 1) * rows; b0 += PL_THREADS) {
        if (b0 >= outer_n) break;  // the whole CTA
        const int64_t w0 = b0 + 32 * w, r = w0 + lane;
        const int64_t len = row_length(ptr, base, outer_n, nnz, r);
        const bool in = chunked(t, len, warp_sum(len));
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (lane == 0 && w0 < outer_n) mask[w0 >> 5] = m;
        const int64_t nch = in ? (len + CHUNK - 1) / CHUNK : 0;
        int64_t x = nch;  // inclusive scan of the warp's chunks
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane == 31) {
            s_rows[w] = __popc(m);
            s_chunks[w] = x;
        }
        __syncthreads();
        int64_t rb = at_row, cb = at_chunk;
        for (int v = 0; v < PL_WARPS; ++v) {
            if (v < w) {
                rb += s_rows[v];
                cb += s_chunks[v];
            }
            at_row += s_rows[v];
            at_chunk += s_chunks[v];
        }
        const int64_t slot = rb + __popc(m & ((1u << lane) - 1)), c0 = cb + x - nch;
        if (in) {
            row[slot] = r;
            first[slot] = (int32_t)c0;
            count[slot] = (int32_t)nch;
        }
        for (unsigned todo = m; todo; todo &= todo - 1) {  // a row's chunks, by the whole warp
            const int l = __ffs(todo) - 1;
            const int64_t n = __shfl_sync(0xffffffffu, nch, l), c = __shfl_sync(0xffffffffu, c0, l);
            const int64_t sl = __shfl_sync(0xffffffffu, slot, l);
            for (int64_t q = lane; q < n; q += 32) chunk_slot[c + q] = (int32_t)sl;
        }
        __syncthreads();
    }
}

// A segment's first position of the order and first group.
struct PlanSegment {
    int64_t pos, group;
};

// CTA per segment: its rows of at most CHUNK entries by bin, stable -- each warp a range of
// consecutive rows, its first place in every bin from the warps' counts -- and the groups of its
// warps.  Bound by the latency of the segment's pointer reads and the ranks' shared-memory
// updates (a segment's CTA walks its rows twice).
template <typename I>
__global__ void __launch_bounds__(BO_THREADS)
bin_order_kernel(int64_t outer_n, int64_t nnz, const I *__restrict__ ptr, int base,
                 const PlanSegment *__restrict__ segs, const int64_t *__restrict__ groups, int64_t ngroups,
                 int64_t nwarps, int32_t *__restrict__ perm, int32_t *__restrict__ warp_group) {
    __shared__ uint32_t s_at[BO_WARPS][NBINS];  // rows of the warp's range in the bin, then their places
    __shared__ uint32_t s_bin[NBINS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < BO_WARPS * NBINS; i += BO_THREADS) (&s_at[0][0])[i] = 0;
    __syncthreads();
    const int64_t s0 = (int64_t)blockIdx.x * BIN_SEGMENT;
    const int64_t a0 = s0 + w * (BIN_SEGMENT / BO_WARPS), a1 = a0 + BIN_SEGMENT / BO_WARPS;
#pragma unroll 4
    for (int64_t r = a0 + lane; r < a1; r += 32) {
        const int64_t len = row_length(ptr, base, outer_n, nnz, r);
        if (r < outer_n && len <= (int64_t)CHUNK) atomicAdd(&s_at[w][bin_of((int)len)], 1u);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < NBINS; b += BO_THREADS) {
        uint32_t n = 0;
        for (int v = 0; v < BO_WARPS; ++v) n += s_at[v][b];
        s_bin[b] = n;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t run = 0;
        for (int b = 0; b < NBINS; ++b) {
            const uint32_t n = s_bin[b];
            s_bin[b] = run;
            run += n;
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < NBINS; b += BO_THREADS) {
        uint32_t run = s_bin[b];
        for (int v = 0; v < BO_WARPS; ++v) {
            const uint32_t n = s_at[v][b];
            s_at[v][b] = run;
            run += n;
        }
    }
    __syncthreads();
    const int64_t pos = segs[blockIdx.x].pos;
#pragma unroll 2
    for (int64_t r = a0 + lane; r < a1; r += 32) {
        const int64_t len = row_length(ptr, base, outer_n, nnz, r);
        const bool in = r < outer_n && len <= (int64_t)CHUNK;
        const int b = in ? bin_of((int)len) : NBINS;
        const unsigned same = __match_any_sync(0xffffffffu, b);
        if (in) {
            const uint32_t at = s_at[w][b];
            perm[pos + at + __popc(same & ((1u << lane) - 1))] = (int32_t)r;
        }
        __syncwarp();
        if (in && lane == __ffs(same) - 1) s_at[w][b] += __popc(same);
        __syncwarp();
    }
    const int64_t g1 = blockIdx.x + 1 < gridDim.x ? segs[blockIdx.x + 1].group : ngroups;
    for (int64_t g = segs[blockIdx.x].group; g < g1; ++g) {
        const int64_t w1 = g + 1 < ngroups ? groups[4 * (g + 1)] : nwarps;
        for (int64_t q = groups[4 * g] + threadIdx.x; q < w1; q += BO_THREADS) warp_group[q] = (int32_t)g;
    }
}

// Host memory that a kernel writes its few counts to: a page that a call has to itself, taken from
// and returned to a list of the process (no page is freed when a thread ends: that is not allowed
// while another thread captures a stream, and would end its capture).  At most MAX_BOXES pages exist;
// p is NULL where none can be had.
constexpr size_t COUNT_BOX = 4096;
constexpr int MAX_BOXES = 64;
std::mutex g_boxes_lock;
char *g_boxes[MAX_BOXES];
int g_boxes_free = 0, g_boxes_made = 0;
struct CountBox {
    char *p = nullptr;
    bool take() {
        std::unique_lock<std::mutex> hold(g_boxes_lock);
        if (g_boxes_free > 0) {
            p = g_boxes[--g_boxes_free];
        } else if (g_boxes_made < MAX_BOXES) {
            ++g_boxes_made;
            hold.unlock();
            void *q = nullptr;
            if (cudaHostAlloc(&q, COUNT_BOX, cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
                p = (char *)q;
            } else {
                cudaGetLastError();
                hold.lock();
                --g_boxes_made;
            }
        }
        return p != nullptr;
    }
    ~CountBox() {
        if (!p) return;
        std::lock_guard<std::mutex> hold(g_boxes_lock);
        g_boxes[g_boxes_free++] = p;
    }
};

template <typename I>
int build_plan(cudaStream_t s, int64_t outer_n, int64_t nnz, const I *ptr, int base, Plan *p) {
    p->outer_n = outer_n;
    p->nnz = nnz;
    const int64_t rows = outer_n <= PL_ALONE ? PL_ALONE : PL_ROWS;
    const int64_t nct = ceil_div(outer_n, rows), nseg = ceil_div(outer_n, BIN_SEGMENT);
    if (nct > 0x7fffffffLL) return fail(GSA_ERR_UNSUPPORTED, "plan: too many outer entries");
    if (outer_n == 0) {  // nothing to launch: a plan of no rows (the stream is synchronized as ever)
        return check_cuda(cudaStreamSynchronize(s), "plan: sync");
    }
    // 1. counts
    Carver sc(nullptr);
    const size_t o_tot = sc.reserve<PlanTotals>(1), o_hist = sc.reserve<uint32_t>((size_t)(nseg * NBINS));
    const size_t zeroed = sc.off;
    const size_t o_cnt = sc.reserve<PlanCount>((size_t)nct);
    const size_t bytes1 = sc.off;
    std::vector<char> copied;
    CountBox box;
    const char *got = nullptr;
    auto count = [&](char *d) {
        plan_stats_kernel<I><<<(unsigned)nct, PL_THREADS, 0, s>>>(outer_n, nnz, ptr, base, rows, (PlanTotals *)(d + o_tot),
                                                                  (PlanCount *)(d + o_cnt), (uint32_t *)(d + o_hist));
        return check_cuda(cudaGetLastError(), "plan_stats_kernel");
    };
    if (nct == 1 && bytes1 <= COUNT_BOX && box.take()) {
        // one CTA: its sums go straight to host memory, without scratch and a copy (30 us a plan with)
        got = box.p;
        int rc = count(box.p);
        if (!rc) rc = check_cuda(cudaStreamSynchronize(s), "plan: sync");
        if (rc) return rc;
    } else {
        copied.resize(bytes1);
        Workspace tmp;
        int rc = tmp.acquire(s, nullptr, 0, bytes1);
        if (rc) return rc;
        char *d = (char *)tmp.p;
        if (nct > 1) rc = check_cuda(cudaMemsetAsync(d, 0, zeroed, s), "plan: clear");
        if (!rc) rc = count(d);
        if (!rc) rc = check_cuda(cudaMemcpyAsync(copied.data(), d, bytes1, cudaMemcpyDeviceToHost, s), "plan: counts");
        if (!rc) rc = check_cuda(cudaStreamSynchronize(s), "plan: sync");
        if (rc) return rc;
        got = copied.data();
    }
    const PlanTotals &tot = *(const PlanTotals *)(got + o_tot);
    const uint32_t *hist = (const uint32_t *)(got + o_hist);
    const PlanCount *cnt = (const PlanCount *)(got + o_cnt);
    p->max_len = (int64_t)tot.max_len;
    // bin order when the natural one would leave over a tenth of the lanes idle (only
    // FP64-bound products use it, where every idle lane is lost FP64 time)
    const double utilisation = tot.held > 0 ? (double)tot.busy / (double)tot.held : 1.0;
    const bool binned = outer_n >= 32 && outer_n <= 0x7fffffffLL && utilisation < 0.9;
    // 2. offsets, groups and warps
    std::vector<PlanFirst> firsts[2];
    int64_t nlong[2] = {0, 0}, nchunks[2] = {0, 0};
    for (int t = 0; t < (binned ? 2 : 1); ++t) {
        firsts[t].resize((size_t)nct);
        for (int64_t b = 0; b < nct; ++b) {
            firsts[t][(size_t)b] = PlanFirst{nlong[t], nchunks[t]};
            nlong[t] += (int64_t)cnt[b].rows[t];
            nchunks[t] += (int64_t)cnt[b].chunks[t];
            if (nchunks[t] > 0x7fffffffLL) return fail(GSA_ERR_UNSUPPORTED, "plan: too many chunks");
        }
    }
    std::vector<PlanSegment> segs;
    std::vector<int64_t> groups;
    int64_t npos = 0, nwarps = 0;
    if (binned) {
        segs.resize((size_t)nseg);
        for (int64_t sg = 0; sg < nseg; ++sg) {
            const uint32_t *h = hist + sg * NBINS;
            segs[(size_t)sg] = PlanSegment{npos, (int64_t)groups.size() / 4};
            // one group per lanes-per-row class: its bins are consecutive, so its rows are
            // sorted by the work of each lane and a warp's 32 / G rows have equal or
            // adjacent lengths (one partial warp per class and segment, not per bin)
            for (int b0 = 0; b0 < NBINS;) {
                const int G = bin_lanes(b0);
                int64_t rows = 0;
                int b1 = b0;
                for (; b1 < NBINS && bin_lanes(b1) == G; ++b1) rows += h[b1];
                if (rows > 0) {
                    if (groups.size() / 4 > 0x7fffffffLL) return fail(GSA_ERR_UNSUPPORTED, "plan: too many bin groups");
                    groups.insert(groups.end(), {nwarps, npos, npos + rows, (int64_t)G});
                    nwarps += ceil_div(rows, 32 / G);
                    npos += rows;
                }
                b0 = b1;
            }
        }
    }
    p->nbin_warps = nwarps;
    p->nplanned = binned ? outer_n : nlong[0];
    if (p->nplanned == 0) return GSA_OK;
    // 3. the plan's arrays: what the host made (one upload), then what the kernels write
    const size_t nmask = (size_t)ceil_div(outer_n, 32);
    Carver up(nullptr);
    const size_t o_groups = up.reserve<int64_t>(groups.size()), o_segs = up.reserve<PlanSegment>(segs.size());
    size_t o_first[2] = {0, 0};
    for (int t = 0; t < 2; ++t) o_first[t] = up.reserve<PlanFirst>(firsts[t].size());
    const size_t o_view = up.reserve<gsa_bin_order>(1);
    const size_t uploaded = up.off;
    size_t o_row[2], o_cfirst[2], o_count[2], o_slot[2], o_mask[2];
    for (int t = 0; t < 2; ++t) {
        o_row[t] = up.reserve<int64_t>((size_t)nlong[t]);
        o_cfirst[t] = up.reserve<int32_t>((size_t)nlong[t]);
        o_count[t] = up.reserve<int32_t>((size_t)nlong[t]);
        o_slot[t] = up.reserve<int32_t>((size_t)nchunks[t]);
        o_mask[t] = up.reserve<uint32_t>(nmask);
    }
    const size_t o_perm = up.reserve<int32_t>((size_t)npos), o_wg = up.reserve<int32_t>((size_t)nwarps);
    int rc = check_cuda(scratch_alloc(&p->mem, align_up(up.off, 256), s), "plan: device memory");
    if (rc) return rc;
    char *d = (char *)p->mem;
    std::vector<char> host(uploaded, 0);
    auto put = [&](size_t at, const void *src, size_t n) {
        if (n) memcpy(host.data() + at, src, n);
    };
    put(o_groups, groups.data(), groups.size() * sizeof(int64_t));
    put(o_segs, segs.data(), segs.size() * sizeof(PlanSegment));
    for (int t = 0; t < 2; ++t) put(o_first[t], firsts[t].data(), firsts[t].size() * sizeof(PlanFirst));
    if (binned) {
        p->order = gsa_bin_order{nwarps, (const int32_t *)(d + o_perm), (const int32_t *)(d + o_wg),
                                 (const int64_t *)(d + o_groups)};
        put(o_view, &p->order, sizeof(gsa_bin_order));
    }
    rc = check_cuda(cudaMemcpyAsync(d, host.data(), uploaded, cudaMemcpyHostToDevice, s), "plan: upload");
    if (rc) return rc;
    PlanSet sets[2];
    for (int t = 0; t < 2; ++t) {
        sets[t] = PlanSet{(const PlanFirst *)(d + o_first[t]), (int64_t *)(d + o_row[t]), (int32_t *)(d + o_cfirst[t]),
                          (int32_t *)(d + o_count[t]), (int32_t *)(d + o_slot[t]), (uint32_t *)(d + o_mask[t])};
        gsa_chunk_set &c = t == 0 ? p->nat : p->bin;
        c.nlong = nlong[t];
        c.nchunks = nchunks[t];
        c.row = sets[t].row;
        c.first = sets[t].first;
        c.count = sets[t].count;
        c.chunk_slot = sets[t].chunk_slot;
        c.skip_mask = sets[t].mask;
    }
    chunk_set_kernel<I><<<dim3((unsigned)nct, binned ? 2 : 1), PL_THREADS, 0, s>>>(outer_n, nnz, ptr, base, rows, sets[0],
                                                                                  sets[1]);
    rc = check_cuda(cudaGetLastError(), "chunk_set_kernel");
    if (rc) return rc;
    if (binned) {
        bin_order_kernel<I><<<(unsigned)nseg, BO_THREADS, 0, s>>>(
            outer_n, nnz, ptr, base, (const PlanSegment *)(d + o_segs), (const int64_t *)(d + o_groups),
            (int64_t)groups.size() / 4, nwarps, (int32_t *)(d + o_perm), (int32_t *)(d + o_wg));
        rc = check_cuda(cudaGetLastError(), "bin_order_kernel");
        if (rc) return rc;
        p->bin_view = (const gsa_bin_order *)(d + o_view);
    }
    // the plan may be used on any stream from here on (and `host` leaves scope)
    return check_cuda(cudaStreamSynchronize(s), "plan: sync");
}

}  // namespace

int plan_create(cudaStream_t s, int itype, int64_t outer_n, int64_t nnz, const void *ptr, int base, Plan *p) {
    if (itype == GSA_IDX32) return build_plan<int32_t>(s, outer_n, nnz, (const int32_t *)ptr, base, p);
    return build_plan<int64_t>(s, outer_n, nnz, (const int64_t *)ptr, base, p);
}

}  // namespace gsa
