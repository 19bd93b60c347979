// Row-block gather: C[o, c] = beta*C[o, c] + alpha * sum_j a_j * op(B)(idx_j, c)
// -- kernel_spmatmul_csr_N! (src/matrix_csr/matrix_csr_kernels.jl:1-22) and
// kernel_spmatmul_csc_T! (src/matrix_csc/matrix_csc_kernels.jl:24-45).
//
// Each CTA of 128 threads owns 128 consecutive outer entries (rows) and one group
// of KC right-hand-side columns; each warp owns 32 of the rows.  From the average
// length of its 32 rows a warp picks G lanes per row (1, 2, ..., 32): a thread
// per row for short rows -- plain loads straight from HBM, where neighbouring
// threads read neighbouring entries so a warp's loads share cache lines, and
// tens of thousands of small CTAs keep enough loads in flight to cover DRAM
// latency without staging -- and groups of G lanes reading consecutive entries
// (coalesced) for longer ones, in G passes over the warp's rows.  For SpMM the
// CTAs of one row block and its column groups are numbered consecutively, so
// they run together and share the row block's entries through L2.
//
// Longer rows, with a plan (gsa_plan_create): the plan lists every row of more
// than CHUNK entries and every row of more than PLAN_LEN entries that is over 4x
// its warp's average, cut into chunks of CHUNK entries; extra CTAs give each
// chunk to one warp (32 lanes, UNROLL loads each in flight).  A row of one chunk
// is summed and stored by its warp; for a longer one each warp stores a partial
// sum, and the warp that completes the row's last chunk adds the partials in chunk
// order and writes the row.  A warp of short rows thus never waits on a long one.
// Without a plan such a row is one group's work like any other.
//
// Every row's summation order is fixed, so results are deterministic.
//
// One source file per value type instantiates this (they compile in parallel).
#pragma once


#include "gsa_rows.cuh"

namespace gsa {

// Resident CTAs per SM the compiler must allow: the one-column kernels of 4- and 8-byte
// values are latency-bound gathers whose speed follows the warps in flight, so they are
// held to 32 registers (16 CTAs of 128 threads, every warp slot of the SM).  So are, less tightly,
// the kernels of many columns of a column-major B, whose loads in flight otherwise take up to 128
// registers (2048^2 grid; us unbounded / held): Float32 KC = 16 at 48 registers 250 / 161 (64: 167),
// KC = 5 to 8 at 48 (KC = 8: 270 / 205), KC = 2 at 40 66 / 59 (32 registers spill: Poisson(10) rows 87
// against 81), ComplexF32 KC = 5 to 8 at 64 (KC = 8: 202 / 168; KC = 6, which the compiler gave 45 and
// loads one after another, on the 1024^2 grid 56 / 39).  Two 4-byte columns of a row-major B take 48
// (32, which the two-stride code fitted, spill 184 bytes: power law, n = 2*10^5, 36 us against 34; rows of 40
// 26 against 22).  Float64 KC = 8, taken for longer rows, is the faster unbounded
// (Poisson(10) rows 383 against 453).  0 leaves the register count to the compiler.
#ifndef GSA_RB_MIN_BLOCKS
#define GSA_RB_MIN_BLOCKS 16
#endif
template <typename V, int KC, int LAY> constexpr int rb_min_blocks() {
    if (KC == 1 && sizeof(V) <= 8) return GSA_RB_MIN_BLOCKS;
    if (LAY == ROWS && KC == 2 && sizeof(V) == 4) return 10;
    if (LAY != COLUMNS) return 0;
    if (sizeof(V) == 4) return KC >= 5 ? 10 : (KC == 2 ? 12 : 0);
    return std::is_same<V, cf32>::value && KC >= 5 ? 8 : 0;
}
// The bin order's ComplexF64 SpMV is held to 8 resident CTAs, which lets the compiler keep 64
// registers (48 without the bound) and more loads in flight: power-law n = 10^6 160 us against
// 170 us on one GB300 (12 CTAs at 40 registers: 177 us, 10 at 48: 167 us, 7 at 72: 163 us, 6 at
// 74: 169 us, 5 at 88: 178 us); the grouped kernel gained nothing from the same bounds.
#ifndef GSA_BINNED_C64_MIN_BLOCKS
#define GSA_BINNED_C64_MIN_BLOCKS 8
#endif
template <typename V, int KC, int LAY> constexpr int binned_min_blocks() {
    return std::is_same<V, cf64>::value && KC == 1 ? GSA_BINNED_C64_MIN_BLOCKS : rb_min_blocks<V, KC, LAY>();
}

// The bin order pays where the FP64 pipe binds: ComplexF64 products (four FMAs per entry)
// and Float64 products with several right-hand sides (one FMA per entry and column); a
// Float64 SpMV is HBM-bound, and there the scattered rows cost more traffic than idle lanes
// cost time (Poisson(10), 2M rows: 112 us natural vs 226 us binned).
template <typename V> constexpr bool bins_possible() {
    return std::is_same<V, cf64>::value || std::is_same<V, double>::value;
}
template <typename V> inline bool bins_pay(int64_t k) {
    return std::is_same<V, cf64>::value || (std::is_same<V, double>::value && k > 1);
}

// One warp sums chunk `chunk` of a chunked row (entries [jb, je), 32 lanes, UNROLL loads
// each in flight).  A row of one chunk is stored at once; otherwise the warp stores its
// partial sum, and the warp that completes the row's last chunk adds the partials in
// chunk order and writes the row.
template <typename V, typename I, int KC, int LAY>
__device__ __forceinline__ void chunk_unit(const CompressedArgs<V, I> &a, int64_t k, const DenseIn<V> &B,
                                           const DenseOut<V> &C, int64_t c0, unsigned cg, int64_t ncg,
                                           int64_t chunk, const PlanRows &L) {
    using O = Off<I>;
    const int lane = threadIdx.x & 31;
    if (chunk >= L.nchunks) return;
    const int slot = L.chunk_slot[chunk];
    const int64_t row = L.row[slot];
    const int nch = L.count[slot];
    const O nz = (O)a.nnz, base = (O)a.base;
    O rb = (O)__ldg(a.ptr + row) - base;
    O re = (O)__ldg(a.ptr + row + 1) - base;
    rb = rb < nz ? rb : nz;
    re = re < nz ? re : nz;
    const O jb = rb + (O)(chunk - L.first[slot]) * (O)CHUNK;
    const O je = jb < re && re - jb > (O)CHUNK ? jb + (O)CHUNK : re;
    V acc[KC];
#pragma unroll
    for (int c = 0; c < KC; ++c) acc[c] = VT<V>::zero();
    if (jb < je) accumulate_range<V, I, KC, 32, UNROLL, LAY>(a, B, jb + (O)lane, je, c0, k, acc);
#pragma unroll
    for (int c = 0; c < KC; ++c) {
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) acc[c] = add(acc[c], shfl_xor(acc[c], m));
    }
    if (nch == 1) {  // the whole row: store it
        if (lane == 0) {
#pragma unroll
            for (int c = 0; c < KC; ++c)
                if (c0 + c < k) C.store(row, c0 + c, acc[c]);
        }
        return;
    }
    V *part = reinterpret_cast<V *>(L.partial);
    int last = 0;
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < KC; ++c)
            if (c0 + c < k) part[chunk * k + c0 + c] = acc[c];
        __threadfence();
        const int prev = atomicAdd(&L.done[slot * ncg + cg], 1);
        last = prev == nch - 1;
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    if (!last) return;
    // the row's last chunk: add the partials in chunk order
    __threadfence();
    if (lane == 0) {
        const int f = L.first[slot];
#pragma unroll
        for (int c = 0; c < KC; ++c) {
            if (c0 + c >= k) continue;
            V t = VT<V>::zero();
            for (int q = 0; q < nch; ++q) t = add(t, ld_coherent(part + (int64_t)(f + q) * k + c0 + c));
            C.store(row, c0 + c, t);
        }
        L.done[slot * ncg + cg] = 0;
    }
}

template <typename V, typename I, int KC, int LAY>
__global__ void __launch_bounds__(RB_THREADS, rb_min_blocks<V, KC, LAY>())
rowblock_kernel(CompressedArgs<V, I> a, int64_t k, DenseIn<V> B, DenseOut<V> C, int64_t ncg,
                int64_t nrb, PlanRows L) {
    // column group fastest; one group (SpMV) needs no division
    const unsigned cta = blockIdx.x;
    const unsigned cg = ncg == 1 ? 0u : cta % (unsigned)ncg;
    const int64_t unit = ncg == 1 ? (int64_t)cta : (int64_t)(cta / (unsigned)ncg);
    const int64_t c0 = (int64_t)cg * KC;
    if (unit >= nrb) {  // chunked rows: a warp per chunk
        chunk_unit<V, I, KC, LAY>(a, k, B, C, c0, cg, ncg, (unit - nrb) * RB_WARPS + (threadIdx.x >> 5), L);
        return;
    }
    // ---- this warp's 32 rows
    warp_unit<V, I, KC, LAY>(a, k, B, C, c0, unit * RB_THREADS + (threadIdx.x & ~31), L.skip_mask);
}

// ---------------------------------------------------------------------------
// Staged rows (GSA_TUNE_STAGE_ROWS = 1; one right-hand side, Float32 or Float64 values, Int32
// indices): the entries of a warp's 32 thread-per-row rows are one contiguous span, which the
// warp copies into shared memory with 16-byte loads -- a lane moves whole 16-byte pieces of
// idx and val, two or three warp instructions where the direct path issues one scalar load
// per entry and lane -- before each lane sums its own row from shared memory.  Warps whose
// rows take several lanes, spans longer than STAGE_CAP entries, spans whose 16-byte pieces
// would pass the end of the arrays and arrays that are not 16-byte aligned take the direct
// path of rowblock_kernel.  Each row is summed in the same order as there (bit-identical).
constexpr int STAGE_CAP = 256;

template <typename V> constexpr bool stage_rows_type() {
    return std::is_same<V, float>::value || std::is_same<V, double>::value;
}

// 12 resident CTAs of 128 threads: 40 registers, and 96 KB (Float32) or 144 KB (Float64) of
// staging per SM
template <typename V, typename I>
__global__ void __launch_bounds__(RB_THREADS, 12)
rowblock_staged_kernel(CompressedArgs<V, I> a, DenseIn<V> B, DenseOut<V> C, int64_t nrb, PlanRows L) {
    static_assert(sizeof(I) == 4, "staged rows take 32-bit offsets");
    constexpr int PIECE = 4;  // entries per 16 bytes of indices (and the unit of the span's ends)
    __shared__ __align__(16) I s_idx[RB_WARPS][STAGE_CAP];
    __shared__ __align__(16) V s_val[RB_WARPS][STAGE_CAP];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t unit = blockIdx.x;
    if (unit >= nrb) {  // chunked rows: a warp per chunk
        chunk_unit<V, I, 1, COLUMNS>(a, 1, B, C, 0, 0u, 1, (unit - nrb) * RB_WARPS + w, L);
        return;
    }
    const int64_t row0 = unit * RB_THREADS + (threadIdx.x & ~31);
    if (row0 >= a.outer_n) return;  // a warp past the last row (uniform: the whole warp leaves)
    uint32_t b, e;
    int skip;
    const int64_t avg = warp_extent(a, row0, L.skip_mask, b, e, skip);
    // lane 0's row exists, so the span [S, E) covers at least one row: S <= b_0 <= e_0 <= E
    const bool valid = row0 + lane < a.outer_n;
    const uint32_t S = __reduce_min_sync(0xffffffffu, valid ? b : 0xffffffffu) & ~(uint32_t)(PIECE - 1);
    const uint32_t E = __reduce_max_sync(0xffffffffu, valid ? e : 0u);
    const uint32_t T = (E + PIECE - 1) & ~(uint32_t)(PIECE - 1);
    if (avg > G1_AVG || T < S || T - S > (uint32_t)STAGE_CAP || (int64_t)T > a.nnz) {
        dispatch_lanes(avg, G1_AVG, [&](auto g) {
            warp_rows<V, I, 1, decltype(g)::value, COLUMNS>(a, 1, B, C, 0, row0, b, e, skip);
        });
        return;
    }
    // the span [S, T) in 16-byte pieces
    const int4 *gi = reinterpret_cast<const int4 *>(a.idx + S);
    int4 *si = reinterpret_cast<int4 *>(&s_idx[w][0]);
    for (uint32_t q = lane; q < (T - S) / PIECE; q += 32) si[q] = __ldcs(gi + q);
    constexpr int VPIECE = 16 / sizeof(V);
    using V4 = typename std::conditional<sizeof(V) == 4, float4, double2>::type;
    const V4 *gv = reinterpret_cast<const V4 *>(a.val + S);
    V4 *sv = reinterpret_cast<V4 *>(&s_val[w][0]);
    for (uint32_t q = lane; q < (T - S) / VPIECE; q += 32) sv[q] = __ldcs(gv + q);
    __syncwarp();
    const uint32_t inner = a.inner_n < 0xffffffffLL ? (uint32_t)a.inner_n : 0xffffffffu;
    const uint32_t base = (uint32_t)a.base;
    V acc = VT<V>::zero();
    uint32_t j = b - S;
    const uint32_t je = e - S;
    for (; j + 3 < je; j += 4) {  // four gathers in flight
        uint32_t ci[4];
        V av[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            ci[u] = (uint32_t)s_idx[w][j + u] - base;
            av[u] = s_val[w][j + u];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) acc = mac(acc, av[u], ci[u] < inner ? B.at((int64_t)ci[u], 0) : VT<V>::zero());
    }
    for (; j < je; ++j) {
        const uint32_t c1 = (uint32_t)s_idx[w][j] - base;
        acc = mac(acc, s_val[w][j], c1 < inner ? B.at((int64_t)c1, 0) : VT<V>::zero());
    }
    if (valid && !skip) C.store(row0 + lane, 0, acc);
}

// Vector rows (GSA_TUNE_STAGE_ROWS = 2; same types as the staged rows): each lane of a
// thread-per-row warp reads its own row's indices and values in aligned 16-byte pieces
// straight into registers -- one 16-byte index load and one or two value loads per four
// entries, where the direct path issues a scalar load per entry and array -- and multiplies the
// entries of each piece that lie in its row, in order (bit-identical to the direct path).  A
// lane whose last piece would pass the end of the arrays uses scalar loads.
template <typename V, typename I>
__global__ void __launch_bounds__(RB_THREADS, rb_min_blocks<V, 1, COLUMNS>())
rowblock_vec_kernel(CompressedArgs<V, I> a, DenseIn<V> B, DenseOut<V> C, int64_t nrb, PlanRows L) {
    static_assert(sizeof(I) == 4, "vector rows take 32-bit offsets");
    const int w = threadIdx.x >> 5;
    const int64_t unit = blockIdx.x;
    if (unit >= nrb) {  // chunked rows: a warp per chunk
        chunk_unit<V, I, 1, COLUMNS>(a, 1, B, C, 0, 0u, 1, (unit - nrb) * RB_WARPS + w, L);
        return;
    }
    const int64_t row0 = unit * RB_THREADS + (threadIdx.x & ~31);
    if (row0 >= a.outer_n) return;  // a warp past the last row (uniform)
    uint32_t b, e;
    int skip;
    const int64_t avg = warp_extent(a, row0, L.skip_mask, b, e, skip);
    if (avg > G1_AVG) {
        dispatch_lanes(avg, G1_AVG, [&](auto g) {
            warp_rows<V, I, 1, decltype(g)::value, COLUMNS>(a, 1, B, C, 0, row0, b, e, skip);
        });
        return;
    }
    const int lane = threadIdx.x & 31;
    const uint32_t inner = a.inner_n < 0xffffffffLL ? (uint32_t)a.inner_n : 0xffffffffu;
    const uint32_t base = (uint32_t)a.base;
    V acc = VT<V>::zero();
    if ((int64_t)((e + 3u) & ~3u) <= a.nnz) {
#pragma unroll 2
        for (uint32_t c = b & ~3u; c < e; c += 4) {
            const int4 iv = __ldcs(reinterpret_cast<const int4 *>(a.idx + c));
            V v[4];
            if constexpr (sizeof(V) == 4) {
                const float4 f = __ldcs(reinterpret_cast<const float4 *>(a.val + c));
                v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
            } else {
                const double2 d0 = __ldcs(reinterpret_cast<const double2 *>(a.val + c));
                const double2 d1 = __ldcs(reinterpret_cast<const double2 *>(a.val + c + 2));
                v[0] = d0.x; v[1] = d0.y; v[2] = d1.x; v[3] = d1.y;
            }
            const uint32_t ci[4] = {(uint32_t)iv.x - base, (uint32_t)iv.y - base, (uint32_t)iv.z - base,
                                    (uint32_t)iv.w - base};
            V x[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const bool in = c + t >= b && c + t < e;
                x[t] = in && ci[t] < inner ? B.at((int64_t)ci[t], 0) : VT<V>::zero();
            }
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (c + t >= b && c + t < e) acc = mac(acc, v[t], x[t]);
        }
    } else {
        for (uint32_t j = b; j < e; ++j) {
            const uint32_t c1 = (uint32_t)a.idx[j] - base;
            acc = mac(acc, a.val[j], c1 < inner ? B.at((int64_t)c1, 0) : VT<V>::zero());
        }
    }
    if (row0 + lane < a.outer_n && !skip) C.store(row0 + lane, 0, acc);
}


// ---------------------------------------------------------------------------
// Bin order: within each segment of BIN_SEGMENT rows the plan sorts the rows by the
// multiply-adds each of their lanes does (rows up to 32 entries with a lane each, longer
// ones with G = 2, 4, 8 or 16 lanes, each lane 17 to 32 entries) and warp w of the order
// takes 32 / G consecutive rows of one lanes-per-row class of one segment.  The lanes of a
// warp then do the same number of multiply-adds, or one apart: FP64 products on GB300 are
// bound by the FP64 pipe, which counts a warp instruction whole however few of its lanes
// are active.  A segment's rows are read close together in time, so the sectors that
// neighbouring rows share are still in L2 when the second of them is read.

template <typename V, typename I, int KC, int LAY>
__global__ void __launch_bounds__(RB_THREADS, binned_min_blocks<V, KC, LAY>())
binned_kernel(CompressedArgs<V, I> a, int64_t k, DenseIn<V> B, DenseOut<V> C, int64_t ncg, gsa_bin_order bv,
              PlanRows L) {
    const unsigned cta = blockIdx.x;
    const unsigned cg = ncg == 1 ? 0u : cta % (unsigned)ncg;
    const int64_t unit = ncg == 1 ? (int64_t)cta : (int64_t)(cta / (unsigned)ncg);
    const int64_t c0 = (int64_t)cg * KC;
    const int64_t w = unit * RB_WARPS + (threadIdx.x >> 5);
    if (w >= bv.nwarps) {  // chunked rows
        chunk_unit<V, I, KC, LAY>(a, k, B, C, c0, cg, ncg, w - bv.nwarps, L);
        return;
    }
    binned_warp<V, I, KC, LAY>(a, k, B, C, c0, w, bv);
}

constexpr size_t WIDE_B_BYTES = (size_t)96 << 20;  // of the 129 MB L2: a B that stays there beside the entries

// Calls f(columns per thread, layout of B), both as compile-time constants.  The FP64 types alone keep
// the general code for a row-major B (its columns are one cache line, so waiting for them in turn
// costs little, and the registers of the other form do: ComplexF64 grid, 16 columns 694 us against
// 731, Float64 200 against 231).
template <typename V, typename F> void by_layout(int KC, Layout lay, F &&f) {
    using std::integral_constant;
    constexpr Layout R = std::is_same<V, double>::value || std::is_same<V, cf64>::value ? ANY : ROWS;
    if constexpr (std::is_same<V, int64_t>::value) {
        if (lay == ANY) {  // a row-major B, short rows (see launch_rowblock)
            using A = integral_constant<int, ANY>;
            if (KC == 1) f(integral_constant<int, 1>{}, A{});
            else if (KC == 2) f(integral_constant<int, 2>{}, A{});
            else if (KC == 4) f(integral_constant<int, 4>{}, A{});
            else f(integral_constant<int, 8>{}, A{});
            return;
        }
    }
    auto with = [&](auto kc) {
        if (lay == ROWS) f(kc, integral_constant<int, R>{});
        else f(kc, integral_constant<int, COLUMNS>{});
    };
    if constexpr (std::is_same<V, double>::value) {
        if (lay == ANY) {  // pairs (see launch_rowblock)
            f(integral_constant<int, 2>{}, integral_constant<int, ANY>{});
            return;
        }
    }
    if constexpr (!std::is_same<V, cf64>::value) {  // widths that are no power of two, and 16
        if (lay == COLUMNS) {
            using C = integral_constant<int, COLUMNS>;
            if (KC == 3) { f(integral_constant<int, 3>{}, C{}); return; }
            if (KC == 5) { f(integral_constant<int, 5>{}, C{}); return; }
            if (KC == 6) { f(integral_constant<int, 6>{}, C{}); return; }
            if (KC == 7) { f(integral_constant<int, 7>{}, C{}); return; }
            if constexpr (sizeof(V) == 4) {
                if (KC == 16) { f(integral_constant<int, 16>{}, C{}); return; }
            }
        }
    }
    if (KC == 1) with(integral_constant<int, 1>{});
    else if (KC == 2) with(integral_constant<int, 2>{});
    else if (KC == 4) with(integral_constant<int, 4>{});
    else with(integral_constant<int, 8>{});
}

// One launch over the k columns of B and C, KC per thread; k is a multiple of KC for lay = COLUMNS.
// (launch_rowblock cuts a call into such launches.)
template <typename V, typename I>
int launch_columns(cudaStream_t s, const CompressedArgs<V, I> &a, int64_t k, int KC, Layout lay, DenseIn<V> B,
                   const DenseOut<V> &C, const Plan *plan, void *ws, size_t ws_bytes) {
    const int64_t nrb = ceil_div(a.outer_n, RB_THREADS), ncg = ceil_div(k, KC);
    B.pairs = KC >= 2 && get_x_pairs() && pairs_ok(B);
    // plan order 0: the bin order where it pays; 1: natural always; 2: the bin order for every
    // FP64 product whose plan has one
    const int order = get_plan_natural();
    const bool binned = plan && plan->nbin_warps > 0 && order != 1 && (order == 2 || bins_pay<V>(k));
    PlanRows L{};
    int64_t chunk_warps = 0;
    const gsa_chunk_set *cs = plan ? (binned ? &plan->bin : &plan->nat) : nullptr;
    if (cs && cs->nlong > 0) {
        const size_t need = rowblock_workspace_size(plan, sizeof(V), k);
        if (ws_bytes < need) return fail(GSA_ERR_INVALID_ARG, "rowblock workspace too small");
        Carver cv(ws);
        int *done = cv.take<int>((size_t)(cs->nlong * ncg));
        void *partial = cv.take<V>((size_t)(cs->nchunks * k));
        int rc = check_cuda(cudaMemsetAsync(done, 0, sizeof(int) * cs->nlong * ncg, s), "plan counters");
        if (rc) return rc;
        L = plan_rows(*cs);
        L.done = done;
        L.partial = partial;
        chunk_warps = cs->nchunks;
    }
    const int64_t units = binned ? ceil_div(plan->nbin_warps + chunk_warps, RB_WARPS)
                                 : nrb + ceil_div(chunk_warps, RB_WARPS);
    const int64_t blocks = units * ncg;
    if (blocks > 0x7fffffffLL) return fail(GSA_ERR_UNSUPPORTED, "too many rows");
    if constexpr (bins_possible<V>()) {  // the only types a bin order runs for: no other instances
        if (binned) {
            const gsa_bin_order bv = plan->order;
            by_layout<V>(KC, lay, [&](auto kc, auto l) {
                binned_kernel<V, I, decltype(kc)::value, decltype(l)::value>
                    <<<(unsigned)blocks, RB_THREADS, 0, s>>>(a, k, B, C, ncg, bv, L);
            });
            return check_cuda(cudaGetLastError(), "binned_kernel");
        }
    }
    if constexpr (stage_rows_type<V>() && sizeof(I) == 4) {
        const bool aligned = ((uintptr_t)a.idx % 16 == 0) && ((uintptr_t)a.val % 16 == 0);
        if (k == 1 && get_stage_rows() == 1 && aligned) {
            rowblock_staged_kernel<V, I><<<(unsigned)blocks, RB_THREADS, 0, s>>>(a, B, C, nrb, L);
            return check_cuda(cudaGetLastError(), "rowblock_staged_kernel");
        }
        if (k == 1 && get_stage_rows() == 2 && aligned) {
            rowblock_vec_kernel<V, I><<<(unsigned)blocks, RB_THREADS, 0, s>>>(a, B, C, nrb, L);
            return check_cuda(cudaGetLastError(), "rowblock_vec_kernel");
        }
    }
    by_layout<V>(KC, lay, [&](auto kc, auto l) {
        rowblock_kernel<V, I, decltype(kc)::value, decltype(l)::value>
            <<<(unsigned)blocks, RB_THREADS, 0, s>>>(a, k, B, C, ncg, nrb, L);
    });
    return check_cuda(cudaGetLastError(), "rowblock_kernel");
}

// The width of the next launch over a column-major B with `left` columns to go, W the best width of a
// group: all of up to 8 columns; W where it divides them; else the largest width down to `least` (and no
// less than half of W) that does, in one launch; else as many groups of W as there are.  Each launch
// reads the matrix again and has its own start and last wave, which costs rows of 40 entries more than
// it gives: halves of W for the rest (7 = 4 + 2 + 1) took, us against this rule, n = 6*10^4: Float32 7
// columns 83 / 72, 15 columns 165 / 132, ComplexF32 5 columns 67 / 56, 12 columns 133 / 115; on the
// 1024^2 grid Float32 3 columns 20 / 14, 7 columns 39 / 28, Float64 5 columns (pairs, one column
// missing) 67 / 60.  Nine columns as 3 x 3 instead of 8 + 1, `least` = 3, give longer rows 3 to 19 %
// (Float32 and ComplexF32; Float64 loses 12 % on Poisson(10) rows) and cost a grid 40 %.
inline int next_width(int64_t left, int W, int least) {
    if (W < 4) return left < W ? (int)left : W;  // a B too wide for L2: no more columns at a time
    if (left <= 8) return (int)left;
    if (left % W == 0) return W;
    for (int w = W < 8 ? W : 8; w >= least; --w)
        if (left % w == 0 && (w == 3 ? left == 9 : 2 * w >= (W < 8 ? W : 8))) return w;
    return left >= W ? W : 8;
}

template <typename V, typename I>
int launch_rowblock(cudaStream_t s, const CompressedArgs<V, I> &a, int64_t k, DenseIn<V> B,
                    DenseOut<V> C, const Plan *plan, void *ws, size_t ws_bytes) {
    if (a.outer_n == 0 || k == 0) return GSA_OK;
    if (a.inner_n == 0) {  // B has no rows: nothing may be read of it, and every entry adds a zero
        B.p = a.val;
        B.rs = 1;
        B.cs = 0;
    }
    if (plan && (plan->outer_n != a.outer_n || plan->nnz != a.nnz))
        return fail(GSA_ERR_INVALID_ARG, "plan was made for another structure");
    // Columns a thread accumulates for SpMM: more share each entry's loads and the row's extent and
    // keep more gathers in flight, fewer keep registers (and so occupancy) low.  Column-major B
    // (each column its own gather), measured with KC = 1 / 2 / 4 / 8 / 16, us on the 2048^2 grid (a
    // lane per row) and on Poisson(10) rows, n = 10^6: Float32, 16 columns 583 / 394 / 289 / 205 / 175
    // and 638 / 667 / 561 / 572 / 575; ComplexF32, 8 columns 348 / 301 / 199 / 168 and 394 / 336 / 331 /
    // 321; Float64, 8 columns 383 / 389 / 370 / 437 and 679 / 465 / 419 / 383; ComplexF64, 8 columns,
    // bound by the FP64 pipe, 1343 / 1377 / 1372 / 1372 and 858 / 885 / 919 / 973.  Hence 16 for 4-byte
    // values, 8 for ComplexF32 and for Float64 (and Int64) rows of several lanes, 4 for shorter
    // ones, 1 for ComplexF64; and 2 for the Float64 rows of several lanes where B does not stay in
    // L2: KC = 2 / 4 / 8, n = 5*10^5, Poisson(10) rows with 76 MB of B 685 / 605 / 609, 91 MB 935 / 877 / 911, 106 MB
    // 1240 / 1188 / 1282, 122 MB 1570 / 1555 / 1635, 183 MB 3176 / 3192 / 3264; the power law 938 / 860 / 861, 1273 /
    // 1249 / 1339, 1698 / 1692 / 1891, 2187 / 2223 / 2424, 4706 / 4668 / 4825 (Int64: all alike from 91 MB on).
    // Row-major B (an entry's values share cache lines, and Float64 reads them in 16-byte pieces): 8
    // columns for the FP64 types (Float64 SpMM of the served mix's matrices, n = 10^6, k = 16: 871 us with
    // 8 against 982 us with 4).  The others, KC = 4 / 8, us on the 1024^2 grid, Poisson(10) rows (n =
    // 3*10^5), the power law (2*10^5) and Poisson(40) rows (6*10^4): Float32, 8 columns 62 / 56, 60 / 62, 73 / 75,
    // 49 / 51, 12 columns 77 / 83, 75 / 83, 91 / 109, 69 / 78; ComplexF32, 5 columns 54 / 46, 53 / 48, 71 / 76, 52 /
    // 44, 8 columns 95 / 93, 82 / 85, 96 / 102, 68 / 75, 16 columns 297 / 293, 196 / 202, 212 / 213, 163 / 177, 31 columns
    // 315 / 270, 260 / 243, 313 / 310, 190 / 187; Int64's longer rows 5 columns 56 / 52, 86 / 77, 53 / 44, 12 columns
    // 107 / 117, 131 / 158, 94 / 106, 31 columns 291 / 262, 362 / 354, 193 / 190.  Hence 4 for 4-byte values, but
    // 8 where that makes one group of a grid's; and 8 for 8-byte values, but 4 for 8 to 23 columns of
    // longer rows.
    const bool rowmajor = B.cs == 1 && B.rs > 1, longer = a.nnz > G1_AVG * a.outer_n;
    const int knob = get_spmm_columns();
    int KC = knob;
    if (KC == 0) {
        if (rowmajor && sizeof(V) == 4) KC = !longer && k > 4 && k <= 8 ? 8 : 4;
        else if (rowmajor && (std::is_same<V, cf32>::value || std::is_same<V, int64_t>::value))
            KC = longer && k >= 8 && k < 24 ? 4 : 8;
        else if (rowmajor) KC = 8;
        else if (sizeof(V) == 4) KC = 16;
        else if (sizeof(V) == 16) KC = 1;
        else if (std::is_same<V, cf32>::value) KC = 8;
        else if (!longer) KC = 4;
        else KC = (size_t)a.inner_n * (size_t)k * sizeof(V) <= WIDE_B_BYTES ? 8 : 2;
    }
    // A row-major B takes the smallest width that covers k, with columns missing in the last group.  A
    // column-major one takes widths that its columns fill (next_width), a launch for each: no kernel
    // has to ask for missing columns.  Two exceptions, both Float64 by pairs in the general code: two
    // columns of longer rows, whose fewer loads in flight are the faster (Poisson(10) rows, n = 3*10^5,
    // 44 us against 48; power law, n = 2*10^5, 47 against 51; rows of 40 the same), and odd k where B is too
    // wide for L2, whose last single column would read the entries once more for one FMA each.
    // (Int64 and a row-major B: the loads of a row's columns issued together pay on longer rows -- power
    // law, 7 columns 179 us / 86 -- but not on a grid's, 2 columns 21.6 us / 23.6, 12 columns 111 / 116.)
    Layout lay = rowmajor ? ROWS : COLUMNS;
    if (rowmajor) {
        if (std::is_same<V, int64_t>::value && !longer) lay = ANY;
        while (KC > 1 && KC / 2 >= k) KC >>= 1;
    } else if (std::is_same<V, double>::value && !knob && k > 1 && ((k == 2 && longer) || (KC == 2 && (k & 1)))) {
        lay = ANY;
        KC = 2;
    }
    const int least = longer && !std::is_same<V, double>::value ? 3 : 4;
    int rc = GSA_OK;
    timer_before(s);
    for (int64_t c = 0; c < k && !rc;) {
        const int64_t left = k - c;
        int w = KC;
        if (lay == COLUMNS && !knob && !std::is_same<V, cf64>::value) w = next_width(left, KC, least);
        while (lay == COLUMNS && w > left) w >>= 1;  // an explicit width, and ComplexF64: halves of it
        const int64_t cols = lay == COLUMNS ? left / w * w : k;
        DenseIn<V> Bc = B;
        DenseOut<V> Cc = C;
        Bc.p += c * B.cs;
        Cc.p += c * C.ld;
        rc = launch_columns<V, I>(s, a, cols, w, lay, Bc, Cc, plan, ws, ws_bytes);
        c += cols;
    }
    timer_after(s);
    return rc;
}

#define GSA_INST_RB(V)                                                                               \
    template int launch_rowblock<V, int32_t>(cudaStream_t, const CompressedArgs<V, int32_t> &, int64_t, \
                                             DenseIn<V>, DenseOut<V>, const Plan *, void *, size_t);  \
    template int launch_rowblock<V, int64_t>(cudaStream_t, const CompressedArgs<V, int64_t> &, int64_t, \
                                             DenseIn<V>, DenseOut<V>, const Plan *, void *, size_t);

}  // namespace gsa
