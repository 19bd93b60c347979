// The grouped kernel (see gsa_batch.cu) and its launch.  One source file per value type
// instantiates this (they compile in parallel).
#pragma once

#include "gsa_rows.cuh"

namespace gsa {

// One value of V from an item's alpha/beta bytes (8-byte loads: the bytes are 8-aligned).
template <typename V>
__device__ __forceinline__ V scalar_at(const unsigned char *p) {
    union { V v; unsigned long long w[sizeof(V) >= 8 ? sizeof(V) / 8 : 1]; unsigned int h; } u;
    if (sizeof(V) >= 8) {
#pragma unroll
        for (int i = 0; i < (int)(sizeof(V) / 8); ++i) u.w[i] = __ldg((const unsigned long long *)p + i);
    } else {
        u.h = __ldg((const unsigned int *)p);
    }
    return u.v;
}

template <typename V, typename I, int KC>
__global__ void __launch_bounds__(RB_THREADS)
grouped_kernel(const gsa_group_item *__restrict__ items, int64_t count, int64_t ntiles, int base,
               int g1_avg, int x_pairs, const int32_t *__restrict__ tile_item) {
    // Each warp finds its tile's item on its own -- lane 0 searches forward from the
    // warp's previous item (a CTA's tiles ascend), the warp reads the item's fields with
    // uniform loads -- so warps never wait for one another between tiles.
    const int lane = threadIdx.x & 31;
    int64_t lo = 0;
    for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        if (tile_item) {  // a batch's table: the tile's item in one load
            lo = __ldg(tile_item + t);
        } else if (lane == 0 && lo + 1 < count && __ldg(&items[lo + 1].first_tile) <= t) {
            int64_t l = lo + 1, h = count - 1;  // last item with first_tile <= t, in (lo, count)
            while (l < h) {
                const int64_t mid = (l + h + 1) >> 1;
                if (__ldg(&items[mid].first_tile) <= t) l = mid;
                else h = mid - 1;
            }
            lo = l;
        }
        if (!tile_item) lo = __shfl_sync(0xffffffffu, lo, 0);
        const gsa_group_item *it = items + lo;
        const int64_t kk = __ldg(&it->k);
        const int64_t ncg = (kk + KC - 1) / KC;
        const int64_t local = t - __ldg(&it->first_tile);
        const int64_t cg = ncg == 1 ? 0 : local % ncg;
        const int64_t unit = ncg == 1 ? local : local / ncg;
        CompressedArgs<V, I> a;
        a.outer_n = __ldg(&it->m);
        a.inner_n = __ldg(&it->n);
        a.nnz = __ldg(&it->nnz);
        a.ptr = (const I *)__ldg((const unsigned long long *)&it->rowptr);
        a.idx = (const I *)__ldg((const unsigned long long *)&it->colval);
        a.val = (const V *)__ldg((const unsigned long long *)&it->nzval);
        a.base = base;
        a.conjA = false;
        const int64_t ldb = __ldg(&it->ldb);
        const bool brow = __ldg(&it->b_rowmajor) != 0;
        DenseIn<V> B;
        B.p = (const V *)__ldg((const unsigned long long *)&it->B);
        B.rs = brow ? ldb : 1;
        B.cs = brow ? 1 : ldb;
        B.conj = false;
        B.pairs = KC >= 2 && x_pairs && std::is_same<V, double>::value && brow && (ldb & 1) == 0 &&
                  ((uintptr_t)B.p & 15) == 0;
        DenseOut<V> C;
        C.p = (V *)__ldg((const unsigned long long *)&it->C);
        C.ld = __ldg(&it->ldc);
        C.alpha = scalar_at<V>(it->alpha);
        C.beta = scalar_at<V>(it->beta);
        C.beta_mode = is_zero(C.beta) ? 0 : (is_one(C.beta) ? 1 : 2);
        C.alpha_one = alpha_one_of(C.alpha);
        const int64_t bin_warps = __ldg(&it->bin_warps);
        if (bin_warps > 0) {  // the plan's bin order: warp w of it
            const int64_t w = unit * RB_WARPS + (threadIdx.x >> 5);
            if (w < bin_warps) {
                const gsa_bin_order *bo = (const gsa_bin_order *)__ldg((const unsigned long long *)&it->bin_order);
                const gsa_bin_order bv{__ldg(&bo->nwarps),
                                       (const int32_t *)__ldg((const unsigned long long *)&bo->perm),
                                       (const int32_t *)__ldg((const unsigned long long *)&bo->warp_group),
                                       (const int64_t *)__ldg((const unsigned long long *)&bo->groups)};
                binned_warp<V, I, KC, ANY>(a, kk, B, C, cg * KC, w, bv);
            }
        } else {
            warp_unit<V, I, KC, ANY>(a, kk, B, C, cg * KC, unit * RB_THREADS + (threadIdx.x & ~31), nullptr, g1_avg);
        }
    }
}

template <typename V, typename I>
int launch_grouped(cudaStream_t s, const gsa_group_item *items, int64_t count, int64_t ntiles, int base, int KC, int g1,
                   const int32_t *tile_item) {
    if (ntiles == 0) return GSA_OK;
    auto kern = KC == 1 ? grouped_kernel<V, I, 1>
              : KC == 2 ? grouped_kernel<V, I, 2>
              : KC == 4 ? grouped_kernel<V, I, 4> : grouped_kernel<V, I, 8>;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, RB_THREADS, 0),
                        "grouped occupancy");
    if (rc) return rc;
    int64_t grid = (int64_t)sms * (per_sm > 0 ? per_sm : 1);
    if (grid > ntiles) grid = ntiles;
    timer_before(s);
    kern<<<(unsigned)grid, RB_THREADS, 0, s>>>(items, count, ntiles, base, g1, get_x_pairs(), tile_item);
    timer_after(s);
    return check_cuda(cudaGetLastError(), "grouped_kernel");
}

#define GSA_INST_GROUPED(V, I)                                                                       \
    template int launch_grouped<V, I>(cudaStream_t, const gsa_group_item *, int64_t, int64_t, int, int, int, \
                                      const int32_t *);

}  // namespace gsa
