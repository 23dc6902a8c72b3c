// The box-mass gather of the plain FP64 form (box_tile.cuh), the lattice gather of the FP32-mixed form
// (lattice_tile.cuh), and the batch's persistent kernels for both.  This translation unit is built with
// FMA contraction: both regroup the reference's sum, so they do not follow its operation order
// and gain nothing from rounding each product on its own; the quantities that integer results depend on
// (bounding boxes, lattice planes, cell centres, the support test of the pair counters) are formed with
// explicitly rounded operations (cart_common.cuh), as in every other form.
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>
#include <vector>

#include "engine.hpp"
#include "kernel_tables.h"

#include "box_tables.h"

namespace kiwi_b200 {
static __constant__ KiwiKernelTable c_tables[KIWI_NUM_KERNELS];
static __constant__ KiwiBoxTable c_box[KIWI_NUM_KERNELS];
}  // namespace kiwi_b200

#include "box_tile.cuh"
#include "lattice_tile.cuh"

namespace kiwi_b200 {

int lattice_init_tables(KiwiCtx* ctx) {
    KIWI_CUDA(ctx, cudaMemcpyToSymbol(c_tables, kiwi_kernel_tables, sizeof(kiwi_kernel_tables)));
    static_assert(sizeof(kiwi_box_tables) == sizeof(KiwiBoxTable) * KIWI_NUM_KERNELS, "one box table per kernel");
    KIWI_CUDA(ctx, cudaMemcpyToSymbol(c_box, kiwi_box_tables, sizeof(kiwi_box_tables)));
    return KIWI_OK;
}

namespace {

// Resident CTAs per SM of the FP32-mixed kernels: two (128 registers), as measured in the FP64 form of this body: the cubic
// kernel's shared memory would fit three, but at the 80 registers three need, its point-wise tiers spill:
// 3.59 G support pairs/s at three against 3.84 G at two on the 2 M-particle log-normal cube.
#ifndef KIWI_LATTICE_MIN_BLOCKS
#define KIWI_LATTICE_MIN_BLOCKS 2
#endif
#ifndef KIWI_LATTICE_GEN_MIN_BLOCKS
#define KIWI_LATTICE_GEN_MIN_BLOCKS 2
#endif
constexpr int kLatMinBlocks = KIWI_LATTICE_MIN_BLOCKS;
constexpr int kLatGenMinBlocks = KIWI_LATTICE_GEN_MIN_BLOCKS;
constexpr size_t kLatMergedDynSmem = kLatDynSmem > kLatGenDynSmem ? kLatDynSmem : kLatGenDynSmem;
#ifndef KIWI_BOX_MIN_BLOCKS
#define KIWI_BOX_MIN_BLOCKS 2
#endif
constexpr int kBoxMinBlocks = KIWI_BOX_MIN_BLOCKS;

// Kernel KERNEL of the tables (NP pieces, powers to DEG; KERNEL < 0: any, `kernel`, with both 0), over items, or
// without them over the tiles tile_map[0 ..) (every tile if null), each tile by one CTA: SEQ cuts it into its
// segments, else no list is longer than one.
template <bool CULL, int KERNEL, int NP, int DEG, bool SEQ>
__global__ void __launch_bounds__(kBoxThreads, kBoxMinBlocks)
    k_cart_box(CartGeom g, DevParticles P, int kernel, const uint32_t* __restrict__ list,
               const int64_t* __restrict__ range, const int32_t* __restrict__ tile_map, const BoxItem* __restrict__ items,
               CartOutputs out, double* __restrict__ sums, DevStats* __restrict__ st) {
    const KiwiBoxTable& T = c_box[KERNEL >= 0 ? KERNEL : kernel];
    if (SEQ) {
        const int64_t t = tile_map ? (int64_t)tile_map[blockIdx.x] : (int64_t)blockIdx.x;
        const int64_t lo = range[2 * t], hi = range[2 * t + 1];
        box_tile<CULL, NP, DEG, true>(g, P, list, lo, hi, box_segment(hi - lo, (int64_t)g.ntx * g.nty * g.ntz), t, out,
                                      nullptr, st, T);
        return;
    }
    BoxItem it{tile_map ? tile_map[blockIdx.x] : (int)blockIdx.x, 0, 1, 0};
    if (items) it = items[blockIdx.x];
    box_item<CULL, NP, DEG>(it, g, P, list, range + 2 * (int64_t)it.tile, it.tile, out, sums, st, T);
}

// The cut tiles' outputs: one CTA per tile (its item of segment 0).
__global__ void __launch_bounds__(256) k_box_combine(CartGeom g, const BoxItem* __restrict__ cut,
                                                     const double* __restrict__ sums, CartOutputs out) {
    const BoxItem it = cut[blockIdx.x];
    box_combine(g, out, it.tile, sums + (int64_t)it.slot * 4 * kTileCells, it.nseg);
}

// The items of the tiles map[first .. first + n) (tiles from `first` on if null), heaviest first by 64 classes of their entry counts (the
// order among the items, and among the places of their sums, does not affect any result).  counts: items, places
// of sums, cut tiles, then the classes' sizes and their running starts (64 each).
constexpr int kBoxClasses = 64;
__device__ __forceinline__ int box_class(int64_t len, int64_t ntiles) {
    const int64_t c = len * kBoxClasses / (box_segment(0, ntiles) + 1);
    return kBoxClasses - 1 - (int)(c < kBoxClasses ? c : kBoxClasses - 1);
}
template <bool EMIT>
__global__ void __launch_bounds__(256) k_box_items(const int64_t* __restrict__ range, int64_t ntiles,
                                                   const int32_t* __restrict__ map, int64_t first, int64_t n,
                                                   int* __restrict__ counts,
                                                   BoxItem* __restrict__ items, BoxItem* __restrict__ cut) {
    __shared__ int s_n[kBoxClasses], s_at[kBoxClasses];
    if (threadIdx.x < kBoxClasses) s_n[threadIdx.x] = 0;
    __syncthreads();
    const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int t = 0, nseg = 0, full = 0, last = 0, at_full = 0, at_last = 0;
    if (w < n) {
        t = map ? map[first + w] : (int)(first + w);
        const int64_t cnt = range[2 * (int64_t)t + 1] - range[2 * (int64_t)t], len = box_segment(cnt, ntiles);
        nseg = cnt > len ? (int)((cnt + len - 1) / len) : 1;
        full = box_class(len, ntiles);
        last = box_class(cnt - (nseg - 1) * len, ntiles);
        if (nseg > 1) at_full = atomicAdd(&s_n[full], nseg - 1);
        at_last = atomicAdd(&s_n[last], 1);
    }
    __syncthreads();
    if (!EMIT) {
        if (threadIdx.x < kBoxClasses && s_n[threadIdx.x]) atomicAdd(&counts[4 + threadIdx.x], s_n[threadIdx.x]);
        int items_n = nseg, places = nseg > 1 ? nseg : 0, tiles = nseg > 1;
        for (int o = 16; o > 0; o >>= 1) {
            items_n += __shfl_down_sync(0xffffffffu, items_n, o);
            places += __shfl_down_sync(0xffffffffu, places, o);
            tiles += __shfl_down_sync(0xffffffffu, tiles, o);
        }
        if ((threadIdx.x & 31) == 0) {
            if (items_n) atomicAdd(&counts[0], items_n);
            if (places) {
                atomicAdd(&counts[1], places);
                atomicAdd(&counts[2], tiles);
            }
        }
        return;
    }
    // the classes' first items, then this block's place in each
    if (threadIdx.x < kBoxClasses) {
        int first = 0;
        for (int c = 0; c < (int)threadIdx.x; ++c) first += counts[4 + c];
        s_at[threadIdx.x] = first + (s_n[threadIdx.x] ? atomicAdd(&counts[4 + kBoxClasses + threadIdx.x], s_n[threadIdx.x]) : 0);
    }
    __syncthreads();
    if (w >= n) return;
    int slot = 0;
    if (nseg > 1) {
        slot = atomicAdd(&counts[4 + 2 * kBoxClasses], nseg);
        cut[atomicAdd(&counts[4 + 2 * kBoxClasses + 1], 1)] = BoxItem{t, 0, nseg, slot};
    }
    for (int s = 0; s + 1 < nseg; ++s) items[s_at[full] + at_full + s] = BoxItem{t, s, nseg, slot};
    items[s_at[last] + at_last] = BoxItem{t, nseg - 1, nseg, slot};
}

// The FP32-mixed form of the cubic lattice kernel (support cells only): edge pairs and lattice points
// evaluated with FP32 tiers (FP64 islands where a plane lies within 1e-3 h of the particle), cell assembly
// and per-cell sums in FP64.
__global__ void __launch_bounds__(kLatThreads, kLatMinBlocks) k_cart_lattice_mixed(CartGeom g, DevParticles P,
                                                                                const uint32_t* __restrict__ list,
                                                                                const int64_t* __restrict__ range,
                                                                                const int32_t* __restrict__ tile_map,
                                                                                CartOutputs out,
                                                                                DevStats* __restrict__ st) {
    const int64_t t = tile_map ? (int64_t)tile_map[blockIdx.x] : (int64_t)blockIdx.x;
    lattice_tile<false>(g, P, list, range, t, t, out, st);
}

// The FP32-mixed form of the generic lattice kernel: edge records and vertex tiers in FP32 (FP64 islands
// where a plane lies within 1e-3 h of the particle), records, cell assembly and per-cell sums in FP64.
__global__ void __launch_bounds__(kLatThreads, kLatGenMinBlocks)
    k_cart_lattice_generic_mixed(CartGeom g, DevParticles P, int kernel, const uint32_t* __restrict__ list,
                                 const int64_t* __restrict__ range, const int32_t* __restrict__ tile_map,
                                 CartOutputs out, DevStats* __restrict__ st) {
    const int64_t t = tile_map ? (int64_t)tile_map[blockIdx.x] : (int64_t)blockIdx.x;
    lattice_tile<true>(g, P, list, range, t, t, out, st, &c_tables[kernel]);
}

// The work of a batch's grids with one kernel (FP64 form), or one lattice family's (FP32-mixed form: whole tiles), in
// one persistent launch: each CTA takes the next of the launch's work items from the work counter and runs the
// same body as the single-grid kernel, so every cell's summation order is that of a single-grid call.
template <int KERNEL, int NP, int DEG>
__global__ void __launch_bounds__(kBoxThreads, 2)
    k_batch_box(const BatchItemDev* __restrict__ items, const int32_t* __restrict__ item_of_tile,
                const BoxItem* __restrict__ work, int64_t nwork, const uint32_t* __restrict__ list,
                const int64_t* __restrict__ range, double* __restrict__ sums, unsigned long long* __restrict__ next) {
    __shared__ long long s_w;
    __shared__ BatchItemDev s_it;  // (in shared memory: the body's registers are full)
    static_assert(sizeof(BatchItemDev) % 8 == 0 && sizeof(BatchItemDev) / 8 <= kBoxThreads, "copied by one step");
    for (;;) {
        if (threadIdx.x == 0) s_w = (long long)atomicAdd(next, 1ull);
        __syncthreads();
        const int64_t w = s_w;
        if (w >= nwork) break;
        const BoxItem wi = work[w];
        const int64_t tg = wi.tile;
        const int64_t* const src = reinterpret_cast<const int64_t*>(items + item_of_tile[tg]);
        if (threadIdx.x < sizeof(BatchItemDev) / 8) reinterpret_cast<int64_t*>(&s_it)[threadIdx.x] = src[threadIdx.x];
        __syncthreads();
        box_item<true, NP, DEG>(wi, s_it.g, s_it.P, list, range + 2 * tg, tg - s_it.tile_base, s_it.out, sums, s_it.st,
                                c_box[KERNEL]);
        __syncthreads();
    }
}

template <int FAMILY>
__global__ void __launch_bounds__(kLatThreads, 2)
    k_batch_mixed(const BatchItemDev* __restrict__ items, const int32_t* __restrict__ item_of_tile,
                  const BoxItem* __restrict__ work, int64_t nwork, const uint32_t* __restrict__ list,
                  const int64_t* __restrict__ range, unsigned long long* __restrict__ next) {
    __shared__ long long s_w;
    for (;;) {
        if (threadIdx.x == 0) s_w = (long long)atomicAdd(next, 1ull);
        __syncthreads();
        const int64_t w = s_w;
        if (w >= nwork) break;
        const int64_t tg = work[w].tile;
        const BatchItemDev& it = items[item_of_tile[tg]];
        const int64_t tl = tg - it.tile_base;
        if (FAMILY == kBatchFamilyMixed || (FAMILY == kBatchFamilyMixedMerged && it.mode == kBatchLattice))
            lattice_tile<false>(it.g, it.P, list, range, tg, tl, it.out, it.st);
        else
            lattice_tile<true>(it.g, it.P, list, range, tg, tl, it.out, it.st, &c_tables[it.kernel]);
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) k_batch_combine(const BatchItemDev* __restrict__ items,
                                                       const int32_t* __restrict__ item_of_tile,
                                                       const BoxItem* __restrict__ cut, const double* __restrict__ sums) {
    const BoxItem wi = cut[blockIdx.x];
    const BatchItemDev& it = items[item_of_tile[wi.tile]];
    box_combine(it.g, it.out, wi.tile - it.tile_base, sums + (int64_t)wi.slot * 4 * kTileCells, wi.nseg);
}

template <int FAMILY>
constexpr size_t mixed_smem() {
    return FAMILY == kBatchFamilyMixed ? kLatDynSmem
                                       : (FAMILY == kBatchFamilyMixedMerged ? kLatMergedDynSmem : kLatGenDynSmem);
}

}  // namespace

template <bool CULL, int KERNEL, int NP, int DEG, bool SEQ>
static int box_launch(KiwiCtx* ctx, int64_t blocks, const CartGeom& g, const DevParticles& P, int kernel,
                      const TileLists& tl, const BoxItem* items, const CartOutputs& out, double* sums, DevStats* st) {
    constexpr size_t smem = BoxCaps<NP, SEQ>::kSmem;
    KIWI_CUDA(ctx, cudaFuncSetAttribute(k_cart_box<CULL, KERNEL, NP, DEG, SEQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem));
    k_cart_box<CULL, KERNEL, NP, DEG, SEQ><<<(unsigned)blocks, kBoxThreads, smem, ctx->stream>>>(g, P, kernel, tl.list, tl.range,
                                                                                      tl.map, items, out, sums, st);
    KIWI_LAUNCHED(ctx);
    return KIWI_OK;
}

template <bool SEQ>
static int box_launch_kernel(KiwiCtx* ctx, int64_t blocks, const CartGeom& g, const DevParticles& P, const KernelChoice& k,
                             const TileLists& tl, const BoxItem* items, const CartOutputs& out, double* sums,
                             DevStats* st, bool full_box) {
    if (k.kernel == 0 && full_box) return box_launch<false, 0, 2, 3, SEQ>(ctx, blocks, g, P, 0, tl, items, out, sums, st);
    if (k.kernel == 0) return box_launch<true, 0, 2, 3, SEQ>(ctx, blocks, g, P, 0, tl, items, out, sums, st);
    if constexpr (SEQ) {  // one CTA per tile (the allocation-free call): one body for the other kernels
        return box_launch<true, -1, 0, 0, SEQ>(ctx, blocks, g, P, k.kernel, tl, items, out, sums, st);
    } else {
#define KIWI_BOX_LAUNCH(K, NP, DEG) \
    if (k.kernel == K) return box_launch<true, K, NP, DEG, false>(ctx, blocks, g, P, K, tl, items, out, sums, st);
        KIWI_BOX_OTHERS(KIWI_BOX_LAUNCH)
#undef KIWI_BOX_LAUNCH
        return set_err(ctx, KIWI_ERR_ARG, "unknown kernel %d", k.kernel);
    }
}

int box_work_next(KiwiCtx* ctx, const TileLists& tl, BoxWork* w) {
    w->all = tl.map ? tl.nmap : tl.ntiles;
    const int64_t first = w->done;
    int64_t n = w->all - first;
    // no list can be longer than a segment: the tiles as they are
    if (tl.total <= box_segment(0, tl.ntiles)) {
        w->n = n;
        w->done = w->all;
        return KIWI_OK;
    }
    constexpr int kCounts = 4 + 2 * kBoxClasses + 2;
    const int64_t most = box_most(tl.ntiles);
    int* counts = nullptr;
    KIWI_TRY(scratch_t(ctx, S_BOX_COUNTS, kCounts, &counts));
    int h[3] = {0, 0, 0};
    // the run: all that is left, or as many tiles as kBoxPlaces hold; half as many as long as their sums cannot be had
    for (;;) {
        if (w->run > 0) n = std::min(n, w->run);
        KIWI_CUDA(ctx, cudaMemsetAsync(counts, 0, sizeof(int) * kCounts, ctx->stream));
        k_box_items<false><<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(tl.range, tl.ntiles, tl.map, first, n,
                                                                                counts, nullptr, nullptr);
        KIWI_LAUNCHED(ctx);
        KIWI_CUDA(ctx, cudaMemcpyAsync(h, counts, sizeof h, cudaMemcpyDeviceToHost, ctx->stream));
        KIWI_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (h[1] > kBoxPlaces && n > kBoxPlaces / most) {
            w->run = kBoxPlaces / most;
            continue;
        }
        w->sums = nullptr;
        if (h[1] == 0) break;
        // (runs take the most that one may need, so that the buffer does not grow from run to run)
        const size_t places = w->run > 0 ? (size_t)(n * most) : (size_t)h[1];
        const int rc = scratch_t(ctx, S_BOX_SUMS, places * 4 * kTileCells, &w->sums);
        if (rc == KIWI_OK) break;
        if (rc != KIWI_ERR_ALLOC || n <= 1) return rc;
        ctx->err.clear();
        w->run = (n + 1) / 2;
    }
    BoxItem *items = nullptr, *cut = nullptr;
    KIWI_TRY(scratch_t(ctx, S_BOX_ITEMS, (size_t)h[0], &items));
    KIWI_TRY(scratch_t(ctx, S_BOX_CUT, (size_t)(h[2] > 0 ? h[2] : 1), &cut));
    k_box_items<true><<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(tl.range, tl.ntiles, tl.map, first, n, counts,
                                                                           items, cut);
    KIWI_LAUNCHED(ctx);
    w->items = items;
    w->n = h[0];
    w->cut = cut;
    w->n_cut = h[2];
    w->done = first + n;
    return KIWI_OK;
}

int box_work_finish(KiwiCtx* ctx, const CartGeom& g, const BoxWork& w, const CartOutputs& out) {
    if (w.n_cut <= 0) return KIWI_OK;
    k_box_combine<<<(unsigned)w.n_cut, 256, 0, ctx->stream>>>(g, w.cut, w.sums, out);
    KIWI_LAUNCHED(ctx);
    return KIWI_OK;
}

int lattice_cart_gather(KiwiCtx* ctx, const CartGeom& g, const DevParticles& P, const KernelChoice& k,
                        const TileLists& tl, const CartOutputs& out, DevStats* d_stats, bool full_box) {
    // without scratch of its own (the allocation-free call), one CTA per tile cuts it
    if (ctx->arena)
        return box_launch_kernel<true>(ctx, tl.map ? tl.nmap : tl.ntiles, g, P, k, tl, nullptr, out, nullptr, d_stats,
                                       full_box);
    BoxWork w;
    do {
        KIWI_TRY(box_work_next(ctx, tl, &w));
        KIWI_TRY(box_launch_kernel<false>(ctx, w.n, g, P, k, tl, w.items, out, w.sums, d_stats, full_box));
        KIWI_TRY(box_work_finish(ctx, g, w, out));
    } while (w.done < w.all);
    return KIWI_OK;
}

void lattice_batch_work(const std::vector<int32_t>& tiles, const std::vector<int64_t>& range,
                        const std::vector<int64_t>& grid_tiles, const std::vector<int32_t>& slot, bool split,
                        std::vector<int32_t>* work, std::vector<int64_t>* weight) {
    work->clear();
    weight->clear();
    for (const int32_t t : tiles) {
        const int64_t cnt = range[2 * (size_t)t + 1] - range[2 * (size_t)t];
        const int64_t len = split ? box_segment(cnt, grid_tiles[(size_t)t]) : cnt;
        const int nseg = cnt > len ? (int)((cnt + len - 1) / len) : 1;
        for (int s = 0; s < nseg; ++s) {
            work->insert(work->end(), {t, s, nseg, nseg > 1 ? slot[(size_t)t] : 0});
            weight->push_back(nseg > 1 ? std::min(len, cnt - s * len) : cnt);
        }
    }
}

int64_t lattice_batch_segments(int64_t cnt, int64_t grid_tiles) {
    const int64_t len = box_segment(cnt, grid_tiles);
    return cnt > len ? (cnt + len - 1) / len : 1;
}

int lattice_batch_combine(KiwiCtx* ctx, const BatchItemDev* d_items, const int32_t* d_item_of_tile, const int32_t* d_cut,
                          int64_t n, const double* sums) {
    if (n <= 0) return KIWI_OK;
    k_batch_combine<<<(unsigned)n, 256, 0, ctx->stream>>>(d_items, d_item_of_tile, reinterpret_cast<const BoxItem*>(d_cut),
                                                          sums);
    KIWI_LAUNCHED(ctx);
    return KIWI_OK;
}

int lattice_mixed_gather(KiwiCtx* ctx, const CartGeom& g, const DevParticles& P, const KernelChoice& k,
                         const TileLists& tl, const CartOutputs& out, DevStats* d_stats) {
    if (tl.ntiles <= 0 || (tl.map && tl.nmap <= 0)) return KIWI_OK;
    const dim3 grid((unsigned)(tl.map ? tl.nmap : tl.ntiles));
    if (!k.cubic) {
        KIWI_CUDA(ctx, cudaFuncSetAttribute(k_cart_lattice_generic_mixed, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)kLatGenDynSmem));
        KIWI_CUDA(ctx, cudaFuncSetAttribute(k_cart_lattice_generic_mixed,
                                            cudaFuncAttributePreferredSharedMemoryCarveout,
                                            (int)kLatCarveout));
        k_cart_lattice_generic_mixed<<<grid, kLatThreads, kLatGenDynSmem, ctx->stream>>>(
            g, P, k.kernel, tl.list, tl.range, tl.map, out, d_stats);
        KIWI_LAUNCHED(ctx);
        return KIWI_OK;
    }
    KIWI_CUDA(ctx, cudaFuncSetAttribute(k_cart_lattice_mixed, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)kLatDynSmem));
    KIWI_CUDA(ctx, cudaFuncSetAttribute(k_cart_lattice_mixed, cudaFuncAttributePreferredSharedMemoryCarveout,
                                        (int)kLatCarveout));
    k_cart_lattice_mixed<<<grid, kLatThreads, kLatDynSmem, ctx->stream>>>(g, P, tl.list, tl.range, tl.map, out,
                                                                          d_stats);
    KIWI_LAUNCHED(ctx);
    return KIWI_OK;
}

template <class F>
static int batch_attr(KiwiCtx* ctx, F* f, size_t smem) {
    KIWI_CUDA(ctx, cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return KIWI_OK;
}

int lattice_batch_prepare(KiwiCtx* ctx) {
#define KIWI_BOX_ATTR(K, NP, DEG) KIWI_TRY(batch_attr(ctx, k_batch_box<K, NP, DEG>, BoxCaps<NP>::kSmem));
    KIWI_BOX_KERNELS(KIWI_BOX_ATTR)
#undef KIWI_BOX_ATTR
    KIWI_TRY(batch_attr(ctx, k_batch_mixed<kBatchFamilyMixed>, mixed_smem<kBatchFamilyMixed>()));
    KIWI_TRY(batch_attr(ctx, k_batch_mixed<kBatchFamilyMixedGeneric>, mixed_smem<kBatchFamilyMixedGeneric>()));
    return batch_attr(ctx, k_batch_mixed<kBatchFamilyMixedMerged>, mixed_smem<kBatchFamilyMixedMerged>());
}

template <int FAMILY>
static void batch_launch_mixed(cudaStream_t stream, const BatchItemDev* d_items, const int32_t* d_item_of_tile,
                               const BoxItem* work, int64_t nwork, const uint32_t* list, const int64_t* range,
                               unsigned long long* d_next, int blocks) {
    k_batch_mixed<FAMILY><<<blocks, kLatThreads, mixed_smem<FAMILY>(), stream>>>(d_items, d_item_of_tile, work, nwork, list,
                                                                              range, d_next);
}

int lattice_batch_gather(KiwiCtx* ctx, int family, const BatchItemDev* d_items, const int32_t* d_item_of_tile,
                         const int32_t* d_work, int64_t nwork, const uint32_t* list,
                         const int64_t* range, double* sums, unsigned long long* d_next, int blocks, bool mixed) {
    const BoxItem* work = reinterpret_cast<const BoxItem*>(d_work);
    const cudaStream_t stream = ctx->stream;
    if (mixed) {
        if (family == kBatchFamilyMixed)
            batch_launch_mixed<kBatchFamilyMixed>(stream, d_items, d_item_of_tile, work, nwork, list, range, d_next, blocks);
        else if (family == kBatchFamilyMixedMerged)
            batch_launch_mixed<kBatchFamilyMixedMerged>(stream, d_items, d_item_of_tile, work, nwork, list, range, d_next,
                                                        blocks);
        else
            batch_launch_mixed<kBatchFamilyMixedGeneric>(stream, d_items, d_item_of_tile, work, nwork, list, range, d_next,
                                                         blocks);
    }
#define KIWI_BOX_BATCH(K, NP, DEG)                                                                                  \
    else if (family == K)                                                                                           \
        k_batch_box<K, NP, DEG><<<blocks, kBoxThreads, BoxCaps<NP>::kSmem, stream>>>(d_items, d_item_of_tile, work, nwork, \
                                                                                  list, range, sums, d_next);
    KIWI_BOX_KERNELS(KIWI_BOX_BATCH)
#undef KIWI_BOX_BATCH
    KIWI_LAUNCHED(ctx);
    return KIWI_OK;
}

}  // namespace kiwi_b200
