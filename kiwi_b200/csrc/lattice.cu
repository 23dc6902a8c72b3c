// The lattice-factorised gather of the plain FP64 form (cubic spline closed form and table-driven generic
// kernels) and the batch's persistent kernel for those two families.  This translation unit is built with
// FMA contraction: the lattice form regroups the reference's sum (lattice_tile.cuh) and evaluates its tiers
// in the triangles' own lengths (lattice_math.cuh), so it does not follow the reference's operation order
// and gains nothing from rounding each product on its own; the quantities that integer results depend on
// (bounding boxes, lattice planes, cell centres, the support test of the pair counters) are formed with
// explicitly rounded operations (cart_common.cuh), as in every other form.
#include <cuda_runtime.h>

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

// Resident CTAs per SM the register budget is sized for: two for both kernels (128 registers).  The cubic
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
#ifndef KIWI_BOX_GEN_MIN_BLOCKS
#define KIWI_BOX_GEN_MIN_BLOCKS 2
#endif
constexpr int kBoxMinBlocks = KIWI_BOX_MIN_BLOCKS;
constexpr int kBoxGenMinBlocks = KIWI_BOX_GEN_MIN_BLOCKS;
constexpr size_t kBoxSmem = BoxCaps<2>::kSmem, kBoxGenSmem = BoxCaps<0>::kSmem;
constexpr size_t kBoxMergedSmem = kBoxSmem > kBoxGenSmem ? kBoxSmem : kBoxGenSmem;

template <bool CULL>
__global__ void __launch_bounds__(kBoxThreads, kBoxMinBlocks) k_cart_box(CartGeom g, DevParticles P,
                                                                         const uint32_t* __restrict__ list,
                                                                         const int64_t* __restrict__ range,
                                                                         const int32_t* __restrict__ tile_map,
                                                                         CartOutputs out, DevStats* __restrict__ st) {
    const int64_t t = tile_map ? (int64_t)tile_map[blockIdx.x] : (int64_t)blockIdx.x;
    box_tile<CULL, 2, 3>(g, P, list, range, t, t, out, st, c_box[0]);
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
    lattice_tile<true, false, false, true>(g, P, list, range, t, t, out, st);
}

// Any kernel of the tables (support cells only).
__global__ void __launch_bounds__(kBoxThreads, kBoxGenMinBlocks) k_cart_box_generic(CartGeom g, DevParticles P, int kernel,
                                                                               const uint32_t* __restrict__ list,
                                                                               const int64_t* __restrict__ range,
                                                                               const int32_t* __restrict__ tile_map,
                                                                               CartOutputs out,
                                                                               DevStats* __restrict__ st) {
    const int64_t t = tile_map ? (int64_t)tile_map[blockIdx.x] : (int64_t)blockIdx.x;
    box_tile<true, 0, 0>(g, P, list, range, t, t, out, st, c_box[kernel]);
}

// The FP32-mixed form of the generic lattice kernel: edge records and vertex tiers in FP32 (FP64 islands
// where a plane lies within 1e-3 h of the particle), records, cell assembly and per-cell sums in FP64.
__global__ void __launch_bounds__(kLatThreads, kLatGenMinBlocks)
    k_cart_lattice_generic_mixed(CartGeom g, DevParticles P, int kernel, const uint32_t* __restrict__ list,
                                 const int64_t* __restrict__ range, const int32_t* __restrict__ tile_map,
                                 CartOutputs out, DevStats* __restrict__ st) {
    const int64_t t = tile_map ? (int64_t)tile_map[blockIdx.x] : (int64_t)blockIdx.x;
    lattice_tile<true, true, false, true>(g, P, list, range, t, t, out, st, &c_tables[kernel]);
}

// The tiles of a batch of grids, one persistent launch per lattice family, or one for both
// (kBatchFamilyLatticeMerged: each tile takes its item's body): each CTA takes the next of the launch's
// tiles (order[w]) from the work counter and runs the same tile body as the single-grid kernel, so every
// cell's summation order is that of a single-grid call.  MIXED: the FP32-mixed tile bodies.
template <int FAMILY, bool MIXED>
__global__ void __launch_bounds__(MIXED ? kLatThreads : kBoxThreads, 2)
    k_batch_lattice(const BatchItemDev* __restrict__ items, const int32_t* __restrict__ item_of_tile,
                    const int32_t* __restrict__ order, int64_t ntiles, const uint32_t* __restrict__ list,
                    const int64_t* __restrict__ range, unsigned long long* __restrict__ next) {
    __shared__ long long s_w;
    for (;;) {
        if (threadIdx.x == 0) s_w = (long long)atomicAdd(next, 1ull);
        __syncthreads();
        const int64_t w = s_w;
        if (w >= ntiles) break;
        const int64_t tg = (int64_t)order[w];
        const BatchItemDev& it = items[item_of_tile[tg]];
        const int64_t tl = tg - it.tile_base;
        const bool cubic = FAMILY == kBatchFamilyLattice || (FAMILY == kBatchFamilyLatticeMerged && it.mode == kBatchLattice);
        if (MIXED) {
            if (cubic) lattice_tile<true, false, false, true>(it.g, it.P, list, range, tg, tl, it.out, it.st);
            else lattice_tile<true, true, false, true>(it.g, it.P, list, range, tg, tl, it.out, it.st, &c_tables[it.kernel]);
        } else {
            if (cubic) box_tile<true, 2, 3>(it.g, it.P, list, range, tg, tl, it.out, it.st, c_box[0]);
            else box_tile<true, 0, 0>(it.g, it.P, list, range, tg, tl, it.out, it.st, c_box[it.kernel]);
        }
        __syncthreads();
    }
}

// The shared memory and block size of a batch launch.
template <int FAMILY, bool MIXED>
constexpr size_t batch_smem() {
    if (MIXED)
        return FAMILY == kBatchFamilyLattice ? kLatDynSmem
                                             : (FAMILY == kBatchFamilyLatticeMerged ? kLatMergedDynSmem : kLatGenDynSmem);
    return FAMILY == kBatchFamilyLattice ? kBoxSmem : (FAMILY == kBatchFamilyLatticeMerged ? kBoxMergedSmem : kBoxGenSmem);
}

}  // namespace

template <class K, class... A>
static int box_launch(KiwiCtx* ctx, K* kernel, size_t smem, dim3 grid, A... args) {
    KIWI_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kernel<<<grid, kBoxThreads, smem, ctx->stream>>>(args...);
    KIWI_LAUNCHED(ctx);
    return KIWI_OK;
}

int lattice_cart_gather(KiwiCtx* ctx, const CartGeom& g, const DevParticles& P, const KernelChoice& k,
                        const TileLists& tl, const CartOutputs& out, DevStats* d_stats, bool full_box) {
    const dim3 grid((unsigned)(tl.map ? tl.nmap : tl.ntiles));
    if (!k.cubic)
        return box_launch(ctx, k_cart_box_generic, kBoxGenSmem, grid, g, P, k.kernel, tl.list, tl.range, tl.map, out,
                          d_stats);
    if (full_box) return box_launch(ctx, k_cart_box<false>, kBoxSmem, grid, g, P, tl.list, tl.range, tl.map, out, d_stats);
    return box_launch(ctx, k_cart_box<true>, kBoxSmem, grid, g, P, tl.list, tl.range, tl.map, out, d_stats);
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

template <int FAMILY, bool MIXED>
static int batch_prepare_t(KiwiCtx* ctx) {
    KIWI_CUDA(ctx, cudaFuncSetAttribute(k_batch_lattice<FAMILY, MIXED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)batch_smem<FAMILY, MIXED>()));
    return KIWI_OK;
}

template <bool MIXED>
static int batch_prepare_form(KiwiCtx* ctx) {
    KIWI_TRY((batch_prepare_t<kBatchFamilyLattice, MIXED>(ctx)));
    KIWI_TRY((batch_prepare_t<kBatchFamilyLatticeGeneric, MIXED>(ctx)));
    return batch_prepare_t<kBatchFamilyLatticeMerged, MIXED>(ctx);
}

int lattice_batch_prepare(KiwiCtx* ctx) {
    KIWI_TRY(batch_prepare_form<false>(ctx));
    return batch_prepare_form<true>(ctx);
}

template <int FAMILY, bool MIXED>
static void batch_launch_t(KiwiCtx* ctx, const BatchItemDev* d_items, const int32_t* d_item_of_tile,
                           const int32_t* d_order, int64_t ntiles, const uint32_t* list, const int64_t* range,
                           unsigned long long* d_next, int blocks) {
    k_batch_lattice<FAMILY, MIXED><<<blocks, MIXED ? kLatThreads : kBoxThreads, batch_smem<FAMILY, MIXED>(), ctx->stream>>>(
        d_items, d_item_of_tile, d_order, ntiles, list, range, d_next);
}

template <bool MIXED>
static void batch_launch_form(KiwiCtx* ctx, int family, const BatchItemDev* d_items, const int32_t* d_item_of_tile,
                              const int32_t* d_order, int64_t ntiles, const uint32_t* list, const int64_t* range,
                              unsigned long long* d_next, int blocks) {
    if (family == kBatchFamilyLattice)
        batch_launch_t<kBatchFamilyLattice, MIXED>(ctx, d_items, d_item_of_tile, d_order, ntiles, list, range, d_next, blocks);
    else if (family == kBatchFamilyLatticeMerged)
        batch_launch_t<kBatchFamilyLatticeMerged, MIXED>(ctx, d_items, d_item_of_tile, d_order, ntiles, list, range,
                                                         d_next, blocks);
    else
        batch_launch_t<kBatchFamilyLatticeGeneric, MIXED>(ctx, d_items, d_item_of_tile, d_order, ntiles, list, range,
                                                          d_next, blocks);
}

int lattice_batch_gather(KiwiCtx* ctx, int family, const BatchItemDev* d_items, const int32_t* d_item_of_tile,
                         const int32_t* d_order, int64_t ntiles, const uint32_t* list, const int64_t* range,
                         unsigned long long* d_next, int blocks, bool mixed) {
    if (mixed)
        batch_launch_form<true>(ctx, family, d_items, d_item_of_tile, d_order, ntiles, list, range, d_next, blocks);
    else
        batch_launch_form<false>(ctx, family, d_items, d_item_of_tile, d_order, ntiles, list, range, d_next, blocks);
    KIWI_LAUNCHED(ctx);
    return KIWI_OK;
}

}  // namespace kiwi_b200
