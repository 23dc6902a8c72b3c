// Adjoint of the Cartesian sph-to-grid stage (no counterpart in the reference, which has no gradients).
//
// The forward pass produces, per cell c, the raw sums M_c = sum_p m_p K_pc and P_c = sum_p m_p K_pc v_p,
// where K_pc = max(Msum_pc, 0) is the particle's kernel mass inside the cell (src/cartesian_grid.cpp:
// 256-277).  Given the cotangents gM_c = dL/dM_c and gP_c = dL/dP_c, the adjoint returns per particle
//   dL/dm_p     = sum_c K_pc (gM_c + v_p . gP_c)
//   dL/dv_p     = m_p sum_c K_pc gP_c
//   dL/dtheta_p = m_p sum_c dK_pc/dtheta (gM_c + v_p . gP_c),   theta = x, y, z, h.
// The per-pair cell integrals are recomputed, not stored, with their derivatives in closed form
// (box_grad.cuh): the derivative of a box mass with respect to a side is the kernel's integral over a face.  A
// clamped pair (Msum < 0) has K = 0 and no gradient.  The pairs are those of the forward's default
// evaluation: the cells of the particle's support bounding box whose closest point lies within the support
// radius.
//
// A box mass depends on offsets / H alone, so dT/dh = (ux dT/dx + uy dT/dy + uz dT/dz) / h with the derivatives
// taken with respect to the particle's coordinates (u = plane - particle).
//
// One CTA takes a run of consecutive (tile, particle) entries, tile by tile: their planes, edge lines and lattice
// points are formed once each as in box_tile.cuh, and then each particle's cells are assembled from their 8 corners
// (value and derivatives alike), weighed with the cells' cotangents and summed to the particle's partial gradient for
// this tile, which goes to its entry.  An entry's partial depends on nothing else in the run, so the
// runs are cut to fill the chip whatever the tiles hold.  k_adjoint_reduce adds each particle's entries in tile
// order.  Deterministic, no atomics on the gradients.
//
// Against forward-mode dual numbers through the point-wise series (one CTA per tile, 255 registers with
// spills): 100 k column particles on 80^3, cubic, forward and backward: 53.8 -> 13.5 ms; 2 k particles on 21 x 19 x 25 (36 tiles), Wendland C4:
// 90.0 -> 1.3 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "binning.cuh"
#include "box_grad.cuh"
#include "box_tile.cuh"
#include "cart_common.cuh"
#include "ctx.hpp"
#include "engine.hpp"
#include "kernel_tables.h"
#include "lattice.cuh"
#include "prims.cuh"

namespace kiwi_b200 {

namespace {

constexpr int kAdjThreads = 512, kAdjWarps = kAdjThreads / 32;
constexpr int kAdjPMax = 32;
constexpr int kAdjComps = 4;  // a point's T and its derivatives with respect to x, y, z
constexpr int kAdjUnit = 128;  // cells a warp sums at a time

static __constant__ KiwiBoxTable c_adj_box[KIWI_NUM_KERNELS];

// Chunk capacities: one CTA per SM (a full 8^3 box has 729 points, 243 edge lines and 27 planes).
template <int NP>
struct AdjCaps {
    static constexpr int kPt = NP == 1 ? 2688 : (NP == 2 ? 2190 : 2040), kPair = NP == 1 ? 1023 : (NP == 2 ? 740 : 576),
                         kPlane = NP == 1 ? 352 : (NP == 2 ? 270 : 200);
    static constexpr int kKinds = NP + 1;  // of edge lines (box_tile.cuh)
    // dynamic shared memory, in doubles: the points' values (and before them the lists of lines), the lists of near
    // and far points, the edge records (and after them the units' sums), the plane records
    static constexpr int kOffL = kAdjComps * kPt;
    static constexpr int kOffE = kOffL + kPt;
    static constexpr int kOffP = kOffE + box_grad_edge_stride(NP) * kPair;
    static constexpr int kEnd = kOffP + box_grad_plane_stride(NP) * kPlane;
    static constexpr size_t kSmem = sizeof(double) * kEnd;
    static_assert(kPair <= 1024 && kPlane <= 512 && kPt <= 4096, "BoxGeo's fields and the listed points'");
    static_assert(kKinds * kPair <= 2 * kAdjComps * kPt, "the lists of lines fit");
    static_assert(8 * (kAdjPMax + kPt / kAdjUnit) <= box_grad_edge_stride(NP) * kPair, "the units' sums fit");
};

struct AdjGrads {
    double *x, *y, *z, *h, *m, *vx, *vy, *vz;
};

// Consecutive entries of one tile: their particles and boxes (box_tile.cuh; a box's `cell` is its first unit), and the
// tile's planes and cell centres.
struct AdjChunk {
    double4 at[kAdjPMax], mv[kAdjPMax];
    int4 geo[kAdjPMax];
    double iH[kAdjPMax];
    uint32_t cmag[kAdjPMax], entry[kAdjPMax];
    double pl[3][kTileX + 1], cc[3][kTileX];
    int bx, by, bz;
    int np, ltot, etot, ptot, utot;
    __device__ __forceinline__ BoxGeo box(int j) const { return BoxGeo{geo[j]}; }
};

// The partial gradients of the sorted entries [blockIdx.x per_block, ..): keys their tiles, list their entry
// numbers, owner the particle of an entry; part receives 8 doubles per entry: dL/dm, dL/d(x, y, z, h),
// dL/d(vx, vy, vz) over the entry's tile.
//
// A chunk is a few boxes at most (a point's and a line's records are three to four times the forward's), so what a
// phase gives to a warp has to be cut across boxes: lines by kind and points by piece are listed over the whole CTA and
// taken 32 of a kind by whichever warp is free, and a box's cells are summed in units of kAdjUnit by different warps,
// the units' sums then added in order.  One CTA holds the whole SM's shared memory: three full boxes instead of one in
// each of two.  The kinds share one copy of the code: two copies of each evaluation overflowed the instruction cache.
// Forward and backward of 100 k column particles on 80^3, cubic: 16.6 ms (warps sorting for themselves, a warp to a
// box: half of the warps' time at the barriers) -> 15.3 (lists, units) -> 14.1 (one copy) -> 13.5 (one CTA per SM).
// KERNEL: the kernel's table; NP, DEG: its pieces and largest power.
template <int KERNEL, int NP, int DEG>
__global__ void __launch_bounds__(kAdjThreads, 1) k_cart_adjoint_box(CartGeom g, DevParticles P,
                                                                     const uint32_t* __restrict__ keys,
                                                                     const uint32_t* __restrict__ list,
                                                                     const uint32_t* __restrict__ owner, int64_t total,
                                                                     int per_block, const double* __restrict__ cot,
                                                                     double* __restrict__ part,
                                                                     DevStats* __restrict__ st) {
    using Caps = AdjCaps<NP>;
    __shared__ AdjChunk s_cp[2];
    // listed lines by kind; near points of the first piece, of later ones, far points; (E)'s and (P)'s next batch
    __shared__ int s_lines[Caps::kKinds], s_pts[3], s_next[2];
    constexpr int kCS = kBoxC + kBoxD + 1;
    __shared__ double s_C[kCS * NP];
    extern __shared__ double s_dyn[];
    const KiwiBoxTable& T = c_adj_box[KERNEL];
    constexpr int n = NP, kPS = box_grad_plane_stride(NP), kES = box_grad_edge_stride(NP);
    double* const s_T = s_dyn;
    double* const s_E = s_dyn + Caps::kOffE;
    double* const s_P = s_dyn + Caps::kOffP;
    uint32_t* const s_list = reinterpret_cast<uint32_t*>(s_T);
    uint32_t* const s_near = reinterpret_cast<uint32_t*>(s_dyn + Caps::kOffL);  // first piece from the front, others the back
    uint32_t* const s_far = s_near + Caps::kPt;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1;
    for (int i = threadIdx.x; i < kCS * n; i += kAdjThreads) {
        const int k = i / kCS, c = i % kCS;
        s_C[i] = c < kBoxC ? T.reg[k].C[c] : (c < kBoxC + kBoxD ? T.reg[k].D[c - kBoxC] : T.reg[k].c);
    }
    auto reset = [&]() {
        if (threadIdx.x < Caps::kKinds) s_lines[threadIdx.x] = 0;
        if (threadIdx.x < 3) s_pts[threadIdx.x] = 0;
        if (threadIdx.x < 2) s_next[threadIdx.x] = 0;
    };
    reset();
    const int64_t ncell = (int64_t)g.nx * g.ny * g.nz;
    unsigned n_eval = 0, n_neg = 0;
    const int64_t beg = (int64_t)blockIdx.x * per_block, end = min(beg + (int64_t)per_block, total);

    // warp 0: the entries from `pos` on that lie in its tile, as many as the capacities take
    auto load_chunk = [&](AdjChunk& c, int64_t pos) {
        const uint32_t t = keys[pos];
        const int tz = (int)(t % g.ntz), ty = (int)((t / g.ntz) % g.nty), tx = (int)(t / ((int64_t)g.ntz * g.nty));
        const int bx = tx * kTileX, by = ty * kTileY, bz = tz * kTileZ;
        if (lane < 3 * (kTileX + 1)) {
            const int a = lane / (kTileX + 1), l = lane % (kTileX + 1);
            const double mn = a == 0 ? g.x_min : (a == 1 ? g.y_min : g.z_min);
            const double d = a == 0 ? g.dpx : (a == 1 ? g.dpy : g.dpz);
            const int b0 = a == 0 ? bx : (a == 1 ? by : bz);
            c.pl[a][l] = add_rn(mn, mul_rn((double)(b0 + l), d));
            if (l < kTileX) c.cc[a][l] = cell_centre(mn, b0 + l, d);
        }
        static_assert(3 * (kTileX + 1) <= 32, "a lane per plane of the tile");
        const int64_t idx = pos + lane;
        const bool in = idx < end && keys[idx] == t;
        int nl = 0, ne = 0, npt = 0, nu = 0, lo0 = 0, lo1 = 0, lo2 = 0, d0 = 0, d1 = 0, d2 = 0;
        double px = 0, py = 0, pz = 0, ph = 1, pm = 0, pvx = 0, pvy = 0, pvz = 0;
        uint32_t e = 0;
        if (in) {
            e = list[idx];
            const uint32_t p = owner[e];
            px = P.x[p]; py = P.y[p]; pz = P.z[p]; ph = P.h[p];
            pm = P.m[p]; pvx = P.vx[p]; pvy = P.vy[p]; pvz = P.vz[p];
            CellBox b;
            bool outside;
            particle_cell_box(g, px, py, pz, ph, b, &outside);
            lo0 = max(b.x0 - bx, 0); lo1 = max(b.y0 - by, 0); lo2 = max(b.z0 - bz, 0);
            d0 = min(b.x1 - bx, kTileX - 1) - lo0 + 1;
            d1 = min(b.y1 - by, kTileY - 1) - lo1 + 1;
            d2 = min(b.z1 - bz, kTileZ - 1) - lo2 + 1;
            const int n0 = d0 + 1, n1 = d1 + 1, n2 = d2 + 1;
            nl = n0 + n1 + n2;
            ne = n0 * n1 + n0 * n2 + n1 * n2;
            npt = n0 * n1 * n2;
            nu = (d0 * d1 * d2 + kAdjUnit - 1) / kAdjUnit;
        }
        int il = nl, ie = ne, ip = npt, iu = nu;
        for (int o = 1; o < 32; o <<= 1) {
            const int vl = __shfl_up_sync(0xffffffffu, il, o), ve = __shfl_up_sync(0xffffffffu, ie, o),
                      vp = __shfl_up_sync(0xffffffffu, ip, o), vu = __shfl_up_sync(0xffffffffu, iu, o);
            if (lane >= o) {
                il += vl;
                ie += ve;
                ip += vp;
                iu += vu;
            }
        }
        const bool fits = in && il <= Caps::kPlane && ie <= Caps::kPair && ip <= Caps::kPt;
        const unsigned no = ~__ballot_sync(0xffffffffu, fits);  // the entries before the first that is not taken
        const int np = no ? __ffs((int)no) - 1 : 32;
        if (lane < np) {
            const double H = mul_rn(g.support_in_h, ph);
            c.at[lane] = double4{px, py, pz, H};
            c.mv[lane] = double4{pm, pvx, pvy, pvz};
            c.iH[lane] = 1.0 / H;
            c.entry[lane] = e;
            c.geo[lane] = box_geo(d0 + 1, d1 + 1, d2 + 1, lo0, lo1, lo2, il - nl, ie - ne, ip - npt, iu - nu);
            c.cmag[lane] = box_cell_magic(d1, d2);
        }
        if (lane == np - 1) {
            c.np = np;
            c.ltot = il;
            c.etot = ie;
            c.ptot = ip;
            c.utot = iu;
            c.bx = bx; c.by = by; c.bz = bz;
        }
    };
    // all warps: a chunk's plane records
    auto form_planes = [&](const AdjChunk* cp) {
        const int off_l = lane < cp->np ? cp->box(lane).plane() : INT_MAX, tot = cp->ltot;
        for (int base = warp * 32; base < tot; base += kAdjThreads) {
            const int j = warp_owner(base, off_l, lane), it = base + lane;
            if (it < tot) {
                const BoxGeo b = cp->box(j);
                int l = it - b.plane();
                const int n0 = b.n0(), n1 = b.n1();
                const int a = (l >= n0) + (l >= n0 + n1);
                l -= a == 0 ? 0 : (a == 1 ? n0 : n0 + n1);
                const double4 at = cp->at[j];
                const double c = a == 0 ? at.x : (a == 1 ? at.y : at.z);
                const int lo = a == 0 ? b.lo0() : (a == 1 ? b.lo1() : b.lo2());
                box_grad_plane<NP, DEG>(T, (cp->pl[a][lo + l] - c) * cp->iH[j], s_P + kPS * it);
            }
        }
    };
    // a lane's item to a list: its place, counted in *count from `first` up or down
    auto append = [&](bool mine, int* count, uint32_t* first, bool down, uint32_t rec) {
        const unsigned m = __ballot_sync(0xffffffffu, mine);
        if (m == 0) return;
        int at = 0;
        if (lane == 0) at = atomicAdd(count, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & below);
        if (mine) first[down ? -at : at] = rec;
    };
    // all warps: a chunk's lines by kind and its points by piece, in any order
    auto list_items = [&](const AdjChunk* cp) {
        {
            const int off_l = lane < cp->np ? cp->box(lane).line() : INT_MAX, tot = cp->etot;
            for (int base = warp * 32; base < tot; base += kAdjThreads) {
                const int j = warp_owner(base, off_l, lane), it = base + lane;
                int kind = -1;
                uint32_t rec = 0;
                if (it < tot) {
                    const BoxGeo b = cp->box(j);
                    int la, lb;
                    b.line_planes(it - b.line(), la, lb);
                    const double p = s_P[kPS * la], q = s_P[kPS * lb];
                    const double D = fma(p, p, q * q);
                    rec = (uint32_t)it | (uint32_t)la << 10 | (uint32_t)lb << 19;
                    kind = n;
                    if (D < 1.0 && !(bg_on(p) && bg_on(q))) {
                        kind = 0;
#pragma unroll
                        for (int k = 0; k + 1 < n; ++k) kind += D >= T.scale[k].b * T.scale[k].b;
                    }
                }
#pragma unroll
                for (int c = 0; c < Caps::kKinds; ++c) append(kind == c, &s_lines[c], s_list + Caps::kPair * c, false, rec);
            }
        }
        {
            const int off_l = lane < cp->np ? cp->box(lane).point() : INT_MAX, tot = cp->ptot;
            // (from the last warp on: the first ones had the lines' last share)
            for (int base = (kAdjWarps - 1 - warp) * 32; base < tot; base += kAdjThreads) {
                const int j = warp_owner(base, off_l, lane), it = base + lane;
                int kind = -1;
                uint32_t rec = 0;
                if (it < tot) {
                    const BoxGeo b = cp->box(j);
                    const int lp = it - b.point(), n0 = b.n0(), n1 = b.n1(), n2 = b.n2();
                    const int i = b.by_n12(lp), rem = lp - i * (n1 * n2);
                    const int jj = b.by_n2(rem), k = rem - jj * n2;
                    const double* const rx = s_P + kPS * (b.plane() + i);
                    const double* const ry = s_P + kPS * (b.plane() + n0 + jj);
                    const double* const rz = s_P + kPS * (b.plane() + n0 + n1 + k);
                    const double x = rx[0], y = ry[0], z = rz[0];
                    const double r2 = fma(x, x, fma(y, y, z * z));
                    rec = (uint32_t)(it | j << 12 | i << 17 | jj << 21 | k << 25);
                    kind = (int)bg_on(x) + (int)bg_on(y) + (int)bg_on(z) > 1 || !(r2 < 1.0)
                               ? 2
                               : (n > 1 && r2 >= T.scale[0].b * T.scale[0].b ? 1 : 0);
                }
                append(kind == 0, &s_pts[0], s_near, false, rec);
                if (n > 1) append(kind == 1, &s_pts[1], s_near + Caps::kPt - 1, true, rec);
                append(kind == 2, &s_pts[2], s_far, false, rec);
            }
        }
    };
    auto next_batch = [&](int* counter) {
        int b = 0;
        if (lane == 0) b = atomicAdd(counter, 1);
        return __shfl_sync(0xffffffffu, b, 0);
    };

    const AdjChunk* cp = &s_cp[0];
    if (warp == 0) load_chunk(s_cp[0], beg);
    __syncthreads();
    form_planes(cp);
    __syncthreads();
    list_items(cp);
    __syncthreads();

    for (int64_t pos = beg; pos < end;) {
        AdjChunk& nx = cp == &s_cp[0] ? s_cp[1] : s_cp[0];
        const int np = cp->np;
        const bool more = pos + np < end;
        if (warp == 0 && more) load_chunk(nx, pos + np);

        // (E) edge lines
        {
            int nb = 0, first[Caps::kKinds];  // batches of each kind, the costly ones first
#pragma unroll
            for (int c = 0; c < Caps::kKinds; ++c) {
                first[c] = nb;
                nb += (s_lines[c] + 31) >> 5;
            }
            for (int b = next_batch(&s_next[0]); b < nb; b = next_batch(&s_next[0])) {
                int c = 0, f = 0;
#pragma unroll
                for (int k = 1; k < Caps::kKinds; ++k)
                    if (b >= first[k]) c = k, f = first[k];
                const int e = 32 * (b - f) + lane;
                if (e >= s_lines[c]) continue;
                const uint32_t rec = s_list[Caps::kPair * c + e];
                double* const E = s_E + kES * (rec & 1023u);
                if (c == n) E[6 * n] = E[6 * n + 1] = E[6 * n + 2] = 0.0;
                else box_grad_edge<NP, DEG>(T, c, s_P + kPS * ((rec >> 10) & 511u), s_P + kPS * (rec >> 19), E);
            }
        }
        __syncthreads();

        // (P) points
        {
            const int nn[3] = {s_pts[0], s_pts[1], s_pts[2]};
            const int b1 = (nn[0] + 31) >> 5, b2 = b1 + ((nn[1] + 31) >> 5), nb = b2 + ((nn[2] + 31) >> 5);
            // a point's values, with the offsets' signs: d/d(particle x) of sgn T(|ux|, ..) = -sgn(uy) sgn(uz) T_x; the sign
            // of a plane through the particle is 0, which leaves the derivative across it (none where two planes meet)
            auto sign = [](double u) { return bg_on(u) ? 0.0 : (u > 0.0 ? 1.0 : -1.0); };
            auto put = [&](int it, int j, double x, double y, double z, const double* v) {
                const double iH = cp->iH[j];
                const double sx = sign(x), sy = sign(y), sz = sign(z);
                s_T[it] = sx * sy * sz * v[0];
                s_T[Caps::kPt + it] = -sy * sz * v[1] * iH;
                s_T[2 * Caps::kPt + it] = -sx * sz * v[2] * iH;
                s_T[3 * Caps::kPt + it] = -sx * sy * v[3] * iH;
            };
            for (int b = next_batch(&s_next[1]); b < nb; b = next_batch(&s_next[1])) {
                const int kind = b < b1 ? 0 : (b < b2 ? 1 : 2);
                const int e = 32 * (b - (kind == 0 ? 0 : (kind == 1 ? b1 : b2))) + lane;
                if (e >= (kind == 0 ? nn[0] : (kind == 1 ? nn[1] : nn[2]))) continue;
                const uint32_t rec = kind == 0 ? s_near[e] : (kind == 1 ? s_near[Caps::kPt - 1 - e] : s_far[e]);
                const int it = (int)(rec & 4095u), j = (int)((rec >> 12) & 31u), i = (int)((rec >> 17) & 15u),
                          jj = (int)((rec >> 21) & 15u), kk = (int)(rec >> 25);
                const BoxGeo bg = cp->box(j);
                const int n0 = bg.n0(), n1 = bg.n1(), n2 = bg.n2();
                const double* const rx = s_P + kPS * (bg.plane() + i);
                const double* const ry = s_P + kPS * (bg.plane() + n0 + jj);
                const double* const rz = s_P + kPS * (bg.plane() + n0 + n1 + kk);
                const double* const E = s_E + kES * bg.line();
                const double* const ez = E + kES * (i * n1 + jj);
                const double* const ey = E + kES * (bg.n01() + i * n2 + kk);
                const double* const ex = E + kES * (bg.n0_12() + jj * n2 + kk);
                const double x = rx[0], y = ry[0], z = rz[0];
                double v[4] = {0.0, 0.0, 0.0, 0.0};
                if (kind == 2) {
                    if ((int)bg_on(x) + (int)bg_on(y) + (int)bg_on(z) < 2) {
                        v[0] = (ez[6 * n] + ey[6 * n]) + ex[6 * n] +
                               ((rx[bg_w(n, n)] + ry[bg_w(n, n)]) + (rz[bg_w(n, n)] + box_centre<NP>(T, n)));
                        v[1] = (ez[6 * n + 1] + ey[6 * n + 1]) + rx[bg_dw(n, n)];
                        v[2] = (ez[6 * n + 2] + ex[6 * n + 1]) + ry[bg_dw(n, n)];
                        v[3] = (ey[6 * n + 2] + ex[6 * n + 2]) + rz[bg_dw(n, n)];
                    }
                } else {
                    int k = kind;  // the point's piece
                    if (NP > 2 && kind == 1) {
                        const double r2 = fma(x, x, fma(y, y, z * z));
#pragma unroll
                        for (int s = 1; s + 1 < n; ++s) k += r2 >= T.scale[s].b * T.scale[s].b;
                    }
                    const double* const C = s_C + kCS * k;
                    box_inside_grad<DEG>(C, C + kBoxC, C[kBoxC + kBoxD], T.deg, n, k, rx, ry, rz, ex, ey, ez, v);
                    if (kind > 0) {
                        v[0] += (rx[bg_w(n, k)] + ry[bg_w(n, k)]) + (rz[bg_w(n, k)] + box_centre<NP>(T, k));
                        v[1] += rx[bg_dw(n, k)];
                        v[2] += ry[bg_dw(n, k)];
                        v[3] += rz[bg_dw(n, k)];
                    }
                }
                put(it, j, x, y, z, v);
            }
        }
        __syncthreads();

        // (C) a warp per unit: its cells in box order over the lanes, weighed by the cotangents, and a fixed-order sum
        // over the lanes, into the edge records' place (dead after (P)); and the next chunk's planes
        double* const s_sum = s_E;
        {
            const int off_l = lane < np ? cp->box(lane).cell() : INT_MAX;
            for (int u = warp; u < cp->utot; u += kAdjWarps) {
                const int j = __popc(__ballot_sync(0xffffffffu, off_l <= u)) - 1;
                double acc[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[c] = 0.0;
                const BoxGeo b = cp->box(j);
                const double4 at = cp->at[j], mv = cp->mv[j];
                const double radius = at.w, sih = g.support_in_h * cp->iH[j];
                const int d1 = b.n1() - 1, d2 = b.n2() - 1, n2 = d2 + 1, n12 = (d1 + 1) * n2;
                const int l0 = b.lo0(), l1 = b.lo1(), l2 = b.lo2();
                const int c0 = kAdjUnit * (u - b.cell()), c1 = min(c0 + kAdjUnit, (b.n0() - 1) * d1 * d2);
                for (int lc = c0 + lane; lc < c1; lc += 32) {
                    int i, jj, k;
                    box_cell(cp->cmag[j], lc, d1, d2, i, jj, k);
                    const double ex = fmax(fabs(at.x - cp->cc[0][l0 + i]) - g.hpx, 0.0);
                    const double ey = fmax(fabs(at.y - cp->cc[1][l1 + jj]) - g.hpy, 0.0);
                    const double ez = fmax(fabs(at.z - cp->cc[2][l2 + k]) - g.hpz, 0.0);
                    if (!(add_rn(add_rn(mul_rn(ex, ex), mul_rn(ey, ey)), mul_rn(ez, ez)) < mul_rn(radius, radius))) continue;
                    ++n_eval;
                    const double* const Tp = s_T + b.point() + i * n12 + jj * n2 + k;
                    const double m1 = (Tp[n12 + n2 + 1] - Tp[n12 + n2]) - (Tp[n12 + 1] - Tp[n12]);
                    const double m0 = (Tp[n2 + 1] - Tp[n2]) - (Tp[1] - Tp[0]);
                    const double msum = m1 - m0;
                    if (msum < 0.0) {
                        ++n_neg;
                        continue;
                    }
                    if (msum == 0.0) continue;
                    const int64_t i3 = ((int64_t)(cp->bx + l0 + i) * g.ny + (cp->by + l1 + jj)) * g.nz + (cp->bz + l2 + k);
                    const double gx = cot[ncell + i3], gy = cot[2 * ncell + i3], gz = cot[3 * ncell + i3];
                    const double gs = fma(mv.w, gz, fma(mv.z, gy, fma(mv.y, gx, cot[i3])));
                    acc[0] = fma(msum, gs, acc[0]);
                    acc[5] = fma(msum, gx, acc[5]);
                    acc[6] = fma(msum, gy, acc[6]);
                    acc[7] = fma(msum, gz, acc[7]);
                    // each derivative's sum over the corners of either plane of its axis: their difference is the cell's,
                    // and weighed with the planes' offsets it is that axis's part of d/dh
                    double dh = 0.0;
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        const double* const q = Tp + (a + 1) * Caps::kPt;
                        const double z11 = q[n12 + n2 + 1] - q[n12 + n2], z10 = q[n12 + 1] - q[n12], z01 = q[n2 + 1] - q[n2],
                                     z00 = q[1] - q[0];
                        const double hi = a == 0 ? z11 - z10 : (a == 1 ? z11 - z01
                                                                       : (q[n12 + n2 + 1] - q[n12 + 1]) - (q[n2 + 1] - q[1]));
                        const double lo = a == 0 ? z01 - z00 : (a == 1 ? z10 - z00 : (q[n12 + n2] - q[n12]) - (q[n2] - q[0]));
                        const int l = a == 0 ? l0 + i : (a == 1 ? l1 + jj : l2 + k);
                        const double x0 = a == 0 ? at.x : (a == 1 ? at.y : at.z);
                        acc[1 + a] = fma(hi - lo, gs, acc[1 + a]);
                        dh = fma(cp->pl[a][l + 1] - x0, hi, dh);
                        dh = fma(-(cp->pl[a][l] - x0), lo, dh);
                    }
                    acc[4] = fma(sih * dh, gs, acc[4]);
                }
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
                double v = 0.0;
#pragma unroll
                for (int c = 0; c < 8; ++c) v = lane == c ? acc[c] : v;
                if (lane < 8) s_sum[8 * u + lane] = v;
            }
        }
        reset();
        if (more) form_planes(&nx);
        __syncthreads();

        // each entry's units in order; and the next chunk's lists
        if (threadIdx.x < 8 * np) {
            const int j = threadIdx.x >> 3, c = threadIdx.x & 7;
            const int u1 = j + 1 < np ? cp->box(j + 1).cell() : cp->utot;
            int u = cp->box(j).cell();
            double v = s_sum[8 * u + c];
            for (++u; u < u1; ++u) v += s_sum[8 * u + c];
            part[8 * (int64_t)cp->entry[j] + c] = c == 0 ? v : cp->mv[j].x * v;
        }
        if (more) list_items(&nx);
        __syncthreads();
        pos += np;
        cp = &nx;
    }
    for (int o = 16; o > 0; o >>= 1) {
        n_eval += __shfl_down_sync(0xffffffffu, n_eval, o);
        n_neg += __shfl_down_sync(0xffffffffu, n_neg, o);
    }
    if (lane == 0) {
        if (n_eval) atomicAdd(&st->evaluated_pairs, (unsigned long long)n_eval);
        if (n_neg) atomicAdd(&st->neg_clamped, (unsigned long long)n_neg);
    }
}

// Each particle's gradient: its entries' partial sums in tile order.
__global__ void k_adjoint_reduce(int64_t n, const int64_t* __restrict__ offs, const double* __restrict__ part,
                                 AdjGrads G) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    double acc[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c] = 0.0;
    for (int64_t e = offs[p]; e < offs[p + 1]; ++e)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[c] += part[8 * e + c];
    if (G.m) G.m[p] = acc[0];
    if (G.x) G.x[p] = acc[1];
    if (G.y) G.y[p] = acc[2];
    if (G.z) G.z[p] = acc[3];
    if (G.h) G.h[p] = acc[4];
    if (G.vx) G.vx[p] = acc[5];
    if (G.vy) G.vy[p] = acc[6];
    if (G.vz) G.vz[p] = acc[7];
}

}  // namespace

int adjoint_init_tables(KiwiCtx* ctx) {
    KIWI_CUDA(ctx, cudaMemcpyToSymbol(c_adj_box, kiwi_box_tables, sizeof(kiwi_box_tables)));
    return KIWI_OK;
}

int cart_adjoint_dev(KiwiCtx* ctx, const DevParticles& P, const CartGeom& g, const KernelChoice& kc,
                     const double* d_cot, const AdjointOutputs& out, KiwiStats* stats) {
    if (kc.tabulated)
        return set_err(ctx, KIWI_ERR_UNSUPPORTED,
                       "the adjoint is available for the analytic integrals (cubic closed form and the generic "
                       "kernels' tables), not for the tabulated one");
    DevStats* d_st = nullptr;
    KIWI_TRY(scratch_t(ctx, S_STATS, 1, &d_st));
    KIWI_CUDA(ctx, cudaMemsetAsync(d_st, 0, sizeof(DevStats), ctx->stream));
    const int64_t n = P.n;
    const int64_t ntiles = (int64_t)g.ntx * g.nty * g.ntz;
    // binning as the forward pass, with the sort carrying each (tile, particle) entry's index
    uint32_t* counts = nullptr;
    TileBox* boxes = nullptr;
    int64_t* offs = nullptr;
    KIWI_TRY(scratch_t(ctx, S_COUNT, (size_t)std::max<int64_t>(n, 1), &counts));
    KIWI_TRY(scratch_t(ctx, S_BOX, (size_t)std::max<int64_t>(n, 1), &boxes));
    KIWI_TRY(scratch_t(ctx, S_OFFS, (size_t)std::max<int64_t>(n, 1) + 1, &offs));
    int64_t* d_total = offs + std::max<int64_t>(n, 1);
    if (n > 0) {
        k_tile_counts<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(g, P, counts, boxes, d_st);
        KIWI_LAUNCHED(ctx);
    }
    KIWI_TRY(exclusive_scan<uint32_t>(ctx, counts, n, offs, d_total));
    int64_t total = 0;
    KIWI_CUDA(ctx, cudaMemcpyAsync(&total, d_total, sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream));
    KIWI_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (total >= (1LL << 32)) return set_err(ctx, KIWI_ERR_LIMIT, "too many (tile, particle) entries: %lld", (long long)total);
    uint32_t *k0, *v0, *k1, *v1;
    double* part = nullptr;
    KIWI_TRY(scratch_t(ctx, S_KEYS0, (size_t)std::max<int64_t>(total, 1), &k0));
    KIWI_TRY(scratch_t(ctx, S_VALS0, (size_t)std::max<int64_t>(total, 1), &v0));
    KIWI_TRY(scratch_t(ctx, S_KEYS1, (size_t)std::max<int64_t>(total, 1), &k1));
    KIWI_TRY(scratch_t(ctx, S_VALS1, (size_t)std::max<int64_t>(total, 1), &v1));
    KIWI_TRY(scratch_t(ctx, S_ADJ_PART, (size_t)8 * std::max<int64_t>(total, 1), &part));
    if (total > 0) {
        uint32_t* owner = nullptr;
        KIWI_TRY(scratch_t(ctx, S_ADJ_OWNER, (size_t)total, &owner));
        k_tile_emit<<<(unsigned)((total + 255) / 256), 256, 0, ctx->stream>>>(g, n, offs, boxes, 0, total, 0u, k0, v0,
                                                                              owner);
        KIWI_LAUNCHED(ctx);
        int key_bits = 1;
        while ((1LL << key_bits) < ntiles) ++key_bits;
        bool second = false;
        KIWI_TRY(radix_sort_pairs(ctx, k0, v0, k1, v1, total, key_bits, &second));
        const uint32_t *sk = second ? k1 : k0, *sv = second ? v1 : v0;
        // entries per CTA: about sixteen CTAs for each of the chip's SMs, so that uneven entries level out,
        // within 16 (two chunks of large boxes) .. 256
        int sms = 148;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
        const int per = (int)std::min<int64_t>(256, std::max<int64_t>(16, total / (16 * (int64_t)sms)));
        const unsigned blocks = (unsigned)((total + per - 1) / per);
#define KIWI_ADJ_LAUNCH(K, NP, DEG)                                                                                      \
    if (kc.kernel == K) {                                                                                               \
        KIWI_CUDA(ctx, cudaFuncSetAttribute(k_cart_adjoint_box<K, NP, DEG>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                            (int)AdjCaps<NP>::kSmem));                                                  \
        k_cart_adjoint_box<K, NP, DEG><<<blocks, kAdjThreads, AdjCaps<NP>::kSmem, ctx->stream>>>(g, P, sk, sv, owner,    \
                                                                                             total, per, d_cot, part,   \
                                                                                             d_st);                     \
    }
        KIWI_BOX_KERNELS(KIWI_ADJ_LAUNCH)
#undef KIWI_ADJ_LAUNCH
        KIWI_LAUNCHED(ctx);
    }
    if (n > 0) {
        AdjGrads G{out.x, out.y, out.z, out.h, out.m, out.vx, out.vy, out.vz};
        k_adjoint_reduce<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(n, offs, part, G);
        KIWI_LAUNCHED(ctx);
    }
    if (stats) {
        DevStats h;
        KIWI_CUDA(ctx, cudaMemcpyAsync(&h, d_st, sizeof(DevStats), cudaMemcpyDeviceToHost, ctx->stream));
        KIWI_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        stats->evaluated_pairs = (int64_t)h.evaluated_pairs;
        stats->neg_clamped = (int64_t)h.neg_clamped;
        stats->skipped_outside = (int64_t)h.skipped_outside;
        stats->tile_pairs = total;
    }
    return KIWI_OK;
}

}  // namespace kiwi_b200
