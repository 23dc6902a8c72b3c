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
// points are formed once each as in box_tile.cuh, and then a warp takes each particle, assembles its cells from
// their 8 corners (value and derivatives alike), weighs them with the cells' cotangents and writes the particle's
// partial gradient for this tile to its entry.  An entry's partial depends on nothing else in the run, so the
// runs are cut to fill the chip whatever the tiles hold.  k_adjoint_reduce adds each particle's entries in tile
// order.  Deterministic, no atomics on the gradients.
//
// Against forward-mode dual numbers through the point-wise series (one CTA per tile, 255 registers with
// spills): 100 k column particles on 80^3, cubic, forward and backward: 53.8 -> 17.2 ms; 2 k particles on 21 x 19 x 25 (36 tiles), Wendland C4:
// 90.0 -> 5.2 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "binning.cuh"
#include "box_grad.cuh"
#include "cart_common.cuh"
#include "ctx.hpp"
#include "engine.hpp"
#include "kernel_tables.h"
#include "lattice.cuh"
#include "prims.cuh"

namespace kiwi_b200 {

namespace {

constexpr int kAdjThreads = 256, kAdjWarps = kAdjThreads / 32;
constexpr int kAdjPMax = 32;
constexpr int kAdjComps = 5;  // a point's T and its derivatives with respect to x, y, z, h

static __constant__ KiwiBoxTable c_adj_box[KIWI_NUM_KERNELS];

// Chunk capacities: two CTAs per SM (a full 8^3 box has 729 points, 243 edge lines and 27 planes).
template <int NP>
struct AdjCaps {
    static constexpr int kN = NP;
    static constexpr int kPt = NP == 1 ? 1280 : (NP == 2 ? 1024 : 800), kPair = NP == 1 ? 512 : (NP == 2 ? 352 : 272),
                         kPlane = NP == 1 ? 192 : (NP == 2 ? 136 : 120);
    static constexpr int kOffE = kAdjComps * kPt;
    static constexpr int kOffP = kOffE + box_grad_edge_stride(kN) * kPair;
    static constexpr int kEnd = kOffP + box_grad_plane_stride(kN) * kPlane;
    static constexpr size_t kSmem = sizeof(double) * kEnd + sizeof(uint32_t) * 64 * kAdjWarps * kN;
    static_assert(kPair <= 1024 && kPlane <= 512, "packed edge entries");
};

struct AdjGrads {
    double *x, *y, *z, *h, *m, *vx, *vy, *vz;
};

struct AdjChunk {
    double x[kAdjPMax], y[kAdjPMax], z[kAdjPMax], H[kAdjPMax], iH[kAdjPMax], m[kAdjPMax], vx[kAdjPMax], vy[kAdjPMax],
        vz[kAdjPMax];
    int lo[kAdjPMax][3], dim[kAdjPMax][3];  // lo relative to the tile
    int loff[kAdjPMax], eoff[kAdjPMax], poff[kAdjPMax];
    uint32_t entry[kAdjPMax];
    uint32_t mag[kAdjPMax][3];   // div_magic of n1', n2' and n1' n2'
    uint32_t cmag[kAdjPMax][2];  // div_magic of n2 and n1 n2
    int np, ltot, etot, ptot;
};

// The partial gradients of the sorted entries [blockIdx.x per_block, ..): keys their tiles, list their entry
// numbers, owner the particle of an entry; part receives 8 doubles per entry: dL/dm, dL/d(x, y, z, h),
// dL/d(vx, vy, vz) over the entry's tile.
// KERNEL: the kernel's table; NP, DEG: its pieces and largest power.
template <int KERNEL, int NP, int DEG>
__global__ void __launch_bounds__(kAdjThreads, 2) k_cart_adjoint_box(CartGeom g, DevParticles P,
                                                                     const uint32_t* __restrict__ keys,
                                                                     const uint32_t* __restrict__ list,
                                                                     const uint32_t* __restrict__ owner, int64_t total,
                                                                     int per_block, const double* __restrict__ cot,
                                                                     double* __restrict__ part,
                                                                     DevStats* __restrict__ st) {
    using Caps = AdjCaps<NP>;
    __shared__ AdjChunk s_cp;
    __shared__ double s_pl[3][kTileX + 1], s_cc[3][kTileX];
    __shared__ double s_C[NP == 2 ? 1 : (kBoxC + kBoxD + 1) * NP];
    __shared__ int64_t s_seg_end;
    extern __shared__ double s_dyn[];
    const KiwiBoxTable& T = c_adj_box[KERNEL];
    constexpr int n = NP, kPS = box_grad_plane_stride(NP), kES = box_grad_edge_stride(NP);
    double* const s_T = s_dyn;
    double* const s_E = s_dyn + Caps::kOffE;
    double* const s_P = s_dyn + Caps::kOffP;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1;
    uint32_t* const s_q = reinterpret_cast<uint32_t*>(s_dyn + Caps::kEnd) + 64 * Caps::kN * warp;
    constexpr int kCS = kBoxC + kBoxD + 1;
    if (NP != 2)
        for (int i = threadIdx.x; i < kCS * n; i += kAdjThreads) {
            const int k = i / kCS, c = i % kCS;
            s_C[i] = c < kBoxC ? T.reg[k].C[c] : (c < kBoxC + kBoxD ? T.reg[k].D[c - kBoxC] : T.reg[k].c);
        }
    const int64_t ncell = (int64_t)g.nx * g.ny * g.nz;
    unsigned n_eval = 0, n_neg = 0;
    const int64_t beg = (int64_t)blockIdx.x * per_block, end = min(beg + (int64_t)per_block, total);

    for (int64_t pos = beg; pos < end;) {
        // the run of this tile's entries
        const int64_t t = keys[pos];
        __syncthreads();
        if (warp == 0) {
            int64_t e = pos;
            for (;;) {  // at most per_block / 32 steps
                const int64_t i = e + lane;
                const unsigned same = __ballot_sync(0xffffffffu, i < end && keys[i] == (uint32_t)t);
                e += __popc(same);
                if (same != 0xffffffffu) break;
            }
            if (lane == 0) s_seg_end = e;
        }
        const int tz = (int)(t % g.ntz), ty = (int)((t / g.ntz) % g.nty), tx = (int)(t / ((int64_t)g.ntz * g.nty));
        const int bx = tx * kTileX, by = ty * kTileY, bz = tz * kTileZ;
        if (threadIdx.x >= 32 && threadIdx.x < 32 + 3 * (kTileX + 1)) {
            const int i = threadIdx.x - 32, a = i / (kTileX + 1), l = i % (kTileX + 1);
            const double mn = a == 0 ? g.x_min : (a == 1 ? g.y_min : g.z_min);
            const double d = a == 0 ? g.dpx : (a == 1 ? g.dpy : g.dpz);
            const int b0 = a == 0 ? bx : (a == 1 ? by : bz);
            s_pl[a][l] = add_rn(mn, mul_rn((double)(b0 + l), d));
            if (l < kTileX) s_cc[a][l] = cell_centre(mn, b0 + l, d);
        }
        __syncthreads();
        const int64_t seg_end = s_seg_end;

        for (; pos < seg_end;) {
            // (L) the next particles, as many as the capacities take
            if (warp == 0) {
                const int64_t idx = pos + lane;
                int nl = 0, ne = 0, npt = 0, lo0 = 0, lo1 = 0, lo2 = 0, d0 = 0, d1 = 0, d2 = 0;
                double px = 0, py = 0, pz = 0, ph = 1, pm = 0, pvx = 0, pvy = 0, pvz = 0;
                uint32_t e = 0;
                if (idx < seg_end) {
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
                }
                int il = nl, ie = ne, ip = npt;
                for (int o = 1; o < 32; o <<= 1) {
                    const int vl = __shfl_up_sync(0xffffffffu, il, o), ve = __shfl_up_sync(0xffffffffu, ie, o),
                              vp = __shfl_up_sync(0xffffffffu, ip, o);
                    if (lane >= o) {
                        il += vl;
                        ie += ve;
                        ip += vp;
                    }
                }
                const bool take = idx < seg_end && il <= Caps::kPlane && ie <= Caps::kPair && ip <= Caps::kPt;
                const int np = __popc(__ballot_sync(0xffffffffu, take));
                AdjChunk& c = s_cp;
                if (take) {
                    const double H = mul_rn(g.support_in_h, ph);
                    c.x[lane] = px; c.y[lane] = py; c.z[lane] = pz; c.H[lane] = H; c.iH[lane] = 1.0 / H;
                    c.m[lane] = pm; c.vx[lane] = pvx; c.vy[lane] = pvy; c.vz[lane] = pvz;
                    c.lo[lane][0] = lo0; c.lo[lane][1] = lo1; c.lo[lane][2] = lo2;
                    c.dim[lane][0] = d0; c.dim[lane][1] = d1; c.dim[lane][2] = d2;
                    c.loff[lane] = il - nl;
                    c.eoff[lane] = ie - ne;
                    c.poff[lane] = ip - npt;
                    c.entry[lane] = e;
                    c.mag[lane][0] = div_magic(d1 + 1);
                    c.mag[lane][1] = div_magic(d2 + 1);
                    c.mag[lane][2] = div_magic((d1 + 1) * (d2 + 1));
                    c.cmag[lane][0] = div_magic(d2);
                    c.cmag[lane][1] = div_magic(d1 * d2);
                }
                if (lane == np - 1) {
                    c.np = np;
                    c.ltot = il;
                    c.etot = ie;
                    c.ptot = ip;
                }
            }
            __syncthreads();
            const AdjChunk* const cp = &s_cp;
            const int np = cp->np;

            // (A) planes
            {
                const int off_l = lane < np ? cp->loff[lane] : INT_MAX, tot = cp->ltot;
                for (int base = warp * 32; base < tot; base += kAdjThreads) {
                    const int j = warp_owner(base, off_l, lane), it = base + lane;
                    const int off = __shfl_sync(0xffffffffu, off_l, j & 31);
                    if (it < tot) {
                        int l = it - off;
                        const int n0 = cp->dim[j][0] + 1, n1 = cp->dim[j][1] + 1;
                        const int a = (l >= n0) + (l >= n0 + n1);
                        l -= a == 0 ? 0 : (a == 1 ? n0 : n0 + n1);
                        const double c = a == 0 ? cp->x[j] : (a == 1 ? cp->y[j] : cp->z[j]);
                        box_grad_plane<NP, DEG>(T, (s_pl[a][cp->lo[j][a] + l] - c) * cp->iH[j], s_P + kPS * it);
                    }
                }
            }
            __syncthreads();

            // (E) edge lines, queued by piece as in box_tile
            {
                const int tot = cp->etot;
                const int off_l = lane < np ? cp->eoff[lane] : INT_MAX;
                int cnt[Caps::kN];
#pragma unroll
                for (int c = 0; c < Caps::kN; ++c) cnt[c] = 0;
                for (int base = warp * 32;; base += kAdjThreads) {
                    const bool last = base >= tot;
                    if (!last) {
                        const int j = warp_owner(base, off_l, lane), it = base + lane;
                        const int off = __shfl_sync(0xffffffffu, off_l, j & 31);
                        int kind = -1;
                        uint32_t rec = 0;
                        if (it < tot) {
                            int e = it - off;
                            const int n0 = cp->dim[j][0] + 1, n1 = cp->dim[j][1] + 1, n2 = cp->dim[j][2] + 1;
                            const int nxy = n0 * n1, nxz = n0 * n2;
                            const int blk = (e >= nxy) + (e >= nxy + nxz);
                            e -= blk == 0 ? 0 : (blk == 1 ? nxy : nxy + nxz);
                            const int pi = div_by(e, cp->mag[j][blk == 0 ? 0 : 1]), qi = e - pi * (blk == 0 ? n1 : n2);
                            const int la = cp->loff[j] + (blk == 2 ? n0 : 0) + pi;
                            const int lb = cp->loff[j] + (blk == 0 ? n0 : n0 + n1) + qi;
                            const double p = s_P[kPS * la], q = s_P[kPS * lb];
                            const double D = fma(p, p, q * q);
                            if (D >= 1.0 || p == 0.0 || q == 0.0) {
                                double* const E = s_E + kES * it + 6 * n;
                                E[0] = E[1] = E[2] = 0.0;
                            } else {
                                kind = 0;
#pragma unroll
                                for (int k = 0; k + 1 < n; ++k) kind += D >= T.scale[k].b * T.scale[k].b;
                                rec = (uint32_t)it | (uint32_t)la << 10 | (uint32_t)lb << 19;
                            }
                        }
#pragma unroll
                        for (int c = 0; c < Caps::kN; ++c) {
                            const unsigned m = __ballot_sync(0xffffffffu, kind == c);
                            if (kind == c) s_q[64 * c + cnt[c] + __popc(m & below)] = rec;
                            cnt[c] += __popc(m);
                        }
                        __syncwarp();
                    }
#pragma unroll
                    for (int c = 0; c < Caps::kN; ++c) {
                        if (cnt[c] >= 32 || (last && cnt[c] > 0)) {
                            const int first = max(cnt[c] - 32, 0);
                            if (first + lane < cnt[c]) {
                                const uint32_t rec = s_q[64 * c + first + lane];
                                box_grad_edge<NP, DEG>(T, c, s_P + kPS * ((rec >> 10) & 511u), s_P + kPS * (rec >> 19),
                                                       s_E + kES * (rec & 1023u));
                            }
                            cnt[c] = first;
                            __syncwarp();
                        }
                    }
                    if (last) break;
                }
            }
            __syncthreads();

            // (P) points
            {
                const int tot = cp->ptot;
                const int off_l = lane < np ? cp->poff[lane] : INT_MAX;
                int cnt = 0;
                // a point's values, with the offsets' signs: d/d(particle x) of sgn T(|ux|, ..) = -sgn(uy) sgn(uz) T_x
                auto put = [&](int it, int j, const double* rx, const double* ry, const double* rz, const double* v) {
                    const double iH = cp->iH[j];
                    const double x = rx[0], y = ry[0], z = rz[0];
                    const double sx = x > 0.0 ? 1.0 : -1.0, sy = y > 0.0 ? 1.0 : -1.0, sz = z > 0.0 ? 1.0 : -1.0;
                    const double tx_ = -sy * sz * v[1] * iH, ty_ = -sx * sz * v[2] * iH, tz_ = -sx * sy * v[3] * iH;
                    s_T[it] = sx * sy * sz * v[0];
                    s_T[Caps::kPt + it] = tx_;
                    s_T[2 * Caps::kPt + it] = ty_;
                    s_T[3 * Caps::kPt + it] = tz_;
                    s_T[4 * Caps::kPt + it] = g.support_in_h * fma(x, tx_, fma(y, ty_, z * tz_));
                };
                for (int base = warp * 32;; base += kAdjThreads) {
                    const bool last = base >= tot;
                    if (!last) {
                        const int j = warp_owner(base, off_l, lane), it = base + lane;
                        const int off = __shfl_sync(0xffffffffu, off_l, j & 31);
                        bool near = false;
                        uint32_t rec = 0;
                        if (it < tot) {
                            const int lp = it - off;
                            const int n0 = cp->dim[j][0] + 1, n1 = cp->dim[j][1] + 1, n2 = cp->dim[j][2] + 1;
                            const int i = div_by(lp, cp->mag[j][2]), rem = lp - i * (n1 * n2);
                            const int jj = div_by(rem, cp->mag[j][1]), k = rem - jj * n2;
                            const double* const rx = s_P + kPS * (cp->loff[j] + i);
                            const double* const ry = s_P + kPS * (cp->loff[j] + n0 + jj);
                            const double* const rz = s_P + kPS * (cp->loff[j] + n0 + n1 + k);
                            const double x = rx[0], y = ry[0], z = rz[0];
                            if (x == 0.0 || y == 0.0 || z == 0.0) {
#pragma unroll
                                for (int c = 0; c < kAdjComps; ++c) s_T[c * Caps::kPt + it] = 0.0;
                            } else if (fma(x, x, fma(y, y, z * z)) < 1.0) {
                                near = true;
                                rec = (uint32_t)j | (uint32_t)i << 5 | (uint32_t)jj << 9 | (uint32_t)k << 13;
                            } else {
                                const double* const E = s_E + kES * cp->eoff[j] + 6 * n;
                                const double* const ez = E + kES * (i * n1 + jj);
                                const double* const ey = E + kES * (n0 * n1 + i * n2 + k);
                                const double* const ex = E + kES * (n0 * (n1 + n2) + jj * n2 + k);
                                const double v[4] = {(ez[0] + ey[0]) + ex[0] +
                                                         ((rx[bg_w(n, n)] + ry[bg_w(n, n)]) +
                                                          (rz[bg_w(n, n)] + box_centre<NP>(T, n))),
                                                     (ez[1] + ey[1]) + rx[bg_dw(n, n)], (ez[2] + ex[1]) + ry[bg_dw(n, n)],
                                                     (ey[2] + ex[2]) + rz[bg_dw(n, n)]};
                                put(it, j, rx, ry, rz, v);
                            }
                        }
                        const unsigned m = __ballot_sync(0xffffffffu, near);
                        if (near) s_q[cnt + __popc(m & below)] = rec;
                        cnt += __popc(m);
                        __syncwarp();
                    }
                    if (cnt >= 32 || (last && cnt > 0)) {
                        const int first = max(cnt - 32, 0);
                        if (first + lane < cnt) {
                            const uint32_t rec = s_q[first + lane];
                            const int j = (int)(rec & 31u), i = (int)((rec >> 5) & 15u), jj = (int)((rec >> 9) & 15u),
                                      kk = (int)(rec >> 13);
                            const int n0 = cp->dim[j][0] + 1, n1 = cp->dim[j][1] + 1, n2 = cp->dim[j][2] + 1;
                            const double* const rx = s_P + kPS * (cp->loff[j] + i);
                            const double* const ry = s_P + kPS * (cp->loff[j] + n0 + jj);
                            const double* const rz = s_P + kPS * (cp->loff[j] + n0 + n1 + kk);
                            const double r2 = fma(rx[0], rx[0], fma(ry[0], ry[0], rz[0] * rz[0]));
                            int k = 0;
#pragma unroll
                            for (int s = 0; s + 1 < n; ++s) k += r2 >= T.scale[s].b * T.scale[s].b;
                            const double* const E = s_E + kES * cp->eoff[j];
                            const double* const ez = E + kES * (i * n1 + jj);
                            const double* const ey = E + kES * (n0 * n1 + i * n2 + kk);
                            const double* const ex = E + kES * (n0 * (n1 + n2) + jj * n2 + kk);
                            double Cl[14], Dl[59], c0, v[4];
                            const double *C = Cl, *D = Dl;
                            if (NP == 2) {  // two pieces, few coefficients each: selected constants
#pragma unroll
                                for (int c = 0; c < 14; ++c) Cl[c] = k ? T.reg[1].C[c] : T.reg[0].C[c];
#pragma unroll
                                for (int c = 0; c < 59; ++c) Dl[c] = k ? T.reg[1].D[c] : T.reg[0].D[c];
                                c0 = k ? T.reg[1].c : T.reg[0].c;
                            } else {
                                C = s_C + kCS * k;
                                D = C + kBoxC;
                                c0 = D[kBoxD];
                            }
                            box_inside_grad<DEG>(C, D, c0, T.deg, n, k, rx, ry, rz, ex, ey, ez, v);
                            if (k > 0) {
                                v[0] += (rx[bg_w(n, k)] + ry[bg_w(n, k)]) + (rz[bg_w(n, k)] + box_centre<NP>(T, k));
                                v[1] += rx[bg_dw(n, k)];
                                v[2] += ry[bg_dw(n, k)];
                                v[3] += rz[bg_dw(n, k)];
                            }
                            put(cp->poff[j] + (i * n1 + jj) * n2 + kk, j, rx, ry, rz, v);
                        }
                        cnt = first;
                        __syncwarp();
                    }
                    if (last) break;
                }
            }
            __syncthreads();

            // (C) a warp per particle: its cells in box order over the lanes, weighed by the cotangents, and a
            // fixed-order sum over the lanes
            for (int j = warp; j < np; j += kAdjWarps) {
                double acc[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[c] = 0.0;
                const double x0 = cp->x[j], y0 = cp->y[j], z0 = cp->z[j], radius = cp->H[j];
                const double vx = cp->vx[j], vy = cp->vy[j], vz = cp->vz[j];
                const int l0 = cp->lo[j][0], l1 = cp->lo[j][1], l2 = cp->lo[j][2];
                const int d1 = cp->dim[j][1], d2 = cp->dim[j][2], d12 = d1 * d2, nc = cp->dim[j][0] * d12;
                const int n2 = d2 + 1, n12 = (d1 + 1) * n2;
                for (int lc = lane; lc < nc; lc += 32) {
                    const int i = div_by(lc, cp->cmag[j][1]), rem = lc - i * d12;
                    const int jj = div_by(rem, cp->cmag[j][0]), k = rem - jj * d2;
                    const double ex = fmax(fabs(x0 - s_cc[0][l0 + i]) - g.hpx, 0.0);
                    const double ey = fmax(fabs(y0 - s_cc[1][l1 + jj]) - g.hpy, 0.0);
                    const double ez = fmax(fabs(z0 - s_cc[2][l2 + k]) - g.hpz, 0.0);
                    if (!(add_rn(add_rn(mul_rn(ex, ex), mul_rn(ey, ey)), mul_rn(ez, ez)) < mul_rn(radius, radius))) continue;
                    ++n_eval;
                    const double* const Tp = s_T + cp->poff[j] + (i * (d1 + 1) + jj) * n2 + k;
                    // component c of the cell's Msum: 0 the value, 1..4 d/d(x, y, z, h)
                    auto cell_sum = [&](int c) {
                        const double* const q = Tp + c * Caps::kPt;
                        const double m1 = (q[n12 + n2 + 1] - q[n12 + n2]) - (q[n12 + 1] - q[n12]);
                        const double m0 = (q[n2 + 1] - q[n2]) - (q[1] - q[0]);
                        return m1 - m0;
                    };
                    const double msum = cell_sum(0);
                    if (msum < 0.0) {
                        ++n_neg;
                        continue;
                    }
                    if (msum == 0.0) continue;
                    const int64_t i3 = ((int64_t)(bx + l0 + i) * g.ny + (by + l1 + jj)) * g.nz + (bz + l2 + k);
                    const double gx = cot[ncell + i3], gy = cot[2 * ncell + i3], gz = cot[3 * ncell + i3];
                    const double gs = fma(vz, gz, fma(vy, gy, fma(vx, gx, cot[i3])));
                    acc[0] = fma(msum, gs, acc[0]);
#pragma unroll
                    for (int c = 1; c <= 4; ++c) acc[c] = fma(cell_sum(c), gs, acc[c]);
                    acc[5] = fma(msum, gx, acc[5]);
                    acc[6] = fma(msum, gy, acc[6]);
                    acc[7] = fma(msum, gz, acc[7]);
                }
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
                double v = 0.0;
#pragma unroll
                for (int c = 0; c < 8; ++c) v = lane == c ? acc[c] : v;
                if (lane < 8) part[8 * (int64_t)cp->entry[j] + lane] = lane == 0 ? v : cp->m[j] * v;
            }
            pos += np;
            __syncthreads();
        }
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
        // entries per CTA: about eight CTAs for each of the chip's 2 x SMs places, so that uneven entries level out,
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
