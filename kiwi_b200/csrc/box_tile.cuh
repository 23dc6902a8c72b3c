// The tile body of the box-mass gather (FP64 form, all kernels): one CTA takes one 8 x 8 x 8 cell tile, shared
// by the single-grid kernels and the batch's persistent kernel.
//
// Per particle of the tile's list, the box of its support clipped to the tile (n0 x n1 x n2 cells) has
// n0' + n1' + n2' planes (n' = n + 1), n0' n1' + n0' n2' + n1' n2' edge lines and n0' n1' n2' lattice points.
// A plane's record, an edge line's record and a point's box mass are formed once each (box_math.cuh); a cell
// of the box is the alternating sum of its eight corners' masses, which is the reference's sum over the cell's
// 6 faces x 4 edges x 2 vertex pyramids regrouped by corner (src/cartesian_grid.cpp:246-259,
// src/kernel_integral.cpp:471-647).
//
// The list (ascending particle index) is walked in chunks, in phases separated by barriers:
//   (E) edge lines, and warp 0 loads the next chunk (particles, boxes, offsets) into the other buffer;
//   (P) points;
//   (C1) every (particle, cell of its box) pair as one flat list: support test, counters, alternating sum; and the
//        next chunk's planes;
//   (C2) each thread adds, for the cells it owns, the chunk's pairs in particle order, so that every cell's sum
//        runs over its particles in ascending index order with no atomics; and the next chunk's lines are listed.
// An item's cost is its kind: a line or a point beyond the support is a few sums, one within it roots, logarithms and
// arctangents, a line in an inner piece those of every piece from there on.  So that no lane waits for another kind's
// work, lines are listed by kind over the whole CTA and taken 32 of a kind at a time, the costly kinds first, by
// whichever warp is free; points (two kinds, forty batches a chunk) a warp sorts for itself, finishing the cheap ones
// at once and queueing the others until it has 32.  Lines queued by warp and kind instead left half of the few
// batches of a chunk part empty and the warps waiting at the barrier: 9 k particles on 37 x 41 x 149, quintic spline
// (three kinds), 4.65 -> 3.7 ms, and 3.2 with one copy of the evaluation for all kinds; 150 k on 131 x 117 x 102, cubic, 5.0 -> 4.7 ms.  With one piece there is one
// costly kind, and a warp's own queue is the faster (100 k on 128^3, Wendland C4: 8.5 against 9.1 ms).
//
// A tile with a long list is cut into segments of box_segment() entries, each summed on its own (by CTAs of their
// own, which leave raw sums for k_box_combine, or one after another in one CTA), and the segments' sums are
// added in list order: a grid of few tiles, or a field with a few dense ones, then fills the chip.  The length
// depends on the tile's own list and the grid's tile count alone, so that every call that maps a tile -- whole
// grid, part, batch, allocation-free -- adds the same numbers in the same order.
//
// What bounds it: the FP64 pipe and the shared-memory loads of the records, about equally (a point within the
// support issues about 150 FP64 instructions and 20 shared loads).
#pragma once

#include <climits>

#include "box_math.cuh"
#include "engine.hpp"
#include "lattice.cuh"
#include "tabulated.cuh"

namespace kiwi_b200 {

// Entries per segment of a tile with cnt entries in a grid of ntiles tiles: 128 (where the whole grid has fewer
// tiles than the chip has places, one tile in eight pieces or more) to 1024 (thousands of tiles: only outliers are cut),
// and at most box_most segments in a tile: 16384 in the grid, or 8 per tile beyond that.
__host__ __device__ __forceinline__ int64_t box_most(int64_t ntiles) {
    return 16384 / ntiles < 8 ? 8 : (16384 / ntiles > 256 ? 256 : 16384 / ntiles);
}
__host__ __device__ __forceinline__ int64_t box_segment(int64_t cnt, int64_t ntiles) {
    const int64_t s0 = ntiles / 4 < 128 ? 128 : (ntiles / 4 > 1024 ? 1024 : ntiles / 4);
    const int64_t s1 = (cnt + box_most(ntiles) - 1) / box_most(ntiles);
    return s0 > s1 ? s0 : s1;
}
// Segments whose raw sums are held at a time (16 KB each: 268 MB).  A call with more takes its tiles in runs, one after
// another: 8 segments a tile would be eight times the outputs of a grid whose every list is long (34 GB on 512^3).  The
// 2 M particles of the log-normal cube on 256^3 have 7405.
constexpr int64_t kBoxPlaces = 16384;

#ifndef KIWI_BOX_THREADS
#define KIWI_BOX_THREADS 256
#endif
constexpr int kBoxThreads = KIWI_BOX_THREADS;
constexpr int kBoxWarps = kBoxThreads / 32;
constexpr int kBoxCells = (kTileCells + kBoxThreads - 1) / kBoxThreads;  // cells a thread owns
constexpr int kBoxPMax = 32;                                            // particles per chunk
#ifndef KIWI_BOX_PT_CAP
#define KIWI_BOX_PT_CAP 2304
#endif
#ifndef KIWI_BOX_PAIR_CAP
#define KIWI_BOX_PAIR_CAP 1024
#endif
#ifndef KIWI_BOX_PLANE_CAP
#define KIWI_BOX_PLANE_CAP 296
#endif
constexpr int kBoxPtCap = KIWI_BOX_PT_CAP;        // lattice points per chunk (a full 8^3 box has 729)
constexpr int kBoxPairCap = KIWI_BOX_PAIR_CAP;    // edge lines per chunk (a full box has 243)
constexpr int kBoxPlaneCap = KIWI_BOX_PLANE_CAP;  // planes per chunk (a full box has 27)
// The tabulated integral's records (box_tab_*): a plane's offset, fraction and index on the table's r0 axis; an edge
// line's fractions and indices on the mu0 and cos phi axes for either of its two distances.
constexpr int kTabPlane = 3, kTabEdge = 6;
// The three-piece kernels' records are larger: fewer lines and planes in the same shared memory.
constexpr int kBoxGenPtCap = 1792, kBoxGenPairCap = 640, kBoxGenPlaneCap = 256;

// SEQ: the segments of a tile one after another, which needs the cells' totals beside the segment's sums.
// TAB (with NP 1): the tabulated integral's records.
template <int NP, bool SEQ = false, bool TAB = false>
struct BoxCaps {
    static constexpr int kN = NP ? NP : KIWI_BOX_PIECES;
    static constexpr int kPS = TAB ? kTabPlane : box_plane_stride(kN), kES = TAB ? kTabEdge : box_edge_stride(kN);
    static constexpr int kPt = TAB ? 2304 : SEQ ? 1536 : (NP == 1 ? 3072 : (NP == 2 ? kBoxPtCap : kBoxGenPtCap));
    static constexpr int kPair = TAB ? 900 : SEQ ? (NP ? 768 : 512) : (NP == 1 ? 1024 : (NP == 2 ? kBoxPairCap : kBoxGenPairCap));
    static constexpr int kPlane = TAB ? 296 : SEQ ? 208 : (NP == 1 ? 448 : (NP == 2 ? kBoxPlaneCap : kBoxGenPlaneCap));
    static constexpr int kKinds = kN + 1;  // of edge lines
    static_assert(kKinds * kPair <= 2 * kPt || TAB, "the lines' lists fit the octant values' place");
    static_assert(kPlane <= 512 && kPair <= 1024 && kPt <= 4096, "BoxGeo's fields");
    // dynamic shared memory, in doubles: the cells' sums, the octant values, the edge and plane records
    static constexpr int kOffT = 4 * kTileCells;
    static constexpr int kOffE = kOffT + kPt;
    static constexpr int kOffP = kOffE + kES * kPair;
    static constexpr int kOffS = kOffP + kPS * kPlane;
    static constexpr int kEnd = kOffS + (SEQ ? 4 * kTileCells : 0);
    static constexpr size_t kSmem = sizeof(double) * kEnd + (TAB ? 0 : sizeof(uint2) * 64 * kBoxWarps);
    // (C1) keeps the pairs' values in the edge records' place (with one piece the records are smaller)
    static_assert((NP ? kES : box_edge_stride(1)) * kPair >= kPt, "pair values fit");
};

// A particle's box clipped to the tile and its places in the chunk, packed so that a thread reads it in one 16-byte
// load (eight to ten 4-byte loads otherwise).
// x: the first plane (9 bits), edge line (10) and lattice point (13); y: the 16-bit magic divisors of n2' and n1' n2'
// (x / n = x * ceil(2^16 / n) >> 16 for the at most 729 points); z: n1', n2' (4 each), n0' n1' (7), n0' (n1' + n2') (8),
// n0' (4); w: the first cell (12), lo relative to the tile (3 each), the 10-bit magic divisor of n1' (the at most 81
// lines of a block).
struct BoxGeo {
    int4 v;
    __device__ __forceinline__ int plane() const { return v.x & 511; }
    __device__ __forceinline__ int line() const { return (v.x >> 9) & 1023; }
    __device__ __forceinline__ int point() const { return (int)((uint32_t)v.x >> 19); }
    __device__ __forceinline__ int cell() const { return v.w & 4095; }
    __device__ __forceinline__ int n1() const { return v.z & 15; }
    __device__ __forceinline__ int n2() const { return (v.z >> 4) & 15; }
    __device__ __forceinline__ int n01() const { return (v.z >> 8) & 127; }
    __device__ __forceinline__ int n0_12() const { return (v.z >> 15) & 255; }
    __device__ __forceinline__ int n0() const { return v.z >> 23; }
    __device__ __forceinline__ int lo0() const { return (v.w >> 12) & 7; }
    __device__ __forceinline__ int lo1() const { return (v.w >> 15) & 7; }
    __device__ __forceinline__ int lo2() const { return (v.w >> 18) & 7; }
    __device__ __forceinline__ int by_n2(int x) const { return (int)(((uint32_t)x * (v.y & 0xffffu)) >> 16); }
    __device__ __forceinline__ int by_n12(int x) const { return (int)(((uint32_t)x * ((uint32_t)v.y >> 16)) >> 16); }
    __device__ __forceinline__ int by_n1(int x) const { return (int)(((uint32_t)x * ((uint32_t)v.w >> 21)) >> 10); }
    // the planes of line e: blocks (x, y) over n0' x n1', (x, z) over n0' x n2', (y, z) over n1' x n2'
    __device__ __forceinline__ void line_planes(int e, int& la, int& lb) const {
        const int a0 = n0(), a1 = n1(), a2 = n2();
        const bool xy = e < n01(), yz = e >= n0_12();
        e -= xy ? 0 : (yz ? n0_12() : n01());
        const int pi = xy ? by_n1(e) : by_n2(e), qi = e - pi * (xy ? a1 : a2);
        la = plane() + (yz ? a0 : 0) + pi;
        lb = plane() + a0 + (xy ? 0 : a1) + qi;
    }
};
__device__ __forceinline__ uint32_t box_magic(int n, int bits) { return ((1u << bits) + (uint32_t)n - 1) / (uint32_t)n; }
// The entry of a box of n0' x n1' x n2' planes.
__device__ __forceinline__ int4 box_geo(int n0, int n1, int n2, int lo0, int lo1, int lo2, int plane, int line, int point,
                                        int cell) {
    return int4{(int)((uint32_t)plane | (uint32_t)line << 9 | (uint32_t)point << 19),
                (int)(box_magic(n2, 16) | box_magic(n1 * n2, 16) << 16),
                n1 | n2 << 4 | (n0 * n1) << 8 | (n0 * (n1 + n2)) << 15 | n0 << 23,
                (int)((uint32_t)cell | (uint32_t)(lo0 | lo1 << 3 | lo2 << 6) << 12 | box_magic(n1, 10) << 21)};
}
// The 16-bit magic divisors of a box's n2 and n1 n2 cells (x / n = x * ceil(2^15 / n) >> 15 for the at most 512).
__device__ __forceinline__ uint32_t box_cell_magic(int d1, int d2) { return box_magic(d2, 15) | box_magic(d1 * d2, 15) << 16; }
__device__ __forceinline__ void box_cell(uint32_t magic, int lc, int d1, int d2, int& i, int& j, int& k) {
    i = (int)(((uint32_t)lc * (magic >> 16)) >> 15);
    const int rem = lc - i * (d1 * d2);
    j = (int)(((uint32_t)rem * (magic & 0xffffu)) >> 15);
    k = rem - j * d2;
}

// One chunk of a tile's particle list: the particles' data and their boxes.
struct BoxChunk {
    double4 at[kBoxPMax];  // x, y, z and the support radius
    double4 mv[kBoxPMax];  // mass, velocities
    int4 geo[kBoxPMax];
    double iH[kBoxPMax];
    uint32_t cmag[kBoxPMax];
    int np, ltot, etot, ptot, ctot;
    __device__ __forceinline__ BoxGeo box(int j) const { return BoxGeo{geo[j]}; }
};

__device__ __forceinline__ void box_add_stat(unsigned long long* dst, unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(dst, v);
}

// x with the sign bits of a, b, c multiplied in.
__device__ __forceinline__ double box_signed(double x, double a, double b, double c) {
    const int s = (__double2hiint(a) ^ __double2hiint(b) ^ __double2hiint(c)) & (int)0x80000000;
    return __hiloint2double(__double2hiint(x) ^ s, __double2loint(x));
}

// The tabulated integral (tab_gridded_c at (cos phi, R_0) = (a1 / r, a1) and (a2 / r, a2) in a wall, r the corner's
// distance in it): a corner's two lookups in a wall need the wall's bin on the r0 axis and, of every
// pair (p, q) of the point's distances, the bins of p / sqrt(p^2 + q^2) on the mu0 axis (as the wall's distance over
// the edge line's) and on the cos phi axis (as the leg over the corner's distance in the wall).  Those are formed once
// per plane and per edge line here, and a point has its lookups left: 6 x 8 table
// entries.  Indices carry whether they were clamped (counted per lookup) and whether they fall in the axis's last
// bin (the lookup is then 0).
constexpr int kTabClamped = 1 << 30, kTabLast = 1 << 29, kTabIndex = (1 << 29) - 1;
__device__ __forceinline__ void box_tab_plane(const TabDev& t, const TabWidths& W, double u, double ih, double* rec) {
    rec[0] = u;
    if (u == 0.0) return;
    double r0 = fabs(u) * ih, fx;
    if (r0 > 2.0) r0 = 2.0;  // beyond 2h the pyramid mass depends on the angles alone
    unsigned clamped = 0;
    const int i = tab_index_fr(W, 0, r0, t.rl, t.nr01, t.nr0, fx, clamped);
    rec[1] = fx;
    rec[2] = __hiloint2double(0, i | (clamped ? kTabClamped : 0));
}
// One of the line's distances p against the other q: rec[0] the fraction on mu0, rec[1] on cos phi, rec[2] both
// indices (mu0 in the low word, cos phi in the high word).
__device__ __forceinline__ void box_tab_edge(const TabDev& t, const TabWidths& W, double p, double s, double is, double* rec) {
    unsigned cj = 0, ck = 0;
    double fy, fz;
    const int j = tab_index_fr(W, 1, p / s, t.mul, t.nR_01 - 1, t.nR_0 - 1, fy, cj);
    const int k = tab_index_fr(W, 2, p * is, t.cphil, t.nphi1 - 1, t.nphi - 1, fz, ck);
    rec[0] = fy;
    rec[1] = fz;
    rec[2] = __hiloint2double(k | (ck ? kTabClamped : 0) | (k == t.nphi1 + t.nphi2 - 1 ? kTabLast : 0),
                              j | (cj ? kTabClamped : 0) | (j == t.nR_01 + t.nR_02 - 1 ? kTabLast : 0));
}
// 32 bytes (aligned) in one load.  Not kept in L1: a scattered 32-byte read would hold a 128-byte line there, and those
// lines were what bounded the reads in flight (17.8 -> 16.0 ms on 200 k particles, 120 x 125 x 130).
__device__ __forceinline__ double4 box_tab_load(const double* p) {
    double4 r;
    asm("ld.global.nc.L1::no_allocate.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
    return r;
}
// One lookup: the wall's record, the mu0 side of one record and the cos phi side of another.
__device__ __forceinline__ double box_tab_lookup(const TabDev& t, const double* wall, const double* mu, const double* phi,
                                                 unsigned& nclamp) {
    const int i = __double2loint(wall[2]) & kTabIndex, jw = __double2loint(mu[2]), kw = __double2hiint(phi[2]);
    nclamp += ((jw & kTabClamped) != 0) + ((kw & kTabClamped) != 0);
    if ((jw | kw) & kTabLast) return 0.0;
    const int j = jw & kTabIndex, k = kw & kTabIndex;
    const double fx = wall[1], fy = mu[0], fz = phi[1];
    double4 a, b;  // rows j and j + 1: (i, k), (i + 1, k), (i, k + 1), (i + 1, k + 1)
    const size_t at = ((size_t)i * (t.nR_0 + 1) + j) * (t.nphi + 1) + k;
    if (t.v4) {
        a = box_tab_load(t.v4 + 4 * at);
        b = box_tab_load(t.v4 + 4 * (at + t.nphi + 1));
    } else {
        a = double4{tab_at(t, i, j, k), tab_at(t, i + 1, j, k), tab_at(t, i, j, k + 1), tab_at(t, i + 1, j, k + 1)};
        b = double4{tab_at(t, i, j + 1, k), tab_at(t, i + 1, j + 1, k), tab_at(t, i, j + 1, k + 1),
                    tab_at(t, i + 1, j + 1, k + 1)};
    }
    const double x00 = fx * a.y + (1 - fx) * a.x;
    const double x10 = fx * b.y + (1 - fx) * b.x;
    const double x01 = fx * a.w + (1 - fx) * a.z;
    const double x11 = fx * b.w + (1 - fx) * b.z;
    const double y0 = fy * x10 + (1 - fy) * x00;
    const double y1 = fy * x11 + (1 - fy) * x01;
    return fz * y1 + (1 - fz) * y0;
}

// A cell's outputs from its sums (src/cartesian_grid.cpp:294-317).
__device__ __forceinline__ void box_store(const CartGeom& g, const CartOutputs& out, int64_t t, int li, double M, double P1,
                                          double P2, double P3) {
    const int tz = (int)(t % g.ntz), ty = (int)((t / g.ntz) % g.nty), tx = (int)(t / ((int64_t)g.ntz * g.nty));
    const int ix = tx * kTileX + li / (kTileZ * kTileY), iy = ty * kTileY + (li / kTileZ) % kTileY,
              iz = tz * kTileZ + li % kTileZ;
    if (ix >= g.nx || iy >= g.ny || iz >= g.nz) return;
    const int64_t ncell = (int64_t)g.nx * g.ny * g.nz;
    const int64_t i3 = ((int64_t)ix * g.ny + iy) * g.nz + iz;
    if (out.density) out.density[i3] = M / g.cell_volume;
    const bool has = M > 0.0;
    if (out.vx) out.vx[i3] = has ? P1 / M : out.meanv[0];
    if (out.vy) out.vy[i3] = has ? P2 / M : out.meanv[1];
    if (out.vz) out.vz[i3] = has ? P3 / M : out.meanv[2];
    if (out.raw4) {
        out.raw4[i3] = M;
        out.raw4[ncell + i3] = P1;
        out.raw4[2 * ncell + i3] = P2;
        out.raw4[3 * ncell + i3] = P3;
    }
}

// A tile's cells from its segments' sums sums[segment][4][cell], added in list order (threads as the caller has).
__device__ __forceinline__ void box_combine(const CartGeom& g, const CartOutputs& out, int64_t t, const double* sums,
                                            int nseg) {
    for (int li = threadIdx.x; li < kTileCells; li += blockDim.x) {
        double a[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) a[c] = sums[c * kTileCells + li];
        for (int s = 1; s < nseg; ++s)
#pragma unroll
            for (int c = 0; c < 4; ++c) a[c] = add_rn(a[c], sums[(4 * (int64_t)s + c) * kTileCells + li]);
        box_store(g, out, t, li, a[0], a[1], a[2], a[3]);
    }
}

// The entries list[beg, end) of tile t: its outputs, or with `sums` their raw sums [4][cell].  SEQ: the list in
// segments of `segment` entries, one after another.
// NP, DEG: the kernel's pieces and largest power, known when compiling (the cubic spline: 2, 3), or 0 for any
// kernel of the tables.  T: the kernel's table in constant memory.
// TAB: the tabulated cubic integral, lookups in tab (NP 1, DEG 0, without CULL: outside the support the lookups do not
// cancel exactly, and the reference keeps what they leave).
template <bool CULL, int NP, int DEG, bool SEQ = false, bool TAB = false>
__device__ __forceinline__ void box_tile(const CartGeom& g, const DevParticles& P, const uint32_t* __restrict__ list,
                                         int64_t beg, int64_t end_all, int64_t segment, int64_t t,
                                         const CartOutputs& out, double* __restrict__ sums, DevStats* __restrict__ st,
                                         const KiwiBoxTable& T, const TabDev tab = TabDev{}) {
    using Caps = BoxCaps<NP, SEQ, TAB>;
    static_assert(!TAB || !CULL, "the tabulated integral takes every cell of a box");
    __shared__ TabWidths s_tw;
    if (TAB && threadIdx.x == 0) s_tw = tab_widths(tab);
    __shared__ BoxChunk s_cp[2];
    constexpr bool kList = !TAB && NP != 1;
    __shared__ int s_lines[Caps::kKinds], s_next;  // listed lines of each kind; (E)'s next batch
    if (threadIdx.x < Caps::kKinds) s_lines[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_next = 0;
    __shared__ double s_pl[3][kTileX + 1], s_cc[3][kTileX];
    __shared__ double s_C[NP == 2 || TAB ? 1 : (kBoxC + 1) * Caps::kN];  // any kernel: c and C of its pieces (lanes differ in piece)
    static_assert(kTileX == kTileY && kTileX == kTileZ, "cubic tiles");
    extern __shared__ double s_dyn[];
    const int n = NP ? NP : T.npiece;
    const int kPS = TAB ? kTabPlane : box_plane_stride(n), kES = TAB ? kTabEdge : box_edge_stride(n);
    double* const s_acc = s_dyn;
    double* const s_T = s_dyn + Caps::kOffT;
    double* const s_E = s_dyn + Caps::kOffE;
    double* const s_P = s_dyn + Caps::kOffP;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1;
    uint2* const s_q = reinterpret_cast<uint2*>(s_dyn + Caps::kEnd) + 64 * warp;
    uint32_t* const s_list = reinterpret_cast<uint32_t*>(s_T);

    const int tz = (int)(t % g.ntz), ty = (int)((t / g.ntz) % g.nty), tx = (int)(t / ((int64_t)g.ntz * g.nty));
    const int bx = tx * kTileX, by = ty * kTileY, bz = tz * kTileZ;
    // the tile's lattice planes and cell centres, formed as the reference forms them
    if (threadIdx.x < 3 * (kTileX + 1)) {
        const int a = threadIdx.x / (kTileX + 1), l = threadIdx.x % (kTileX + 1);
        const double mn = a == 0 ? g.x_min : (a == 1 ? g.y_min : g.z_min), d = a == 0 ? g.dpx : (a == 1 ? g.dpy : g.dpz);
        const int b0 = a == 0 ? bx : (a == 1 ? by : bz);
        s_pl[a][l] = add_rn(mn, mul_rn((double)(b0 + l), d));
        if (l < kTileX) s_cc[a][l] = cell_centre(mn, b0 + l, d);
    }
    if (NP != 2 && !TAB)
        for (int i = threadIdx.x; i < (kBoxC + 1) * n; i += kBoxThreads) {
            const int k = i / (kBoxC + 1), c = i % (kBoxC + 1);
            s_C[i] = c < kBoxC ? T.reg[k].C[c] : T.reg[k].c;
        }
    for (int i = threadIdx.x; i < 4 * kTileCells; i += kBoxThreads) s_acc[i] = 0.0;

    // work counters: 32-bit per thread, flushed to the 64-bit totals every 2^16 chunks and at the end
    unsigned n_bbox = 0, n_sphere = 0, n_eval = 0, n_neg = 0, n_warn = 0, n_eo = 0, n_em = 0, n_ei = 0, n_vp = 0,
             n_clamp = 0, n_chunks = 0;
    auto flush = [&]() {
        box_add_stat(&st->bbox_pairs, n_bbox);
        box_add_stat(&st->sphere_pairs, n_sphere);
        box_add_stat(&st->evaluated_pairs, n_eval);
        box_add_stat(&st->neg_clamped, n_neg);
        box_add_stat(&st->neg_warned, n_warn);
        box_add_stat(&st->edge_outer, n_eo);
        box_add_stat(&st->edge_middle, n_em);
        box_add_stat(&st->edge_inner, n_ei);
        box_add_stat(&st->vertex_pyramids, n_vp);
        if (TAB) box_add_stat(&st->table_clamps, n_clamp);
        n_bbox = n_sphere = n_eval = n_neg = n_warn = n_eo = n_em = n_ei = n_vp = n_clamp = 0;
    };
    // the end of the segment at hand (a chunk never crosses it)
    auto segment_end = [&](int64_t at) { return SEQ ? min(at + segment, end_all) : end_all; };
    int64_t end = segment_end(beg);

    // warp 0: the chunk of the particle list starting at `at` (as many particles as the capacities take)
    auto load_chunk = [&](BoxChunk* dst, int64_t at, int64_t end) {
        const int64_t idx = at + lane;
        int nl = 0, ne = 0, npt = 0, ncl = 0, lo0 = 0, lo1 = 0, lo2 = 0, d0 = 0, d1 = 0, d2 = 0;
        double px = 0, py = 0, pz = 0, ph = 1, pm = 0, pvx = 0, pvy = 0, pvz = 0;
        if (idx < end) {
            const uint32_t p = list[idx];
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
            ncl = d0 * d1 * d2;
        }
        int il = nl, ie = ne, ip = npt, ic = ncl;
        for (int o = 1; o < 32; o <<= 1) {
            const int vl = __shfl_up_sync(0xffffffffu, il, o), ve = __shfl_up_sync(0xffffffffu, ie, o);
            const int vp = __shfl_up_sync(0xffffffffu, ip, o), vc = __shfl_up_sync(0xffffffffu, ic, o);
            if (lane >= o) {
                il += vl;
                ie += ve;
                ip += vp;
                ic += vc;
            }
        }
        const bool take = idx < end && il <= Caps::kPlane && ie <= Caps::kPair && ip <= Caps::kPt;
        const int np = __popc(__ballot_sync(0xffffffffu, take));
        if (take) {
            const double H = mul_rn(g.support_in_h, ph);
            dst->at[lane] = double4{px, py, pz, H};
            dst->mv[lane] = double4{pm, pvx, pvy, pvz};
            dst->iH[lane] = 1.0 / (TAB ? ph : H);
            dst->geo[lane] = box_geo(d0 + 1, d1 + 1, d2 + 1, lo0, lo1, lo2, il - nl, ie - ne, ip - npt, ic - ncl);
            dst->cmag[lane] = box_cell_magic(d1, d2);
        }
        if (lane == np - 1) {
            dst->np = np;
            dst->ltot = il;
            dst->etot = ie;
            dst->ptot = ip;
            dst->ctot = ic;
        }
    };
    // all warps: a chunk's plane records
    auto form_planes = [&](const BoxChunk* cp) {
        const int off_l = lane < cp->np ? cp->box(lane).plane() : INT_MAX, tot = cp->ltot;
        for (int base = warp * 32; base < tot; base += kBoxThreads) {
            const int j = warp_owner(base, off_l, lane), it = base + lane;
            if (it < tot) {
                const BoxGeo b = cp->box(j);
                int l = it - b.plane();
                const int n0 = b.n0(), n1 = b.n1();
                const int a = (l >= n0) + (l >= n0 + n1);
                l -= a == 0 ? 0 : (a == 1 ? n0 : n0 + n1);
                const double4 at = cp->at[j];
                const double c = a == 0 ? at.x : (a == 1 ? at.y : at.z);
                const double u = s_pl[a][(a == 0 ? b.lo0() : (a == 1 ? b.lo1() : b.lo2())) + l] - c;
                if constexpr (TAB) box_tab_plane(tab, s_tw, u, cp->iH[j], s_P + kPS * it);
                else box_plane<NP, DEG>(T, u * cp->iH[j], s_P + kPS * it);
            }
        }
    };

    // the kind of particle j's line: the piece it lies in, or n beyond the support and in a particle's plane (nothing to
    // form); and the entry to form it from
    auto line_kind = [&](const BoxChunk* cp, int j, int it, uint32_t& rec) {
        const BoxGeo b = cp->box(j);
        int la, lb;
        b.line_planes(it - b.line(), la, lb);
        const double p = s_P[kPS * la], q = s_P[kPS * lb];
        const double D = fma(p, p, q * q);
        rec = (uint32_t)it | (uint32_t)la << 10 | (uint32_t)lb << 19;
        if (D >= 1.0 || p == 0.0 || q == 0.0) {
            n_eo += 2;
            return Caps::kN;
        }
        int kind = 0;
#pragma unroll
        for (int k = 0; k + 1 < n; ++k) kind += D >= T.scale[k].b * T.scale[k].b;
        if (kind == 0) n_ei += 2;
        else n_em += 2;
        return kind;
    };
    // all warps: the lines of a chunk by kind, into the octant values' place (free from (C2) to (P)), in any order
    auto list_lines = [&](const BoxChunk* cp) {
        const int off_l = lane < cp->np ? cp->box(lane).line() : INT_MAX, tot = cp->etot;
        for (int base = warp * 32; base < tot; base += kBoxThreads) {
            const int j = warp_owner(base, off_l, lane), it = base + lane;
            int kind = -1;
            uint32_t rec = 0;
            if (it < tot) kind = line_kind(cp, j, it, rec);
#pragma unroll
            for (int c = 0; c < Caps::kKinds; ++c) {
                const unsigned m = __ballot_sync(0xffffffffu, kind == c);
                if (m == 0) continue;
                int at = 0;
                if (lane == 0) at = atomicAdd(&s_lines[c], __popc(m));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (kind == c) s_list[Caps::kPair * c + at + __popc(m & below)] = rec;
            }
        }
    };
    auto next_batch = [&]() {
        int b = 0;
        if (lane == 0) b = atomicAdd(&s_next, 1);
        return __shfl_sync(0xffffffffu, b, 0);
    };

    bool first_segment = true;
    BoxChunk* cp = &s_cp[0];
    if (warp == 0 && beg < end) load_chunk(cp, beg, end);
    __syncthreads();
    if (beg < end) form_planes(cp);
    if constexpr (kList) {
        __syncthreads();
        if (beg < end) list_lines(cp);
    }
    __syncthreads();

    for (int64_t pos = beg; pos < end_all;) {
        BoxChunk* const nx = cp == &s_cp[0] ? &s_cp[1] : &s_cp[0];
        const int np = cp->np;
        const bool more = pos + np < end_all;
        const bool ends = SEQ && pos + np == end;  // the segment's last chunk
        if (ends) end = segment_end(end);
        if (warp == 0 && more) load_chunk(nx, pos + np, end);

        // (E) edge lines
        if constexpr (TAB) {
            const int off_l = lane < np ? cp->box(lane).line() : INT_MAX;
            for (int base = warp * 32; base < cp->etot; base += kBoxThreads) {
                const int j = warp_owner(base, off_l, lane), it = base + lane;
                if (it < cp->etot) {
                    int la, lb;
                    cp->box(j).line_planes(it - cp->box(j).line(), la, lb);
                    const double p = fabs(s_P[kPS * la]), q = fabs(s_P[kPS * lb]);
                    if (p != 0.0 && q != 0.0) {
                        const double s = sqrt(p * p + q * q), is = 1.0 / s;
                        box_tab_edge(tab, s_tw, p, s, is, s_E + kES * it);
                        box_tab_edge(tab, s_tw, q, s, is, s_E + kES * it + 3);
                    }
                }
            }
        } else if constexpr (!kList) {
            const int tot = cp->etot;
            const int off_l = lane < np ? cp->box(lane).line() : INT_MAX;
            uint32_t* const s_ql = reinterpret_cast<uint32_t*>(s_q);
            int cnt = 0;
            for (int base = warp * 32;; base += kBoxThreads) {
                const bool last = base >= tot;
                if (!last) {
                    const int j = warp_owner(base, off_l, lane), it = base + lane;
                    bool near = false;
                    uint32_t rec = 0;
                    if (it < tot) {
                        near = line_kind(cp, j, it, rec) == 0;
                        if (!near) s_E[kES * it + 2 * n] = 0.0;
                    }
                    const unsigned m = __ballot_sync(0xffffffffu, near);
                    if (near) s_ql[cnt + __popc(m & below)] = rec;
                    cnt += __popc(m);
                    __syncwarp();
                }
                // (the queue gains at most 32 entries per step, so one batch per step keeps it below 32)
                if (cnt >= 32 || (last && cnt > 0)) {
                    const int first = max(cnt - 32, 0);
                    if (first + lane < cnt) {
                        const uint32_t rec = s_ql[first + lane];
                        box_edge<NP, DEG>(T, 0, s_P + kPS * ((rec >> 10) & 511u), s_P + kPS * (rec >> 19), s_E + kES * (rec & 1023u));
                    }
                    cnt = first;
                    __syncwarp();
                }
                if (last) break;
            }
        } else {
            int nb = 0, first[Caps::kKinds];  // batches of each kind, the costly ones first
#pragma unroll
            for (int c = 0; c < Caps::kKinds; ++c) {
                first[c] = nb;
                nb += (s_lines[c] + 31) >> 5;
            }
            for (int b = next_batch(); b < nb; b = next_batch()) {
                int c = 0, f = 0;
#pragma unroll
                for (int k = 1; k < Caps::kKinds; ++k)
                    if (b >= first[k]) c = k, f = first[k];
                const int e = 32 * (b - f) + lane;
                if (e >= s_lines[c]) continue;
                const uint32_t rec = s_list[Caps::kPair * c + e];
                double* const E = s_E + kES * (rec & 1023u);
                if (c == Caps::kN) E[2 * n] = 0.0;
                else box_edge<NP, DEG>(T, c, s_P + kPS * ((rec >> 10) & 511u), s_P + kPS * (rec >> 19), E);
            }
        }
        __syncthreads();

        // (P) lattice points
        if constexpr (TAB) {
            const int off_l = lane < np ? cp->box(lane).point() : INT_MAX;
            for (int base = warp * 32; base < cp->ptot; base += kBoxThreads) {
                const int j = warp_owner(base, off_l, lane), it = base + lane;
                if (it < cp->ptot) {
                    const BoxGeo b = cp->box(j);
                    const int lp = it - b.point(), n1 = b.n1(), n2 = b.n2();
                    const int i = b.by_n12(lp), rem = lp - i * (n1 * n2);
                    const int jj = b.by_n2(rem), k = rem - jj * n2;
                    const double* const rx = s_P + kPS * (b.plane() + i);
                    const double* const ry = s_P + kPS * (b.plane() + b.n0() + jj);
                    const double* const rz = s_P + kPS * (b.plane() + b.n0() + n1 + k);
                    if (rx[0] == 0.0 || ry[0] == 0.0 || rz[0] == 0.0) {
                        s_T[it] = 0.0;
                    } else {
                        // a line's first three entries are of its first axis's distance, the others of its second's
                        const double* const E = s_E + kES * b.line();
                        const double* const xy = E + kES * (i * n1 + jj);
                        const double* const xz = E + kES * (b.n01() + i * n2 + k);
                        const double* const yz = E + kES * (b.n0_12() + rem);
                        double f = box_tab_lookup(tab, rx, xy, yz, n_clamp) + box_tab_lookup(tab, rx, xz, yz + 3, n_clamp);
                        f = f + (box_tab_lookup(tab, ry, xy + 3, xz, n_clamp) + box_tab_lookup(tab, ry, yz, xz + 3, n_clamp));
                        f = f + (box_tab_lookup(tab, rz, xz + 3, xy, n_clamp) + box_tab_lookup(tab, rz, yz + 3, xy + 3, n_clamp));
                        n_clamp += ((__double2loint(rx[2]) & kTabClamped) != 0) + ((__double2loint(ry[2]) & kTabClamped) != 0) +
                                   ((__double2loint(rz[2]) & kTabClamped) != 0);
                        s_T[it] = box_signed(f, rx[0], ry[0], rz[0]);
                        n_vp += 6;
                    }
                }
            }
        } else {
            const int tot = cp->ptot;
            const int off_l = lane < np ? cp->box(lane).point() : INT_MAX;
            int cnt = 0;
            const double far_c = box_centre<NP>(T, n);
            for (int base = warp * 32;; base += kBoxThreads) {
                const bool last = base >= tot;
                if (!last) {
                    const int j = warp_owner(base, off_l, lane), it = base + lane;
                    bool near = false;
                    uint2 rec{0, 0};
                    if (it < tot) {
                        const BoxGeo b = cp->box(j);
                        const int lp = it - b.point(), n0 = b.n0(), n1 = b.n1(), n2 = b.n2();
                        const int i = b.by_n12(lp), rem = lp - i * (n1 * n2);
                        const int jj = b.by_n2(rem), k = rem - jj * n2;
                        const int lx = b.plane() + i, dly = n0 - i + jj, dlz = n1 - jj + k;  // its planes, and its lines:
                        const int exy = b.line() + i * n1 + jj, dxz = b.n01() + i * n2 + k - (i * n1 + jj), dyz = n2 * dly;
                        const double* const rx = s_P + kPS * lx;
                        const double* const ry = rx + kPS * dly;
                        const double* const rz = ry + kPS * dlz;
                        const double x = rx[0], y = ry[0], z = rz[0];
                        if (x == 0.0 || y == 0.0 || z == 0.0) {
                            s_T[it] = 0.0;
                        } else if (fma(x, x, fma(y, y, z * z)) < 1.0) {
                            near = true;
                            rec = uint2{(uint32_t)(it | exy << 12 | lx << 22), (uint32_t)(dly | dlz << 5 | dxz << 10 | dyz << 18)};
                        } else {
                            const double* const E = s_E + kES * exy + 2 * n;
                            const double f = (E[0] + E[kES * dxz]) + E[kES * (dxz + dyz)] +
                                             ((rx[1 + 2 * n] + ry[1 + 2 * n]) + (rz[1 + 2 * n] + far_c));
                            s_T[it] = box_signed(f, x, y, z);
                            n_vp += 6;
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
                        const uint2 rec = s_q[first + lane];
                        const int it = (int)(rec.x & 4095u);
                        const double* const rx = s_P + kPS * (int)(rec.x >> 22);
                        const double* const ry = rx + kPS * (int)(rec.y & 31u);
                        const double* const rz = ry + kPS * (int)((rec.y >> 5) & 31u);
                        const double x = rx[0], y = ry[0], z = rz[0];
                        const double ax = fabs(x), ay = fabs(y), az = fabs(z);
                        const double r2 = fma(x, x, fma(y, y, z * z));
                        int k = 0;  // the point's piece
#pragma unroll
                        for (int s = 0; s + 1 < n; ++s) k += r2 >= T.scale[s].b * T.scale[s].b;
                        const double* const exy = s_E + kES * (int)((rec.x >> 12) & 1023u) + k;
                        const double* const exz = exy + kES * (int)((rec.y >> 10) & 255u);
                        const double* const eyz = exz + kES * (int)(rec.y >> 18);
                        // the smallest offset first: the other two's angles are then at most pi/4
                        const bool mx = ax <= ay && ax <= az, my = !mx && ay <= az;
                        const double* const r0 = mx ? rx : (my ? ry : rz);
                        const double* const r1 = mx ? ry : rx;
                        const double* const r2_ = mx || my ? rz : ry;
                        double Cl[14], c0;
                        const double* C = Cl;
                        if (NP == 2) {  // two pieces, six coefficients each: selected constants
#pragma unroll
                            for (int c = 0; c < 14; ++c) Cl[c] = k ? T.reg[1].C[c] : T.reg[0].C[c];
                            c0 = k ? T.reg[1].c : T.reg[0].c;
                        } else {
                            C = s_C + (kBoxC + 1) * k;
                            c0 = C[kBoxC];
                        }
                        double f = box_inside<DEG>(C, c0, T.deg, ax, ay, az, r2, eyz[0], eyz[n], exz[0], exz[n], exy[0],
                                                   exy[n], fabs(r0[0]), r0[2 + k], fabs(r1[0]), r1[1], r1[2 + k],
                                                   fabs(r2_[0]), r2_[1], r2_[2 + k]);
                        if (k > 0) f += ((rx[1 + n + k] + ry[1 + n + k]) + (rz[1 + n + k] + box_centre<NP>(T, k)));
                        s_T[it] = box_signed(f, x, y, z);
                        n_vp += 6;
                    }
                    cnt = first;
                    __syncwarp();
                }
                if (last) break;
            }
        }
        __syncthreads();

        // (C1) the chunk's (particle, cell) pairs, into the edge records' place (dead after (P))
        double* const s_cm = s_E;
        if (threadIdx.x < Caps::kKinds) s_lines[threadIdx.x] = 0;  // for the next chunk
        if (threadIdx.x == 0) s_next = 0;
        if (more) form_planes(nx);
        {
            const int tot = cp->ctot;
            const int off_l = lane < np ? cp->box(lane).cell() : INT_MAX;
            for (int base = warp * 32; base < tot; base += kBoxThreads) {
                const int j = warp_owner(base, off_l, lane), it = base + lane;
                if (it < tot) {
                    const BoxGeo b = cp->box(j);
                    const int d1 = b.n1() - 1, d2 = b.n2() - 1;
                    int i, jj, k;
                    box_cell(cp->cmag[j], it - b.cell(), d1, d2, i, jj, k);
                    ++n_bbox;
                    const double4 at = cp->at[j];
                    const double radius = at.w;
                    const double ex = fmax(fabs(at.x - s_cc[0][b.lo0() + i]) - g.hpx, 0.0);
                    const double ey = fmax(fabs(at.y - s_cc[1][b.lo1() + jj]) - g.hpy, 0.0);
                    const double ez = fmax(fabs(at.z - s_cc[2][b.lo2() + k]) - g.hpz, 0.0);
                    // the support test of the pair counters, rounded as the host restatement rounds it
                    const bool in = add_rn(add_rn(mul_rn(ex, ex), mul_rn(ey, ey)), mul_rn(ez, ez)) < mul_rn(radius, radius);
                    n_sphere += in;
                    double msum = 0.0;
                    if (!CULL || in) {
                        ++n_eval;
                        const int n2 = d2 + 1, n12 = (d1 + 1) * n2;
                        const double* const Tp = s_T + b.point() + i * n12 + jj * n2 + k;
                        const double m1 = (Tp[n12 + n2 + 1] - Tp[n12 + n2]) - (Tp[n12 + 1] - Tp[n12]);
                        const double m0 = (Tp[n2 + 1] - Tp[n2]) - (Tp[1] - Tp[0]);
                        msum = m1 - m0;
                        if (msum < 0.0) {
                            ++n_neg;
                            if (msum <= -0.01) ++n_warn;
                            msum = 0.0;
                        }
                    }
                    s_cm[it] = msum;
                }
            }
        }
        __syncthreads();

        // (C2) the owned cells' sums: a warp's 32 cells are four z rows of one x slab; it visits the particles whose
        // boxes reach them
        const BoxGeo mine = cp->box(lane < np ? lane : 0);
#pragma unroll
        for (int c = 0; c < kBoxCells; ++c) {
            const int li = threadIdx.x + c * kBoxThreads;
            if (kTileCells % kBoxThreads && (li & ~31) >= kTileCells) break;
            const int lx = li / (kTileZ * kTileY), ly = (li / kTileZ) % kTileY, lz = li % kTileZ;
            const int ly0 = ly & ~3;
            bool hit = false;
            if (lane < np) {
                const int i = lx - mine.lo0(), j0 = mine.lo1();
                hit = i >= 0 && i < mine.n0() - 1 && j0 < ly0 + 4 && j0 + mine.n1() - 1 > ly0;
            }
            unsigned todo = __ballot_sync(0xffffffffu, hit);
            if (todo == 0 && !ends) continue;
            double a0 = s_acc[li], a1 = s_acc[kTileCells + li];
            double a2 = s_acc[2 * kTileCells + li], a3 = s_acc[3 * kTileCells + li];
            for (; todo; todo &= todo - 1) {
                const int j = __ffs((int)todo) - 1;
                const BoxGeo b = cp->box(j);
                const int i = lx - b.lo0(), jj = ly - b.lo1(), k = lz - b.lo2();
                const int d1 = b.n1() - 1, d2 = b.n2() - 1;
                if ((unsigned)jj >= (unsigned)d1 || (unsigned)k >= (unsigned)d2) continue;
                const double4 mv = cp->mv[j];
                const double msum = s_cm[b.cell() + (i * d1 + jj) * d2 + k], mm = msum * mv.x;
                if (msum == 0.0) continue;  // (not by mm: a mass or velocity that is not finite shows in its cells)
                a0 = add_rn(a0, mm);
                a1 = fma(mm, mv.y, a1);
                a2 = fma(mm, mv.z, a2);
                a3 = fma(mm, mv.w, a3);
            }
            if (SEQ && ends) {  // the first segment's sums as they are, the others' added
                const double v[4] = {a0, a1, a2, a3};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    double& tot = s_dyn[Caps::kOffS + q * kTileCells + li];
                    tot = first_segment ? v[q] : add_rn(tot, v[q]);
                }
                a0 = a1 = a2 = a3 = 0.0;
            }
            s_acc[li] = a0;
            s_acc[kTileCells + li] = a1;
            s_acc[2 * kTileCells + li] = a2;
            s_acc[3 * kTileCells + li] = a3;
        }
        if (ends) first_segment = false;
        if constexpr (kList)
            if (more) list_lines(nx);
        __syncthreads();
        pos += np;
        cp = nx;
        if (++n_chunks == (1u << 16)) {
            flush();
            n_chunks = 0;
        }
    }

    const double* const fin = SEQ && !first_segment ? s_dyn + Caps::kOffS : s_acc;
#pragma unroll
    for (int c = 0; c < kBoxCells; ++c) {
        const int li = threadIdx.x + c * kBoxThreads;
        if (kTileCells % kBoxThreads && li >= kTileCells) break;
        const double M = fin[li], P1 = fin[kTileCells + li], P2 = fin[2 * kTileCells + li], P3 = fin[3 * kTileCells + li];
        if (sums) {
            sums[li] = M;
            sums[kTileCells + li] = P1;
            sums[2 * kTileCells + li] = P2;
            sums[3 * kTileCells + li] = P3;
        } else {
            box_store(g, out, t, li, M, P1, P2, P3);
        }
    }
    flush();
}

// Runs one item; range: the tile's list.
template <bool CULL, int NP, int DEG, bool TAB = false>
__device__ __forceinline__ void box_item(const BoxItem& it, const CartGeom& g, const DevParticles& P,
                                         const uint32_t* __restrict__ list, const int64_t* __restrict__ range,
                                         int64_t t, const CartOutputs& out, double* __restrict__ sums,
                                         DevStats* __restrict__ st, const KiwiBoxTable& T, const TabDev tab = TabDev{}) {
    const int64_t lo = range[0], hi = range[1];
    const int64_t len = box_segment(hi - lo, (int64_t)g.ntx * g.nty * g.ntz);
    const int64_t beg = lo + it.seg * len, end = it.nseg > 1 ? min(beg + len, hi) : hi;
    box_tile<CULL, NP, DEG, false, TAB>(g, P, list, beg, end, 0, t, out,
                            it.nseg > 1 ? sums + (int64_t)(it.slot + it.seg) * 4 * kTileCells : nullptr, st, T, tab);
}

}  // namespace kiwi_b200
