#!/usr/bin/env python3
"""Exact-rational derivation of the box-mass tables: the kernel mass T(x, y, z) of the box between a particle
and a point at offsets x, y, z > 0 (lengths in units of the support radius H), for the six SPH kernels.

Writes ``kiwi_b200/csrc/box_tables.h``.  Between breakpoints a kernel is a polynomial, W = sum_n w_n r^n, so
T needs the box moments V_n = int_box r^n dV.  With M_k = int rho^k dphi along an edge line (r0 the distance
to a wall, R0 the edge line's distance within it, t the leg along the edge, r the distance to the point) and
K_k = M_k - r0^k phi, the divergence theorem gives (n + 3)(n + 2) V_n = sum over the six right triangles of
r0 K_{n+2}, and the recurrences (no division by a length)

  K_k = r0^2 K_{k-2} + R0 L_{k-2},   L_m = int rho^m ds = (t r^m + m p^2 L_{m-2}) / (m + 1),  p^2 = r0^2 + R0^2,
  L_{-1} = atanh(t / r),  L_0 = t,  K_0 = 0,  r0 K_{-1} = ang - phi,  ang = atan(r0 t / (R0 r)).

The two triangles of a wall have phi_1 + phi_2 = pi/2 and ang_1 + ang_2 = pi/2 - A, A = atan(a b / (r0 r)), and
the three A sum to pi/2.  Hence, with e1, e2, e3 the elementary symmetric functions of x^2, y^2, z^2,

  sum_n w_n V_n = xyz E(r, e2, e3) + sum_pairs xy Q(x^2, y^2) atanh(z / r) - sum_walls a(x) A_x
                = xyz C(r, e2, e3) / r + sum_pairs xy Q(x^2, y^2) (atanh(z / r) - z / r) - sum_walls a(x) A_x,
  a(x) = sum_{n odd} w_n x^(n+3) / ((n+3)(n+2)),   C = r E + sum_pairs Q.

The first form's terms are of order one and cancel to T <= 1/8; taking each logarithm's leading term into the
polynomial leaves terms of T's own order (a third of the rounding error).  C, a polynomial in r, e2 and e3, is
stored in powers of r - c, c the piece's outer end b for the splines and CENTRE b for the Wendland kernels (one
piece of a high degree), so that its own terms cancel little where the cells' masses are smallest, nor about the
particle, where T is: with 3/4, cells of 0.02 H about the particle of the Wendland C6 kernel erred by 1.5e-12 of their
mass, with 3/8 by 1e-14, and the cells at the support's end as before.

A kernel with several pieces is the sum over its breakpoints b of difference kernels W_s - W_{s+1} supported on
r < b.  Where the point lies beyond b, the difference kernel's mass follows from the directions in which the
sphere ends before the box does: with m its mass / (4 pi), the octant's mass less the caps beyond the walls plus
the caps beyond two walls, (pi/2) m - (pi/2) sum_walls h(x) + sum_pairs g(x, y),

  f(p) = p c1 - sum_{n even} w_n p^(n+3) / ((n+3)(n+2)),  c1 = N(b) + m / b,  N(q) = sum_n w_n q^(n+2) / ((n+3)(n+2)),
  h(p) = m + a(p) - f(p) for p < b (it vanishes at b with several derivatives), 0 beyond,
  g(p, q) = pq t G(p^2, q^2) + pq Q(p^2, q^2) atanh(t / b) - (phi_p - ang_p) f(p) + ang_p h(p) + the same of q,
            t = sqrt(b^2 - p^2 - q^2), phi_p = atan(t / q), ang_p = atan(p t / (q b)); 0 for t^2 <= 0.

f and h are stored in powers of b - p for p near b, where h is small, and in powers of p (f, a) for the rest.

The derivative with respect to x is the kernel's integral over the box's face at x, from the same recurrences:

  dT/dx = yz D(r, x^2, y^2 z^2) / r + y R(x^2, y^2) (atanh(z / r) - z / r) + z R(x^2, z^2) (atanh(y / r) - y / r)
          - a'(x) A_x  inside,    -(pi/2) h'(x) + g_p(x, y) + g_p(x, z)  beyond b,
  -g_p(p, q) = (phi - ang) f'(p) - ang h'(p) - q t A(p^2, q^2) - q R(p^2, q^2) atanh(t / b),

D in powers of r - c like C, R and A (the triangle ending on the sphere) in powers of p^2 and p^2 + q^2.

A face of a general cell is a sum over its edges' right triangles, whose cones' masses share all this: with
delta = phi - ang at the triangle's far vertex, in piece k,

  cone(r0, R0, t) = r0 R0 [t V(r, r0^2, p^2) / r + B(r0^2, p^2) (atanh(t / r) - t / r)] - delta a(r0)
                    + sum_{s<k} [m_s delta - h_s(r0) phi + e_s(r0, R0)],
  e(r0, R0) = r0 R0 [t_b A(r0^2, p^2) + B atanh(t_b / b)] - delta_b f(r0) + ang_b h(r0),

the subscript b marking the point where the edge line leaves the sphere of radius b (kiwi_cone_tables).

The polynomials of the arctangent and the logarithm (kiwi_b200/csrc/fastmath.cuh) interpolate
atan(x) / x in x^2 on [0, 1] and (log(1 + f) - f) / f^2 in f about 0 at Chebyshev points, in exact rational
arithmetic; the logarithm's argument is reduced by a table of reciprocals with their logarithms.

Usage:  python gen_box_tables.py            (write the header)
        python gen_box_tables.py --check    (exit 1 if the committed header is stale)
"""
from __future__ import annotations

import math
import os
import struct
import sys
from decimal import Decimal, getcontext
from fractions import Fraction as Q

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from gen_kernel_tables import KERNELS, _num  # noqa: E402

HERE = os.path.dirname(os.path.abspath(__file__))
OUT = os.path.normpath(os.path.join(HERE, "..", "csrc", "box_tables.h"))

getcontext().prec = 60
PI = Decimal("3.14159265358979323846264338327950288419716939937510582097494")


# ---- sparse polynomials {exponent tuple: Fraction} in (X, Y, Z) = (r0^2, R0^2, t^2)

def padd(a, b, s=Q(1)):
    r = dict(a)
    for m, v in b.items():
        r[m] = r.get(m, Q(0)) + s * v
    return {m: v for m, v in r.items() if v}


def pmul(a, b):
    r = {}
    for m, v in a.items():
        for n, w in b.items():
            k = tuple(i + j for i, j in zip(m, n))
            r[k] = r.get(k, Q(0)) + v * w
    return {m: v for m, v in r.items() if v}


def pscale(a, s):
    return {m: v * s for m, v in a.items()}


def ppow(a, n):
    r = {(0, 0, 0): Q(1)}
    for _ in range(n):
        r = pmul(r, a)
    return r


XP, YP, ZP = {(1, 0, 0): Q(1)}, {(0, 1, 0): Q(1)}, {(0, 0, 1): Q(1)}
PP = padd(XP, YP)
RR = padd(PP, ZP)
ONE3 = {(0, 0, 0): Q(1)}


def lam(m):
    """L_m = t [r if m odd] lam(m) + nu(m) p^(m+1) L_{-1}."""
    if m <= 0:
        return {} if m < 0 else ONE3
    head = ppow(RR, m // 2)
    return pscale(padd(head, pscale(pmul(PP, lam(m - 2)), Q(m))), Q(1, m + 1))


def nu(m):
    return Q(1) if m == -1 else Q(m, m + 1) * nu(m - 2)


def tri(k):
    """r0 K_k: (poly of r0 R0 t [times r for odd k], poly of r0 R0 L_{-1}); the coefficient of (ang - phi) is
    X^((k+1)/2) for odd k."""
    if k == 0 or k == -1:
        return {}, {}
    A, B = tri(k - 2)
    A = padd(pmul(XP, A), lam(k - 2))
    B = pmul(XP, B)
    if k % 2:
        B = padd(B, pscale(ppow(PP, (k - 1) // 2), nu(k - 2)))
    return A, B


def permuted(a, perm):
    return {tuple(m[perm[i]] for i in range(3)): v for m, v in a.items()}


def symmetric_to_e(a):
    """A symmetric polynomial of (X, Y, Z) as {(i1, i2, i3): coef} of e1^i1 e2^i2 e3^i3."""
    e1 = RR
    e2 = padd(padd(pmul(XP, YP), pmul(YP, ZP)), pmul(XP, ZP))
    e3 = pmul(pmul(XP, YP), ZP)
    out, rest = {}, dict(a)
    while rest:
        m = max(rest)  # the leading monomial, exponents descending
        v = rest[m]
        i = (m[0] - m[1], m[1] - m[2], m[2])
        assert min(i) >= 0
        out[i] = v
        rest = padd(rest, pmul(pmul(ppow(e1, i[0]), ppow(e2, i[1])), ppow(e3, i[2])), -v)
    return out


def symmetric2_to_ps(a):
    """A polynomial symmetric in (X, Y) (no Z) as {(i, j): coef} of P^i S^j, P = X + Y, S = XY."""
    out, rest = {}, {m: v for m, v in a.items()}
    while rest:
        m = max(rest)
        v = rest[m]
        i = (m[0] - m[1], m[1])
        assert min(i) >= 0 and m[2] == 0
        out[i] = v
        rest = padd(rest, pmul(ppow(PP, i[0]), ppow(pmul(XP, YP), i[1])), -v)
    return out


PERMS = [(0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)]


def moment(n):
    """V_n (without its a(x) A_x terms): (e-poly of xyz [times r for odd n], PS-poly of xy atanh(z / r))."""
    A, B = tri(n + 2)
    sym = {}
    for p in PERMS:
        sym = padd(sym, permuted(A, p))
    s = Q(1, (n + 3) * (n + 2))
    b2 = padd(B, permuted(B, (1, 0, 2)))
    return pscale(symmetric_to_e(sym), s), pscale(symmetric2_to_ps(b2), s)


def edge_poly(n, b):
    """pq t G(P, S): the pair of triangles ending on the sphere of radius b (t^2 = b^2 - P, r = b)."""
    A, _ = tri(n + 2)
    sym = padd(A, permuted(A, (1, 0, 2)))
    by_z = {}
    for m, v in sym.items():
        by_z.setdefault(m[2], {})[(m[0], m[1], 0)] = v
    zpoly = padd({(0, 0, 0): b * b}, PP, Q(-1))
    tot = {}
    for k, a in by_z.items():
        tot = padd(tot, pmul(a, ppow(zpoly, k)))
    s = Q(1, (n + 3) * (n + 2)) * (b if n % 2 else 1)
    return pscale(symmetric2_to_ps(tot), s)


# array layouts: exponents of each coefficient
CENTRE, CONE_CENTRE = Q(3, 8), Q(3, 4)
# C: powers of r - c for each e2^j e3^l: 13 | e2: 9 | e2^2: 5 | e3: 7 | e2 e3: 3 | e2^3: 1 | e3^2: 1
C_BLOCKS = [((0, 0), 13), ((1, 0), 9), ((2, 0), 5), ((0, 1), 7), ((1, 1), 3), ((3, 0), 1), ((0, 2), 1)]
LAY_Q = [(i, 0) for i in range(1, 7)] + [(i, 1) for i in range(5)] + [(i, 2) for i in range(3)] + [(0, 3)]
LAY_G = [(i, 0) for i in range(6)] + [(i, 1) for i in range(4)] + [(i, 2) for i in range(2)]


# D: powers of r - c for each X^i S^j (X = x^2, S = y^2 z^2), largest total weight 12
D_BLOCKS = [((i, j), 13 - 2 * i - 4 * j) for j in range(4) for i in range(7) if 13 - 2 * i - 4 * j > 0]
LAY_R = [(i, j) for i in range(7) for j in range(7 - i)]   # X^i P^j
LAY_A = [(i, j) for i in range(6) for j in range(6 - i)]


def laid(poly, layout):
    assert set(poly) <= set(layout), (sorted(poly), layout)
    return [poly.get(m, Q(0)) for m in layout]


def to_xp(a):
    """A polynomial in (X, Y) as {(i, j): coef} of X^i P^j, P = X + Y (Y = P - X)."""
    out = {}
    for (i, j, k), v in a.items():
        assert k == 0
        for u in range(j + 1):
            key = (i + u, j - u)
            out[key] = out.get(key, Q(0)) + v * math.comb(j, u) * (-1) ** u
    return {m: v for m, v in out.items() if v}


def to_xes(a):
    """A polynomial symmetric in (Y, Z) as {(i, l, j): coef} of X^i e1^l S^j, S = YZ, Y + Z = e1 - X."""
    out, rest = {}, dict(a)
    while rest:
        m = max(rest, key=lambda t: (t[1], t[2], t[0]))
        v, s = rest[m], m[1] - m[2]
        assert s >= 0
        rest = padd(rest, pmul({(m[0], 0, 0): Q(1)}, pmul(ppow(padd(YP, ZP), s), ppow(pmul(YP, ZP), m[2]))), -v)
        for u in range(s + 1):
            key = (m[0] + u, s - u, m[2])
            out[key] = out.get(key, Q(0)) + v * math.comb(s, u) * (-1) ** u
    return {m: v for m, v in out.items() if v}


def face(n):
    """The face moment of r^n: (yz [times r for odd n], y atanh(z / r)) coefficients, as polynomials in X, Y, Z."""
    A, B = tri(n + 2)
    s = Q(1, n + 2)
    return pscale(padd(A, permuted(A, (0, 2, 1))), s), pscale(B, s), pscale(A, s)


def add_into(dst, src, s):
    for m, v in src.items():
        dst[m] = dst.get(m, Q(0)) + s * v
        if not dst[m]:
            del dst[m]


def shifted(c, b):
    """Coefficients of sum c[i] r^i in powers of r - b."""
    out = [Q(0)] * len(c)
    for i, v in enumerate(c):
        for k in range(i + 1):
            out[k] += v * math.comb(i, k) * b ** (i - k)
    return out


def region(w, c0):
    """Tables of one piece sum_n w[n] r^n: C (about r = c0), Q, a (rational, without the normalisation)."""
    C, QQ, a = {}, {}, [Q(0)] * 6
    D, R = {}, {}
    for n, c in w.items():
        A2, B1, _ = face(n)
        for (i, l, j), v in to_xes(A2).items():
            D.setdefault((i, j), [Q(0)] * 13)[2 * l + 1 + n % 2] += c * v
        for (i, l, j), v in to_xes(padd(B1, permuted(B1, (0, 2, 1)))).items():
            D.setdefault((i, j), [Q(0)] * 13)[2 * l] += c * v
        add_into(R, to_xp(B1), c)
        V, B = moment(n)
        pairs = {}  # the three pairs' Q as a symmetric polynomial
        for (i, j), v in B.items():
            one = pscale(pmul(ppow(PP, i), ppow(pmul(XP, YP), j)), v)
            for perm in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
                pairs = padd(pairs, permuted(one, perm))
        for poly, up in ((V, 1 + n % 2), (symmetric_to_e(pairs), 0)):
            for (i1, i2, i3), v in poly.items():  # e1^i1 = r^(2 i1)
                C.setdefault((i2, i3), [Q(0)] * 13)[2 * i1 + up] += c * v
        add_into(QQ, B, c)
        if n % 2:
            a[(n - 1) // 2] += c / ((n + 3) * (n + 2))
    flat = []
    for key, size in C_BLOCKS:
        block = C.pop(key, [Q(0)] * 13)
        assert not any(block[size:])
        flat += shifted(block[:size], c0)
    assert not C
    dflat = []
    for key, size in D_BLOCKS:
        block = D.pop(key, [Q(0)] * 13)
        assert not any(block[size:])
        dflat += shifted(block[:size], c0)
    assert not D
    return {"c": c0, "C": flat, "Q": laid(QQ, LAY_Q), "a": a, "D": dflat, "R": laid(R, LAY_R)}


def scale(d, b):
    """Tables of a difference kernel sum_n d[n] r^n on r < b: m, G, Q, f and a in powers of p, f and h in powers
    of b - p."""
    m = sum(c * b ** (n + 3) / (n + 3) for n, c in d.items())
    N = sum(c * b ** (n + 2) / ((n + 3) * (n + 2)) for n, c in d.items())
    G, f, h, A = {}, [Q(0)] * 15, [Q(0)] * 15, {}
    f[1] = N + m / b
    for n, c in d.items():
        add_into(G, edge_poly(n, b), c)
        one, zpoly = {}, padd({(0, 0, 0): b * b}, PP, Q(-1))
        for m3, v in face(n)[2].items():  # t^2 = b^2 - P, r = b
            one = padd(one, pmul({(m3[0], m3[1], 0): v}, ppow(zpoly, m3[2])))
        add_into(A, to_xp(one), c * (b if n % 2 else 1))
        v = c / ((n + 3) * (n + 2))
        if n % 2:
            h[n + 3] += v
        else:
            f[n + 3] -= v
    assert f[14] == 0 and not any(f[0::2]) and not any(h[1::2]) and not any(h[:4])
    fp, ap = f[1::2], h[4::2]
    h = [x - y for x, y in zip(h, f)]
    h[0] += m
    flip = lambda c: [v * (-1) ** i for i, v in enumerate(shifted(c, b))]  # noqa: E731
    return {"b": b, "m": m, "G": laid(G, LAY_G), "fp": fp, "ap": ap, "f": flip(f)[:14],
            "h": flip(h), "A": laid(A, LAY_A)}


V_BLOCKS = [((i, d - i), 13 - 2 * d) for d in range(7) for i in range(d + 1)]  # powers of r - c for each X^i P^j


def to_xpr(a):
    """A polynomial in (X, Y, Z) as {(i, j, l): coef} of X^i P^j r^(2l), Y = P - X, Z = r^2 - P."""
    out = {}
    for (i, j, k), v in a.items():
        for u in range(j + 1):
            for w in range(k + 1):
                key = (i + u, j - u + k - w, w)
                c = v * math.comb(j, u) * (-1) ** u * math.comb(k, w) * (-1) ** (k - w)
                out[key] = out.get(key, Q(0)) + c
    return {m: v for m, v in out.items() if v}


def cone_region(w, c0):
    V, B, a = {}, {}, [Q(0)] * 6
    for n, c in w.items():
        A1, B1 = tri(n + 2)
        c = c / ((n + 3) * (n + 2))
        for (i, j, l), v in to_xpr(A1).items():
            V.setdefault((i, j), [Q(0)] * 13)[2 * l + 1 + n % 2] += c * v
        b = to_xp(B1)
        for (i, j), v in b.items():
            V.setdefault((i, j), [Q(0)] * 13)[0] += c * v
        add_into(B, b, c)
        if n % 2:
            a[(n - 1) // 2] += c
    flat = []
    for key, size in V_BLOCKS:
        block = V.pop(key, [Q(0)] * 13)
        assert not any(block[size:])
        flat += shifted(block[:size], c0)
    assert not V
    return {"c": c0, "V": flat, "B": laid(B, LAY_R), "a": a}


def cone_scale(d, b):
    A, zpoly = {}, padd({(0, 0, 0): b * b}, PP, Q(-1))
    for n, c in d.items():
        one = {}
        for m3, v in tri(n + 2)[0].items():  # t^2 = b^2 - P, r = b
            one = padd(one, pmul({(m3[0], m3[1], 0): v}, ppow(zpoly, m3[2])))
        add_into(A, to_xp(one), c * (b if n % 2 else 1) / ((n + 3) * (n + 2)))
    s = scale(d, b)
    return {"b": b, "m": s["m"], "fp": s["fp"], "ap": s["ap"], "f": s["f"], "h": s["h"], "A": laid(A, LAY_A)}


def kernel_box(K):
    polys = [dict(p.c) for p in K.piece_polys()]
    a3 = K.a3_times_pi()
    regs = [region(p, b if K.spline else CENTRE * b) for p, b in zip(polys, K.breaks)]
    scs = []
    for s, b in enumerate(K.breaks):
        nxt = polys[s + 1] if s + 1 < len(polys) else {}
        d = dict(polys[s])
        for n, c in nxt.items():
            d[n] = d.get(n, Q(0)) - c
        scs.append(scale({n: c for n, c in d.items() if c}, b))
    top = max(n for p in polys for n in p)
    cregs = [cone_region(p, b if K.spline else CONE_CENTRE * b) for p, b in zip(polys, K.breaks)]
    cscs = []
    for s, b in enumerate(K.breaks):
        nxt = polys[s + 1] if s + 1 < len(polys) else {}
        d = {n: polys[s].get(n, Q(0)) - nxt.get(n, Q(0)) for n in set(polys[s]) | set(nxt)}
        cscs.append(cone_scale({n: c for n, c in d.items() if c}, b))
    return {"creg": cregs, "cscale": cscs, "key": K.key, "npiece": len(polys), "deg": top, "a3pi": a3, "reg": regs, "scale": scs}


# the stored rows of a piece and of a difference kernel
REG = ("C", "Q", "a", "D", "R")
SCL = ("G", "fp", "ap", "f", "h", "A")
CREG = ("V", "B", "a")
CSCL = ("fp", "ap", "f", "h", "A")


# ---- the two univariate polynomials

def interpolate(values, nodes):
    """Monomial coefficients (Fractions) of the interpolant: Newton's divided differences, expanded."""
    n = len(nodes)
    c = list(values)
    for j in range(1, n):
        for i in range(n - 1, j - 1, -1):
            c[i] = (c[i] - c[i - 1]) / (nodes[i] - nodes[i - j])
    poly = [c[-1]]
    for i in range(n - 2, -1, -1):
        shifted = [Q(0)] + poly
        poly = [shifted[k] - (nodes[i] * poly[k] if k < len(poly) else 0) for k in range(len(shifted))]
        poly[0] += c[i]
    return poly


def atan_over_x(z):
    """atan(x) / x at x^2 = z in [0, 1] by Euler's series sum 4^k (k!)^2 / (2k+1)! z^k / (1+z)^(k+1)."""
    y = z / (1 + z)
    term, tot = 1 / (1 + z), Q(0)
    for k in range(150):
        tot += term
        term = Q((term * y * Q(2 * (k + 1), 2 * k + 3)).limit_denominator(10 ** 60))
        if term < Q(1, 10 ** 40):
            break
    return tot.limit_denominator(10 ** 50)


def log1p_rest(f):
    """(log(1 + f) - f) / f^2 for small f."""
    return sum(Q((-1) ** (k + 1), k + 2) * f ** k for k in range(30))


def chebyshev_poly(fn, lo, hi, n):
    nodes = [Q(0.5 * (lo + hi) + 0.5 * (hi - lo) * math.cos(math.pi * (2 * k + 1) / (2 * n))).limit_denominator(10 ** 12)
             for k in range(n)]
    return interpolate([fn(z) for z in nodes], nodes)


N_ATAN, N_LOG, LOG_BITS = 22, 5, 6
LOG_HI0 = 0x3fe6a09e  # the high word of sqrt(1/2)


def log_table():
    """Per cell of 2^(20 - LOG_BITS) high words from sqrt(1/2) on: the reciprocal of its middle and minus that
    reciprocal's logarithm; 1 and 0 in the cell that holds 1.  And the largest |m reciprocal - 1| of any cell."""
    def value(hi):
        return struct.unpack("<d", struct.pack("<Q", hi << 32))[0]

    out, most = [], 0.0
    for i in range(1 << LOG_BITS):
        lo, hi = (value(LOG_HI0 + ((i + k) << (20 - LOG_BITS))) for k in (0, 1))
        inv = 1.0 if lo < 1.0 < hi else 2.0 / (lo + hi)
        out += [inv, float(-Decimal(inv).ln()) + 0.0]
        most = max(most, abs(lo * inv - 1.0), abs(hi * inv - 1.0))
    return out, most


def rounded(v, a3=None):
    """A rational, times a3 / pi if given, rounded to double."""
    if a3 is None:
        return float(v)
    d = Decimal(v.numerator) / Decimal(v.denominator) * Decimal(a3.numerator) / Decimal(a3.denominator) / PI
    return float(d)


def tables():
    out = []
    for K in KERNELS:
        t = kernel_box(K)
        a3 = t["a3pi"]
        rnd = lambda row: [rounded(v, a3) for v in row]  # noqa: E731
        out.append({"key": t["key"], "npiece": t["npiece"], "deg": t["deg"],
                    "creg": [{"c": float(r["c"]), **{k: rnd(r[k]) for k in CREG}} for r in t["creg"]],
                    "cscale": [{"b": float(s["b"]), "m": rounded(s["m"], a3), **{k: rnd(s[k]) for k in CSCL}}
                               for s in t["cscale"]],
                    "reg": [{"c": float(r["c"]), **{k: rnd(r[k]) for k in REG}} for r in t["reg"]],
                    "scale": [{"b": float(s["b"]), "m": rounded(s["m"], a3), "G": rnd(s["G"]),
                               **{k: rnd(s[k]) for k in SCL[1:]}} for s in t["scale"]]})
    return out


def _row(v):
    return "{" + ", ".join(_num(x) for x in v) + "}"


def header_text():
    T = tables()
    zr = {"c": 0.0, "C": [0.0] * 39, "Q": [0.0] * 15, "a": [0.0] * 6, "D": [0.0] * 84, "R": [0.0] * 28}
    zs = {"b": 0.0, "m": 0.0, "G": [0.0] * 12, "fp": [0.0] * 7, "ap": [0.0] * 6,
          "f": [0.0] * 14, "h": [0.0] * 15, "A": [0.0] * 21}
    L = [
        "// GENERATED by kiwi_b200/tables/gen_box_tables.py -- do not edit by hand.",
        "// Box-mass tables of the six SPH kernels (lengths in units of the support radius), normalised, derived in",
        "// exact rational arithmetic and rounded once to double; the formulas they enter stand in the generator.",
        "// Coefficient orders (powers):",
        "//   C:    (r - c)^0..12 | e2 ..8 | e2^2 ..4 | e3 ..6 | e2 e3 ..2 | e2^3 | e3^2",
        "//   Q:    P^1..6 | S P^0..4 | S^2 P^0..2 | S^3        (P = p^2 + q^2, S = p^2 q^2)",
        "//   G:    P^0..5 | S P^0..3 | S^2 P^0..1",
        "//   a, ap: x^4, x^6, .. x^14       fp: p, p^3, .. p^13       f, h: (b - p)^0..",
        "//   D:    (r - c)^0.. for each X^i S^j, i inner, 13 - 2 i - 4 j terms   R, A: X^i P^0.., i outer, total 6 and 5",
        "#pragma once",
        "",
        "#define KIWI_BOX_PIECES 3",
        "",
        "typedef struct KiwiBoxRegion {",
        "    double c, C[39], Q[15], a[6], D[84], R[28];",
        "} KiwiBoxRegion;",
        "typedef struct KiwiBoxScale {",
        "    double b, ib, m, G[12], fp[7], ap[6], f[14], h[15], A[21];",
        "} KiwiBoxScale;",
        "typedef struct KiwiBoxTable {",
        "    int npiece;                       /* pieces: piece k holds scale[k-1].b <= r < scale[k].b */",
        "    int deg;                          /* largest power of r */",
        "    KiwiBoxRegion reg[KIWI_BOX_PIECES];",
        "    KiwiBoxScale scale[KIWI_BOX_PIECES]; /* the difference kernel ending at b: piece k minus piece k+1 */",
        "} KiwiBoxTable;",
        "",
        "#ifndef KIWI_BOX_QUALIFIER",
        "#define KIWI_BOX_QUALIFIER static const",
        "#endif",
        "",
        "KIWI_BOX_QUALIFIER KiwiBoxTable kiwi_box_tables[6] = {",
    ]
    for t in T:
        L.append(f"    {{ /* {t['key']} */ {t['npiece']}, {t['deg']},")
        L.append("      {" + ",\n       ".join(
            "{" + _num(r["c"]) + ",\n        " + ",\n        ".join(_row(r[k]) for k in REG) + "}"
            for r in t["reg"] + [zr] * (3 - t["npiece"])) + "},")
        L.append("      {" + ",\n       ".join(
            "{" + f"{_num(s['b'])}, {_num(1.0 / s['b'] if s['b'] else 0.0)}, {_num(s['m'])},\n        " + ",\n        ".join(_row(s[k]) for k in SCL) +
            "}" for s in t["scale"] + [zs] * (3 - t["npiece"])) + "}},")
    L.append("};")
    L.append("")
    zr = {"c": 0.0, "V": [0.0] * 140, "B": [0.0] * 28, "a": [0.0] * 6}
    zs = {"b": 0.0, "m": 0.0, "fp": [0.0] * 7, "ap": [0.0] * 6, "f": [0.0] * 14, "h": [0.0] * 15, "A": [0.0] * 21}
    L += [
        "// The cones' tables.  V: (r - c)^0.. for each X^i P^j, by i + j, then i, 13 - 2 (i + j) terms; B like R.",
        "typedef struct KiwiConeRegion {",
        "    double c, V[140], B[28], a[6];",
        "} KiwiConeRegion;",
        "typedef struct KiwiConeScale {",
        "    double b, ib, m, fp[7], ap[6], f[14], h[15], A[21];",
        "} KiwiConeScale;",
        "typedef struct KiwiConeTable {",
        "    int npiece, deg;",
        "    KiwiConeRegion reg[KIWI_BOX_PIECES];",
        "    KiwiConeScale scale[KIWI_BOX_PIECES];",
        "} KiwiConeTable;",
        "",
        "KIWI_BOX_QUALIFIER KiwiConeTable kiwi_cone_tables[6] = {",
    ]
    for t in T:
        L.append(f"    {{ /* {t['key']} */ {t['npiece']}, {t['deg']},")
        L.append("      {" + ",\n       ".join(
            "{" + _num(r["c"]) + ",\n        " + ",\n        ".join(_row(r[k]) for k in CREG) + "}"
            for r in t["creg"] + [zr] * (3 - t["npiece"])) + "},")
        L.append("      {" + ",\n       ".join(
            "{" + f"{_num(s['b'])}, {_num(1.0 / s['b'] if s['b'] else 0.0)}, {_num(s['m'])},\n        " + ",\n        ".join(_row(s[k]) for k in CSCL) +
            "}" for s in t["cscale"] + [zs] * (3 - t["npiece"])) + "}},")
    L.append("};")
    L.append("")
    L.append("// atan(x) / x in powers of x^2 on [0, 1], and (log(1 + f) - f) / f^2 in powers of f")
    L.append(f"#define KIWI_N_ATAN {N_ATAN}")
    L.append("#define KIWI_ATAN_COEFS " + ", ".join(_num(float(c)) for c in chebyshev_poly(atan_over_x, 0.0, 1.0, N_ATAN)))
    table, most = log_table()
    L.append(f"// the logarithm's cells: pairs (reciprocal of the middle, minus its logarithm); |f| <= {most:.6f}")
    L.append(f"#define KIWI_LOG_BITS {LOG_BITS}")
    L.append(f"#define KIWI_LOG_HI0 0x{LOG_HI0:x}")
    L.append("#define KIWI_LOG_TABLE " + ", ".join(_num(v) for v in table))
    L.append(f"#define KIWI_N_LOG {N_LOG}")
    L.append("#define KIWI_LOG_COEFS " + ", ".join(_num(float(c)) for c in chebyshev_poly(log1p_rest, -most, most, N_LOG)))
    L.append("")
    return "\n".join(L)


def main(argv):
    text = header_text()
    if "--check" in argv:
        cur = open(OUT).read() if os.path.exists(OUT) else ""
        if cur != text:
            print(f"{OUT} is stale: rerun gen_box_tables.py")
            return 1
        print(f"{OUT} is up to date")
        return 0
    with open(OUT, "w") as f:
        f.write(text)
    print("wrote", OUT)
    return 0


if __name__ == "__main__":
    sys.exit(main(sys.argv[1:]))
