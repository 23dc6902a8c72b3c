"""What this framework is measured on: the calls its users make, over the sizes they make them at.

Cartesian maps (sph_to_grid on the device and from host arrays; cubic, generic, tabulated and FP32-mixed
forms), their gradients through the autograd binding, batches of snapshots, and Voronoi maps.  Inputs follow
the repository's own recipes (kiwi_b200/workloads.py: the gas column and the log-normal cube), with the
smoothing length taken from the recipe's known density instead of a neighbour search, so that they are made
quickly.  The Voronoi tessellation is a periodic block of jittered sites, copied.

`exact` integrates the kernel mass of each cell by Gauss-Legendre quadrature along the cell's edges: the mass
of the cone from the particle over a right triangle (wall distance r0, edge distance R0) is
1/(4 pi) int dphi r0 (N(rho(phi)) - N(r0)), N' = M(rho) / rho^2, M(rho) the kernel mass within rho.
"""
import math

import numpy as np
import torch

import kiwi_b200
from kiwi_b200 import autograd as kiwi_autograd

GRADS = ("x", "y", "z", "h", "m", "vx", "vy", "vz")


def listed():
    return [
        # the smallest call: a few particles on a coarse grid (a quick look, a unit test); latency and launches
        {"name": "grid_smallest", "kind": "grid", "field": "uniform", "n": 64, "nx": 12, "ny": 12, "nz": 12,
         "kernel": "cubic_spline", "form": "fp64"},
        # the example cutout's size: 7,300 gas particles on 100 x 100 x 410 cells of 0.02 pc, from host arrays into
        # pinned host arrays, as the command-line stage's user has them
        {"name": "cutout_from_host", "kind": "host", "field": "column", "n": 7300, "nx": 100, "ny": 100, "nz": 410,
         "kernel": "cubic_spline", "form": "fp64"},
        # a small snapshot with the quintic kernel on an odd grid: density and velocities
        {"name": "column_quintic", "kind": "grid", "field": "column", "n": 9001, "nx": 37, "ny": 41, "nz": 149,
         "kernel": "quintic_spline", "form": "fp64"},
        # an ordinary snapshot of a turbulent cloud on a ragged grid, device arrays
        {"name": "cloud_ragged", "kind": "grid", "field": "lognormal", "n": 150_000, "nx": 131, "ny": 117, "nz": 102,
         "kernel": "cubic_spline", "form": "fp64"},
        # the benchmark's size: 2 M particles of a log-normal cube on 256^3 cells
        {"name": "cloud_large", "kind": "grid", "field": "lognormal", "n": 2_000_000, "nx": 256, "ny": 256, "nz": 256,
         "kernel": "cubic_spline", "form": "fp64"},
        # a snapshot of a code that uses a Wendland kernel
        {"name": "cloud_wendland_c4", "kind": "grid", "field": "lognormal", "n": 100_000, "nx": 128, "ny": 128,
         "nz": 128, "kernel": "wendland_c4", "form": "fp64"},
        # the reference's lookup-table option
        {"name": "cloud_tabulated", "kind": "grid", "field": "lognormal", "n": 200_000, "nx": 120, "ny": 125,
         "nz": 130, "kernel": "cubic_spline", "form": "tabulated"},
        # the approximate fast form
        {"name": "cloud_fp32_mixed", "kind": "grid", "field": "lognormal", "n": 500_000, "nx": 192, "ny": 192,
         "nz": 192, "kernel": "cubic_spline", "form": "fp32_mixed"},
        # forward and backward through the autograd binding, as a fit of a snapshot to an observed map runs them
        {"name": "gradient_column", "kind": "gradient", "field": "column_cube", "n": 100_000, "nx": 80, "ny": 80,
         "nz": 80, "kernel": "cubic_spline", "form": "fp64"},
        {"name": "gradient_small_wendland", "kind": "gradient", "field": "column_cube", "n": 2000, "nx": 21, "ny": 19,
         "nz": 25, "kernel": "wendland_c4", "form": "fp64"},
        # a time series of small snapshots with mixed kernels, mapped in one launch
        {"name": "batch_of_snapshots", "kind": "batch", "field": "column", "items": 16, "n_min": 1000, "n_max": 20_000,
         "res_min": 24, "res_max": 64, "n": 16 * 6300, "nx": 16 * 41, "ny": 41, "nz": 41, "kernel": "cubic_spline",
         "form": "fp64"},
        # a snapshot mapped to Voronoi cells, one particle per cell, the tessellation resident on the GPU
        {"name": "voronoi_map", "kind": "voronoi", "field": "tile", "n": 64_000, "nx": 5, "ny": 5, "nz": 5,
         "kernel": "cubic_spline", "form": "fp64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cubic", "cubic", "cubic", "generic", "tabulated", "fp32", "host", "gradient", "batch", "voronoi"])
    generic = rng.choice(["quartic_spline", "quintic_spline", "wendland_c2", "wendland_c4", "wendland_c6"])
    field = rng.choice(["column", "lognormal", "lognormal"])

    def grid(lo, hi, n_lo, n_hi, **more):
        res = _log_int(rng, lo, hi)
        nx, ny, nz = (max(3, int(res * rng.uniform(0.8, 1.1))) for _ in range(3))
        # particles per cell from sparse to dense, as the recipes' grids have them
        n = min(n_hi, max(n_lo, int(nx * ny * nz * math.exp(rng.uniform(math.log(0.02), math.log(0.3))))))
        return {"field": field, "n": n, "nx": nx, "ny": ny, "nz": nz, **more}

    if kind == "cubic":
        return {"kind": "grid", "kernel": "cubic_spline", "form": "fp64", **grid(10, 210, 40, 1_500_000)}
    if kind == "generic":
        return {"kind": "grid", "kernel": generic, "form": "fp64", **grid(12, 110, 60, 200_000)}
    if kind == "tabulated":
        return {"kind": "grid", "kernel": "cubic_spline", "form": "tabulated", **grid(24, 150, 500, 500_000)}
    if kind == "fp32":
        return {"kind": "grid", "kernel": "cubic_spline", "form": "fp32_mixed", **grid(24, 200, 500, 1_000_000)}
    if kind == "host":
        return {"kind": "host", "kernel": "cubic_spline", "form": "fp64", **grid(16, 150, 100, 300_000),
                "field": "column"}
    if kind == "gradient":
        return {"kind": "gradient", "kernel": rng.choice(["cubic_spline", "cubic_spline", generic]), "form": "fp64",
                **grid(16, 60, 300, 60_000), "field": "column_cube"}
    if kind == "batch":
        items = rng.randint(4, 16)
        lo, hi = _log_int(rng, 500, 2000), _log_int(rng, 4000, 16_000)
        rlo, rhi = rng.randint(13, 30), rng.randint(34, 64)
        mid = int(math.sqrt(rlo * rhi))
        return {"kind": "batch", "field": "column", "items": items, "n_min": lo, "n_max": hi, "res_min": rlo,
                "res_max": rhi, "n": items * int(math.sqrt(lo * hi)), "nx": items * mid, "ny": mid, "nz": mid,
                "kernel": "cubic_spline", "form": "fp64"}
    nx, ny, nz = (rng.randint(1, 4) for _ in range(3))
    return {"kind": "voronoi", "field": "tile", "n": int(512 * nx * ny * nz * rng.uniform(0.5, 1.2)), "nx": nx,
            "ny": ny, "nz": nz, "kernel": rng.choice(["cubic_spline", "cubic_spline", generic]), "form": "fp64"}


# ------------------------------------------------------------------------------------------------- inputs

# h = hfact (m / rho)^(1/3) and the support in h, per kernel
HFACT = {"cubic_spline": 1.2, "quartic_spline": 1.1, "quintic_spline": 1.0, "wendland_c2": 1.3, "wendland_c4": 1.5,
         "wendland_c6": 1.6}
SUPPORT = {"cubic_spline": 2.0, "quartic_spline": 2.5, "quintic_spline": 3.0, "wendland_c2": 2.0, "wendland_c4": 2.0,
           "wendland_c6": 2.0}


def _finish(rng, pos, density, mass, hfact):
    """The snapshot's arrays: the smoothing length of the local number density with the scatter a neighbour
    count leaves in it, i.i.d. velocities."""
    n = len(pos)
    h = hfact * density ** (-1.0 / 3.0) * np.exp(0.045 * rng.standard_normal(n))
    vel = rng.standard_normal((n, 3))
    P = {k: np.ascontiguousarray(pos[:, a]) for a, k in enumerate(("x", "y", "z"))}
    P.update({k: np.ascontiguousarray(vel[:, a]) for a, k in enumerate(("vx", "vy", "vz"))})
    P["m"], P["h"] = np.full(n, mass), h
    return P


def _column(rng, n, box, hfact, sigma=0.15):
    """60 % uniform, 40 % in a Gaussian filament along z."""
    box = np.asarray(box)
    nu = int(round(0.6 * n))
    pos = rng.random((n, 3)) * box
    pos[nu:, :2] = 0.5 * box[:2] + sigma * rng.standard_normal((n - nu, 2))
    pos[:, :2] = np.abs(pos[:, :2])
    pos[:, :2] = np.minimum(pos[:, :2], 2 * box[:2] - pos[:, :2])
    r2 = ((pos[:, :2] - 0.5 * box[:2]) ** 2).sum(axis=1)
    dens = nu / box.prod() + (n - nu) / box[2] * np.exp(-0.5 * r2 / sigma ** 2) / (2 * math.pi * sigma ** 2)
    return _finish(rng, pos, dens, 0.05, hfact), (0.0, float(box[0]), 0.0, float(box[1]), 0.0, float(box[2]))


def _lognormal(rng, n, hfact, size=10.0, sigma_ln=1.5):
    """Particles sampling a log-normal density field with P(k) ~ k^-4, the domain padded by the largest support."""
    mesh = 128 if n > 300_000 else 64
    fk = np.fft.rfftn(rng.standard_normal((mesh, mesh, mesh)))
    kx, kz = np.fft.fftfreq(mesh), np.fft.rfftfreq(mesh)
    k2 = kx[:, None, None] ** 2 + kx[None, :, None] ** 2 + kz[None, None, :] ** 2
    k2[0, 0, 0] = np.inf
    g = np.fft.irfftn(fk / k2, s=(mesh, mesh, mesh))
    rho = np.exp(sigma_ln * (g - g.mean()) / g.std()).reshape(-1)
    rho /= rho.sum()
    cum = np.cumsum(rho)
    cells = np.minimum(np.searchsorted(cum, np.sort(rng.random(n)) * cum[-1]), mesh ** 3 - 1)
    dx = size / mesh
    pos = (np.stack(np.unravel_index(cells, (mesh, mesh, mesh)), axis=1) + rng.random((n, 3))) * dx
    order = rng.permutation(n)
    # a neighbour search smooths the emptiest regions: no length beyond an eighth of the box
    P = _finish(rng, pos[order], n * rho[cells[order]] / dx ** 3, 1000.0 / n, hfact)
    P["h"] = np.minimum(P["h"], size / 8)
    pad = float(2.0 * P["h"].max())
    return P, (-pad, size + pad) * 3


def _snapshot(case, seed):
    rng = np.random.default_rng([seed, case["n"], case["nx"]])
    n, hf = case["n"], HFACT[case["kernel"]]
    if case["field"] == "uniform":
        P = _finish(rng, rng.random((n, 3)), np.full(n, float(n)), 0.05, hf)
        P["h"] = rng.uniform(0.05, 0.15, n)
        return P, (0.0, 1.0) * 3
    if case["field"] == "column":
        return _column(rng, n, (2.0, 2.0, 8.2), hf)
    if case["field"] == "column_cube":
        return _column(rng, n, (4.0, 4.0, 4.0), hf)
    return _lognormal(rng, n, hf)


def _batch_items(case, seed):
    rng, sizes = np.random.default_rng([seed, case["items"], case["n_max"]]), np.random.default_rng(case["n_max"])
    out = []
    for i in range(case["items"]):
        n = int(round(math.exp(sizes.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        res = int(round(math.exp(sizes.uniform(math.log(case["res_min"]), math.log(case["res_max"])))))
        kernel = ("cubic_spline", "quintic_spline", "wendland_c4")[i % 3]
        P, bounds = _column(rng, n, (2.0, 2.0, 8.2), HFACT[kernel])
        out.append((P, bounds, (res, res, res), kernel))
    return out


TILE = 8  # sites per axis of the periodic block


def _tile_geometry(rng, device):
    """The Voronoi cells of a periodic block of TILE^3 jittered lattice sites of unit spacing, each formed on
    its own as the intersections of its bisector planes.  Returns sites (s, 3) and, per cell in a row,
    faces = (cell, neighbour site, neighbour block offset) with their vertices in order around the face,
    relative to the cell's site."""
    s = TILE ** 3
    lat = np.stack(np.meshgrid(*[np.arange(TILE)] * 3, indexing="ij"), axis=-1).reshape(s, 3)
    sites = torch.tensor(lat + 0.5 + rng.uniform(-0.33, 0.33, (s, 3)), device=device)
    lat = torch.tensor(lat, device=device)
    off = torch.tensor([(i, j, k) for i in range(-3, 4) for j in range(-3, 4) for k in range(-3, 4)
                        if (i, j, k) != (0, 0, 0)], device=device)
    nl = lat[:, None, :] + off[None]                               # neighbours' lattice positions
    blk = torch.div(nl, TILE, rounding_mode="floor")
    nm = nl - blk * TILE
    nid = (nm[..., 0] * TILE + nm[..., 1]) * TILE + nm[..., 2]
    d = sites[nid] + blk * TILE - sites[:, None, :]                 # bisector of d: v . d = |d|^2 / 2
    near = (d * d).sum(-1).argsort(dim=1, stable=True)[:, :44]
    d = torch.gather(d, 1, near[..., None].expand(-1, -1, 3))
    nid, blk = torch.gather(nid, 1, near), torch.gather(blk, 1, near[..., None].expand(-1, -1, 3))
    half = 0.5 * (d * d).sum(-1)
    tri = torch.combinations(torch.arange(44, device=device), 3)
    verts, owner, planes = [], [], []
    for lo in range(0, s, 64):
        D, Hh = d[lo:lo + 64], half[lo:lo + 64]
        a, b, c = (D[:, tri[:, q]] for q in range(3))
        ha, hb, hc = (Hh[:, tri[:, q], None] for q in range(3))
        bc, ca, ab = torch.linalg.cross(b, c), torch.linalg.cross(c, a), torch.linalg.cross(a, b)
        det = (a * bc).sum(-1, keepdim=True)
        v = (ha * bc + hb * ca + hc * ab) / det
        ok = (det.abs()[..., 0] > 1e-9) & ((v * v).sum(-1) < 9.0)
        ci, ti = torch.nonzero(ok, as_tuple=True)
        v, t = v[ci, ti], tri[ti]
        slack = (D[ci] * v[:, None, :]).sum(-1) - Hh[ci]
        slack.scatter_(1, t, -1.0)
        keep = (slack < 0.0).all(dim=1)
        verts.append(v[keep])
        owner.append(ci[keep] + lo)
        planes.append(t[keep])
    v, own, pl = torch.cat(verts), torch.cat(owner), torch.cat(planes)
    # (cell, plane) incidences, each face's vertices sorted by angle, clockwise seen from outside
    v3, own3, pl3 = v.repeat(3, 1), own.repeat(3), pl.t().reshape(-1)
    nrm = d[own3, pl3]
    key = own3 * 64 + pl3
    uniq, inv, cnt = torch.unique(key, return_inverse=True, return_counts=True)
    # (the mean is formed per face in a fixed order on the host: a floating-point scatter has none)
    inv_h = inv.cpu().numpy()
    mean = np.stack([np.bincount(inv_h, weights=v3[:, a].cpu().numpy()) for a in range(3)], axis=1)
    mean = torch.tensor(mean, device=device) / cnt[:, None]
    axis = torch.nn.functional.one_hot(nrm.abs().argmin(dim=1), 3).to(nrm)
    e1 = torch.linalg.cross(nrm, axis)
    e1 = e1 / (e1 * e1).sum(-1, keepdim=True).sqrt()
    e2 = torch.linalg.cross(e1, nrm) / (nrm * nrm).sum(-1, keepdim=True).sqrt()
    w = v3 - mean[inv]
    ang = torch.atan2((w * e2).sum(-1), (w * e1).sum(-1))
    order = np.lexsort((ang.cpu().numpy(), inv_h))
    v3, cnt = v3.cpu().numpy()[order], cnt.cpu().numpy()
    big = cnt >= 3
    take = np.repeat(big, cnt)
    cell, plane = uniq.cpu().numpy() // 64, uniq.cpu().numpy() % 64
    return {"sites": sites.cpu().numpy(), "cell": cell[big], "nbr": nid.cpu().numpy()[cell, plane][big],
            "blk": blk.cpu().numpy()[cell, plane][big], "count": cnt[big], "verts": v3[take]}


def _tessellation(case, seed, device):
    """nx x ny x nz copies of the block: the CSR geometry map_voronoi_device takes, the sites, the particles
    (scattered about the sites as gas is about generators moved to their cells' centroids) and their cells."""
    rng = np.random.default_rng([seed, case["n"], case["nx"], case["ny"], case["nz"]])
    T = _tile_geometry(rng, device)
    s, dims = TILE ** 3, np.array([case["nx"], case["ny"], case["nz"]])
    scale = 5.0 / (TILE * dims.max())
    copies = np.stack(np.meshgrid(*[np.arange(k) for k in dims], indexing="ij"), axis=-1).reshape(-1, 3)
    nb, nf = len(copies), len(T["cell"])
    shift = copies[:, None, :] + T["blk"][None]
    inside = ((shift >= 0) & (shift < dims)).all(axis=-1)
    nbr = (((shift[..., 0] * dims[1]) + shift[..., 1]) * dims[2] + shift[..., 2]) * s + T["nbr"][None]
    face_nbr = np.where(inside, nbr, -1).astype(np.int32).reshape(-1)
    per_cell = np.bincount(T["cell"], minlength=s)
    face_off = np.concatenate([[0], np.cumsum(np.tile(per_cell, nb))])
    vert_off = np.concatenate([[0], np.cumsum(np.tile(T["count"], nb))])
    vcell = np.repeat(T["cell"], T["count"])
    base = T["sites"][vcell] + T["verts"]
    vxyz = ((base[None] + (copies * TILE)[:, None, :]) * scale).reshape(-1)
    sites = ((T["sites"][None] + (copies * TILE)[:, None, :]) * scale).reshape(-1, 3)
    # cell volumes: pyramids from the site over each face's fan of triangles
    rel = T["verts"]
    start = np.concatenate([[0], np.cumsum(T["count"])])[:-1]
    first = np.repeat(start, T["count"])
    nxt = np.arange(len(rel)) + 1
    nxt = np.where(nxt - first == np.repeat(T["count"], T["count"]), first, nxt)
    vol6 = np.abs(np.einsum("ij,ij->i", rel[first], np.cross(rel, rel[nxt])))
    volume = np.tile(np.bincount(vcell, weights=vol6, minlength=s) / 6.0, nb) * scale ** 3
    n, nc = case["n"], nb * s
    who = rng.permutation(nc)[:n] if n <= nc else np.concatenate([np.arange(nc), rng.integers(0, nc, n - nc)])
    pos = sites[who] + 0.15 * scale * rng.standard_normal((n, 3))
    lo, hi = 0.02 * scale, (dims * TILE - 0.02) * scale
    pos = np.clip(pos, lo, hi)
    P = _finish(rng, pos, np.full(n, scale ** -3), 0.05, HFACT[case["kernel"]])
    # home cell: the nearest site among the lattice neighbours of the particle
    pt, st = torch.tensor(pos, device=device), torch.tensor(sites, device=device)
    lat = torch.tensor(np.floor(pos / scale).astype(np.int64), device=device)
    lim = torch.tensor(dims * TILE, device=device)
    best = torch.full((n,), math.inf, dtype=torch.float64, device=device)
    home = torch.full((n,), -1, dtype=torch.int32, device=device)
    for o in [(i, j, k) for i in (-2, -1, 0, 1, 2) for j in (-2, -1, 0, 1, 2) for k in (-2, -1, 0, 1, 2)]:
        q = lat + torch.tensor(o, device=device)
        ok = ((q >= 0) & (q < lim)).all(dim=1)
        q = q.clamp(min=0).minimum(lim - 1)
        blk, loc = q // TILE, q % TILE
        cid = ((blk[:, 0] * dims[1] + blk[:, 1]) * dims[2] + blk[:, 2]) * s + (loc[:, 0] * TILE + loc[:, 1]) * TILE + loc[:, 2]
        d2 = ((st[cid] - pt) ** 2).sum(dim=1)
        better = ok & (d2 < best)
        best, home = torch.where(better, d2, best), torch.where(better, cid.int(), home)
    cells = {"face_off": face_off.astype(np.int64), "vert_off": vert_off.astype(np.int64), "vxyz": vxyz,
             "face_nbr": face_nbr, "volume": volume}
    return P, home, cells, sites, scale


def _integrator(case):
    return kiwi_b200.make_kernel_integrator(case["kernel"], use_tabulated_integral=case["form"] == "tabulated")


def _out(case, nc, device):
    """What the call is asked for.  A column fills its grid, so density and velocities; a padded or sparse
    grid has cells that only graze a support, whose velocity is a ratio of rounding errors, so there the
    program asks for the density and the raw sums (mass and momenta) and divides where it needs to."""
    def new(k):
        return torch.empty(k, dtype=torch.float64, device=device)

    if case["field"] in ("column", "tile"):
        return {k: new(nc) for k in ("density", "vx", "vy", "vz")}
    return {"density": new(nc), "raw4": new(4 * nc)}


def _to(P, device):
    return {k: torch.from_numpy(v).to(device) for k, v in P.items()}


def prepare(case, seed):
    device = torch.device("cuda", 0)
    kind = case["kind"]
    state = {"case": case, "kernel": _integrator(case), "precision": "fp32_mixed" if case["form"] == "fp32_mixed" else "fp64"}
    if kind == "batch":
        items = []
        for P, bounds, shape, kernel in _batch_items(case, seed):
            items.append({"particles": _to(P, device), "bounds": bounds, "shape": shape,
                          "kernel": kiwi_b200.make_kernel_integrator(kernel), "out": _out(case, math.prod(shape), device)})
        torch.cuda.synchronize()
        state["items"], state["batch"] = items, kiwi_b200.Batch(items)
        return state
    if kind == "voronoi":
        P, home, cells, _, _ = _tessellation(case, seed, device)
        state.update(particles=_to(P, device), home=home, cells=_to(cells, device),
                     out=_out(case, len(cells["volume"]), device))
        torch.cuda.synchronize()
        return state
    P, bounds = _snapshot(case, seed)
    shape = (case["nx"], case["ny"], case["nz"])
    state.update(bounds=bounds, shape=shape)
    if kind == "host":
        state["particles"] = P
        pinned = torch.empty((4, math.prod(shape)), dtype=torch.float64, pin_memory=True)
        state["pinned"], state["out"] = pinned, [pinned[i].numpy() for i in range(4)]
        return state
    state["particles"] = _to(P, device)
    if kind == "gradient":
        rng = np.random.default_rng([seed, 7])
        state["cotangent"] = torch.from_numpy(rng.standard_normal((4,) + shape)).to(device)
        for v in state["particles"].values():
            v.requires_grad_(True)
    else:
        state["out"] = _out(case, math.prod(shape), device)
    torch.cuda.synchronize()
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "batch":
        state["batch"].run()
        return [it["out"] for it in state["items"]]
    if kind == "voronoi":
        kiwi_b200.map_voronoi_device(state["particles"], state["home"], state["cells"], state["out"],
                                     kernel=state["kernel"])
        return state["out"]
    if kind == "host":
        r = kiwi_b200.sph_to_grid(state["particles"], state["bounds"], state["shape"], kernel=state["kernel"],
                                  out=state["out"])
        return {"density": r.density, "vx": r.vx, "vy": r.vy, "vz": r.vz}
    if kind == "gradient":
        P = state["particles"]
        raw = kiwi_autograd.sph_to_grid_raw(*[P[k] for k in GRADS], state["bounds"], state["shape"],
                                            kernel=state["kernel"])
        grads = torch.autograd.grad(raw, [P[k] for k in GRADS], state["cotangent"])
        return {"raw": raw.detach(), **dict(zip(GRADS, grads))}
    kiwi_b200.sph_to_grid_device(state["particles"], state["bounds"], state["shape"], state["out"],
                                 kernel=state["kernel"], precision=state["precision"])
    return state["out"]


# ------------------------------------------------------------------------------------------------- work

def _pairs(P, bounds, shape, kernel):
    """Expected (particle, cell) pairs within support: the cells a ball meets, for a random place on the grid."""
    cell = [(bounds[2 * a + 1] - bounds[2 * a]) / shape[a] for a in range(3)]
    r = SUPPORT[kernel] * P["h"]
    a, b, c = cell
    met = a * b * c + 2 * r * (a * b + b * c + c * a) + math.pi * r ** 2 * (a + b + c) + 4 / 3 * math.pi * r ** 3
    if len(r) == 0:
        return 0.0
    return float(np.minimum(met / (a * b * c), math.prod(shape)).sum())


def work(case):
    """Bytes: each particle and cell array once.  Operations per (particle, cell) pair within support: its one
    new lattice point's value (a root, two reciprocals, three logarithms, five arctangents at 20 operations
    each, six short series), its share of the edge lines and its sum; a Voronoi pair has half of its cell's
    15 faces of 5 edges to evaluate, two series each."""
    kind = case["kind"]
    if kind == "voronoi":
        cells = TILE ** 3 * case["nx"] * case["ny"] * case["nz"]
        reach = SUPPORT[case["kernel"]] * HFACT[case["kernel"]]
        pairs = case["n"] * (1 + 4 * reach + 3 * math.pi * reach ** 2 / 2 + 4 / 3 * math.pi * reach ** 3)
        return {"bytes": case["n"] * 68 + cells * (15.5 * (5.2 * 24 + 12) + 8 + 8 + 32), "flops": pairs * 7.5 * 5.2 * 2 * 200}
    if kind == "batch":
        todo = [(P, b, s, k) for P, b, s, k in _batch_items(case, 0)]
    else:
        P, bounds = _snapshot(case, 0)
        todo = [(P, bounds, (case["nx"], case["ny"], case["nz"]), case["kernel"])]
    bytes_, flops = 0.0, 0.0
    outs = 4 if case["field"] == "column" else 5
    for P, bounds, shape, kernel in todo:
        n, nc, pairs = len(P["h"]), math.prod(shape), _pairs(P, bounds, shape, kernel)
        per = 40 if case["form"] == "tabulated" else 600 if kernel == "cubic_spline" else 1200
        if kind == "gradient":
            bytes_ += n * 64 * 3 + nc * 32 * 2
            flops += pairs * per * 4
        else:
            bytes_ += n * 64 + nc * 8 * outs
            flops += pairs * per
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------------------------------------------- exact values

# kernels as sums of truncated powers of q = r / h: (normalisation, [(coefficient, breakpoint, power)]), or a
# Wendland polynomial times (1 - q/2)^power
_SPLINES = {
    "cubic_spline": (1 / math.pi, [(0.25, 2.0, 3), (-1.0, 1.0, 3)]),
    "quartic_spline": (1 / (20 * math.pi), [(1.0, 2.5, 4), (-5.0, 1.5, 4), (10.0, 0.5, 4)]),
    "quintic_spline": (1 / (120 * math.pi), [(1.0, 3.0, 5), (-6.0, 2.0, 5), (15.0, 1.0, 5)]),
}
_WENDLAND = {
    "wendland_c2": (21 / (16 * math.pi), 4, [1.0, 2.0]),
    "wendland_c4": (495 / (256 * math.pi), 6, [1.0, 3.0, 35 / 12]),
    "wendland_c6": (1365 / (512 * math.pi), 8, [1.0, 4.0, 25 / 4, 4.0]),
}


def _kernel_regions(kernel):
    """(breakpoints, N): N[k] holds the coefficients by power of q (from q^-1) of the antiderivative of
    M(q) / q^2 on region k, M the mass within q h; the last region lies beyond the support (M = 1)."""
    from numpy.polynomial import polynomial as pl

    if kernel in _SPLINES:
        norm, terms = _SPLINES[kernel]
        breaks = sorted(b for _, b, _ in terms)
        polys = []
        for b in breaks:
            w = np.zeros(1)
            for c, t, p in terms:
                if t >= b:
                    w = pl.polyadd(w, c * pl.polypow([t, -1.0], p))
            polys.append(norm * w)
    else:
        norm, p, poly = _WENDLAND[kernel]
        breaks, polys = [2.0], [norm * pl.polymul(pl.polypow([1.0, -0.5], p), poly)]
    N, mass, val, lo = [], 0.0, 0.0, 0.0
    for b, w in zip(breaks, polys):
        M = pl.polyint(4 * math.pi * pl.polymul([0.0, 0.0, 1.0], w))
        M[0] = mass - (pl.polyval(lo, M) - M[0])
        n = np.zeros(len(M))                      # n[j] multiplies q^(j - 1); M has no q^1 term
        for j, c in enumerate(M):
            if j != 1 and c != 0.0:
                n[j] = c / (j - 1)
        at = (lambda q, n=n: sum(c * q ** (j - 1) for j, c in enumerate(n) if c != 0.0))
        n[1] += val - (at(lo) if lo > 0 else 0.0)
        mass, val, lo = pl.polyval(b, M), at(b), b
        N.append(n)
    N.append(np.array([-1.0, val + 1.0 / lo]))
    width = max(len(n) for n in N)
    return breaks, np.stack([np.pad(n, (0, width - len(n))) for n in N])


class _Quadrature:
    def __init__(self, kernel, device, nodes=40):
        self.breaks, N = _kernel_regions(kernel)
        self.N = torch.tensor(N, device=device)
        x, w = np.polynomial.legendre.leggauss(nodes)
        self.x, self.w = torch.tensor(0.5 * (x + 1), device=device), torch.tensor(0.5 * w, device=device)

    def _n(self, q, region):
        c = self.N[region]
        s = torch.zeros_like(q)
        for j in range(c.shape[-1] - 1, 0, -1):
            s = s * q + c[..., j]
        return s + c[..., 0] / q

    def cone(self, r0, R0, t):
        """Kernel mass (lengths in h) of the cone over the right triangle with legs R0 and t in the plane at r0,
        all > 0.  With tan(phi) = sinh(v) the integrand has no singularity within pi/2 of the real axis."""
        brk = torch.tensor(self.breaks, dtype=torch.float64, device=r0.device)
        reg0 = torch.bucketize(r0.detach(), brk)
        n0 = self._n(r0, reg0)
        end = torch.asinh(t / R0)
        lo, total = torch.zeros_like(end), torch.zeros_like(end)
        for k in range(len(self.breaks) + 1):
            if k < len(self.breaks):
                c = torch.sqrt((self.breaks[k] ** 2 - r0 * r0).clamp(min=0.0)) / R0
                hi = torch.minimum(torch.acosh(c.clamp(min=1.0)).detach(), end)
            else:
                hi = end
            v = lo[:, None] + (hi - lo)[:, None] * self.x
            ch = torch.cosh(v)
            rho = torch.sqrt((r0 * r0)[:, None] + (R0 * R0)[:, None] * ch * ch)
            f = (self._n(rho, torch.full((1, 1), k, dtype=torch.long, device=r0.device)) - n0[:, None]) / ch
            total = total + (hi - lo) * (f * self.w).sum(-1)
            lo = hi
        return r0 * total / (4 * math.pi)

    def octant(self, a, b, c):
        """Kernel mass of the box between the particle and a point at offsets a, b, c > 0."""
        s = torch.zeros_like(a)
        for r0, p, q in ((a, b, c), (b, a, c), (c, a, b)):
            s = s + self.cone(r0, p, q) + self.cone(r0, q, p)
        return s


def _ragged(count):
    """Owner and index within it of every element of lists of these lengths."""
    owner = torch.repeat_interleave(torch.arange(len(count), device=count.device), count)
    first = torch.cumsum(count, 0) - count
    return owner, torch.arange(len(owner), device=count.device) - first[owner]


def _grid_chunks(P, bounds, shape, kernel, points):
    """Slices of the particles with about `points` lattice points each."""
    lo, dim = _boxes(P, bounds, shape, kernel)
    cum = torch.cumsum((dim + 1).prod(dim=1), 0).cpu().numpy()
    at, out = 0, []
    while at < len(cum):
        base = cum[at - 1] if at else 0
        to = max(at + 1, int(np.searchsorted(cum, base + points)))
        out.append(slice(at, to))
        at = to
    return out, (int(cum[-1]) if len(cum) else 0)


def _boxes(P, bounds, shape, kernel):
    lo, hi = [], []
    for a, k in enumerate(("x", "y", "z")):
        cell = (bounds[2 * a + 1] - bounds[2 * a]) / shape[a]
        r = SUPPORT[kernel] * P["h"]
        lo.append((torch.floor((P[k] - r - bounds[2 * a]) / cell) - 1).clamp(0, shape[a] - 1))
        hi.append((torch.floor((P[k] + r - bounds[2 * a]) / cell) + 1).clamp(0, shape[a] - 1))
    lo, hi = torch.stack(lo, 1).long().detach(), torch.stack(hi, 1).long().detach()
    return lo, hi - lo + 1


def _cell_masses(Q, P, bounds, shape, kernel):
    """Every (particle, cell of its box) pair's kernel mass: (owner, flat cell, mass)."""
    lo, dim = _boxes(P, bounds, shape, kernel)
    npt = dim + 1
    own, at = _ragged(npt.prod(dim=1))
    n = npt[own]
    ijk = torch.stack([at // (n[:, 1] * n[:, 2]), (at // n[:, 2]) % n[:, 1], at % n[:, 2]], dim=1)
    off = []
    for a, k in enumerate(("x", "y", "z")):
        cell = (bounds[2 * a + 1] - bounds[2 * a]) / shape[a]
        off.append((bounds[2 * a] + (lo[own, a] + ijk[:, a]).double() * cell - P[k][own]) / P["h"][own])
    sign = torch.sign(off[0]) * torch.sign(off[1]) * torch.sign(off[2])
    T = sign.detach() * Q.octant(*[o.abs().clamp(min=1e-30) for o in off])
    first = torch.cumsum(npt.prod(dim=1), 0) - npt.prod(dim=1)
    owc, atc = _ragged(dim.prod(dim=1))
    d, n = dim[owc], npt[owc]
    i, j, k = atc // (d[:, 1] * d[:, 2]), (atc // d[:, 2]) % d[:, 1], atc % d[:, 2]
    base = first[owc] + (i * n[:, 1] + j) * n[:, 2] + k
    n2, n12 = n[:, 2], n[:, 1] * n[:, 2]
    m = ((T[base + n12 + n2 + 1] - T[base + n12 + n2]) - (T[base + n12 + 1] - T[base + n12])
         - ((T[base + n2 + 1] - T[base + n2]) - (T[base + 1] - T[base])))
    flat = ((lo[owc, 0] + i) * shape[1] + lo[owc, 1] + j) * shape[2] + lo[owc, 2] + k
    return owc, flat, m


def _sums(owner, flat, mass, P, nc):
    mm = mass * P["m"][owner]
    out = [torch.zeros(nc, dtype=torch.float64, device=mm.device).index_add(0, flat, w)
           for w in (mm, mm * P["vx"][owner], mm * P["vy"][owner], mm * P["vz"][owner])]
    return torch.stack(out)


def _fields(raw, volume, P, case):
    M = raw[0]
    if "raw4" in _out(case, 1, "cpu"):
        return {"density": M / volume, "raw4": raw.reshape(-1)}
    v = [torch.where(M > 0, raw[1 + a] / M, P[k].mean()) for a, k in enumerate(("vx", "vy", "vz"))]
    return {"density": M / volume, "vx": v[0], "vy": v[1], "vz": v[2]}


def _exact_grid(P, bounds, shape, case, kernel, limit=100_000_000):
    chunks, total = _grid_chunks(P, bounds, shape, kernel, 100_000)
    if total > limit:
        return None
    Q, nc = _Quadrature(kernel, P["x"].device), math.prod(shape)
    raw = torch.zeros((4, nc), dtype=torch.float64, device=P["x"].device)
    for c in chunks:
        Pc = {k: v[c] for k, v in P.items()}
        raw += _sums(*_cell_masses(Q, Pc, bounds, shape, kernel), Pc, nc)
    volume = math.prod((bounds[2 * a + 1] - bounds[2 * a]) / shape[a] for a in range(3))
    return _fields(raw, volume, P, case)


def _exact_gradient(P, bounds, shape, case, cot):
    chunks, total = _grid_chunks(P, bounds, shape, case["kernel"], 25_000)
    if total > 6_000_000:
        return None
    Q, nc = _Quadrature(case["kernel"], P["x"].device), math.prod(shape)
    raw = torch.zeros((4, nc), dtype=torch.float64, device=P["x"].device)
    grads = {k: [] for k in GRADS}
    for c in chunks:
        Pc = {k: v[c].clone().requires_grad_(True) for k, v in P.items()}
        part = _sums(*_cell_masses(Q, Pc, bounds, shape, case["kernel"]), Pc, nc)
        for k, g in zip(GRADS, torch.autograd.grad(part, [Pc[k] for k in GRADS], cot.reshape(4, nc))):
            grads[k].append(g)
        raw += part.detach()
    return {"raw": raw.reshape((4,) + tuple(shape)), **{k: torch.cat(v) for k, v in grads.items()}}


def _exact_voronoi(case, seed, device):
    """Each (particle, cell) pair within reach: the cell's faces' triangle fans about the particle's foot point."""
    if case["n"] > 4000:
        return None
    P, _, cells, sites, scale = _tessellation(case, seed, device)
    P = _to(P, device)
    Q, kernel = _Quadrature(case["kernel"], device), case["kernel"]
    st, nc = torch.tensor(sites, device=device), len(cells["volume"])
    fo, vo = torch.tensor(cells["face_off"], device=device), torch.tensor(cells["vert_off"], device=device)
    vx = torch.tensor(cells["vxyz"], device=device).reshape(-1, 3)
    raw = torch.zeros((4, nc), dtype=torch.float64, device=device)
    pos = torch.stack([P["x"], P["y"], P["z"]], 1)
    for lo in range(0, case["n"], 32):
        Pc = {k: v[lo:lo + 32] for k, v in P.items()}
        p, h = pos[lo:lo + 32], Pc["h"]
        near = ((p[:, None] - st[None]) ** 2).sum(-1).sqrt() < SUPPORT[kernel] * h[:, None] + 2.0 * scale
        who, cell = torch.nonzero(near, as_tuple=True)
        o1, f = _ragged((fo[1:] - fo[:-1])[cell])
        f = f + fo[cell][o1]
        o2, e = _ragged((vo[1:] - vo[:-1])[f])
        first, cnt = vo[f][o2], (vo[1:] - vo[:-1])[f][o2]
        pair = o1[o2]
        at, q, hh = cell[pair], p[who[pair]], h[who[pair], None]
        A, B = (vx[first + e] - q) / hh, (vx[first + (e + 1) % cnt] - q) / hh
        # the face's plane from the sum of its fan's cross products, turned outwards
        V0 = vx[first]
        fan = torch.linalg.cross(vx[first + e] - V0, vx[first + (e + 1) % cnt] - V0)
        area = torch.zeros((len(f), 3), dtype=torch.float64, device=device).index_add(0, o2, fan)[o2]
        nrm = area / area.norm(dim=1, keepdim=True)
        turn = torch.sign((nrm * (V0 - st[at])).sum(1))
        nrm = nrm * turn[:, None]
        d = (nrm * A).sum(1)
        r0, foot = d.abs(), nrm * d[:, None]
        a, b = A - foot, B - foot
        edge = b - a
        ln = edge.norm(dim=1, keepdim=True)
        edge = edge / ln
        R0 = torch.linalg.cross(a, edge).norm(dim=1)
        sa, sb = (a * edge).sum(1), (b * edge).sum(1)
        out = torch.linalg.cross(edge, nrm)                         # in the plane, across the edge
        side = torch.sign((out * a).sum(1))                         # which side of the edge the foot point is on
        ok = (r0 > 1e-14) & (R0 > 1e-14) & (ln[:, 0] > 1e-14)
        val = torch.zeros_like(r0)
        for s, sg in ((sb, 1.0), (sa, -1.0)):
            m = ok & (s.abs() > 1e-14)
            val[m] += sg * torch.sign(s[m]) * Q.cone(r0[m], R0[m], s[m].abs())
        val = val * side * turn * torch.sign(d)
        mass = torch.zeros(len(who), dtype=torch.float64, device=device).index_add(0, pair, val)
        raw += _sums(who, cell, mass, Pc, nc)
    return _fields(raw, torch.tensor(cells["volume"], device=device), P, case)


def exact(case, seed):
    device = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
    kind = case["kind"]
    if case["form"] == "tabulated":
        return None  # the option's value is its table's, not the integral's
    if kind == "voronoi":
        return _exact_voronoi(case, seed, device)
    if kind == "batch":
        items = [(_to(P, device), bounds, shape, kernel) for P, bounds, shape, kernel in _batch_items(case, seed)]
        if sum(_grid_chunks(P, b, s, k, 100_000)[1] for P, b, s, k in items) > 150_000_000:
            return None
        return [_exact_grid(P, b, s, case, k) for P, b, s, k in items]
    P, bounds = _snapshot(case, seed)
    P, shape = _to(P, device), (case["nx"], case["ny"], case["nz"])
    if kind == "gradient":
        cot = np.random.default_rng([seed, 7]).standard_normal((4,) + shape)
        return _exact_gradient(P, bounds, shape, case, torch.from_numpy(cot).to(device))
    return _exact_grid(P, bounds, shape, case, case["kernel"])
