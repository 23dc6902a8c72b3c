"""Every kernel through every entry point that maps a grid: the whole grid, parts, a batch of all kernels, and the
allocation-free call, whose one body serves five of them with sizes read at run time.  The same bits."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_segments import _particles

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

KERNELS = ["cubic_spline", "quartic_spline", "quintic_spline", "wendland_c2", "wendland_c4", "wendland_c6"]
BOUNDS = (0.0, 1.0) * 3


def _new(nc):
    out = {k: torch.full((nc,), np.nan, dtype=torch.float64, device="cuda") for k in ("density", "vx", "vy", "vz")}
    out["raw4"] = torch.full((4 * nc,), np.nan, dtype=torch.float64, device="cuda")
    return out


def _noalloc(kiwi, P, shape, ki, out):
    f = kiwi.load_library().kiwi_sph_to_grid_device_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.POINTER(kiwi.KiwiParticles), C.POINTER(kiwi.KiwiCartGrid), C.POINTER(kiwi.KiwiKernelSel),
                  C.c_int] + [C.POINTER(C.c_double)] * 5 + [C.POINTER(kiwi.KiwiStats), C.c_char_p, C.c_size_t]
    Ps, _ = kiwi._particles_struct(P, device=True)
    ptr = [C.cast(C.c_void_p(int(out[k].data_ptr())), C.POINTER(C.c_double)) for k in ("density", "vx", "vy", "vz", "raw4")]
    sel, st, err = ki.sel(), kiwi.KiwiStats(), C.create_string_buffer(256)
    rc = f(None, C.byref(Ps), C.byref(kiwi.KiwiCartGrid((C.c_double * 6)(*BOUNDS), *shape)), C.byref(sel), kiwi.KIWI_FP64,
           *ptr, C.byref(st), err, 256)
    torch.cuda.synchronize()
    assert rc == 0, err.value


# supports of a cell or two, and of half the grid
@pytest.mark.parametrize("hmax,shape", [(0.06, (25, 17, 40)), (0.3, (17, 16, 23))])
def test_every_kernel_has_one_result(kiwi, ctx, hmax, shape):
    nc = int(np.prod(shape))
    P = _particles(torch, 1500, hmax, 12)
    items = []
    for k in KERNELS:
        ki, whole, parts, na, item = kiwi.make_kernel_integrator(k), _new(nc), _new(nc), _new(nc), _new(nc)
        torch.cuda.synchronize()
        kiwi.sph_to_grid_device(P, BOUNDS, shape, whole, kernel=ki, ctx=ctx)
        for p in range(3):
            kiwi.sph_to_grid_device(P, BOUNDS, shape, parts, kernel=ki, ctx=ctx, part=p, n_parts=3)
        _noalloc(kiwi, P, shape, ki, na)
        for q in whole:
            assert torch.equal(parts[q], whole[q]), (k, q)
            assert torch.equal(na[q], whole[q]), (k, q)
        items.append(({"particles": P, "bounds": BOUNDS, "shape": shape, "kernel": ki, "out": item}, whole))
    batch = kiwi.Batch([i[0] for i in items], ctx=ctx)
    batch.run()
    batch.close()
    for k, (item, whole) in zip(KERNELS, items):
        for q in whole:
            assert torch.equal(item["out"][q], whole[q]), (k, q)
