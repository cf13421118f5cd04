"""Device pointers that a kernel cannot use as they lie are copied first: arrays
off their alignment, pinned host memory, results written over the targets."""
import ctypes as C

import numpy as np
import pytest

from sph_2_b200 import Config, Context, _lib as L, ic

pytestmark = pytest.mark.gpu
NAMES = ["x", "y", "z", "vx", "vy", "vz", "m", "h", "u"]


def _shifted(a, by):
    """A device copy of `a` that begins `by` bytes off a 256-byte boundary."""
    import torch
    raw = np.frombuffer(a.tobytes(), np.uint8)
    t = torch.zeros(len(raw) + 256, dtype=torch.uint8, device="cuda")
    t[by:by + len(raw)] = torch.tensor(raw, device="cuda")
    return t, t.data_ptr() + by


def _state(n):
    rng = np.random.default_rng(n)
    a = {k: rng.normal(size=n) for k in NAMES}
    a["h"], a["m"] = np.abs(a["h"]) + 0.1, np.abs(a["m"])
    return a


@pytest.mark.parametrize("by", [1, 4, 8, "pinned"])
@pytest.mark.parametrize("n", [1, 1000, 70_001])
def test_load(n, by):
    import torch
    a = _state(n)
    if by == "pinned":
        keep = [torch.tensor(a[k]).pin_memory() for k in NAMES]
        ptr = [t.data_ptr() for t in keep]
    else:
        keep, ptr = zip(*(_shifted(a[k], by) for k in NAMES))
    torch.cuda.synchronize()
    lib = L.load()
    with Context(Config(n_max=n, precision="mixed")) as ctx:
        L.check(lib.sph_load(ctx.handle, n, None, *map(C.c_void_p, ptr), 0), "load")
        for k in NAMES:
            assert np.array_equal(ctx.get(k), a[k]), k


@pytest.mark.parametrize("by", [0, 2, 4, "over"])
@pytest.mark.parametrize("spline", [True, False])
def test_direct_sums(by, spline):
    import torch
    n, nt = 3000, 700
    d = ic.evrard(n, seed=1)
    tg = np.random.default_rng(3).choice(n, nt, replace=False).astype(np.int32)
    eps = np.linspace(0.01, 0.02, n)
    lib = L.load()
    with Context(Config(n_max=n, precision="fp64")) as ctx:
        ctx.load(d["pos"], d["vel"], d["m"], d["h"], d["u"])
        ctx.sort()
        want = ctx.gravity_direct_spline(eps, tg) if spline else np.column_stack(ctx.gravity_direct(tg))
        width = want.shape[1]
        kt, pt = _shifted(tg, 0 if by == "over" else by)
        ke, pe = _shifted(eps, 0 if by == "over" else by)
        if by == "over":        # the results begin where the targets do
            ko = torch.zeros(width * nt, dtype=torch.float64, device="cuda")
            ko.view(torch.int32)[:nt] = torch.tensor(tg, device="cuda")
            off, pt = 0, ko.data_ptr()
            ko, po = ko.view(torch.uint8), ko.data_ptr()
        else:
            off = by
            ko, po = _shifted(np.zeros(width * nt), by)
        torch.cuda.synchronize()
        if spline:
            L.check(lib.sph_gravity_direct_spline(ctx.handle, C.c_void_p(pe), nt, C.c_void_p(pt),
                                                  C.c_void_p(po), 0), "spline")
        else:
            L.check(lib.sph_gravity_direct(ctx.handle, nt, C.c_void_p(pt), C.c_void_p(po), 0), "direct")
        got = np.frombuffer(ko.cpu().numpy()[off:off + 8 * width * nt].tobytes())
        assert np.array_equal(got.reshape(nt, width), want)
