"""Loads in every form (host arrays below and above the staging size, device
arrays, null velocities, one cloud and several) and the drop-in functions on
NumPy arrays, CUDA tensors and mixtures give one and the same state."""
import ctypes as C

import numpy as np
import pytest

from sph_2_b200 import Config, Context, _lib as L, ic
from sph_2_b200 import libsx as X

pytestmark = pytest.mark.gpu
NAMES = ["x", "y", "z", "vx", "vy", "vz", "m", "h", "u"]


@pytest.mark.parametrize("n", [1, 3, 16384, 16385])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_load(n, precision):
    import torch
    rng = np.random.default_rng(n)
    a = {k: rng.normal(size=n) for k in NAMES}
    a["h"], a["m"] = np.abs(a["h"]) + 0.1, np.abs(a["m"])
    cloud = np.sort(rng.integers(0, 3, n)).astype(np.int32)
    dev = {k: torch.tensor(v, device="cuda") for k, v in a.items()}
    dcl = torch.tensor(cloud, device="cuda")
    torch.cuda.synchronize()
    lib = L.load()
    with Context(Config(n_max=n, n_cloud_max=3, precision=precision, dt_fixed=0.25)) as ctx:
        for host in (1, 0):
            for cl in (None, cloud):
                for null_v in (False, True):
                    src = [a[k].ctypes.data if host else dev[k].data_ptr() for k in NAMES]
                    if null_v:
                        src[3:6] = [None] * 3
                    pc = None if cl is None else (cl.ctypes.data if host else dcl.data_ptr())
                    ctx.set("x", np.full(ctx.n, 7.0)) if ctx.n else None
                    L.check(lib.sph_load(ctx.handle, n, C.c_void_p(pc), *map(C.c_void_p, src), host), "load")
                    assert ctx.n == n and ctx.n_clouds == (1 if cl is None else cloud.max() + 1)
                    for k in NAMES:
                        want = np.zeros(n) if null_v and k[0] == "v" else a[k]
                        assert np.array_equal(ctx.get(k), want), k
                    for k in ("ax_sph", "az_grav", "divV", "pot", "dudt_prev"):
                        assert not ctx.get(k).any()
                    assert np.array_equal(ctx.ids(), np.arange(n)) and (ctx.dt == 0.25).all()
                    assert np.array_equal(ctx.debug_array("p0_h"), a["h"])
                    assert np.allclose(ctx.debug_array("p1_m"), a["m"], rtol=1e-7)


def test_drop_in_functions_on_every_kind_of_array():
    import torch
    n = 1500
    rng = np.random.default_rng(4)
    d = ic.evrard(n, seed=2)
    pos, m, h = d["pos"], d["m"], d["h"] * 1.1
    v, rho = rng.normal(size=(n, 3)), rng.uniform(1, 2, n)
    P, c, dv, cv = (rng.uniform(0.5, 1.5, n) for _ in range(4))
    eps = rng.uniform(0.01, 0.02, n)
    T = lambda a: torch.tensor(a, device="cuda")
    f32 = lambda a: torch.tensor(a, device="cuda", dtype=torch.float32)
    # integers, float32, wider and strided position arrays are converted
    wide = np.concatenate([pos, rng.normal(size=(n, 2))], 1)
    want = X.getDensity(pos, m, h)
    assert np.array_equal(X.getDensity(wide, m, h), want)
    assert np.array_equal(X.getDensity(np.asfortranarray(pos), m, h), want)
    assert np.array_equal(X.getDensity(T(wide), T(m), T(h)).cpu().numpy(), want)
    assert np.array_equal(X.getDensity(T(wide)[:, :3], T(m), T(h)).cpu().numpy(), want)
    assert np.array_equal(X.getDensity(f32(pos), f32(m), f32(h)).cpu().numpy(),
                          X.getDensity(pos.astype(np.float32), m.astype(np.float32), h.astype(np.float32)))
    with pytest.raises(ValueError):
        X.getDensity(T(pos), m, T(h))
    a = X.getAcc_sph_shear(pos, v, rho, P, c, h, m, dv, cv, 1.0)
    b = X.getAcc_sph_shear(T(pos), T(v), T(rho), P, T(c), T(h), T(m), dv, T(cv), 1.0)   # some on the host
    assert b.is_cuda and b.is_contiguous() and np.array_equal(b.cpu().numpy(), a)
    g = X.getAcc_g_smth_mimj_mpi(0, n, pos, m, 1.5, eps)
    for e in (T(eps), eps, list(eps)):
        t = X.getAcc_g_smth_mimj_mpi(0, n, T(pos), T(m), 1.5, e)
        assert t.is_cuda and np.array_equal(t.cpu().numpy(), g)
    r = X.getAcc_g_smth_mimj_mpi(10, 700, pos, m, 1.5, eps)
    assert np.array_equal(X.getAcc_g_smth_mimj_mpi(10, 700, T(pos), T(m), 1.5, T(eps)).cpu().numpy(), r)
