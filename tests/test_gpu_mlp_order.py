"""The launches of training steps overlap in programmatic stream order: a step's
gradient must see the weights of the update before it, and an update all of the
gradient's slots.  Many steps in one call give the weights, to the bit, of one step
a call with the device idle between them."""
import ctypes as C

import numpy as np
import pytest

from sph_2_b200 import Config, Context, _lib as L, cooling

pytestmark = pytest.mark.gpu
NORM = np.array([0, 0, 0, 1, 1, 1, 0, 1], np.float32)


@pytest.mark.parametrize("n", [31, 4096, 296 * 32 + 5])
def test_steps_in_a_row(n):
    import torch
    rng = np.random.default_rng(n)
    X = torch.tensor(rng.normal(size=(n, 3)).astype(np.float32), device="cuda")
    t = torch.tanh(X @ torch.tensor([0.5, -1.0, 0.3], device="cuda"))
    P = cooling.init_params(seed=3)
    torch.cuda.synchronize()

    def train(c, steps):
        L.check(L.load().sph_mlp_train(c.handle, n, C.c_void_p(X.data_ptr()), C.c_void_p(t.data_ptr()), n,
                                       steps, C.c_float(1e-2), C.byref(C.c_float())), "train", c.handle)

    with Context(Config(n_max=1024, precision="mixed")) as a, Context(Config(n_max=1024, precision="mixed")) as b:
        a.mlp_set(P, NORM)
        b.mlp_set(P, NORM)
        train(a, 200)
        for _ in range(200):
            train(b, 1)
            torch.cuda.synchronize()
        pa, pb = a.mlp_get()[0], b.mlp_get()[0]
    assert np.isfinite(pa).all() and not np.array_equal(pa, P)
    assert np.array_equal(pa, pb)
