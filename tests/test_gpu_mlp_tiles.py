"""The surrogate's gradient over row counts at the edges of its tiles (32 rows,
two resident blocks on each of 148 SMs) against the NumPy restatement with the
same BF16 rounding points, and a training step against Adam on that gradient."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from sph_2_b200 import Config, Context, _lib as L, cooling

pytestmark = pytest.mark.gpu
NORM = np.array([0, 0, 0, 1, 1, 1, 0, 1], np.float32)
PARTS = [(0, 192), (192, 256), (256, 4352), (4352, 4416), (4416, 4480), (4480, 4481)]


def rows(n, seed):
    rng = np.random.default_rng(seed)
    X = rng.normal(size=(n, 3)).astype(np.float32)
    return X, np.tanh(X @ np.array([0.5, -1.0, 0.3], np.float32)).astype(np.float32)


def params(seed):
    P = cooling.init_params(seed=seed)
    P[192:256] = np.linspace(-0.1, 0.1, 64)
    P[4352:4416] = np.linspace(0.1, -0.1, 64)
    return P


@pytest.mark.parametrize("n", [1, 31, 32, 33, 4096, 296 * 32, 296 * 32 + 1, 50_007])
def test_gradient(n):
    X, t = rows(n, n)
    P = params(5)
    with Context(Config(n_max=1024, precision="mixed")) as c:
        c.mlp_set(P, NORM)
        g, loss = c.mlp_grad(X, t)
        g2, loss2 = c.mlp_grad(X, t)
    assert np.array_equal(g, g2) and loss == loss2      # sums in block order
    go, lo = O.mlp_grad_bf16(X, t, *cooling.unpack(P))
    assert abs(loss - lo) < 1e-3 * lo
    for a, b in PARTS:
        # BF16 roundings of activations and errors: 2^-9 each, a few in a chain
        assert np.linalg.norm(g[a:b] - go[a:b]) < 2e-2 * np.linalg.norm(go[a:b]) + 1e-12, (a, b)


@pytest.mark.parametrize("n,batch", [(40, 64), (1000, 300), (4096, 4096)])
def test_training_steps_are_adam_on_the_gradient(n, batch):
    """Three steps over consecutive minibatches (wrapping) equal Adam applied to
    mlp_grad of each."""
    import torch
    X, t = rows(n, 3)
    P = params(6)
    nb, lr = max(1, n // batch), 1e-3
    with Context(Config(n_max=1024, precision="mixed")) as c:
        want, m, v = P.astype(np.float64), np.zeros(len(P)), np.zeros(len(P))
        for s in range(3):
            b = slice((s % nb) * batch, min((s % nb) * batch + batch, n))
            c.mlp_set(want.astype(np.float32), NORM)
            g, loss = c.mlp_grad(X[b], t[b])
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g.astype(np.float64) ** 2
            want = want - lr * (m / (1 - 0.9 ** (s + 1))) / (np.sqrt(v / (1 - 0.999 ** (s + 1))) + 1e-8)
        c.mlp_set(P, NORM)
        dX, dt = torch.as_tensor(X, device="cuda"), torch.as_tensor(t, device="cuda")
        last = C.c_float()
        torch.cuda.synchronize()
        L.check(L.load().sph_mlp_train(c.handle, n, C.c_void_p(dX.data_ptr()), C.c_void_p(dt.data_ptr()),
                                       batch, 3, C.c_float(lr), C.byref(last)), "sph_mlp_train", c.handle)
        got, _ = c.mlp_get()
    # where a weight's BF16 copy rounds the other way the next gradients part:
    # a few per cent of the step on a few weights
    step = np.linalg.norm(want - P)
    assert np.linalg.norm(got - want) < 2e-2 * step
    assert abs(last.value - loss) < 1e-2 * loss
