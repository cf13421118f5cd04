"""Position and velocity arrays with fewer than three columns raise, as NumPy
arrays and as CUDA tensors."""
import numpy as np
import pytest

from sph_2_b200 import libsx as X


class _OnDevice:
    """A stand-in for a CUDA tensor where there is no GPU."""
    is_cuda = True

    def __init__(self, a):
        self.a, self.shape, self.ndim = a, a.shape, a.ndim

    def __getitem__(self, k):
        return _OnDevice(self.a[k])

    def to(self, dtype):
        import torch
        return torch.as_tensor(self.a).to(dtype)


@pytest.mark.parametrize("wrap", [lambda a: a, _OnDevice])
@pytest.mark.parametrize("shapes", [[(9, 2)], [(9, 3), (9, 2)], [(9, 1)], [(9, 2), (9, 3)], [(9,)]])
def test_columns_refuse_narrow_arrays(wrap, shapes):
    with pytest.raises(IndexError):
        X._columns([wrap(np.ones(s)) for s in shapes], [wrap(np.ones(9))])


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["numpy", "cuda"])
def test_functions_refuse_narrow_arrays(kind):
    import torch
    T = (lambda a: a) if kind == "numpy" else (lambda a: torch.tensor(a, device="cuda"))
    rng = np.random.default_rng(0)
    n = 500
    pos, vel = rng.uniform(size=(n, 3)), rng.normal(size=(n, 3))
    one = T(np.ones(n))
    m, h = T(np.full(n, 1.0 / n)), T(np.full(n, 0.2))
    X.div_curlVel(T(pos), T(vel), one, m, h)
    for p, v in ((pos[:, :2], vel), (pos, vel[:, :2]), (pos[:, :1], vel[:, :1])):
        with pytest.raises(IndexError):
            X.div_curlVel(T(p), T(v), one, m, h)
    with pytest.raises(IndexError):
        X.getDensity(T(pos[:, :2]), m, h)
    with pytest.raises(IndexError):
        X.getAcc_g_smth_mimj_mpi(0, n, T(pos[:, :2]), m, 1.0, np.full(n, 0.01))
    # (n, 3, 1) is as good as (n, 3)
    assert np.array_equal(np.asarray(X.getDensity(T(pos[:, :, None]), m, h).tolist()),
                          np.asarray(X.getDensity(T(pos), m, h).tolist()))
