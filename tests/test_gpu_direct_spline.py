"""The spline-softened direct sum at the edges of its split (32 targets and
1024 sources per cluster) against the oracle's restatement of the reference,
for all targets, a few of them, and row ranges."""
import numpy as np
import pytest

from oracle import oracle as O
from sph_2_b200 import Config, Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1023, 1025, 2500])
def test_direct_spline(n):
    rng = np.random.default_rng(n)
    pos = rng.normal(size=(n, 3))
    if n > 2:
        pos[2] = pos[0]                         # coincident: no force between them
    m = rng.uniform(0.5, 1.5, n) / n
    eps = rng.uniform(0.01, 0.5, n)             # many pairs inside the support
    want = O.ref_getAcc_g_smth_mimj(0, n, pos + (1e-300 if n > 2 else 0.0), m, 1.3, eps) if n < 3 else None
    if n >= 3:
        # the reference divides by the coincident pair's distance: sum it apart
        dx = pos[None] - pos[:, None]
        r = np.sqrt((dx ** 2).sum(2))
        e = 0.5 * (eps[None] + eps[:, None])
        with np.errstate(all="ignore"):
            q = r / e
            f = np.where(q <= 1, (4 / 3 - 1.2 * q ** 2 + 0.5 * q ** 3) / e ** 3,
                         np.where(q <= 2, -1 / 15 + 8 / 3 * q ** 3 - 3 * q ** 4 + 1.2 * q ** 5 - q ** 6 / 6,
                                  1.0) / r ** 3)
        f[r == 0.0] = 0.0
        want = 1.3 * (f[..., None] * m[None, :, None] * dx).sum(1)
    scale = max(np.abs(want).max(), 1e-30)
    with Context(Config(n_max=max(n, 64), precision="fp64", G=1.3)) as ctx:
        ctx.load(pos, None, m, np.full(n, 0.1), None)
        ctx.sort()
        ctx.build_tree()
        ids = ctx.ids()
        slot = np.empty(n, np.int32)
        slot[ids] = np.arange(n, dtype=np.int32)
        got = ctx.gravity_direct_spline(eps, slot)
        # some 25 roundings a pair, summed over n of them in 32 parts
        assert np.abs(got - want).max() < 1e-12 * scale
        few = slot[rng.integers(0, n, min(n, 37))]
        assert np.array_equal(ctx.gravity_direct_spline(eps, few), got[ids[few]])
        # the partial fields of a partition of the rows add up
        cuts = [0, n // 3, n // 2, n]
        parts = [ctx.gravity_direct_spline_rows(eps, a, b) for a, b in zip(cuts[:-1], cuts[1:])]
        assert np.abs(sum(parts) - want).max() < 1e-12 * scale
