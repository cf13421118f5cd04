"""The block walk's stack at the settings that fill it most: buckets of one
particle and small opening angles.  Nothing may be left out of the sums: the
oracle's interaction counts, and its field."""
import numpy as np
import pytest

from oracle import oracle as O
from sph_2_b200 import Config, Context, ic

pytestmark = pytest.mark.gpu


def _positions(kind, n):
    if kind == "evrard":
        return ic.evrard(n, seed=3)["pos"]
    rng = np.random.default_rng(1)
    if kind == "core":      # three quarters of the particles within a hundredth of the radius
        k = n // 4
        r = np.concatenate([0.01 * rng.uniform(0, 1, n - k) ** (1 / 3), rng.uniform(0, 1, k) ** (1 / 3)])
    else:                   # as many in every octave of radius: past the stack's reserve
        r = 10.0 ** rng.uniform(-6.0, 0.0, n)
    d = rng.normal(size=(n, 3))
    return r[:, None] * d / np.linalg.norm(d, axis=1)[:, None]


# 4 warps a group up to 200 particles per SM (29,600), 2 above
@pytest.mark.parametrize("kind,n,theta", [("evrard", 29_000, 0.05), ("evrard", 100_000, 0.05),
                                          ("evrard", 110_000, 0.1), ("core", 29_000, 0.05),
                                          ("core", 112_000, 0.1), ("octaves", 29_000, 0.05),
                                          ("octaves", 29_000, 0.1), ("octaves", 112_000, 0.1)])
def test_every_node_is_summed(kind, n, theta):
    pos, leaf = _positions(kind, n), 1
    with Context(Config(n_max=n, precision="fp64", theta=theta, leaf_size=leaf)) as ctx:
        ctx.load(pos, np.zeros((n, 3)), np.full(n, 1.0 / n), np.full(n, 0.01), np.ones(n))
        ctx.sort()
        ctx.build_tree()
        ctx.gravity()
        assert ctx.status()["stack_overflow"] == 0
        x, y, z = (ctx.get_pos(True)[:, k].copy() for k in range(3))
        keys, _ = ctx.sort_info()
        acc, _, nc, npart = O.bh_walk(x, y, z, ctx.get("m", True), ctx.get("h", True), np.sort(keys),
                                      theta, 1e-2, leaf_size=leaf)
        cnt = ctx.counters()
        assert (cnt["cells"], cnt["particles"]) == (int(nc.sum()), int(npart.sum()))
        # up to a hundred thousand terms of some 30 roundings, in another order
        assert np.abs(ctx.get_acc("grav", True) - acc).max() < 1e-11 * np.abs(acc).max()
