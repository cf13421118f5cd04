"""The walk on both sides of the lines between 4, 2 and 1 warps per group, in
particles per SM: FP64 against the oracle's interaction counts and field, FP32
against the FP64 direct sum within the opening angle's error, for a flat cloud,
whose walks are short, and a sphere."""
import numpy as np
import pytest

from oracle import oracle as O
from sph_2_b200 import Config, Context, ic

pytestmark = pytest.mark.gpu
SMS = 148


def _loaded(flat, n, precision, **kw):
    pos = ic.evrard(n, seed=3)["pos"][np.random.default_rng(1).permutation(n)]
    if flat:
        pos = pos * [1.0, 1.0, 0.01]
    ctx = Context(Config(n_max=n, precision=precision, flags=16, **kw))
    ctx.load(pos, np.zeros((n, 3)), np.full(n, 1.0 / n), np.full(n, 0.01), np.ones(n))
    ctx.sort()
    ctx.build_tree()
    ctx.gravity()
    return ctx


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("n", [200 * SMS, 200 * SMS + 1])
def test_walk_fp64(n, flat):
    with _loaded(flat, n, "fp64", theta=0.6) as ctx:
        x, y, z = ctx.get_pos(True).T.copy()
        keys, _ = ctx.sort_info()
        acc, pot, nc, npart = O.bh_walk(x, y, z, ctx.get("m", True), ctx.get("h", True), np.sort(keys), 0.6, 1e-2,
                                        leaf_size=8, want_pot=True)
        cnt = ctx.counters()
        assert (cnt["cells"], cnt["particles"]) == (int(nc.sum()), int(npart.sum()))
        assert ctx.status()["stack_overflow"] == 0
        # thousands of terms of some 30 roundings, in another order
        assert np.abs(ctx.get_acc("grav", True) - acc).max() < 1e-12 * np.abs(acc).max()
        assert np.abs(ctx.get("pot", True) - pot).max() < 1e-12 * np.abs(pot).max()


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("n,local", [(150 * SMS, True), (150 * SMS + 1, True), (340 * SMS, True), (340 * SMS + 1, True),
                                     (150 * SMS + 1, False), (400 * SMS, False), (400 * SMS + 1, False)])
def test_walk_mixed(n, local, flat):
    kw = dict(theta=0.35, theta_local=0.28, theta_small=0.45, small_cell=128) if local else dict(theta=0.5)
    with _loaded(flat, n, "mixed", **kw) as ctx:
        tg = np.random.default_rng(0).choice(n, 2000, replace=False).astype(np.int32)
        ad, pd = ctx.gravity_direct(tg)
        a = ctx.get_acc("grav", True)[tg]
        assert ctx.status()["stack_overflow"] == 0
        # a quadrupole walk's truncation goes as theta^3, about 1e-3 of the field for
        # theta 0.5 and a third of that for 0.35
        err = np.sqrt(np.mean(np.sum((a - ad) ** 2, 1) / np.sum(ad * ad, 1)))
        assert err < 1e-3, err
        assert np.abs(ctx.get("pot", True)[tg] - pd).max() < 1e-3 * np.abs(pd).max()
