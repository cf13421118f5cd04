"""The neighbour-sum passes on both sides of each line of their lanes per
particle (32, 16, 8, the configured 4), phase by phase and through the fused
list and density pass, against the oracle's list sums."""
import numpy as np
import pytest

from oracle import oracle as O
from sph_2_b200 import Config, Context, ic

pytestmark = pytest.mark.gpu
SMS = 148


def _rel(a, b):
    return np.abs(np.asarray(a) - b).max() / (np.abs(b).max() + 1e-300)


# sums of about a hundred terms: 1e-10 in FP64, 3e-5 in FP32, ten times that
# for the differences of the velocity and pressure terms
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 3e-5)])
@pytest.mark.parametrize("n", [150, 21 * SMS, 21 * SMS + 1, 75 * SMS, 75 * SMS + 1, 300 * SMS, 300 * SMS + 1])
def test_pass_lanes(n, precision, tol):
    d = ic.evrard(n, seed=5)
    vel = np.random.default_rng(2).normal(scale=0.2, size=(n, 3))
    with Context(Config(n_max=n, precision=precision, theta=0.7, av_mode="gadget", balsara=True)) as ctx:
        for fused in (False, True):
            ctx.load(d["pos"], vel, d["m"], d["h"], d["u"])
            if fused:
                ctx.prologue()
                ctx.step(1)
            else:
                ctx.sort()
                ctx.build_tree()
                ctx.smoothing_h(); ctx.neighbours(); ctx.density(); ctx.divcurl(); ctx.forces(); ctx.dudt()
            x, y, z = ctx.get_pos(True).T.copy()
            v, m, h, u = ctx.get_vel(True), ctx.get("m", True), ctx.get("h", True), ctx.get("u", True)
            off, lst = O.neighbours(x, y, z, h)
            rho = O.density_list(x, y, z, m, h, off, lst)
            P, c = O.ref_pressure(rho, u, 5 / 3), O.ref_sound_speed(u, 5 / 3)
            dv, cv = O.divcurl_list(x, y, z, *v.T.copy(), rho, m, h, off, lst)
            acc, du, vs = O.force_list(x, y, z, *v.T.copy(), rho, P, c, h, m, dv, cv, 1.0, 2.0, 0.1, 1, 1,
                                       off, lst)
            assert _rel(ctx.get("rho", True), rho) < tol
            go, gl = ctx.neighbour_lists()
            assert np.array_equal(go, off) and np.array_equal(gl, lst)
            if fused:
                continue  # the step's last kick has moved v and u on since its passes
            assert _rel(ctx.get("divV", True), dv) < 10 * tol
            assert _rel(ctx.get("curlV", True), cv) < 10 * tol
            assert _rel(ctx.get_acc("sph", True), acc) < 10 * tol
            assert _rel(ctx.get("dudt", True), du) < 10 * tol
            assert _rel(ctx.get("vsig", True), vs) < 10 * tol


@pytest.mark.parametrize("heavy", [0.0, 0.3])
def test_marked_lists(heavy):
    """The lists that the rows cannot show to be complete: most of them before
    any list has told the rows how far to reach (searched by groups), a few
    after that (one by one)."""
    n = 20_000
    d = ic.evrard(n, seed=6)
    m = d["m"] * np.where(np.random.default_rng(4).random(n) < heavy, 12.0, 1.0)
    with Context(Config(n_max=n, precision="fp64", max_ngb=512)) as ctx:
        ctx.load(d["pos"], d["vel"], m, d["h"], d["u"])
        ctx.sort()
        ctx.build_tree()
        marked = []
        for _ in range(2):
            ctx.smoothing_h()
            ctx.neighbours()
            marked.append(int(ctx.debug_array("tree_search")[:n].sum()))
            x, y, z = ctx.get_pos(True).T.copy()
            off, lst = O.neighbours(x, y, z, ctx.get("h", True))
            assert np.diff(off).max() <= 512
            go, gl = ctx.neighbour_lists()
            assert np.array_equal(go, off) and np.array_equal(gl, lst)
        assert marked[0] > n // 8 and (marked[1] > n // 8) == (heavy > 0)
