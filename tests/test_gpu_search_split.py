"""The searches take 8, 4, 2 or 1 lanes per particle by the cloud's size; every
form gives the exact lists and the reference's own count and k-th neighbour
smoothing lengths, at the sizes where the form changes (per SM of a 148-SM
B200) and at the smallest ones."""
import numpy as np
import pytest

from oracle import oracle as O
from sph_2_b200 import Config, Context, ic

pytestmark = pytest.mark.gpu
SM = 148
SIZES = [1, 2, 33, 68 * SM, 68 * SM + 1, 140 * SM + 1, 300 * SM, 300 * SM + 1]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", SIZES)
def test_lists_and_newton_h(n, precision):
    d = ic.evrard(n, seed=n % 1000)
    h0 = d["h"] * np.random.default_rng(1).uniform(0.7, 1.4, n)
    with Context(Config(n_max=n, precision=precision)) as ctx:
        ctx.load(d["pos"], d["vel"], d["m"], h0, d["u"])
        ctx.sort()
        ctx.build_tree()
        # tree-search lists of the given h
        ctx.neighbours()
        x, y, z = ctx.get_pos(True).T.copy()
        oo, ol = O.neighbours(x, y, z, ctx.get("h", True))
        off, lst = ctx.neighbour_lists()
        assert np.array_equal(off, oo) and np.array_equal(lst, ol)
        if n < 100:
            return      # fewer particles than the target count: no root
        ctx.smoothing_h()
        h = ctx.get("h", True)
        st = ctx.status()
        assert st["h_noconv"] == 0 and st["stack_overflow"] == 0, st
        # two iterations that each stop within 1e-3 of the root
        ho, _, bad = O.newton_h(x, y, z, ctx.get("m", True), h)
        assert bad == 0 and np.max(np.abs(h / ho - 1)) < 2e-3
        # lists from the candidate rows
        ctx.neighbours()
        oo, ol = O.neighbours(x, y, z, h)
        off, lst = ctx.neighbour_lists()
        assert np.array_equal(off, oo) and np.array_equal(lst, ol)


@pytest.mark.parametrize("n", [60, 2_000, 68 * SM + 1, 140 * SM + 1, 300 * SM + 1])
def test_count_and_kth_h_equal_the_reference(n):
    d = ic.evrard(n, seed=n % 1000)
    h0 = d["h"] * np.random.default_rng(2).uniform(0.6, 1.5, n)
    pos = np.ascontiguousarray(d["pos"])
    a, b = n // 2 - min(n // 2, 100), n // 2 + min(n // 2, 100)
    with Context(Config(n_max=n, precision="fp64")) as ctx:
        ctx.load(pos, d["vel"], d["m"], h0, d["u"])
        ctx.sort()
        ctx.build_tree()
        ctx.smoothing_h_count()
        assert ctx.status(reset=True)["h_noconv"] == 0
        assert np.array_equal(ctx.get("h")[a:b], O.ref_h_smooth_fast(a, b, pos, h0))
        ctx.set("h", h0)
        ctx.smoothing_length_kth(50)
        assert ctx.status()["h_noconv"] == 0
        assert np.array_equal(ctx.get("h")[a:b], O.ref_smoothing_length(a, b, pos))


def test_count_h_with_equal_distances():
    """A lattice: many neighbours at the very same distance, where no trial
    radius separates the window's two distances from their equals."""
    g = np.arange(9.0)
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    n = len(pos)
    h0 = np.full(n, 1.3)
    with Context(Config(n_max=n, precision="fp64")) as ctx:
        ctx.load(pos, None, None, h0, None)
        ctx.sort()
        ctx.build_tree()
        ctx.smoothing_length_kth(50)
        assert np.array_equal(ctx.get("h"), O.ref_smoothing_length(0, n, pos))
        # the window is wider than any jump of a lattice point's counts
        ctx.set("h", h0)
        ctx.smoothing_h_count(n_target=50, n_tol=20, max_iter=400)
        assert ctx.status(reset=True)["h_noconv"] == 0
        h = ctx.get("h")
        cnt = (np.linalg.norm(pos[:, None] - pos[None], axis=2) < 2 * h[:, None]).sum(1)
        assert ((cnt >= 30) & (cnt <= 70)).all()
