"""Searches of clouds whose tree is as deep as the keys allow and whose radii take
in most of it: nothing may be left out of the rows when the stack fills up.  The
k-th neighbour and count smoothing lengths are then the reference's, bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O
from sph_2_b200 import Config, Context

pytestmark = pytest.mark.gpu


def _octaves(n):
    """as many particles in every octave of radius"""
    rng = np.random.default_rng(n)
    r = 10.0 ** rng.uniform(-6, 0, n)
    d = rng.normal(size=(n, 3))
    return r[:, None] * d / np.linalg.norm(d, axis=1)[:, None]


# a warp per particle, 8, 4, 2 and 1 lanes each
@pytest.mark.parametrize("n", [4000, 8000, 15_000, 30_000, 60_000])
@pytest.mark.parametrize("leaf", [1, 8])
def test_deep_trees(n, leaf):
    pos = _octaves(n)
    h0 = np.full(n, 0.05)
    a, b = n // 2, n // 2 + 100
    with Context(Config(n_max=n, precision="fp64", leaf_size=leaf, max_ngb=512)) as ctx:
        ctx.load(pos, None, None, h0, None)
        ctx.sort()
        ctx.build_tree()
        ctx.smoothing_h()
        assert ctx.status(reset=True)["stack_overflow"] == 0
        ctx.set("h", h0)
        ctx.smoothing_h_count(max_iter=2000)
        assert ctx.status(reset=True)["stack_overflow"] == 0
        ctx.set("h", h0)
        ctx.smoothing_length_kth(50)
        st = ctx.status(reset=True)
        assert st["stack_overflow"] == 0
        if st["h_noconv"] == 0:
            assert np.array_equal(ctx.get("h")[a:b], O.ref_smoothing_length(a, b, pos))
        # exact lists of radii that grow with the distance from the centre
        h = 0.05 * np.linalg.norm(pos, axis=1)
        ctx.set("h", h)
        ctx.neighbours()
        st = ctx.status()
        assert st["stack_overflow"] == 0 and st["ngb_overflow"] == 0
        x, y, z = ctx.get_pos(True).T.copy()
        oo, ol = O.neighbours(x, y, z, ctx.get("h", True))
        off, lst = ctx.neighbour_lists()
        assert np.array_equal(off, oo) and np.array_equal(lst, ol)
