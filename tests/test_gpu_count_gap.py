"""The count iteration of a particle with a dense clump just outside its window:
a search widened past the clump overflows its row, and the iteration has to go
on with the narrow steps that end inside the window."""
import numpy as np
import pytest

from oracle import oracle as O
from sph_2_b200 import Config, Context

pytestmark = pytest.mark.gpu


def _ball(rng, n, r0, r1):
    d = rng.normal(size=(n, 3))
    r = rng.uniform(r0 ** 3, r1 ** 3, n) ** (1 / 3)
    return r[:, None] * d / np.linalg.norm(d, axis=1)[:, None]


def _around(rng, clump, at):
    """A particle at the origin with 30 others within 1, 30 from 1.02 to 1.12
    and `clump` in a ball at distance `at`."""
    axis = rng.normal(size=3)
    return np.concatenate([np.zeros((1, 3)), _ball(rng, 30, 0.0, 1.0), _ball(rng, 30, 1.02, 1.12),
                           _ball(rng, clump, 0.0, 0.02) + at * axis / np.linalg.norm(axis)])


@pytest.mark.parametrize("max_ngb,clump,at", [(512, 700, 1.2), (512, 2000, 1.16), (128, 300, 1.2), (60, 40, 1.2)])
@pytest.mark.parametrize("copies", [1, 60, 400])
def test_clump_outside_the_window(max_ngb, clump, at, copies):
    rng = np.random.default_rng(clump)
    pos = np.concatenate([_around(rng, clump, at) + 20.0 * np.array([k % 8, k // 8 % 8, k // 64])
                          for k in range(copies)])
    each = len(pos) // copies
    one = np.concatenate([np.full(61, 0.465), np.full(each - 61, 0.005)])
    h0 = np.tile(one, copies)
    n = len(pos)
    centre = np.arange(copies) * each
    with Context(Config(n_max=n, precision="fp64", max_ngb=max_ngb)) as ctx:
        ctx.load(pos, None, None, h0, None)
        ctx.sort()
        ctx.build_tree()
        ctx.smoothing_h_count(max_iter=2000)
        h = ctx.get("h")
        for i in centre[:: max(1, copies // 4)]:
            assert h[i] == O.ref_h_smooth_fast(i, i + 1, pos, h0, 2000)[0]
