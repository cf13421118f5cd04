"""Sort tiles that do not wait for one another but count the keys before them,
which is what a tile does whose wait has passed its limit: the same keys and
permutation, bit for bit, at the edges of the sort's three forms."""
import numpy as np
import pytest

from oracle import oracle as O
from sph_2_b200 import Config, Context, _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 512, 513, 50_000, 50_001, 130_000, 130_001, 300_003])
@pytest.mark.parametrize("kind", ["random", "equal"])
def test_counting_tiles(n, kind):
    rng = np.random.default_rng(n)
    pos = rng.normal(size=(n, 3)) if kind == "random" else np.full((n, 3), 0.25)
    if kind == "random" and n > 20:
        pos[5:15] = pos[3]                       # ties keep their order
    with Context(Config(n_max=n, precision="mixed")) as ctx:
        ctx.load(pos)
        ctx.set_params(flags=L.FLAG_SORT_COUNT)
        want = O.morton_keys(*(pos[:, k].copy() for k in range(3)))
        ctx.sort()
        keys, perm = ctx.sort_info()
        assert np.array_equal(keys, want)
        assert np.array_equal(perm, O.sort_perm(want))
        assert np.array_equal(np.sort(ctx.ids()), np.arange(n))
        assert ctx.status()["wait_timeout"] == 0
