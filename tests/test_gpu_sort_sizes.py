"""The radix sort at the edges of its tiles and of its forms (512, 1024 and 2048
keys to a tile): keys and the stable permutation bit for bit, random and with
every key equal, one cloud and several."""
import numpy as np
import pytest

from oracle import oracle as O
from sph_2_b200 import Config, Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 511, 512, 513, 50_000, 50_001, 130_000, 130_001, 700_003])
@pytest.mark.parametrize("kind", ["random", "equal", "clouds"])
def test_sort(n, kind):
    rng = np.random.default_rng(n)
    pos = rng.normal(size=(n, 3)) if kind != "equal" else np.full((n, 3), 0.25)
    if kind == "random" and n > 20:
        pos[5:15] = pos[3]                       # ties keep their order
    cloud = None
    if kind == "clouds":
        cloud = np.sort(rng.integers(0, 5, n)).astype(np.int32)
        cloud[-1] = 4
    with Context(Config(n_max=n, n_cloud_max=5, precision="mixed")) as ctx:
        ctx.load(pos, cloud=cloud)
        for _ in range(2):                        # the second from sorted input
            p = ctx.get_pos(True)
            cl = None if cloud is None else cloud[ctx.ids()]
            ctx.sort()
            keys, perm = ctx.sort_info()
            bits = None if cloud is None else O.morton_bits(5)
            want = O.morton_keys(*(p[:, k].copy() for k in range(3)), cl, bits) if cl is not None \
                else O.morton_keys(*(p[:, k].copy() for k in range(3)))
            assert np.array_equal(keys, want)
            assert np.array_equal(perm, O.sort_perm(want))
        assert ctx.status()["wait_timeout"] == 0
