"""The climb above the groups (512 groups to a block in shared memory, the nodes
that reach beyond a block through device memory): every node record, h_max and
opening radius bit for bit with the oracle, after a build, after h changed
(the h_max climb of a tree search) and after steps, for clouds within one
block, across several, and for several clouds."""
import numpy as np
import pytest

from oracle import oracle as O
from sph_2_b200 import Config, Context, ic

pytestmark = pytest.mark.gpu


def check(ctx, cloud, theta):
    t = ctx.tree()
    x, y, z = ctx.get_pos(True).T.copy()
    m, h = ctx.get("m", True), ctx.get("h", True)
    cl = None if cloud is None else cloud[ctx.ids()]
    node, hmax = O.tree_moments(t["child"], t["first"], t["last"], x, y, z, m, h, cl)
    n = len(x)
    assert np.array_equal(t["node"].view(np.uint64), node.view(np.uint64))
    assert np.array_equal(t["hmax"], hmax)
    assert np.array_equal(t["open_r2"][: n - 1], O.open_r2(node, theta)[: n - 1])


@pytest.mark.parametrize("n,clouds", [(2, 1), (33, 1), (65, 2), (9_000, 1), (12_000, 1), (60_007, 1),
                                      (30_000, 7), (250_001, 1)])
def test_records(n, clouds):
    rng = np.random.default_rng(n)
    d = ic.evrard(n, seed=n % 97)
    cloud = np.sort(rng.integers(0, clouds, n)).astype(np.int32) if clouds > 1 else None
    theta = 0.6
    with Context(Config(n_max=n, n_cloud_max=clouds, precision="fp64", theta=theta)) as ctx:
        ctx.load(d["pos"], d["vel"], d["m"] * rng.uniform(0.5, 1.5, n), d["h"], d["u"], cloud=cloud)
        ctx.sort()
        ctx.build_tree()
        check(ctx, cloud, theta)
        ctx.set("h", d["h"] * rng.uniform(0.5, 1.5, n))
        ctx.neighbours()                     # refits h_max
        t = ctx.tree()
        h = ctx.get("h", True)
        first, last = t["first"], t["last"]
        some = rng.integers(0, 2 * n - 1, 300)
        assert all(t["hmax"][k] == h[first[k]:last[k] + 1].max() for k in some)
        ctx.build_tree()                     # the arrival counters are clear again
        check(ctx, cloud, theta)
