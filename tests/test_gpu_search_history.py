"""The h iteration's choice between a warp per particle and eight lanes follows
the last iteration's longest search, which is part of neither a loaded state nor
a restart file: a load and a restart, read or written, begin it anew, so that
they repeat bit for bit whatever the context ran before."""
import numpy as np
import pytest

from sph_2_b200 import Config, Context

pytestmark = pytest.mark.gpu
SMS = 148
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "u", "h", "rho", "dudt", "ax_grav", "ax_sph")


def _cfg(n, precision, **kw):
    return Config(n_max=n, precision=precision, max_ngb=256, theta=0.5, **kw)


def _core(n, seed):
    """A dense core in a thin halo: rim particles whose searches of eight lanes
    reach the core, which is what the choice is for."""
    rng = np.random.default_rng(seed)
    k = n // 8
    r = np.concatenate([0.05 * rng.uniform(0, 1, n - k) ** (1 / 3), rng.uniform(0.1, 1.0, k)])
    d = rng.normal(size=(n, 3))
    pos = r[:, None] * d / np.linalg.norm(d, axis=1)[:, None]
    # near the radius of 64 neighbours: the core's, and 0.1 to 0.5 in the halo
    h = np.where(r < 0.06, 0.5 * 0.05 * (64 / n) ** (1 / 3), 0.5 * r)
    return pos, 0.1 * rng.normal(size=(n, 3)), np.full(n, 1.0 / n), h, np.full(n, 0.05)


def _uniform(n, seed):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(-1.0, 1.0, size=(n, 3))
    return pos, np.zeros((n, 3)), np.full(n, 1.0 / n), np.full(n, (64 / n) ** (1 / 3)), np.full(n, 0.05)


def _same(a, b):
    for f in FIELDS:
        assert np.array_equal(a.get(f), b.get(f)), f


# the choice is there from 34 to 68 particles per SM
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [34 * SMS + 1, 8000, 68 * SMS])
def test_restart_of_a_dense_core(tmp_path, n, precision):
    path = tmp_path / "restart.bin"
    kw = dict(dt_fixed=1e-4)
    with Context(_cfg(n, precision, **kw)) as a, Context(_cfg(n, precision, **kw)) as b, \
            Context(_cfg(n, precision, **kw)) as used:
        a.load(*_core(n, 3))
        a.prologue()
        a.step(4)
        a.write_restart(path)
        used.load(*_uniform(n, 4))
        used.prologue()
        used.step(2)
        for c in (b, used):
            c.read_restart(path)
        for c in (a, b, used):
            c.step(3)
            c.sync()
        _same(a, b)
        _same(a, used)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [34 * SMS + 1, 8000, 68 * SMS])
def test_load_into_a_used_context(n, precision):
    def run(ctx):
        ctx.load(*_core(n, 5))
        ctx.sort()
        ctx.build_tree()
        ctx.smoothing_h()
        return ctx.get("h")
    with Context(_cfg(n, precision)) as a:
        first = run(a)
        assert np.array_equal(run(a), first)
        a.load(*_uniform(n, 6))
        a.sort()
        a.build_tree()
        a.smoothing_h()
        assert np.array_equal(run(a), first)
