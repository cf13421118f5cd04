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


def _small_steps(d, h, cap, K, lo, hi, frac, rounds, max_iter):
    """The iteration over rows of at most K candidates, widened by 8 % past h at a
    time: h where it ends inside the window, None where the rounds run out.
    d: the particle's sorted distances, cap: half the first radius."""
    it = 0
    for _ in range(rounds):
        c = np.searchsorted(d, 2.0 * cap, "right")
        if c > K:
            cap *= max(0.5, np.cbrt(0.5 * K / c))
            continue
        lim = cap * (1.0 - 1e-12)
        n = lambda r: np.searchsorted(d[:c], r, "left")
        if h > lim:
            if n(2.0 * lim) <= hi:
                cap = h * 1.08
                continue
            while h > lim:
                h -= frac * h
                it += 1
        while h <= lim and it <= max_iter:
            if n(2.0 * h) > hi:
                h -= frac * h
            elif n(2.0 * h) < lo:
                h += frac * h
            else:
                return h
            it += 1
        cap = h * 1.08
    return None


@pytest.mark.parametrize("n,K,target,tol", [(6000, 64, 56, 4), (6000, 64, 58, 1), (30_000, 64, 50, 5), (3000, 128, 120, 6)])
def test_rows_barely_above_the_window(n, K, target, tol):
    """Where small steps of the radius end inside the window, so does the
    iteration, with the same h."""
    rng = np.random.default_rng(n + K)
    pos = rng.uniform(-1.0, 1.0, size=(n, 3))
    h0 = (target / n) ** (1 / 3) * rng.uniform(0.3, 1.2, n)
    with Context(Config(n_max=n, precision="fp64", max_ngb=K)) as ctx:
        ctx.load(pos, None, None, h0, None)
        ctx.sort()
        ctx.build_tree()
        ctx.smoothing_h_count(n_target=target, n_tol=tol, max_iter=1500)
        h = ctx.get("h")
    ended = 0
    for i in rng.integers(0, n, 400):
        dx, dy, dz = (pos - pos[i]).T
        d = np.sort(np.sqrt(dx * dx + dy * dy + dz * dz))
        want = _small_steps(d, h0[i], 1.08 * h0[i], K, target - tol, target + tol, 0.003, 16, 1500)
        if want is not None:
            ended += 1
            assert h[i] == want
    assert ended
