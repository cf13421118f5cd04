"""The cooling solve takes most signs of its residual from bounds, table edges
and an enclosed root; every row must end where the plain bracket and bisection
(the oracle's) ends, with the same count, for tables that rise, fall and
wiggle, states inside and far outside the table, and degenerate inputs."""
import numpy as np
import pytest

from oracle import oracle as O
from sph_2_b200 import Config, Context, cooling, ic

pytestmark = pytest.mark.gpu


def table(kind, nb):
    if kind == "default":
        return ic.cooling_table(nb, 1.0, 8.0)
    rng = np.random.default_rng(nb)
    slope = {"rise": rng.uniform(0.0, 6.0, nb), "fall": rng.uniform(-4.0, -0.1, nb),
             "wiggle": rng.uniform(-6.0, 6.0, nb), "flat": np.zeros(nb)}[kind]
    lam = np.concatenate([[0.0], np.cumsum(slope * 7.0 / nb)])
    return lam - lam.mean() - 23.5


def solve(tab, rho, u, dt, **kw):
    p = dict(cooling.DEFAULT, n_bins=len(tab) - 1, **kw)
    with Context(Config(n_max=1024, precision="mixed")) as ctx:
        ctx.cooling_setup(p, tab)
        got = ctx.cool_solve(rho, u, dt)
    want = O.do_cooling(tab, p["logT0"], p["logT1"], p["mu"], p["gamma"], p["XH"], p["gamma_heat"],
                        rho, u, dt, tol=p["tol"], max_iter=p["max_iter"])
    return got, want


def check(got, want):
    u, it = got
    uo, ito = want
    # the same decisions; where the residual's own rounding (a last place of
    # log10 or exp10) decides, the two may part by a bisection's tolerance
    same = (it == ito) & (np.abs(u - uo) <= 1e-12 * np.abs(uo))
    assert same.mean() > 0.999, same.mean()


@pytest.mark.parametrize("kind,nb", [("default", 128), ("rise", 128), ("fall", 64), ("wiggle", 96),
                                     ("wiggle", 4096), ("flat", 8), ("rise", 1), ("fall", 1)])
@pytest.mark.parametrize("heat", [2e-26, 0.0, 1e-22])
def test_same_decisions_as_the_plain_iteration(kind, nb, heat):
    rng = np.random.default_rng(nb)
    n = 20_000
    rho = 10.0 ** rng.uniform(-25.0, -17.0, n)
    u = cooling.u_of_T(10.0 ** rng.uniform(-1.0, 9.5, n))      # below and above the table
    dt = 10.0 ** rng.uniform(5.0, 15.0, n)
    check(*solve(table(kind, nb), rho, u, dt, gamma_heat=heat))


@pytest.mark.parametrize("tol,max_iter", [(1e-3, 200), (1e-9, 200), (1e-6, 5), (2.0, 200)])
def test_stopping_rules(tol, max_iter):
    rho, u, dt = cooling.sample_states(5_001, seed=8)
    check(*solve(table("default", 128), rho, u, dt, tol=tol, max_iter=max_iter))


def test_degenerate_rows():
    """No step, no density, zero and negative energies, magnitudes outside the
    FP32 range: the plain iteration's answer, whatever it is."""
    rho = np.array([1e-21, 1e-21, 1e-60, 1e-21, 1e-21, 1e-21, 1e-21, 1e10])
    u = np.array([1e11, 1e11, 1e11, 1e-30, 1e40, 1e11, 1e11, 1e11])
    dt = np.array([0.0, 1e300, 1e12, 1e12, 1e12, 1e-300, -1e10, 1e12])
    (ug, ig), (uo, io) = solve(table("default", 128), rho, u, dt)
    assert np.array_equal(ig, io)
    assert np.allclose(ug, uo, rtol=1e-9, atol=0.0, equal_nan=True)
