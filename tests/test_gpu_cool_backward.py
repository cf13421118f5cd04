"""The cooling solve of rows outside the shortcuts' range (a step back in time,
a heating rate below zero): every sign from the FP64 residual, so the same
iterates as the plain bracket and bisection (the oracle's)."""
import numpy as np
import pytest

from oracle import oracle as O
from sph_2_b200 import Config, Context, cooling, ic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heat,sign", [(2e-26, -1.0), (-2e-26, 1.0), (-2e-26, -1.0), (0.0, -1.0)])
@pytest.mark.parametrize("tol", [1e-6, 1e-9])
def test_same_decisions_as_the_plain_iteration(heat, sign, tol):
    rng = np.random.default_rng(3)
    n = 20_000
    rho = 10.0 ** rng.uniform(-25.0, -17.0, n)
    u = cooling.u_of_T(10.0 ** rng.uniform(0.0, 9.0, n))
    dt = sign * 10.0 ** rng.uniform(5.0, 13.0, n)
    tab = ic.cooling_table(128, 1.0, 8.0)
    p = dict(cooling.DEFAULT, n_bins=128, gamma_heat=heat, tol=tol)
    with Context(Config(n_max=1024, precision="mixed")) as ctx:
        ctx.cooling_setup(p, tab)
        got, it = ctx.cool_solve(rho, u, dt)
    want, ito = O.do_cooling(tab, p["logT0"], p["logT1"], p["mu"], p["gamma"], p["XH"], heat, rho, u, dt,
                             tol=tol, max_iter=p["max_iter"])
    # where the residual's own rounding (a last place of log10 or exp10)
    # decides, the two may part by a bisection's tolerance
    same = (it == ito) & ((np.abs(got - want) <= 1e-12 * np.abs(want)) | (got == want))
    assert same.mean() > 0.999, same.mean()
