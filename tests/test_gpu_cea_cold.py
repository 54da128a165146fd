"""Equilibrium of cells far below the transport fits' range: the fits' exponentials leave
the double range there, and the mixture viscosity is what plain divisions give (a term
over an infinite sum is 0)."""
import numpy as np
import pytest

from shared_cfd_b200 import cea

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [1, 300, 3000])
def test_cold_cells_match_restatement(gpu, orc, tiles):
    """Register and shared-memory launch shapes.  T converges to 1e-9 relative and ln mu is
    within 200 here, so mu agrees to 2e-7; 1e-6 is asked for."""
    d = cea.h2_air_data()
    with cea.Cea(d, lib=gpu) as g, cea.Cea(d, lib=orc) as o:
        rho, Y, e, T = cea.random_states(o.info(), 8, seed=3)
        states = [np.tile(np.tile(x, 5), tiles) for x in (rho, Y, e, T)]
        states[2] = states[2] * np.tile(np.repeat([-1.0, -0.9, -0.5, 0.5, 2.0], 8), tiles)
        rho, Y, e, T = states
        n = rho.size
        ref = o.solve(rho[:40], Y[:, :40], e[:40], T[:40], o.initial_n(40))
        got = g.solve(rho, Y, e, T, g.initial_n(n))
    assert ref["T"].min() < 20.0 and (ref["mu"] < 1e-80).any()
    for k in ("T", "kappa", "MWave", "mu"):
        for lo in (0, n - 40):
            np.testing.assert_allclose(got[k][lo:lo + 40], ref[k], rtol=1e-6, atol=0.0, equal_nan=True, err_msg=k)
    np.testing.assert_array_equal(got["iters"][:40], ref["iters"])
