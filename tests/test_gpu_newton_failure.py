"""A cell whose temperature iteration does not converge: the step reports E_TNEWTON and the
cell keeps the thermodynamic properties it had, run for run the same."""
import numpy as np
import pytest

from shared_cfd_b200 import abi, cases
from shared_cfd_b200.solver import Solver, SolverError

pytestmark = pytest.mark.gpu


def test_failed_cell_keeps_its_properties(gpu):
    case = cases.reacting_step(scale=1.0 / 64.0, inner=2)
    q = case.q.copy()
    q[0, 3, 4, -1] *= -1.0  # no temperature has this energy
    nY = case.nY
    for _ in range(2):
        s = Solver(case, lib=gpu)
        try:
            s.upload(q=q)
            with pytest.raises(SolverError) as e:
                s.prepare(1)
            _, w, vhi, _ = s.download()
        finally:
            s.close()
        assert e.value.code == abi.E_TNEWTON
        np.testing.assert_array_equal(vhi[0, 3, 4], case.vhi[0, 3, 4])
        # p, gamma, the total enthalpy, R and mu
        keep = [3, nY + 4, nY + 5, nY + 6, nY + 7]
        np.testing.assert_array_equal(w[0, 3, 4][keep], case.w[0, 3, 4][keep])
        assert np.isfinite(w).all() and np.isfinite(vhi).all()
