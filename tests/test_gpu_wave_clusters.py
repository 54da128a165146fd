"""The sweeps on clusters of 8 CTAs (tasks of 128 rows), which a device part without room
for 16 takes: the same bits as on 16, over one to three times as many tasks, and the
tuning report says which ran, and why where neither did."""
import numpy as np
import pytest

from shared_cfd_b200 import abi, cases
from shared_cfd_b200.solver import Solver

from helpers import run_case
from test_gpu_wave_edges import one_block

pytestmark = pytest.mark.gpu


def sweep_report(case, lib):
    s = Solver(case, lib=lib)
    try:
        return s.tuning()["sweep"]
    finally:
        s.close()


@pytest.mark.parametrize("nj", [128, 129, 300])
@pytest.mark.parametrize("kind", ["ideal", "dual", "species9"])
def test_clusters_of_eight_match_sixteen(gpu, monkeypatch, kind, nj):
    monkeypatch.delenv("SCFD_SWEEP_CLUSTER", raising=False)
    if kind == "species9":
        base = cases.reacting_step(scale=1.0 / 64.0, inner=3)
    else:
        scheme = abi.SCHEME_DUAL if kind == "dual" else abi.SCHEME_LUSGS
        base = cases.forward_step(0, n=4, scheme=scheme, viscous=1,
                                  dt_mode=abi.DT_GLOBAL if kind == "dual" else abi.DT_LOCAL)
    case = one_block(base, 141, nj, seed=nj)
    if kind == "dual":
        case.desc.num_internal_loop, case.desc.cfl_tau, case.desc.res_rate_err = 4, 5.0, 1e300
    for precision in (abi.PREC_FP64, abi.PREC_MIXED):
        case.desc.precision = precision
        wide, a = sweep_report(case, gpu), run_case(case, gpu, 2)
        with monkeypatch.context() as m:
            m.setenv("SCFD_SWEEP_CLUSTER", "8")
            narrow, b = sweep_report(case, gpu), run_case(case, gpu, 2)
        assert wide["kind"] == narrow["kind"] == "cluster wavefront"
        assert (wide["cluster_ctas"], wide["tasks"]) == (16, -(-nj // 256))
        assert (narrow["cluster_ctas"], narrow["tasks"]) == (8, -(-nj // 128))
        np.testing.assert_array_equal(a["q"], b["q"])


def test_generic_sweeps_say_why(gpu, monkeypatch):
    monkeypatch.setenv("SCFD_SWEEP_LEGACY", "1")
    assert sweep_report(cases.flat_plate(24, 16), gpu) == {"kind": "generic", "reason": "SCFD_SWEEP_LEGACY"}
