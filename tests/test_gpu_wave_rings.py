"""The sweeps' rings beyond their first turn (k_wave.cu): the hand-off ring holds 32 chunks
of 4 columns, so planes of more than 128 columns reuse its places (and wait for their
release), inside a task and, above 256 rows, between two tasks; a cluster of a later task
starts with the counts that the one before left.  Bounds as in test_gpu_wave_edges.py."""
import pytest

from shared_cfd_b200 import abi, cases

from helpers import rel_l2, run_case
from test_gpu_wave_edges import one_block

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj", [(127, 9), (133, 257), (261, 265)])
@pytest.mark.parametrize("kind", ["ideal", "species9"])
def test_wrapped_rings(gpu, orc, kind, ni, nj):
    if kind == "ideal":
        base = cases.forward_step(0, n=4, scheme=abi.SCHEME_LUSGS, dt_mode=abi.DT_LOCAL, viscous=1)
        base.desc.cfl = 2.0
    else:
        base = cases.reacting_step(scale=1.0 / 64.0, inner=3)
        base.desc.scheme = abi.SCHEME_LUSGS
    case = one_block(base, ni, nj, seed=ni * 1000 + nj)
    ref = run_case(case, orc, 2)
    assert ref["stats"].status == 0
    for precision, bound in ((abi.PREC_FP64, 1e-10), (abi.PREC_MIXED, 1e-4)):
        case.desc.precision = precision
        got = run_case(case, gpu, 2)
        assert got["stats"].status == 0
        assert rel_l2(case, got["q"], ref["q"]) <= bound


@pytest.mark.parametrize("ni,nj", [(134, 67), (150, 267)])
@pytest.mark.parametrize("scheme", [abi.SCHEME_DUAL, abi.SCHEME_PRECON, abi.SCHEME_PRECON_LUSGS])
def test_wrapped_rings_preconditioned(gpu, orc, scheme, ni, nj):
    local = scheme != abi.SCHEME_DUAL
    base = cases.forward_step(0, n=4, scheme=scheme, viscous=1, dt_mode=abi.DT_LOCAL if local else abi.DT_GLOBAL)
    case = one_block(base, ni, nj, seed=ni * 1000 + nj)
    case.desc.num_internal_loop = 4
    case.desc.cfl_tau = 5.0
    case.desc.cfl = 0.8 if local else case.desc.cfl
    case.desc.res_rate_err = 1e300
    ref = run_case(case, orc, 2)
    for precision, bound in ((abi.PREC_FP64, 1e-10), (abi.PREC_MIXED, 1e-4)):
        case.desc.precision = precision
        got = run_case(case, gpu, 2)
        assert rel_l2(case, got["q"], ref["q"]) <= bound
