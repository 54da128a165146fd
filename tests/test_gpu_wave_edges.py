"""The cluster-wavefront sweeps (k_wave.cu) at the sizes where their schedule can go
wrong: planes of one column or row fewer and more than a strip (8 rows), a record
slot (8 steps), a hand-off chunk (4 columns), a CTA (2 strips) and a task (256 rows),
against the CPU restatement.  FP64 within 1e-10 relative L2 of q as elsewhere; the
mixed path's sweeps carry FP32 rounding (6e-8 per value) through a few dozen
operations per cell, so q stays within 1e-4 of the restatement."""
import numpy as np
import pytest

from shared_cfd_b200 import abi, cases
from shared_cfd_b200.solver import Case

from helpers import rel_l2, run_case

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (3, 7), (4, 8), (5, 9), (7, 15), (8, 17), (9, 33), (25, 255), (6, 256), (33, 257), (17, 520)]


def one_block(base, ni, nj, seed):
    """A rectangular plane with the base case's descriptor, tables and first cell's
    state, zero-gradient sides, disturbed."""
    xs = np.linspace(0.0, 0.01 * ni / 64, ni + 1)
    rs = np.linspace(0.01, 0.01 + 0.01 * nj / 64, nj + 1)
    c = Case([cases.rect_plane(xs, rs)], abi.Desc.from_buffer_copy(base.desc), chem=base.chem)
    cases.fill_all(c, 0, base.q[0, 3, 3], base.w[0, 3, 3], base.vhi[0, 3, 3])
    c.bcs = cases.all_sides([(ni, nj)], abi.BC_EXTRAP)
    return cases.perturb(c, seed=seed, amp=0.01)


@pytest.mark.parametrize("ni,nj", SIZES)
@pytest.mark.parametrize("kind", ["ideal", "species9"])
def test_sweep_edges(gpu, orc, kind, ni, nj):
    if kind == "ideal":
        base = cases.forward_step(0, n=4, scheme=abi.SCHEME_LUSGS, dt_mode=abi.DT_LOCAL, viscous=1)
        base.desc.cfl = 2.0
    else:
        base = cases.reacting_step(scale=1.0 / 64.0, inner=3)
    case = one_block(base, ni, nj, seed=ni * 1000 + nj)
    ref = run_case(case, orc, 2)
    got = run_case(case, gpu, 2)
    assert got["stats"].status == 0 and ref["stats"].status == 0
    assert rel_l2(case, got["q"], ref["q"]) <= 1e-10
    if kind == "species9":
        # NR's limiter scales the whole update by a factor that a trace species with an
        # FP32-rounded Dq may set (2e-4 of q here, whatever the sweep): the mixed sweep
        # is checked on the LU-SGS step, which has no limiter
        case.desc.scheme = abi.SCHEME_LUSGS
        ref = run_case(case, orc, 2)
    case.desc.precision = abi.PREC_MIXED
    mixed = run_case(case, gpu, 2)
    assert mixed["stats"].status == 0 and ref["stats"].status == 0
    assert rel_l2(case, mixed["q"], ref["q"]) <= 1e-4


@pytest.mark.parametrize("n", [3, 8, 9, 33])
@pytest.mark.parametrize("scheme", [abi.SCHEME_DUAL, abi.SCHEME_PRECON, abi.SCHEME_PRECON_LUSGS])
def test_preconditioned_sweep_edges(gpu, orc, scheme, n):
    local = scheme != abi.SCHEME_DUAL
    case = cases.forward_step(0, n=n, scheme=scheme, viscous=1, dt_mode=abi.DT_LOCAL if local else abi.DT_GLOBAL)
    case = cases.perturb(case, seed=n)
    case.desc.num_internal_loop = 6
    case.desc.cfl_tau = 5.0
    case.desc.cfl = 0.8 if local else case.desc.cfl
    case.desc.res_rate_err = 1e300
    ref = run_case(case, orc, 2)
    got = run_case(case, gpu, 2)
    assert rel_l2(case, got["q"], ref["q"]) <= 1e-10
    case.desc.precision = abi.PREC_MIXED
    assert rel_l2(case, run_case(case, gpu, 2)["q"], ref["q"]) <= 1e-4


def test_records_without_room_take_the_generic_sweeps(gpu, monkeypatch):
    """A grid whose fields fit on the device and whose strip records do not runs as it
    does without them, bit for bit."""
    import torch
    from shared_cfd_b200.solver import Solver

    monkeypatch.setenv("SCFD_AUTOTUNE", "0")
    case = cases.flat_plate(768, 512)

    def used():
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        s = Solver(case, gpu)
        took = before - torch.cuda.mem_get_info()[0]
        s.close()
        return took

    torch.cuda.init()
    used()
    full = used()
    monkeypatch.setenv("SCFD_SWEEP_LEGACY", "1")
    ref = run_case(case, gpu, 2)
    fields = used()
    monkeypatch.delenv("SCFD_SWEEP_LEGACY")
    records = 8 * 40 * 768 * 512  # 40 doubles a cell
    assert full - fields >= records
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (full + fields) // 2, dtype=torch.uint8, device="cuda")
    try:
        got = run_case(case, gpu, 2)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert got["stats"].status == 0
    assert np.array_equal(got["q"][0], ref["q"][0])
