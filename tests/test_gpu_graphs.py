"""Steps replayed from CUDA graphs, one or eight to a graph, give the bits of steps that
are enqueued one by one; and the graph of eight is built when a context has run enough
steps to pay for it."""
import numpy as np
import pytest

from shared_cfd_b200 import abi, cases
from shared_cfd_b200.solver import Solver

pytestmark = pytest.mark.gpu

CASES = {
    "sod": lambda: cases.sod(100, 4),
    "plate": lambda: cases.flat_plate(40, 24),
    "channel": lambda: cases.adjoint_channel(n=12),
    "precon_lusgs": lambda: cases.forward_step(0, n=5, scheme=abi.SCHEME_PRECON_LUSGS, viscous=1, dt_mode=abi.DT_LOCAL),
}


def runs(case, lib, lengths):
    s = Solver(case, lib=lib)
    try:
        s.upload()
        s.prepare(1)
        seen = []
        for n in lengths:
            st = s.run(1, n)
            seen.append((n, s.launch_count(), s.tuning().get("graph_steps"), st.tt, st.dt_grbl))
        q, w, _, _ = s.download()
        return q, w, s.download_qp(), seen
    finally:
        s.close()


@pytest.mark.parametrize("kind", list(CASES))
@pytest.mark.parametrize("lengths", [[2, 211], [3, 33, 90, 61, 40]])
def test_graph_runs_match_eager_steps(gpu, monkeypatch, kind, lengths):
    monkeypatch.setenv("SCFD_AUTOTUNE", "0")  # one kernel shape on both sides
    case = CASES[kind]()
    monkeypatch.delenv("SCFD_GRAPH", raising=False)
    *got, seen = runs(case, gpu, lengths)
    monkeypatch.setenv("SCFD_GRAPH", "0")
    *ref, plain = runs(case, gpu, lengths)
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)
    for (n, launches, steps, *times), (_, eager_launches, none, *eager_times) in zip(seen, plain):
        assert launches == eager_launches and times == eager_times and none is None
    # runs of eight steps or more add up to 160 before the long graph is there
    total = np.cumsum([n if n >= 8 else 0 for n in lengths])
    assert [steps for _, _, steps, *_ in seen] == [8 if t >= 160 else 1 for t in total]


def test_inner_loops_replay_single_steps(gpu):
    case = cases.reacting_step(scale=1.0 / 64.0, inner=2)
    case.desc.thermo = abi.THERMO_CHEMKIN_COLD
    case.desc.res_rate_err = 1e300
    *_, seen = runs(case, gpu, [200])
    assert seen[0][2] == 1
