"""What a solver does without where device memory is short (SCFD_MEM_LIMIT stands for a
smaller device): first the staging of whole fields, so that copies to and from the host go
in parts, then the sweeps' strip records, then it refuses."""
import numpy as np
import pytest

from shared_cfd_b200 import abi, cases
from shared_cfd_b200.solver import Solver, SolverError

pytestmark = pytest.mark.gpu

STAGING = 64 << 20


def run(case, lib):
    s = Solver(case, lib=lib)
    try:
        report = s.tuning()
        s.upload()
        s.prepare(1)
        s.run(1, 2)
        return report, s.download()[:3]
    finally:
        s.close()


@pytest.mark.parametrize("kind", ["plate", "step"])
def test_memory_runs_out_step_by_step(gpu, monkeypatch, kind):
    monkeypatch.setenv("SCFD_AUTOTUNE", "0")  # one kernel shape in all runs
    for name in ("SCFD_MEM_LIMIT", "SCFD_SWEEP_LEGACY"):
        monkeypatch.delenv(name, raising=False)
    # w takes more than one part: 9 doubles of 1.05 M cells, 17 of 0.52 M
    case = cases.flat_plate(1300, 800) if kind == "plate" else cases.reacting_step(scale=0.7, inner=2)
    whole, ref = run(case, gpu)
    assert whole["memory"]["staging_bytes"] > STAGING and whole["sweep"]["kind"] == "cluster wavefront"

    monkeypatch.setenv("SCFD_MEM_LIMIT", str(whole["memory"]["arena_bytes"] - 1))
    parts, got = run(case, gpu)
    assert parts["memory"]["staging_bytes"] == STAGING and parts["sweep"] == whole["sweep"]
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)

    monkeypatch.setenv("SCFD_MEM_LIMIT", str(parts["memory"]["arena_bytes"] - 1))
    bare, got = run(case, gpu)
    assert bare["sweep"] == {"kind": "generic", "reason": "no memory for the strip records"}
    with monkeypatch.context() as m:
        m.delenv("SCFD_MEM_LIMIT")
        m.setenv("SCFD_SWEEP_LEGACY", "1")
        _, ref = run(case, gpu)
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)

    monkeypatch.setenv("SCFD_MEM_LIMIT", str(bare["memory"]["arena_bytes"] - 1))
    with pytest.raises(SolverError) as e:
        run(case, gpu)
    assert e.value.code == abi.E_CUDA
