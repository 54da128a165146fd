"""The CUDA library's C symbols: only scfd_*, so that none is taken by (or takes over) a
function of the host program."""
import subprocess

from test_abi import cuda_lib_path


def test_c_symbols_carry_the_prefix():
    out = subprocess.check_output(["nm", "-D", "--defined-only", cuda_lib_path()], text=True)
    names = [line.split()[2] for line in out.splitlines()]
    assert [n for n in names if not n.startswith(("_Z", "scfd_"))] == []
