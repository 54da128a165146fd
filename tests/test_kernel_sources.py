"""Rules of the kernels' sources that neither the compiler nor a run shows: what breaks
them is undefined, whatever a device makes of it."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "shared_cfd_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_sweep_barriers_are_initialised_once():
    """An mbarrier that is live may not be initialised again: one statement initialises
    all of a sweep CTA's barriers, each with the arrivals of its phases."""
    src = source("k_wave.cu")
    assert len(re.findall(r"\bmbar_init\(", src)) == 1
    assert re.search(r"for \(int k = threadIdx\.x; k < UPC \* L::NBAR; k \+= kThreads\)\s*mbar_init\(", src)


def test_dynamic_shared_memory_is_declared_aligned():
    """Every kernel reads its dynamic shared memory as doubles or 16-byte vectors (k_cea's
    species tables as double2 in all its kernels), so each declares that alignment."""
    found = 0
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            for decl in re.findall(r"extern __shared__[^;]*;", source(name)):
                found += 1
                assert re.search(r"__align__\((16|32|64|128)\)", decl), (name, decl)
    assert found >= 7


def test_sweep_winds_down_with_its_copies():
    """A sweep CTA whose wait gave up stays until the bulk copies on their way into its
    shared memory have landed: that pause stands before the cluster's last barrier."""
    src = source("k_wave.cu")
    kernel = src[src.index("k_wave(View v, WaveArgs a)"):src.index("records_to_tile(")]
    tail = kernel[kernel.rindex("cluster_sync();", 0, kernel.rindex("cluster_sync();")):]
    assert re.search(r"\*s_bail\b|s_bail\) != 0", tail) and "kDrain" in tail
