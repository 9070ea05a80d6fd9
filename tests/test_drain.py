"""A kernel that gives up waits for the loads it has in flight, and for no others (csrc/drain.h): against a model of the barriers."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_drain_waits_for_what_is_in_flight(tmp_path):
    exe = str(tmp_path / "drain_check")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", os.path.join(HERE, "drain_check.cpp"), "-o", exe], check=True,
                   capture_output=True, text=True)
    assert subprocess.run([exe], capture_output=True, text=True, timeout=60).stdout == "ok\n"


# tc_intra_grp.cuh has waits of its own for the two buffers that its loads take in turn
@pytest.mark.parametrize("source", ["tc_dbc_tma", "tc_state_tma", "tc_walk_tma", "tc_scan_tma", "tc_dx_tma", "tc_scan_ws", "tc_bmm_tma",
                                    "tc_dcb_tma", "tc_intra", "tc_intra_sums"])
def test_every_kernel_with_loads_waits_for_them(source):
    """A kernel's text, from one __global__ to the next, and the functions before the first: a load is asked for, so one is waited for on
    the way out.  It cannot be made to happen on a GPU without breaking the kernel."""
    with open(os.path.join(HERE, "..", "bi-mamba2_b200", "csrc", source + ".cuh")) as f:
        before, *kernels = f.read().split("__global__")
    for part in (before + k for k in kernels):
        assert ("tma_load" in part or "feed.start()" in part) <= ("drain_loads(" in part or "feed.leave()" in part), part[len(before):][:200]


@pytest.mark.parametrize("source", ["tc_intra", "tc_intra_sums"])
def test_a_load_that_does_not_arrive_is_reported(source):
    """The intra-chunk kernels leave reporting to umma_drain, which a tile that never arrived does not reach."""
    with open(os.path.join(HERE, "..", "bi-mamba2_b200", "csrc", source + ".cuh")) as f:
        after = f.read().split("ok = mbar_wait(&sh.free_bar[0], 0);")[1]
    assert "atomicExch(status, kErrMmaTimeout);" in after.split("__syncthreads_and")[0]
