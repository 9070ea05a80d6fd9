"""The backward's second stream (csrc/side_stream.h) rejoins on every way out of a call: compiled here against a fake CUDA
runtime, where a launch or an event call can be made to fail without a GPU."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def test_second_stream_rejoins_on_every_way_out(tmp_path):
    if not os.path.exists(os.path.join(CUDA, "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    exe = str(tmp_path / "side_stream_check")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-isystem", CUDA, os.path.join(HERE, "side_stream_check.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    run = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert run.stdout == "ok\n", run.stdout
