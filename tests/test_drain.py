"""A kernel that gives up waits for the loads it has in flight, and for no others (csrc/drain.h): against a model of the barriers."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_drain_waits_for_what_is_in_flight(tmp_path):
    exe = str(tmp_path / "drain_check")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", os.path.join(HERE, "drain_check.cpp"), "-o", exe], check=True,
                   capture_output=True, text=True)
    assert subprocess.run([exe], capture_output=True, text=True, timeout=60).stdout == "ok\n"
