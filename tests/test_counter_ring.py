"""tim_rt_trace_dev's work counters (csrc/counter_ring.h): 4,096 calls in flight share no word."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


def test_calls_in_flight_share_no_counter(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "counter_ring_check"
    subprocess.run([cxx, "-std=c++17", "-O1", f"-I{HERE.parent / 'tim_raytracing_b200' / 'csrc'}",
                    str(HERE / "c" / "counter_ring_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
