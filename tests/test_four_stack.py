"""The any-hit walk's stack rule (csrc/four_stack.h) on trees of every number of levels,
under the address and undefined-behaviour sanitizers."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


def test_every_walk_keeps_to_its_words(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "four_stack_check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-g", "-fsanitize=undefined,address", "-fno-sanitize-recover=all",
                    f"-I{HERE.parent / 'tim_raytracing_b200' / 'csrc'}", str(HERE / "c" / "four_stack_check.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split() == ["walks", "1920", "bad", "0", "waits", "many"]
