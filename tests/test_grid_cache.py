"""The cache of the persistent kernels' grid sizes (csrc/grid_cache.h) holds every stack
size that a launch can ask for, up to the deepest 8-wide tree of a batch, under UBSan."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


def test_every_stack_size_has_its_place(tmp_path):
    cxx, cuda = shutil.which("g++"), Path("/usr/local/cuda/include")
    if cxx is None or not (cuda / "cuda_runtime_api.h").exists():
        pytest.skip("no C++ compiler or CUDA headers")
    exe = tmp_path / "grid_cache_check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-g", "-fsanitize=undefined,address", "-fno-sanitize-recover=all", f"-I{cuda}",
                    f"-I{HERE.parent / 'tim_raytracing_b200' / 'csrc'}", str(HERE / "c" / "grid_cache_check.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split() == ["sizes", "47", "wrong", "0"]   # 2 * 16 + 2 stack words, 12 beside them
