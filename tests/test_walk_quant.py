"""CPU property test of the 8-wide walk's box test (csrc/trace_quant.cuh) against
CollideBox, on seeded cases built to sit on the decision boundary
(tests/c/quant_box_check.c): it loses no box that the reference enters."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.mark.parametrize("seed", [1, 2])
def test_box_test_against_collide_box(tmp_path, seed):
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    exe = tmp_path / "quant_box_check"
    subprocess.run([cc, "-O2", "-ffp-contract=off", "-fno-fast-math", str(HERE / "c" / "quant_box_check.c"), "-o", str(exe),
                    "-lm"], check=True)
    r = subprocess.run([str(exe), "4000000", str(seed)], capture_output=True, text=True)
    words = r.stdout.split()
    got = dict(zip(words[0::2], map(int, words[1::2])))
    assert r.returncode == 0, r.stdout + r.stderr
    assert got["lost"] == 0
    assert got["tested"] > 1_000_000 and got["entered"] > 100_000 and got["missed"] > 100_000
