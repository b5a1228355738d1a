"""CPU property test of the box tests of the binary form's two walks
(csrc/trace_any.cuh, csrc/trace_pair.cuh) against CollideBox, on seeded cases built to
sit on the decision boundary (tests/c/walk_box_check.c): the any-hit test loses no box
that the reference enters, and the closest-hit test decides nothing the reference
decides otherwise."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.mark.parametrize("seed", [1, 2])
def test_box_tests_against_collide_box(tmp_path, seed):
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    exe = tmp_path / "walk_box_check"
    subprocess.run([cc, "-O2", "-ffp-contract=off", "-fno-fast-math", str(HERE / "c" / "walk_box_check.c"), "-o", str(exe),
                    "-lm"], check=True)
    r = subprocess.run([str(exe), "2000000", str(seed)], capture_output=True, text=True)
    words = r.stdout.split()
    got = dict(zip(words[0::2], map(int, words[1::2])))
    assert r.returncode == 0, r.stdout + r.stderr
    assert got["any_lost"] == 0 and got["pair_wrong"] == 0
    # the cases do exercise both outcomes
    assert got["any_cases"] > 1_000_000 and got["any_accept"] > 100_000
    assert got["pair_decided"] > 100_000 and got["pair_open"] > 100_000
