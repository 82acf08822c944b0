"""The choice between the column-by-column and the tensor-memory kernels, on
structures where one side was measured faster by 15 % or more (CPU only; the
library's own layout.cpp and rule, through tests/choice_check.cpp).  A long 1-D
matrix with small leaves fills few rows of the tensor-memory kernels' tiles and
pays for whole groups of four or eight columns; a matrix with higher ranks does
not."""

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from qhmat_gb300.construct import spatial_partition

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "qhmat_gb300" / "csrc"
RANKS = {1: (6, 6), 2: (17, 11), 3: (33, 21)}  # neighbouring, admissible


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = tmp_path_factory.mktemp("choice") / "choice_check"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", "-o", str(exe), str(ROOT / "tests" / "choice_check.cpp"),
                    str(CSRC / "layout.cpp")], check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("n,dim,leaf,one_by_one,several", [
    (16384, 1, 16, (1, 2, 3, 4, 5, 9), (8, 16, 24, 64)),
    (20000, 1, 64, (1, 2, 3), (6, 8, 12, 16, 64)),
    (300, 1, 64, (1, 2), (3, 4, 5, 9, 16)),
    (2048, 1, 32, (1, 2), (3, 4, 5, 9, 16)),
    (9001, 2, 16, (1, 2, 3), (6, 8, 12, 16, 64)),
    (9001, 2, 64, (1, 2), (3, 4, 5, 9, 16)),
    (4000, 3, 64, (1, 2), (3, 4, 5, 9, 16)),
])
def test_faster_kernels_are_chosen(checker, n, dim, leaf, one_by_one, several):
    _, rects = spatial_partition(np.random.default_rng(3).random((n, dim)), leaf)
    lines = [f"{n} 152", " ".join(map(str, one_by_one + several + (0,)))]
    for r0, r1, c0, c1, admissible in (b[:5] for b in rects):
        rank = max(1, min(RANKS[dim][1 if admissible else 0], min(r1 - r0, c1 - c0) // 2))
        lines.append(f"{r0} {r1} {c0} {c1} {0 if (r0, r1) == (c0, c1) else rank}")
    r = subprocess.run([str(checker)], input="\n".join(lines), capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split() == ["0"] * len(one_by_one) + ["1"] * len(several)
