"""The tensor-memory kernels' work lists cover the layout exactly once, within
the sizes of the kernels' stages (CPU only, through tests/worklist_check.cpp)."""

import os
import shutil
import subprocess
from pathlib import Path

import pytest

from conftest import GOLDEN_CASES

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "qhmat_gb300" / "csrc"


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = tmp_path_factory.mktemp("worklists") / "worklist_check"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", "-o", str(exe), str(ROOT / "tests" / "worklist_check.cpp"),
                    str(CSRC / "layout.cpp")], check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("chunks", ["", "1"])
@pytest.mark.parametrize("name", GOLDEN_CASES)
def test_work_lists(checker, name, chunks):
    env = dict(os.environ, QHMAT_GB300_PART_CHUNKS=chunks)
    r = subprocess.run([str(checker), str(ROOT / "tests" / "golden" / f"{name}.qhmat")], capture_output=True, text=True,
                       env=env)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout + r.stderr
