"""The page populator of to_dense's output (CPU only, through
tests/pages_check.cpp): it works without the threads that cannot be made."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = tmp_path_factory.mktemp("pages") / "pages_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", f"-I{ROOT / 'qhmat_gb300' / 'csrc'}", "-o", str(exe),
                    str(ROOT / "tests" / "pages_check.cpp")], check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("failing", [0, 1, 2, 3])
def test_threads_that_cannot_be_made(checker, failing):
    r = subprocess.run([str(checker), str(failing)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("OK"), (r.returncode, r.stdout, r.stderr)
