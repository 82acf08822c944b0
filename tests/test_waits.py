"""The bounded wait of the tensor-memory kernels (CPU only, through
tests/waits_check.cpp): the preceding kernel's time is not counted, a phase that
never completes runs the wait out, and a block that gives up ends its waits."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_bounded_wait(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "waits_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Werror", f"-I{ROOT / 'qhmat_gb300' / 'csrc'}", "-o", str(exe),
                    str(ROOT / "tests" / "waits_check.cpp")], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout
