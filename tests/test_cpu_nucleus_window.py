"""The value buckets of rows without a top-k cut, compiled for the host (tests/native/nucleus_window.cpp)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_bucket_ends(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    binary = tmp_path / "nucleus_window"
    build = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-I",
                            str(ROOT / "flash_gordon_b200" / "csrc" / "cuda"),
                            str(ROOT / "tests" / "native" / "nucleus_window.cpp"), "-o", str(binary)],
                           capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    run = subprocess.run([str(binary)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout
    assert int(run.stdout) > 1_000_000
