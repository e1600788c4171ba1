"""The serving loop's growing device blocks, on the CPU: a growth that the pool
refuses leaves a block empty, not with the size it had before."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_block_holds_what_it_says_after_a_failed_growth(tmp_path):
    exe = tmp_path / "serve_block_check"
    subprocess.run(["g++", "-std=c++20", "-O1", "-Wall", "-Wextra", "-Werror", f"-I{ROOT / 'oceanlib_b200' / 'csrc'}",
                    str(ROOT / "tests" / "native" / "serve_block_check.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
