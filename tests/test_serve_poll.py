"""The serving dispatcher's watch over the batch in flight, on the CPU."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_watch_sees_the_end_of_a_batch_under_steady_work(tmp_path):
    exe = tmp_path / "serve_poll_check"
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", "-Wall", "-Wextra", "-Werror",
                    f"-I{ROOT / 'oceanlib_b200' / 'csrc'}",
                    str(ROOT / "tests" / "native" / "serve_poll_check.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout + res.stderr
