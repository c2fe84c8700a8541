"""Host units of the pass schedules, compiled by the host compiler alone."""
from __future__ import annotations

import os
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_schedule_choice_host_unit(tmp_path):
    """Built-in schedules by rows x images, and what set and tuned pairs keep."""
    nvcc = Path(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"))
    out = tmp_path / "test_sched"
    res = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", f"-I{nvcc.parent.parent / 'include'}",
                          f"-I{ROOT / 'include'}", f"-I{ROOT / 'glscv_gb300' / 'csrc'}",
                          str(ROOT / "tests" / "cpp" / "test_sched.cpp"), "-o", str(out)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    run = subprocess.run([str(out)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and "ALL OK" in run.stdout, run.stdout
