"""The serving loop's failure path against a fake CUDA runtime, on the CPU."""
from __future__ import annotations

import os
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "glscv_gb300" / "csrc"


def test_failed_launch_keeps_its_memory_until_idle(tmp_path):
    """A request whose launches fail half way gives its device memory back only
    when what was issued before has finished."""
    nvcc = Path(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"))
    out = tmp_path / "test_serve_failure"
    res = subprocess.run(["g++", "-std=c++17", "-O1", f"-I{nvcc.parent.parent / 'include'}",
                          f"-I{ROOT / 'include'}", f"-I{CSRC}",
                          str(ROOT / "tests" / "cpp" / "test_serve_failure.cpp"),
                          str(CSRC / "serve.cpp"), "-lpthread", "-o", str(out)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    run = subprocess.run([str(out)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0 and "ALL OK" in run.stdout, run.stdout
