"""The launch shape of a visibility batch (rg_internal.h, vis_launch) up to the
largest count an int holds, checked on the CPU: every segment in exactly one
block, blocks within their bounds, and no signed overflow on the way."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "restir-vulkan_gb300" / "csrc"


def test_every_count_has_a_shape(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not found")
    exe = tmp_path / "vis_launch_check"
    cmd = [nvcc, "-std=c++17", "-O1", "-Xcompiler", "-fsanitize=undefined,-fno-sanitize-recover=all", f"-I{CSRC}",
           str(ROOT / "tests" / "vis_launch_check.cu"), "-o", str(exe), "-lubsan"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    assert int(r.stdout) == 3 + 6 * 5 + 3
