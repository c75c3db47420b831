"""The host-buffer calls' per-thread caches belong to a device, and a capture is uploaded in parts only
where that hides more than it costs: tests/cpp/host_cache.cpp runs both against a fake CUDA
runtime of two devices (no GPU)."""
from __future__ import annotations

import subprocess
from pathlib import Path

from backprojector_gb300 import build

SRC = Path(__file__).resolve().parent / "cpp" / "host_cache.cpp"


def test_caches_follow_the_device(tmp_path):
    exe = tmp_path / "host_cache"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{build.INCLUDE}", f"-I{build.CSRC}",
                    f"-I{build.CUDA_HOME / 'include'}", str(SRC), "-o", str(exe)], check=True,
                   capture_output=True, text=True)
    r = subprocess.run([str(exe)])
    assert r.returncode == 0, f"check on line {r.returncode} of {SRC.name}"
