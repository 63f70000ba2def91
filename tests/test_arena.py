"""Device memory kept between calls (librpa_gb300/csrc/device_arena.cpp), compiled for the host over a stand-in
for the CUDA runtime: what is unused, in the call itself, in idle arenas or in a call on another thread, makes
room for an allocation that fails; buffers that fit the device fit whatever sizes went before; nothing is lost
or freed twice."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_arenas(tmp_path):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    inc = Path(nvcc).resolve().parents[1] / "include"
    if not (inc / "cuda_runtime.h").exists():
        pytest.skip("no CUDA headers")
    exe = tmp_path / "arena_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", str(inc), str(ROOT / "tests" / "arena_check.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
