"""Waits of the tensor-core kernels that run out: a wait on an mbarrier that nothing arrives at gives up
after its limit of wall time and returns (needs a GB300)."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def _nvcc():
    return os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def test_waits_end_at_their_limit(tmp_path):
    exe = tmp_path / "wait_check"
    subprocess.run([_nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17", "-I",
                    str(ROOT / "librpa_gb300" / "csrc"), str(ROOT / "tests" / "wait_check.cu"), "-o", str(exe)], check=True)
    lines = subprocess.run([str(exe)], capture_output=True, text=True, check=True, timeout=60).stdout.split("\n")
    got = [[float(x) for x in ln.split()] for ln in lines if ln]
    assert [g[0] for g in got] == [0, 20, 100]
    for _, done, ms in got:
        # 200 units of 2^20 ns; a poll may be suspended for a while, and the clock is read every 256 of them
        assert done == 0 and 200 <= ms <= 1000, got


def test_launches_after_one_that_gave_up_do_nothing(lib, tmp_path):
    from librpa_gb300.build import ARCH, CFLAGS, PKG
    exe = tmp_path / "t1_give_up_check"
    subprocess.run([_nvcc(), *ARCH, *[f for f in CFLAGS if f not in ("-Xptxas", "-warn-spills")],
                    str(ROOT / "tests" / "t1_give_up_check.cu"), "-o", str(exe), "-L", str(PKG), "-l:liblibrpa_gb300.so",
                    "-Xlinker", "-rpath", "-Xlinker", str(PKG), "-ldl"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
