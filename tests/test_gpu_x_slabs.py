"""X = C G of the tensor-core chi0 contraction, formed for some atoms at a time so that it takes a bounded amount of
memory beside its re-ordered copy (needs a GB300)."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def test_slabs_of_x(lib, tmp_path):
    from librpa_gb300.build import ARCH, CFLAGS, PKG
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "x_slab_check"
    subprocess.run([nvcc, *ARCH, *[f for f in CFLAGS if f not in ("-Xptxas", "-warn-spills")],
                    str(ROOT / "tests" / "x_slab_check.cu"), "-o", str(exe), "-L", str(PKG), "-l:liblibrpa_gb300.so",
                    "-Xlinker", "-rpath", "-Xlinker", str(PKG), "-ldl"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
