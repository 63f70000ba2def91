"""The Gauss-Jordan solve of W_c (needs a GB300), in shared memory and, for more than 311 columns a side, in
global memory: residuals, and the flag for a zero column or a NaN; and the LU form of E_c with more q points than
one batch of its matrices holds, against the Cholesky form."""
import os
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import librpa_gb300 as L
from librpa_gb300.synthetic import small_periodic

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def test_gauss_jordan_forms(lib, tmp_path):
    from librpa_gb300.build import ARCH, CFLAGS, PKG
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "gj_check"
    subprocess.run([nvcc, *ARCH, *[f for f in CFLAGS if f not in ("-Xptxas", "-warn-spills")],
                    str(ROOT / "tests" / "gj_check.cu"), "-o", str(exe), "-L", str(PKG), "-l:liblibrpa_gb300.so",
                    "-Xlinker", "-rpath", "-Xlinker", str(PKG), "-ldl"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    lines = [ln.split() for ln in out.stdout.strip().split("\n")]
    assert len(lines) == 8 * 4 * 2 + 4 * 4
    for N, M, staged, kind, residual, bad in lines:
        what = (N, M, staged, kind, residual, bad)
        if int(kind) < 2:
            # a diagonal of 4 sqrt(N) beside entries of at most 1 (singular values within about 4 +- 1.2 of
            # sqrt(N)): condition below 4, N roundings of 2^-53 an entry on each side
            assert int(bad) == 0 and float(residual) <= 1e-15 * (10 + int(N)), what
        else:
            assert int(bad) == 1, what


def test_lu_of_several_batches():
    # 16 frequencies of complex 800 x 800: 164 MB a q point, 24 of the 25 in the first batch of 4 GB
    s = small_periodic(1, [2], [800], (5, 5, 1), nocc=1, seed=21, nfreq=16)
    assert L.n_ibz(s) == 25
    perq = {}
    for path in (L.EC_LU_FP64, L.EC_CHOL_FP64):
        with L.Handler() as h:
            L.load_system(h, s)
            h.set_gb300_options(L.gb300_options(chi0_precision=L.CHI0_FP64, ec_path=path))
            _, q = h.get_rpa_correlation_energy(L.Options(nfreq=16, tfgrids_type=L.Minimax, minimax_emin=s.minimax_emin,
                                                          minimax_emax=s.minimax_emax), 25)
            perq[path] = np.asarray(q)
            assert h.stats()["ec_lu_fallback_q"] == 0
    lu, chol = perq[L.EC_LU_FP64], perq[L.EC_CHOL_FP64]
    # N 2^-52 1e3 absolute, times frequency weights of below 50 Ha in all over 2 pi; points differ by far more
    assert np.abs(lu - chol).max() <= 1e-11 * 800
    assert len({complex(v) for v in lu}) > 12
