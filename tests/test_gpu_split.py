"""The three-piece BF16 split of the chi0 contraction (needs a GB300): the pieces add up to the value, hi and
mid are the nearest ones, and the three of the nine products that the contraction leaves out stay as small
as rounding to nearest makes them."""
import os
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("split")
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17", "-I",
                    str(ROOT / "librpa_gb300" / "csrc"), str(ROOT / "tests" / "split_check.cu"), "-o", str(tmp / "exe")],
                   check=True)

    def run(x):
        (tmp / "in").write_bytes(np.ascontiguousarray(x, dtype=np.float32).tobytes())
        subprocess.run([str(tmp / "exe"), str(tmp / "in"), str(tmp / "out")], check=True, timeout=60)
        w = np.fromfile(tmp / "out", dtype=np.uint32).reshape(-1, 3)
        lohi = np.stack([w & 0xffff, w >> 16], axis=1).reshape(-1, 3)  # element 0 in the low half
        return (lohi << 16).astype(np.uint32).view(np.float32).astype(np.float64)  # [value][hi, mid, lo]
    return run


def _half_ulp(x):
    """Half the distance of BF16 numbers around x (8 significant bits)."""
    return np.ldexp(1.0, np.frexp(np.abs(x))[1] - 9)


def test_pieces_are_nearest_and_exact(split):
    rng = np.random.default_rng(3)
    x = (rng.standard_normal(1 << 16) * np.exp2(rng.integers(-60, 60, 1 << 16))).astype(np.float32)
    edge = np.array([0.0, -0.0, 1.0, 1.99999988, -1.99999988, 1.00390625, 1.001953125, 1.0039062, 255.99998, 3e38, -1e-30, 0.1],
                    dtype=np.float32)
    x = np.concatenate([x, edge])
    p, v = split(x), x.astype(np.float64)
    assert (p.sum(axis=1) == v).all()
    r1 = v - p[:, 0]
    assert (np.abs(r1) <= _half_ulp(v)).all()
    assert (np.abs(r1 - p[:, 1]) <= np.where(r1 == 0.0, 0.0, _half_ulp(r1))).all()


def test_not_a_number_and_infinity_stay(split):
    p = split(np.array([np.inf, -np.inf, np.nan, 1.0], dtype=np.float32))
    with np.errstate(invalid="ignore"):
        s = p.sum(axis=1)
    assert not np.isfinite(s[:3]).any() and s[3] == 1.0


def test_products_left_out(split):
    # hi lies within 2^-9 of the value's binade, mid within 2^-9 of the rest's: what is left out is below
    # 2 x 2^-9 x 2^-17 of the largest product, its rms about a tenth of 2^-24 (0.3 with pieces cut off)
    rng = np.random.default_rng(4)
    a, b = (split(rng.standard_normal(1 << 17).astype(np.float32)) for _ in range(2))
    left = a[:, 1] * b[:, 2] + a[:, 2] * b[:, 1] + a[:, 2] * b[:, 2]
    rms = np.sqrt(np.mean((left / (a.sum(axis=1) * b.sum(axis=1))) ** 2))
    assert rms <= 0.2 * 2.0 ** -24
