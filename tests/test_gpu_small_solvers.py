"""Edges of the small dense solvers (needs a GB300): the Cholesky's 64-wide diagonal blocks (last block of
1 to 64 rows) through the tensor-core Cholesky's self-test; the Gauss-Jordan solve of W_c, whose
columns go to the CTAs of a cluster four at a time, through the Gamma-point G0W0 against the oracle; and
the LU of E_c, whose columns go the same way to clusters of 1 to 8 CTAs, against the form with one CTA, and
the panels of the complex Cholesky, through E_c against the LU form."""
import ctypes
import math

import numpy as np
import pytest

import librpa_gb300 as L
from conftest import oracle_input
from librpa_gb300.synthetic import cluster_gamma, small_periodic
from oracle.gw_oracle import g0w0_gamma
from oracle.rpa_oracle import Options as OOpts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 63, 65, 66, 127, 128, 129, 190])
def test_cholesky_diagonal_blocks(lib, N):
    rel = ctypes.c_double(float("nan"))
    dl = lib.librpa_gb300_selftest_chol_ozaki(N, 3, 7 + N, 0, 0.05, ctypes.byref(rel))
    assert not math.isnan(dl), lib.librpa_get_last_error(None).decode()
    # two FP64 factorisations of a matrix of condition below 1e3: N 2^-52 each, with the condition
    assert dl <= 1e-11 * N and rel.value <= 1e-12, (dl, rel.value)


@pytest.mark.parametrize("nabf", [(1, 2), (3, 4), (15, 16), (16, 17), (20, 45), (60, 70)])
def test_wc_solve_through_g0w0(nabf):
    s = cluster_gamma("gj", 2, [(3, nabf[0]), (4, nabf[1])], 3, nfreq=6)
    s.nao, s.nabf = list(s.nao), list(s.nabf)
    s.v_cut = s.Vq
    nb = s.n_bands
    vxc = np.zeros((1, 1, nb))
    ref = g0w0_gamma(oracle_input(s), s.v_cut, vxc, OOpts(nfreq=6, minimax_emin=s.minimax_emin, minimax_emax=s.minimax_emax))
    with L.Handler() as h:
        L.load_system(h, s)
        h.set_gb300_options(L.gb300_options(chi0_precision=L.CHI0_FP64, ec_path=L.EC_LU_FP64))
        o = L.Options(nfreq=6, tfgrids_type=L.Minimax, minimax_emin=s.minimax_emin, minimax_emax=s.minimax_emax)
        h.lib.librpa_build_g0w0_sigma(h.h, ctypes.byref(o))
        h._check()
        got = h.g0w0_sigc_iw(0, 0, nb, 6)
    want = np.asarray(ref["sigc_iw"][0]).reshape(got.shape)
    # FP64 throughout; the frequency-to-time weights of a 6-point window amplify rounding by up to 1e3
    assert np.abs(got - want).max() <= 1e-11 * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("kind", [0, 1, 2], ids=["uniform", "ties", "not_a_number"])
@pytest.mark.parametrize("N,batch,complex_", [
    (1, 3, 0), (3, 16, 1), (4, 16, 0),          # fewer column groups than CTAs of the cluster
    (32, 16, 1), (33, 16, 0), (70, 38, 1),      # whole groups, a last group of one and of two columns
    (304, 2, 1), (320, 2, 1), (450, 2, 0),      # columns in shared memory, in global memory
    (30, 39, 1), (31, 77, 0), (30, 153, 1),     # clusters of 4, 2 and 1
    (120, 153, 1),                              # one CTA a matrix, in global memory
])
def test_lu_log_determinant(lib, N, batch, complex_, kind):
    d = lib.librpa_gb300_selftest_lu(N, batch, complex_, kind, 3 + N)
    assert not math.isnan(d), lib.librpa_get_last_error(None).decode()
    # the same operations per element in the same order; the compiler may fuse them differently: N 2^-52 with
    # the condition of a random matrix (below 1e4 N)
    assert d <= 1e-11 * N * N, d


@pytest.mark.parametrize("nabf", [(16, 17), (31, 33), (32, 33), (48, 49), (64, 65)])
def test_complex_cholesky_panels(nabf):
    # rows below a 32-wide panel: 1, 32, 33, 65, 97 (a CTA takes 32)
    s = small_periodic(2, [3, 2], list(nabf), (2, 1, 1), nocc=1, seed=12, nfreq=6)
    perq = {}
    for path in (L.EC_LU_FP64, L.EC_CHOL_FP64):
        with L.Handler() as h:
            L.load_system(h, s)
            h.set_gb300_options(L.gb300_options(chi0_precision=L.CHI0_FP64, ec_path=path))
            _, q = h.get_rpa_correlation_energy(L.Options(nfreq=6, tfgrids_type=L.Minimax, minimax_emin=s.minimax_emin,
                                                          minimax_emax=s.minimax_emax), L.n_ibz(s))
            perq[path] = np.asarray(q)
            assert h.stats()["ec_lu_fallback_q"] == 0
    # ln det and tr of N x N matrices near 1 with V of condition below 1e3: N 2^-52 1e3 absolute, times
    # frequency weights of below 50 Ha in all over 2 pi
    N = sum(nabf)
    assert np.abs(perq[L.EC_LU_FP64] - perq[L.EC_CHOL_FP64]).max() <= 1e-11 * N
