"""The CUDA-core chi0 contraction (FP64 and FP32) at the edges of its tiles and parts, against the oracle
(needs a GB300): ABF counts around the mu tile of 48 and the nu tiles of 48, 96 and 144, NAO counts around
the quads of j and i, one to many columns per cluster part, one cell and several.

Tolerance, relative to the largest entry.  FP64: sums of at most K = n_cells n_ao a few hundred terms a j,
300 * 2^-53 and the same again for X, G and the transforms, below 1e-12; FP32: 300 * 2^-24 = 1.8e-5."""
import numpy as np
import pytest

import librpa_gb300 as L
from conftest import oracle_input
from librpa_gb300.synthetic import small_periodic
from oracle.rpa_oracle import Options as OOpts, rpa_correlation_energy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nao,nabf,period", [
    ([4, 1], [48, 3], (1, 1, 1)),
    ([5, 4], [49, 47], (1, 1, 1)),
    ([13], [40], (2, 2, 1)),
    ([3, 2], [96, 97], (1, 1, 1)),
    ([36, 7], [144, 30], (1, 1, 1)),
    ([8, 9], [145, 50], (2, 1, 1)),
    ([2], [1], (1, 1, 1)),
])
def test_chi0_simt_edges(nao, nabf, period):
    s = small_periodic(len(nao), nao, nabf, period, nocc=1, seed=5, nfreq=6)
    o = rpa_correlation_energy(oracle_input(s), OOpts(nfreq=6, minimax_emin=s.minimax_emin, minimax_emax=s.minimax_emax))
    for prec, tol in ((L.CHI0_FP64, 1e-12), (L.CHI0_FP32, 300 * 2.0 ** -24)):
        with L.Handler() as h:
            L.load_system(h, s)
            h.set_gb300_options(L.gb300_options(chi0_precision=prec, ec_path=L.EC_LU_FP64, keep_chi0=1))
            h.get_rpa_correlation_energy(L.Options(nfreq=6, tfgrids_type=L.Minimax, minimax_emin=s.minimax_emin,
                                                   minimax_emax=s.minimax_emax), L.n_ibz(s))
            for iw in (0, 5):
                for iq in range(L.n_ibz(s)):
                    blocks = o["chi0q"][iw][iq]
                    top = max(np.abs(b).max() for b in blocks.values())
                    for (I, J), ref in blocks.items():
                        got = h.get_chi0_block(iw, iq, I, J, s.nabf[I], s.nabf[J])
                        assert np.abs(got - ref).max() <= tol * top, (prec, iw, iq, I, J)
