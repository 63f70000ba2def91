"""The CUDA-core chi0 contraction takes atoms of at most 46 NAOs in FP64 and 87 in FP32 (needs a GB300): the largest
run, in FP64 against the oracle, and one more NAO is refused.

Tolerance, relative to the largest entry: sums of n_ao n_ao terms in FP64, 49^2 2^-53 and the transforms, below 1e-11."""
import numpy as np
import pytest

import librpa_gb300 as L
from conftest import oracle_input
from librpa_gb300.synthetic import small_periodic
from oracle.rpa_oracle import Options as OOpts, rpa_correlation_energy

pytestmark = pytest.mark.gpu


def _run(h, s, prec):
    L.load_system(h, s)
    h.set_gb300_options(L.gb300_options(chi0_precision=prec, ec_path=L.EC_LU_FP64, keep_chi0=1))
    return h.get_rpa_correlation_energy(L.Options(nfreq=6, tfgrids_type=L.Minimax, minimax_emin=s.minimax_emin,
                                                  minimax_emax=s.minimax_emax), L.n_ibz(s))[0]


def test_most_orbitals_in_fp64():
    s = small_periodic(2, [46, 3], [50, 7], (1, 1, 1), nocc=1, seed=15, nfreq=6)
    o = rpa_correlation_energy(oracle_input(s), OOpts(nfreq=6, minimax_emin=s.minimax_emin, minimax_emax=s.minimax_emax))
    with L.Handler() as h:
        _run(h, s, L.CHI0_FP64)
        for iw in (0, 5):
            blocks = o["chi0q"][iw][0]
            top = max(np.abs(b).max() for b in blocks.values())
            for (I, J), ref in blocks.items():
                got = h.get_chi0_block(iw, 0, I, J, s.nabf[I], s.nabf[J])
                assert np.abs(got - ref).max() <= 1e-11 * top, (iw, I, J)


def test_most_orbitals_in_fp32():
    with L.Handler() as h:
        assert np.isfinite(_run(h, small_periodic(1, [87], [60], (1, 1, 1), nocc=1, seed=15, nfreq=6), L.CHI0_FP32))


@pytest.mark.parametrize("nao,prec", [(47, L.CHI0_FP64), (88, L.CHI0_FP32)])
def test_one_more_is_refused(nao, prec):
    s = small_periodic(1, [nao], [4], (1, 1, 1), nocc=1, seed=15, nfreq=6)
    with L.Handler() as h, pytest.raises(Exception, match="too large for the SIMT"):
        _run(h, s, prec)
