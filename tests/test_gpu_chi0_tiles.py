"""The tensor-core chi0 contraction at the edges of its tiles (needs a GB300): chi0(q, omega) of the
default path against the FP64 path of the same inputs, over the NAO counts at which a producer's unit
of j changes (4, 5, 8, 9, 12, 13, 14, 15, 16, 17, 32), the ABF counts at which the accumulator layout
changes (16, 17, 48, 49, 64, 65, 80, 96, 128), atoms of unequal size in one tile, NAO totals that are
not a multiple of 4, and cell counts on both sides of the shift table's 32.

Tolerance.  A chi0 entry sums K = n_cells n_ao products per j; the contraction rounds to FP32 after every
64 of them, once per piece of the split and once per row q <= 2 * 32 of E, and X = C G once per 64 of its
K: below 64 + 64 + 3 + K/64 roundings of 2^-24, under 300 for the sizes here.  300 * 2^-24 = 1.8e-5,
relative to the largest entry."""
import numpy as np
import pytest

import librpa_gb300 as L
from librpa_gb300.synthetic import small_periodic

pytestmark = pytest.mark.gpu
TOL = 300 * 2.0 ** -24


def _chi0(s, prec):
    with L.Handler() as h:
        L.load_system(h, s)
        h.set_gb300_options(L.gb300_options(chi0_precision=prec, stage=L.STAGE_CHI0))
        o = L.Options(nfreq=6, tfgrids_type=L.Minimax, parallel_routing=L.LIBRI, minimax_emin=s.minimax_emin,
                      minimax_emax=s.minimax_emax)
        h.get_rpa_correlation_energy(o, L.n_ibz(s))
        assert h.stats()["chi0_precision_used"] == prec
        return h.chi0_qw()


@pytest.mark.parametrize("nao,nabf,period", [
    ([4, 5], [16, 17], (1, 1, 1)),
    ([8, 9], [48, 15], (2, 1, 1)),
    ([12, 13], [49, 40], (1, 1, 1)),
    ([14, 15, 3], [64, 20, 9], (1, 2, 1)),
    ([16, 17], [65, 33], (1, 1, 1)),
    ([32, 2], [128, 5], (1, 1, 1)),
    ([26, 13, 5], [96, 60, 20], (1, 1, 1)),
    ([10, 11], [80, 130 - 2], (3, 1, 1)),
    ([5], [7], (4, 4, 2)),
    ([3], [6], (3, 11, 1)),
    ([1, 2], [1, 2], (1, 1, 1)),
])
def test_chi0_tile_edges(nao, nabf, period):
    s = small_periodic(len(nao), nao, nabf, period, nocc=1, seed=11)
    ref, got = _chi0(s, L.CHI0_FP64), _chi0(s, L.CHI0_BF16X3)
    assert np.isfinite(got).all()
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
