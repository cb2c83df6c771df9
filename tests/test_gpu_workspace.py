"""The workspace of a split Gaussian request: linear in the mesh points at a given number
of bands in the window, but for the rate partials, one per state and 32 rows.  With
all eight bands of 14^3 points in the window these are 15 MB; one per state and 16
final states would be 241 MB.
"""
import numpy as np
import pytest

from elphbolt_gb300 import _lib, synthetic as S

pytestmark = pytest.mark.gpu


def test_wide_window():
    from elphbolt_gb300.build import build
    from elphbolt_gb300.wannier import Wannier, el_rates_batch
    build()
    W = Wannier(S.make_wannier(S.make_crystal_si_like(), 8, supercell=(2, 2, 2), seed=4))
    peak = {}
    try:
        e = W.el_wann(kvecs=S.mesh_kvecs((14, 14, 14)))
        mid = float(np.median(e))
        for m1 in (7, 14):
            req = S.RateRequest(mesh=(m1, 14, 14), enref=mid, fsthick=1.0 + float(np.abs(e - mid).max()), chempot=mid,
                                T=300.0)
            (out,), stats, _ = el_rates_batch([W], [req], precision=_lib.PREC_SPLIT_TF32, nslots=1)
            assert out["nstates"] == 8 * m1 * 14 * 14
            peak[m1] = stats["peak_workspace_bytes"]
    finally:
        W.deallocate_wannier()
    # rounding up to tiles, and constants, only make twice the half mesh's the larger one
    partials = 8 * 14**3 * (-(-14**3 // 256) * 8) * 8
    assert peak[14] <= 2 * peak[7] + partials, (peak[14] - 2 * peak[7], partials)
