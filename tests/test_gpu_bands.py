"""FP64 rates against the oracle for numbers of bands on both sides of every capacity of
the stage-A rotation (multiples of 4), few and many states per k-point.  Rates
within 1e-10 relative, the FP64 form's bound.
"""
import numpy as np
import pytest

from elphbolt_gb300 import _lib, synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw", [2, 3, 4, 5, 8, 9, 12, 13, 16, 17, 20, 21, 24, 25, 28, 29, 32])
def test_band_counts(oracle_lib, nw):
    from elphbolt_gb300.build import build
    from elphbolt_gb300.wannier import Wannier
    build()
    mesh = (3, 2, 2)
    wd = S.make_wannier(S.make_crystal_si_like(), nw, supercell=(2, 2, 2), seed=nw)
    O = oracle_lib.Wannier(wd)
    e = O.el_wann(S.mesh_kvecs(mesh))[0]
    mid = float(np.median(e)) + 0.003
    d = np.sort(np.abs(e - mid).ravel())
    win = float(0.5 * (d[min(len(d), 40) - 1] + d[min(len(d) - 1, 40)])) + (0.01 if len(d) <= 40 else 0.0)
    req = S.RateRequest(mesh=mesh, enref=mid, fsthick=win, chempot=mid, T=300.0, sigma=0.1)
    ref = O.el_rates(req)
    W = Wannier(wd)
    out = W.el_rates(req, precision=_lib.PREC_FP64)
    W.deallocate_wannier()
    assert np.array_equal(out["indexlist"], ref["indexlist"])
    m = ref["rates"] > 0
    assert m.any() and np.all(out["rates"][~m] == 0)
    assert np.max(np.abs(out["rates"][m] - ref["rates"][m]) / ref["rates"][m]) <= 1e-10
