"""The FP64 epilogue's groups of final states: windows of one state to several thousand,
whose groups hold one final state or several and end full or ragged, for few initial
states (a wedge) as for all.  Every rate is the sum of its vertices' X+ and X-,
formed in compensated FP64 but for the sum over the modes of a vertex: within
(nb + 4) 2^-53 of the exact sum of the listed values.
"""
import math

import numpy as np
import pytest

from elphbolt_gb300 import _lib, synthetic as S, symmetry as Y

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def W():
    from elphbolt_gb300.build import build
    from elphbolt_gb300.wannier import Wannier
    build()
    w = Wannier(S.make_wannier(S.make_crystal_si_like(), 2, supercell=(2, 2, 2), seed=3))
    yield w
    w.deallocate_wannier()


# final states: 1 to 2 bands of every point; the group's size is about a 512th of them
@pytest.mark.parametrize("delta,prec", [(0, _lib.PREC_FP64), (2, _lib.PREC_FP64), (2, _lib.PREC_SPLIT_TF32)])
@pytest.mark.parametrize("mesh,wedge", [((2, 1, 1), False), ((5, 5, 5), False), ((8, 8, 4), False), ((8, 8, 8), True),
                                        ((9, 9, 9), True), ((11, 11, 11), True), ((12, 12, 12), True)])
def test_rates_are_the_sums_of_their_vertices(W, mesh, wedge, delta, prec):
    e = W.el_wann(kvecs=S.mesh_kvecs(mesh))
    mid = float(np.median(e))
    req = S.RateRequest(mesh=mesh, enref=mid, fsthick=1.0 + float(np.abs(e - mid).max()), chempot=mid, T=300.0,
                        delta_kind=delta, sigma=0.05)
    W.set_symmetry(Y.crystal_symmetry(S.make_crystal_si_like())[0] if wedge else None)
    try:
        o = W.el_rates(req, precision=prec, vertices=True, cap=12_000_000)
    finally:
        W.set_symmetry(None)
    nin = 2 * int(np.prod(mesh))
    assert o["stats"]["nstates_inwindow"] == nin and o["vertices"] == o["nstates"] * nin * 6 <= 12_000_000
    x = np.stack([o["xp"], o["xm"]], axis=1).reshape(o["nstates"], -1)
    ref = np.array([math.fsum(r) for r in x])
    assert np.all(np.abs(o["rates"].ravel() - ref) <= (6 + 4) * 2.0**-53 * ref)
