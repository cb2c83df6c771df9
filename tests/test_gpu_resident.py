"""A crystal's resident device data is complete when its handle is: no call adds to
it afterwards, so that the serving loop's budget, checked at its creation and
against its slots' workspaces, covers everything.  Checked by the smallest budget
that a server accepts for the crystal, before and after a call of every entry
point that multiplies by a resident operand.
"""
import numpy as np
import pytest

from elphbolt_gb300 import _lib, synthetic as S
from tests.cases import case

pytestmark = pytest.mark.gpu


def smallest_budget(W):
    from elphbolt_gb300.serve import Server
    lo, hi = 0, 1 << 30
    while hi - lo > 1:
        mid = (lo + hi) // 2
        try:
            Server([W], hbm_budget_bytes=mid).close()
            hi = mid
        except _lib.EphgError:
            lo = mid
    return hi


def test_calls_add_nothing_to_the_resident_data():
    from elphbolt_gb300.build import build
    from elphbolt_gb300.wannier import Wannier
    build()
    wd, req = case("tiny")
    W = Wannier(wd)
    try:
        before = smallest_budget(W)
        k = np.array([[0.1, 0.2, 0.3]])
        W.el_wann(kvecs=k, velocities=True)
        W.ph_wann(qvecs=k, velocities=True)
        W.gkRp(kvec=k)
        W.gReq(qvec=k)
        e = float(np.sort(W.el_wann(kvecs=S.mesh_kvecs(req.mesh)).ravel())[0])
        for window in ({}, dict(enref=e, fsthick=1e-6)):   # sums and, for the few rows of one state, products
            W.el_rates(S.RateRequest(**{**req.__dict__, **window}), precision=_lib.PREC_FP64)
        assert smallest_budget(W) == before
    finally:
        W.deallocate_wannier()
