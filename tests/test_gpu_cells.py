"""The FP64 rate path's Fourier sums over cells, one dimension at a time, and the
tabulated simplex deltas, against the oracle: meshes of one, two, odd and uneven points per dimension (mirrored
outputs v and m - v, the unpaired v = 0 and v = m / 2), cell ranges that are not
symmetric about zero, more cells than mesh points, and windows so narrow that
the contractions run as matrix products.  Rates within 1e-10 relative, the FP64
form's bound.
"""
import dataclasses

import numpy as np
import pytest

from elphbolt_gb300 import _lib, synthetic as S

pytestmark = pytest.mark.gpu


def crystal(kind):
    if kind == "odd":       # nw 5, nb 9, uneven supercell
        return S.make_wannier(S.make_crystal_multi(3, np.random.Generator(np.random.PCG64(7))), 5, supercell=(2, 2, 3),
                              seed=13)
    wd = S.make_wannier(S.make_crystal_si_like(), 4, supercell=(3, 3, 3), seed=21)
    if kind == "shifted":   # vertex cells from zero up in one dimension, with gaps in another
        keep = wd.rcells_q[:, 0] >= 0
        R = wd.rcells_q[keep] * np.array([1, 2, 1])
        D = np.zeros_like(wd.Dphwann[keep])   # on-site springs only: the same positive phonons at every q
        D[np.flatnonzero(~R.any(axis=1))[0]] = np.diag(np.linspace(0.02, 0.2, wd.numbranches))
        return dataclasses.replace(wd, rcells_q=R, rcells_g=R.copy(), Dphwann=np.asfortranarray(D),
                                   phwsdeg=wd.phwsdeg[keep], gwsdeg=wd.gwsdeg[keep],
                                   gwann=np.asfortranarray(wd.gwann[..., keep]))
    return wd


@pytest.mark.parametrize("window", [4.0, 0.08])
@pytest.mark.parametrize("mesh", [(1, 1, 7), (2, 3, 5), (6, 2, 1), (4, 4, 4), (9, 3, 2)])
@pytest.mark.parametrize("kind", ["sym", "odd", "shifted"])
def test_fp64_rates(oracle_lib, kind, mesh, window):
    from elphbolt_gb300.build import build
    from elphbolt_gb300.wannier import Wannier
    build()
    wd = crystal(kind)
    k = np.linspace(0, 1, int(np.prod(mesh)), endpoint=False)
    O = oracle_lib.Wannier(wd)
    e = O.el_wann(S.mesh_kvecs(mesh))[0]
    mu = float(np.sort(e.ravel())[len(k) * wd.numwannbands // 2]) + 0.01     # some state is in every window
    req = S.RateRequest(mesh=mesh, enref=mu, fsthick=window, chempot=mu, T=300.0, sigma=0.05)
    ref = O.el_rates(req)
    W = Wannier(wd)
    out = W.el_rates(req, precision=_lib.PREC_FP64)
    W.deallocate_wannier()
    assert np.array_equal(out["indexlist"], ref["indexlist"])
    m = ref["rates"] > 0
    assert np.all(out["rates"][~m] == 0)
    assert np.max(np.abs(out["rates"][m] - ref["rates"][m]) / ref["rates"][m], initial=0.0) <= 1e-10


@pytest.mark.parametrize("delta", [1, 2])
@pytest.mark.parametrize("mesh", [(1, 1, 7), (2, 3, 5), (6, 2, 1), (5, 4, 3)])
def test_simplex_rates(oracle_lib, mesh, delta):
    """Triangle / tetrahedron deltas on meshes whose cells wrap onto themselves (a
    corner then appears several times in one simplex), windows that cut simplices
    (corners outside count as zero energy) and the phonon side, whose delta sits
    at the initial state."""
    from elphbolt_gb300.build import build
    from elphbolt_gb300.wannier import Wannier
    build()
    wd = crystal("odd")
    O = oracle_lib.Wannier(wd)
    e = np.sort(O.el_wann(S.mesh_kvecs(mesh))[0].ravel())
    mu = float(e[len(e) // 2]) + 0.01
    W = Wannier(wd)
    for window in (4.0, 0.7):
        req = S.RateRequest(mesh=mesh, enref=mu, fsthick=window, chempot=mu, T=300.0, delta_kind=delta)
        ref = O.el_rates(req)["rates"]
        refp = O.ph_rates(req, spindeg=2)["rates_phe"]
        out = W.ph_rates(req, precision=_lib.PREC_FP64, electrons=True)
        for a, b in ((out["rates"], ref), (out["rates_phe"], refp)):
            assert np.max(np.abs(a - b)) <= 1e-10 * np.max(np.abs(b), initial=0.0)
    W.deallocate_wannier()
