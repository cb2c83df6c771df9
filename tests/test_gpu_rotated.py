"""The generic split form's second stage, which rotates its accumulators to the
bands of the window before it writes them: against the FP64 form on meshes whose
rows, positions and window states end inside a tile, a 32-row group and a block,
with one band of the window and with all of them, from the electrons' and the
phonons' side.  Vertices within 1e-5, the split form's bound; rates as the sums
of the vertices, formed in FP32.
"""
import numpy as np
import pytest

from elphbolt_gb300 import _lib, synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", [4.0, 0.08])
@pytest.mark.parametrize("mesh", [(1, 1, 7), (3, 5, 2), (5, 7, 6)])
@pytest.mark.parametrize("nw,nat", [(8, 3), (8, 4), (8, 6), (16, 2), (16, 4), (24, 2), (32, 2)])
def test_rotated(oracle_lib, nw, nat, mesh, window):
    from elphbolt_gb300.build import build
    from elphbolt_gb300.wannier import Wannier
    build()
    crys = S.make_crystal_si_like() if nat == 2 else \
        S.make_crystal_multi(nat, np.random.Generator(np.random.PCG64(nat)))
    wd = S.make_wannier(crys, nw, supercell=(2, 2, 3), seed=31)
    e = np.sort(oracle_lib.Wannier(wd).el_wann(S.mesh_kvecs(mesh))[0].ravel())
    mu = float(e[len(e) // 2]) + 0.01     # some state is in every window
    req = S.RateRequest(mesh=mesh, enref=mu, fsthick=window, chempot=mu, T=300.0, sigma=0.05)

    W = Wannier(wd)
    (a, pa), (b, pb) = ((W.el_rates(req, precision=p, vertices=True, cap=400000),
                         W.ph_rates(req, precision=p, electrons=True, vertices=True, cap=400000))
                        for p in (_lib.PREC_SPLIT_TF32, _lib.PREC_FP64))
    W.deallocate_wannier()
    for x, y, keys in ((a, b, ("g2", "xp", "xm")), (pa, pb, ("g2", "y"))):
        for key in keys:
            assert x[key].shape == y[key].shape
            assert np.all(np.abs(x[key] - y[key]) <= 1e-5 * np.abs(y[key]) + 1e-6 * np.max(np.abs(y[key]), initial=0))
    if a["vertices"] > 400000:
        return
    # a state's rate is the sum of its vertices' X+ and X-: in FP32 over a row's positive terms
    rows = [np.sort((o["xp"] + o["xm"]).reshape(o["nstates"], -1).sum(axis=1)) for o in (a, b)]
    rates = [np.sort(o["rates"][o["rates"] > 0]) for o in (a, b)]
    unit = rates[1].sum() / rows[1].sum()
    rows = rows[0][rows[0] > 0] * unit
    assert np.all(np.abs(rates[0] - rows) <= (nw * wd.numbranches + 8) * 2.0**-24 * rows)
