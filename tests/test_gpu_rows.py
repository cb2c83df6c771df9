"""A k- or q-point's results are the same bits whatever other points share its call:
rows at the edges of the products' chunks (8 and 32 rows) and widths, and on both
sides of the 4,096 rows of one launch.  Degenerate eigenvectors would otherwise come
in another gauge from another call.
"""
import numpy as np
import pytest

from elphbolt_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def W():
    from elphbolt_gb300.build import build
    from elphbolt_gb300.wannier import Wannier
    build()
    w = Wannier(S.make_wannier(S.make_crystal_si_like(), 4, supercell=(3, 3, 3), seed=21))
    yield w
    w.deallocate_wannier()


K = np.random.default_rng(8).uniform(0, 1, (4100, 3))
SPANS = [(0, 1), (0, 7), (0, 9), (3, 24), (0, 25), (0, 33), (100, 300), (4090, 4097), (4096, 4100)]


def test_bands_and_phonons(W):
    for f in (lambda k: W.el_wann(kvecs=k, velocities=True, evecs=True),
              lambda k: W.ph_wann(qvecs=k, velocities=True, evecs=True)):
        whole = f(K)
        for a, b in SPANS:
            for x, y in zip(f(np.asfortranarray(K[a:b])), whole):
                assert np.array_equal(x, y[a:b]), (a, b)


def test_half_transformed_vertices(W):
    for f in (lambda k: W.gkRp(kvec=k), lambda k: W.gReq(qvec=k)):
        whole = f(K[:70])
        for a, b in SPANS[:6]:
            assert np.array_equal(f(np.asfortranarray(K[a:b])), whole[..., a:b]), (a, b)
