"""The eigensolver's blocks of several matrices: sizes that leave lanes, pairs and
warps part-filled, batches on both sides of the line at which matrices are taken
together and with a last block that is not full.  Energies against the oracle
within 1e-10 eV, sum_b E_b v_b v_b^H likewise, eigenvectors orthonormal to 1e-12.
"""
import numpy as np
import pytest

from elphbolt_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw", [2, 3, 6, 7, 8, 9, 12, 13, 16, 24, 31, 32])
def test_eigensolver_batches(oracle_lib, nw):
    from elphbolt_gb300.build import build
    from elphbolt_gb300.wannier import Wannier
    build()
    wd = S.make_wannier(S.make_crystal_si_like(), nw, supercell=(2, 2, 2), seed=50 + nw)
    ks = np.random.default_rng(nw).uniform(-1, 1, (1219, 3))
    ks[5] = 0
    eo, vo, _ = oracle_lib.Wannier(wd).el_wann(ks)
    W = Wannier(wd)
    for nk in (1, 3, 1215, 1216, 1217, 1219):
        e, v = W.el_wann(kvecs=ks[-nk:], evecs=True)
        assert np.max(np.abs(e - eo[-nk:])) <= 1e-10
        assert np.max(np.abs(np.einsum("kbi,kci->kbc", v.conj(), v) - np.eye(nw))) <= 1e-12
        for i in (0, nk // 2, nk - 1):
            H, Ho = ((w[i].T * x[i]) @ w[i].conj() for w, x in ((v, e), (vo[-nk:], eo[-nk:])))
            assert np.max(np.abs(H - Ho)) <= 1e-10
    W.deallocate_wannier()
