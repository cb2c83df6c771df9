"""|g|^2 lists whose vertices all have a block of their own: more chunks than one
launch takes, so that the list runs in pieces, in device memory that is bounded
whatever the number of cells and blocks: beside the inputs, the phases, the cell
sums and the digits hold at most 256 MB each.

Tolerance as for the lists of a few blocks: FP64 rotations, 1e-13 of the sum of
magnitudes.
"""
import numpy as np
import pytest

from elphbolt_gb300 import _lib, synthetic as S

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_a_block_per_vertex():
    torch = pytest.importorskip("torch")
    from elphbolt_gb300.build import build
    from elphbolt_gb300.wannier import Wannier
    build()
    L = _lib.load()
    wd = S.make_wannier(S.make_crystal_si_like(), 2, supercell=(8, 8, 8), seed=3)   # 617 cells
    n, nw, nb, nws = 1500, 2, 6, wd.nwsk
    rng = np.random.default_rng(5)

    def c(*shape):
        return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    gm = np.asfortranarray(c(nw, nw, nb, nws, n))
    ek, ekp, eq = c(n, nw), c(n, nw), c(n, nb)
    q = np.round(rng.uniform(0, 1, (n, 3)) * 64) / 64     # q.R exact
    en = rng.uniform(0.01, 0.05, n)
    gi = rng.permutation(n) + 1
    W = Wannier(wd)
    try:
        W.g2_batch(q[:1], q[:1], ek[:1], ekp[:1], eq[:1], en[:1], gm[..., :1], [1])   # first-use allocations
        assert L.ephg_trim_memory() == _lib.EPHG_OK
        free0 = torch.cuda.mem_get_info()[0]
        out = W.g2_batch(q, q, ek, ekp, eq, en, gm, gi)
        used = free0 - torch.cuda.mem_get_info()[0]
    finally:
        W.deallocate_wannier()
    a = (q @ wd.rcells_q.T) % 1.0
    ph = np.exp(2j * np.pi * a) / wd.phwsdeg
    g = np.array([np.einsum("r,ijsr,j,i,s", ph[v], gm[..., gi[v] - 1], ek[v], ekp[v].conj(),
                            eq[v] / np.sqrt(np.repeat(wd.crystal.masses, 3)), optimize=True) for v in range(n)])
    mag = np.array([np.einsum("r,ijsr,j,i,s", np.abs(ph[v]), np.abs(gm[..., gi[v] - 1]), np.abs(ek[v]), np.abs(ekp[v]),
                              np.abs(eq[v]) / np.sqrt(np.repeat(wd.crystal.masses, 3)), optimize=True) for v in range(n)])
    assert np.all(np.abs(out - 0.5 * g.real**2 / en * S.C.g2unitfactor - 0.5 * g.imag**2 / en * S.C.g2unitfactor)
                  <= 1e-13 * 0.5 * mag**2 / en * S.C.g2unitfactor)
    assert used <= gm.nbytes + 3 * 256 * MB + 64 * MB     # 64 MB: the lists and the pool's granularity
