"""Polar phonons with velocities at arbitrary q against the oracle: crystals whose
sums fill part of a block, all of it (5 atoms: 120 Hermitian elements) and more
than one element per thread (6 and 10 atoms), a dielectric tensor that is not a
multiple of the unit one.  Frequencies within 1e-10, velocities within 1e-7 of the
largest, with and without the velocities asked for.
"""
import dataclasses

import numpy as np
import pytest

from elphbolt_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


def polar_crystal(nat):
    rng = np.random.Generator(np.random.PCG64(nat))
    crys = S.make_crystal_multi(nat, rng)
    born = rng.uniform(-0.1, 0.1, (3, 3, nat)) + 0.2 * np.eye(3)[:, :, None] * (-1.0) ** np.arange(nat)
    born -= born.mean(axis=2, keepdims=True)     # neutral
    eps = 7.0 * np.eye(3) + np.array([[0.5, 0.3, 0.1], [0.3, -0.4, 0.2], [0.1, 0.2, 0.0]])
    crys = dataclasses.replace(crys, polar=True, epsilon=eps, born=np.asfortranarray(born))
    return S.make_wannier(crys, 2, supercell=(3, 2, 2), seed=nat, spring_range=(30.0, 60.0))


@pytest.mark.parametrize("nat", [2, 3, 5, 6, 10])
def test_polar_velocities(oracle_lib, nat):
    from elphbolt_gb300.build import build
    from elphbolt_gb300.wannier import Wannier
    build()
    wd = polar_crystal(nat)
    qs = np.random.default_rng(2).uniform(0, 1, (23, 3))
    eo, _, vo, st = oracle_lib.Wannier(wd).ph_wann(qs, velocities=True)
    assert st == 0
    W = Wannier(wd)
    e, v = W.ph_wann(qvecs=qs, velocities=True)
    e0 = W.ph_wann(qvecs=qs)
    W.deallocate_wannier()
    assert np.max(np.abs(e - eo)) <= 1e-10 and np.max(np.abs(e0 - eo)) <= 1e-10
    assert np.max(np.abs(v - vo)) <= 1e-7 * np.max(np.abs(vo))
