"""Half-transformed vertices at arbitrary k against sums in extended precision (the lists
of tests/test_gpu_xgemm.py have k.R exact).

Tolerance, derived: beside the 12 2^-53 per term of an exact k.R, the library rounds
k_d R_d once per dimension to FP64, an angle error of up to 2 pi 2^-53 |k_d R_d| each.
The reference's k.R is exact to 2^-62: products of 53 bits with R below 2^9 fit
extended precision's 64.
"""
import numpy as np
import pytest

from elphbolt_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,span", [(3, 0.5), (25, 1.0), (40, 7.0)])
def test_arbitrary_k(n, span):
    from elphbolt_gb300.build import build
    from elphbolt_gb300.wannier import Wannier
    build()
    wd = S.make_wannier(S.make_crystal_si_like(), 4, supercell=(4, 4, 4), seed=6)
    k = np.asfortranarray(np.random.default_rng(n).uniform(-span, span, (n, 3)))
    W = Wannier(wd)
    outs = [(W.gkRp(kvec=k), wd.rcells_k, wd.elwsdeg, np.moveaxis(wd.gwann, 2, 0)),
            (W.gReq(qvec=k), wd.rcells_g, wd.gwsdeg, np.moveaxis(wd.gwann, [4, 2], [0, 4]))]
    W.deallocate_wannier()
    for out, R, deg, x in outs:
        kr = k.astype(np.longdouble) @ R.T.astype(np.longdouble)
        a = (kr - np.round(kr)) * (2 * np.longdouble("3.14159265358979323846264338327950288"))
        ph = (np.cos(a) + 1j * np.sin(a)) / deg.astype(np.longdouble)
        ref = np.tensordot(ph, x.astype(np.clongdouble), axes=(1, 0))
        term = (12 + 2 * np.pi * (np.abs(k) @ np.abs(R).T)) * 2.0**-53 / deg
        tol = np.tensordot(term, np.abs(x.real) + np.abs(x.imag), axes=(1, 0))
        d = (np.moveaxis(out, -1, 0) - ref).astype(np.complex128)
        assert np.all(np.abs(d.real) <= tol) and np.all(np.abs(d.imag) <= tol)
