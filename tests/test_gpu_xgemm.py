"""FP64 products by exact splitting (g(k,Rp), g(Re,q), |g|^2 lists) against sums in
extended precision: phase rows around the chunks of 32 and the MMA widths, column
counts and cell counts that leave tiles ragged, more cells than one accumulation
holds, columns of very different magnitude, and non-finite values.

Tolerance, derived: the split sum is exact to ~2^-60 of the largest product and
rounded once, 2^-53 of the result.  The k-points are multiples of 1/64, so k.R is
exact and the reference's phases are exact to extended precision; the library's
are products of three table entries of error 2^-53 each, two complex products and
a scaling, under 9 2^-53 in all.  So each element is within 12 2^-53
sum_R |phase_R| |x_R|.
"""
import dataclasses

import numpy as np
import pytest

from elphbolt_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def W_of():
    from elphbolt_gb300.build import build
    from elphbolt_gb300.wannier import Wannier
    build()
    made = []

    def make(wd):
        W = Wannier(wd)
        made.append(W)
        return W
    yield make
    for W in made:
        W.deallocate_wannier()


def crystal(kind):
    if kind == "odd":      # nw 5, nb 9: 225 columns per cell
        return S.make_wannier(S.make_crystal_multi(3, np.random.Generator(np.random.PCG64(7))), 5, supercell=(2, 2, 3),
                              seed=13)
    if kind == "long":     # more cells than one accumulation of 320
        return S.make_wannier(S.make_crystal_si_like(), 2, supercell=(7, 7, 7), seed=3)
    return S.make_wannier(S.make_crystal_si_like(), 4, supercell=(3, 3, 3), seed=21)


def phases(k, R, deg):
    a = (k @ R.T) % 1.0 * (2 * np.longdouble("3.14159265358979323846264338327950288"))   # exact up to the last product
    return (np.cos(a) + 1j * np.sin(a)) / deg.astype(np.longdouble)


def check(out, ph, x):
    """out (n, ...), ph (n, R), x (R, ...)"""
    ref = np.tensordot(ph.astype(np.clongdouble), x.astype(np.clongdouble), axes=(1, 0))
    tol = 12 * 2.0 ** -53 * np.tensordot(np.abs(ph), np.abs(x.real) + np.abs(x.imag), axes=(1, 0))
    d = (out - ref).astype(np.complex128)
    assert np.all(np.abs(d.real) <= tol) and np.all(np.abs(d.imag) <= tol)


def points(n):
    k = np.round(np.random.default_rng(n).uniform(0, 1, (n, 3)) * 64) / 64   # k.R exact: the same arguments on both sides
    k[0] = 0
    return k


@pytest.mark.parametrize("kind,n", [("odd", 1), ("odd", 8), ("odd", 9), ("odd", 33), ("even", 31), ("even", 32),
                                    ("even", 70), ("long", 5)])
def test_gkRp_gReq(W_of, kind, n):
    wd = crystal(kind)
    if kind == "even":     # columns over 60 orders of magnitude, and an empty one
        g = wd.gwann * (10.0 ** np.linspace(-30, 30, wd.nwsq))
        g[0, 0, :, 0, 0] = 0.0
        wd = dataclasses.replace(wd, gwann=np.asfortranarray(g))
    W = W_of(wd)
    k = points(n)
    g = wd.gwann           # (i, j, Re, s, Rp)
    out = W.gkRp(kvec=k)   # (i, j, s, Rp, n)
    check(np.moveaxis(out, -1, 0), phases(k, wd.rcells_k, wd.elwsdeg), np.moveaxis(g, 2, 0))
    out = W.gReq(qvec=k)   # (i, j, s, Re, n)
    check(np.moveaxis(out, -1, 0), phases(k, wd.rcells_g, wd.gwsdeg), np.moveaxis(g, [4, 2], [0, 4]))


def test_non_finite_values_stay_in_their_columns(W_of):
    wd = crystal("even")
    g = wd.gwann.copy(order="F")
    g[1, 2, 5, 3, 7] = np.nan
    g[0, 1, 4, 2, 6] = np.inf
    out = W_of(dataclasses.replace(wd, gwann=g)).gkRp(kvec=points(3))
    bad = ~np.isfinite(out)
    expect = np.zeros(out.shape, dtype=bool)
    expect[1, 2, 3, 7] = expect[0, 1, 2, 6] = True
    assert np.array_equal(bad, expect)


@pytest.mark.parametrize("nv,ngm,side", [(1, 1, "ph"), (33, 1, "el"), (97, 5, "ph"), (40, 60, "el")])
def test_g2_groups(W_of, nv, ngm, side):
    """Vertices in any order of their blocks, blocks no vertex uses, chunks of 1 to 32."""
    wd = crystal("odd")
    W = W_of(wd)
    rng = np.random.default_rng(nv)
    nw, nb, nws = 5, 9, wd.nwsk

    def c(*shape):
        return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    gm = c(nw, nw, nb, nws, ngm)
    ek, ekp, eq = c(nv, nw), c(nv, nw), c(nv, nb)
    k, q = points(nv), points(nv + 1)[1:]
    en = rng.uniform(0.01, 0.05, nv)
    en[0] = 0.0 if nv > 1 else en[0]
    gi = rng.integers(1, ngm + 1, nv)
    out = W.g2_batch(k, q, ek, ekp, eq, en, gm, gi, wannspace=side)
    ph = phases(q if side == "ph" else k, wd.rcells_q, wd.phwsdeg)
    m = np.sqrt(np.repeat(wd.crystal.masses, 3))
    g = np.einsum("vr,ijsrv,vj,vi,vs->v", ph, gm[..., gi - 1], ek, ekp.conj(), eq / m)
    with np.errstate(divide="ignore"):
        ref = np.where(en == 0, 0.0, 0.5 * np.abs(g) ** 2 / en * S.C.g2unitfactor)
    # FP64 rotations of ~nw nw nb terms: 1e-12 of the result's scale
    scale = 0.5 * np.einsum("vr,ijsrv,vj,vi,vs->v", np.abs(ph), np.abs(gm[..., gi - 1]), np.abs(ek), np.abs(ekp),
                            np.abs(eq) / m) ** 2 / np.where(en == 0, 1.0, en) * S.C.g2unitfactor
    assert np.all(np.abs(out - ref) <= 1e-13 * scale)
