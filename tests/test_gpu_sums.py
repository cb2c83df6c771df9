"""The FP64 rate path's Fourier sums over cells, one dimension at a time, on their own (the
requests of small meshes take the product with the phases): meshes of one, two, odd and
even points per dimension (mirrored outputs v and m - v, the unpaired v = 0 and
v = m / 2), cells not symmetric about zero, with gaps, one only, more than the mesh
has points; some or all rows; columns around a block's 128.

Tolerance, derived: a dimension's sum over its h = max |r| pairs is a chain of h + 2
roundings of terms that a root of 2^-53 relative error multiplies; a scaling and the
three dimensions in all: sum_d (2 h_d + 6) 2^-53 of the sum of magnitudes.
"""
import ctypes as ct

import numpy as np
import pytest

from elphbolt_gb300 import _lib

pytestmark = pytest.mark.gpu


def cells_of(kind):
    if kind == "one":
        return np.zeros((1, 3), dtype=np.int64)
    box = np.array([(i, j, k) for i in range(-3, 4) for j in range(-2, 3) for k in range(-4, 5)])
    if kind == "ball":
        return box[(box**2 @ [1, 1, 1]) <= 12]
    if kind == "box":
        return box
    r = box[box[:, 0] >= 0] * [1, 3, 1] + [2, 0, -3]      # from 2 up, every third, from -7 up to 1
    return r[np.random.default_rng(1).permutation(len(r))[:70]]


@pytest.fixture(scope="module")
def lib():
    from elphbolt_gb300.build import build
    build()
    L = _lib.load()
    L.ephg_debug_cells_fourier.argtypes = [ct.c_int64, _lib.c_i64p, _lib.c_dp, _lib.c_i64p, ct.c_int64, _lib.c_dp,
                                           ct.c_int64, _lib.c_i64p, _lib.c_dp]
    L.ephg_debug_cells_fourier.restype = ct.c_int
    return L


def p(a, t=_lib.c_dp):
    return None if a is None else a.ctypes.data_as(t)


@pytest.mark.parametrize("nc,share,scaled", [(1, 1.0, False), (127, 0.3, True), (130, 1.0, True)])
@pytest.mark.parametrize("mesh", [(1, 1, 7), (2, 3, 5), (6, 2, 1), (4, 4, 4), (9, 3, 2), (13, 12, 10)])
@pytest.mark.parametrize("kind", ["one", "ball", "box", "shifted"])
def test_sums(lib, kind, mesh, nc, share, scaled):
    R = np.asfortranarray(cells_of(kind))
    rng = np.random.default_rng(nc)
    x = rng.standard_normal((len(R), nc)) + 1j * rng.standard_normal((len(R), nc))
    scale = 1.0 / rng.integers(1, 7, len(R)) if scaled else None
    N = int(np.prod(mesh))
    rows = np.sort(rng.permutation(N)[:max(1, int(share * N))]).astype(np.int64)
    out = np.full((len(rows), nc), np.nan, dtype=np.complex128)
    m = np.array(mesh, dtype=np.int64)
    rc = lib.ephg_debug_cells_fourier(len(R), p(R, _lib.c_i64p), p(scale), p(m, _lib.c_i64p), nc, p(x), len(rows),
                                      p(rows, _lib.c_i64p), p(out))
    assert rc == _lib.EPHG_OK, lib.ephg_last_error()
    k = np.stack([rows % m[0], rows // m[0] % m[1], rows // (m[0] * m[1])], axis=1)
    frac = sum(((k[:, d:d + 1] * R[:, d]) % m[d]).astype(np.longdouble) / int(m[d]) for d in range(3))
    a = frac * (2 * np.longdouble("3.14159265358979323846264338327950288"))
    w = np.ones(len(R)) if scale is None else scale
    ref = (np.cos(a) + 1j * np.sin(a)) @ (w[:, None] * x.astype(np.clongdouble))
    tol = (np.sum(2 * np.abs(R).max(axis=0)) + 18) * 2.0**-53 * (w @ (np.abs(x.real) + np.abs(x.imag)))
    d = (out - ref).astype(np.complex128)
    assert np.all(np.abs(d.real) <= tol) and np.all(np.abs(d.imag) <= tol)
