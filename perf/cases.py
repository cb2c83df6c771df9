"""The work that users of the e-ph vertex library have it do, as measurable cases.

Each case is one pass through a public entry point of ``elphbolt_gb300`` (the
Python mirror of the C ABI), on seeded synthetic crystals in the reference's
layouts.  A handle (``Wannier``) is what a program keeps: ``prepare`` makes it,
``run`` calls it with host arrays, as every caller of the C ABI does.

Kinds:

* ``bands``    ``el_wann`` at arbitrary k (band paths, random fine points)
* ``phonons``  ``ph_wann`` at arbitrary q or on a mesh, polar or not
* ``gkRp``, ``gReq``  the half-transformed vertices of the IBZ points
* ``g2``       |g|^2 of a vertex list from given half-transformed vertices
* ``rates``    a whole RTA-rate request (``el_rates``, ``el_rates_sets`` or
  ``ph_rates``): FP64 drop-in or split form, Gaussian / triangle / tetrahedron
* ``batch``    many requests on several crystals in one call

``exact`` restates what each returns in 64 bits with numpy and torch alone: the
Fourier sums on a mesh as FFTs of the folded cells, LAPACK eigensolvers, and
every vertex formula written out.
"""
import functools
import math

import numpy as np
import torch

from elphbolt_gb300 import _lib, synthetic as S
from elphbolt_gb300.wannier import Wannier, el_rates_batch

FP64, SPLIT = _lib.PREC_FP64, _lib.PREC_SPLIT_TF32


# ------------------------------------------------------------------ cases
def _rates(name, mesh, nw=8, nat=2, cells=6, split=True, delta=0, polar=False, ph=False, sets=1, window=0.5,
           T=300.0, sigma=0.010):
    c = dict(kind="rates", m1=mesh[0], m2=mesh[1], m3=mesh[2], nw=nw, nat=nat, cells=cells, split=split, delta=delta,
             polar=polar, ph=ph, sets=sets, window=window, T=T, sigma=sigma)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a band-structure path: a few hundred k-points, energies and velocities (smallest calls: latency)
        dict(name="bands_path", kind="bands", nw=8, nat=2, cells=6, n=200, vel=True),
        # the phonon set-up of a polar crystal (phonon.f90:208-214): the whole 12^3 q mesh, with velocities
        dict(name="phonons_polar_mesh", kind="phonons", nw=4, nat=2, cells=6, n=1728, vel=True, polar=True),
        # calculate_gkRp / calculate_gReq over the IBZ points of the Si example (25 k, 16 q)
        dict(name="gkRp_ibz", kind="gkRp", nw=8, nat=2, cells=6, n=25),
        dict(name="gReq_ibz", kind="gReq", nw=8, nat=2, cells=6, n=16),
        # the per-vertex entry point, as a host code that walks the vertices of a few k-points calls it
        dict(name="g2_vertices", kind="g2", nw=8, nat=2, cells=5, n=4001, blocks=5, side="ph"),
        # the drop-in: plain FP64 rates of the Si-like crystal on 12^3, the library's default precision
        _rates("rates_fp64_12", (12, 12, 12), split=False),
        # the reference's own delta (tetrahedra), split form, on an uneven mesh
        _rates("rates_tetra_split", (10, 12, 11), cells=5, delta=2),
        # the headline request: split form, 24^3
        _rates("rates_split_24", (24, 24, 24)),
        # the smallest served request: 8^3
        _rates("rates_split_8", (8, 8, 8), cells=4),
        # a larger cell (16 Wannier bands, 4 atoms): the generic split path, odd mesh
        _rates("rates_split_nw16", (13, 13, 13), nw=16, nat=4, cells=4, window=0.3),
        # phonon and electron side of a polar crystal in one sweep
        _rates("phrates_polar_fp64", (9, 10, 9), cells=4, split=False, polar=True, ph=True),
        # many requests of uneven size on crystals of different shapes in one call
        dict(name="batch_mixed", kind="batch", requests=16, lo=8, hi=13, crystals=4),
    ]


# (nw, atoms, WS supercell) of the batch's crystals: the fused shape and three generic ones
BATCH_SHAPES = [(8, 2, 5), (16, 2, 4), (8, 4, 4), (24, 2, 4)]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(c):
    """Rough multiply-adds of a rates case, FP64 ones weighted by how much slower they run."""
    N = c["m1"] * c["m2"] * c["m3"]
    nws = {4: 93, 5: 165, 6: 279}[c["cells"]]
    nb = 3 * c["nat"]
    ns = N * min(1.0, 0.9 * c["window"] / 0.5) * c["nw"] / 8
    contraction = N * nws * c["nw"] * nb * (ns + c["nw"] * nws)
    vertices = 100.0 * ns * ns * nb * c["sets"]
    if not c["split"]:
        return 100 * contraction + 40 * vertices
    return contraction * (1 if c["nw"] == 8 and c["nat"] == 2 else 2) + (40 * vertices if c["delta"] else vertices)


def draw(rng):
    kind = rng.choice(["bands", "phonons", "gkRp", "gReq", "g2", "rates", "rates", "rates", "rates", "batch"])
    nw, nat, cells = rng.choice([(4, 2, 4), (8, 2, 6), (8, 2, 5), (8, 3, 4), (16, 2, 4), (16, 4, 4)])
    if kind == "bands":
        return dict(kind=kind, nw=nw, nat=nat, cells=cells, n=_logint(rng, 16, 4096), vel=rng.random() < 0.6)
    if kind == "phonons":
        polar = rng.random() < 0.5
        return dict(kind=kind, nw=4, nat=2 if polar else nat, cells=rng.choice([4, 5, 6]), n=_logint(rng, 16, 4096),
                    vel=rng.random() < 0.6, polar=polar)
    if kind in ("gkRp", "gReq"):
        return dict(kind=kind, nw=nw, nat=nat, cells=cells, n=_logint(rng, 1, 40))
    if kind == "g2":
        return dict(kind=kind, nw=nw, nat=nat, cells=rng.choice([4, 5]), n=_logint(rng, 64, 8192),
                    blocks=rng.randint(1, 8), side=rng.choice(["ph", "el"]))
    if kind == "batch":
        return dict(kind=kind, requests=rng.randint(4, 16), lo=rng.randint(6, 8), hi=rng.randint(9, 13),
                    crystals=rng.randint(2, 4))
    split = rng.random() < 0.6
    delta = rng.choice([0, 0, 0, 1, 2])
    polar = nat == 2 and rng.random() < 0.25
    ph = rng.random() < 0.3
    sets = rng.randint(2, 4) if not ph and rng.random() < 0.25 else 1
    m = _logint(rng, 6, 24)
    mesh = [max(5, m + rng.choice([-1, 0, 0, 1])) for _ in range(3)]
    c = _rates(None, mesh, nw=nw, nat=nat, cells=cells, split=split, delta=delta, polar=polar, ph=ph, sets=sets,
               window=round(rng.uniform(0.15, 0.5), 3), T=round(rng.uniform(100.0, 600.0), 1),
               sigma=round(rng.uniform(0.005, 0.020), 5))
    limit = _cost(next(x for x in listed() if x["name"] == "rates_fp64_12"))
    while _cost(c) > limit and max(c["m1"], c["m2"], c["m3"]) > 5:   # no more than the listed drop-in request
        k = max(("m1", "m2", "m3"), key=lambda x: c[x])
        c[k] -= 1
    return c


# ---------------------------------------------------------------- crystals
@functools.lru_cache(maxsize=None)
def _geometry(nat, cells, polar):
    """Crystal, Wigner-Seitz cells and their degeneracies: geometry only, the same for every seed."""
    if polar:
        crys = S.make_crystal_sic_like()
    elif nat == 2:
        crys = S.make_crystal_si_like()
    else:
        crys = S.make_crystal_multi(nat, np.random.Generator(np.random.PCG64(40 + nat)))
    return (crys,) + S.wigner_seitz(crys.lattvecs, (cells,) * 3)


def _crystal(nw, nat, cells, seed, polar=False, vertex=True):
    """Wannier data with the package's synthetic distributions (``synthetic.make_wannier``): one band structure per
    shape, so that its window holds the same states for every seed; springs and g(Re,Rp) from the seed, g drawn on
    the GPU; without ``vertex`` (calls that read no g) zeros stand for it."""
    crys, R, deg = _geometry(nat, cells, polar)
    rng = np.random.Generator(np.random.PCG64(seed))
    rlen = np.linalg.norm((crys.lattvecs * S.ANG_PER_NM) @ R.T, axis=0)
    env = np.exp(-rlen / 2.0)
    bands = np.random.Generator(np.random.PCG64(1000 * nw + 10 * nat + cells))
    H = np.asfortranarray(S._hermitian_paired(bands, R, nw, env) / S.C.Ryd2eV)
    D = S._springs(crys, R, (cells,) * 3, rng, 5.0, 15.0)
    nws, nb = len(R), 3 * nat
    if vertex:
        gen = torch.Generator(device="cuda").manual_seed(seed)
        e = torch.tensor(env, device="cuda")
        g = torch.randn((nws, nb, nws, nw, nw, 2), generator=gen, dtype=torch.float64, device="cuda")   # C order of F
        g *= (0.1 / math.sqrt(2.0) * S.EV_PER_ANG_TO_RY_PER_BOHR) * (e[:, None] * e)[:, None, :, None, None, None]
        g = torch.view_as_complex(g).cpu().numpy().T
    else:
        g = np.zeros((nws, nb, nws, nw, nw), dtype=np.complex128).T
    wd = S.WannierData(crystal=crys, numwannbands=nw, numbranches=nb, coarse_qmesh=np.full(3, cells, dtype=np.int64),
                       rcells_k=R.copy(), rcells_q=R.copy(), rcells_g=R.copy(), elwsdeg=deg.copy(), phwsdeg=deg.copy(),
                       gwsdeg=deg.copy(), Hwann=H, Dphwann=np.asfortranarray(D), gwann=g)
    wd.midgap = S._midgap(wd, nw // 2)
    return wd


def _requests(case, wd):
    """The parameter sets of a rates case: one request, or several that differ in T and sigma."""
    mu = wd.midgap + 0.6
    return [S.RateRequest(mesh=(case["m1"], case["m2"], case["m3"]), enref=mu, fsthick=case["window"], chempot=mu + 0.02 * p,
                          T=case["T"] + 50.0 * p, delta_kind=case["delta"], sigma=case["sigma"] * (1 + 0.2 * p))
            for p in range(case["sets"])]


def _batch(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    wds = [_crystal(nw, nat, cells, seed + 1 + i) for i, (nw, nat, cells) in enumerate(BATCH_SHAPES[:case["crystals"]])]
    reqs = []
    for i in range(case["requests"]):
        # sizes are the case's, spread over its range; only values come from the seed
        m = case["lo"] + (5 * i) % (case["hi"] - case["lo"] + 1)
        w = wds[i % len(wds)]
        reqs.append((i % len(wds), S.si_like_request(w, (m, m, m), window=0.1 + 0.03 * (i % 8),
                                                     T=float(rng.uniform(250.0, 350.0)))))
    return wds, reqs


def _points(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed + 5))
    n = case["n"]
    if case["kind"] == "bands":      # straight segments between random corners, as a band path
        ends = rng.uniform(-0.5, 0.5, (5, 3))
        t = np.linspace(0.0, 4.0, n, endpoint=False)
        i = t.astype(int)
        return ends[i] + (t - i)[:, None] * (ends[i + 1] - ends[i])
    m = round(n ** (1.0 / 3.0))
    if m ** 3 == n:                  # a whole mesh, shifted by a seeded offset
        return S.mesh_kvecs((m, m, m)) + rng.uniform(0.0, 1.0 / m, 3)
    return rng.uniform(0.0, 1.0, (n, 3))


def _unit(rng, n, w):
    v = rng.standard_normal((n, w)) + 1j * rng.standard_normal((n, w))
    return np.asfortranarray(v / np.linalg.norm(v, axis=1, keepdims=True))


def _vertices(case, wd, seed):
    """A vertex list: blocks of half-transformed vertices (decaying as the real-space ones) and unit eigenvectors."""
    rng = np.random.Generator(np.random.PCG64(seed + 9))
    nw, nb, nws, n = wd.numwannbands, wd.numbranches, wd.nwsk, case["n"]
    env = np.exp(-np.linalg.norm((wd.crystal.lattvecs * S.ANG_PER_NM) @ wd.rcells_q.T, axis=0) / 2.0)
    gm = rng.standard_normal((case["blocks"], nws, nb, nw, nw)) + 1j * rng.standard_normal((case["blocks"], nws, nb, nw, nw))
    gm *= (0.1 * S.EV_PER_ANG_TO_RY_PER_BOHR) * env[None, :, None, None, None]
    return dict(kvecs=np.asfortranarray(rng.uniform(0, 1, (n, 3))), qvecs=np.asfortranarray(rng.uniform(0, 1, (n, 3))),
                el_evec_k=_unit(rng, n, nw), el_evec_kp=_unit(rng, n, nw), ph_evec_q=_unit(rng, n, nb),
                ph_en=rng.uniform(0.005, 0.06, n), gmixed=gm.T, gm_index=np.sort(rng.integers(1, case["blocks"] + 1, n)),
                wannspace=case["side"])


def _inputs(case, seed):
    kind = case["kind"]
    if kind == "batch":
        wds, reqs = _batch(case, seed)
        return dict(wds=wds, reqs=reqs)
    wd = _crystal(case["nw"], case["nat"], case["cells"], seed, polar=case.get("polar", False),
                  vertex=kind in ("rates", "gkRp", "gReq"))
    if kind == "rates":
        return dict(wd=wd, reqs=_requests(case, wd))
    if kind == "g2":
        return dict(wd=wd, args=_vertices(case, wd, seed))
    return dict(wd=wd, points=_points(case, seed))


def prepare(case, seed):
    s = dict(_inputs(case, seed), case=case)
    if case["kind"] == "batch":
        s["W"] = [Wannier(w) for w in s.pop("wds")]
    else:
        s["W"] = Wannier(s.pop("wd"))
    return s


def run(s):
    case, W = s["case"], s["W"]
    kind = case["kind"]
    if kind == "bands":
        return W.el_wann(kvecs=s["points"], velocities=case["vel"])
    if kind == "phonons":
        return W.ph_wann(qvecs=s["points"], velocities=case["vel"])
    if kind == "gkRp":
        return W.gkRp(kvec=s["points"])
    if kind == "gReq":
        return W.gReq(qvec=s["points"])
    if kind == "g2":
        return W.g2_batch(**s["args"])
    if kind == "batch":
        outs, _, _ = el_rates_batch([W[c] for c, _ in s["reqs"]], [r for _, r in s["reqs"]], precision=SPLIT)
        return [dict(rates=o["rates"], indexlist=o["indexlist"]) for o in outs]
    prec = SPLIT if case["split"] else FP64
    if case["ph"]:
        o = W.ph_rates(s["reqs"][0], precision=prec, electrons=True)
        return dict(rates=o["rates"], indexlist=o["indexlist"], rates_phe=o["rates_phe"])
    if case["sets"] > 1:
        return [dict(rates=o["rates"], indexlist=o["indexlist"]) for o in W.el_rates_sets(s["reqs"], precision=prec)]
    o = W.el_rates(s["reqs"][0], precision=prec)
    return dict(rates=o["rates"], indexlist=o["indexlist"])


def work(case):
    """Inputs read once and outputs written once; operations of the plain method: the Fourier sums as separable or
    direct sums, whichever is fewer, and about 300 operations a vertex."""
    kind = case["kind"]
    if kind == "batch":
        tot = dict(bytes=0.0, flops=0.0)
        for i in range(case["requests"]):
            nw, nat, cells = BATCH_SHAPES[i % case["crystals"]]
            m = case["lo"] + (5 * i) % (case["hi"] - case["lo"] + 1)
            w = work(_rates(None, (m, m, m), nw=nw, nat=nat, cells=cells, window=0.1 + 0.03 * (i % 8)))
            tot = {k: tot[k] + w[k] for k in tot}
        return tot
    nw, nb = case["nw"], 3 * case["nat"]
    nws = {4: 93, 5: 165, 6: 279}[case["cells"]]
    if kind == "bands":
        n, c = case["n"], nw * nw * (4 if case["vel"] else 1)
        return dict(bytes=8.0 * n * (3 + nw * (4 if case["vel"] else 1)) + 16.0 * nws * nw * nw,
                    flops=8.0 * n * nws * c + 100.0 * n * nw ** 3)
    if kind == "phonons":
        n, c = case["n"], nb * nb * (4 if case["vel"] else 1)
        return dict(bytes=8.0 * n * (3 + nb * (4 if case["vel"] else 1)) + 16.0 * nws * nb * nb,
                    flops=8.0 * n * nws * c + 100.0 * n * nb ** 3)
    if kind in ("gkRp", "gReq"):
        col = nw * nw * nb * nws
        return dict(bytes=16.0 * col * (nws + case["n"]), flops=8.0 * case["n"] * nws * col)
    if kind == "g2":
        n, col = case["n"], nw * nw * nb
        return dict(bytes=16.0 * case["blocks"] * col * nws + 16.0 * n * (2 * nw + nb + 4), flops=8.0 * n * nws * col)
    m = (case["m1"], case["m2"], case["m3"])
    N = m[0] * m[1] * m[2]
    e = 2 * case["cells"] - 1
    column = min(N * nws, e * e * m[2] * e + e * m[1] * m[2] * e + N * e)   # multiply-adds of one column's Fourier sum
    ns = N * min(1.0, 0.9 * case["window"] / 0.5) * nw / 8
    col = nw * nw * nb * nws
    return dict(bytes=16.0 * col * nws + 8.0 * N * (nw * case["sets"] + (nb if case["ph"] else 0)),
                flops=8.0 * column * (col + ns * nw * nb) + 300.0 * ns * ns * nb * case["sets"])


# ------------------------------------------------------------------- exact
def _t(a, dtype=None):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")


def _mass(crys):
    return np.repeat(crys.masses, 3)


def _wraps(crys, R, cells):
    """Per (iat, jat, cell): the shortest supercell images R + w N of the bond (wannier.f90:532-582)."""
    sh = np.array([(i, j, k) for k in range(-3, 4) for j in range(-3, 4) for i in range(-3, 4)])
    out = {}
    for ia in range(crys.numatoms):
        for ja in range(crys.numatoms):
            vl = (R - crys.basis[:, ia] + crys.basis[:, ja]) / cells
            iv = np.trunc(vl)
            v = (vl - iv)[:, None, :] + sh[None]
            d = np.linalg.norm(v @ crys.lattvecs.T, axis=2)
            keep = np.abs(d - d.min(axis=1, keepdims=True)) < 1e-6
            out[ia, ja] = [(R[r] + (sh[keep[r]] - iv[r]) * cells).astype(int) for r in range(len(R))]
    return out


def _polar(crys, cells, q):
    """Long-range terms at q (n,3): the matrix added to D before the mass factors, its q-derivatives and the vector
    L (wannier.f90:784-901, 1013-1071)."""
    b2nm = S.C.bohr2nm
    rec = crys.reclattvecs
    a1 = np.linalg.norm(crys.lattvecs[:, 0])
    alph = (2 * np.pi / a1 * b2nm) ** 2
    fac = 8 * np.pi / (crys.volume / b2nm ** 3)
    m = np.arange(-cells, cells + 1)
    G = np.stack(np.meshgrid(m, m, m, indexing="ij"), -1).reshape(-1, 3) @ rec.T * b2nm
    tau = (crys.lattvecs @ crys.basis).T / b2nm
    eps, Z = crys.epsilon, crys.born
    na = crys.numatoms

    def terms(g):     # g (M,3) that pass the cut: f, p (M,na), z (M,na,3)
        qeq = np.einsum("mi,ij,mj->m", g, eps, g)
        ok = (qeq > 0) & (qeq / alph / 4 < 14.0)
        g, qeq = g[ok], qeq[ok]
        return g, qeq, np.exp(-qeq / alph / 4) / qeq, np.exp(1j * g @ tau.T), np.einsum("mi,ija->maj", g, Z)

    g, qeq, f, p, z = terms(G)
    Da = np.zeros((na, 3, na, 3), complex)
    for a in range(na):
        fn = np.einsum("mcj,m,mc->mj", z, p[:, a], p.conj())
        Da[a, :, a, :] = -np.einsum("m,mi,mj->ij", f, z[:, a], fn)
    D = np.zeros((len(q), 3 * na, 3 * na), complex)
    dD = np.zeros((3, len(q), 3 * na, 3 * na), complex)
    L = np.zeros((len(q), 3 * na), complex)
    for i, qi in enumerate(q):
        g, qeq, f, p, z = terms(G + (rec @ qi) * b2nm)
        w = (p[:, :, None] * z).reshape(len(f), -1)
        D[i] = fac * ((w * f[:, None]).T @ w.conj() + Da.reshape(3 * na, 3 * na))
        L[i] = 1j * fac * (f[:, None] * w.conj()).sum(0)
        zz = z.reshape(len(f), -1)
        for x in range(3):
            dge = g @ (eps[x, :] + eps[:, x])
            Zx = np.repeat(Z[x].T.reshape(-1)[None], len(f), 0)      # Z(x, i, a) by 3 a + i
            P = np.repeat(p, 3, axis=1)
            dc = (0.25 / alph + 1.0 / qeq) * dge
            pa = (P * f[:, None])
            dr = np.repeat(tau[:, x], 3)
            re = np.einsum("mi,mj->ij", pa * Zx, (P * zz).conj()) + np.einsum("mi,mj->ij", pa * zz, (P * Zx).conj())
            wf = np.einsum("mi,mj->ij", pa * zz, (P * zz).conj())
            dD[x, i] = fac * b2nm * (re - np.einsum("mi,mj->ij", pa * zz * dc[:, None], (P * zz).conj())
                                     + 1j * (dr[:, None] - dr[None, :]) * wf)
    return D, dD, L


def _exact_phonons(wd, q, vel=False):
    """omega (eV), eigenvectors (columns), velocities (km/s) and the polar vector L at q (n,3) (wannier.f90:585-782)."""
    crys, R, cells = wd.crystal, wd.rcells_q, int(wd.coarse_qmesh[0])
    nb, na = wd.numbranches, crys.numatoms
    D = np.zeros((len(q), nb, nb), complex)
    dD = np.zeros((3, len(q), nb, nb), complex)
    rc = R @ crys.lattvecs.T
    wr = _wraps(crys, R, cells)
    for ia in range(na):
        for ja in range(na):
            ph = np.stack([np.exp(2j * np.pi * (q @ wr[ia, ja][r].T)).sum(1) / (wd.phwsdeg[r] * len(wr[ia, ja][r]))
                           for r in range(len(R))], 1)
            blk = wd.Dphwann[:, 3 * ia:3 * ia + 3, 3 * ja:3 * ja + 3]
            sl = (slice(None), slice(3 * ia, 3 * ia + 3), slice(3 * ja, 3 * ja + 3))
            D[sl] = np.einsum("qr,rab->qab", ph, blk)
            for x in range(3):
                dD[x][sl] = np.einsum("qr,rab->qab", ph * (1j * rc[:, x]), blk)
    L = None
    if crys.polar:
        lD, ldD, L = _polar(crys, cells, q)
        D, dD = D + lD, dD + ldD
    m = _mass(crys)
    mn = S.C.Ryd2amu / np.sqrt(m[:, None] * m[None, :])
    D, dD = D * mn, dD * mn
    w, V = np.linalg.eigh(0.5 * (D + np.conj(np.transpose(D, (0, 2, 1)))))
    e = np.copysign(np.sqrt(np.abs(w)), w)
    v = None
    if vel:
        with np.errstate(divide="ignore", invalid="ignore"):
            v = np.stack([np.einsum("qas,qab,qbs->qs", V.conj(), dD[x], V).real / (2 * e) for x in range(3)], 2)
        v *= S.C.Ryd2radTHz
    e = e * S.C.Ryd2eV
    gam = np.all(q == 0, axis=1)
    e[np.ix_(gam, np.arange(nb) < 3)] = 0.0
    if vel:
        v[gam] = 0.0
    e[(e < 0) & (e > -0.005)] = 0.0
    return e, V, v, L


def _exact_bands(wd, k, vel=False):
    ph = np.exp(2j * np.pi * (k @ wd.rcells_k.T)) / wd.elwsdeg
    nws, nw = wd.nwsk, wd.numwannbands
    H = (ph @ wd.Hwann.reshape(nws, -1, order="C")).reshape(-1, nw, nw)
    e, V = np.linalg.eigh(0.5 * (H + np.conj(np.transpose(H, (0, 2, 1)))))
    v = None
    if vel:
        rc = wd.rcells_k @ wd.crystal.lattvecs.T
        Hc = np.ascontiguousarray(wd.Hwann).reshape(nws, -1)
        v = np.stack([np.einsum("kab,kac,kcb->kb", V.conj(), ((ph * (1j * rc[:, x])) @ Hc).reshape(-1, nw, nw), V).real
                      for x in range(3)], 2) * S.C.Ryd2radTHz
    return e * S.C.Ryd2eV, V, v


def _tetra(kind, mesh, widx, ens):
    """Simplices of the window mesh with their sorted vertex energies (delta.f90:494-788): per window k the list of
    (sorted energies of every band, the label of the vertex that is this k)."""
    m1, m2, m3 = mesh
    pos = {int(p): i for i, p in enumerate(widx)}
    corner = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 0), (0, 0, 1), (1, 0, 1), (0, 1, 1), (1, 1, 1)]
    sets = ([(1, 2, 3), (1, 3, 4)] if kind == 1 else
            [(1, 2, 3, 6), (1, 3, 5, 6), (3, 5, 6, 7), (3, 6, 7, 8), (3, 4, 6, 8), (2, 3, 4, 6)])
    nv, most = len(sets[0]), 6 if kind == 1 else 24
    nwv, nw = ens.shape
    ev = np.full((nwv, most, nw, nv), np.nan)
    lab = np.zeros((nwv, most), int)
    cnt = np.zeros(nwv, int)
    for p in widx:
        c = [(int(p) % m1 + a) % m1 + m1 * (((int(p) // m1) % m2 + b) % m2 + m2 * ((int(p) // (m1 * m2) + d) % m3))
             for a, b, d in corner]
        for t in sets:
            at = [pos.get(c[x - 1], -1) for x in t]
            se = np.sort(np.stack([ens[i] if i >= 0 else np.zeros(nw) for i in at], 1), axis=1)
            for l, i in enumerate(at):
                if i >= 0:
                    ev[i, cnt[i]], lab[i, cnt[i]] = se, l + 1
                    cnt[i] += 1
    return ev, lab


def _weights_triangle(e, E):
    """Per vertex label, the weight in the two energy ranges of a triangle (delta.f90:790-881)."""
    e1, e2, e3 = E
    f = lambda a, b: (e - b) / (a - b)   # noqa: E731
    lo, hi = (e1 < e) & (e <= e2), (e2 < e) & (e <= e3)
    pairs = [(f(e2, e1) * (f(e1, e2) + f(e1, e3)), f(e2, e3) * f(e1, e3)), (f(e2, e1) ** 2, f(e2, e3) ** 2),
             (f(e2, e1) * f(e3, e1), f(e2, e3) * (f(e3, e1) + f(e3, e2)))]
    zero = torch.zeros_like(e)
    return [torch.where(lo, a, torch.where(hi, b, zero)) / (e3 - e1) for a, b in pairs]


def _weights_tetra(e, E):
    """Per vertex label, the weight in the three energy ranges of a tetrahedron (delta.f90:61-225), with the forms
    for equal vertex energies (corners outside the window sit at zero)."""
    e1, e2, e3, e4 = E
    x1, x2, x3, x4 = e1 - e, e2 - e, e3 - e, e4 - e
    d21, d31, d41, d32, d42, d43 = e2 - e1, e3 - e1, e4 - e1, e3 - e2, e4 - e2, e4 - e3
    r1, r2, r3 = (e1 <= e) & (e <= e2), (e2 <= e) & (e <= e3), (e3 <= e) & (e <= e4)
    zero = torch.zeros_like(e)
    c1 = x1 ** 3 / d21 / d31 / d41
    c4 = x4 ** 3 / d41 / d42 / d43
    # the quadratic products of the middle range
    p = [x3 * x2 / d42 / d32, x4 * x1 / d41 / d42, x3 * x1 / d32 / d41]
    q = [x4 * x1 / d42 / d31, x4 * x2 / d42 / d32, x3 * x1 / d31 / d32]
    u = [x3 * x2 / d42 / d31, x4 * x2 / d42 / d41, x3 * x1 / d31 / d41]
    v = [x3 * x2 / d32 / d31, x4 * x1 / d41 / d31, x4 * x2 / d32 / d41]
    mid = [-0.5 * (x3 / d31 ** 2 * sum(p) + x4 / d41 ** 2 * sum(q)),
           -0.5 * (x3 / d32 ** 2 * sum(u) + x4 / d42 ** 2 * sum(v)),
           0.5 * (x2 / d32 ** 2 * sum(u) + x1 / d31 ** 2 * sum(p)),
           0.5 * (x2 / d42 ** 2 * sum(v) + x1 / d41 ** 2 * sum(q))]
    mid23 = [-0.5 * (x4 * x1 / d41 / d42 + x1 / d41 + x4 / d41 ** 2 * (x4 * x1 / d42 / d31 + x4 / d42 + x1 / d31)),
             -0.5 * (x4 / d42 / d41 + x4 / d42 ** 2 * (x4 * x1 / d41 / d31 + 1.0)),
             0.5 * (x4 / d42 / d41 + x1 / d31 / d41 + x1 / d31 ** 2 * (x4 * x1 / d41 / d42 + x1 / d41)),
             0.5 * (x1 / d41 ** 2 * (x4 * x1 / d42 / d31 + x4 / d42 + x1 / d31))]
    low = [(x2 / d21 + x3 / d31 + x4 / d41) * x1 ** 2 / d41 / d31 / d21, -c1 / d21, -c1 / d31, -c1 / d41]
    top = [c4 / d41, c4 / d42, c4 / d43, -(x3 / d43 + x2 / d42 + x1 / d41) * x4 ** 2 / d41 / d42 / d43]
    top34 = [x4 ** 2 / d41 ** 2 / d42 + zero, zero, zero, zero]
    out = []
    for i in range(4):
        a = torch.where(e1 == e2, zero, low[i])
        b = torch.where(e2 == e3, mid23[i], mid[i])
        c = torch.where(e3 == e4, top34[i], top[i])
        out.append(torch.where(r1, a, torch.where(r2, b, torch.where(r3, c, zero))))
    return out


def _delta_simplex(kind, e, ev, lab, N):
    """The simplex deltas at e (j, f, s): ev (f, t, nv) sorted energies (NaN: no simplex), lab (f, t) vertex labels."""
    acc = torch.zeros_like(e)
    for t in range(ev.shape[1]):
        w = (_weights_triangle if kind == 1 else _weights_tetra)(e, [ev[None, :, t, i, None] for i in range(ev.shape[2])])
        v = lab[None, :, t, None]
        x = torch.zeros_like(e)
        for i, wi in enumerate(w):
            x = torch.where(v == i + 1, wi, x)
        acc += torch.where(torch.isnan(ev[None, :, t, 0, None]), torch.zeros_like(x), x)
    return torch.where(acc < 1e-12, torch.zeros_like(acc), acc) / ((2 if kind == 1 else 6) * N)


def _fold(X, R, mesh):
    """sum over cells R (rows of X) of e^{2 pi i k.R} X for every mesh point, rows in muxed order: cells folded onto
    the mesh, then one FFT."""
    m1, m2, m3 = mesh
    Rm = R % np.asarray(mesh)
    at = _t((Rm[:, 2] * m2 + Rm[:, 1]) * m1 + Rm[:, 0])
    box = torch.zeros((m1 * m2 * m3,) + X.shape[1:], dtype=X.dtype, device=X.device)
    torch.view_as_real(box).index_add_(0, at, torch.view_as_real(X.contiguous()))
    f = torch.fft.ifftn(box.reshape((m3, m2, m1) + X.shape[1:]), dim=(0, 1, 2), norm="forward")
    return f.reshape((m1 * m2 * m3,) + X.shape[1:])


def _exact_rates(wd, reqs, ph=False, spindeg=2):
    """rates (nwv, nw) per request, the window's indexlist and the ph-e rates (N, nb) of requests that share a window."""
    C, mesh = S.C, reqs[0].mesh
    N, nw, nb, nws = int(np.prod(mesh)), wd.numwannbands, wd.numbranches, wd.nwsk
    R = wd.rcells_k
    k = S.mesh_kvecs(mesh)
    ens, V, _ = _exact_bands(wd, k)
    om, Vq, _, L = _exact_phonons(wd, k)
    u = np.transpose(Vq, (0, 2, 1)) / np.sqrt(_mass(wd.crystal))        # u[q, s, c]
    inw = np.abs(ens - reqs[0].enref) <= reqs[0].fsthick
    widx = np.nonzero(inw.any(1))[0]
    fk, fb = np.nonzero(inw[widx])                                      # window states in order
    p = widx[fk]
    nst, nwv = len(p), len(widx)
    E = _t(ens[p, fb])
    U = _t(np.transpose(V, (0, 2, 1))[p, fb])                           # U[state, c]
    om_t, u_t, p_t = _t(om), _t(u), _t(p)
    glp = _t(np.einsum("qc,qsc->qs", L, u)) if L is not None else None
    deg = _t(wd.elwsdeg, torch.float64)
    # stage A: g(k,Rp) on the mesh by FFT over Re, the initial band, the k half of the Rp phase
    g = torch.from_numpy(wd.gwann.T)                                    # (Rp, s, Re, j, i)
    B = torch.empty((nst, nws, nb, nw), dtype=torch.complex128, device="cuda")
    step = max(1, (1 << 30) // (16 * N * nw * nw * nb))
    for r0 in range(0, nws, step):
        x = g[r0:r0 + step].cuda().permute(2, 0, 1, 3, 4) / deg[:, None, None, None, None]
        gk = _fold(x, R, mesh)                                          # (N, rp, s, mp, np)
        for j0 in range(0, nst, 512):
            j = slice(j0, j0 + 512)
            B[j, r0:r0 + step] = torch.einsum("jm,jrsmn->jrsn", U[j], gk[p_t[j]])
        del gk, x
    phk = torch.exp(-2j * np.pi * (_t(k[p]) @ _t(R, torch.float64).T).to(torch.complex128)) / deg
    B *= phk[:, :, None, None]
    # stage B and the vertices, a few initial states at a time
    kint = np.stack([widx % mesh[0], (widx // mesh[0]) % mesh[1], widx // (mesh[0] * mesh[1])], 1)
    kf, m_t = _t(kint[fk]), _t(np.asarray(mesh))
    w_t, fk_t = _t(widx), _t(fk)
    acc = [torch.zeros(nst, dtype=torch.float64, device="cuda") for _ in reqs]
    phr = torch.zeros(N * nb, dtype=torch.float64, device="cuda")
    simplex = None
    if reqs[0].delta_kind:
        ev, lab = _tetra(reqs[0].delta_kind, mesh, widx, ens[widx])
        simplex = _t(ev[fk, :, fb]), _t(lab[fk])
    tp = 2 * np.pi / C.hbar_eVps
    js = max(1, min(512, (1 << 28) // (N * nw * nb), (1 << 26) // (nst * nb * nb), (1 << 23) // (nst * nb)))
    for j0 in range(0, nst, js):
        j = slice(j0, min(nst, j0 + js))
        G = _fold(B[j].transpose(0, 1), R, mesh)[w_t]                    # (nwv, j, s, np)
        h = torch.einsum("fn,fjsn->jfs", U.conj(), G[fk_t])
        d = torch.remainder(kf[None] - kf[j, None], m_t)
        q = d[..., 0] + mesh[0] * (d[..., 1] + mesh[1] * d[..., 2])      # (j, f)
        gs = torch.einsum("jfsc,jfc->jfs", u_t[q], h)
        if glp is not None:
            gs = gs + glp[q] * torch.einsum("fn,jn->jf", U.conj(), U[j])[..., None]
        w = om_t[q]
        g2 = torch.where(w == 0, torch.zeros_like(w), 0.5 * gs.abs() ** 2 / w * C.g2unitfactor)
        live = w >= 0.5e-3
        Ej, Ef = E[j, None, None], E[None, :, None]
        for i, r in enumerate(reqs):
            kT = C.kB * r.T
            fermi = lambda x: 1.0 / (torch.exp((x - r.chempot) / kT) + 1.0)   # noqa: E731, B023
            if simplex is None:
                dl = lambda x: torch.exp(-0.5 * ((x - Ef) / r.sigma) ** 2) / (math.sqrt(2 * np.pi) * r.sigma * N)   # noqa: E731, B023
            else:
                dl = lambda x: _delta_simplex(r.delta_kind, x, *simplex, N)    # noqa: E731, B023
            bose = torch.where(w != 0, 1.0 / torch.expm1(w / kT), torch.zeros_like(w))
            x = g2 * (bose + fermi(Ej + w)) * dl(Ej + w) + g2 * (1 + bose - fermi(Ej - w)) * dl(Ej - w)
            acc[i][j] = tp * torch.where(live, x, torch.zeros_like(x)).sum((1, 2))
            if ph:
                if simplex is None:
                    dy = dl(Ej + w)
                else:      # delta(E' - omega) at the initial electron
                    dy = _delta_simplex(r.delta_kind, (Ef - w).transpose(0, 1), simplex[0][j], simplex[1][j], N).transpose(0, 1)
                y = tp * g2 * fermi(Ej) * (1 - fermi(Ej + w)) / (1 + bose) * dy
                at = (q[..., None] * nb + torch.arange(nb, device="cuda")).reshape(-1)
                phr.index_add_(0, at, spindeg * torch.where(live, y, torch.zeros_like(y)).reshape(-1))
    rates = []
    for a in acc:
        o = np.zeros((nwv, nw))
        o[fk, fb] = a.cpu().numpy()
        rates.append(o)
    return rates, widx.astype(np.int64) + 1, phr.reshape(N, nb).cpu().numpy()


def exact(case, seed):
    kind, s = case["kind"], _inputs(case, seed)
    if kind == "batch":
        out = []
        for c, r in s["reqs"]:
            rates, idx, _ = _exact_rates(s["wds"][c], [r])
            out.append(dict(rates=rates[0], indexlist=idx))
        return out
    wd = s["wd"]
    if kind == "bands":
        e, _, v = _exact_bands(wd, s["points"], case["vel"])
        return (e, v) if case["vel"] else e
    if kind == "phonons":
        e, _, v, _ = _exact_phonons(wd, s["points"], case["vel"])
        return (e, v) if case["vel"] else e
    if kind in ("gkRp", "gReq"):
        ph = _t(np.exp(2j * np.pi * (s["points"] @ wd.rcells_k.T)) / wd.elwsdeg)
        g = torch.from_numpy(wd.gwann.T)      # (Rp, s, Re, j, i)
        out = torch.empty((len(ph), wd.nwsk) + (wd.numbranches, wd.numwannbands, wd.numwannbands), dtype=torch.complex128)
        if kind == "gkRp":
            for r in range(wd.nwsk):
                x = g[r].cuda().transpose(0, 1)
                out[:, r] = (ph @ x.reshape(wd.nwsk, -1)).reshape((-1,) + x.shape[1:]).cpu()
        else:
            for r in range(wd.nwsk):
                x = g[:, :, r].cuda()
                out[:, r] = (ph @ x.reshape(wd.nwsk, -1)).reshape((-1,) + x.shape[1:]).cpu()
        return out.numpy().T
    if kind == "g2":
        a = s["args"]
        w = a["qvecs"] if a["wannspace"] == "ph" else a["kvecs"]
        ph = _t(np.exp(2j * np.pi * (w @ wd.rcells_q.T)) / wd.phwsdeg)
        gm = _t(a["gmixed"].T)                # (block, cell, s, j, i)
        u = _t(a["ph_evec_q"] / np.sqrt(_mass(wd.crystal)))
        out = torch.empty(len(u), dtype=torch.complex128, device="cuda")
        at = _t(a["gm_index"]) - 1
        for b in range(case["blocks"]):
            i = torch.nonzero(at == b)[:, 0]
            G = torch.einsum("vr,rsmn->vsmn", ph[i], gm[b])
            h = torch.einsum("vsmn,vm->vsn", G, _t(a["el_evec_k"])[i])
            out[i] = torch.einsum("vsn,vn,vs->v", h, _t(a["el_evec_kp"]).conj()[i], u[i])
        return (0.5 * out.abs() ** 2 / _t(a["ph_en"]) * S.C.g2unitfactor).cpu().numpy()
    rates, idx, phr = _exact_rates(wd, s["reqs"], ph=case["ph"])
    if case["ph"]:
        return dict(rates=rates[0], indexlist=idx, rates_phe=phr)
    out = [dict(rates=r, indexlist=idx) for r in rates]
    return out if case["sets"] > 1 else out[0]
