// ephg_polar.cu - the long-range dipole terms of polar crystals on the device:
// dyn_nonanalytic (wannier.f90:784-901) and long_range_prefac (:1013-1071).
//
// For a box vector G and g = G + q, with per-atom phases p_a = e^{i g.tau_a},
// z_a(j) = sum_i g_i born(i, j, a) and w(3a+i) = p_a z_a(i), the G + q term of
// dyn_nonanalytic is a rank-one update
//   D += f w w^H,   f = e^{-qeq/4alph}/qeq,
// and long_range_prefac is sum_c L(c) u(c), L = i fac conj(sum_g f w).
//
// One block per q, bound by the FP64 pipe, so what counts is FP64 instructions on
// full warps: the cut is tested in FP32 with a margin (a few per cent of the box
// vectors pass), the candidates are listed in the reference's loop order and one
// thread per candidate decides the cut in FP64 and forms its factors.  For q on
// the mesh (first cell) only the box vectors that can pass for some q of the cell
// are tested; the others never contribute.  Fixed order throughout: deterministic
// sums.
//
// With velocities (k_polar_vel) the sums' Hermitian halves, the candidates split over as
// many slices as the block has threads per item: 1,728 q, 13^3 box: 0.18 ms (1.13 ms with
// the FP64 test on every box vector, its terms formed in partly filled warps and ~70
// operations per element and vector; 0.32 with the derivative's outer products whole).
// Without (k_polar) an element is summed by one thread in the loop order, from
// f p_a conj(p_b) per pair of atoms and z.  The tensor-core rates round the
// eigenvectors to FP32 in the gauge that the eigensolver leaves them in, which the
// last bit of D decides where an off-diagonal element is all rounding: sums in
// another order move those rates by 1e-7, so here the order stays the loop's.  D of a call
// with velocities therefore differs from that of one without in its last bits.
#include <algorithm>

#include "ephg_common.cuh"
#include "ephg_kernels.cuh"

namespace ephg {

constexpr double BOHR2NM = 0.052917721092;   // params.f90:53
constexpr int PL_THREADS = 128;
constexpr int PL_LIST = 512;     // candidates listed before they are worked off
constexpr int PL_SMEM = 96 * 1024;

__device__ inline double geg(const double *eps, const double g[3]) {   // dot_product(g, matmul(epsilon, g))
  double acc = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) acc += g[i] * (eps[i] * g[0] + eps[i + 3] * g[1] + eps[i + 6] * g[2]);
  return acc;
}

// The cut in FP32 for up to PL_LIST box vectors from c0 on, the candidates listed in
// order; returns their number.  The margin covers FP32's rounding of all terms.
__device__ inline int pl_candidates(const PolarDev &P, const float *Gf, int M, const double qc[3], int &c0, int *list,
                                    int *wcount) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float qcf[3] = {(float)qc[0], (float)qc[1], (float)qc[2]};
  float epsf[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) epsf[i] = (float)P.eps[i];
  const float lim = (float)(4.0 * P.alph * P.gmax) * 1.00001f;
  int nl = 0;
  for (; c0 < M && nl <= PL_LIST - PL_THREADS; c0 += PL_THREADS) {
    const int gi = c0 + tid;
    bool cand = false;
    if (gi < M) {
      float g[3], a[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const float b = Gf[3 * gi + d];
        g[d] = b + qcf[d];
        a[d] = fabsf(b) + fabsf(qcf[d]);
      }
      float s = 0.f, t = 0.f;   // qeq and the size of its terms
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          s += g[i] * epsf[i + 3 * j] * g[j];
          t += a[i] * fabsf(epsf[i + 3 * j]) * a[j];
        }
      cand = s - 1e-5f * t < lim;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, cand);
    __syncthreads();   // wcount of the previous pass has been read
    if (lane == 0) wcount[warp] = __popc(bal);
    __syncthreads();
    int off = nl;
    for (int w = 0; w < PL_THREADS / 32; ++w) {
      if (w < warp) off += wcount[w];
      nl += wcount[w];
    }
    if (cand) list[off + __popc(bal & ((1u << lane) - 1u))] = gi;
  }
  return nl;
}

// q in nm^-1 x bohr: matmul(reclattvecs, q) * bohr2nm
__device__ inline void pl_q(const PolarDev &P, int q, int nq, const int *qp, int m1, int m2, int m3, const double *qv,
                            double qc[3]) {
  double qf[3];
  if (qp) {
    const int p = qp[q];
    qf[0] = (double)(p % m1) / m1;
    qf[1] = (double)((p / m1) % m2) / m2;
    qf[2] = (double)(p / (m1 * m2)) / m3;
  } else {
    qf[0] = qv[q];
    qf[1] = qv[q + nq];
    qf[2] = qv[q + 2 * nq];
  }
  for (int d = 0; d < 3; ++d) qc[d] = (P.rec[d] * qf[0] + P.rec[d + 3] * qf[1] + P.rec[d + 6] * qf[2]) * BOHR2NM;
}

// Candidates worked off at a time, entry bytes each.
static int pl_entries(size_t entry) { return std::min(PL_THREADS, (int)(PL_SMEM / entry)); }

// Without velocities.  Entry of a candidate: f, z (nb), p_a (re, im; nat), then (DA false)
// f p_a conj(p_b) per pair of atoms.  DA: the q-independent sum (wannier.f90:843-867)
//   D(3a+i, 3a+j) -= f z_a(i) sum_c z_c(j) e^{i g.(tau_a - tau_c)}.
// NU: matrix + vector elements per thread (nb^2 + nb <= NU * PL_THREADS).
// G / Gf / M: the box vectors to test, FP64 and FP32.
__host__ __device__ inline int pl_entry_doubles(int nat, bool da) { return 1 + 5 * nat + (da ? 0 : 2 * nat * nat); }

template <int NU, bool DA>
__global__ void __launch_bounds__(PL_THREADS) k_polar(PolarDev P, const double *G, const float *Gf, int M, int nq,
                                                      const int *qp, int m1, int m2, int m3, const double *qv, int nent,
                                                      double2 *Dq, int64_t ldd, double2 *Lq) {
  extern __shared__ double pse[];
  __shared__ int list[PL_LIST];
  __shared__ int wcount[PL_THREADS / 32];
  const int q = blockIdx.x, tid = threadIdx.x;
  const int nat = P.nat, nb = P.nb, ne = nb * nb, esz = pl_entry_doubles(nat, DA);
  double qc[3] = {0.0, 0.0, 0.0};
  if (!DA) pl_q(P, q, nq, qp, m1, m2, m3, qv, qc);
  double2 acc[NU];
#pragma unroll
  for (int u = 0; u < NU; ++u) acc[u] = make_double2(0.0, 0.0);
  for (int c0 = 0; c0 < M;) {
    const int nl = pl_candidates(P, Gf, M, qc, c0, list, wcount);
    for (int l0 = 0; l0 < nl; l0 += nent) {
      const int n = min(nent, nl - l0);
      __syncthreads();   // the list is written, the previous entries have been read
      if (tid < n) {
        const int gi = list[l0 + tid];
        double g[3];
        for (int d = 0; d < 3; ++d) g[d] = G[3 * gi + d] + qc[d];
        const double qeq = geg(P.eps, g);
        const bool pass = qeq > 0.0 && qeq / P.alph / 4.0 < P.gmax;
        const double f = pass ? exp(-qeq / P.alph / 4.0) / qeq : 0.0;   // 0: the terms leave every sum as it is
        double *e = pse + (size_t)tid * esz, *z = e + 1, *p = z + nb, *fq = p + 2 * nat;
        e[0] = f;
        for (int a = 0; a < nat; ++a) {
          const double arg = g[0] * P.tau[3 * a] + g[1] * P.tau[3 * a + 1] + g[2] * P.tau[3 * a + 2];
          double sn, cs;
          sincos(arg, &sn, &cs);
          p[2 * a] = cs;
          p[2 * a + 1] = sn;
          for (int j = 0; j < 3; ++j) {
            const double *Z = P.born + 3 * j + 9 * a;
            z[3 * a + j] = g[0] * Z[0] + g[1] * Z[1] + g[2] * Z[2];
          }
        }
        if (!DA && Dq)
          for (int b = 0; b < nat; ++b)
            for (int a = 0; a < nat; ++a) {
              const double2 pa = make_double2(p[2 * a], p[2 * a + 1]), pb = make_double2(p[2 * b], p[2 * b + 1]);
              fq[2 * (a + nat * b)] = f * (pa.x * pb.x + pa.y * pb.y);
              fq[2 * (a + nat * b) + 1] = f * (pa.y * pb.x - pa.x * pb.y);
            }
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const int el = tid + u * PL_THREADS;
        if (el < ne && Dq) {
          const int i = el % nb, j = el / nb, a = i / 3, b = j / 3;
          if (DA) {
            if (a != b) continue;
            for (int k = 0; k < n; ++k) {
              const double *e = pse + (size_t)k * esz, *z = e + 1, *p = z + nb;
              const double2 pa = make_double2(p[2 * a], p[2 * a + 1]);
              double2 fn = make_double2(0.0, 0.0);
              for (int c = 0; c < nat; ++c) {
                const double2 pc = make_double2(p[2 * c], p[2 * c + 1]);
                const double zc = z[3 * c + j % 3];
                fn.x += zc * (pa.x * pc.x + pa.y * pc.y);   // z * pa * conj(pc)
                fn.y += zc * (pa.y * pc.x - pa.x * pc.y);
              }
              const double t = e[0] * z[i];
              acc[u].x -= t * fn.x;
              acc[u].y -= t * fn.y;
            }
          } else {
            const double *zi = pse + 1 + i, *zj = pse + 1 + j, *fq = pse + 1 + 5 * nat + 2 * (a + nat * b);
#pragma unroll 4
            for (int k = 0; k < n; ++k) {
              const size_t o = (size_t)k * esz;
              const double zz = zi[o] * zj[o];
              acc[u].x += fq[o] * zz;
              acc[u].y += fq[o + 1] * zz;
            }
          }
        } else if (el >= ne && el < ne + nb && Lq) {
          const int c = el - ne, a = c / 3;
          for (int k = 0; k < n; ++k) {   // f conj(p_a) z(c)
            const double *e = pse + (size_t)k * esz;
            const double t = e[0] * e[1 + c];
            acc[u].x += t * e[1 + nb + 2 * a];
            acc[u].y -= t * e[2 + nb + 2 * a];
          }
        }
      }
    }
  }
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    const int el = tid + u * PL_THREADS;
    if (el < ne && Dq) {
      const int i = el % nb, j = el / nb;
      if (DA) {
        Dq[el] = acc[u];
        continue;
      }
      const double mn = 1.0 / sqrt(P.masses[i / 3] * P.masses[j / 3]) * Ryd2amu;
      double2 d = acc[u];
      if (P.Da) d = cadd(d, P.Da[el]);
      double2 &o = Dq[q * ldd + el];
      o = cadd(o, cscale(d, P.fac * mn));
    } else if (el >= ne && el < ne + nb && Lq) {
      Lq[(size_t)q * nb + (el - ne)] = make_double2(-P.fac * acc[u].y, P.fac * acc[u].x);   // i fac * acc
    }
  }
}

// With velocities.  With r = w w^H of a candidate, the derivative along x of sum f r is
//   dD_x(i,j) = born(x,i) P(a,j) + conj(born(x,j) P(b,i)) + i (tau_a - tau_b)(x) D(i,j) - 2 W_x(i,j),
//   P(a,j) = sum f p_a conj(w_j),  W_x = sum f dgeg_x (1/4alph + 1/qeq) / 2 r
// for i, j of atoms a, b: beside the nat nb sums of P only D and the W_x are summed, which are
// Hermitian: 12 FP64 operations per candidate on nb (nb + 1) / 2 elements instead of 16 on
// nb^2, and no vector per direction to prepare.
// Entry of a candidate (double2): w (nb), f p_a (nat), (f, W_0's weight), (W_1's, W_2's).
// NU: items per thread (nb (nb + 1) / 2 and nat nb <= NU * PL_THREADS).
__host__ __device__ inline int pv_entry(int nat) { return 4 * nat + 2; }

template <int NU>
__global__ void __launch_bounds__(PL_THREADS) k_polar_vel(PolarDev P, const double *G, const float *Gf, int M, int nq,
                                                          const int *qp, int m1, int m2, int m3, const double *qv,
                                                          int nent, double2 *Dq, double2 *dDq, int64_t ldd) {
  extern __shared__ double2 psm[];   // entries; at the end the sums
  __shared__ int list[PL_LIST];
  __shared__ int wcount[PL_THREADS / 32];
  const int q = blockIdx.x;
  const int nat = P.nat, nb = P.nb, ne = nb * nb, nh = nb * (nb + 1) / 2, np = nat * nb, esz = pv_entry(nat);
  const int tid = threadIdx.x;
  double qc[3];
  pl_q(P, q, nq, qp, m1, m2, m3, qv, qc);
  // Hermitian items (i >= j) and P items, each tid + u PL_THREADS, or (NU = 1) split over
  // as many slices of the candidates as the block has threads per item
  const int hsl = NU == 1 ? PL_THREADS / nh : 1, psl = NU == 1 ? PL_THREADS / np : 1;
  const int hs = NU == 1 ? tid / nh : 0, h0 = NU == 1 ? tid % nh : tid;
  const int ps = NU == 1 ? tid / np : 0, p0 = NU == 1 ? tid % np : tid;
  int hi[NU], hj[NU];
  double2 acc[NU][4], pacc[NU];
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    const int it = h0 + u * PL_THREADS;
    int i = 0;
    while ((i + 1) * (i + 2) / 2 <= it) ++i;
    hi[u] = hs < hsl && it < nh ? i : -1;
    hj[u] = it - i * (i + 1) / 2;
    pacc[u] = make_double2(0.0, 0.0);
#pragma unroll
    for (int x = 0; x < 4; ++x) acc[u][x] = make_double2(0.0, 0.0);
  }
  for (int c0 = 0; c0 < M;) {
    const int nl = pl_candidates(P, Gf, M, qc, c0, list, wcount);
    for (int l0 = 0; l0 < nl; l0 += nent) {
      const int n = min(nent, nl - l0);
      __syncthreads();   // the list is written, the previous entries have been read
      if (tid < n) {
        const int gi = list[l0 + tid];
        double g[3];
        for (int d = 0; d < 3; ++d) g[d] = G[3 * gi + d] + qc[d];
        const double qeq = geg(P.eps, g);
        const bool pass = qeq > 0.0 && qeq / P.alph / 4.0 < P.gmax;
        const double f = pass ? exp(-qeq / P.alph / 4.0) / qeq : 0.0;
        const double dgc = pass ? 0.5 * f * (0.25 / P.alph + 1.0 / qeq) : 0.0;
        double dge[3];
        for (int x = 0; x < 3; ++x)
          dge[x] = dgc * ((P.eps[x] + P.eps[3 * x]) * g[0] + (P.eps[x + 3] + P.eps[3 * x + 1]) * g[1] +
                          (P.eps[x + 6] + P.eps[3 * x + 2]) * g[2]);
        double2 *e = psm + (size_t)tid * esz;
        for (int a = 0; a < nat; ++a) {
          double sn, cs;
          sincos(g[0] * P.tau[3 * a] + g[1] * P.tau[3 * a + 1] + g[2] * P.tau[3 * a + 2], &sn, &cs);
          for (int i = 0; i < 3; ++i) {
            const double *Z = P.born + 3 * i + 9 * a;
            const double z = g[0] * Z[0] + g[1] * Z[1] + g[2] * Z[2];
            e[3 * a + i] = make_double2(cs * z, sn * z);
          }
          e[nb + a] = make_double2(f * cs, f * sn);
        }
        e[nb + nat] = make_double2(f, dge[0]);
        e[nb + nat + 1] = make_double2(dge[1], dge[2]);
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < NU; ++u)
        if (hi[u] >= 0)
          for (int k = hs; k < n; k += hsl) {
            const double2 *e = psm + (size_t)k * esz;
            const double2 wi = e[hi[u]], wj = e[hj[u]], f0 = e[nb + nat], f1 = e[nb + nat + 1];
            const double2 r = make_double2(wi.x * wj.x + wi.y * wj.y, wi.y * wj.x - wi.x * wj.y);
            acc[u][0].x += f0.x * r.x;
            acc[u][0].y += f0.x * r.y;
            acc[u][1].x += f0.y * r.x;
            acc[u][1].y += f0.y * r.y;
            acc[u][2].x += f1.x * r.x;
            acc[u][2].y += f1.x * r.y;
            acc[u][3].x += f1.y * r.x;
            acc[u][3].y += f1.y * r.y;
          }
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const int it = p0 + u * PL_THREADS;
        if (ps < psl && it < np)
          for (int k = ps; k < n; k += psl) {
            const double2 *e = psm + (size_t)k * esz;
            cfma(pacc[u], e[nb + it / nb], cconj(e[it % nb]));
          }
      }
    }
  }
  // ---- the slices' sums in order, into the first slice's places
  __syncthreads();
  double2 *pp = psm + (size_t)hsl * 4 * nh;   // [psl][np], behind [hsl][4][nh]
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    const int it = h0 + u * PL_THREADS, ip = p0 + u * PL_THREADS;
    if (hi[u] >= 0)
#pragma unroll
      for (int x = 0; x < 4; ++x) psm[(hs * 4 + x) * nh + it] = acc[u][x];
    if (ps < psl && ip < np) pp[ps * np + ip] = pacc[u];
  }
  __syncthreads();
  for (int t = tid; t < 4 * nh + np; t += PL_THREADS) {
    double2 *o = t < 4 * nh ? psm + t : pp + (t - 4 * nh);
    const int n = t < 4 * nh ? hsl : psl, step = t < 4 * nh ? 4 * nh : np;
    double2 v = *o;
    for (int sl = 1; sl < n; ++sl) v = cadd(v, o[sl * step]);
    *o = v;
  }
  __syncthreads();
  auto herm = [&](int x, int i, int j) {
    const int hi_ = max(i, j), lo = min(i, j);
    const double2 v = psm[x * nh + hi_ * (hi_ + 1) / 2 + lo];
    return i >= j ? v : cconj(v);
  };
  for (int el = tid; el < ne; el += PL_THREADS) {
    const int i = el % nb, j = el / nb, a = i / 3, b = j / 3;
    const double mn = 1.0 / sqrt(P.masses[a] * P.masses[b]) * Ryd2amu;
    const double2 d0 = herm(0, i, j);
    if (Dq) {
      double2 &o = Dq[q * ldd + el];
      o = cadd(o, cscale(P.Da ? cadd(d0, P.Da[el]) : d0, P.fac * mn));
    }
    const double2 pi = pp[a * nb + j], pj = cconj(pp[b * nb + i]);
    for (int x = 0; x < 3; ++x) {
      const double zi = P.born[x + 3 * (i % 3) + 9 * a], zj = P.born[x + 3 * (j % 3) + 9 * b];
      const double rr = P.tau[3 * a + x] - P.tau[3 * b + x];
      const double2 w = herm(1 + x, i, j);
      const double2 d = make_double2(zi * pi.x + zj * pj.x - rr * d0.y - 2.0 * w.x,
                                     zi * pi.y + zj * pj.y + rr * d0.x - 2.0 * w.y);
      double2 &o = dDq[q * ldd + x * ne + el];
      o = cadd(o, cscale(d, P.fac * BOHR2NM * mn));
    }
  }
}

// The box vectors of a launch: all, or those that some q of the first cell can need.
struct PolarBox {
  const double *G;
  const float *Gf;
  int M;
};

template <int NU, bool DA>
static void polar_run(const PolarDev &P, const PolarBox &B, int nq, const int *qp, const int mesh[3], const double *qv,
                      double2 *Dq, int64_t ldd, double2 *Lq, cudaStream_t st) {
  static OncePerDevice attr;
  attr([] { cudaFuncSetAttribute(k_polar<NU, DA>, cudaFuncAttributeMaxDynamicSharedMemorySize, PL_SMEM); });
  const size_t entry = pl_entry_doubles(P.nat, DA) * sizeof(double);
  const int nent = pl_entries(entry);
  k_polar<NU, DA><<<nq, PL_THREADS, nent * entry, st>>>(P, B.G, B.Gf, B.M, nq, qp, mesh ? mesh[0] : 1,
                                                        mesh ? mesh[1] : 1, mesh ? mesh[2] : 1, qv, nent, Dq, ldd, Lq);
}

template <bool DA>
static void polar_dispatch(const PolarDev &P, const PolarBox &B, int nq, const int *qp, const int mesh[3],
                           const double *qv, double2 *Dq, int64_t ldd, double2 *Lq, cudaStream_t st) {
  const int nel = P.nb * P.nb + P.nb;   // matrix + vector elements
  if (nel <= PL_THREADS) polar_run<1, DA>(P, B, nq, qp, mesh, qv, Dq, ldd, Lq, st);
  else if (nel <= 3 * PL_THREADS) polar_run<3, DA>(P, B, nq, qp, mesh, qv, Dq, ldd, Lq, st);
  else polar_run<9, DA>(P, B, nq, qp, mesh, qv, Dq, ldd, Lq, st);
}

template <int NU>
static void polar_vel_run(const PolarDev &P, const PolarBox &B, int nq, const int *qp, const int mesh[3],
                          const double *qv, double2 *Dq, double2 *dDq, int64_t ldd, cudaStream_t st) {
  static OncePerDevice attr;
  attr([] { cudaFuncSetAttribute(k_polar_vel<NU>, cudaFuncAttributeMaxDynamicSharedMemorySize, PL_SMEM); });
  const int nh = P.nb * (P.nb + 1) / 2, np = P.nat * P.nb;
  const size_t entry = (size_t)pv_entry(P.nat) * sizeof(double2);
  const int nent = pl_entries(entry);
  const size_t sums = sizeof(double2) * ((NU == 1 ? PL_THREADS / nh : 1) * 4 * nh + (NU == 1 ? PL_THREADS / np : 1) * np);
  k_polar_vel<NU><<<nq, PL_THREADS, std::max(nent * entry, sums), st>>>(
      P, B.G, B.Gf, B.M, nq, qp, mesh ? mesh[0] : 1, mesh ? mesh[1] : 1, mesh ? mesh[2] : 1, qv, nent, Dq, dDq, ldd);
}

void launch_polar_q(const PolarDev &P, int nq, const int *qp, const int mesh[3], const double *qv, double2 *Dq,
                    double2 *dDq, int64_t ldd, double2 *Lq, cudaStream_t st) {
  if (nq <= 0 || (!Dq && !dDq && !Lq)) return;
  // mesh q lie in the first cell: the box vectors that can pass the cut there suffice
  const PolarBox B = qp ? PolarBox{P.Gcell, P.Gcellf, P.Mcell} : PolarBox{P.G, P.Gf, P.M};
  if (!dDq) {
    polar_dispatch<false>(P, B, nq, qp, mesh, qv, Dq, ldd, Lq, st);
    return;
  }
  if (P.nb * (P.nb + 1) / 2 <= PL_THREADS) polar_vel_run<1>(P, B, nq, qp, mesh, qv, Dq, dDq, ldd, st);
  else polar_vel_run<5>(P, B, nq, qp, mesh, qv, Dq, dDq, ldd, st);
  if (Lq) polar_dispatch<false>(P, B, nq, qp, mesh, qv, nullptr, ldd, Lq, st);
}

void launch_polar_da(const PolarDev &P, double2 *Da, cudaStream_t st) {
  PolarDev Pa = P;
  Pa.Da = nullptr;
  polar_dispatch<true>(Pa, PolarBox{P.G, P.Gf, P.M}, 1, nullptr, nullptr, nullptr, Da, 0, nullptr, st);
}

__global__ void k_glprefac(int nq, int nb, const double2 *Lq, const double2 *u, double2 *glp, float2 *glpf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;   // (q, s)
  if (i >= nq * nb) return;
  const int q = i / nb;
  double2 acc = make_double2(0.0, 0.0);
  for (int c = 0; c < nb; ++c) cfma(acc, Lq[(size_t)q * nb + c], u[(size_t)i * nb + c]);
  glp[i] = acc;
  if (glpf) glpf[i] = make_float2((float)acc.x, (float)acc.y);
}

void launch_glprefac(int nq, int nb, const double2 *Lq, const double2 *u, double2 *glp, float2 *glpf,
                     cudaStream_t st) {
  if (nq <= 0) return;
  k_glprefac<<<(nq * nb + 255) / 256, 256, 0, st>>>(nq, nb, Lq, u, glp, glpf);
}

}  // namespace ephg
