// ephg_polar.cu - the long-range dipole terms of polar crystals on the device:
// dyn_nonanalytic (wannier.f90:784-901) and long_range_prefac (:1013-1071).
//
// For a box vector G and g = G + q, with per-atom phases p_a = e^{i g.tau_a},
// z_a(j) = sum_i g_i born(i, j, a) and w(3a+i) = p_a z_a(i), the G + q term of
// dyn_nonanalytic is a rank-one update
//   D += f w w^H,   f = e^{-qeq/4alph}/qeq,
// its derivative along x is M_x + M_x^H with the outer product
//   M_x += f v_x w^H,   v_x(3a+i) = p_a born(x, i, a) + (i tau_a(x) - dgeg_x (1/4alph + 1/qeq) / 2) w(3a+i),
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
// With velocities (k_polar_vel) every thread sums outer products, the candidates
// split over as many slices as the block has threads per matrix element: 1,728 q,
// 13^3 box: 0.32 ms (1.13 ms with the FP64 test on every box vector, its terms
// formed in partly filled warps and ~70 operations per element and vector).
// Without (k_polar) an element is summed by one thread in the loop order, from
// f p_a conj(p_b) per pair of atoms and z.  The tensor-core rates round the
// eigenvectors to FP32 in the gauge that the eigensolver leaves them in, which the
// last bit of D decides where an off-diagonal element is all rounding: sums in
// another order move those rates by 1e-7, so here the order stays the loop's.
#include <algorithm>
#include <mutex>

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

// With velocities.  Entry of a candidate: complex vectors of nb values: w, f w (right and
// left factors), f v_x for x = 0..2.
constexpr int PV_VECTORS = 5;

template <int NU>
__global__ void __launch_bounds__(PL_THREADS) k_polar_vel(PolarDev P, const double *G, const float *Gf, int M, int nq,
                                                          const int *qp, int m1, int m2, int m3, const double *qv,
                                                          int nent, double2 *Dq, double2 *dDq, int64_t ldd,
                                                          double2 *Lq) {
  extern __shared__ double2 psm[];   // [nent][vectors][nb]
  __shared__ int list[PL_LIST];
  __shared__ int wcount[PL_THREADS / 32];
  constexpr int NV = PV_VECTORS;
  const int q = blockIdx.x;
  const int nat = P.nat, nb = P.nb, ne = nb * nb;
  const int tid = threadIdx.x;
  double qc[3];
  pl_q(P, q, nq, qp, m1, m2, m3, qv, qc);
  // thread's elements: el = tid + u PL_THREADS of the nb^2 matrix and nb vector elements, or
  // (NU = 1) element tid % nel of slice tid / nel
  const int nel = ne + nb, nsl = NU == 1 ? PL_THREADS / nel : 1;
  const int slice = NU == 1 ? tid / nel : 0, el0 = NU == 1 ? tid % nel : tid;
  const bool work = slice < nsl;
  double2 acc[NU], dacc[NU][3];
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    acc[u] = make_double2(0.0, 0.0);
#pragma unroll
    for (int x = 0; x < 3; ++x) dacc[u][x] = make_double2(0.0, 0.0);
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
        const double dgc = pass ? 0.5 * (0.25 / P.alph + 1.0 / qeq) : 0.0;
        double dge[3];
        for (int x = 0; x < 3; ++x)
          dge[x] = dgc * ((P.eps[x] + P.eps[3 * x]) * g[0] + (P.eps[x + 3] + P.eps[3 * x + 1]) * g[1] +
                          (P.eps[x + 6] + P.eps[3 * x + 2]) * g[2]);
        double2 *e = psm + (size_t)tid * NV * nb;
        for (int a = 0; a < nat; ++a) {
          double sn, cs;
          sincos(g[0] * P.tau[3 * a] + g[1] * P.tau[3 * a + 1] + g[2] * P.tau[3 * a + 2], &sn, &cs);
          for (int i = 0; i < 3; ++i) {
            const double *Z = P.born + 3 * i + 9 * a;
            const double z = g[0] * Z[0] + g[1] * Z[1] + g[2] * Z[2];
            const double2 w = make_double2(cs * z, sn * z);
            e[3 * a + i] = w;
            e[nb + 3 * a + i] = cscale(w, f);
            for (int x = 0; x < 3; ++x) {
              const double t = P.tau[3 * a + x];
              e[(2 + x) * nb + 3 * a + i] = make_double2(f * (cs * Z[x] - dge[x] * w.x - t * w.y),
                                                         f * (sn * Z[x] - dge[x] * w.y + t * w.x));
            }
          }
        }
      }
      __syncthreads();
      if (work)
#pragma unroll
        for (int u = 0; u < NU; ++u) {
          const int el = el0 + u * PL_THREADS;
          if (el < ne) {
            const int i = el % nb, j = el / nb;
            for (int k = slice; k < n; k += nsl) {
              const double2 *e = psm + (size_t)k * NV * nb;
              const double2 r = cconj(e[j]);
              cfma(acc[u], e[nb + i], r);
#pragma unroll
              for (int x = 0; x < 3; ++x) cfma(dacc[u][x], e[(2 + x) * nb + i], r);
            }
          } else if (el < nel && Lq) {
            for (int k = slice; k < n; k += nsl) acc[u] = cadd(acc[u], psm[(size_t)k * NV * nb + nb + (el - ne)]);
          }
        }
    }
  }
  // ---- the slices' sums in order; M_x and its transpose meet in shared memory
  __syncthreads();
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    const int el = el0 + u * PL_THREADS;
    if (work && el < nel) {
      psm[(size_t)(slice * 4) * nel + el] = acc[u];
#pragma unroll
      for (int x = 0; x < 3; ++x) psm[(size_t)(slice * 4 + 1 + x) * nel + el] = dacc[u][x];
    }
  }
  __syncthreads();
  auto sum = [&](int c, int el) {
    double2 t = psm[(size_t)c * nel + el];
    for (int sl = 1; sl < nsl; ++sl) t = cadd(t, psm[(size_t)(sl * 4 + c) * nel + el]);
    return t;
  };
  for (int el = tid; el < nel; el += PL_THREADS) {
    if (el < ne) {
      const int i = el % nb, j = el / nb;
      const double mn = 1.0 / sqrt(P.masses[i / 3] * P.masses[j / 3]) * Ryd2amu;
      if (Dq) {
        double2 d = sum(0, el);
        if (P.Da) d = cadd(d, P.Da[el]);
        double2 &o = Dq[q * ldd + el];
        o = cadd(o, cscale(d, P.fac * mn));
      }
      for (int x = 0; x < 3; ++x) {
        double2 &o = dDq[q * ldd + x * ne + el];
        o = cadd(o, cscale(cadd(sum(1 + x, el), cconj(sum(1 + x, j + nb * i))), P.fac * BOHR2NM * mn));
      }
    } else if (Lq) {
      const double2 t = sum(0, el);
      Lq[(size_t)q * nb + (el - ne)] = make_double2(P.fac * t.y, P.fac * t.x);   // i fac conj(t)
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
  // once per process: changing a kernel attribute can wait for the device's queued work
  static std::once_flag once;
  std::call_once(once, [] {
    cudaFuncSetAttribute(k_polar<NU, DA>, cudaFuncAttributeMaxDynamicSharedMemorySize, PL_SMEM);
  });
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
                          const double *qv, double2 *Dq, double2 *dDq, int64_t ldd, double2 *Lq, cudaStream_t st) {
  static std::once_flag once;
  std::call_once(once, [] {
    cudaFuncSetAttribute(k_polar_vel<NU>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * PL_SMEM);
  });
  const int nel = P.nb * P.nb + P.nb;
  const size_t entry = (size_t)PV_VECTORS * P.nb * sizeof(double2);
  const int nent = pl_entries(entry);
  const size_t sums = (size_t)(NU == 1 ? PL_THREADS / nel : 1) * 4 * nel * sizeof(double2);
  k_polar_vel<NU><<<nq, PL_THREADS, std::max(nent * entry, sums), st>>>(
      P, B.G, B.Gf, B.M, nq, qp, mesh ? mesh[0] : 1, mesh ? mesh[1] : 1, mesh ? mesh[2] : 1, qv, nent, Dq, dDq, ldd, Lq);
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
  const int nel = P.nb * P.nb + P.nb;
  if (nel <= PL_THREADS) polar_vel_run<1>(P, B, nq, qp, mesh, qv, Dq, dDq, ldd, Lq, st);
  else if (nel <= 3 * PL_THREADS) polar_vel_run<3>(P, B, nq, qp, mesh, qv, Dq, dDq, ldd, Lq, st);
  else polar_vel_run<9>(P, B, nq, qp, mesh, qv, Dq, dDq, ldd, Lq, st);
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
