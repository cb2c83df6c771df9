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
// vectors pass), the candidates are listed in the reference's loop order, one
// thread per candidate decides the cut in FP64 and forms w and v_x, and every
// thread then sums outer products, the candidates split over as many slices as
// the block has threads per matrix element.  Fixed order throughout:
// deterministic sums.  For q on the mesh (first cell) only the box vectors that
// can pass for some q of the cell are tested; the others never contribute.
// 1,728 q with velocities, 13^3 box: 0.32 ms (1.13 ms with the FP64 test on every box
// vector, its terms formed in partly filled warps and ~70 operations per
// element and vector).
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

// Entry of a candidate: complex vectors of nb values: w, f w (right and left factors),
// with VEL f v_x for x = 0..2.  DA (the q-independent sum, wannier.f90:843-867): the right
// factor is sum_c w(3c + i % 3), the left one -f w, and only blocks of one atom are kept.
static int pl_vectors(bool vel) { return vel ? 5 : 2; }
static int pl_entries(int nb, bool vel) {
  return std::min(PL_THREADS, (int)(PL_SMEM / (pl_vectors(vel) * nb * sizeof(double2))));
}

// NU: matrix + vector elements per thread (nb^2 + nb <= NU * PL_THREADS).
// G / Gf / M: the box vectors to test, FP64 and FP32.
template <int NU, bool VEL, bool DA>
__global__ void __launch_bounds__(PL_THREADS) k_polar(PolarDev P, const double *G, const float *Gf, int M, int nq,
                                                      const int *qp, int m1, int m2, int m3, const double *qv, int nent,
                                                      double2 *Dq, double2 *dDq, int64_t ldd, double2 *Lq) {
  extern __shared__ double2 psm[];   // [nent][vectors][nb]
  __shared__ int list[PL_LIST];
  __shared__ int wcount[PL_THREADS / 32];
  constexpr int NV = VEL ? 5 : 2;
  const int q = blockIdx.x;
  const int nat = P.nat, nb = P.nb, ne = nb * nb;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double qc[3] = {0.0, 0.0, 0.0};
  if (!DA) {
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
    for (int d = 0; d < 3; ++d)   // matmul(reclattvecs, q) * bohr2nm
      qc[d] = (P.rec[d] * qf[0] + P.rec[d + 3] * qf[1] + P.rec[d + 6] * qf[2]) * BOHR2NM;
  }
  const float qcf[3] = {(float)qc[0], (float)qc[1], (float)qc[2]};
  float epsf[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) epsf[i] = (float)P.eps[i];
  const float lim = (float)(4.0 * P.alph * P.gmax) * 1.00001f;
  // thread's elements: el = tid + u PL_THREADS of the nb^2 matrix and nb vector elements, or
  // (NU = 1) element tid % nel of slice tid / nel
  const int nel = ne + nb, nsl = NU == 1 ? PL_THREADS / nel : 1;
  const int slice = NU == 1 ? tid / nel : 0, el0 = NU == 1 ? tid % nel : tid;
  const bool work = slice < nsl;
  double2 acc[NU], dacc[VEL ? NU : 1][3];
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    acc[u] = make_double2(0.0, 0.0);
    if (VEL)
#pragma unroll
      for (int x = 0; x < 3; ++x) dacc[u][x] = make_double2(0.0, 0.0);
  }
  for (int c0 = 0; c0 < M;) {
    // ---- list the candidates of the next box vectors, in order
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
    // ---- work them off
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
        double dge[3] = {0.0, 0.0, 0.0};
        if (VEL)
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
            e[nb + 3 * a + i] = cscale(w, DA ? -f : f);
            if (VEL)
              for (int x = 0; x < 3; ++x) {
                const double t = P.tau[3 * a + x];
                e[(2 + x) * nb + 3 * a + i] = make_double2(f * (cs * Z[x] - dge[x] * w.x - t * w.y),
                                                           f * (sn * Z[x] - dge[x] * w.y + t * w.x));
              }
          }
        }
        if (DA)
          for (int i = 0; i < 3; ++i) {
            double2 t = make_double2(0.0, 0.0);
            for (int a = 0; a < nat; ++a) t = cadd(t, e[3 * a + i]);
            for (int a = 0; a < nat; ++a) e[3 * a + i] = t;
          }
      }
      __syncthreads();
      if (work)
#pragma unroll
        for (int u = 0; u < NU; ++u) {
          const int el = el0 + u * PL_THREADS;
          if (el < ne) {
            const int i = el % nb, j = el / nb;
            if (DA && i / 3 != j / 3) continue;
            for (int k = slice; k < n; k += nsl) {
              const double2 *e = psm + (size_t)k * NV * nb;
              const double2 r = cconj(e[j]);
              cfma(acc[u], e[nb + i], r);
              if (VEL)
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
  const int nq4 = VEL ? 4 : 1;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    const int el = el0 + u * PL_THREADS;
    if (work && el < nel) {
      psm[(size_t)(slice * nq4) * nel + el] = acc[u];
      if (VEL)
#pragma unroll
        for (int x = 0; x < 3; ++x) psm[(size_t)(slice * nq4 + 1 + x) * nel + el] = dacc[u][x];
    }
  }
  __syncthreads();
  auto sum = [&](int c, int el) {
    double2 t = psm[(size_t)c * nel + el];
    for (int sl = 1; sl < nsl; ++sl) t = cadd(t, psm[(size_t)(sl * nq4 + c) * nel + el]);
    return t;
  };
  for (int el = tid; el < nel; el += PL_THREADS) {
    if (el < ne) {
      const int i = el % nb, j = el / nb;
      if (DA) {
        Dq[el] = sum(0, el);
        continue;
      }
      const double mn = 1.0 / sqrt(P.masses[i / 3] * P.masses[j / 3]) * Ryd2amu;
      if (Dq) {
        double2 d = sum(0, el);
        if (P.Da) d = cadd(d, P.Da[el]);
        double2 &o = Dq[q * ldd + el];
        o = cadd(o, cscale(d, P.fac * mn));
      }
      if (VEL && dDq)
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

template <int NU, bool VEL, bool DA>
static void polar_run(const PolarDev &P, const double *G, const float *Gf, int M, int nq, const int *qp,
                      const int mesh[3], const double *qv, double2 *Dq, double2 *dDq, int64_t ldd, double2 *Lq,
                      cudaStream_t st) {
  // once per process: changing a kernel attribute can wait for the device's queued work
  static std::once_flag once;
  std::call_once(once, [] {
    cudaFuncSetAttribute(k_polar<NU, VEL, DA>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * PL_SMEM);
  });
  const int nent = pl_entries(P.nb, VEL), nel = P.nb * P.nb + P.nb;
  const size_t entries = (size_t)nent * pl_vectors(VEL) * P.nb;
  const size_t sums = (size_t)(NU == 1 ? PL_THREADS / nel : 1) * (VEL ? 4 : 1) * nel;
  k_polar<NU, VEL, DA><<<nq, PL_THREADS, std::max(entries, sums) * sizeof(double2), st>>>(
      P, G, Gf, M, nq, qp, mesh ? mesh[0] : 1, mesh ? mesh[1] : 1, mesh ? mesh[2] : 1, qv, nent, Dq, dDq, ldd, Lq);
}

template <bool VEL, bool DA>
static void polar_dispatch(const PolarDev &P, const double *G, const float *Gf, int M, int nq, const int *qp,
                           const int mesh[3], const double *qv, double2 *Dq, double2 *dDq, int64_t ldd, double2 *Lq,
                           cudaStream_t st) {
  const int nel = P.nb * P.nb + P.nb;   // matrix + vector elements
  if (nel <= PL_THREADS) polar_run<1, VEL, DA>(P, G, Gf, M, nq, qp, mesh, qv, Dq, dDq, ldd, Lq, st);
  else if (nel <= 3 * PL_THREADS) polar_run<3, VEL, DA>(P, G, Gf, M, nq, qp, mesh, qv, Dq, dDq, ldd, Lq, st);
  else polar_run<9, VEL, DA>(P, G, Gf, M, nq, qp, mesh, qv, Dq, dDq, ldd, Lq, st);
}

void launch_polar_q(const PolarDev &P, int nq, const int *qp, const int mesh[3], const double *qv, double2 *Dq,
                    double2 *dDq, int64_t ldd, double2 *Lq, cudaStream_t st) {
  if (nq <= 0 || (!Dq && !dDq && !Lq)) return;
  // mesh q lie in the first cell: the box vectors that can pass the cut there suffice
  const double *G = qp ? P.Gcell : P.G;
  const float *Gf = qp ? P.Gcellf : P.Gf;
  const int M = qp ? P.Mcell : P.M;
  if (dDq) polar_dispatch<true, false>(P, G, Gf, M, nq, qp, mesh, qv, Dq, dDq, ldd, Lq, st);
  else polar_dispatch<false, false>(P, G, Gf, M, nq, qp, mesh, qv, Dq, nullptr, ldd, Lq, st);
}

void launch_polar_da(const PolarDev &P, double2 *Da, cudaStream_t st) {
  PolarDev Pa = P;
  Pa.Da = nullptr;
  polar_dispatch<false, true>(Pa, P.G, P.Gf, P.M, 1, nullptr, nullptr, nullptr, Da, nullptr, 0, nullptr, st);
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
