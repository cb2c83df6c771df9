// ephg_kernels.cu - FP64 set-up and drop-in kernels of the e-ph vertex path.
//
// Phase tables, Fourier sums over cells, the batched Hermitian Jacobi eigensolver (one to
// four matrices per block), the FP64 complex GEMM of the call that may not allocate, and
// the per-(state, final states) epilogue that forms |g|^2, X+- and the RTA rate partials.
// Each kernel names the reference lines it restates.
#include <algorithm>
#include <cstdio>
#include <type_traits>
#include <vector>

#include "../../include/ephg_debug.h"
#include "ephg_kernels.cuh"

namespace ephg {

static constexpr double PI = 3.141592653589793;   // 4*atan(1), params.f90:44
static constexpr double TWOPI = 2.0 * PI;

// =================================================================== phases

__global__ void k_roots(int L, double2 *roots) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= L) return;
  double s, c;
  sincospi(2.0 * (double)t / (double)L, &s, &c);
  roots[t] = make_double2(c, s);
}

void launch_roots(int L, double2 *roots, cudaStream_t st) {
  k_roots<<<(L + 255) / 256, 256, 0, st>>>(L, roots);
}

// exact integer modular phase index of k (mesh index p) and integer R
__device__ inline int phase_index(int p, const int mesh[3], int L, int r1, int r2, int r3) {
  int v1 = p % mesh[0];
  int v2 = (p / mesh[0]) % mesh[1];
  int v3 = p / (mesh[0] * mesh[1]);
  int64_t t = (int64_t)v1 * r1 * (L / mesh[0]) + (int64_t)v2 * r2 * (L / mesh[1]) +
              (int64_t)v3 * r3 * (L / mesh[2]);
  return (int)floormod(t, L);
}

__global__ void k_phase_mesh(int nrows, const int *rowp, int m1, int m2, int m3, int L, int nR,
                             const int *R, const double *deg, int conj, const double2 *roots,
                             double2 *out, int64_t ldo) {
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)nrows * nR) return;
  int row = (int)(idx / nR), r = (int)(idx % nR);
  int p = rowp ? rowp[row] : row;
  const int mesh[3] = {m1, m2, m3};
  int t = phase_index(p, mesh, L, R[3 * r], R[3 * r + 1], R[3 * r + 2]);
  double2 v = roots[t];
  if (conj) v.y = -v.y;
  if (deg) { v.x /= deg[r]; v.y /= deg[r]; }
  out[(int64_t)row * ldo + r] = v;
}

void launch_phase_mesh(int nrows, const int *rowp, const int mesh[3], int L, int nR,
                       const int *R, const double *deg, int conj, const double2 *roots,
                       double2 *out, int64_t ldo, cudaStream_t st) {
  int64_t n = (int64_t)nrows * nR;
  if (n == 0) return;
  k_phase_mesh<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(nrows, rowp, mesh[0], mesh[1],
                                                             mesh[2], L, nR, R, deg, conj,
                                                             roots, out, ldo);
}

// ---- a Fourier sum over integer cells onto a whole mesh, one dimension at a time ----
// On a mesh, sum_R e^{2 pi i k.R} X(R) separates: with X placed on the box of
// cell coordinates [lo, lo + ext) per dimension (zero where there is no cell),
// three 1-D sums of ext terms each replace the N_k x N_R phase matrix and its
// GEMM (for H(k), wannier.f90:467-479: ~40x fewer FP64 flops at 24^3, 6^3 WS).
// Every factor e^{2 pi i v (r + lo) / m} is the exact integer-indexed root of
// unity.  One pass: out[a][v][b][e] = sum_r root(v (r + lo) L / m) in[a][r][b][e],
// or with TRANS out[a][b][v][e]: the second and third passes write [r1][v3][v2]
// and then [v3][v2][v1], the muxed mesh index v1 + m1 (v2 + m2 v3) in row order.
template <bool TRANS>
__global__ void k_dft1(int64_t total, int R, int B, int M, int nn, int lo, int Lm, int L,
                       const double2 *__restrict__ roots, const double2 *__restrict__ in,
                       double2 *__restrict__ out) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int e = (int)(idx % nn);
  int64_t t = idx / nn;
  const int b = (int)(t % B);
  t /= B;
  const int v = (int)(t % M);
  const int64_t a = t / M;
  double2 acc = make_double2(0.0, 0.0);
  for (int r = 0; r < R; ++r)
    cfma(acc, roots[floormod((int64_t)v * (r + lo) * Lm, L)], in[((a * R + r) * B + b) * nn + e]);
  out[TRANS ? ((a * B + b) * M + v) * nn + e : idx] = acc;
}

void launch_mesh_fourier(const double2 *box, const int lo[3], const int ext[3], int nn, const int mesh[3], int L,
                         const double2 *roots, double2 *t1, double2 *t2, double2 *out, cudaStream_t st) {
  const int64_t n1 = (int64_t)ext[0] * ext[1] * mesh[2] * nn, n2 = (int64_t)ext[0] * mesh[1] * mesh[2] * nn,
                n3 = (int64_t)mesh[0] * mesh[1] * mesh[2] * nn;
  // along R3: [r1 r2][r3][e] -> [r1 r2][v3][e]
  k_dft1<false><<<(unsigned)((n1 + 255) / 256), 256, 0, st>>>(n1, ext[2], 1, mesh[2], nn, lo[2], L / mesh[2], L,
                                                              roots, box, t1);
  // along R2: [r1][r2][v3][e] -> [r1][v3][v2][e]
  k_dft1<true><<<(unsigned)((n2 + 255) / 256), 256, 0, st>>>(n2, ext[1], mesh[2], mesh[1], nn, lo[1], L / mesh[1],
                                                             L, roots, t1, t2);
  // along R1: [r1][v3 v2][e] -> [v3 v2][v1][e], rows in muxed mesh order
  k_dft1<true><<<(unsigned)((n3 + 255) / 256), 256, 0, st>>>(n3, ext[0], mesh[1] * mesh[2], mesh[0], nn, lo[0],
                                                             L / mesh[0], L, roots, t2, out);
}

// ---- the same for many columns at once: the contractions of the FP64 rate path ----
// Both contractions of the rate path are Fourier sums of cells onto mesh points
// (stage A: g(Re,Rp) over Re for every column of g; stage B: the state operand
// over Rp).  As matrix products against the phase matrix they are bound by the
// FP64 pipe (1.25 TFLOP/s), so what counts is FP64 instructions: one dimension
// at a time needs ~25x fewer of them (12^3 mesh, 279 cells: 402k complex
// multiply-adds a column become 25k), and the symmetric range of cells halves
// them twice more.  With s_r = x_r + x_-r and d_r = x_r - x_-r,
//   y_v = x_0 + sum_r cos(2 pi v r / m) s_r + i sin(2 pi v r / m) d_r,
// and y_-v has the same two sums with the second one subtracted: 4 FMA serve two
// cells and two outputs that take 16 as complex products.
//
// One thread owns a column of one line (all of its outputs), so that loads and
// stores run along the columns and the roots are shared-memory broadcasts; a
// line's s and d sit in shared memory, [2 h + 1][128 threads].  An FP64
// instruction of a warp holds the pipe for 16 cycles, so the ~3 shared loads
// per 4 FMA are hidden at any occupancy of a few warps.  Measured, 12^3, nw 8, nb 6,
// 279 cells (both contractions): 14.7 ms, 0.95 of the FP64 rate for the instructions
// counted by cells_fourier_cost; matrix products on that pipe took 468 ms at 1.23 TFLOP/s.
constexpr int CF_THREADS = 128;
constexpr int CF_MAXM = 1024;                 // mesh points per dimension (shared root table)
constexpr int CF_SMEM = 160 * 1024;

struct CellDft {
  int64_t nlines;
  int B, m, Lm;          // lines (a, b): a = line / B, b = line % B; m outputs; root step L / m
  int lo, ext, h;        // cell coordinates [lo, lo + ext), h = max |r|
  const int *tab;        // [a][ext]: input row group or -1
  int nc, ncb;           // columns, column blocks
  const double2 *in, *roots;
  int64_t ldi, ldo;
  const double *scale;   // per input row group (nullable)
  const int *rowmap;     // output row of (line, v) (nullable: line m + v)
  double2 *out;
};

__global__ void __launch_bounds__(CF_THREADS) k_cells_dft(CellDft g) {
  extern __shared__ double2 cfs[];
  double2 *sr = cfs, *sx = cfs + g.m + threadIdx.x;   // sx[u * CF_THREADS]: x_0, then s_r, d_r
  const int64_t line = blockIdx.x / g.ncb;
  const int c = (int)(blockIdx.x % g.ncb) * CF_THREADS + threadIdx.x;
  const int a = (int)(line / g.B), b = (int)(line % g.B);
  for (int t = threadIdx.x; t < g.m; t += CF_THREADS) sr[t] = g.roots[(int64_t)t * g.Lm];
  const int *tab = g.tab + (int64_t)a * g.ext;
  const bool live = c < g.nc;
  auto fetch = [&](int r) {
    const int u = r - g.lo;
    const int t = (live && u >= 0 && u < g.ext) ? tab[u] : -1;
    if (t < 0) return make_double2(0.0, 0.0);
    const double2 x = g.in[((int64_t)t * g.B + b) * g.ldi + c];
    return g.scale ? cscale(x, g.scale[t]) : x;
  };
  const double2 x0 = fetch(0);
#pragma unroll 2
  for (int r = 1; r <= g.h; ++r) {
    const double2 p = fetch(r), q = fetch(-r);
    sx[(2 * r - 1) * CF_THREADS] = cadd(p, q);
    sx[2 * r * CF_THREADS] = csub(p, q);
  }
  __syncthreads();
  if (!live) return;
  for (int v = 0; 2 * v <= g.m; ++v) {
    const int w = (v == 0 || 2 * v == g.m) ? -1 : g.m - v;   // the mirrored output
    int64_t o1 = line * g.m + v, o2 = w < 0 ? -1 : line * g.m + w;
    if (g.rowmap) {
      o1 = g.rowmap[o1];
      if (o2 >= 0) o2 = g.rowmap[o2];
      if (o1 < 0 && o2 < 0) continue;
    }
    double2 P = x0, Q = make_double2(0.0, 0.0);
    int idx = 0;
#pragma unroll 4
    for (int r = 1; r <= g.h; ++r) {
      idx += v;
      if (idx >= g.m) idx -= g.m;
      const double2 e = sr[idx], s = sx[(2 * r - 1) * CF_THREADS], d = sx[2 * r * CF_THREADS];
      P.x = fma(e.x, s.x, P.x);
      P.y = fma(e.x, s.y, P.y);
      Q.x = fma(e.y, d.x, Q.x);
      Q.y = fma(e.y, d.y, Q.y);
    }
    if (o1 >= 0) g.out[o1 * g.ldo + c] = make_double2(P.x - Q.y, P.y + Q.x);
    if (o2 >= 0) g.out[o2 * g.ldo + c] = make_double2(P.x + Q.y, P.y - Q.x);
  }
}

static int cells_h(const CellTab &t, int d) { return std::max(0, std::max(-t.lo[d], t.lo[d] + t.ext[d] - 1)); }

static size_t cells_smem(const CellTab &t, int d, int m) {
  return sizeof(double2) * ((size_t)m + (size_t)(2 * cells_h(t, d) + 1) * CF_THREADS);
}

double cells_fourier_cost(const CellTab &t, const int mesh[3], int64_t rows) {
  if (!t.ok) return INFINITY;
  for (int d = 0; d < 3; ++d)
    if (mesh[d] > CF_MAXM || cells_smem(t, d, mesh[d]) > (size_t)CF_SMEM) return INFINITY;
  auto line = [&](int d) {   // a line's instructions: 4 h + 4 per output pair, 4 h to form s and d
    const double h = cells_h(t, d);
    return (mesh[d] / 2 + 1) * (4 * h + 4) + 4 * h;
  };
  const double full = (double)mesh[0] * mesh[1] * mesh[2];
  return t.npair * line(2) + (double)t.n1 * mesh[2] * line(1) +
         (double)mesh[1] * mesh[2] * line(0) * std::min(1.0, 2.0 * rows / full);
}

void launch_cells_fourier(const CellTab &t, const double2 *in, int64_t ldi, const double *scale, int nc,
                          const int mesh[3], int L, const double2 *roots, double2 *t1, double2 *t2,
                          const int *rowmap, double2 *out, int64_t ldo, cudaStream_t st) {
  if (nc <= 0) return;
  static OncePerDevice attr;
  attr([] { cudaFuncSetAttribute(k_cells_dft, cudaFuncAttributeMaxDynamicSharedMemorySize, CF_SMEM); });
  auto pass = [&](int d, int64_t A, int B, const int *tab, const double2 *src, int64_t ls, const double *sc,
                  const int *map, double2 *dst, int64_t ld) {
    CellDft g;
    g.nlines = A * B;
    g.B = B;
    g.m = mesh[d];
    g.Lm = L / mesh[d];
    g.lo = t.lo[d];
    g.ext = t.ext[d];
    g.h = cells_h(t, d);
    g.tab = tab;
    g.nc = nc;
    g.ncb = (nc + CF_THREADS - 1) / CF_THREADS;
    g.in = src;
    g.roots = roots;
    g.ldi = ls;
    g.ldo = ld;
    g.scale = sc;
    g.rowmap = map;
    g.out = dst;
    k_cells_dft<<<(unsigned)(g.nlines * g.ncb), CF_THREADS, cells_smem(t, d, mesh[d]), st>>>(g);
  };
  pass(2, t.npair, 1, t.tab1, in, ldi, scale, nullptr, t1, nc);                    // [pair][v3]
  pass(1, t.n1, mesh[2], t.tab2, t1, nc, nullptr, nullptr, t2, nc);                // [r1][v3][v2]
  pass(0, 1, mesh[1] * mesh[2], t.tab3, t2, nc, nullptr, rowmap, out, ldo);        // [v3 v2][v1]: muxed mesh rows
}

__global__ void k_row_map(int nrows, const int *rows, int *rowmap) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nrows) rowmap[rows[i]] = i;
}

void launch_row_map(int N, int nrows, const int *rows, int *rowmap, cudaStream_t st) {
  cudaMemsetAsync(rowmap, 0xFF, (size_t)N * sizeof(int), st);
  if (nrows > 0) k_row_map<<<(nrows + 255) / 256, 256, 0, st>>>(nrows, rows, rowmap);
}

// expi(twopi * dot_product(k, R)) / deg, misc.f90:588 with wannier.f90:467,1097
__global__ void k_phase_frac(int nrows, const double *kv, int nR, const int *R,
                             const double *deg, double2 *out, int64_t ldo) {
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)nrows * nR) return;
  int row = (int)(idx / nR), r = (int)(idx % nR);
  double dot = kv[row] * (double)R[3 * r];
  dot += kv[row + nrows] * (double)R[3 * r + 1];
  dot += kv[row + 2 * nrows] * (double)R[3 * r + 2];
  double s, c;
  sincos(TWOPI * dot, &s, &c);
  double2 v = make_double2(c, s);
  if (deg) { v.x /= deg[r]; v.y /= deg[r]; }
  out[(int64_t)row * ldo + r] = v;
}

void launch_phase_frac(int nrows, const double *kv, int nR, const int *R, const double *deg,
                       double2 *out, int64_t ldo, cudaStream_t st) {
  int64_t n = (int64_t)nrows * nR;
  if (n == 0) return;
  k_phase_frac<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(nrows, kv, nR, R, deg, out, ldo);
}

// The same for many rows (row r the vector perm[r], r itself if perm is null; kv's column
// stride ldk), from tables of e^{2 pi i k_d n} over the cells' range (lo, ext) of each dimension:
// two complex products per cell instead of an FP64 sincos of ~40 operations, and the
// angles are rounded per dimension and exactly reduced.  A block takes ROWS rows: four
// where there are many, one where the call waits for a few.
// 4,001 rows of 165 cells: 36 us (63 with a sincos and two divisions per cell).
constexpr int PC_TAB = 128, PC_THREADS = 128;

template <int ROWS>
__global__ void __launch_bounds__(PC_THREADS) k_phase_cells(int nrows, const double *kv, int64_t ldk, const int *perm,
                                                            int nR, const int *R, const double *deg, int lo0, int lo1,
                                                            int lo2, int e0, int e1, int e2, double2 *out,
                                                            int64_t ldo) {
  constexpr int T = PC_THREADS / ROWS;   // threads of a row
  __shared__ double2 tabs[ROWS][PC_TAB];
  const int lane = threadIdx.x % T, w = threadIdx.x / T;
  const int row = blockIdx.x * ROWS + w;
  const bool live = row < nrows;
  double2 *tab = tabs[w];
  if (live) {
    const int64_t k = perm ? perm[row] : row;
    const double k0 = kv[k], k1 = kv[k + ldk], k2 = kv[k + 2 * ldk];
    for (int i = lane; i < e0 + e1 + e2; i += T) {
      const double x = i < e0 ? k0 * (lo0 + i) : i < e0 + e1 ? k1 * (lo1 + i - e0) : k2 * (lo2 + i - e0 - e1);
      sincospi(2.0 * x, &tab[i].y, &tab[i].x);
    }
  }
  __syncthreads();
  if (!live) return;
  for (int r = lane; r < nR; r += T) {
    double2 v = cmul(cmul(tab[R[3 * r] - lo0], tab[e0 + R[3 * r + 1] - lo1]), tab[e0 + e1 + R[3 * r + 2] - lo2]);
    if (deg) v = cscale(v, 1.0 / deg[r]);
    out[(int64_t)row * ldo + r] = v;
  }
}

// ranges too long for the tables
__global__ void k_phase_list(int nrows, const double *kv, int64_t ldk, const int *perm, int nR, const int *R,
                             const double *deg, double2 *out, int64_t ldo) {
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)nrows * nR) return;
  const int row = (int)(idx / nR), r = (int)(idx % nR);
  const int64_t k = perm ? perm[row] : row;
  double dot = kv[k] * (double)R[3 * r];
  dot += kv[k + ldk] * (double)R[3 * r + 1];
  dot += kv[k + 2 * ldk] * (double)R[3 * r + 2];
  double s, c;
  sincos(TWOPI * dot, &s, &c);
  const double d = deg ? deg[r] : 1.0;
  out[(int64_t)row * ldo + r] = make_double2(c / d, s / d);
}

void launch_phase_cells(int nrows, const double *kv, int64_t ldk, const int *perm, int nR, const int *R,
                        const double *deg, const int lo[3], const int ext[3], double2 *out, int64_t ldo,
                        cudaStream_t st) {
  const int64_t n = (int64_t)nrows * nR;
  if (n <= 0) return;
  auto go = [&](auto kernel, int rows) {
    kernel<<<(nrows + rows - 1) / rows, PC_THREADS, 0, st>>>(nrows, kv, ldk, perm, nR, R, deg, lo[0], lo[1], lo[2],
                                                             ext[0], ext[1], ext[2], out, ldo);
  };
  if (ext[0] + ext[1] + ext[2] <= PC_TAB)
    nrows > 2048 ? go(k_phase_cells<4>, 4) : go(k_phase_cells<1>, 1);
  else
    k_phase_list<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(nrows, kv, ldk, perm, nR, R, deg, out, ldo);
}

// ============================================================ FP64 GEMM
// C[M][N] = A[M][K] * B[K][N], complex double, row-major.  32x64 tile per 256-thread
// block, 2x4 complex outputs per thread; FP64-FMA bound on GB300.  For the call that
// may not allocate; every other product runs on the tensor cores (launch_xgemm), which
// needs a buffer for its digits.
constexpr int ZBM = 32, ZBN = 64, ZBK = 8, ZRM = ZBM / 16;

__global__ void __launch_bounds__(256) k_zgemm(int M, int N, int K, const double2 *__restrict__ A,
                                               int64_t lda, const double2 *__restrict__ B,
                                               int64_t ldb, double2 *__restrict__ C, int64_t ldc) {
  __shared__ double2 sA[ZBK][ZBM + 1];
  __shared__ double2 sB[ZBK][ZBN];
  const int t = threadIdx.x, tx = t % 16, ty = t / 16;
  const int64_t m0 = (int64_t)blockIdx.y * ZBM, n0 = (int64_t)blockIdx.x * ZBN;
  double2 acc[ZRM][4];
#pragma unroll
  for (int i = 0; i < ZRM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_double2(0.0, 0.0);
  for (int k0 = 0; k0 < K; k0 += ZBK) {
    for (int idx = t; idx < ZBM * ZBK; idx += 256) {
      int row = idx / ZBK, kk = idx % ZBK;
      int64_t gm = m0 + row;
      int gk = k0 + kk;
      sA[kk][row] = (gm < M && gk < K) ? A[gm * lda + gk] : make_double2(0.0, 0.0);
    }
    for (int idx = t; idx < ZBK * ZBN; idx += 256) {
      int kb = idx / ZBN, col = idx % ZBN;
      int64_t gn = n0 + col;
      int gkb = k0 + kb;
      sB[kb][col] = (gn < N && gkb < K) ? B[(int64_t)gkb * ldb + gn] : make_double2(0.0, 0.0);
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < ZBK; ++kk) {
      double2 a[ZRM], b[4];
#pragma unroll
      for (int i = 0; i < ZRM; ++i) a[i] = sA[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = sB[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < ZRM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) cfma(acc[i][j], a[i], b[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < ZRM; ++i) {
    int64_t gm = m0 + ty + 16 * i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int64_t gn = n0 + tx + 16 * j;
      if (gn < N) C[gm * ldc + gn] = acc[i][j];
    }
  }
}

void launch_zgemm(int M, int N, int K, const double2 *A, int64_t lda, const double2 *B,
                  int64_t ldb, double2 *C, int64_t ldc, cudaStream_t st) {
  if (M <= 0 || N <= 0) return;
  dim3 grid((N + ZBN - 1) / ZBN, (M + ZBM - 1) / ZBM);
  k_zgemm<<<grid, 256, 0, st>>>(M, N, K, A, lda, B, ldb, C, ldc);
}

// ====================================================== Jacobi eigensolver
// Hermitian matrices, n <= 32.  Parallel cyclic Jacobi with the round-robin ordering:
// n/2 disjoint rotations per step, n-1 steps per sweep (Golub & Van Loan sec. 8.5.4).
// Stands in for zheev('V','U') at wannier.f90:489 and :732.
//
// A block of T threads takes G matrices together.  A warp's FP64 instruction costs the
// same with 3 active lanes as with 32, and a step has n/2 rotations and n^2/2 element
// pairs: the lanes are therefore dealt out over the matrices that still have sweeps to
// do (n = 6, one matrix per warp: 3 and 18 of 32 lanes; half the FP64 instructions are
// then the rotations').  Every element's arithmetic, and the norms' order, are those of
// one matrix alone.  Matrices lie in shared memory with an odd leading dimension, which
// rows and columns alike read without bank conflicts.
//
// Mixed precision, because GB300's FP64 rate is a sixtieth of its FP32 rate:
//  1. FP32 sweeps bring the matrix to near-diagonal form (off-diagonal norm
//     ~1e-5 of the total) and accumulate their rotations in Q;
//  2. two Newton-Schulz steps X <- X (3I - X^H X) / 2 in FP64 make Q unitary to
//     FP64 rounding (from ~1e-6);
//  3. B = Q^H A Q in FP64 has A's eigenvalues to FP64 rounding;
//  4. FP64 sweeps on B, accumulating into V = Q, converge quadratically from
//     there: two or three sweeps instead of six or seven from A.
constexpr int EIG_MAXSWEEP = 40;
constexpr int EIG_MAXSWEEP32 = 12;

// round-robin pair `lane` (< m / 2) of step r, m players: (p, q) with p < q
__device__ __forceinline__ void rr_pair(int r, int m, int lane, int &p, int &q) {
  int a, b;
  if (lane == 0) {
    a = 0;
    b = (r % (m - 1)) + 1;
  } else {
    a = ((r + lane) % (m - 1)) + 1;
    b = ((r - lane + (m - 1)) % (m - 1)) + 1;
  }
  p = min(a, b);
  q = max(a, b);
}

// x / d for x d < 2^32, from inv_of(d)
__device__ __forceinline__ unsigned inv_of(int d) { return d == 1 ? 0u : 0xffffffffu / (unsigned)d + 1u; }
__device__ __forceinline__ int div_by(int x, unsigned inv) { return inv ? (int)__umulhi((unsigned)x, inv) : x; }

constexpr int EIG_G = 4;       // matrices per block at most

// What a block's sweeps share: which matrices are done, their last off-diagonal norms.
struct EigState {
  int done[EIG_G];
  double prev[EIG_G];
};

// The matrices of a block that still have sweeps to do, four bits each.
__device__ __forceinline__ int eig_active(const EigState &es, int G, unsigned &map) {
  int na = 0;
  map = 0;
  for (int g = 0; g < G; ++g)
    if (!es.done[g]) map |= (unsigned)g << (4 * na++);
  return na;
}

// Index helpers of a block's items: n, n / 2 pairs (n even; odd n has a dummy player).
struct EigDims {
  int n, m, half, ld, size;          // size: doubles2 of one matrix's storage
  unsigned inv_n, inv_half, inv_hn, inv_nn;
};

// A rotation's factors from a_pq = (ax, ay), rr = |a_pq| and d = a_qq - a_pp: the lane with
// `phase` returns e^{i phi} = (ax, ay) / rr, the other (c, t = tan), each with two of the
// four divisions.
__device__ __forceinline__ float2 rotation_f32(bool phase, float ax, float ay, float d, float rr) {
  const float u = (phase ? ax : d) / (phase ? rr : 2.f * rr);   // tau
  const bool big = fabsf(u) > 1e18f;
  const float num = phase ? ay : big ? 0.5f : u >= 0.f ? 1.f : -1.f;
  const float v = num / (phase ? rr : big ? u : fabsf(u) + sqrtf(1.f + u * u));
  return phase ? make_float2(u, v) : make_float2(rsqrtf(1.f + v * v), v);
}

// (tot, off) summed over the warp's lanes by a butterfly, the two in opposite halves.
template <typename F>
__device__ __forceinline__ void warp_sums(F &tot, F &off, int lane) {
  F v = lane < 16 ? tot : off;
  const F w = lane < 16 ? off : tot;
  v += __shfl_xor_sync(0xffffffffu, w, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  tot = __shfl_sync(0xffffffffu, v, 0);
  off = __shfl_sync(0xffffffffu, v, 16);
}

// FP32 sweeps on A (float2, column-major) accumulating into Q until the off-diagonal
// norm is 1e-10 of the total or stalls below 1e-6 of it; P4 / PI: the step's rotations
// (c, s, e^{i phi}) and pairs.  base: the block's first matrix, dim.size apart.
template <int T>
__device__ void jacobi_f32(const EigDims &e, double2 *base, EigState &es, int G, int tid) {
  const int n = e.n, ld = e.ld, nn = n * n, half = e.half, lane = tid & 31, warp = tid >> 5;
  auto fA = [&](int g) { return (float2 *)(base + (size_t)g * e.size + 2 * ld * n); };
  auto fQ = [&](int g) { return (float2 *)(base + (size_t)g * e.size + 2 * ld * n) + ld * n; };
  auto fP = [&](int g) { return (float4 *)(base + (size_t)g * e.size + 4 * ld * n); };
  auto fI = [&](int g) { return (int2 *)(base + (size_t)g * e.size + 4 * ld * n + 16); };
  unsigned map;
  int na = eig_active(es, G, map);
  for (int sweep = 0; sweep < EIG_MAXSWEEP32; ++sweep) {
    for (int a = warp; a < na; a += T / 32) {
      const int g = (map >> (4 * a)) & 15;
      const float2 *A = fA(g);
      float off = 0.f, tot = 0.f;
      for (int idx = lane; idx < nn; idx += 32) {
        const int j = div_by(idx, e.inv_n), i = idx - j * n;
        const float2 v = A[i + ld * j];
        const float a2 = v.x * v.x + v.y * v.y;
        tot += a2;
        if (i != j) off += a2;
      }
      warp_sums(tot, off, lane);
      // done at 1e-10 of the total, or once it stalls near FP32's floor; a
      // non-finite norm also stops it (Q is then not used)
      const float prev = (float)es.prev[g];
      __syncwarp();
      if (lane == 0) {
        es.done[g] = !(off > 1e-10f * tot) || (off <= 1e-6f * tot && off > 0.25f * prev);
        es.prev[g] = off;
      }
    }
    __syncthreads();
    na = eig_active(es, G, map);
    if (na == 0) return;
    const int cnt = na * half * n, cntv = (cnt + 31) & ~31;
    for (int r = 0; r < e.m - 1; ++r) {
      for (int idx = tid; idx < 2 * na * half; idx += T) {
        const int v = idx >> 1, a = div_by(v, e.inv_half), l = v - a * half, g = (map >> (4 * a)) & 15;
        const bool phase = idx & 1;
        const float2 *A = fA(g);
        int p, q;
        rr_pair(r, e.m, l, p, q);
        float2 out = make_float2(1.f, 0.f);
        if (q < n) {
          const float2 apq = A[p + ld * q];
          const float rr = hypotf(apq.x, apq.y);
          if (rr > 0.f) out = rotation_f32(phase, apq.x, apq.y, A[q + ld * q].x - A[p + ld * p].x, rr);
          if (rr > 0.f && !phase) out.y *= out.x;   // s = t c
        }
        ((float2 *)(fP(g) + l))[phase] = out;   // (c, s); e^{i phi}
        if (!phase) fI(g)[l] = make_int2(p, q < n ? q : -1);
      }
      __syncthreads();
      // columns: A <- A J;  J = [[c, s], [-s e^{-i phi}, c e^{-i phi}]]
      for (int idx = tid; idx < cnt; idx += T) {
        const int a = div_by(idx, e.inv_hn), w = idx - a * half * n, k = div_by(w, e.inv_n), i = w - k * n;
        const int g = (map >> (4 * a)) & 15;
        const int2 pq = fI(g)[k];
        if (pq.y < 0) continue;
        const float4 r4 = fP(g)[k];
        float2 *xp = fA(g) + i + ld * pq.x, *xq = fA(g) + i + ld * pq.y;
        const float2 aip = *xp, aiq = *xq;
        const float2 t = make_float2(r4.z * aiq.x + r4.w * aiq.y, r4.z * aiq.y - r4.w * aiq.x);
        *xp = make_float2(r4.x * aip.x - r4.y * t.x, r4.x * aip.y - r4.y * t.y);
        *xq = make_float2(r4.y * aip.x + r4.x * t.x, r4.y * aip.y + r4.x * t.y);
      }
      __syncthreads();
      // rows: A <- J^H A, its diagonal kept real; Q <- Q J, by other warps
      for (int idx = tid; idx < cntv + cnt; idx += T) {
        const bool row = idx < cntv;
        const int v = row ? idx : idx - cntv;
        if (v >= cnt) continue;
        const int a = div_by(v, e.inv_hn), w = v - a * half * n, k = div_by(w, e.inv_n), i = w - k * n;
        const int g = (map >> (4 * a)) & 15;
        const int2 pq = fI(g)[k];
        if (pq.y < 0) continue;
        const float4 r4 = fP(g)[k];
        if (row) {
          float2 *A = fA(g) + ld * i;
          const float2 apj = A[pq.x], aqj = A[pq.y];
          const float2 t = make_float2(r4.z * aqj.x - r4.w * aqj.y, r4.z * aqj.y + r4.w * aqj.x);
          const float2 np = make_float2(r4.x * apj.x - r4.y * t.x, r4.x * apj.y - r4.y * t.y);
          const float2 nq = make_float2(r4.y * apj.x + r4.x * t.x, r4.y * apj.y + r4.x * t.y);
          A[pq.x] = make_float2(np.x, i == pq.x ? 0.f : np.y);
          A[pq.y] = make_float2(nq.x, i == pq.y ? 0.f : nq.y);
        } else {
          float2 *xp = fQ(g) + i + ld * pq.x, *xq = fQ(g) + i + ld * pq.y;
          const float2 vip = *xp, viq = *xq;
          const float2 t = make_float2(r4.z * viq.x + r4.w * viq.y, r4.z * viq.y - r4.w * viq.x);
          *xp = make_float2(r4.x * vip.x - r4.y * t.x, r4.x * vip.y - r4.y * t.y);
          *xq = make_float2(r4.y * vip.x + r4.x * t.x, r4.y * vip.y + r4.x * t.y);
        }
      }
      __syncthreads();
    }
  }
}

// C = op(X) Y for the block's n x n complex FP64 matrices (X, Y, C: offsets in a matrix's
// storage), op(X) = X^H if XH.
template <int T, bool XH>
__device__ void group_matmul(const EigDims &e, double2 *base, int ng, int X, int Y, int C, int tid) {
  const int n = e.n, ld = e.ld;
  for (int idx = tid; idx < ng * n * n; idx += T) {
    const int g = div_by(idx, e.inv_nn), w = idx - g * n * n, jj = div_by(w, e.inv_n), i = w - jj * n;
    double2 *M = base + (size_t)g * e.size;
    const double2 *x = M + X + (XH ? ld * i : i), *y = M + Y + ld * jj;
    double2 acc = make_double2(0.0, 0.0);
    for (int k = 0; k < n; ++k) {
      if (XH) cfma_cj(acc, x[k], y[k]);
      else cfma(acc, x[ld * k], y[k]);
    }
    M[C + i + ld * jj] = acc;
  }
  __syncthreads();
}

// Bound by FP64 instructions: one holds an SM sub-partition for 64 cycles.  A rotation's two
// normalisations therefore run on two lanes, and V <- V J in other warps than A <- J^H A.
// Against one warp per matrix: 13,824 matrices of n = 8 and of n = 6 2.37 -> 1.44 ms, 2,197
// of n = 16 and of n = 12 2.64 -> 1.80, 1,728 of n = 6 154 -> 100 us, 200 of n = 8
// 115 -> 82 (175,000 cycles a matrix: a third in the FP32 sweeps, half in the FP64 ones).
template <int T>
__global__ void __launch_bounds__(T) k_heig(int batch, int n, int G, const double2 *__restrict__ A, int64_t stride,
                                            double *__restrict__ w, double2 *__restrict__ V, int *err) {
  extern __shared__ double2 sm[];
  __shared__ EigState es;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int mat0 = blockIdx.x * G, ng = min(G, batch - mat0), nn = n * n;
  EigDims e;
  e.n = n;
  e.m = n + (n & 1);         // even number of players (dummy = n)
  e.half = e.m / 2;
  e.ld = n | 1;
  e.size = 4 * e.ld * n + 3 * 16;
  e.inv_n = inv_of(n);
  e.inv_half = inv_of(e.half);
  e.inv_hn = inv_of(e.half * n);
  e.inv_nn = inv_of(nn);
  const int ld = e.ld, half = e.half;
  // a matrix's storage: A, V, two temporaries (the FP32 phase inside the first), per
  // pair (c, s), (ph.x, ph.y), (p, q)
  const int oV = ld * n, oT = 2 * ld * n, oT2 = 3 * ld * n, oP = 4 * ld * n;
  for (int idx = tid; idx < ng * nn; idx += T) {
    const int g = div_by(idx, e.inv_nn), v0 = idx - g * nn, j = div_by(v0, e.inv_n), i = v0 - j * n;
    const double2 *Am = A + (size_t)(mat0 + g) * stride;
    double2 v;
    if (i < j) {                       // averaged upper triangle (wannier.f90:481-486)
      double2 aij = Am[i + n * j], aji = Am[j + n * i];
      v = make_double2(0.5 * (aij.x + aji.x), 0.5 * (aij.y - aji.y));
    } else if (i > j) {
      double2 aij = Am[i + n * j], aji = Am[j + n * i];
      v = make_double2(0.5 * (aji.x + aij.x), -0.5 * (aji.y - aij.y));
    } else {
      v = make_double2(Am[i + n * i].x, 0.0);
    }
    double2 *M = sm + (size_t)g * e.size;
    M[i + ld * j] = v;
    float2 *fA = (float2 *)(M + oT), *fQ = fA + ld * n;
    fA[i + ld * j] = make_float2((float)v.x, (float)v.y);
    fQ[i + ld * j] = make_float2(i == j ? 1.f : 0.f, 0.f);
  }
  if (tid < EIG_G) {
    es.done[tid] = tid >= ng;
    es.prev[tid] = INFINITY;
  }
  __syncthreads();
  // 1. FP32 sweeps
  jacobi_f32<T>(e, sm, es, G, tid);
  for (int g = warp; g < ng; g += T / 32) {
    double2 *M = sm + (size_t)g * e.size;
    const float2 *fQ = (const float2 *)(M + oT) + ld * n;
    bool finite = true;
    for (int idx = lane; idx < nn; idx += 32) {
      const int j = div_by(idx, e.inv_n), o = idx - j * n + ld * j;
      const float2 q = fQ[o];
      finite = finite && isfinite(q.x) && isfinite(q.y);
      M[oV + o] = make_double2((double)q.x, (double)q.y);
    }
    if (!__all_sync(0xffffffffu, finite)) {   // FP32 overflowed: the FP64 sweeps start from A itself
      for (int idx = lane; idx < nn; idx += 32) {
        const int j = div_by(idx, e.inv_n), i = idx - j * n;
        M[oV + i + ld * j] = make_double2(i == j ? 1.0 : 0.0, 0.0);
      }
    }
  }
  __syncthreads();
  if (tid < EIG_G) {
    es.done[tid] = tid >= ng;
    es.prev[tid] = INFINITY;
  }
  // 2. Q unitary to FP64 rounding: X <- X (3I - X^H X) / 2, twice
  for (int it = 0; it < 2; ++it) {
    group_matmul<T, true>(e, sm, ng, oV, oV, oT, tid);
    for (int idx = tid; idx < ng * nn; idx += T) {
      const int g = div_by(idx, e.inv_nn), v0 = idx - g * nn, j = div_by(v0, e.inv_n), i = v0 - j * n;
      double2 &t = sm[(size_t)g * e.size + oT + i + ld * j];
      t = make_double2((i == j ? 3.0 : 0.0) - t.x, -t.y);
    }
    __syncthreads();
    group_matmul<T, false>(e, sm, ng, oV, oT, oT2, tid);
    for (int idx = tid; idx < ng * nn; idx += T) {
      const int g = div_by(idx, e.inv_nn), v0 = idx - g * nn, j = div_by(v0, e.inv_n), o = v0 - j * n + ld * j;
      double2 *M = sm + (size_t)g * e.size;
      M[oV + o] = cscale(M[oT2 + o], 0.5);
    }
    __syncthreads();
  }
  // 3. B = Q^H A Q, made exactly Hermitian (its rounding is below the FP64 sweeps' floor)
  group_matmul<T, false>(e, sm, ng, 0, oV, oT, tid);
  group_matmul<T, true>(e, sm, ng, oV, oT, 0, tid);
  for (int idx = tid; idx < ng * nn; idx += T) {
    const int g = div_by(idx, e.inv_nn), v0 = idx - g * nn, j = div_by(v0, e.inv_n), i = v0 - j * n;
    double2 *M = sm + (size_t)g * e.size;
    if (i < j) {
      const double2 bij = M[i + ld * j], bji = M[j + ld * i];
      const double2 v = make_double2(0.5 * (bij.x + bji.x), 0.5 * (bij.y - bji.y));
      M[i + ld * j] = v;
      M[j + ld * i] = cconj(v);
    } else if (i == j) {
      M[i + ld * j].y = 0.0;
    }
  }
  __syncthreads();
  // 4. FP64 sweeps on B, accumulating into V = Q
  unsigned map;
  int na = eig_active(es, G, map);
  for (int sweep = 0; sweep < EIG_MAXSWEEP && na > 0; ++sweep) {
    for (int a = warp; a < na; a += T / 32) {
      const int g = (map >> (4 * a)) & 15;
      const double2 *M = sm + (size_t)g * e.size;
      double off = 0.0, tot = 0.0;
      for (int idx = lane; idx < nn; idx += 32) {
        const int j = div_by(idx, e.inv_n), i = idx - j * n;
        double2 v = M[i + ld * j];
        double a2 = v.x * v.x + v.y * v.y;
        tot += a2;
        if (i != j) off += a2;
      }
      warp_sums(tot, off, lane);
      // Converged: the off-diagonal norm is ~7 eps of the matrix norm, or it has
      // reached the FP64 rounding floor (the rotations leave a_pq at rounding
      // level rather than zero, so the floor sits near 1e-31..1e-30 of the total
      // and may not pass the first test): below 1e-26 of the total and no longer
      // falling by 4x per sweep.
      const double prev_off = es.prev[g];
      __syncwarp();
      if (lane == 0) {
        es.done[g] = off <= 1e-30 * tot || off == 0.0 || (off <= 1e-26 * tot && off > 0.25 * prev_off);
        es.prev[g] = off;
      }
    }
    __syncthreads();
    na = eig_active(es, G, map);
    if (na == 0) break;
    const int cnt = na * half * n, cntv = (cnt + 31) & ~31;
    for (int r = 0; r < e.m - 1; ++r) {
      // Rotations, two lanes each: both find the angle, the even one makes (c, s) unitary to
      // FP64 rounding, the odd one e^{i phi}; comparisons are on the integer images.
      for (int idx = tid; idx < 2 * na * half; idx += T) {
        const int v0 = idx >> 1, a = div_by(v0, e.inv_half), l = v0 - a * half;
        const bool phase = idx & 1;
        double2 *M = sm + (size_t)((map >> (4 * a)) & 15) * e.size, *sP = M + oP;
        int p, q;
        rr_pair(r, e.m, l, p, q);
        double2 out = make_double2(1.0, 0.0);
        if (q < n) {
          // The rotation angle is computed in FP32 on operands scaled by the
          // power of two of a_pq (GB300's FP64 divide / sqrt are slow); the
          // rotation is then made unitary to FP64 rounding, so it is an exact
          // similarity transform that leaves a_pq ~ 1e-7 of its value.  Later
          // rotations remove that residual; a_pq is not forced to zero.  With
          // |a_qq - a_pp| > 1e30 |a_pq| the rotation is negligible and skipped.
          const double2 apq = M[p + ld * q];
          const double d = M[q + ld * q].x - M[p + ld * p].x;
          const int ex = (max(__double2hiint(apq.x) & 0x7fffffff, __double2hiint(apq.y) & 0x7fffffff) >> 20) - 1023;
          if (ex > -1000 && ex < 1000) {
            const double sc = __hiloint2double((1023 - ex) << 20, 0);   // 2^-ex: max |a_pq| -> [1, 2)
            const float ax = (float)(apq.x * sc), ay = (float)(apq.y * sc);
            const double dsc = d * sc;
            const float rr = sqrtf(ax * ax + ay * ay);
            if ((__double_as_longlong(dsc) & 0x7fffffffffffffffll) <= __double_as_longlong(1e30)) {
              const float2 ct = rotation_f32(phase, ax, ay, (float)dsc, rr);
              const double x = (double)ct.x, y = (double)ct.y * (phase ? 1.0 : x);   // s = t c
              // two Newton steps of 1/sqrt(r2) from 1: x^2 + y^2 = 1 in FP64
              const double r2 = x * x + y * y;
              double f = 1.5 - 0.5 * r2;
              f = f * (1.5 - 0.5 * r2 * f * f);
              out = make_double2(x * f, y * f);
            }
          }
        }
        sP[3 * l + phase] = out;   // (c, s); e^{i phi}
        if (!phase) *(int2 *)(sP + 3 * l + 2) = make_int2(p, q < n ? q : -1);
      }
      __syncthreads();
      // columns: A <- A J;  J = [[c, s], [-s e^{-i phi}, c e^{-i phi}]]
      for (int idx = tid; idx < cnt; idx += T) {
        const int a = div_by(idx, e.inv_hn), v0 = idx - a * half * n, k = div_by(v0, e.inv_n), i = v0 - k * n;
        double2 *M = sm + (size_t)((map >> (4 * a)) & 15) * e.size;
        const double2 *sP = M + oP + 3 * k;
        const int2 pq = *(const int2 *)(sP + 2);
        if (pq.y < 0) continue;
        double2 *xp = M + ld * pq.x + i, *xq = M + ld * pq.y + i;
        const double c = sP[0].x, s = sP[0].y;
        const double2 phc = make_double2(sP[1].x, -sP[1].y);
        const double2 aip = *xp, aiq = *xq;
        const double2 t = cmul(phc, aiq);
        *xp = make_double2(c * aip.x - s * t.x, c * aip.y - s * t.y);
        *xq = make_double2(s * aip.x + c * t.x, s * aip.y + c * t.y);
      }
      __syncthreads();
      // rows: A <- J^H A, its diagonal kept real; V <- V J, by other warps
      for (int idx = tid; idx < cntv + cnt; idx += T) {
        const bool row = idx < cntv;
        const int v = row ? idx : idx - cntv;
        if (v >= cnt) continue;
        const int a = div_by(v, e.inv_hn), v0 = v - a * half * n, k = div_by(v0, e.inv_n), i = v0 - k * n;
        double2 *M = sm + (size_t)((map >> (4 * a)) & 15) * e.size;
        const double2 *sP = M + oP + 3 * k;
        const int2 pq = *(const int2 *)(sP + 2);
        if (pq.y < 0) continue;
        const double c = sP[0].x, s = sP[0].y;
        if (row) {
          const double2 ph = sP[1];
          M += ld * i;
          const double2 apj = M[pq.x], aqj = M[pq.y];
          const double2 t = cmul(ph, aqj);
          const double2 np = make_double2(c * apj.x - s * t.x, c * apj.y - s * t.y);
          const double2 nq = make_double2(s * apj.x + c * t.x, s * apj.y + c * t.y);
          M[pq.x] = make_double2(np.x, i == pq.x ? 0.0 : np.y);
          M[pq.y] = make_double2(nq.x, i == pq.y ? 0.0 : nq.y);
        } else {
          const double2 phc = make_double2(sP[1].x, -sP[1].y);
          double2 *xp = M + oV + ld * pq.x + i, *xq = M + oV + ld * pq.y + i;
          const double2 vip = *xp, viq = *xq;
          const double2 t = cmul(phc, viq);
          *xp = make_double2(c * vip.x - s * t.x, c * vip.y - s * t.y);
          *xq = make_double2(s * vip.x + c * t.x, s * vip.y + c * t.y);
        }
      }
      __syncthreads();
    }
  }
  if (na > 0 && tid == 0) atomicOr(err, DERR_EIG);   // not converged
  // sort ascending by rank (ties by index), write eigenvalues and columns
  for (int idx = tid; idx < ng * n; idx += T) {
    const int g = div_by(idx, e.inv_n), i = idx - g * n;
    const double2 *M = sm + (size_t)g * e.size;
    double di = M[i + ld * i].x;
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      double dj = M[j + ld * j].x;
      rank += (dj < di) || (dj == di && j < i);
    }
    w[(size_t)(mat0 + g) * n + rank] = di;
    for (int c = 0; c < n; ++c) V[(size_t)(mat0 + g) * nn + c + n * rank] = M[oV + c + ld * i];
  }
}

template <int T>
static void heig_run(int batch, int n, int G, const double2 *A, int64_t stride, double *w, double2 *V, int *err,
                     cudaStream_t st) {
  static OncePerDevice attr;
  attr([] { cudaFuncSetAttribute(k_heig<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024); });
  const size_t smem = (size_t)G * (4 * (n | 1) * n + 3 * 16) * sizeof(double2);   // 67 KB at most (n = 32)
  k_heig<T><<<(batch + G - 1) / G, T, smem, st>>>(batch, n, G, A, stride, w, V, err);
}

void launch_heig(int batch, int n, const double2 *A, int64_t stride, double *w, double2 *V,
                 int *err, cudaStream_t st) {
  if (batch <= 0) return;
  // Small batches are bound by the latency of one matrix, whose phases more warps shorten;
  // from a few matrices per SM sub-partition on by FP64 instructions, which taking matrices
  // together saves where one leaves lanes idle.  Microseconds at G = 1 / together:
  //   512 of n = 8:    90 / 103 (G = 4)      1,728 of n = 6:  133 / 100 (G = 4)
  //   2,197 of n = 12: 659 / 613 (G = 2)     2,197 of n = 16: 1,190 / 1,242 (G = 2)
  const bool many = batch >= 8 * num_sms();
  if (n <= 8) {
    if (many) heig_run<128>(batch, n, 4, A, stride, w, V, err, st);
    else heig_run<64>(batch, n, 1, A, stride, w, V, err, st);
  } else {
    heig_run<128>(batch, n, n <= 12 && many ? 2 : 1, A, stride, w, V, err, st);
  }
}

// ============================================================ electrons
// el_wann post-processing (wannier.f90:499-520): energies (eV, + scissor),
// evecs(k,b,:) = eigenvector b, velocities by Feynman-Hellmann.  A thread per band
// and direction (y = 0 also writes the band's energy and vector) in blocks of one
// warp: a few hundred k-points then reach most SMs, where one thread per band in
// blocks of 128 left 200 k-points on 13 of them (45 us; now 17).
__global__ void __launch_bounds__(32) k_el_post(int nk, int nw, const double *w, const double2 *V, const double2 *C,
                                                int64_t ldc, const double *scissor, double *energies_f, double *vel_f,
                                                double2 *evecs_f, double *ens_i) {
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= nk * nw) return;
  int k = idx / nw, b = idx % nw;
  const size_t nn = (size_t)nw * nw;
  const double2 *Vk = V + (size_t)k * nn;
  const int p = blockIdx.y;
  if (p == 0) {
    double e = w[(size_t)k * nw + b] * Ryd2eV;
    if (scissor) e += scissor[b];
    if (energies_f) energies_f[k + (int64_t)nk * b] = e;
    if (ens_i) ens_i[(size_t)k * nw + b] = e;
    if (evecs_f)
      for (int c = 0; c < nw; ++c) evecs_f[k + (int64_t)nk * (b + (int64_t)nw * c)] = Vk[c + nw * b];
  }
  if (vel_f) {
    const double2 *dH = C + (int64_t)k * ldc + (size_t)(1 + p) * nn;
    double2 acc = make_double2(0.0, 0.0);
    for (int r = 0; r < nw; ++r) {
      double2 mv = make_double2(0.0, 0.0);
      for (int c = 0; c < nw; ++c) cfma(mv, dH[r + nw * c], Vk[c + nw * b]);
      cfma_cj(acc, Vk[r + nw * b], mv);
    }
    vel_f[k + (int64_t)nk * (b + (int64_t)nw * p)] = acc.x * Ryd2radTHz;
  }
}

void launch_el_post(int nk, int nw, const double *w, const double2 *V, const double2 *C,
                    int64_t ldc, int with_vel, const double *scissor, double *energies_f,
                    double *vel_f, double2 *evecs_f, double *ens_i, cudaStream_t st) {
  int n = nk * nw;
  if (n == 0) return;
  k_el_post<<<dim3((n + 31) / 32, with_vel && vel_f ? 3 : 1), 32, 0, st>>>(nk, nw, w, V, C, ldc, scissor, energies_f,
                                                                        with_vel ? vel_f : nullptr, evecs_f, ens_i);
}

// ============================================================= phonons
// ph_wann post-processing (wannier.f90:740-780); a thread per mode and direction, as k_el_post
__global__ void __launch_bounds__(32) k_ph_post(int nq, int nb, const int *qp, const double *qv, const double *w,
                          const double2 *V, const double2 *dDq, int64_t ldd, int with_vel,
                          const double *masses, double *energies_f, double2 *evecs_f,
                          double *vel_f, double *om_i, double2 *u_i, float2 *u_f, int *err) {
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= nq * nb) return;
  int q = idx / nb, s = idx % nb;
  const size_t nn = (size_t)nb * nb;
  double o2 = w[(size_t)q * nb + s];
  double e = sqrt(fabs(o2));
  if (o2 < 0.0 || signbit(o2)) e = -e;          // sign(sqrt(abs(w)), w)
  const double2 *Vq = V + (size_t)q * nn;
  const int p = blockIdx.y;
  const bool gamma = qp ? (qp[q] == 0) : (qv[q] == 0.0 && qv[q + nq] == 0.0 && qv[q + 2 * nq] == 0.0);
  if (with_vel && vel_f) {
    const double2 *dD = dDq + (size_t)q * ldd + p * nn;
    double2 acc = make_double2(0.0, 0.0);
    for (int r = 0; r < nb; ++r) {
      double2 mv = make_double2(0.0, 0.0);
      for (int c = 0; c < nb; ++c) cfma(mv, dD[r + nb * c], Vq[c + nb * s]);
      cfma_cj(acc, Vq[r + nb * s], mv);
    }
    vel_f[q + (int64_t)nq * (s + (int64_t)nb * p)] = gamma ? 0.0 : acc.x / (2.0 * e) * Ryd2radTHz;
  }
  if (p) return;
  e *= Ryd2eV;
  if (gamma && s < 3) e = 0.0;
  if (e < -0.005) atomicOr(err, DERR_NEG_PHONON);
  else if (e < 0.0 && e > -0.005) e = 0.0;
  if (energies_f) energies_f[q + (int64_t)nq * s] = e;
  if (om_i) om_i[(size_t)q * nb + s] = e;
  if (evecs_f)
    for (int c = 0; c < nb; ++c) evecs_f[q + (int64_t)nq * (s + (int64_t)nb * c)] = Vq[c + nb * s];
  if (u_i || u_f)
    for (int c = 0; c < nb; ++c) {
      // u(ip) = ph_evec(ip)/sqrt(mass) (wannier.f90:937-942)
      double2 u = make_double2(Vq[c + nb * s].x / sqrt(masses[c / 3]), Vq[c + nb * s].y / sqrt(masses[c / 3]));
      if (u_i) u_i[((size_t)q * nb + s) * nb + c] = u;
      if (u_f) u_f[((size_t)q * nb + s) * nb + c] = make_float2((float)u.x, (float)u.y);
    }
}

void launch_ph_post(int nq, int nb, const int *qp, const double *qv, const double *w,
                    const double2 *V, const double2 *dDq, int64_t ldd, int with_vel, const double *masses,
                    double *energies_f, double2 *evecs_f, double *vel_f, double *om_i,
                    double2 *u_i, float2 *u_f, int *err, cudaStream_t st) {
  int n = nq * nb;
  if (n == 0) return;
  k_ph_post<<<dim3((n + 31) / 32, with_vel && vel_f ? 3 : 1), 32, 0, st>>>(nq, nb, qp, qv, w, V, dDq, ldd, with_vel, masses,
                                             energies_f, evecs_f, vel_f, om_i, u_i, u_f, err);
}

// ======================================================= g(Re,Rp) layouts
// epmatwp order (i, j, Re, s, Rp) -> stage-A matrix G[Re][n], n = i + nw*(j + nw*(s + nb*Rp)),
// so that one row of the GEMM output is gmixed(nw,nw,nb,nwsq) of gkRp (wannier.f90:1085).
__global__ void k_permute_gwann(int nw, int nb, int nwsk, int nwsg, const double2 *raw,
                                double2 *G) {
  const int64_t Nn = (int64_t)nw * nw * nb * nwsg;
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= Nn * nwsk) return;
  int64_t re = idx / Nn, n = idx % Nn;
  int64_t nn = (int64_t)nw * nw;
  int64_t ij = n % nn, s = (n / nn) % nb, rp = n / (nn * nb);
  G[idx] = raw[ij + nn * (re + (int64_t)nwsk * (s + (int64_t)nb * rp))];
}

void launch_permute_gwann(int nw, int nb, int nwsk, int nwsg, const double2 *raw, double2 *G,
                          cudaStream_t st) {
  int64_t n = (int64_t)nw * nw * nb * nwsg * nwsk;
  k_permute_gwann<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(nw, nb, nwsk, nwsg, raw, G);
}

// ================================================================ gReq
__global__ void k_permute_greq(int nq, int nw, int nb, int nwsk, const double2 *in,
                               double2 *out) {
  int64_t per = (int64_t)nw * nw * nb * nwsk;
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= per * nq) return;
  int64_t q = idx / per, r = idx % per;
  // out (i, j, s, Re) <- in (i, j, Re, s)
  int64_t ij = r % ((int64_t)nw * nw);
  int64_t rest = r / ((int64_t)nw * nw);
  int64_t s = rest % nb, re = rest / nb;
  out[q * per + r] = in[q * per + ij + (int64_t)nw * nw * (re + (int64_t)nwsk * s)];
}

void launch_permute_greq(int nq, int nw, int nb, int nwsk, const double2 *in, double2 *out,
                         cudaStream_t st) {
  int64_t n = (int64_t)nq * nw * nw * nb * nwsk;
  if (n == 0) return;
  k_permute_greq<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(nq, nw, nb, nwsk, in, out);
}

// ============================================================= g2 batch
// |g|^2 of the vertices of a list (wannier.f90:903-1011) from their cell sums
// G(n', m', s') = sum_R e^{2 pi i q.R} / deg gmixed(n', m', s', R), which come from one product
// per right-hand side (launch_xgemm_chunks): one warp per vertex rotates them by the
// electrons and the mode, lanes along (n', s').  row v of G is vertex perm[v].
// The sum over cells comes first because it is linear in the given blocks: the
// rotation then runs once per vertex instead of once per vertex and cell.
__global__ void __launch_bounds__(128) k_g2_vertices(int nv, const int *perm, int64_t ld, int nw, int nb,
                                                     const double2 *G, const double2 *ek, const double2 *ekp,
                                                     const double2 *eq, const double *ph_en, const double *masses,
                                                     const double2 *Lv, double *g2) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= nv) return;
  const int64_t v = perm[row];
  const double en = ph_en[v];
  if (en == 0.0) {
    if (lane == 0) g2[v] = 0.0;
    return;
  }
  const double2 *g = G + (int64_t)row * nw * nw * nb;
  double2 gb = make_double2(0.0, 0.0);
  for (int o = lane; o < nw * nb; o += 32) {
    const int np = o % nw, sp = o / nw;
    double2 h = make_double2(0.0, 0.0);
    for (int mp = 0; mp < nw; ++mp) cfma(h, ek[v + ld * mp], g[np + nw * (mp + (int64_t)nw * sp)]);
    // conj(U_k'(n')) u(s') / sqrt(M)
    const double rm = 1.0 / sqrt(masses[sp / 3]);
    cfma(gb, cmul(cconj(ekp[v + ld * np]), cscale(eq[v + ld * sp], rm)), h);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gb.x += __shfl_xor_sync(0xffffffffu, gb.x, o);
    gb.y += __shfl_xor_sync(0xffffffffu, gb.y, o);
  }
  if (lane == 0) {
    if (Lv) {   // polar: + long_range_prefac(q, u) * dot_product(el_evec_kp, el_evec_k) (wannier.f90:998-1006)
      double2 gl = make_double2(0.0, 0.0), unm = make_double2(0.0, 0.0);
      for (int sp = 0; sp < nb; ++sp) {
        double2 u = eq[v + ld * sp];
        u = make_double2(u.x / sqrt(masses[sp / 3]), u.y / sqrt(masses[sp / 3]));
        cfma(gl, Lv[(size_t)v * nb + sp], u);
      }
      for (int c = 0; c < nw; ++c) cfma_cj(unm, ekp[v + ld * c], ek[v + ld * c]);
      cfma(gb, gl, unm);
    }
    g2[v] = 0.5 * (gb.x * gb.x + gb.y * gb.y) / en * g2unitfactor;
  }
}

void launch_g2_vertices(int nv, const int *perm, int64_t ld, int nw, int nb, const double2 *G, const double2 *ek,
                        const double2 *ekp, const double2 *eq, const double *ph_en, const double *masses,
                        const double2 *Lv, double *g2, cudaStream_t st) {
  if (nv > 0) k_g2_vertices<<<(nv + 3) / 4, 128, 0, st>>>(nv, perm, ld, nw, nb, G, ek, ekp, eq, ph_en, masses, Lv, g2);
}

// ============================================================ q indices
// q = k' - k folded onto the mesh, on integers (vector.f90:86-102 computes the
// same through fractional coordinates and nint).
__global__ void k_kq_index(int m1, int m2, int m3, int nk, const int64_t *k_idx, int nkp,
                           const int64_t *kp_idx, int64_t *q_idx, int *err) {
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)nk * nkp) return;
  int i = (int)(idx % nk), j = (int)(idx / nk);
  int64_t N = (int64_t)m1 * m2 * m3;
  int64_t a = k_idx[i] - 1, b = kp_idx[j] - 1;
  if (a < 0 || a >= N || b < 0 || b >= N) { atomicOr(err, DERR_INDEX); q_idx[idx] = -1; return; }
  int64_t a1 = a % m1, a2 = (a / m1) % m2, a3 = a / ((int64_t)m1 * m2);
  int64_t b1 = b % m1, b2 = (b / m1) % m2, b3 = b / ((int64_t)m1 * m2);
  int64_t q1 = floormod(b1 - a1, m1), q2 = floormod(b2 - a2, m2), q3 = floormod(b3 - a3, m3);
  q_idx[idx] = (q3 * m2 + q2) * m1 + q1 + 1;   // mux_vector base 0 (misc.f90:906)
}

void launch_kq_index(const int mesh[3], int nk, const int64_t *k_idx, int nkp,
                     const int64_t *kp_idx, int64_t *q_idx, int *err, cudaStream_t st) {
  int64_t n = (int64_t)nk * nkp;
  if (n == 0) return;
  k_kq_index<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(mesh[0], mesh[1], mesh[2], nk, k_idx,
                                                          nkp, kp_idx, q_idx, err);
}

// ======================================================= rate pipeline
__global__ void k_window_flags(int N, int nw, const double *ens, double enref, double fsthick,
                               int *flag) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= N) return;
  int in = 0;
  for (int b = 0; b < nw; ++b) in |= fabs(ens[(size_t)p * nw + b] - enref) <= fsthick;
  flag[p] = in;     // apply_energy_window, electron.f90:613-621
}

void launch_window_flags(int N, int nw, const double *ens, double enref, double fsthick,
                         int *flag, cudaStream_t st) {
  k_window_flags<<<(N + 255) / 256, 256, 0, st>>>(N, nw, ens, enref, fsthick, flag);
}

__global__ void k_state_flags(int nwv, int nw, const int *widx, const double *ens, double enref,
                              double fsthick, int *flag, int *nin_k) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nwv) return;
  int p = widx[i], c = 0;
  for (int m = 0; m < nw; ++m) {
    int f = fabs(ens[(size_t)p * nw + m] - enref) <= fsthick;
    flag[(size_t)i * nw + m] = f;
    c += f;
  }
  nin_k[i] = c;
}

void launch_state_flags(int nwv, int nw, const int *widx, const double *ens, double enref,
                        double fsthick, int *flag, int *nin_k, cudaStream_t st) {
  k_state_flags<<<(nwv + 255) / 256, 256, 0, st>>>(nwv, nw, widx, ens, enref, fsthick, flag,
                                                    nin_k);
}

__global__ void k_iota(int n, int *out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = i;
}
void launch_iota(int n, int *out, cudaStream_t st) {
  if (n > 0) k_iota<<<(n + 255) / 256, 256, 0, st>>>(n, out);
}

// Stage A rotation over the initial band (the U_k half of wannier.f90:960-978),
// with the k-half of the Rp phase, conj(e^{2 pi i k.Rp})/phwsdeg(Rp), folded in
// so that the Rp Fourier of all states is one sum against e^{2 pi i k'.Rp}.
// FP64-pipe bound: nw complex multiply-adds and one multiply per output, the
// phases from a table.  Lanes are states, so that the stores run along the states
// (the epilogue's lanes); each warp stages its states' nw x nw blocks through
// shared memory in whole rows, ROT64_V values of each state at a time.
// 12^3, nw 8, nb 6, 279 cells, 1,679 states: 1.74 ms (1.1 at the FP64 rate; 2.63 with each
// lane reading its own block).  With the phases tabulated but one state's columns after the
// other's it took 1.34; the epilogue, whose lanes are states, gained more from this order.
constexpr int ROT64_THREADS = 64, ROT64_V = 32;

// A thread's sums over the initial band, one per final one, stay in registers: CAP of them, the next
// multiple of 4 from nw on, or nw = CAP known to the compiler (EXACT).  With 32 for every nw
// the registers and the unrolled tail are paid by all: 9^3, nb 6, 1,200 states, with 32 / with CAP:
// nw 3 0.33 / 0.11 ms, nw 5 0.49 / 0.18, nw 10 1.07 / 0.50, nw 12 1.34 / 0.55, nw 20 3.11 / 1.35,
// nw 24 3.89 / 1.83; nw 32 5.57, with nw known 3.56.
template <int CAP, bool EXACT>
__global__ void __launch_bounds__(ROT64_THREADS) k_rotate_states_fp64(int j0, int j1, int i0, const int *st_code,
                                                                      int nw_, int nb, int nws, int64_t blk0,
                                                                      const int *widx,
                                                                      const double2 *U, const double2 *gk,
                                                                      int64_t ldgk, const double2 *phk, double2 *B,
                                                                      int64_t ldb, int sc, int nst) {
  __shared__ double2 sg[ROT64_THREADS * (ROT64_V + 1)];
  const int nw = EXACT ? CAP : nw_;
  const int lane = threadIdx.x & 31, wj = j0 + blockIdx.x * ROT64_THREADS + (threadIdx.x & ~31);
  const int j = wj + lane;
  const bool live = j < j1;
  const int code = live ? st_code[j] : 0;
  const int i = live ? code / nw : i0, m = code % nw;
  const int64_t u = blockIdx.y;
  const int rp = (int)((blk0 + u) / nb), s = (int)((blk0 + u) % nb);
  const double2 *Uk = U + ((size_t)widx[i] * nw + m) * nw;
  const double2 *g = gk + (int64_t)nw * nw * u;
  double2 *tile = sg + (threadIdx.x & ~31) * (ROT64_V + 1);
  const int mpc = ROT64_V / nw, nv = min(32, j1 - wj);   // initial bands per pass; the warp's states
  double2 acc[CAP];
#pragma unroll
  for (int np = 0; np < CAP; ++np) acc[np] = make_double2(0.0, 0.0);
  for (int mp0 = 0; mp0 < nw; mp0 += mpc) {
    const int nm = min(mpc, nw - mp0), n = nw * nm;
    __syncwarp();
    for (int t = 0; t < nv; ++t) {   // state t's values, contiguous in gk
      const double2 *src = g + (int64_t)(__shfl_sync(0xffffffffu, i, t) - i0) * ldgk + nw * mp0;
      for (int v = lane; v < n; v += 32) tile[t * (ROT64_V + 1) + v] = src[v];
    }
    __syncwarp();
    if (live)
      for (int mp = 0; mp < nm; ++mp) {
        const double2 um = Uk[mp0 + mp], *row = tile + lane * (ROT64_V + 1) + nw * mp;
#pragma unroll
        for (int np = 0; np < CAP; ++np)
          if (np < nw) cfma(acc[np], um, row[np]);
      }
  }
  if (!live) return;
  const double2 ph = phk[(int64_t)i * nws + rp];
  // columns of a chunk of sc states: [n' + nw s'][state]
  const int jc = j / sc * sc, ns = min(sc, nst - jc);
  double2 *out = B + (int64_t)rp * ldb + (int64_t)jc * nw * nb + (int64_t)nw * s * ns + (j - jc);
#pragma unroll
  for (int np = 0; np < CAP; ++np)
    if (np < nw) out[(int64_t)np * ns] = cmul(ph, acc[np]);
}

void launch_rotate_states_fp64(int j0, int j1, int i0, const int *st_code, int nw, int nb, int nws, int64_t blk0,
                               int64_t nblk, const int *widx, const double2 *U, const double2 *gk, int64_t ldgk,
                               const double2 *phk, double2 *B, int64_t ldb, int sc, int nst, cudaStream_t st) {
  if (j1 <= j0) return;
  for (int64_t b = 0; b < nblk; b += 32768) {   // grid.y
    dim3 grid((j1 - j0 + ROT64_THREADS - 1) / ROT64_THREADS, (unsigned)std::min<int64_t>(nblk - b, 32768));
    auto go = [&](auto k) {
      k<<<grid, ROT64_THREADS, 0, st>>>(j0, j1, i0, st_code, nw, nb, nws, blk0 + b, widx, U, gk + b * nw * nw, ldgk, phk,
                                        B, ldb, sc, nst);
    };
    auto upto = [&](auto cap) {
      constexpr int C = decltype(cap)::value;
      nw == C ? go(k_rotate_states_fp64<C, true>) : go(k_rotate_states_fp64<C, false>);
    };
    switch ((nw + 3) / 4) {
      case 1: upto(std::integral_constant<int, 4>()); break;
      case 2: upto(std::integral_constant<int, 8>()); break;
      case 3: upto(std::integral_constant<int, 12>()); break;
      case 4: upto(std::integral_constant<int, 16>()); break;
      case 5: upto(std::integral_constant<int, 20>()); break;
      case 6: upto(std::integral_constant<int, 24>()); break;
      case 7: upto(std::integral_constant<int, 28>()); break;
      default: upto(std::integral_constant<int, 32>()); break;
    }
  }
}

__global__ void k_bose(int n, const double *om, double T, double *bose) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double e = om[i];
  // Bose = 1/expm1(e/kB/T) (misc.f90:992-999), zero for zero-energy phonons (interactions.f90:2287)
  bose[i] = (e != 0.0) ? 1.0 / expm1(e / kB / T) : 0.0;
}

void launch_bose(int N, int nb, const double *om, double T, double *bose, cudaStream_t st) {
  int n = N * nb;
  k_bose<<<(n + 255) / 256, 256, 0, st>>>(n, om, T, bose);
}

// ------------------------------------------------- simplex deltas as tables
// The triangle and tetrahedron deltas (delta.f90:790-881, 61-225) of one final
// state (k', n) are functions of the energy alone: over the up to 24 tetrahedra
// (6 triangles) that share the corner k', each contributes a product of linear
// factors between its sorted vertex energies.  Between consecutive vertex
// energies of all of them the sum is one cubic, so a table of (breakpoint,
// cubic) replaces 24 range tests and formulas with five to seven FP64 divisions
// each: an evaluation is a binary search and ten FP64 operations.
//
// The cubic of (b_i-1, b_i] is kept in Bernstein form, coefficients over
// (e - b_i-1) and (b_i - e): they are the formulas' blossoms, sums of products
// of factors of one sign, so the tails keep their relative accuracy, as in the
// formulas themselves.  Vertex energies of corners outside the window are zero,
// as the reference leaves them (delta.f90:494-646); equal energies give
// intervals of no width, which are never looked up, so the formulas' special
// cases for them need no counterpart.
struct SimplexEntry {
  double e[4];      // sorted vertex energies
  double c1[4];     // first range: x_1 x_1 (or x_1) times sum_i c1_i x_i, x_i = e_i - e
  double c3[4];     // last range: the same with the last vertex
  double m[5];      // middle range of a tetrahedron: S^2 (m0 a + m1 b) + Q^2 (m2 b + m3 a) + m4 x_label S Q
  int label;        // 0-based vertex label; -1: no simplex (its cell is outside the window)
};

// corners of a mesh cell used by the simplices, and the simplices as corner lists (delta.f90)
__constant__ int kTri[2][3] = {{1, 2, 3}, {1, 3, 4}};
__constant__ int kTet[6][4] = {{1, 2, 3, 6}, {1, 3, 5, 6}, {3, 5, 6, 7}, {3, 6, 7, 8}, {3, 4, 6, 8}, {2, 3, 4, 6}};

__device__ void simplex_coefs(int kind, SimplexEntry &t) {
  const double *e = t.e;
  const int v = t.label;
  for (int i = 0; i < 4; ++i) t.c1[i] = t.c3[i] = 0.0;
  for (int i = 0; i < 5; ++i) t.m[i] = 0.0;
  const double r21 = 1.0 / (e[1] - e[0]), r31 = 1.0 / (e[2] - e[0]), r32 = 1.0 / (e[2] - e[1]);
  if (kind == 1) {
    if (v == 0) {
      t.c1[1] = -r21 * r21 * r31;
      t.c1[2] = -r31 * r21 * r31;
      t.c3[2] = r32 * r31 * r31;
    } else if (v == 1) {
      t.c1[0] = r21 * r21 * r31;
      t.c3[2] = r32 * r32 * r31;
    } else {
      t.c1[0] = r21 * r31 * r31;
      t.c3[0] = -r31 * r32 * r31;
      t.c3[1] = -r32 * r32 * r31;
    }
    return;
  }
  const double r41 = 1.0 / (e[3] - e[0]), r42 = 1.0 / (e[3] - e[1]), r43 = 1.0 / (e[3] - e[2]);
  const double k1 = r21 * r31 * r41, k3 = r41 * r42 * r43;
  if (v == 0) {
    t.c1[1] = r21 * k1;
    t.c1[2] = r31 * k1;
    t.c1[3] = r41 * k1;
    t.c3[3] = k3 * r41;
    t.m[0] = -0.5 * r31 * r31 * r42 * r32;
    t.m[1] = -0.5 * r31 * r31 * r32 * r41;
    t.m[2] = -0.5 * r41 * r41 * r42 * r31;
    t.m[3] = -0.5 * r41 * r41 * r42 * r32;
    t.m[4] = -0.5 * (r31 * r31 * r41 * r42 + r41 * r41 * r31 * r32);
  } else if (v == 1) {
    t.c1[0] = -k1 * r21;
    t.c3[3] = k3 * r42;
    t.m[0] = -0.5 * r32 * r32 * r42 * r31;
    t.m[1] = -0.5 * r32 * r32 * r31 * r41;
    t.m[2] = -0.5 * r42 * r42 * r41 * r31;
    t.m[3] = -0.5 * r42 * r42 * r32 * r41;
    t.m[4] = -0.5 * (r32 * r32 * r42 * r41 + r42 * r42 * r32 * r31);
  } else if (v == 2) {
    t.c1[0] = -k1 * r31;
    t.c3[3] = k3 * r43;
    t.m[0] = 0.5 * r32 * r32 * r42 * r31;
    t.m[1] = 0.5 * r32 * r32 * r42 * r41;
    t.m[2] = 0.5 * r31 * r31 * r41 * r42;
    t.m[3] = 0.5 * r31 * r31 * r32 * r41;
    t.m[4] = 0.5 * (r32 * r32 * r31 * r41 + r31 * r31 * r42 * r32);
  } else {
    t.c1[0] = -k1 * r41;
    t.c3[0] = -r41 * k3;
    t.c3[1] = -r42 * k3;
    t.c3[2] = -r43 * k3;
    t.m[0] = 0.5 * r42 * r42 * r32 * r31;
    t.m[1] = 0.5 * r42 * r42 * r32 * r41;
    t.m[2] = 0.5 * r41 * r41 * r42 * r31;
    t.m[3] = 0.5 * r41 * r41 * r31 * r32;
    t.m[4] = 0.5 * (r42 * r42 * r41 * r31 + r41 * r41 * r42 * r32);
  }
}

// beta += the Bernstein coefficients (times the binomials) of a product of three
// linear factors given by their values at the two ends
__device__ __forceinline__ void blossom(double *beta, double x0, double x1, double y0, double y1, double z0, double z1) {
  const double p = x0 * y0, q = x1 * y1, r = fma(x0, y1, x1 * y0);
  beta[0] = fma(p, z0, beta[0]);
  beta[1] = fma(r, z0, fma(p, z1, beta[1]));
  beta[2] = fma(r, z1, fma(q, z0, beta[2]));
  beta[3] = fma(q, z1, beta[3]);
}

// One block per final state: its simplices from the 8 (4) mesh cells that have k'
// as a corner, their vertex energies ranked, one thread per interval.  FP64 bound
// (~60 operations per interval and simplex that covers it).
constexpr int SX_THREADS = 96;

__global__ void __launch_bounds__(SX_THREADS) k_simplex_tab(int kind, int m1, int m2, int m3, const int2 *fin,
                                                            const int *widx, const int *rowmap, const double *ens,
                                                            int nw, SimplexTab t) {
  __shared__ SimplexEntry en[24];
  __shared__ double bp[SX_MAX];
  __shared__ int nbp;
  const int f = blockIdx.x, tid = threadIdx.x;
  const int nv = kind == 1 ? 3 : 4, per = kind == 1 ? 2 : 6, ne = nv * per;
  const int2 fs = fin[f];
  const int p = widx[fs.x];
  const int mesh[3] = {m1, m2, m3};
  if (tid == 0) nbp = 0;
  if (tid < ne) {   // simplex tid / nv of the cell whose corner (tid % nv) is k'
    const int tk = tid / nv, tl = tid % nv;
    auto corner = [&](int l) { return (kind == 1 ? kTri[tk][l] : kTet[tk][l]) - 1; };
    const int a = corner(tl);
    const int pc[3] = {p % m1, (p / m1) % m2, p / (m1 * m2)};
    int o[3];
    for (int d = 0; d < 3; ++d) {   // the cell's origin: k' minus the corner's offset
      o[d] = pc[d] - ((a >> d) & 1);
      if (o[d] < 0) o[d] += mesh[d];
    }
    SimplexEntry x;
    x.label = rowmap[o[0] + m1 * (o[1] + m2 * o[2])] >= 0 ? tl : -1;
    if (x.label >= 0) {
      for (int l = 0; l < nv; ++l) {
        int c[3];
        for (int d = 0; d < 3; ++d) {
          c[d] = o[d] + ((corner(l) >> d) & 1);
          if (c[d] >= mesh[d]) c[d] -= mesh[d];
        }
        const int mux = c[0] + m1 * (c[1] + m2 * c[2]);
        x.e[l] = rowmap[mux] >= 0 ? ens[(size_t)mux * nw + fs.y] : 0.0;
      }
      for (int u = 1; u < nv; ++u)
        for (int w = u; w > 0 && x.e[w] < x.e[w - 1]; --w) {
          const double y = x.e[w];
          x.e[w] = x.e[w - 1];
          x.e[w - 1] = y;
        }
      if (kind == 1) x.e[3] = x.e[2];
      simplex_coefs(kind, x);
    }
    en[tid] = x;
  }
  __syncthreads();
  // rank the vertex energies
  for (int u = tid; u < nv * ne; u += SX_THREADS) {
    const SimplexEntry &x = en[u / nv];
    if (x.label < 0) continue;
    const double e = x.e[u % nv];
    int rank = 0;
    for (int w = 0; w < nv * ne; ++w) {
      const SimplexEntry &y = en[w / nv];
      if (y.label < 0) continue;
      const double ye = y.e[w % nv];
      rank += (ye < e) || (ye == e && w < u);
    }
    bp[rank] = e;
    atomicAdd(&nbp, 1);
  }
  __syncthreads();
  const int n = nbp;
  if (tid == 0) t.n[f] = n;
  for (int i = tid; i < n; i += SX_THREADS) {
    const double b1 = bp[i], b0 = i ? bp[i - 1] : b1, w = b1 - b0;
    double beta[4] = {0.0, 0.0, 0.0, 0.0};
    if (w > 0.0)
      for (int u = 0; u < ne; ++u) {
        const SimplexEntry &x = en[u];
        if (x.label < 0 || b0 < x.e[0] || b1 > x.e[nv - 1]) continue;
        double l[4], r[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          l[c] = x.e[c] - b0;
          r[c] = x.e[c] - b1;
        }
        const bool first = b1 <= x.e[1], last = b0 >= x.e[nv - 2];
        if (first || last) {
          const double *k = first ? x.c1 : x.c3;
          const double zl = k[0] * l[0] + k[1] * l[1] + k[2] * l[2] + k[3] * l[3];
          const double zr = k[0] * r[0] + k[1] * r[1] + k[2] * r[2] + k[3] * r[3];
          const double xl = first ? l[0] : l[nv - 1], xr = first ? r[0] : r[nv - 1];
          if (kind == 1) blossom(beta, xl, xr, 1.0, 1.0, zl, zr);
          else blossom(beta, xl, xr, xl, xr, zl, zr);
        } else {
          const bool lo = x.label < 2;
          const double Sl = lo ? l[2] : l[1], Sr = lo ? r[2] : r[1], Ql = lo ? l[3] : l[0], Qr = lo ? r[3] : r[0];
          const double al = lo ? l[1] : l[2], ar = lo ? r[1] : r[2], bl = lo ? l[0] : l[3], br = lo ? r[0] : r[3];
          blossom(beta, Sl, Sr, Sl, Sr, x.m[0] * al + x.m[1] * bl, x.m[0] * ar + x.m[1] * br);
          blossom(beta, Ql, Qr, Ql, Qr, x.m[2] * bl + x.m[3] * al, x.m[2] * br + x.m[3] * ar);
          blossom(beta, Sl, Sr, Ql, Qr, x.m[4] * l[x.label], x.m[4] * r[x.label]);
        }
      }
    const double rw = w > 0.0 ? 1.0 / w : 0.0, r3 = rw * rw * rw;
    const size_t at = (size_t)f * t.stride + i;
    t.key[at] = (float)b1;
    t.b[at] = b1;
    t.lo[at] = make_double2(beta[0] * r3, beta[1] * r3);
    t.hi[at] = make_double2(beta[2] * r3, beta[3] * r3);
  }
}

void launch_simplex_tab(int kind, const int mesh[3], int nin, const int2 *fin, const int *widx, const int *rowmap,
                        const double *ens, int nw, const SimplexTab &t, cudaStream_t st) {
  if (nin > 0)
    k_simplex_tab<<<nin, SX_THREADS, 0, st>>>(kind, mesh[0], mesh[1], mesh[2], fin, widx, rowmap, ens, nw, t);
}

// the delta of final state f at energy e, before the 1 / (simplices per cell N)
__device__ __forceinline__ double simplex_delta(const SimplexTab &t, int f, double e) {
  const int n = t.n[f];
  const size_t at = (size_t)f * t.stride;
  const float *key = t.key + at;
  const double *b = t.b + at;
  // the first breakpoint >= e: found on the breakpoints rounded to FP32 (rounding is
  // monotone, so that one is at or before it), then settled in FP64
  const float ef = (float)e;
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (key[mid] < ef) lo = mid + 1; else hi = mid;
  }
  while (lo < n && b[lo] < e) ++lo;
  if (lo == 0 || lo == n) return 0.0;
  const double u = e - b[lo - 1], v = b[lo] - e;
  const double2 p = t.lo[at + lo], q = t.hi[at + lo];
  const double acc = fma(fma(p.x, v, p.y * u), v * v, fma(q.x, v, q.y * u) * (u * u));
  return acc < 1.0e-12 ? 0.0 : acc;
}

// ------------------------------------------------------- FP64 rate epilogue
// Window bands of the window k' as a list of final states (k', n), in order
__global__ void k_final_states(int nwv, int nw, const int *widx, const double *ens, double enref, double fsthick,
                               const int *cum, int2 *fin) {
  const int ip = blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= nwv) return;
  int f = cum[ip];
  for (int n = 0; n < nw; ++n)
    if (fabs(ens[(size_t)widx[ip] * nw + n] - enref) <= fsthick) fin[f++] = make_int2(ip, n);
}

void launch_final_states(int nwv, int nw, const int *widx, const double *ens, double enref, double fsthick,
                         const int *cum, int2 *fin, cudaStream_t st) {
  k_final_states<<<(nwv + 127) / 128, 128, 0, st>>>(nwv, nw, widx, ens, enref, fsthick, cum, fin);
}

__global__ void k_mode_tab(int n, const double *om, const double *bose, double T, double const_tp, ModeRec *mt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double o = om[i];
  mt[i] = ModeRec{o, o >= 0.5e-3 ? const_tp * (0.5 / o * g2unitfactor) : 0.0, bose[i], exp(o / kB / T)};
}

void launch_mode_tab(int n, const double *om, const double *bose, double T, double const_tp, ModeRec *mt,
                     cudaStream_t st) {
  k_mode_tab<<<(n + 127) / 128, 128, 0, st>>>(n, om, bose, T, const_tp, mt);
}

// Vertices of (initial state j, final state f): the k' rotation, the phonon mix,
// |g|^2 (wannier.f90:937-1009), X+- (interactions.f90:2278-2332, 2353) and the RTA
// rate (interactions.f90:3012-3034).  With the phonon side requested, also Y of
// the same vertex (interactions.f90:1857-1870, 1897: the (k, m, k + q, n, s) vertex
// of phonon state (q, s) is the (k, m, k', n, s) vertex here, q = k' - k) added
// into the phonon state's rate.
//
// Bound by the FP64 pipe (16 cycles per warp instruction on an SM), so the split
// keeps every lane on a vertex of its own and every FP64 instruction on the
// result: a thread is one initial state and walks epf_per(nin) final states, the
// same ones as its neighbours.  There is no divergence over the window bands,
// U_k' and the delta's table are read by broadcast, the sum over final states
// stays in the thread (compensated), and the occupations need no exponential:
// f(E + w) = 1 / (1 + e^x e^v) and 1 - f(E - w) = 1 / (1 + e^-x e^v), x = (E - mu) / kT
// per state, v = w / kT per mode.  12^3, nw 8, nb 6 (2.8 M pairs): 4.2 ms (3.9 at the
// FP64 rate for its ~850 instructions a pair; 5.1 with 16 final states per thread); one thread per (k', state) with a loop
// over the bands took 15.1 ms.  Tetrahedra, 10x12x11 (1.8 M pairs): 2.6 ms + 0.32 ms for
// the tables; with every simplex's formula at every vertex 511 ms.
template <bool F32>
__device__ __forceinline__ double2 epf_load(const FinalIn &c, int64_t off) {
  if (F32) return make_double2((double)c.re[off], (double)c.im[off]);
  return c.z[off];
}

template <bool F32, bool SIMPLEX, bool PH>
__global__ void __launch_bounds__(EPF_THREADS) k_epilogue_final(int j0, int ns, FinalIn c, RateParams rp, EpiData d,
                                                                double *partial, int nblk) {
  const int2 it = epf_item((int64_t)blockIdx.x * EPF_THREADS + threadIdx.x, ns);
  const int jl = it.x, grp = it.y;
  if (grp >= nblk) return;
  const int j = j0 + jl;
  const int nw = rp.nw, nb = rp.nb;
  const int code = d.st_code[j];
  const int p = d.sidx[code / nw], m = code % nw;
  const double E = d.ens[(size_t)p * nw + m];
  const double kT = kB * rp.T, x = (E - rp.chempot) / kT;
  const double ex = exp(x), emx = exp(-x);
  const double f1 = 1.0 / (ex + 1.0);
  const double isig = SIMPLEX ? 0.0 : 1.0 / rp.sigma;
  const double dnorm = SIMPLEX ? rp.inv_nk / (rp.delta_kind == 1 ? 2.0 : 6.0)
                               : (1.0 / sqrt(TWOPI)) / rp.sigma * rp.inv_nk;
  const int a1 = p % rp.mesh[0], a2 = (p / rp.mesh[0]) % rp.mesh[1], a3 = p / (rp.mesh[0] * rp.mesh[1]);
  const double2 *Uk = d.U + ((size_t)p * nw + m) * nw;
  double sum = 0.0, comp = 0.0;
  const int f0 = grp * epf_per(d.nin), fe = min(d.nin, f0 + epf_per(d.nin));
  for (int f = f0; f < fe; ++f) {
    const int2 fs = d.fin[f];
    const int pp = d.widx[fs.x];
    const double eps = d.ens[(size_t)pp * nw + fs.y];
    const double2 *Ukp = d.U + ((size_t)pp * nw + fs.y) * nw;
    int q1 = pp % rp.mesh[0] - a1, q2 = (pp / rp.mesh[0]) % rp.mesh[1] - a2, q3 = pp / (rp.mesh[0] * rp.mesh[1]) - a3;
    q1 += q1 < 0 ? rp.mesh[0] : 0;
    q2 += q2 < 0 ? rp.mesh[1] : 0;
    q3 += q3 < 0 ? rp.mesh[2] : 0;
    const int q = q1 + rp.mesh[0] * (q2 + rp.mesh[1] * q3);
    const int64_t base = (int64_t)fs.x * c.ldc + jl * c.js;
    double2 h[32];
    for (int s = 0; s < nb; ++s) {
      double2 a = make_double2(0.0, 0.0);
      for (int np = 0; np < nw; ++np) cfma_cj(a, Ukp[np], epf_load<F32>(c, base + (np + nw * s) * c.xs));
      h[s] = a;
    }
    double2 unm = make_double2(0.0, 0.0);   // dot_product(el_evec_kp, el_evec_k), polar crystals
    if (d.glp)
      for (int n = 0; n < nw; ++n) cfma_cj(unm, Ukp[n], Uk[n]);
    double acc = 0.0;
    for (int s = 0; s < nb; ++s) {
      const int qs = q * nb + s;
      const ModeRec mt = d.mt[qs];
      double2 g = make_double2(0.0, 0.0);
      const double2 *u = d.u + (size_t)qs * nb;
      for (int sp = 0; sp < nb; ++sp) cfma(g, u[sp], h[sp]);
      if (d.glp) cfma(g, d.glp[qs], unm);   // long-range term (wannier.f90:998-1006)
      const double gg = fma(g.x, g.x, g.y * g.y);
      double xp = 0.0, xm = 0.0, y = 0.0;
      if (mt.cx != 0.0) {
        double dp, dm;
        if (SIMPLEX) {
          dp = simplex_delta(d.sx, f, E + mt.om) * dnorm;
          dm = simplex_delta(d.sx, f, E - mt.om) * dnorm;
        } else {
          const double tp = ((E + mt.om) - eps) * isig, tm = ((E - mt.om) - eps) * isig;
          dp = dnorm * exp(-0.5 * tp * tp);
          dm = dnorm * exp(-0.5 * tm * tm);
        }
        double A = fma(ex, mt.ev, 1.0), B = fma(emx, mt.ev, 1.0);
        if (mt.ev > 1e260) {   // omega / kT > 600: the factors may leave FP64's range one by one
          const double v = mt.om / kT;
          A = 1.0 + exp(x + v);
          B = 1.0 + exp(v - x);
        }
        const double gc = gg * mt.cx, fp = 1.0 / A;
        xp = gc * (mt.bose + fp) * dp;
        xm = gc * (mt.bose + 1.0 / B) * dm;
        if (PH) {
          // Y: delta(E' - omega) at the initial electron (k, m), interactions.f90:1862; the Gaussian is even
          const double dy = SIMPLEX ? simplex_delta(d.sx, j, eps - mt.om) * dnorm : dp;
          y = gc * (f1 * (1.0 - fp) / (1.0 + mt.bose)) * dy;
          if (d.phr && y != 0.0) atomicAdd(d.phr + q + (size_t)rp.N * s, d.ph_scale * y);
        }
      }
      acc += xp + xm;
      if (d.g2) {
        const int64_t off = (int64_t)j * d.per_state + (int64_t)f * nb + s;
        if (off < d.cap) {
          d.g2[off] = mt.om == 0.0 ? 0.0 : 0.5 * gg / mt.om * g2unitfactor;
          if (d.xp) d.xp[off] = xp;
          if (d.xm) d.xm[off] = xm;
          if (d.yv) d.yv[off] = y;
        }
      }
    }
    const double t = sum + acc;   // compensated (Neumaier)
    comp += (fabs(sum) >= fabs(acc)) ? (sum - t) + acc : (acc - t) + sum;
    sum = t;
  }
  partial[(size_t)j * nblk + grp] = sum + comp;
}

void launch_epilogue_final(int j0, int j1, const FinalIn &c, const RateParams &rp, const EpiData &d, double *partial,
                           int nblk, cudaStream_t st) {
  const int ns = j1 - j0;
  if (ns <= 0 || d.nin <= 0) return;
  const unsigned grid = (unsigned)epf_grid(ns, d.nin);
  const bool ph = d.phr || d.yv, simplex = rp.delta_kind != 0;
  auto go = [&](auto k) { k<<<grid, EPF_THREADS, 0, st>>>(j0, ns, c, rp, d, partial, nblk); };
  if (c.z) {
    if (simplex) ph ? go(k_epilogue_final<false, true, true>) : go(k_epilogue_final<false, true, false>);
    else ph ? go(k_epilogue_final<false, false, true>) : go(k_epilogue_final<false, false, false>);
  } else {
    if (simplex) ph ? go(k_epilogue_final<true, true, true>) : go(k_epilogue_final<true, true, false>);
    else ph ? go(k_epilogue_final<true, false, true>) : go(k_epilogue_final<true, false, false>);
  }
}

// rates(ik, m) = compensated sum of the block partials in block order
__global__ void k_rate_final(int nst, int nblk, const double *partial, const int *st_code, int nw,
                             int N, double *rates_f) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nst) return;
  double s = 0.0, c = 0.0;
  for (int b = 0; b < nblk; ++b) {
    double x = partial[(size_t)j * nblk + b], t = s + x;
    c += (fabs(s) >= fabs(x)) ? (s - t) + x : (x - t) + s;
    s = t;
  }
  int code = st_code[j];
  rates_f[(code / nw) + (int64_t)N * (code % nw)] = s + c;
}

void launch_rate_final(int nst, int nblk, const double *partial, const int *st_code, int nw,
                       int N, double *rates_f, cudaStream_t st) {
  if (nst <= 0) return;
  k_rate_final<<<(nst + 127) / 128, 128, 0, st>>>(nst, nblk, partial, st_code, nw, N, rates_f);
}

// ------------------------------------------ degenerate-subspace averaging
// The gauge fixing of plot_along_path (wannier.f90:1332-1384, the same loops
// in test/check_interactions_symmetries.f90:330-384) on a |g|^2 vertex list in
// the electron side's order (state j, final state f = (k', n), branch s),
// FP64.  Three passes in the reference's order, each over groups of one index
// with the others fixed: branches s of q = k' - k (phonon energies), initial
// bands m of each k, final bands n of each k' (electron energies); a member's
// partners are those with |E - E'| < thres.  Mode 0 restates the reference's
// loops literally, in place: member a becomes the mean, summed in member
// order, of its partners' values as they are at that moment (so a later member
// sees its predecessors' new values); mode 1 takes every mean from the values
// before the pass.  One thread per group set; groups of a pass are disjoint.
constexpr int DEG_MAXG = 64;

__device__ void deg_group(int mode, double thres, int c, double *v, int64_t st, const double *e) {
  double tmp[DEG_MAXG];
  if (mode == 1)
    for (int a = 0; a < c; ++a) tmp[a] = v[a * st];
  for (int a = 0; a < c; ++a) {
    int cnt = 0;
    double aux = 0.0;
    for (int b = 0; b < c; ++b)
      if (fabs(e[a] - e[b]) < thres) {
        ++cnt;
        aux += mode == 0 ? v[b * st] : tmp[b];
      }
    v[a * st] = aux / (double)cnt;
  }
}

// window bands of mesh point p in band order: their count, bands in `band`
__device__ __forceinline__ int window_bands(const double *ens, int p, int nw, double enref, double fsthick, int *band,
                                            double *e) {
  int c = 0;
  for (int n = 0; n < nw; ++n) {
    const double x = ens[(size_t)p * nw + n];
    if (fabs(x - enref) <= fsthick) {
      band[c] = n;
      e[c] = x;
      ++c;
    }
  }
  return c;
}

struct DegList {
  double *g2;
  const int *st_code, *arow, *widx, *cum, *first_state;
  const double *ens, *om;
  int nst, nA, nwv, nw, nb, mesh[3];
  int64_t per;          // entries per state: nin * nb
  double enref, fsthick, thres;
  int mode;
};

// pass 1: branches, per (state, k' row)
__global__ void k_deg_branches(DegList L) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)L.nst * L.nwv) return;
  const int j = (int)(t / L.nwv), b = (int)(t % L.nwv);
  const int p = L.arow[L.st_code[j] / L.nw], pp = L.widx[b];
  const int a1 = p % L.mesh[0], a2 = (p / L.mesh[0]) % L.mesh[1], a3 = p / (L.mesh[0] * L.mesh[1]);
  const int b1 = pp % L.mesh[0], b2 = (pp / L.mesh[0]) % L.mesh[1], b3 = pp / (L.mesh[0] * L.mesh[1]);
  const int q = (int)(floormod(b1 - a1, L.mesh[0]) +
                      L.mesh[0] * (floormod(b2 - a2, L.mesh[1]) + L.mesh[1] * floormod(b3 - a3, L.mesh[2])));
  double e[DEG_MAXG];
  for (int s = 0; s < L.nb; ++s) e[s] = L.om[(size_t)q * L.nb + s];
  const int nf = L.cum[b + 1] - L.cum[b];
  for (int r = 0; r < nf; ++r)
    deg_group(L.mode, L.thres, L.nb, L.g2 + (int64_t)j * L.per + (int64_t)(L.cum[b] + r) * L.nb, 1, e);
}

// pass 2: initial bands, per (initial k row, final state); the states of one
// k row are consecutive, in band order
__global__ void k_deg_initial(DegList L, int nin) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)L.nA * nin) return;
  const int a = (int)(t / nin), f = (int)(t % nin);
  const int j0 = L.first_state[a], c = L.first_state[a + 1] - j0;
  if (c <= 0) return;
  const int p = L.arow[a];
  double e[DEG_MAXG];
  for (int i = 0; i < c; ++i) e[i] = L.ens[(size_t)p * L.nw + L.st_code[j0 + i] % L.nw];
  for (int s = 0; s < L.nb; ++s)
    deg_group(L.mode, L.thres, c, L.g2 + (int64_t)j0 * L.per + (int64_t)f * L.nb + s, L.per, e);
}

// pass 3: final bands, per (state, k' row)
__global__ void k_deg_final(DegList L) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)L.nst * L.nwv) return;
  const int j = (int)(t / L.nwv), b = (int)(t % L.nwv);
  int band[DEG_MAXG];
  double e[DEG_MAXG];
  const int c = window_bands(L.ens, L.widx[b], L.nw, L.enref, L.fsthick, band, e);
  for (int s = 0; s < L.nb; ++s)
    deg_group(L.mode, L.thres, c, L.g2 + (int64_t)j * L.per + (int64_t)L.cum[b] * L.nb + s, L.nb, e);
}

int launch_degenerate_average(double *g2, int64_t per, int nin, const int *st_code, const int *arow, const int *widx,
                              const int *cum, const int *first_state, const double *ens, const double *om, int nst,
                              int nA, int nwv, int nw, int nb, const int mesh[3], double enref, double fsthick,
                              double thres, int mode, cudaStream_t st) {
  if (nw > DEG_MAXG || nb > DEG_MAXG) return 1;
  DegList L{g2, st_code, arow, widx, cum, first_state, ens, om, nst, nA, nwv, nw, nb, {mesh[0], mesh[1], mesh[2]},
            per, enref, fsthick, thres, mode};
  const int64_t n1 = (int64_t)nst * nwv, n2 = (int64_t)nA * nin;
  if (n1 > 0) k_deg_branches<<<(unsigned)((n1 + 127) / 128), 128, 0, st>>>(L);
  if (n2 > 0) k_deg_initial<<<(unsigned)((n2 + 127) / 128), 128, 0, st>>>(L, nin);
  if (n1 > 0) k_deg_final<<<(unsigned)((n1 + 127) / 128), 128, 0, st>>>(L);
  return 0;
}

}  // namespace ephg

extern "C" int ephg_debug_epilogue_grid(int nstates, int nin, int64_t *grid) {
  using namespace ephg;
  if (nstates <= 0 || nin <= 0 || !grid) return EPHG_ERR_ARG;
  grid[0] = epf_grid(nstates, nin);
  grid[1] = grid[2] = 1;
  const int64_t ng = epf_blocks(nin);
  if (ng * epf_per(nin) < nin || (ng - 1) * epf_per(nin) >= nin) return EPHG_ERR_INDEX;
  std::vector<bool> seen((size_t)(nstates * ng));
  int64_t left = nstates * ng;
  for (int64_t t = 0; t < grid[0] * EPF_THREADS; ++t) {
    const int2 p = epf_item(t, nstates);
    if (p.y >= ng) continue;
    if (p.x < 0 || p.x >= nstates || p.y < 0 || seen[(size_t)(p.x + nstates * (int64_t)p.y)]) return EPHG_ERR_INDEX;
    seen[(size_t)(p.x + nstates * (int64_t)p.y)] = true;
    --left;
  }
  return left ? EPHG_ERR_INDEX : EPHG_OK;
}

extern "C" int ephg_debug_once_per_device(int n, const int *devices, int *ran) {
  if (n <= 0 || !devices || !ran) return EPHG_ERR_ARG;
  ephg::OncePerDevice once;
  for (int i = 0; i < n; ++i) {
    ran[i] = 0;
    once.on(devices[i], [&] { ran[i] = 1; });
  }
  return EPHG_OK;
}
