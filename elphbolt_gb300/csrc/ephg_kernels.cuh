// ephg_kernels.cuh - launchers of the library's kernels (internal interface).
#pragma once
#include "ephg_common.cuh"

namespace ephg {

// ---- phases ----
void launch_roots(int L, double2 *roots, cudaStream_t st);
// out[row*ldo + r] = e^{2 pi i k_row . R_r} (/ deg_r if deg) (conjugated if conj);
// k on the mesh (row -> mesh index rowp[row], or row itself if rowp == nullptr)
void launch_phase_mesh(int nrows, const int *rowp, const int mesh[3], int L, int nR,
                       const int *R, const double *deg, int conj, const double2 *roots,
                       double2 *out, int64_t ldo, cudaStream_t st);
// same for arbitrary fractional k: kv (nrows,3) column-major as the reference
void launch_phase_frac(int nrows, const double *kv, int nR, const int *R, const double *deg,
                       double2 *out, int64_t ldo, cudaStream_t st);
// The same for the vectors perm[0..nrows) of kv (0..nrows - 1 if null; column stride ldk); lo, ext: the
// range of the cell coordinates per dimension; deg nullable; out rows at stride ldo
void launch_phase_cells(int nrows, const double *kv, int64_t ldk, const int *perm, int nR, const int *R,
                        const double *deg, const int lo[3], const int ext[3], double2 *out, int64_t ldo,
                        cudaStream_t st);

// out[p][e] = sum_R e^{2 pi i k_p.R} X(R)[e] for every point p of the mesh (muxed
// order), X given on the box of cell coordinates [lo, lo + ext) per dimension
// (box[((r1 ext2 + r2) ext3 + r3) nn + e], zero where there is no cell); three
// 1-D passes through t1 (ext1 ext2 m3 nn) and t2 (ext1 m2 m3 nn).
void launch_mesh_fourier(const double2 *box, const int lo[3], const int ext[3], int nn, const int mesh[3], int L,
                         const double2 *roots, double2 *t1, double2 *t2, double2 *out, cudaStream_t st);

// ---- Fourier sum of many columns over integer cells, one dimension at a time ----
// The cells of a Wigner-Seitz set as nested index tables (device): tab1 [npair][ext3]
// the cell of (R1, R2 of the pair, R3) or -1; tab2 [n1][ext2] the pair of (R1, R2)
// or -1; tab3 [ext1] the R1 slot or -1.  ok: every cell is distinct and the tables fit.
struct CellTab {
  bool ok = false;
  int lo[3] = {0, 0, 0}, ext[3] = {1, 1, 1};
  int npair = 0, n1 = 0;
  const int *tab1 = nullptr, *tab2 = nullptr, *tab3 = nullptr;
};
// FP64 instructions per column of launch_cells_fourier; infinity where it cannot run
double cells_fourier_cost(const CellTab &t, const int mesh[3], int64_t rows);
// Cycles of one SM for 128 columns: four warps' FP64 instructions at 16 cycles each, as measured
inline double cells_fourier_cycles(const CellTab &t, const int mesh[3], int64_t rows) {
  return 60.0 * cells_fourier_cost(t, mesh, rows);
}
// work rows (double2 per column) of t1 and t2
inline int64_t cells_t1_rows(const CellTab &t, const int mesh[3]) { return (int64_t)t.npair * mesh[2]; }
inline int64_t cells_t2_rows(const CellTab &t, const int mesh[3]) { return (int64_t)t.n1 * mesh[1] * mesh[2]; }
// out[rowmap[p]][c] = sum_cells e^{2 pi i k_p.R} scale[cell] in[cell][c], c < nc, for the mesh
// points p with rowmap[p] >= 0; in rows at stride ldi, out rows at stride ldo; scale nullable.
void launch_cells_fourier(const CellTab &t, const double2 *in, int64_t ldi, const double *scale, int nc,
                          const int mesh[3], int L, const double2 *roots, double2 *t1, double2 *t2,
                          const int *rowmap, double2 *out, int64_t ldo, cudaStream_t st);
// rowmap[p] = i for p = rows[i], -1 elsewhere (N mesh points)
void launch_row_map(int N, int nrows, const int *rows, int *rowmap, cudaStream_t st);

// ---- FP64 complex GEMM: C[M][N] = A[M][K] * B[K][N], row-major ----
void launch_zgemm(int M, int N, int K, const double2 *A, int64_t lda, const double2 *B,
                  int64_t ldb, double2 *C, int64_t ldc, cudaStream_t st);

// ---- Hermitian eigensolver (batched, n <= 32) ----
// A: batch matrices (n,n) column-major, `stride` values apart, upper triangle forced
// Hermitian as in wannier.f90:481-486.  w: (batch, n) ascending;
// V: (batch, n, n) column-major, columns = eigenvectors.
void launch_heig(int batch, int n, const double2 *A, int64_t stride, double *w, double2 *V,
                 int *err, cudaStream_t st);

// ---- electron / phonon post-processing ----
// C: (nk, 4*nw*nw) from the H(k) GEMM (H, dH_x, dH_y, dH_z), nvel = 0 or 3
void launch_el_post(int nk, int nw, const double *w, const double2 *V, const double2 *C,
                    int64_t ldc, int with_vel, const double *scissor, double *energies_f,
                    double *vel_f, double2 *evecs_f, double *ens_i, cudaStream_t st);

// omega, Gamma / negative handling, velocities; outputs in reference layout
// (energies_f (nq,nb), evecs_f (nq,nb,nb), vel_f (nq,nb,3)) and/or internal
// (om_i [q][s], u_i [q][s][c] = evec/sqrt(M_c)).
void launch_ph_post(int nq, int nb, const int *qp, const double *qv, const double *w,
                    const double2 *V, const double2 *dDq, int64_t ldd, int with_vel, const double *masses,
                    double *energies_f, double2 *evecs_f, double *vel_f, double *om_i,
                    double2 *u_i, float2 *u_f, int *err, cudaStream_t st);

// ---- gkRp / gReq layout helpers ----
void launch_permute_gwann(int nw, int nb, int nwsk, int nwsg, const double2 *raw, double2 *G,
                          cudaStream_t st);
// gReq GEMM output (nq, [i,j,Re,s]) -> (nw,nw,nb,nwsk,nq) column-major
void launch_permute_greq(int nq, int nw, int nb, int nwsk, const double2 *in, double2 *out,
                         cudaStream_t st);

// ---- g2 of a vertex list (wannier.f90:903-1011) ----
// G (nv rows of nw nw nb): the cell sums of vertices perm[0..nv); the vertex arrays' column
// stride is ld.  Lv (ld, nb), nullable: the polar long-range vector of each vertex's q
void launch_g2_vertices(int nv, const int *perm, int64_t ld, int nw, int nb, const double2 *G, const double2 *ek,
                        const double2 *ekp, const double2 *eq, const double *ph_en, const double *masses,
                        const double2 *Lv, double *g2, cudaStream_t st);

// ---- polar long-range terms (wannier.f90:784-901, 1013-1071) ----
// Crystal data of a polar crystal on the device (ephg_set_polar).  The Ewald
// sums run over the box of reciprocal-lattice vectors m1 b1 + m2 b2 + m3 b3,
// |m_i| <= coarse_qmesh(i), with the cut qeq / (4 alph) < gmax.
struct PolarDev {
  int nat = 0, nb = 0, M = 0;
  const double *G = nullptr;      // [M][3] box vectors, Cartesian 1/bohr, in the reference's loop order
  const double *Gcell = nullptr;  // [Mcell][3] those of them that can pass the cut for q in the first cell
  int Mcell = 0;
  const float *Gf = nullptr, *Gcellf = nullptr;   // the same in FP32, for the first test of the cut
  const double *born = nullptr;   // born(x, ipol, at) at x + 3 ipol + 9 at
  const double *tau = nullptr;    // [nat][3] Cartesian basis, bohr
  const double2 *Da = nullptr;    // (nb,nb) column-major: the q-independent sum (before fac)
  const double *masses = nullptr; // per atom, amu
  double eps[9];                  // dielectric tensor, column-major
  double rec[9];                  // reciprocal vectors (columns, 1/nm, with 2 pi)
  double alph = 0, gmax = 14.0, fac = 0;   // tpiba^2 (1/bohr^2), cut, 8 pi / volume (1/bohr^3)
};
// Per q (mesh index qp[q] on `mesh`, else crystal coordinates qv (nq,3)
// column-major): Dq[q] += massnorm * dyn_l(q) (nullable; matrices ldd values apart),
// dDq[q] += massnorm * ddyn_l(q) * bohr2nm (nullable; three matrices per q, ldd apart), and
// Lq[q][c] (nullable) with long_range_prefac(q, u) = sum_c Lq[q][c] u[c].
void launch_polar_q(const PolarDev &P, int nq, const int *qp, const int mesh[3], const double *qv,
                    double2 *Dq, double2 *dDq, int64_t ldd, double2 *Lq, cudaStream_t st);
// The q-independent part of dyn_nonanalytic into Da (nb,nb), once per crystal.
void launch_polar_da(const PolarDev &P, double2 *Da, cudaStream_t st);
// glp[q][s] = sum_c Lq[q][c] u[q][s][c] (u = evec / sqrt(M)), and its fp32 copy (nullable)
void launch_glprefac(int nq, int nb, const double2 *Lq, const double2 *u, double2 *glp, float2 *glpf,
                     cudaStream_t st);

// ---- q index table (vector.f90:86-102 on integers) ----
void launch_kq_index(const int mesh[3], int nk, const int64_t *k_idx, int nkp,
                     const int64_t *kp_idx, int64_t *q_idx, int *err, cudaStream_t st);

// ---- rate pipeline ----
void launch_window_flags(int N, int nw, const double *ens, double enref, double fsthick,
                         int *flag, cudaStream_t st);
void launch_state_flags(int nwv, int nw, const int *widx, const double *ens, double enref,
                        double fsthick, int *flag, int *nin_k, cudaStream_t st);
void launch_iota(int n, int *out, cudaStream_t st);
// Stage A rotation: B[Rp][c] (ldb) for states j in [j0,j1) of k-chunk [i0, i0+kc) and the
// (mode, cell) blocks s + nb Rp in [blk0, blk0 + nblk) that gk holds (nw nw values each):
// B = phk[k][Rp] * sum_m' U_k[m][m'] gk(n',m',s',Rp), phk = conj(e^{2 pi i k.Rp})/deg(Rp) (row stride nws).
// Columns: chunks of sc states (the last one shorter), within a chunk [n' + nw s'][state].
void launch_rotate_states_fp64(int j0, int j1, int i0, const int *st_code, int nw, int nb, int nws, int64_t blk0,
                               int64_t nblk, const int *widx, const double2 *U, const double2 *gk, int64_t ldgk,
                               const double2 *phk, double2 *B, int64_t ldb, int sc, int nst, cudaStream_t st);
// Per (q, s), FP64 epilogue: omega, 2 pi / hbar g2unitfactor / (2 omega) (0 below 0.5 meV), n(omega), e^(omega / kT)
struct alignas(16) ModeRec {
  double om, cx, bose, ev;
};
// Triangle / tetrahedron deltas of the final states as tables (launch_simplex_tab):
// per final state the sorted breakpoints b (key: rounded to FP32) and for each the
// Bernstein coefficients (lo, hi) of the interval that ends there.
constexpr int SX_MAX = 96;
struct SimplexTab {
  int stride;           // entries per final state: 96, or 18 for triangles
  int *n;
  float *key;
  double *b;
  double2 *lo, *hi;
};
struct EpiData {
  const int *widx;      // window (k' row) -> mesh index
  const int *st_code;   // state -> i*nw + m, i the state's k row (an A-row)
  const int *sidx;      // A-row (the k of initial states) -> mesh index
  const int *cum;       // window k' -> first (k',n) final-state rank
  const double *ens;    // [p][b] eV
  const double2 *U;     // [p][b][c]
  const float2 *Uf;     // same in fp32 (split path)
  const double *om;     // [q][s] eV
  const double2 *u;     // [q][s][c] evec/sqrt(M)
  const float2 *uf;     // same in fp32
  const double *bose;   // [q][s]
  // FP64 epilogue: the final states (window k' row, band), the (q, s) table of
  // launch_mode_tab and, for the triangle / tetrahedron deltas, theirs
  const int2 *fin;
  int nin;
  const ModeRec *mt;
  SimplexTab sx;
  int64_t per_state;    // vertices per initial state
  double *g2, *xp, *xm; // optional vertex lists
  int64_t cap;
  // phonon side (ibzq 'Y' + the ph-e rates), both nullable: phr (N, nb)
  // column-major receives ph_scale * Y summed over the vertices of each (q, s)
  // (device atomics); yv is the optional per-vertex Y list in the order of g2
  double *phr, *yv;
  double ph_scale;      // el%spindeg
  // polar crystals: glp[q][s] = long_range_prefac(q, u_s), added to each vertex
  // as glp * <U_k'[n]|U_k[m]> (wannier.f90:998-1006); nullable
  const double2 *glp;
  const float2 *glpf;   // same in fp32 (split path)
};
// Parameter sets of a merged request (ephg_el_rates_sets): requests that differ
// only in T, sigma and chempot share their vertices and |g|^2, so the
// contractions run once and the rate epilogue once per set.  Set 0 is the
// request itself (its RateParams, EpiData.bose and partial buffer); sets 1..n-1
// carry their own parameters, FP64 Bose factors and rate partials.
constexpr int MAX_SETS = 8;   // EPHG_MAX_SETS
struct RateSets {
  int n;
  RateParams rp[MAX_SETS];
  double *bose[MAX_SETS];      // [q][s] per set (set 0: EpiData.bose)
  const ModeRec *mt[MAX_SETS]; // FP64 epilogue: [q][s] per set (set 0: EpiData.mt)
  double *partial[MAX_SETS];   // [j][iblk] per set (set 0: the caller's partial)
};
// Final states of the window rows in order: fin[cum[ip] + rank] = (ip, band)
void launch_final_states(int nwv, int nw, const int *widx, const double *ens, double enref, double fsthick,
                         const int *cum, int2 *fin, cudaStream_t st);
// The simplex tables of nin final states (kind 1 triangles, 2 tetrahedra); rowmap: mesh point -> window row or -1
void launch_simplex_tab(int kind, const int mesh[3], int nin, const int2 *fin, const int *widx, const int *rowmap,
                        const double *ens, int nw, const SimplexTab &t, cudaStream_t st);
// the mode table of n (q, s)
void launch_mode_tab(int n, const double *om, const double *bose, double T, double const_tp, ModeRec *mt,
                     cudaStream_t st);
// FP64 epilogue over the states [j0, j1): the Rp sums G(x = n' + nw s') of (window row ip,
// state j) at ip ldc + x xs + (j - j0) js, in FP64 (z) or as FP32 planes (re, im).  Rate
// partials [j][group of epf_per(nin) final states].
constexpr int EPF_THREADS = 128;
// A thread's final states: one while there are few, so that a request of few states fills the chip
// and waits for one vertex instead of 16 in a row; more where the partials, added up one after the
// other per state, would take longer than a further vertex (both grow with nin; about 512
// partials), at most 16.  Stage C in ms with 1 / 2 / 4 / 16 (one thread per window row and
// state, its bands in turn, before): nw 4, 36 states 0.07 / 0.09 / 0.14 / 0.48 (0.14); nw 16,
// 740 states 2.5 / 2.7 / 2.8 / 8.0 (5.7); nw 8, 1,984 states 6.5 / 6.0 / 5.8 / 6.6 (18.4); wedge of 82
// states with 2,238 final states 0.94 / 0.66 / 0.50 / 0.60 (0.78).
__host__ __device__ inline int epf_per(int nin) {
  const int n = (nin + 511) / 512;
  return n < 1 ? 1 : n > 16 ? 16 : n;
}
inline int epf_blocks(int nin) { return (nin + epf_per(nin) - 1) / epf_per(nin); }
// Its grid is one-dimensional over the (state, group) pairs, states fastest: no lane idles for want
// of states, and a mesh of 2^24 points has more groups than the other grid dimensions hold (65,535).
inline int64_t epf_grid(int ns, int nin) { return ((int64_t)ns * epf_blocks(nin) + EPF_THREADS - 1) / EPF_THREADS; }
// (state, group) of thread t
__host__ __device__ inline int2 epf_item(int64_t t, int ns) { return make_int2((int)(t % ns), (int)(t / ns)); }
struct FinalIn {
  const double2 *z = nullptr;
  const float *re = nullptr, *im = nullptr;
  int64_t ldc = 0, xs = 1, js = 0;
};
void launch_epilogue_final(int j0, int j1, const FinalIn &c, const RateParams &rp, const EpiData &d, double *partial,
                           int nblk, cudaStream_t st);
void launch_bose(int N, int nb, const double *om, double T, double *bose, cudaStream_t st);
void launch_rate_final(int nst, int nblk, const double *partial, const int *st_code, int nw,
                       int N, double *rates_f, cudaStream_t st);
// degenerate-subspace averaging of a vertex list (3 launches); 1 if nw or nb > 64
int launch_degenerate_average(double *g2, int64_t per, int nin, const int *st_code, const int *arow, const int *widx,
                              const int *cum, const int *first_state, const double *ens, const double *om, int nst,
                              int nA, int nwv, int nw, int nb, const int mesh[3], double enref, double fsthick,
                              double thres, int mode, cudaStream_t st);

}  // namespace ephg
