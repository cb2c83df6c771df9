// ephg_api.cu - the C ABI (include/ephg.h): handle, uploads and the
// orchestration of the e-ph vertex path on one GPU and one CUDA stream.
#include <cub/device/device_scan.cuh>
#include <cub/device/device_select.cuh>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/ephg.h"
#include "../../include/ephg_debug.h"
#include "ephg_kernels.cuh"
#include "ephg_tc.cuh"
#include "ephg_ws.cuh"
#include "ephg_handle.cuh"
#include "ephg_sym.cuh"
#include "ephg_xgemm.cuh"

using namespace ephg;

#define fail ephg::api_fail

static thread_local std::string g_err;

int ephg::api_fail(int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

#define CK(call)                                                                          \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess)                                                                \
      return fail(EPHG_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__, #call,                \
                  cudaGetErrorString(e_));                                                \
  } while (0)

#define CKL()                                                                             \
  do {                                                                                    \
    cudaError_t e_ = cudaGetLastError();                                                  \
    if (e_ != cudaSuccess)                                                                \
      return fail(EPHG_ERR_CUDA, "%s:%d launch: %s", __FILE__, __LINE__,                   \
                  cudaGetErrorString(e_));                                                \
  } while (0)

namespace {

int gcd_i(int a, int b) { return b == 0 ? a : gcd_i(b, a % b); }
int lcm3(const int m[3]) {
  int l = m[0];
  l = l / gcd_i(l, m[1]) * m[1];
  l = l / gcd_i(l, m[2]) * m[2];
  return l;
}

// ws_wrapping_vectors (wannier.f90:532-582), q independent: evaluated once per
// (R, atom pair) at create time instead of once per q.
std::vector<int> ws_wrap(const double lvec[9], const double vl[3], double eps) {
  int iv0[3];
  double wl[3];
  for (int i = 0; i < 3; ++i) {
    iv0[i] = (int)std::trunc(vl[i]);
    wl[i] = vl[i] - (double)iv0[i];
  }
  double d = 1.79769313486231570815e308;
  auto norm = [&](int i, int j, int k) {
    double v[3] = {wl[0] + i, wl[1] + j, wl[2] + k}, wc[3];
    for (int r = 0; r < 3; ++r) wc[r] = lvec[r] * v[0] + lvec[r + 3] * v[1] + lvec[r + 6] * v[2];
    return std::sqrt(wc[0] * wc[0] + wc[1] * wc[1] + wc[2] * wc[2]);
  };
  for (int k = -3; k <= 3; ++k)
    for (int j = -3; j <= 3; ++j)
      for (int i = -3; i <= 3; ++i) {
        double nr = norm(i, j, k);
        if (std::fabs(nr - d) < eps) {
        } else if (nr < d) d = nr;
      }
  std::vector<int> out;
  for (int k = -3; k <= 3; ++k)
    for (int j = -3; j <= 3; ++j)
      for (int i = -3; i <= 3; ++i)
        if (std::fabs(norm(i, j, k) - d) < eps) {
          out.push_back(i - iv0[0]);
          out.push_back(j - iv0[1]);
          out.push_back(k - iv0[2]);
        }
  return out;
}

// The nested cell tables of launch_cells_fourier (rows r: n cells, 3 ints each),
// packed one after the other; offsets off[0..2].  False: cells repeat or span
// too large a box, and the sums run as matrix products instead.
bool cell_tables(const std::vector<int> &r, int n, CellTab &t, std::vector<int> &tab, size_t off[3]) {
  if (n <= 0) return false;
  for (int d = 0; d < 3; ++d) {
    int lo = r[d], hi = r[d];
    for (int i = 1; i < n; ++i) {
      lo = std::min(lo, r[3 * i + d]);
      hi = std::max(hi, r[3 * i + d]);
    }
    if ((int64_t)hi - lo > 1023 || lo < -1023 || hi > 1023) return false;
    t.lo[d] = lo;
    t.ext[d] = hi - lo + 1;
  }
  std::map<std::pair<int, int>, int> pair;
  std::map<int, int> slot;
  for (int i = 0; i < n; ++i) {
    slot.emplace(r[3 * i], 0);
    pair.emplace(std::make_pair(r[3 * i], r[3 * i + 1]), 0);
  }
  int k = 0;
  for (auto &x : slot) x.second = k++;
  k = 0;
  for (auto &x : pair) x.second = k++;
  t.n1 = (int)slot.size();
  t.npair = (int)pair.size();
  off[0] = 0;
  off[1] = (size_t)t.npair * t.ext[2];
  off[2] = off[1] + (size_t)t.n1 * t.ext[1];
  tab.assign(off[2] + t.ext[0], -1);
  for (int i = 0; i < n; ++i) {
    const int *R = &r[3 * (size_t)i];
    const int p = pair[{R[0], R[1]}], s = slot[R[0]];
    int &cell = tab[off[0] + (size_t)p * t.ext[2] + (R[2] - t.lo[2])];
    if (cell >= 0) return false;
    cell = i;
    tab[off[1] + (size_t)s * t.ext[1] + (R[1] - t.lo[1])] = p;
    tab[off[2] + (R[0] - t.lo[0])] = s;
  }
  return true;
}

}  // namespace


static int read_err(ephg_handle *h, int *word) {
  CK(cudaMemcpyAsync(word, h->err, sizeof(int), cudaMemcpyDeviceToHost, h->st));
  CK(cudaStreamSynchronize(h->st));
  CK(cudaMemsetAsync(h->err, 0, sizeof(int), h->st));
  return EPHG_OK;
}

int ephg::api_check_err(ephg_handle *h) {
  int w = 0;
  int rc = read_err(h, &w);
  if (rc) return rc;
  if (w & DERR_NEG_PHONON) return fail(EPHG_ERR_NEG_PHONON, "Large negative phonon energy found!");
  if (w & DERR_EIG) return fail(EPHG_ERR_EIG, "Jacobi eigensolver did not converge");
  if (w & DERR_INDEX) return fail(EPHG_ERR_INDEX, "device index check failed");
  if (w & DERR_TIMEOUT) return fail(EPHG_ERR_TIMEOUT, "bounded device wait gave up");
  return EPHG_OK;
}

// workspace failures carry their own message
#define WSFAIL(rc) fail((rc), "%s", h->ws.msg.c_str())

// Small host arrays (tables built on the host, caller arrays of a few MB) reach
// the device through one pinned staging buffer of the library instead of the
// driver's staging of pageable memory, whose occasional page pinning cost
// handle creation ~15 ms every few calls.  Arrays above kStageMax are copied
// directly (the caller's pinned arrays stay asynchronous).
constexpr size_t kStageMax = (size_t)64 << 20;
static int staged_copy(void *dst, const void *src, size_t bytes, cudaStream_t st) {
  static std::mutex mu;
  static void *stage = nullptr;
  static size_t cap = 0;
  std::lock_guard<std::mutex> lk(mu);
  if (cap < bytes) {
    if (stage) cudaFreeHost(stage);
    stage = nullptr;
    cap = 0;
    size_t want = std::max<size_t>(bytes, (size_t)8 << 20);
    if (cudaMallocHost(&stage, want) != cudaSuccess) {
      cudaGetLastError();
      stage = nullptr;
      CK(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));   // no pinned memory: the plain path
      return EPHG_OK;
    }
    cap = want;
  }
  memcpy(stage, src, bytes);
  CK(cudaMemcpyAsync(dst, stage, bytes, cudaMemcpyHostToDevice, st));
  CK(cudaStreamSynchronize(st));   // the staging buffer is free again for the next copy
  return EPHG_OK;
}

template <typename T>
// n elements from the library pool on st, copied from src; the bytes are added to *acc
static int upload(T **dst, const T *src, size_t n, cudaStream_t st, int64_t *acc = nullptr) {
  const size_t b = std::max<size_t>(n, 1) * sizeof(T);
  CK(pool_alloc((void **)dst, b, st));
  if (acc) *acc += (int64_t)b;
  if (n && n * sizeof(T) <= kStageMax) return staged_copy(*dst, src, n * sizeof(T), st);
  if (n) CK(cudaMemcpyAsync(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice, st));
  return EPHG_OK;
}

extern "C" {

const char *ephg_last_error(void) { return g_err.c_str(); }

int ephg_device_count(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

int ephg_trim_memory(void) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(EPHG_ERR_CUDA, "trim_memory: no device");
  cudaMemPool_t pool = lib_pool(dev);
  if (!pool) return fail(EPHG_ERR_CUDA, "trim_memory: no memory pool");
  CK(cudaDeviceSynchronize());   // frees still queued on streams reach the pool first
  CK(cudaMemPoolTrimTo(pool, 0));
  return EPHG_OK;
}

int ephg_destroy(ephg_handle *h) {
  if (!h) return EPHG_OK;
  void *ptrs[] = {h->Rk, h->Rq, h->Rg, h->degk, h->degq, h->degg, h->Hext, h->Hbox, h->Dbox, h->graw, h->G64,
                  h->masses, h->Dcell, h->RD, h->err, h->kposk, h->kposq, h->polar_G, h->polar_Gcell,
                  h->polar_born, h->polar_tau, h->polar_Da, h->polar_Gf, h->cellk_tab, h->cellq_tab, h->rdegk, h->exp_H, h->exp_G, h->exp_raw, h->exp_D};
  // stream-ordered frees back to the library pool, which keeps the memory
  // mapped for the next handle
  for (void *p : ptrs)
    if (p) cudaFreeAsync(p, h->st);
  h->ws.release();
  tc::free_split(h->split, h->st);
  cudaStreamSynchronize(h->st);
  if (h->st) cudaStreamDestroy(h->st);
  delete h;
  return EPHG_OK;
}

int ephg_create(const ephg_wannier_desc *d, ephg_handle **out) {
  if (!d || !out) return fail(EPHG_ERR_ARG, "null argument");
  *out = nullptr;
  if (ephg_device_count() <= 0) return fail(EPHG_ERR_CUDA, "no CUDA device visible");
  if (d->numwannbands < 1 || d->numwannbands > 32)
    return fail(EPHG_ERR_ARG, "numwannbands must be in [1, 32]");
  if (d->numbranches != 3 * d->numatoms || d->numbranches > 32)
    return fail(EPHG_ERR_ARG, "numbranches must be 3*numatoms <= 32");
  if (d->nwsg != d->nwsq)
    return fail(EPHG_ERR_ARG, "nwsg must equal nwsq (the vertex Fourier uses rcells_q, wannier.f90:947)");
  for (int64_t i = 0; i < 3 * d->nwsq; ++i)
    if (d->rcells_g[i] != d->rcells_q[i])
      return fail(EPHG_ERR_ARG, "rcells_g must equal rcells_q (wannier.f90:947-951,988-990)");
  for (int64_t i = 0; i < d->nwsq; ++i)
    if (d->gwsdeg[i] != d->phwsdeg[i]) return fail(EPHG_ERR_ARG, "gwsdeg must equal phwsdeg");
  for (int i = 0; i < 3; ++i)
    if (d->coarse_qmesh[i] <= 0) return fail(EPHG_ERR_ARG, "Bad input(s) in wannier.");
  ephg_handle *h = new ephg_handle();
  int rc = EPHG_OK;
  auto bail = [&](int r) {
    ephg_destroy(h);
    return r;
  };
  if (cudaGetDevice(&h->device) != cudaSuccess) return bail(fail(EPHG_ERR_CUDA, "cudaGetDevice"));
  if (cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking) != cudaSuccess)
    return bail(fail(EPHG_ERR_CUDA, "cudaStreamCreate"));
  h->ws.st = h->st;
  h->nw = (int)d->numwannbands;
  h->nb = (int)d->numbranches;
  h->nwsk = (int)d->nwsk;
  h->nwsq = (int)d->nwsq;
  h->nwsg = (int)d->nwsg;
  h->nat = (int)d->numatoms;
  for (int i = 0; i < 3; ++i) h->cq[i] = (int)d->coarse_qmesh[i];
  for (int i = 0; i < 9; ++i) h->lattvecs[i] = d->lattvecs[i];
  h->masses_h.assign(d->masses, d->masses + h->nat);
  h->basis_h.assign(d->basis, d->basis + 3 * h->nat);
  const int nw = h->nw, nb = h->nb, nwsk = h->nwsk, nwsq = h->nwsq;
  h->Nn = (int64_t)nw * nw * nb * nwsq;
  // R lists as (n,3) int rows and degeneracies as doubles
  auto rows = [](const int64_t *r, int n) {
    std::vector<int> v(3 * (size_t)n);
    for (int i = 0; i < n; ++i)
      for (int c = 0; c < 3; ++c) v[3 * i + c] = (int)r[i + (int64_t)n * c];
    return v;
  };
  std::vector<int> rk = rows(d->rcells_k, nwsk), rq = rows(d->rcells_q, nwsq), rg = rows(d->rcells_g, nwsq);
  std::vector<double> dk(d->elwsdeg, d->elwsdeg + nwsk), dq(d->phwsdeg, d->phwsdeg + nwsq),
      dg(d->gwsdeg, d->gwsdeg + nwsq);
  if ((rc = upload(&h->Rk, rk.data(), rk.size(), h->st, &h->resident_bytes)) || (rc = upload(&h->Rq, rq.data(), rq.size(), h->st, &h->resident_bytes)) ||
      (rc = upload(&h->Rg, rg.data(), rg.size(), h->st, &h->resident_bytes)) || (rc = upload(&h->degk, dk.data(), dk.size(), h->st, &h->resident_bytes)) ||
      (rc = upload(&h->degq, dq.data(), dq.size(), h->st, &h->resident_bytes)) || (rc = upload(&h->degg, dg.data(), dg.size(), h->st, &h->resident_bytes)) ||
      (rc = upload(&h->masses, d->masses, (size_t)h->nat, h->st, &h->resident_bytes)))
    return bail(rc);
  for (int c = 0; c < 3; ++c) {   // range of the Rp coordinates
    int lo = nwsq > 0 ? rq[c] : 0, hi = lo;
    for (int r = 0; r < nwsq; ++r) {
      lo = std::min(lo, rq[3 * r + c]);
      hi = std::max(hi, rq[3 * r + c]);
    }
    h->qlo[c] = lo;
    h->qext[c] = hi - lo + 1;
  }
  {   // the cells of the two Fourier sums of g
    auto cells = [&](const std::vector<int> &r, int n, CellTab &t, int **dev) -> int {
      std::vector<int> tab;
      size_t off[3];
      if (!cell_tables(r, n, t, tab, off)) return EPHG_OK;
      const int e = upload(dev, tab.data(), tab.size(), h->st, &h->resident_bytes);
      if (e) return e;
      t.tab1 = *dev + off[0];
      t.tab2 = *dev + off[1];
      t.tab3 = *dev + off[2];
      t.ok = true;
      return EPHG_OK;
    };
    std::vector<double> rd(nwsk);
    for (int r = 0; r < nwsk; ++r) rd[r] = 1.0 / dk[r];
    if ((rc = cells(rk, nwsk, h->cellk, &h->cellk_tab)) || (rc = cells(rq, nwsq, h->cellq, &h->cellq_tab)) ||
        (rc = upload(&h->rdegk, rd.data(), rd.size(), h->st, &h->resident_bytes)))
      return bail(rc);
  }
  // H(Re) with the velocity companions i*rcart*H (wannier.f90:466-478)
  {
    const size_t nn = (size_t)nw * nw;
    std::vector<double2> hx((size_t)nwsk * 4 * nn);
    for (int r = 0; r < nwsk; ++r) {
      double R[3] = {(double)rk[3 * r], (double)rk[3 * r + 1], (double)rk[3 * r + 2]}, rc3[3];
      for (int i = 0; i < 3; ++i)
        rc3[i] = h->lattvecs[i] * R[0] + h->lattvecs[i + 3] * R[1] + h->lattvecs[i + 6] * R[2];
      for (size_t e = 0; e < nn; ++e) {
        size_t ib = e % nw, jb = e / nw;
        const double *src = d->Hwann + 2 * (r + (size_t)nwsk * (ib + (size_t)nw * jb));
        double2 v = make_double2(src[0], src[1]);
        hx[(size_t)r * 4 * nn + e] = v;
        for (int p = 0; p < 3; ++p)
          hx[(size_t)r * 4 * nn + (1 + p) * nn + e] = make_double2(-rc3[p] * v.y, rc3[p] * v.x);
      }
    }
    if ((rc = upload(&h->Hext, hx.data(), hx.size(), h->st, &h->resident_bytes))) return bail(rc);
    // H(Re) / deg(Re) on the box of Re coordinates, for the mesh Fourier sums
    int hi[3];
    for (int c = 0; c < 3; ++c) {
      h->hlo[c] = hi[c] = nwsk > 0 ? rk[c] : 0;
      for (int r = 0; r < nwsk; ++r) {
        h->hlo[c] = std::min(h->hlo[c], rk[3 * r + c]);
        hi[c] = std::max(hi[c], rk[3 * r + c]);
      }
      h->hext[c] = hi[c] - h->hlo[c] + 1;
    }
    const size_t nbox = (size_t)h->hext[0] * h->hext[1] * h->hext[2];
    if (nbox > ((size_t)1 << 22)) return bail(fail(EPHG_ERR_ARG, "Re cells span too large a box"));
    std::vector<double2> hb(nbox * nn, make_double2(0.0, 0.0));
    for (int r = 0; r < nwsk; ++r) {
      const size_t cell = ((size_t)(rk[3 * r] - h->hlo[0]) * h->hext[1] + (rk[3 * r + 1] - h->hlo[1])) * h->hext[2] +
                          (rk[3 * r + 2] - h->hlo[2]);
      for (size_t e = 0; e < nn; ++e) {
        const double2 v = hx[(size_t)r * 4 * nn + e];
        hb[cell * nn + e] = make_double2(v.x / dk[r], v.y / dk[r]);
      }
    }
    if ((rc = upload(&h->Hbox, hb.data(), hb.size(), h->st, &h->resident_bytes))) return bail(rc);
  }
  // g(Re,Rp): raw epmatwp order and the stage-A layout
  {
    size_t n = (size_t)nw * nw * nwsk * nb * nwsq;
    if ((rc = upload(&h->graw, (const double2 *)d->gwann, n, h->st, &h->resident_bytes))) return bail(rc);
    if (pool_alloc((void **)&h->G64, n * sizeof(double2), h->st) != cudaSuccess)
      return bail(fail(EPHG_ERR_NOMEM, "device allocation of g(Re,Rp), %zu bytes", n * 16));
    h->resident_bytes += (int64_t)(n * sizeof(double2));
    launch_permute_gwann(nw, nb, nwsk, nwsq, h->graw, h->G64, h->st);
  }
  // Phonon terms.  D(q) is one Fourier sum per element over the wrapped vectors R':
  // X_ab(R') = massnorm_ab sum of D(iuc)_ab / (deg nwrap) over the (pair(a, b), iuc) whose
  // shortest wraps include R', and its q derivatives the sums of i rcart(iuc) times the
  // same terms.  On a mesh X runs on the box of R' (launch_mesh_fourier), at arbitrary
  // q the distinct R' are the cells of one product (ph_wann).
  {
    const int nat = h->nat, ne = nb * nb;
    struct Wrap {
      int r[3];
      double rden;
    };
    std::vector<Wrap> wraps;
    std::vector<int> woff(1, 0);   // wraps of entry (pair = iat + nat jat, iuc), in that order
    for (int jat = 0; jat < nat; ++jat)
      for (int iat = 0; iat < nat; ++iat)
        for (int iuc = 0; iuc < nwsq; ++iuc) {
          double dist[3];
          for (int c = 0; c < 3; ++c)
            dist[c] = ((double)rq[3 * iuc + c] - d->basis[c + 3 * iat] + d->basis[c + 3 * jat]) / (double)h->cq[c];
          const std::vector<int> w = ws_wrap(h->lattvecs, dist, 1.0e-6);
          const int nwrap = (int)w.size() / 3;
          for (int iw = 0; iw < nwrap; ++iw) {
            Wrap x;
            for (int c = 0; c < 3; ++c) x.r[c] = rq[3 * iuc + c] + w[3 * iw + c] * h->cq[c];
            x.rden = 1.0 / (double)(d->phwsdeg[iuc] * nwrap);
            wraps.push_back(x);
          }
          woff.push_back((int)wraps.size());
        }
    for (int c = 0; c < 3; ++c) {
      int lo = wraps.empty() ? 0 : wraps[0].r[c], hi = lo;
      for (const Wrap &x : wraps) {
        lo = std::min(lo, x.r[c]);
        hi = std::max(hi, x.r[c]);
      }
      h->dlo[c] = lo;
      h->dext[c] = hi - lo + 1;
    }
    const size_t nbox = (size_t)h->dext[0] * h->dext[1] * h->dext[2];
    if (nbox > ((size_t)1 << 22)) return bail(fail(EPHG_ERR_ARG, "phonon cells span too large a box"));
    auto box = [&](const Wrap &x) {
      return ((size_t)(x.r[0] - h->dlo[0]) * h->dext[1] + (x.r[1] - h->dlo[1])) * h->dext[2] + (x.r[2] - h->dlo[2]);
    };
    std::vector<int> slot(nbox, -1), cells;   // distinct R', in box order
    for (const Wrap &x : wraps) slot[box(x)] = 0;
    for (size_t b = 0; b < nbox; ++b)
      if (slot[b] == 0) {
        slot[b] = h->nD++;
        cells.insert(cells.end(), {(int)(b / ((size_t)h->dext[1] * h->dext[2])) + h->dlo[0],
                                   (int)(b / h->dext[2] % h->dext[1]) + h->dlo[1], (int)(b % h->dext[2]) + h->dlo[2]});
      }
    std::vector<double2> xb(nbox * ne, make_double2(0.0, 0.0)), xc((size_t)h->nD * 4 * ne, make_double2(0.0, 0.0));
    const double2 *Dw = (const double2 *)d->Dphwann;
    for (int e = 0; e < ne; ++e) {
      const int a = e % nb, b = e / nb;
      const int pair = (a / 3) + nat * (b / 3);
      const double massnorm = 1.0 / std::sqrt(d->masses[a / 3] * d->masses[b / 3]) * Ryd2amu;
      for (int iuc = 0; iuc < nwsq; ++iuc) {
        const int en = pair * nwsq + iuc;
        const double2 dv = Dw[iuc + (size_t)nwsq * (a + (size_t)nb * b)];
        double rc3[3];
        for (int i = 0; i < 3; ++i)
          rc3[i] = h->lattvecs[i] * rq[3 * iuc] + h->lattvecs[i + 3] * rq[3 * iuc + 1] + h->lattvecs[i + 6] * rq[3 * iuc + 2];
        for (int wv = woff[en]; wv < woff[en + 1]; ++wv) {
          const double f = wraps[wv].rden * massnorm;
          const double2 t = make_double2(f * dv.x, f * dv.y);
          const size_t at = box(wraps[wv]);
          double2 *x = &xb[at * ne + e], *y = &xc[(size_t)slot[at] * 4 * ne + e];
          x->x += t.x;
          x->y += t.y;
          y->x += t.x;
          y->y += t.y;
          for (int i = 0; i < 3; ++i) {
            y[(1 + i) * ne].x -= rc3[i] * t.y;
            y[(1 + i) * ne].y += rc3[i] * t.x;
          }
        }
      }
    }
    if ((rc = upload(&h->Dbox, xb.data(), xb.size(), h->st, &h->resident_bytes)) ||
        (rc = upload(&h->Dcell, xc.data(), xc.size(), h->st, &h->resident_bytes)) ||
        (rc = upload(&h->RD, cells.data(), cells.size(), h->st, &h->resident_bytes)))
      return bail(rc);
  }
  // contraction order of the split form: cells by decreasing |R| (ties by index),
  // so that the decaying Wannier-space terms are summed smallest first
  {
    auto order = [&](const std::vector<int> &r, int n) {
      std::vector<double> len(n);
      for (int i = 0; i < n; ++i) {
        double c[3];
        for (int d = 0; d < 3; ++d)
          c[d] = h->lattvecs[d] * r[3 * i] + h->lattvecs[d + 3] * r[3 * i + 1] + h->lattvecs[d + 6] * r[3 * i + 2];
        len[i] = std::sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
      }
      std::vector<int> idx(n), pos(n);
      for (int i = 0; i < n; ++i) idx[i] = i;
      std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return len[a] > len[b]; });
      for (int p = 0; p < n; ++p) pos[idx[p]] = p;
      return pos;
    };
    std::vector<int> pk = order(rk, nwsk), pq = order(rq, nwsq);
    if ((rc = upload(&h->kposk, pk.data(), pk.size(), h->st, &h->resident_bytes)) || (rc = upload(&h->kposq, pq.data(), pq.size(), h->st, &h->resident_bytes)))
      return bail(rc);
  }
  // column exponents of the operands that launch_xgemm multiplies by: part of the resident data, so
  // that no request allocates beside its workspace (four bytes a column; one pass over each operand)
  {
    const struct {
      int **e;
      int64_t n;
      int K;
      const double2 *B;
    } ops[] = {{&h->exp_H, 4 * (int64_t)nw * nw, nwsk, h->Hext},
               {&h->exp_G, h->Nn, nwsk, h->G64},
               {&h->exp_raw, (int64_t)nw * nw * nb * nwsk, nwsq, h->graw},
               {&h->exp_D, 4 * (int64_t)nb * nb, h->nD, h->Dcell}};
    for (const auto &o : ops) {
      if (o.n <= 0) continue;
      if (pool_alloc((void **)o.e, (size_t)o.n * sizeof(int), h->st) != cudaSuccess)
        return bail(fail(EPHG_ERR_NOMEM, "device allocation of column exponents, %lld bytes", (long long)(4 * o.n)));
      h->resident_bytes += o.n * (int64_t)sizeof(int);
      launch_colexp(o.n, o.K, o.B, *o.e, h->st);
    }
  }
  if (pool_alloc((void **)&h->err, sizeof(int), h->st) != cudaSuccess)
    return bail(fail(EPHG_ERR_CUDA, "device allocation of the error word"));
  if (cudaMemsetAsync(h->err, 0, sizeof(int), h->st) != cudaSuccess) return bail(fail(EPHG_ERR_CUDA, "memset"));
  if (cudaStreamSynchronize(h->st) != cudaSuccess || cudaGetLastError() != cudaSuccess)
    return bail(fail(EPHG_ERR_CUDA, "create: %s", cudaGetErrorString(cudaGetLastError())));
  *out = h;
  return EPHG_OK;
}

// ------------------------------------------------------------- polar
// The crystal fields of a polar crystal (crys%polar, epsilon, born;
// crystal.f90:45-49) and what the long-range terms derive from them:
// reciprocal vectors and volume (crystal.f90:282-293), the Cartesian basis in
// bohr, the box of reciprocal-lattice vectors and the q-independent part of
// dyn_nonanalytic (wannier.f90:843-867), formed once.
int ephg_set_polar(ephg_handle *h, const double *epsilon, const double *born) {
  if (!h) return fail(EPHG_ERR_ARG, "set_polar: bad arguments");
  if (epsilon && !born) return fail(EPHG_ERR_ARG, "set_polar: born effective charges are required");
  for (void *p : {(void *)h->polar_G, (void *)h->polar_Gcell, (void *)h->polar_born, (void *)h->polar_tau,
                  (void *)h->polar_Da, (void *)h->polar_Gf})
    if (p) cudaFreeAsync(p, h->st);
  CK(cudaStreamSynchronize(h->st));
  h->polar_G = h->polar_Gcell = h->polar_born = h->polar_tau = nullptr;
  h->polar_Da = nullptr;
  h->polar_Gf = nullptr;
  h->polar_on = false;
  if (!epsilon) return EPHG_OK;   // non-polar
  const double bohr2nm = 0.052917721092, pi = 4.0 * atan(1.0), twopi = 2.0 * pi;   // params.f90
  const int nat = h->nat, nb = h->nb;
  const double *a = h->lattvecs;
  ephg::PolarDev P;
  for (int i = 0; i < 3; ++i) {
    const int j = (i + 1) % 3, k = (j + 1) % 3;
    P.rec[0 + 3 * i] = a[1 + 3 * j] * a[2 + 3 * k] - a[2 + 3 * j] * a[1 + 3 * k];
    P.rec[1 + 3 * i] = a[2 + 3 * j] * a[0 + 3 * k] - a[0 + 3 * j] * a[2 + 3 * k];
    P.rec[2 + 3 * i] = a[0 + 3 * j] * a[1 + 3 * k] - a[1 + 3 * j] * a[0 + 3 * k];
  }
  const double vol = fabs(a[0] * P.rec[0] + a[1] * P.rec[1] + a[2] * P.rec[2]);
  for (double &r : P.rec) r *= twopi / vol;
  const double a1 = sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
  const double tpiba = twopi / a1 * bohr2nm;
  P.alph = tpiba * tpiba;
  P.gmax = 14.0;
  P.fac = 8.0 * pi / (vol / (bohr2nm * bohr2nm * bohr2nm));
  for (int i = 0; i < 9; ++i) P.eps[i] = epsilon[i];
  std::vector<double> G, tau(3 * (size_t)nat);
  for (int m1 = -h->cq[0]; m1 <= h->cq[0]; ++m1)
    for (int m2 = -h->cq[1]; m2 <= h->cq[1]; ++m2)
      for (int m3 = -h->cq[2]; m3 <= h->cq[2]; ++m3)
        for (int d = 0; d < 3; ++d) G.push_back((m1 * P.rec[d] + m2 * P.rec[d + 3] + m3 * P.rec[d + 6]) * bohr2nm);
  for (int at = 0; at < nat; ++at)
    for (int d = 0; d < 3; ++d) {
      const double *b = &h->basis_h[3 * (size_t)at];
      tau[3 * at + d] = (a[d] * b[0] + a[d + 3] * b[1] + a[d + 6] * b[2]) / bohr2nm;
    }
  // The box vectors that can pass the cut qeq < 4 alph gmax for some q of the
  // first cell (the mesh q): qeq >= lmin |G + q|^2 >= lmin (|G| - qmax)^2, with
  // lmin a Gershgorin lower bound of the symmetric part of epsilon and qmax the
  // longest corner of the cell.  Without a positive bound nothing is dropped.
  double lmin = INFINITY, qmax = 0.0;
  for (int i = 0; i < 3; ++i) {
    double off = 0.0;
    for (int j = 0; j < 3; ++j)
      if (j != i) off += fabs(0.5 * (epsilon[i + 3 * j] + epsilon[j + 3 * i]));
    lmin = std::min(lmin, epsilon[i + 3 * i] - off);
  }
  for (int c = 0; c < 8; ++c) {
    double v[3];
    for (int d = 0; d < 3; ++d)
      v[d] = ((c & 1) * P.rec[d] + ((c >> 1) & 1) * P.rec[d + 3] + ((c >> 2) & 1) * P.rec[d + 6]) * bohr2nm;
    qmax = std::max(qmax, sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]));
  }
  std::vector<double> Gc;
  const double rcut = lmin > 0.0 ? sqrt(4.0 * P.alph * P.gmax / lmin) * (1.0 + 1e-9) + qmax : INFINITY;
  for (size_t i = 0; i < G.size(); i += 3) {
    const double n = sqrt(G[i] * G[i] + G[i + 1] * G[i + 1] + G[i + 2] * G[i + 2]);
    if (n < rcut) Gc.insert(Gc.end(), {G[i], G[i + 1], G[i + 2]});
  }
  P.nat = nat;
  P.nb = nb;
  P.M = (int)(G.size() / 3);
  P.Mcell = (int)(Gc.size() / 3);
  P.masses = h->masses;
  int rc;
  std::vector<float> Gf(G.begin(), G.end());
  Gf.insert(Gf.end(), Gc.begin(), Gc.end());
  if ((rc = upload(&h->polar_Gf, Gf.data(), Gf.size(), h->st)) || (rc = upload(&h->polar_G, G.data(), G.size(), h->st)) ||
      (rc = upload(&h->polar_Gcell, Gc.data(), Gc.size(), h->st)) ||
      (rc = upload(&h->polar_born, born, 9 * (size_t)nat, h->st)) ||
      (rc = upload(&h->polar_tau, tau.data(), tau.size(), h->st)))
    return rc;
  CK(pool_alloc((void **)&h->polar_Da, (size_t)nb * nb * sizeof(double2), h->st));
  P.G = h->polar_G;
  P.Gcell = h->polar_Gcell;
  P.Gf = h->polar_Gf;
  P.Gcellf = h->polar_Gf + G.size();
  P.born = h->polar_born;
  P.tau = h->polar_tau;
  launch_polar_da(P, h->polar_Da, h->st);
  CKL();
  CK(cudaStreamSynchronize(h->st));
  P.Da = h->polar_Da;
  h->polar = P;
  h->polar_on = true;
  return EPHG_OK;
}

// ------------------------------------------------------------- symmetry
int ephg_crystal_symmetry(const double *lattvecs, int64_t natoms, const double *basis, const int64_t *atomtypes,
                          double symprec, int64_t maxops, int64_t *nops, int64_t *rotations, double *translations) {
  if (!lattvecs || natoms < 1 || !basis || !atomtypes || !nops || (maxops > 0 && !rotations))
    return fail(EPHG_ERR_ARG, "crystal_symmetry: bad arguments");
  std::vector<ephg::SymOp> ops;
  if (ephg::crystal_symmetry(lattvecs, (int)natoms, basis, atomtypes, symprec, ops))
    return fail(EPHG_ERR_ARG, "crystal_symmetry: no symmetry found (symprec must be > 0)");
  *nops = (int64_t)ops.size();
  if ((int64_t)ops.size() > maxops)
    return fail(EPHG_ERR_ARG, "crystal_symmetry: %lld operations, room for %lld", (long long)ops.size(),
                (long long)maxops);
  for (size_t o = 0; o < ops.size(); ++o) {
    for (int k = 0; k < 9; ++k) rotations[9 * o + k] = ops[o].W[k];
    if (translations)
      for (int d = 0; d < 3; ++d) translations[3 * o + d] = ops[o].t[d];
  }
  return EPHG_OK;
}

int ephg_set_symmetry(ephg_handle *h, int64_t nsymm, const int64_t *rotations) {
  if (!h || nsymm < 0 || (nsymm > 0 && !rotations) || nsymm > 192)
    return fail(EPHG_ERR_ARG, "set_symmetry: bad arguments");
  h->sym_rot.assign(rotations, rotations + 9 * nsymm);
  if (nsymm > 0) {   // every rotation must be a lattice symmetry (an integer reciprocal rotation)
    const int m1[3] = {1, 1, 1};
    std::vector<int> K;
    const char *why = "";
    if (ephg::mesh_qrotations(h->lattvecs, (int)nsymm, rotations, m1, K, &why)) {
      h->sym_rot.clear();
      return fail(EPHG_ERR_ARG, "set_symmetry: %s", why);
    }
  }
  return EPHG_OK;
}

int ephg_irred_wedge(const double *lattvecs, int64_t nsymm, const int64_t *rotations, const int64_t mesh[3],
                     int64_t nk, const int64_t *indexlist, int64_t *nirred, int64_t *indexlist_irred, int64_t *nequiv,
                     int64_t *fbz2ibz) {
  if (!lattvecs || nsymm < 0 || (nsymm > 0 && !rotations) || !mesh || !nirred || !indexlist_irred)
    return fail(EPHG_ERR_ARG, "irred_wedge: bad arguments");
  for (int i = 0; i < 3; ++i)
    if (mesh[i] <= 0 || mesh[i] > 1024) return fail(EPHG_ERR_ARG, "irred_wedge: bad mesh");
  const int m[3] = {(int)mesh[0], (int)mesh[1], (int)mesh[2]};
  const int64_t N = mesh[0] * mesh[1] * mesh[2];
  const int64_t n = indexlist ? nk : N;
  std::vector<int> K;
  const char *why = "";
  if (nsymm > 0 && ephg::mesh_qrotations(lattvecs, (int)nsymm, rotations, m, K, &why))
    return fail(EPHG_ERR_ARG, "irred_wedge: %s", why);
  const int nops = (int)(K.size() / 9);
  // points of the list by muxed index (0-based); -1 outside it
  std::vector<int64_t> pos(N, -1);
  for (int64_t i = 0; i < n; ++i) {
    const int64_t p = indexlist ? indexlist[i] - 1 : i;
    if (p < 0 || p >= N) return fail(EPHG_ERR_ARG, "irred_wedge: index out of range");
    if (i > 0 && indexlist && indexlist[i] <= indexlist[i - 1])
      return fail(EPHG_ERR_ARG, "irred_wedge: indexlist must be sorted ascending");
    pos[p] = i;
  }
  // find_irred_wedge (symmetry.f90:303-452): the first point of each orbit, in list order
  std::vector<int64_t> rep(n);
  int64_t nir = 0;
  for (int64_t i = 0; i < n; ++i) {
    const int64_t p = indexlist ? indexlist[i] - 1 : i;
    const int v0 = (int)(p % m[0]), v1 = (int)((p / m[0]) % m[1]), v2 = (int)(p / ((int64_t)m[0] * m[1]));
    int64_t best = p;
    for (int s = 0; s < nops; ++s) {
      const int *k = &K[9 * s];
      const int64_t a = floormod((int64_t)k[0] * v0 + (int64_t)k[3] * v1 + (int64_t)k[6] * v2, m[0]);
      const int64_t b = floormod((int64_t)k[1] * v0 + (int64_t)k[4] * v1 + (int64_t)k[7] * v2, m[1]);
      const int64_t c = floormod((int64_t)k[2] * v0 + (int64_t)k[5] * v1 + (int64_t)k[8] * v2, m[2]);
      const int64_t img = a + m[0] * (b + m[1] * c);
      if (pos[img] < 0) return fail(EPHG_ERR_ARG, "Severe error: Could not find irreducible wedge.");
      best = std::min(best, img);
    }
    rep[i] = pos[best];
  }
  std::vector<int64_t> ibz_of(n, -1);
  for (int64_t i = 0; i < n; ++i)
    if (rep[i] == i) {
      ibz_of[i] = nir;
      indexlist_irred[nir] = indexlist ? indexlist[i] : i + 1;
      if (nequiv) nequiv[nir] = 0;
      ++nir;
    }
  for (int64_t i = 0; i < n; ++i) {
    const int64_t r = ibz_of[rep[i]];
    if (nequiv) nequiv[r]++;
    if (fbz2ibz) fbz2ibz[i] = r + 1;
  }
  *nirred = nir;
  return EPHG_OK;
}

// ------------------------------------------------------------- el_wann
int ephg_el_wann(ephg_handle *h, int64_t nk, const double *kvecs, double *energies,
                 double *velocities, double *evecs, const double *scissor) {
  if (!h || nk < 0 || (nk > 0 && (!kvecs || !energies)))
    return fail(EPHG_ERR_ARG, "el_wann: bad arguments");
  if (velocities && !evecs)
    return fail(EPHG_ERR_ARG, "In el_wann, velocity is present but not eigenvecs.");
  if (nk == 0) return EPHG_OK;
  const int nw = h->nw, nwsk = h->nwsk;
  const size_t nn = (size_t)nw * nw;
  const int with_vel = velocities != nullptr;
  const int ncol = with_vel ? 4 * (int)nn : (int)nn;
  double *kv, *w, *ens, *vel, *sc = nullptr;
  double2 *P, *C, *V, *ev;
  int rc;
  if ((rc = wsget(h->ws, "el_kv", (size_t)nk * 3, &kv)) || (rc = wsget(h->ws, "el_P", (size_t)nk * nwsk, &P)) ||
      (rc = wsget(h->ws, "el_C", (size_t)nk * ncol, &C)) || (rc = wsget(h->ws, "el_w", (size_t)nk * nw, &w)) ||
      (rc = wsget(h->ws, "el_V", (size_t)nk * nn, &V)) || (rc = wsget(h->ws, "el_e", (size_t)nk * nw, &ens)) ||
      (rc = wsget(h->ws, "el_vel", with_vel ? (size_t)nk * nw * 3 : 1, &vel)) ||
      (rc = wsget(h->ws, "el_ev", evecs ? (size_t)nk * nn : 1, &ev)))
    return WSFAIL(rc);
  if (scissor) {
    if ((rc = wsget(h->ws, "el_sc", (size_t)nw, &sc))) return WSFAIL(rc);
    CK(cudaMemcpyAsync(sc, scissor, nw * sizeof(double), cudaMemcpyHostToDevice, h->st));
  }
  CK(cudaMemcpyAsync(kv, kvecs, (size_t)nk * 3 * sizeof(double), cudaMemcpyHostToDevice, h->st));
  launch_phase_cells((int)nk, kv, nk, nullptr, nwsk, h->Rk, h->degk, h->hlo, h->hext, P, nwsk, h->st);
  if ((rc = launch_xgemm(h->ws, (int)nk, ncol, nwsk, P, nwsk, h->Hext, 4 * (int64_t)nn, h->exp_H, C, ncol, h->err, h->st)))
    return WSFAIL(rc);
  launch_heig((int)nk, nw, C, ncol, w, V, h->err, h->st);
  launch_el_post((int)nk, nw, w, V, C, ncol, with_vel, sc, ens, with_vel ? vel : nullptr,
                 evecs ? ev : nullptr, nullptr, h->st);
  h->launches += 5;
  CKL();
  CK(cudaMemcpyAsync(energies, ens, (size_t)nk * nw * sizeof(double), cudaMemcpyDeviceToHost, h->st));
  if (evecs) CK(cudaMemcpyAsync(evecs, ev, (size_t)nk * nn * sizeof(double2), cudaMemcpyDeviceToHost, h->st));
  if (with_vel) CK(cudaMemcpyAsync(velocities, vel, (size_t)nk * nw * 3 * sizeof(double), cudaMemcpyDeviceToHost, h->st));
  return ephg::api_check_err(h);
}

// ------------------------------------------------------------- ph_wann
int ephg_ph_wann(ephg_handle *h, int64_t nq, const double *qvecs, double *energies,
                 double *evecs, double *velocities) {
  if (!h || nq < 0 || (nq > 0 && (!qvecs || !energies)))
    return fail(EPHG_ERR_ARG, "ph_wann: bad arguments");
  if (velocities && !evecs)
    return fail(EPHG_ERR_ARG, "In ph_wann, velocity is present but not eigenvecs.");
  if (nq == 0) return EPHG_OK;
  const int nb = h->nb;
  const size_t nn = (size_t)nb * nb;
  const int with_vel = velocities != nullptr;
  const int ncol = (with_vel ? 4 : 1) * (int)nn;   // D(q), then its three derivatives
  const int64_t qb = std::max<int64_t>(1, std::min<int64_t>(nq, ((int64_t)1 << 28) / (16 * std::max(1, h->nD))));
  double *qv, *w, *ens, *vel;
  double2 *P, *Dq, *V, *ev;
  int rc;
  if ((rc = wsget(h->ws, "ph_qv", (size_t)nq * 3, &qv)) || (rc = wsget(h->ws, "ph_D", (size_t)nq * ncol, &Dq)) ||
      (rc = wsget(h->ws, "ph_P", (size_t)qb * h->nD, &P)) ||
      (rc = wsget(h->ws, "ph_w", (size_t)nq * nb, &w)) || (rc = wsget(h->ws, "ph_V", (size_t)nq * nn, &V)) ||
      (rc = wsget(h->ws, "ph_e", (size_t)nq * nb, &ens)) ||
      (rc = wsget(h->ws, "ph_vel", with_vel ? (size_t)nq * nb * 3 : 1, &vel)) ||
      (rc = wsget(h->ws, "ph_ev", evecs ? (size_t)nq * nn : 1, &ev)))
    return WSFAIL(rc);
  CK(cudaMemcpyAsync(qv, qvecs, (size_t)nq * 3 * sizeof(double), cudaMemcpyHostToDevice, h->st));
  for (int64_t q0 = 0; q0 < nq; q0 += qb) {
    const int n = (int)std::min(qb, nq - q0);
    launch_phase_cells(n, qv + q0, nq, nullptr, h->nD, h->RD, nullptr, h->dlo, h->dext, P, h->nD, h->st);
    if ((rc = launch_xgemm(h->ws, n, ncol, h->nD, P, h->nD, h->Dcell, 4 * (int64_t)nn, h->exp_D, Dq + q0 * ncol, ncol,
                           h->err, h->st)))
      return WSFAIL(rc);
    h->launches += 3;
  }
  double2 *dDq = Dq + nn;
  if (h->polar_on)   // non-analytic correction (wannier.f90:684-705)
    launch_polar_q(h->polar, (int)nq, nullptr, nullptr, qv, Dq, with_vel ? dDq : nullptr, ncol, nullptr, h->st);
  launch_heig((int)nq, nb, Dq, ncol, w, V, h->err, h->st);
  launch_ph_post((int)nq, nb, nullptr, qv, w, V, dDq, ncol, with_vel, h->masses, ens,
                 evecs ? ev : nullptr, with_vel ? vel : nullptr, nullptr, nullptr, nullptr, h->err,
                 h->st);
  h->launches += 3;
  CKL();
  CK(cudaMemcpyAsync(energies, ens, (size_t)nq * nb * sizeof(double), cudaMemcpyDeviceToHost, h->st));
  if (evecs) CK(cudaMemcpyAsync(evecs, ev, (size_t)nq * nn * sizeof(double2), cudaMemcpyDeviceToHost, h->st));
  if (with_vel) CK(cudaMemcpyAsync(velocities, vel, (size_t)nq * nb * 3 * sizeof(double), cudaMemcpyDeviceToHost, h->st));
  return ephg::api_check_err(h);
}

// ---------------------------------------------------------------- gkRp
int ephg_gkRp(ephg_handle *h, int64_t nk, const double *kvecs, double *gmixed) {
  if (!h || nk < 0 || (nk > 0 && (!kvecs || !gmixed))) return fail(EPHG_ERR_ARG, "gkRp: bad arguments");
  if (nk == 0) return EPHG_OK;
  const int nwsk = h->nwsk;
  const int64_t chunk = std::max<int64_t>(1, std::min<int64_t>(nk, (int64_t)(1u << 30) / (h->Nn * 16)));
  double *kv;
  double2 *P, *C;
  int rc;
  if ((rc = wsget(h->ws, "gk_kv", (size_t)chunk * 3, &kv)) || (rc = wsget(h->ws, "gk_P", (size_t)chunk * nwsk, &P)) ||
      (rc = wsget(h->ws, "gk_C", (size_t)chunk * h->Nn, &C)))
    return WSFAIL(rc);
  std::vector<double> kc((size_t)chunk * 3);
  for (int64_t k0 = 0; k0 < nk; k0 += chunk) {
    int64_t n = std::min(chunk, nk - k0);
    for (int c = 0; c < 3; ++c)
      for (int64_t i = 0; i < n; ++i) kc[i + n * c] = kvecs[(k0 + i) + nk * c];
    CK(cudaMemcpyAsync(kv, kc.data(), (size_t)n * 3 * sizeof(double), cudaMemcpyHostToDevice, h->st));
    launch_phase_cells((int)n, kv, n, nullptr, nwsk, h->Rk, h->degk, h->hlo, h->hext, P, nwsk, h->st);
    if ((rc = launch_xgemm(h->ws, (int)n, h->Nn, nwsk, P, nwsk, h->G64, h->Nn, h->exp_G, C, h->Nn, h->err, h->st)))
      return WSFAIL(rc);
    h->launches += 3;
    CKL();
    CK(cudaMemcpyAsync(gmixed + 2 * k0 * h->Nn, C, (size_t)n * h->Nn * sizeof(double2),
                       cudaMemcpyDeviceToHost, h->st));
    CK(cudaStreamSynchronize(h->st));
  }
  return ephg::api_check_err(h);
}

// ---------------------------------------------------------------- gReq
int ephg_gReq(ephg_handle *h, int64_t nq, const double *qvecs, double *gmixed) {
  if (!h || nq < 0 || (nq > 0 && (!qvecs || !gmixed))) return fail(EPHG_ERR_ARG, "gReq: bad arguments");
  if (nq == 0) return EPHG_OK;
  const int nw = h->nw, nb = h->nb, nwsk = h->nwsk, nwsg = h->nwsg;
  const int64_t per = (int64_t)nw * nw * nb * nwsk;
  const int64_t chunk = std::max<int64_t>(1, std::min<int64_t>(nq, (int64_t)(1u << 30) / (per * 16)));
  double *qv;
  double2 *P, *C, *O;
  int rc;
  if ((rc = wsget(h->ws, "gq_qv", (size_t)chunk * 3, &qv)) || (rc = wsget(h->ws, "gq_P", (size_t)chunk * nwsg, &P)) ||
      (rc = wsget(h->ws, "gq_C", (size_t)chunk * per, &C)) || (rc = wsget(h->ws, "gq_O", (size_t)chunk * per, &O)))
    return WSFAIL(rc);
  std::vector<double> qc((size_t)chunk * 3);
  for (int64_t q0 = 0; q0 < nq; q0 += chunk) {
    int64_t n = std::min(chunk, nq - q0);
    for (int c = 0; c < 3; ++c)
      for (int64_t i = 0; i < n; ++i) qc[i + n * c] = qvecs[(q0 + i) + nq * c];
    CK(cudaMemcpyAsync(qv, qc.data(), (size_t)n * 3 * sizeof(double), cudaMemcpyHostToDevice, h->st));
    // sum_Rp e^{2 pi i q.Rp}/gwsdeg * g(i,j,Re,s,Rp): rows of the raw array are Rp
    launch_phase_cells((int)n, qv, n, nullptr, nwsg, h->Rg, h->degg, h->qlo, h->qext, P, nwsg, h->st);
    if ((rc = launch_xgemm(h->ws, (int)n, per, nwsg, P, nwsg, h->graw, per, h->exp_raw, C, per, h->err, h->st)))
      return WSFAIL(rc);
    launch_permute_greq((int)n, nw, nb, nwsk, C, O, h->st);
    h->launches += 4;
    CKL();
    CK(cudaMemcpyAsync(gmixed + 2 * q0 * per, O, (size_t)n * per * sizeof(double2),
                       cudaMemcpyDeviceToHost, h->st));
    CK(cudaStreamSynchronize(h->st));
  }
  return ephg::api_check_err(h);
}

// ------------------------------------------------------------------ g2
int ephg_g2(ephg_handle *h, int64_t wannspace, int64_t nv, const double *kvecs,
            const double *qvecs, const double *el_evec_k, const double *el_evec_kp,
            const double *ph_evec_q, const double *ph_en, int64_t ngm, const double *gmixed,
            const int64_t *gm_index, double *g2_out) {
  if (!h || nv < 0) return fail(EPHG_ERR_ARG, "g2: bad arguments");
  if (wannspace != EPHG_WANNSPACE_EL && wannspace != EPHG_WANNSPACE_PH)
    return fail(EPHG_ERR_ARG, "Invalid value of wannspace in call to g2_epw. Exiting.");
  if (nv == 0) return EPHG_OK;
  for (int64_t v = 0; v < nv; ++v)
    if (gm_index[v] < 1 || gm_index[v] > ngm) return fail(EPHG_ERR_ARG, "g2: gm_index out of range");
  const int nw = h->nw, nb = h->nb;
  const int nws = wannspace == EPHG_WANNSPACE_PH ? h->nwsg : h->nwsk;
  const int64_t per = (int64_t)nw * nw * nb, gstride = per * nws;
  // vertices grouped by their block, as chunks of rows that share one; pieces of whole
  // chunks whose phases, cell sums and digits fit bounded buffers
  std::vector<int64_t> at(ngm + 1, 0);
  for (int64_t v = 0; v < nv; ++v) at[gm_index[v]]++;
  for (int64_t b = 0; b < ngm; ++b) at[b + 1] += at[b];
  std::vector<int> perm(nv);
  for (int64_t v = 0; v < nv; ++v) perm[at[gm_index[v] - 1]++] = (int)v;
  std::vector<int4> chunks;
  int most = 1;   // rows of the longest chunk
  for (int64_t r = 0; r < nv;) {
    const int64_t b = gm_index[perm[r]];
    int64_t e = r + 1;
    while (e < nv && e - r < XG_CHUNK && gm_index[perm[e]] == b) ++e;
    chunks.push_back(make_int4((int)r, (int)(e - r), (int)(b - 1), 0));
    most = std::max(most, (int)(e - r));
    r = e;
  }
  // rows of a piece: phases (nws values) and cell sums (per); chunks: digits
  const int64_t bound = (int64_t)1 << 28;
  const int64_t row_most = bound / (16 * std::max<int64_t>(per, nws));
  const int64_t chunk_most = std::min<int64_t>(XG_MAXCHUNKS, bound / xgemm_chunk_bytes(most, nws));
  std::vector<std::pair<int64_t, int64_t>> piece;   // first row, first chunk
  int64_t rows = 0;
  for (size_t c = 0; c < chunks.size(); ++c) {
    const int64_t r = chunks[c].x, e = r + chunks[c].y;
    if (piece.empty() || e - piece.back().first > row_most || (int64_t)c - piece.back().second >= chunk_most)
      piece.push_back({r, (int64_t)c});
    chunks[c].x = (int)(r - piece.back().first);
    rows = std::max(rows, e - piece.back().first);
  }
  piece.push_back({nv, (int64_t)chunks.size()});
  double *qv, *en, *out;
  double2 *ek, *ekp, *eq, *gm, *P, *G;
  int *pd;
  int4 *cd;
  int rc;
  if ((rc = wsget(h->ws, "g2_qv", (size_t)nv * 3, &qv)) || (rc = wsget(h->ws, "g2_en", (size_t)nv, &en)) ||
      (rc = wsget(h->ws, "g2_out", (size_t)nv, &out)) || (rc = wsget(h->ws, "g2_ek", (size_t)nv * nw, &ek)) ||
      (rc = wsget(h->ws, "g2_ekp", (size_t)nv * nw, &ekp)) || (rc = wsget(h->ws, "g2_eq", (size_t)nv * nb, &eq)) ||
      (rc = wsget(h->ws, "g2_gm", (size_t)ngm * gstride, &gm)) || (rc = wsget(h->ws, "g2_perm", (size_t)nv, &pd)) ||
      (rc = wsget(h->ws, "g2_chunks", chunks.size(), &cd)) || (rc = wsget(h->ws, "g2_P", (size_t)(rows * nws), &P)) ||
      (rc = wsget(h->ws, "g2_G", (size_t)(rows * per), &G)))
    return WSFAIL(rc);
  const double *kq = wannspace == EPHG_WANNSPACE_PH ? qvecs : kvecs;
  CK(cudaMemcpyAsync(gm, gmixed, (size_t)ngm * gstride * sizeof(double2), cudaMemcpyHostToDevice, h->st));
  CK(cudaMemcpyAsync(qv, kq, (size_t)nv * 3 * sizeof(double), cudaMemcpyHostToDevice, h->st));
  CK(cudaMemcpyAsync(en, ph_en, (size_t)nv * sizeof(double), cudaMemcpyHostToDevice, h->st));
  CK(cudaMemcpyAsync(ek, el_evec_k, (size_t)nv * nw * sizeof(double2), cudaMemcpyHostToDevice, h->st));
  CK(cudaMemcpyAsync(ekp, el_evec_kp, (size_t)nv * nw * sizeof(double2), cudaMemcpyHostToDevice, h->st));
  CK(cudaMemcpyAsync(eq, ph_evec_q, (size_t)nv * nb * sizeof(double2), cudaMemcpyHostToDevice, h->st));
  CK(cudaMemcpyAsync(pd, perm.data(), (size_t)nv * sizeof(int), cudaMemcpyHostToDevice, h->st));
  CK(cudaMemcpyAsync(cd, chunks.data(), chunks.size() * sizeof(int4), cudaMemcpyHostToDevice, h->st));
  const int *R = wannspace == EPHG_WANNSPACE_PH ? h->Rq : h->Rk;
  const double *deg = wannspace == EPHG_WANNSPACE_PH ? h->degq : h->degk;
  double2 *Lv = nullptr;
  if (h->polar_on) {   // the long-range term of each vertex's q (wannier.f90:998-1006)
    double *qp = qv;
    if (wannspace != EPHG_WANNSPACE_PH) {
      if ((rc = wsget(h->ws, "g2_qp", (size_t)nv * 3, &qp))) return WSFAIL(rc);
      CK(cudaMemcpyAsync(qp, qvecs, (size_t)nv * 3 * sizeof(double), cudaMemcpyHostToDevice, h->st));
    }
    if ((rc = wsget(h->ws, "g2_L", (size_t)nv * nb, &Lv))) return WSFAIL(rc);
    launch_polar_q(h->polar, (int)nv, nullptr, nullptr, qp, nullptr, nullptr, 0, Lv, h->st);
    h->launches += 1;
  }
  const int *ce;
  if ((rc = xgemm_colexp(h->ws, ngm, per, nws, gm, gstride, &ce, h->st))) return WSFAIL(rc);
  for (size_t p = 0; p + 1 < piece.size(); ++p) {
    const int64_t r0 = piece[p].first, c0 = piece[p].second;
    const int n = (int)(piece[p + 1].first - r0);
    launch_phase_cells(n, qv, nv, pd + r0, nws, R, deg, wannspace == EPHG_WANNSPACE_PH ? h->qlo : h->hlo,
                       wannspace == EPHG_WANNSPACE_PH ? h->qext : h->hext, P, nws, h->st);
    if ((rc = launch_xgemm_chunks(h->ws, cd + c0, (int)(piece[p + 1].second - c0), most, n, per, nws, P, nws, gm, per,
                                  gstride, ce, G, per, h->err, h->st)))
      return WSFAIL(rc);
    launch_g2_vertices(n, pd + r0, nv, nw, nb, G, ek, ekp, eq, en, h->masses, Lv, out, h->st);
    h->launches += 5;
  }
  CKL();
  CK(cudaMemcpyAsync(g2_out, out, (size_t)nv * sizeof(double), cudaMemcpyDeviceToHost, h->st));
  return ephg::api_check_err(h);
}

// ------------------------------------------------------------ kq index
int ephg_kq_index(ephg_handle *h, const int64_t mesh[3], int64_t nk, const int64_t *k_idx,
                  int64_t nkp, const int64_t *kp_idx, int64_t *q_idx) {
  if (!h || !mesh || nk < 0 || nkp < 0) return fail(EPHG_ERR_ARG, "kq_index: bad arguments");
  for (int i = 0; i < 3; ++i)
    if (mesh[i] <= 0) return fail(EPHG_ERR_ARG, "kq_index: bad mesh");
  if (nk == 0 || nkp == 0) return EPHG_OK;
  int m[3] = {(int)mesh[0], (int)mesh[1], (int)mesh[2]};
  int64_t *a, *b, *q;
  int rc;
  if ((rc = wsget(h->ws, "kq_a", (size_t)nk, &a)) || (rc = wsget(h->ws, "kq_b", (size_t)nkp, &b)) ||
      (rc = wsget(h->ws, "kq_q", (size_t)nk * nkp, &q)))
    return WSFAIL(rc);
  CK(cudaMemcpyAsync(a, k_idx, nk * sizeof(int64_t), cudaMemcpyHostToDevice, h->st));
  CK(cudaMemcpyAsync(b, kp_idx, nkp * sizeof(int64_t), cudaMemcpyHostToDevice, h->st));
  launch_kq_index(m, (int)nk, a, (int)nkp, b, q, h->err, h->st);
  h->launches += 1;
  CKL();
  CK(cudaMemcpyAsync(q_idx, q, (size_t)nk * nkp * sizeof(int64_t), cudaMemcpyDeviceToHost, h->st));
  return ephg::api_check_err(h);
}

}  // extern "C"

// ------------------------------------------------------------- rates
namespace {

struct EvTimer {
  cudaEvent_t e[6];
  EvTimer() { for (auto &x : e) cudaEventCreate(&x); }
  ~EvTimer() { for (auto &x : e) cudaEventDestroy(x); }
};

}  // namespace


// the device error word of an execution view: read, clear, translate
static int check_err_view(const ExecView &x) {
  int w = 0;
  CK(cudaMemcpyAsync(&w, x.err, sizeof(int), cudaMemcpyDeviceToHost, x.st));
  CK(cudaStreamSynchronize(x.st));
  CK(cudaMemsetAsync(x.err, 0, sizeof(int), x.st));
  if (w & DERR_NEG_PHONON) return fail(EPHG_ERR_NEG_PHONON, "Large negative phonon energy found!");
  if (w & DERR_EIG) return fail(EPHG_ERR_EIG, "Jacobi eigensolver did not converge");
  if (w & DERR_INDEX) return fail(EPHG_ERR_INDEX, "device index check failed");
  if (w & DERR_TIMEOUT) return fail(EPHG_ERR_TIMEOUT, "bounded device wait gave up");
  return EPHG_OK;
}

#define WSFAILX(rc) fail((rc), "%s", x.ws->msg.c_str())

static_assert(ephg::MAX_SETS == EPHG_MAX_SETS, "parameter-set bound of the C interface");

int ephg::check_sets(int64_t n, const ephg_rate_request *reqs) {
  if (n < 1 || n > MAX_SETS) return fail(EPHG_ERR_ARG, "el_rates_sets: nsets must be 1..%d", MAX_SETS);
  const ephg_rate_request &a = reqs[0];
  for (int64_t p = 0; p < n; ++p) {
    const ephg_rate_request &b = reqs[p];
    if (b.mesh[0] != a.mesh[0] || b.mesh[1] != a.mesh[1] || b.mesh[2] != a.mesh[2] || b.enref != a.enref ||
        b.fsthick != a.fsthick || b.delta_kind != a.delta_kind || b.precision != a.precision)
      return fail(EPHG_ERR_ARG, "el_rates_sets: set %lld differs from set 0 in more than T, sigma and chempot",
                  (long long)p);
    if (!(b.T > 0)) return fail(EPHG_ERR_ARG, "el_rates_sets: T must be > 0 (set %lld)", (long long)p);
    if (b.delta_kind == 0 && !(b.sigma > 0))
      return fail(EPHG_ERR_ARG, "el_rates_sets: sigma must be > 0 (set %lld)", (long long)p);
  }
  return EPHG_OK;
}

int ephg::el_rates_view(ephg_handle *h, const ExecView &x, const ephg_rate_request *req, double *rates,
                        int64_t *indexlist, ephg_rate_stats *stats, double *g2, double *xplus, double *xminus,
                        int64_t cap, const PhOut *ph, const DegAvgReq *avg, const SetsOut *sets) {
  if (!h || !req || (!ph && !avg && (!rates || !indexlist)) || (ph && !ph->rates_phe) || (avg && (ph || !avg->g2)))
    return fail(EPHG_ERR_ARG, "el_rates: bad arguments");
  if (sets) {
    if (ph || avg || g2 || sets->reqs != req || !sets->rates) return fail(EPHG_ERR_ARG, "el_rates_sets: bad arguments");
    int rc0 = check_sets(sets->n, sets->reqs);
    if (rc0) return rc0;
    for (int p = 0; p < sets->n; ++p)
      if (!sets->rates[p]) return fail(EPHG_ERR_ARG, "el_rates_sets: rates[%d] is NULL", p);
  }
  const int nsets = sets ? sets->n : 1;
  for (int i = 0; i < 3; ++i)
    if (req->mesh[i] <= 0) return fail(EPHG_ERR_ARG, "el_rates: bad mesh");
  if (req->delta_kind < 0 || req->delta_kind > 2) return fail(EPHG_ERR_ARG, "el_rates: bad delta_kind");
  if (req->delta_kind == 0 && !(req->sigma > 0)) return fail(EPHG_ERR_ARG, "el_rates: sigma must be > 0");
  if (!(req->T > 0)) return fail(EPHG_ERR_ARG, "el_rates: T must be > 0");
  if (req->precision != EPHG_PREC_FP64 && req->precision != EPHG_PREC_SPLIT_TF32)
    return fail(EPHG_ERR_ARG, "el_rates: bad precision");
  const int64_t N64 = req->mesh[0] * req->mesh[1] * req->mesh[2];
  if (N64 > (1 << 24)) return fail(EPHG_ERR_ARG, "el_rates: mesh too large");
  const int N = (int)N64;
  const int mesh[3] = {(int)req->mesh[0], (int)req->mesh[1], (int)req->mesh[2]};
  const int L = lcm3(mesh);
  const int nw = h->nw, nb = h->nb, nwsk = h->nwsk, nwsq = h->nwsq;
  const size_t nn = (size_t)nw * nw;
  const int ncol = nw * nb;   // columns per initial state in stage B
  const bool split = req->precision == EPHG_PREC_SPLIT_TF32;
  cudaStream_t st = x.st;
  int rc;
  int64_t launches0 = (*x.launches);
  EvTimer ev;
  (*x.ta).reset();
  (*x.tb).reset();
  CK(cudaEventRecord(ev.e[0], st));
  // ---- set-up: electrons on the full mesh (el_wann, electron.f90:364) ----
  double2 *roots, *Hk, *V, *Dq, *Vq, *u;
  double *w, *ens, *wq, *om, *bose, *rates_d;
  int *flag, *widx, *nwv_d, *sflag, *iota, *st_code, *nst_d, *nin_k, *cum;
  if ((rc = wsget((*x.ws), "r_roots", (size_t)L, &roots)) || (rc = wsget((*x.ws), "r_Hk", (size_t)N * nn, &Hk)) || (rc = wsget((*x.ws), "r_w", (size_t)N * nw, &w)) ||
      (rc = wsget((*x.ws), "r_V", (size_t)N * nn, &V)) || (rc = wsget((*x.ws), "r_ens", (size_t)N * nw, &ens)) ||
      (rc = wsget((*x.ws), "r_flag", (size_t)N, &flag)) || (rc = wsget((*x.ws), "r_widx", (size_t)N, &widx)) ||
      (rc = wsget((*x.ws), "r_nwv", 4, &nwv_d)) || (rc = wsget((*x.ws), "r_iota", (size_t)N * nw, &iota)) ||
      (rc = wsget((*x.ws), "r_Dq", (size_t)N * nb * nb, &Dq)) || (rc = wsget((*x.ws), "r_wq", (size_t)N * nb, &wq)) ||
      (rc = wsget((*x.ws), "r_Vq", (size_t)N * nb * nb, &Vq)) || (rc = wsget((*x.ws), "r_om", (size_t)N * nb, &om)) ||
      (rc = wsget((*x.ws), "r_u", (size_t)N * nb * nb, &u)) || (rc = wsget((*x.ws), "r_bose", (size_t)N * nb, &bose)) ||
      (rc = wsget((*x.ws), "r_rates", (size_t)N * nw, &rates_d)))
    return WSFAILX(rc);
  launch_roots(L, roots, st);
  {   // H(k) on the whole mesh: the Re sum one dimension at a time
    double2 *t1, *t2;
    if ((rc = wsget((*x.ws), "r_ht1", (size_t)h->hext[0] * h->hext[1] * mesh[2] * nn, &t1)) ||
        (rc = wsget((*x.ws), "r_ht2", (size_t)h->hext[0] * mesh[1] * mesh[2] * nn, &t2)))
      return WSFAILX(rc);
    launch_mesh_fourier(h->Hbox, h->hlo, h->hext, (int)nn, mesh, L, roots, t1, t2, Hk, st);
  }
  launch_heig(N, nw, Hk, nn, w, V, x.err, st);
  launch_el_post(N, nw, w, V, nullptr, 0, 0, nullptr, nullptr, nullptr, nullptr, ens, st);
  // ---- crystal symmetry: every mesh point takes the energies of its orbit's
  // representative, the irreducible point (electron.f90:363-385, 531-546); the
  // eigenvectors stay the point's own (:431-437).  The electron side then
  // starts from the irreducible window points only; the phonon side needs
  // every window k and keeps them all.
  const int nsymm = (int)(h->sym_rot.size() / 9);
  const bool ibz = nsymm > 0 && !ph;
  int *rep = nullptr;
  if (nsymm > 0) {
    std::vector<int> K;
    const char *why = "";
    if (ephg::mesh_qrotations(h->lattvecs, nsymm, h->sym_rot.data(), mesh, K, &why))
      return fail(EPHG_ERR_ARG, "el_rates: %s", why);
    int *Kd;
    double *ens_m;
    if ((rc = wsget((*x.ws), "r_symK", K.size(), &Kd)) || (rc = wsget((*x.ws), "r_rep", (size_t)N, &rep)) ||
        (rc = wsget((*x.ws), "r_ensm", (size_t)N * nw, &ens_m)))
      return WSFAILX(rc);
    CK(cudaMemcpyAsync(Kd, K.data(), K.size() * sizeof(int), cudaMemcpyHostToDevice, st));
    launch_sym_rep(N, mesh, (int)(K.size() / 9), Kd, rep, st);
    launch_map_ens(N, nw, rep, ens, ens_m, st);
    ens = ens_m;
    (*x.launches) += 2;
  }
  // ---- window (apply_energy_window, electron.f90:597-636) ----
  launch_window_flags(N, nw, ens, req->enref, req->fsthick, flag, st);
  launch_iota(N * nw, iota, st);
  size_t tmp_bytes = 0, tb2 = 0, tb3 = 0;
  cub::DeviceSelect::Flagged(nullptr, tmp_bytes, iota, flag, widx, nwv_d, N, st);
  if ((rc = wsget((*x.ws), "r_sflag", (size_t)N * nw, &sflag)) || (rc = wsget((*x.ws), "r_stcode", (size_t)N * nw, &st_code)) ||
      (rc = wsget((*x.ws), "r_nst", 4, &nst_d)) || (rc = wsget((*x.ws), "r_nink", (size_t)N + 1, &nin_k)) ||
      (rc = wsget((*x.ws), "r_cum", (size_t)N + 1, &cum)))
    return WSFAILX(rc);
  cub::DeviceSelect::Flagged(nullptr, tb2, iota, sflag, st_code, nst_d, N * nw, st);
  cub::DeviceScan::ExclusiveSum(nullptr, tb3, nin_k, cum, N + 1, st);
  void *cubtmp;
  if ((rc = x.ws->get("r_cub", std::max(tmp_bytes, std::max(tb2, tb3)), &cubtmp))) return WSFAILX(rc);
  size_t tbytes = std::max(tmp_bytes, std::max(tb2, tb3));
  cub::DeviceSelect::Flagged(cubtmp, tbytes, iota, flag, widx, nwv_d, N, st);
  (*x.launches) += 8;
  CKL();
  int nwv = 0;
  CK(cudaMemcpyAsync(&nwv, nwv_d, sizeof(int), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if ((rc = check_err_view(x))) return rc;
  if (nwv == 0) return fail(EPHG_ERR_EMPTY_WINDOW, "No states found within Fermi window.");
  // ---- phonons on the q mesh (phonon.f90:208-214) ----
  {   // D(q) on the whole mesh: the sum over wrapped cells one dimension at a time
    double2 *t1, *t2;
    const size_t ne = (size_t)nb * nb;
    if ((rc = wsget((*x.ws), "r_dt1", (size_t)h->dext[0] * h->dext[1] * mesh[2] * ne, &t1)) ||
        (rc = wsget((*x.ws), "r_dt2", (size_t)h->dext[0] * mesh[1] * mesh[2] * ne, &t2)))
      return WSFAILX(rc);
    launch_mesh_fourier(h->Dbox, h->dlo, h->dext, (int)ne, mesh, L, roots, t1, t2, Dq, st);
  }
  double2 *Lq = nullptr, *glp = nullptr;
  float2 *glpf = nullptr;
  if (h->polar_on) {   // dyn_nonanalytic into D(q) and the long-range vector of every mesh q
    if ((rc = wsget((*x.ws), "r_Lq", (size_t)N * nb, &Lq)) || (rc = wsget((*x.ws), "r_glp", (size_t)N * nb, &glp)) ||
        (split && (rc = wsget((*x.ws), "r_glpf", (size_t)N * nb, &glpf))))
      return WSFAILX(rc);
    launch_polar_q(h->polar, N, iota, mesh, nullptr, Dq, nullptr, (int64_t)nb * nb, Lq, st);
    (*x.launches) += 1;
  }
  launch_heig(N, nb, Dq, (int64_t)nb * nb, wq, Vq, x.err, st);
  float2 *uf = nullptr;
  if (split && (rc = wsget((*x.ws), "r_uf", (size_t)N * nb * nb, &uf))) return WSFAILX(rc);
  launch_ph_post(N, nb, iota, nullptr, wq, Vq, nullptr, 0, 0, h->masses, nullptr, nullptr, nullptr, om,
                 u, uf, x.err, st);
  launch_bose(N, nb, om, req->T, bose, st);
  RateSets rs;
  memset(&rs, 0, sizeof rs);
  rs.n = nsets;
  for (int p = 1; p < nsets; ++p) {   // the other parameter sets' Bose factors
    if ((rc = wsget((*x.ws), ("r_bose" + std::to_string(p)).c_str(), (size_t)N * nb, &rs.bose[p])))
      return WSFAILX(rc);
    launch_bose(N, nb, om, sets->reqs[p].T, rs.bose[p], st);
    (*x.launches) += 1;
  }
  if (h->polar_on) {   // long_range_prefac(q, u_s) for every (q, s)
    launch_glprefac(N, nb, Lq, u, glp, glpf, st);
    (*x.launches) += 1;
  }
  // ---- final states: window bands of the window k' (their ranks, cum) ----
  launch_state_flags(nwv, nw, widx, ens, req->enref, req->fsthick, sflag, nin_k, st);
  CK(cudaMemsetAsync(nin_k + nwv, 0, sizeof(int), st));
  tbytes = std::max(tmp_bytes, std::max(tb2, tb3));
  cub::DeviceScan::ExclusiveSum(cubtmp, tbytes, nin_k, cum, nwv + 1, st);
  std::vector<int> widx_h(nwv), code_h;
  CK(cudaMemcpyAsync(widx_h.data(), widx, nwv * sizeof(int), cudaMemcpyDeviceToHost, st));
  // ---- A-rows: the k of the initial states, the window points or, with
  // crystal symmetry, the irreducible ones (IBZ blocks, find_irred_wedge with
  // blocks, electron.f90:553-577), in window order ----
  int nA = nwv;
  const int *arow = widx;
  std::vector<int> arow_h;
  if (ibz) {
    std::vector<int> rep_h(N);
    CK(cudaMemcpyAsync(rep_h.data(), rep, (size_t)N * sizeof(int), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    for (int i = 0; i < nwv; ++i)
      if (rep_h[widx_h[i]] == widx_h[i]) arow_h.push_back(widx_h[i]);
    nA = (int)arow_h.size();
    int *arow_d, *ninA;
    if ((rc = wsget((*x.ws), "r_arow", (size_t)nA, &arow_d)) || (rc = wsget((*x.ws), "r_ninA", (size_t)nA, &ninA)))
      return WSFAILX(rc);
    CK(cudaMemcpyAsync(arow_d, arow_h.data(), (size_t)nA * sizeof(int), cudaMemcpyHostToDevice, st));
    arow = arow_d;
    launch_state_flags(nA, nw, arow, ens, req->enref, req->fsthick, sflag, ninA, st);
  }
  // ---- initial states (demux_state order, interactions.f90:2169-2191) ----
  tbytes = std::max(tmp_bytes, std::max(tb2, tb3));
  cub::DeviceSelect::Flagged(cubtmp, tbytes, iota, sflag, st_code, nst_d, nA * nw, st);
  (*x.launches) += 7;
  CKL();
  int nst = 0, nin = 0;
  CK(cudaMemcpyAsync(&nst, nst_d, sizeof(int), cudaMemcpyDeviceToHost, st));
  CK(cudaMemcpyAsync(&nin, cum + nwv, sizeof(int), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if ((rc = check_err_view(x))) return rc;
  if (!ibz) arow_h = widx_h;
  code_h.resize(nst);
  CK(cudaMemcpyAsync(code_h.data(), st_code, nst * sizeof(int), cudaMemcpyDeviceToHost, st));
  EpiData ed;
  memset(&ed, 0, sizeof ed);
  CK(cudaStreamSynchronize(st));
  std::vector<int> first_state(nA + 1, nst);
  for (int j = nst - 1; j >= 0; --j) first_state[code_h[j] / nw] = j;
  for (int i = nA - 1; i >= 0; --i)
    if (first_state[i] > first_state[i + 1]) first_state[i] = first_state[i + 1];
  if (avg) {   // degenerate-subspace averaging of the caller's vertex list, no contraction
    const int64_t per = (int64_t)nin * nb, vtot = (int64_t)nst * per;
    if (avg->nv != vtot)
      return fail(EPHG_ERR_ARG, "g2_average_degenerate: the list has %lld entries, the request's vertex list %lld",
                  (long long)avg->nv, (long long)vtot);
    double *g2d;
    int *fsd;
    if ((rc = wsget((*x.ws), "r_vg2", (size_t)vtot, &g2d)) || (rc = wsget((*x.ws), "r_fsd", (size_t)nA + 1, &fsd)))
      return WSFAILX(rc);
    CK(cudaMemcpyAsync(g2d, avg->g2, (size_t)vtot * sizeof(double), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(fsd, first_state.data(), (size_t)(nA + 1) * sizeof(int), cudaMemcpyHostToDevice, st));
    if (launch_degenerate_average(g2d, per, nin, st_code, arow, widx, cum, fsd, ens, om, nst, nA, nwv, nw, nb, mesh,
                                  req->enref, req->fsthick, avg->thres, avg->mode, st))
      return fail(EPHG_ERR_ARG, "g2_average_degenerate: nw and nb must be <= 64");
    (*x.launches) += 3;
    CKL();
    CK(cudaMemcpyAsync(avg->g2, g2d, (size_t)vtot * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (indexlist)
      for (int i = 0; i < nA; ++i) indexlist[i] = (int64_t)arow_h[i] + 1;
    if ((rc = check_err_view(x))) return rc;
    if (stats) {
      memset(stats, 0, sizeof *stats);
      stats->nwv = nA;
      stats->nstates_inwindow = nin;
      stats->nstates = nst;
      stats->vertices = vtot;
      stats->pairs = (int64_t)nst * nwv;
    }
    return EPHG_OK;
  }
  CK(cudaEventRecord(ev.e[1], st));
  x.yield();   // serving: hand the GPU to a smaller request before the contractions
  // ---- stage A: g(k,Rp) for window k, rotation over m, k-half of the Rp phase ----
  const int64_t ldb = (int64_t)ncol * nst;
  const int64_t Nn = h->Nn;
  RateParams rp;
  for (int i = 0; i < 3; ++i) rp.mesh[i] = mesh[i];
  rp.N = N;
  rp.nw = nw;
  rp.nb = nb;
  rp.enref = req->enref;
  rp.fsthick = req->fsthick;
  rp.chempot = req->chempot;
  rp.T = req->T;
  rp.delta_kind = (int)req->delta_kind;
  rp.sigma = req->sigma;
  rp.inv_nk = 1.0 / (double)N;
  rp.const_tp = 2.0 * 3.141592653589793 / hbar_eVps;
  ed.widx = widx;
  ed.sidx = arow;
  ed.st_code = st_code;
  ed.cum = cum;
  ed.ens = ens;
  ed.U = V;
  ed.om = om;
  ed.u = u;
  ed.uf = uf;
  ed.bose = bose;
  ed.glp = glp;
  ed.glpf = glpf;
  ed.per_state = (int64_t)nin * nb;
  ed.nin = nin;
  double *g2d = nullptr, *xpd = nullptr, *xmd = nullptr, *yd = nullptr, *phr = nullptr;
  int64_t vtot = (int64_t)nst * nin * nb;
  int64_t vcap = std::min<int64_t>(cap, vtot);
  const bool want_y = ph && ph->y;
  const bool lists = (g2 || want_y) && vcap > 0;
  if (lists) {
    if ((rc = wsget((*x.ws), "r_vg2", (size_t)vcap, &g2d)) || (rc = wsget((*x.ws), "r_vxp", (size_t)vcap, &xpd)) ||
        (rc = wsget((*x.ws), "r_vxm", (size_t)vcap, &xmd)) ||
        (want_y && (rc = wsget((*x.ws), "r_vy", (size_t)vcap, &yd))))
      return WSFAILX(rc);
    ed.g2 = g2d;
    ed.xp = xpd;
    ed.xm = xmd;
    ed.yv = yd;
    ed.cap = vcap;
  }
  if (ph) {
    // the phonon states' rates, summed by the epilogues' atomics (ibzq 'Y' + ph-e rates)
    if ((rc = wsget((*x.ws), "r_phr", (size_t)N * nb, &phr))) return WSFAILX(rc);
    CK(cudaMemsetAsync(phr, 0, (size_t)N * nb * sizeof(double), st));
    ed.phr = phr;
    ed.ph_scale = ph->spindeg;
  }
  // FP64 epilogues (the FP64 form; the simplex deltas of both): final states, mode
  // tables of every parameter set and the deltas' tables
  const bool final_epi = !split || req->delta_kind != 0;
  if (final_epi) {
    int2 *fin;
    if ((rc = wsget((*x.ws), "e_fin", (size_t)nin, &fin))) return WSFAILX(rc);
    launch_final_states(nwv, nw, widx, ens, req->enref, req->fsthick, cum, fin, st);
    for (int p = 0; p < nsets; ++p) {
      ModeRec *mt;
      if ((rc = wsget((*x.ws), ("e_mt" + std::to_string(p)).c_str(), (size_t)N * nb, &mt))) return WSFAILX(rc);
      launch_mode_tab(N * nb, om, p ? rs.bose[p] : bose, p ? sets->reqs[p].T : req->T, rp.const_tp, mt, st);
      rs.mt[p] = mt;
    }
    ed.fin = fin;
    ed.mt = rs.mt[0];
    (*x.launches) += 1 + nsets;
    if (req->delta_kind != 0) {
      SimplexTab &t = ed.sx;
      int *map;
      t.stride = req->delta_kind == 1 ? 18 : SX_MAX;
      const size_t ne = (size_t)nin * t.stride;
      if ((rc = wsget((*x.ws), "e_sxn", (size_t)nin, &t.n)) || (rc = wsget((*x.ws), "e_sxk", ne, &t.key)) ||
          (rc = wsget((*x.ws), "e_sxb", ne, &t.b)) || (rc = wsget((*x.ws), "e_sxl", ne, &t.lo)) ||
          (rc = wsget((*x.ws), "e_sxh", ne, &t.hi)) || (rc = wsget((*x.ws), "a_map", (size_t)N, &map)))
        return WSFAILX(rc);
      launch_row_map(N, nwv, widx, map, st);
      launch_simplex_tab((int)req->delta_kind, mesh, nin, fin, widx, map, ens, nw, t, st);
      (*x.launches) += 2;
    }
    CKL();
  }
  // blocks of the rate partials: of final states in the FP64 epilogues, else of 32 (fused) or 128 rows
  const int nblk_max = final_epi ? epf_blocks(nin) : (nwv + 255) / 256 * 8;
  int nblk = nblk_max;
  double *partial;
  if ((rc = wsget((*x.ws), "r_partial", (size_t)nst * nblk_max, &partial))) return WSFAILX(rc);
  rs.rp[0] = rp;
  rs.bose[0] = bose;
  rs.partial[0] = partial;
  for (int p = 1; p < nsets; ++p) {
    rs.rp[p] = rp;
    rs.rp[p].T = sets->reqs[p].T;
    rs.rp[p].sigma = sets->reqs[p].sigma;
    rs.rp[p].chempot = sets->reqs[p].chempot;
    if ((rc = wsget((*x.ws), ("r_partial" + std::to_string(p)).c_str(), (size_t)nst * nblk_max, &rs.partial[p])))
      return WSFAILX(rc);
  }
  if (!split) {
    // Each contraction is a Fourier sum of cells onto mesh points: one dimension at a
    // time on the FP64 pipe (launch_cells_fourier), which forms whole mesh lines, or as a
    // product with the rows' phases on the tensor cores (launch_xgemm), whose time grows
    // with rows times cells.  Whichever is estimated shorter per column; of 300 measured
    // contractions (6^3 to 24^3, 43 to 279 cells, 20 to 2,500 rows) the choice is within 5%
    // of the better one in 285, the others being calls of a few columns (under 30 us).  Sums / products in ms, stage A: 12^3, 279 cells, 1,678 rows
    // 8.8 / 14.4, 955 rows 7.8 / 8.0, 397 rows 6.5 / 3.5, 60 rows 5.6 / 0.6; 9x10x9, 93 cells,
    // 756 rows 1.09 / 1.10; 24^3, 93 cells, 1,001 rows 4.0 / 1.4.
    const bool sepA = cells_fourier_cycles(h->cellk, mesh, nA) < xgemm_cycles(nA, nwsk);
    const bool sepB = cells_fourier_cycles(h->cellq, mesh, nwv) < xgemm_cycles(nwv, nwsq);
    const int64_t per = (int64_t)nw * nw, nper = (int64_t)nb * nwsq;   // columns of one (mode, Rp) block; blocks
    const int64_t bound = (int64_t)1 << 31;
    double2 *Pk = nullptr, *t1 = nullptr, *t2 = nullptr, *gk, *B, *Pq = nullptr, *Cb, *phk;
    int *rowmap = nullptr;
    const int64_t a1 = cells_t1_rows(h->cellk, mesh), a2 = cells_t2_rows(h->cellk, mesh);
    const int64_t b1 = cells_t1_rows(h->cellq, mesh), b2 = cells_t2_rows(h->cellq, mesh);
    // stage A as sums: ra blocks at a time, all rows; as products: kc rows at a time, all blocks
    const int64_t ra = sepA ? std::max<int64_t>(1, std::min<int64_t>(nper, bound / ((a1 + a2 + nA) * per * 16))) : nper;
    const int64_t kc = sepA ? nA : std::max<int64_t>(1, std::min<int64_t>(nA, bound / (Nn * 16)));
    // states per chunk of stage B
    const int64_t brows = sepB ? b1 + b2 + nwv : nwv;
    const int64_t sc = std::max<int64_t>(1, std::min<int64_t>({(int64_t)nst, (int64_t)32768, bound / (brows * ncol * 16)}));
    const int64_t n1 = std::max(sepA ? a1 * ra * per : 0, sepB ? b1 * sc * ncol : 0);
    const int64_t n2 = std::max(sepA ? a2 * ra * per : 0, sepB ? b2 * sc * ncol : 0);
    if ((!sepA && (rc = wsget((*x.ws), "a_Pk", (size_t)kc * nwsk, &Pk))) ||
        (n1 && (rc = wsget((*x.ws), "a_t1", (size_t)n1, &t1))) || (n2 && (rc = wsget((*x.ws), "a_t2", (size_t)n2, &t2))) ||
        (rc = wsget((*x.ws), "a_gk", (size_t)kc * ra * per, &gk)) || (rc = wsget((*x.ws), "a_B", (size_t)nwsq * ldb, &B)) ||
        (rc = wsget((*x.ws), "a_phk", (size_t)nA * nwsq, &phk)) || (rc = wsget((*x.ws), "a_map", (size_t)N, &rowmap)) ||
        (!sepB && (rc = wsget((*x.ws), "b_Pq", (size_t)nwv * nwsq, &Pq))) ||
        (rc = wsget((*x.ws), "b_C", (size_t)nwv * ncol * sc, &Cb)))
      return WSFAILX(rc);
    launch_phase_mesh(nA, arow, mesh, L, nwsq, h->Rq, h->degq, 1, roots, phk, nwsq, st);
    (*x.launches) += 1;
    if (sepA) {
      launch_row_map(N, nA, arow, rowmap, st);
      (*x.launches) += 1;
      for (int64_t r0 = 0; r0 < nper; r0 += ra) {
        const int64_t nr = std::min<int64_t>(ra, nper - r0);
        (*x.ta).begin(st);
        launch_cells_fourier(h->cellk, h->G64 + r0 * per, Nn, h->rdegk, (int)(nr * per), mesh, L, roots, t1, t2, rowmap,
                             gk, nr * per, st);
        (*x.ta).end(st);
        launch_rotate_states_fp64(0, nst, 0, st_code, nw, nb, nwsq, r0, nr, arow, V, gk, nr * per, phk, B, ldb,
                                  (int)sc, nst, st);
        (*x.launches) += 4;
      }
    } else {
      for (int64_t i0 = 0; i0 < nA; i0 += kc) {
        const int n = (int)std::min<int64_t>(kc, nA - i0);
        launch_phase_mesh(n, arow + i0, mesh, L, nwsk, h->Rk, h->degk, 0, roots, Pk, nwsk, st);
        (*x.ta).begin(st);
        if ((rc = launch_xgemm(*x.ws, n, Nn, nwsk, Pk, nwsk, h->G64, Nn, h->exp_G, gk, Nn, x.err, st))) return WSFAILX(rc);
        (*x.ta).end(st);
        launch_rotate_states_fp64(first_state[i0], first_state[i0 + n], (int)i0, st_code, nw, nb, nwsq, 0, nper, arow, V,
                                  gk, Nn, phk, B, ldb, (int)sc, nst, st);
        (*x.launches) += 3;
      }
    }
    CK(cudaEventRecord(ev.e[2], st));
    // ---- stage B + C: Rp Fourier against e^{2 pi i k'.Rp}, then the epilogue ----
    if (sepB) launch_row_map(N, nwv, widx, rowmap, st);
    else launch_phase_mesh(nwv, widx, mesh, L, nwsq, h->Rq, nullptr, 0, roots, Pq, nwsq, st);
    (*x.launches) += 1;
    for (int64_t j0 = 0; j0 < nst; j0 += sc) {
      int ns = (int)std::min<int64_t>(sc, nst - j0);
      (*x.tb).begin(st);
      if (sepB) {
        launch_cells_fourier(h->cellq, B + j0 * ncol, ldb, nullptr, ns * ncol, mesh, L, roots, t1, t2, rowmap, Cb,
                             (int64_t)ns * ncol, st);
      } else if ((rc = launch_xgemm(*x.ws, nwv, (int64_t)ns * ncol, nwsq, Pq, nwsq, B + j0 * ncol, ldb, nullptr, Cb,
                                    (int64_t)ns * ncol, x.err, st))) {
        return WSFAILX(rc);
      }
      (*x.tb).end(st);
      (*x.launches) += 3;
      FinalIn in;
      in.z = Cb;
      in.ldc = (int64_t)ns * ncol;
      in.xs = ns;
      in.js = 1;
      launch_epilogue_final((int)j0, (int)j0 + ns, in, rp, ed, partial, nblk, st);
      for (int p = 1; p < nsets; ++p) {   // the same sums under the other parameter sets
        EpiData ep = ed;
        ep.bose = rs.bose[p];
        ep.mt = rs.mt[p];
        launch_epilogue_final((int)j0, (int)j0 + ns, in, rs.rp[p], ep, rs.partial[p], nblk, st);
        (*x.launches) += 1;
      }
      (*x.launches) += 1;
    }
  } else {
    rc = tc::split_rates_stage(h->split, *x.ws, st, h->G64, h->nwsk, nwsq, Nn, nw, nb, nwv, nst,
                               mesh, L, roots, widx, arow, nA, st_code, first_state, h->Rk, h->degk, h->kposk,
                               h->Rq, h->degq, h->kposq, V, rp, ed, partial, nblk_max, &nblk,
                               ev.e[2], x.launches, x.ta, x.tb, &h->split_mu, x.chunk_us, x.yield, &x.bm,
                               x.chunk_bytes, nsets > 1 ? &rs : nullptr);
    if (rc) return fail(rc, "split path: %s", tc::last_error());
  }
  CKL();
  CK(cudaMemsetAsync(rates_d, 0, (size_t)N * nw * sizeof(double), st));
  launch_rate_final(nst, nblk, partial, st_code, nw, N, rates_d, st);
  (*x.launches) += 1;
  std::vector<double *> rates_sets(nsets, rates_d);
  for (int p = 1; p < nsets; ++p) {
    if ((rc = wsget((*x.ws), ("r_rates" + std::to_string(p)).c_str(), (size_t)N * nw, &rates_sets[p])))
      return WSFAILX(rc);
    CK(cudaMemsetAsync(rates_sets[p], 0, (size_t)N * nw * sizeof(double), st));
    launch_rate_final(nst, nblk, rs.partial[p], st_code, nw, N, rates_sets[p], st);
    (*x.launches) += 1;
  }
  CK(cudaEventRecord(ev.e[3], st));
  if (rates) CK(cudaMemcpyAsync(rates, rates_d, (size_t)N * nw * sizeof(double), cudaMemcpyDeviceToHost, st));
  for (int p = 1; p < nsets; ++p)
    CK(cudaMemcpyAsync(sets->rates[p], rates_sets[p], (size_t)N * nw * sizeof(double), cudaMemcpyDeviceToHost, st));
  if (ph) CK(cudaMemcpyAsync(ph->rates_phe, phr, (size_t)N * nb * sizeof(double), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if (indexlist)   // the rows of the rates: the A-rows
    for (int i = 0; i < nA; ++i) indexlist[i] = (int64_t)arow_h[i] + 1;
  if (lists) {
    if (g2) CK(cudaMemcpyAsync(g2, g2d, vcap * sizeof(double), cudaMemcpyDeviceToHost, st));
    if (g2 && xplus) CK(cudaMemcpyAsync(xplus, xpd, vcap * sizeof(double), cudaMemcpyDeviceToHost, st));
    if (g2 && xminus) CK(cudaMemcpyAsync(xminus, xmd, vcap * sizeof(double), cudaMemcpyDeviceToHost, st));
    if (want_y) CK(cudaMemcpyAsync(ph->y, yd, vcap * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
  }
  if ((rc = check_err_view(x))) return rc;
  if (stats) {
    float t01 = 0, t12 = 0, t23 = 0, t03 = 0;
    cudaEventElapsedTime(&t01, ev.e[0], ev.e[1]);
    cudaEventElapsedTime(&t12, ev.e[1], ev.e[2]);
    cudaEventElapsedTime(&t23, ev.e[2], ev.e[3]);
    cudaEventElapsedTime(&t03, ev.e[0], ev.e[3]);
    stats->nwv = nA;
    stats->nstates_inwindow = nin;
    stats->nstates = nst;
    stats->vertices = vtot;
    stats->pairs = (int64_t)nst * nwv;
    stats->kernel_launches = (*x.launches) - launches0;
    stats->ms_setup = t01;
    stats->ms_stage_a = t12;
    stats->ms_stage_bc = t23;
    stats->ms_total = t03;
    stats->stage_a_gflop = 8.0 * (double)nA * nwsk * (double)Nn * 1e-9;
    stats->stage_b_gflop = 8.0 * (double)nwv * nwsq * (double)ncol * nst * 1e-9;
    stats->ms_gemm_a = (*x.ta).total_ms();
    stats->ms_gemm_b = (*x.tb).total_ms();
    stats->gemm_a_launches = (*x.ta).n;
    stats->gemm_b_launches = (*x.tb).n;
  }
  return EPHG_OK;
}

extern "C" int ephg_el_rates(ephg_handle *h, const ephg_rate_request *req, double *rates,
                             int64_t *indexlist, ephg_rate_stats *stats, double *g2,
                             double *xplus, double *xminus, int64_t cap) {
  if (!h) return fail(EPHG_ERR_ARG, "el_rates: bad arguments");
  const ExecView x{h->st, h->err, &h->ws, &h->timer_a, &h->timer_b, &h->launches};
  return el_rates_view(h, x, req, rates, indexlist, stats, g2, xplus, xminus, cap);
}

extern "C" int ephg_el_rates_sets(ephg_handle *h, int64_t nsets, const ephg_rate_request *reqs, double *const *rates,
                                  int64_t *indexlist, ephg_rate_stats *stats) {
  if (!h || !reqs || !rates || !indexlist) return fail(EPHG_ERR_ARG, "el_rates_sets: bad arguments");
  int rc = check_sets(nsets, reqs);
  if (rc) return rc;
  const ExecView x{h->st, h->err, &h->ws, &h->timer_a, &h->timer_b, &h->launches};
  const SetsOut so{(int)nsets, reqs, rates};
  return el_rates_view(h, x, &reqs[0], rates[0], indexlist, stats, nullptr, nullptr, nullptr, 0, nullptr, nullptr,
                       &so);
}

extern "C" int ephg_g2_average_degenerate(ephg_handle *h, const ephg_rate_request *req, int64_t mode, double thres,
                                          int64_t nv, double *g2) {
  if (!h || !req || !g2 || nv < 0) return fail(EPHG_ERR_ARG, "g2_average_degenerate: bad arguments");
  if (mode != EPHG_DEGAVG_REFERENCE && mode != EPHG_DEGAVG_MEAN)
    return fail(EPHG_ERR_ARG, "g2_average_degenerate: bad mode");
  const ExecView x{h->st, h->err, &h->ws, &h->timer_a, &h->timer_b, &h->launches};
  const DegAvgReq avg{g2, nv, (int)mode, thres > 0 ? thres : 1.0e-6};
  return el_rates_view(h, x, req, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0, nullptr, &avg);
}

extern "C" int ephg_ph_rates(ephg_handle *h, const ephg_rate_request *req, int64_t spindeg, double *rates_phe,
                             double *el_rates, int64_t *indexlist, ephg_rate_stats *stats, double *g2, double *y,
                             int64_t cap) {
  if (!h || !rates_phe) return fail(EPHG_ERR_ARG, "ph_rates: bad arguments");
  // "spindeg can be 1 or 2.", electron.f90:164-166
  if (spindeg < 1 || spindeg > 2) return fail(EPHG_ERR_ARG, "ph_rates: spindeg must be 1 or 2");
  const ExecView x{h->st, h->err, &h->ws, &h->timer_a, &h->timer_b, &h->launches};
  const PhOut ph{rates_phe, y, (double)spindeg};
  return el_rates_view(h, x, req, el_rates, indexlist, stats, g2, nullptr, nullptr, cap, &ph);
}

// The FP64 rate path's sums over cells on their own (include/ephg_debug.h).
extern "C" int ephg_debug_cells_fourier(int64_t ncells, const int64_t *cells, const double *scale, const int64_t mesh[3],
                                        int64_t nc, const double *in, int64_t nrows, const int64_t *rows, double *out) {
  if (ncells <= 0 || !cells || !mesh || nc <= 0 || !in || nrows <= 0 || !rows || !out)
    return fail(EPHG_ERR_ARG, "debug_cells_fourier: bad arguments");
  const int m[3] = {(int)mesh[0], (int)mesh[1], (int)mesh[2]};
  const int64_t N = mesh[0] * mesh[1] * mesh[2];
  std::vector<int> r(3 * (size_t)ncells), rw(nrows), tab;
  for (int64_t i = 0; i < ncells; ++i)
    for (int c = 0; c < 3; ++c) r[3 * i + c] = (int)cells[i + ncells * c];
  for (int64_t i = 0; i < nrows; ++i) {
    if (rows[i] < 0 || rows[i] >= N) return fail(EPHG_ERR_ARG, "debug_cells_fourier: row outside the mesh");
    rw[i] = (int)rows[i];
  }
  CellTab t;
  size_t off[3];
  if (!cell_tables(r, (int)ncells, t, tab, off)) return fail(EPHG_ERR_ARG, "debug_cells_fourier: cells");
  t.ok = true;
  if (std::isinf(cells_fourier_cost(t, m, nrows))) return fail(EPHG_ERR_ARG, "debug_cells_fourier: mesh");
  const int L = lcm3(m);
  Workspace ws;
  int *td, *rd, *map, rc;
  double *sd = nullptr;
  double2 *roots, *t1, *t2, *a, *b;
  if ((rc = wsget(ws, "tab", tab.size(), &td)) || (rc = wsget(ws, "rows", rw.size(), &rd)) ||
      (rc = wsget(ws, "map", (size_t)N, &map)) || (rc = wsget(ws, "roots", (size_t)L, &roots)) ||
      (scale && (rc = wsget(ws, "scale", (size_t)ncells, &sd))) ||
      (rc = wsget(ws, "t1", (size_t)(cells_t1_rows(t, m) * nc), &t1)) ||
      (rc = wsget(ws, "t2", (size_t)(cells_t2_rows(t, m) * nc), &t2)) ||
      (rc = wsget(ws, "in", (size_t)(ncells * nc), &a)) || (rc = wsget(ws, "out", (size_t)(nrows * nc), &b))) {
    ws.release();
    return fail(rc, "%s", ws.msg.c_str());
  }
  t.tab1 = td + off[0];
  t.tab2 = td + off[1];
  t.tab3 = td + off[2];
  cudaMemcpy(td, tab.data(), tab.size() * sizeof(int), cudaMemcpyHostToDevice);
  cudaMemcpy(rd, rw.data(), rw.size() * sizeof(int), cudaMemcpyHostToDevice);
  if (scale) cudaMemcpy(sd, scale, (size_t)ncells * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(a, in, (size_t)(ncells * nc) * sizeof(double2), cudaMemcpyHostToDevice);
  launch_roots(L, roots, nullptr);
  launch_row_map((int)N, (int)nrows, rd, map, nullptr);
  launch_cells_fourier(t, a, nc, sd, (int)nc, m, L, roots, t1, t2, map, b, nc, nullptr);
  const cudaError_t e = cudaMemcpy(out, b, (size_t)(nrows * nc) * sizeof(double2), cudaMemcpyDeviceToHost);
  ws.release();
  return e == cudaSuccess && cudaGetLastError() == cudaSuccess
             ? EPHG_OK
             : fail(EPHG_ERR_CUDA, "debug_cells_fourier: %s", cudaGetErrorString(e));
}
