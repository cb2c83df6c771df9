// ephg_xgemm.cu - FP64 complex products on the tensor cores by exact splitting.
//
// The arbitrary-k Fourier sums (H(k), g(k,Rp), g(Re,q), the Rp sums of a vertex
// list) are products of a few rows of phases with a tall resident matrix.  As
// FP64 multiply-adds they are bound by the FP64 pipe (1.25 TFLOP/s), 60 times
// under the memory traffic they need.  Here each real operand is split into
// nine signed 7-bit digits of a fixed point per column (63 bits: an FP64 number
// to well below its own rounding), digits are exact in BF16, and the products of
// digits i and j with i + j = l are integers that the FP32 accumulators of
// tcgen05.mma hold exactly: the method of Ozaki, Ogita, Oishi and Rump
// (Numerical Algorithms 59, 2012).
//
//   sum_k a_k b_k = sum_l 2^(-7 l - 12) S_l,   S_l = sum over i + j = l, k of integers |d| <= 64
//
// Levels have an accumulator each, 7 and 8 one together (nine of the widest chunk do not
// fit TMEM; every chunk width takes the same eight, so that a row's result does not depend
// on how many rows share its call); |S_l| <= (l + 1) 4096 K stays within 2^24
// for the XG_KGROUP positions summed at a time for l <= 5; above that (2^-54 of the
// result) only for sums not of one sign throughout, and an FP32 rounding there no
// longer counts.  Products beyond level 8 (2^-63), and the tall operand's first digit with
// the phases' last (2^-62 of one phase), are left out.  The result is the
// exact sum of the products to ~2^-60 of the largest term, rounded once: its error is at or below that of the FP64
// multiply-adds it replaces (g(Re,q), 279 cells, against sums of the same phases in
// extended precision: 5.5e-17 relative; the multiply-adds 7.6e-16).
//
// The tall matrix is the M operand: a tile is 128 of its columns, with K running
// over (cell, re | im), so that one product gives C = A B for up to 32 rows of
// phases as columns (row m: real and imaginary part).  A level's accumulator lies
// beside the next level's, as the phases' digit planes do in shared memory, so one
// MMA of up to 256 columns takes a digit of the tall operand with several digits of
// the phases.  The tall operand's digits are
// formed where they are used: sixteen warps read the FP64 values (coalesced along
// the columns, each once per chunk of phase rows) and write the nine BF16 planes of
// a stage in the swizzled layout the MMA reads; HBM sees the FP64 matrix only.
// The phases' digits are formed once per call and arrive by bulk copies.  Two
// stages of 104 KB; 44 digit products per stage, the tensor core is the bound
// (about one cycle a column at these widths), the splitting runs beside it.
//
// Measured: g(k,Rp) at 25 k, nw 8, nb 6, 279 cells: 0.29 ms (6.70 as FP64 multiply-adds);
// 200 H(k) with velocities, nw 8: 0.053 ms (0.61); 1,728 D(q) with derivatives, nb 6, 339
// wrapped cells: 0.072 ms (1.16 in the kernel that summed them in FP64).  On the way: one
// MMA per digit pair 0.46 ms, descriptors formed in loops 0.49 ms (the issuing thread
// was the bound), one FP64 drain warp per quadrant 0.32 ms.
#include <cuda_bf16.h>

#include <algorithm>
#include <climits>

#include "../../include/ephg.h"
#include "ephg_ptx.cuh"
#include "ephg_xgemm.cuh"

namespace ephg {

using namespace tc;

constexpr int XG_D = 9, XG_DA = XG_D - 1;              // digits; the phases' last one meets none (below)
constexpr int XG_ROWS = 128, XG_M = XG_CHUNK;          // tile columns of B; phase rows of a chunk
constexpr int XG_W = 2 * XG_M;                         // most MMA columns of a level
constexpr int XG_CELLS = 16, XG_KV = 2 * XG_CELLS;     // cells and K values per stage
constexpr int XG_KGROUP = 320 / XG_CELLS;              // stages per accumulation: 640 K values
constexpr int XG_PLANE_B = XG_ROWS * XG_KV * 2;        // 8 KB per digit
constexpr int XG_PLANE_A = XG_W * XG_KV * 2;           // at most 4 KB per digit
constexpr int XG_STAGE_B = XG_D * XG_PLANE_B, XG_STAGE_A = XG_DA * XG_PLANE_A;
constexpr int XG_STAGE = (XG_STAGE_B + XG_STAGE_A + 1023) / 1024 * 1024;
constexpr int XG_LEVELS = XG_D - 1;                    // accumulators of W columns; level 8 shares the last
static_assert(XG_LEVELS * XG_W <= 512, "the levels' accumulators fit TMEM");
constexpr int XG_STAGES = 2;
constexpr int XG_SMEM = XG_STAGES * XG_STAGE + 1024 + 256;
constexpr int XG_CONV = 512, XG_EPI = 256;             // converter and epilogue threads
constexpr int XG_THREADS = 64 + XG_CONV + XG_EPI;
constexpr int XG_BATCH = 4096;                         // phase rows per launch (bounds the digit buffer)
constexpr int XG_BAD = INT_MAX;                        // exponent of a column with a non-finite value

// x as 62-bit fixed point of 2^e (|x| <= 2^e), biased so that the nine digits are plain
// bit fields: digit i = field i - 64
__device__ __forceinline__ uint64_t xg_fixed(double x, int e) {
  const uint64_t u = (uint64_t)__double_as_longlong(x);
  const int ex = (int)((u >> 52) & 0x7ff);
  uint64_t m = (u & 0xFFFFFFFFFFFFFull) << 10;
  if (ex) m |= 1ull << 62;
  const int sh = 1023 + e - max(ex, 1);   // >= 0
  m = sh < 64 ? m >> sh : 0;
  constexpr uint64_t BIAS = 0x4081020408102040ull;   // 64 sum_i 128^i, i = 0..8
  const uint64_t sg = (uint64_t)((int64_t)u >> 63);
  return BIAS + ((m ^ sg) - sg);
}

// digits I of two values as a BF16 pair, digit i with its weight 2^(-7 i - 6): the fields under the
// exponent of 128.0 are the numbers 128 + field, exactly (digit 0 reaches +64: field 128, 256.0)
template <int I>
__device__ __forceinline__ uint32_t xg_digit2(uint64_t a, uint64_t b) {
  constexpr uint32_t mask = I == 0 ? 0x00FF00FFu : 0x007F007Fu;
  const uint32_t f = __byte_perm((uint32_t)(a >> (56 - 7 * I)), (uint32_t)(b >> (56 - 7 * I)), 0x5410);
  const uint32_t n = (f & mask) | 0x43004300u;
  const float w = __uint_as_float((uint32_t)(127 - 7 * I - 6) << 23);
  const __nv_bfloat162 w2 = __float2bfloat162_rn(w), o2 = __float2bfloat162_rn(-192.0f * w);
  __nv_bfloat162 r = __hfma2(*reinterpret_cast<const __nv_bfloat162 *>(&n), w2, o2);
  return *reinterpret_cast<uint32_t *>(&r);
}

// the planes of digits I .. D - 1
template <int D, int I = 0>
__device__ __forceinline__ void xg_store(uint8_t *p, int plane, const uint64_t *v) {
  if constexpr (I < D) {
    *(uint4 *)(p + I * plane) = make_uint4(xg_digit2<I>(v[0], v[1]), xg_digit2<I>(v[2], v[3]), xg_digit2<I>(v[4], v[5]),
                                           xg_digit2<I>(v[6], v[7]));
    xg_store<D, I + 1>(p, plane, v);
  }
}

// byte of row r, 16-byte chunk q of a K-major tile of 64-byte rows, SWIZZLE_64B
__device__ __forceinline__ int xg_swz(int r, int q) { return r * 64 + ((q ^ ((r >> 1) & 3)) << 4); }

// Largest exponent of each column of B[K][N] (2^e bounds its values), XG_BAD if a value is not finite
__global__ void __launch_bounds__(256) k_col_exp(int64_t N, int K, const double2 *B, int64_t ldb, int64_t bstride,
                                                 int *cexp) {
  __shared__ int sm[8][32];
  B += blockIdx.y * bstride;
  cexp += blockIdx.y * N;
  const int64_t n = (int64_t)blockIdx.x * 32 + threadIdx.x;
  int e = 0;
  if (n < N)
    for (int k = threadIdx.y; k < K; k += 8) {
      const double2 x = B[(int64_t)k * ldb + n];
      e = max(e, max((__double2hiint(x.x) >> 20) & 0x7ff, (__double2hiint(x.y) >> 20) & 0x7ff));
    }
  sm[threadIdx.y][threadIdx.x] = e;
  __syncthreads();
  if (threadIdx.y == 0 && n < N) {
    for (int y = 1; y < 8; ++y) e = max(e, sm[y][threadIdx.x]);
    cexp[n] = e == 0x7ff ? XG_BAD : max(e, 1) - 1022;
  }
}

// chunk c of up to 32 rows of A: its first row, row count and right-hand side
__device__ __forceinline__ int4 xg_chunk(const int4 *chunks, int M, int rpc, int c) {
  if (chunks) return chunks[c];
  return make_int4(c * rpc, min(rpc, M - c * rpc), 0, 0);
}

// The phases' digit tiles [chunk][stage][XG_DA digits][W rows][64 B, swizzled] (4 W threads):
// MMA row 2 m holds (re, -im) and row 2 m + 1 (im, re) of A[m][cell] along K.
__global__ void __launch_bounds__(256) k_xg_phases(const int4 *chunks, int M, int rpc, int W, int K, int kch,
                                                   const double2 *A, int64_t lda, uint8_t *dig, int *bad) {
  const int r = threadIdx.x >> 2, q = threadIdx.x & 3;   // MMA row, 16-byte chunk (4 cells)
  const int kc = blockIdx.x, mc = blockIdx.y;
  const int4 ch = xg_chunk(chunks, M, rpc, mc);
  const int m = ch.x + (r >> 1);
  uint64_t v[8];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int k = kc * XG_CELLS + 4 * q + c;
    double2 a = make_double2(0.0, 0.0);
    if ((r >> 1) < ch.y && k < K) a = A[(int64_t)m * lda + k];
    // a product of three table entries may round to a few units above 1; anything else beyond is no phase
    // (a non-finite k) and the row's results are NaN
    constexpr long long ONE = 0x3ff0000000000000ll, ABS = 0x7fffffffffffffffll;
    const long long ax = __double_as_longlong(a.x) & ABS, ay = __double_as_longlong(a.y) & ABS;
    if (ax > ONE || ay > ONE) {
      if (ax > ONE + 64 || ay > ONE + 64) bad[m] = 1;
      if (ax > ONE) a.x = copysign(1.0, a.x);
      if (ay > ONE) a.y = copysign(1.0, a.y);
    }
    v[2 * c] = xg_fixed((r & 1) ? a.y : a.x, 0);
    v[2 * c + 1] = xg_fixed((r & 1) ? a.x : -a.y, 0);
  }
  xg_store<XG_DA>(dig + ((size_t)mc * kch + kc) * (XG_DA * 64 * W) + xg_swz(r, q), 64 * W, v);
}

// 2^e sum_l 2^(-7 l - 12) S_l, rounded once, in integer arithmetic: eight FP64 operations a value
// on GB300's FP64 pipe had made the drain a fifth of a tile's time
__device__ __forceinline__ double xg_value(const int *s, int e) {
  if (e == XG_BAD) return __longlong_as_double(0x7ff8000000000000ll);
  const long long hi = (long long)s[0] * (1 << 21) + (long long)s[1] * (1 << 14) + (long long)s[2] * 128 + s[3];
  const long long lo = (long long)s[4] * (1 << 28) + (long long)s[5] * (1 << 21) + (long long)s[6] * (1 << 14) +
                       (long long)s[7] * 128 + s[8];
  constexpr int LB = 35;
  constexpr uint64_t LM = (1ull << LB) - 1;
  long long h = hi + (lo >> LB);                     // the sum is 2^-68 (h 2^35 + l), 0 <= l < 2^35
  uint64_t l = (uint64_t)lo & LM;
  const bool neg = h < 0;
  if (neg) {
    h = ~h + (l == 0);
    l = (0 - l) & LM;
  }
  if (h == 0 && l == 0) return 0.0;
  // leading bit to bit 63 (z places above where h's bit 63 has it)
  const int z = h ? __clzll(h) : __clzll((long long)l) + LB;
  uint64_t m;
  if (z <= LB) m = ((uint64_t)h << z) | (l >> (LB - z));
  else m = (h ? (uint64_t)h << z : 0) | (l << (z - LB));
  const uint64_t m53 = (m >> 11) + ((m >> 10) & 1);  // 53 bits, rounded to nearest
  const int ex = e + 1052 - z;                       // value m53 2^(ex - 1074)
  if (ex < 1 || ex > 2044) return (neg ? -1.0 : 1.0) * ldexp((double)m53, ex - 1074);
  return __longlong_as_double((long long)(((uint64_t)ex << 52) + m53) | (neg ? (long long)0x8000000000000000ull : 0));
}

struct XgArgs {
  int M, K, kch, mch;
  int rpc;                      // rows per chunk
  const int4 *chunks;           // null: one right-hand side, rows in order
  int64_t N, ldb, ldc, bstride; // bstride: values between right-hand sides
  int64_t estride;              // exponents per right-hand side
  int64_t units;                // (tile of B, chunk of A), chunks fastest
  const double2 *B;
  const uint8_t *dig;
  const int *cexp, *bad;
  double2 *C;
  int *err;
};

// kind::f16 with BF16 operands, FP32 accumulators, K-major, M = 128
__device__ constexpr uint32_t idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(XG_ROWS >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
          d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

// One K step: digit I of the tall operand with the phases' digits J.., up to 256 columns of
// adjacent levels per MMA.  All addresses and descriptors are constants off two bases:
// the issuing thread had been slower than the tensor core with them formed in loops.
template <int W, int I = 0, int J = 0>
__device__ __forceinline__ void xg_products(uint32_t tmem, uint64_t b, uint64_t a, uint32_t more) {
  constexpr int end = XG_LEVELS - I;
  constexpr int n = end - J < 256 / W ? end - J : 256 / W;
  umma_bf16(tmem + (I + J) * W, b + I * (XG_PLANE_B >> 4), a + J * (W * 4), idesc_bf16(n * W), I ? 1u : more);
  if constexpr (J + n < end) {
    xg_products<W, I, J + n>(tmem, b, a, more);
  } else if constexpr (I + 1 < XG_LEVELS) {
    xg_products<W, I + 1, 0>(tmem, b, a, more);
  } else {   // level 8 into level 7's accumulator
#pragma unroll
    for (int i = 1; i < XG_D; ++i)
      umma_bf16(tmem + 7 * W, b + i * (XG_PLANE_B >> 4), a + (8 - i) * (W * 4), idesc_bf16(W), 1u);
  }
}

__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

template <int W>
__global__ void __launch_bounds__(XG_THREADS, 1) k_xgemm(XgArgs g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *full = (uint64_t *)(smem + XG_STAGES * XG_STAGE);
  uint64_t *empty = full + XG_STAGES;
  uint64_t *tfull = empty + XG_STAGES;
  uint64_t *tempty = tfull + 1;
  uint64_t *drain = tempty + 1;
  uint32_t *tslot = (uint32_t *)(drain + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < XG_STAGES; ++s) {
      mbar_init(&full[s], XG_CONV + 1);   // the converters and the phases' bulk copy
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, XG_EPI);
    mbar_init(drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;

  if (warp == 0) {
    if (lane == 0) {   // ---- the phases' digit tiles
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int64_t u = blockIdx.x; u < g.units && ok; u += gridDim.x) {
        const uint32_t bytes = XG_DA * 64 * W;
        const uint8_t *src = g.dig + (size_t)(u % g.mch) * g.kch * bytes;
        for (int kc = 0; kc < g.kch; ++kc) {
          if (!mbar_wait(&empty[stage], phase ^ 1, g.err)) { ok = false; break; }
          mbar_expect_tx(&full[stage], bytes);
          bulk_load(smem + stage * XG_STAGE + XG_STAGE_B, src + (size_t)kc * bytes, bytes, &full[stage]);
          if (++stage == XG_STAGES) { stage = 0; phase ^= 1; }
        }
      }
      // every issued stage has landed and been read before the CTA can exit
      for (int s = 0; s < XG_STAGES; ++s) mbar_wait(&empty[stage], phase ^ 1, g.err), stage = (stage + 1) % XG_STAGES,
                                            phase ^= (stage == 0);
    }
  } else if (warp == 1) {
    if (lane == 0) {   // ---- MMA issuer
      int stage = 0, it = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int64_t u = blockIdx.x; u < g.units && ok; u += gridDim.x) {
        for (int k0 = 0; k0 < g.kch && ok; k0 += XG_KGROUP, ++it) {
          if (!mbar_wait(tempty, (it & 1) ^ 1, g.err)) { ok = false; break; }
          tc_fence_after();
          const int k1 = min(g.kch, k0 + XG_KGROUP);
          for (int kc = k0; kc < k1; ++kc) {
            if (!mbar_wait(&full[stage], phase, g.err)) { ok = false; break; }
            tc_fence_after();
            const uint64_t bd = sdesc(smem + stage * XG_STAGE), ad = sdesc(smem + stage * XG_STAGE + XG_STAGE_B);
#pragma unroll
            for (int ks = 0; ks < XG_KV / 16; ++ks) {   // addresses in the descriptors count 16 bytes
              const uint64_t bk = bd + 2 * ks, ak = ad + 2 * ks;
              const uint32_t more = (kc > k0 || ks > 0) ? 1u : 0u;
              xg_products<W>(tmem, bk, ak, more);
            }
            umma_commit(&empty[stage]);
            if (++stage == XG_STAGES) { stage = 0; phase ^= 1; }
          }
          if (ok) umma_commit(tfull);
        }
      }
      // a wait gave up: let the MMAs already issued retire before TMEM is freed
      if (!ok) {
        umma_commit(drain);
        mbar_wait(drain, 0, g.err);
      }
    }
  } else if (warp < 2 + XG_CONV / 32) {   // ---- converters: B's digits of a stage, one 16-byte chunk of each plane per thread
    const int t = threadIdx.x - 64, r = t & 127, q = t >> 7;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int64_t u = blockIdx.x; u < g.units && ok; u += gridDim.x) {
      const int64_t n = (u / g.mch) * XG_ROWS + r;
      const int64_t rhs = xg_chunk(g.chunks, g.M, g.rpc, (int)(u % g.mch)).z;
      const bool live = n < g.N;
      int e = live ? g.cexp[rhs * g.estride + n] : 0;
      if (e == XG_BAD) e = 1024;   // the results are NaN; any finite digits do
      const double2 *col = g.B + rhs * g.bstride + n;
      double2 next[4];   // the next stage's values are in flight while this one's are split
      auto fetch = [&](int kc) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int k = kc * XG_CELLS + 4 * q + c;
          next[c] = live && k < g.K ? col[(int64_t)k * g.ldb] : make_double2(0.0, 0.0);
        }
      };
      fetch(0);
      for (int kc = 0; kc < g.kch; ++kc) {
        uint64_t v[8];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          v[2 * c] = xg_fixed(next[c].x, e);
          v[2 * c + 1] = xg_fixed(next[c].y, e);
        }
        if (kc + 1 < g.kch) fetch(kc + 1);
        if (!mbar_wait(&empty[stage], phase ^ 1, g.err)) { ok = false; break; }
        xg_store<XG_D>(smem + stage * XG_STAGE + xg_swz(r, q), XG_PLANE_B, v);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_arrive(&full[stage]);
        if (++stage == XG_STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else {   // ---- epilogue: warp w reads TMEM lane quadrant w % 4, a thread every other 4 of a column's results
    const int quad = warp & 3, half = (warp - 2 - XG_CONV / 32) >> 2;
    const uint32_t tr = tmem + ((uint32_t)(quad * 32) << 16);
    int it = 0;
    bool ok = true;
    for (int64_t u = blockIdx.x; u < g.units && ok; u += gridDim.x) {
      const int4 ch = xg_chunk(g.chunks, g.M, g.rpc, (int)(u % g.mch));
      const int mrows = ch.y;
      const int64_t n = (u / g.mch) * XG_ROWS + quad * 32 + lane;
      const bool live = n < g.N;
      const int e = live ? g.cexp[ch.z * g.estride + n] : 0;
      const unsigned badm = __ballot_sync(0xffffffffu, lane < mrows && g.bad[ch.x + lane]);
      for (int k0 = 0; k0 < g.kch; k0 += XG_KGROUP, ++it) {
        if (!mbar_wait(tfull, it & 1, g.err)) { ok = false; break; }
        tc_fence_after();
#pragma unroll 1
        for (int c0 = 4 * half; c0 < 2 * mrows; c0 += 8) {
          uint32_t a[XG_LEVELS][4];
          __syncwarp();
#pragma unroll
          for (int l = 0; l < XG_LEVELS; ++l) tmem_ld4_nowait(tr + l * W + c0, a[l]);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 4; c += 2) {
            double2 z;
#pragma unroll
            for (int y = 0; y < 2; ++y) {
              int s[XG_D];
#pragma unroll
              for (int l = 0; l < XG_LEVELS; ++l)   // S_l; the last accumulator holds levels 7 and 8
                s[l] = __float2int_rn(__uint_as_float(a[l][c + y]) *
                                      __uint_as_float((uint32_t)(127 + 7 * l + 12) << 23));
              s[8] = __float2int_rn(128.0f * (__uint_as_float(a[7][c + y]) * 0x1p61f - (float)s[7]));
              (y ? z.y : z.x) = xg_value(s, e);
            }
            const int m = ch.x + (c0 + c) / 2;
            if (live && c0 + c < 2 * mrows) {
              if (badm >> ((c0 + c) / 2) & 1) z.x = z.y = __longlong_as_double(0x7ff8000000000000ll);
              double2 *o = g.C + (int64_t)m * g.ldc + n;
              if (k0) {
                const double2 p = *o;
                z.x += p.x;
                z.y += p.y;
              }
              *o = z;
            }
          }
        }
        tc_fence_before();
        mbar_arrive(tempty);
      }
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

static void col_exp(int64_t nrhs, int64_t N, int K, const double2 *B, int64_t ldb, int64_t bstride, int *cexp,
                    cudaStream_t st) {
  for (int64_t b = 0; b < nrhs; b += 32768)   // grid.y
    k_col_exp<<<dim3((unsigned)((N + 31) / 32), (unsigned)std::min<int64_t>(nrhs - b, 32768)), dim3(32, 8), 0, st>>>(
        N, K, B + b * bstride, ldb, bstride, cexp + b * N);
}

int xgemm_colexp(Workspace &ws, int64_t nrhs, int64_t N, int K, const double2 *B, int64_t bstride, const int **cexp,
                 cudaStream_t st) {
  int *e;
  const int rc = wsget(ws, "x_exp", (size_t)(nrhs * N), &e);
  if (rc) return rc;
  col_exp(nrhs, N, K, B, N, bstride, e, st);
  *cexp = e;
  return EPHG_OK;
}

void launch_colexp(int64_t N, int K, const double2 *B, int *e, cudaStream_t st) {
  col_exp(1, N, K, B, N, 0, e, st);
}

template <int W>
static void xg_run(const XgArgs &g, cudaStream_t st) {
  static OncePerDevice attr;
  attr([] { cudaFuncSetAttribute(k_xgemm<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, XG_SMEM); });
  k_xgemm<W><<<(unsigned)std::min<int64_t>(g.units, num_sms()), XG_THREADS, XG_SMEM, st>>>(g);
}

// MMA columns of a level for chunks of up to `rows` rows
static int xg_width(int rows) { return (2 * rows + 15) / 16 * 16; }

int64_t xgemm_chunk_bytes(int most, int K) {
  return (int64_t)((K + XG_CELLS - 1) / XG_CELLS) * XG_DA * 64 * xg_width(most);
}

// one launch over mch chunks (dig sized for them)
static void xg_launch(XgArgs &g, const double2 *A, int64_t lda, uint8_t *dig, int *bad, cudaStream_t st) {
  g.dig = dig;
  g.bad = bad;
  g.units = (g.N + XG_ROWS - 1) / XG_ROWS * g.mch;
  const int W = xg_width(g.rpc);
  k_xg_phases<<<dim3(g.kch, g.mch), 4 * W, 0, st>>>(g.chunks, g.M, g.rpc, W, g.K, g.kch, A, lda, dig, bad);
  W == 16 ? xg_run<16>(g, st) : W == 32 ? xg_run<32>(g, st) : W == 48 ? xg_run<48>(g, st) : xg_run<64>(g, st);
}

int launch_xgemm(Workspace &ws, int M, int64_t N, int K, const double2 *A, int64_t lda, const double2 *B, int64_t ldb,
                 const int *cexp, double2 *C, int64_t ldc, int *err, cudaStream_t st) {
  if (M <= 0 || N <= 0) return EPHG_OK;
  const int kch = (K + XG_CELLS - 1) / XG_CELLS, mb = std::min(M, XG_BATCH);
  uint8_t *dig;
  int *bad, *ce = nullptr;
  int rc;
  if ((rc = wsget(ws, "x_dig", (size_t)((mb + XG_M - 1) / XG_M) * kch * XG_STAGE_A, &dig)) ||
      (rc = wsget(ws, "x_bad", (size_t)M, &bad)) || (!cexp && (rc = wsget(ws, "x_exp", (size_t)N, &ce))))
    return rc;
  if (!cexp) {
    col_exp(1, N, K, B, ldb, 0, ce, st);
    cexp = ce;
  }
  cudaMemsetAsync(bad, 0, (size_t)M * sizeof(int), st);
  for (int m0 = 0; m0 < M; m0 += XG_BATCH) {
    XgArgs g{};
    g.M = std::min(XG_BATCH, M - m0);
    g.K = K;
    g.kch = kch;
    g.mch = (g.M + XG_M - 1) / XG_M;
    g.rpc = (g.M + g.mch - 1) / g.mch;   // even chunks
    g.N = N;
    g.ldb = ldb;
    g.ldc = ldc;
    g.B = B;
    g.cexp = cexp;
    g.C = C + (int64_t)m0 * ldc;
    g.err = err;
    xg_launch(g, A + (int64_t)m0 * lda, lda, dig, bad + m0, st);
  }
  if (cudaGetLastError() != cudaSuccess) {
    ws.msg = "xgemm: launch failed";
    return EPHG_ERR_CUDA;
  }
  return EPHG_OK;
}

int launch_xgemm_chunks(Workspace &ws, const int4 *chunks, int nchunks, int most, int rows, int64_t N, int K, const double2 *A,
                        int64_t lda, const double2 *B, int64_t ldb, int64_t bstride, const int *cexp, double2 *C,
                        int64_t ldc, int *err, cudaStream_t st) {
  if (nchunks <= 0) return EPHG_OK;
  const int kch = (K + XG_CELLS - 1) / XG_CELLS;
  uint8_t *dig;
  int *bad;
  int rc;
  if ((rc = wsget(ws, "x_dig", (size_t)(nchunks * xgemm_chunk_bytes(most, K)), &dig)) ||
      (rc = wsget(ws, "x_bad", (size_t)rows, &bad)))
    return rc;
  cudaMemsetAsync(bad, 0, (size_t)rows * sizeof(int), st);
  XgArgs g{};
  g.chunks = chunks;
  g.K = K;
  g.kch = kch;
  g.mch = nchunks;
  g.rpc = most;
  g.N = N;
  g.ldb = ldb;
  g.ldc = ldc;
  g.bstride = bstride;
  g.estride = ldb;
  g.B = B;
  g.cexp = cexp;
  g.C = C;
  g.err = err;
  xg_launch(g, A, lda, dig, bad, st);
  if (cudaGetLastError() != cudaSuccess) {
    ws.msg = "xgemm: launch failed";
    return EPHG_ERR_CUDA;
  }
  return EPHG_OK;
}

}  // namespace ephg
