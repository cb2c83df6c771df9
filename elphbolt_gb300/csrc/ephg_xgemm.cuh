// ephg_xgemm.cuh - FP64 complex products on the tensor cores by exact splitting.
#pragma once
#include "ephg_ws.cuh"

namespace ephg {

// C[M][N] = A[M][K] B[K][N], complex FP64, row-major, |A| <= 1 (phases).  cexp: B's column
// exponents (nullable: formed per call in ws).  err: device error word of the bounded waits.
// Returns 0, or an EPHG_ERR code with ws.msg set.
int launch_xgemm(Workspace &ws, int M, int64_t N, int K, const double2 *A, int64_t lda, const double2 *B, int64_t ldb,
                 const int *cexp, double2 *C, int64_t ldc, int *err, cudaStream_t st);
// Cycles of one SM for 128 columns of a product of M rows: chunks of up to 32 rows, each splitting
// B's K values anew.  Fitted to launches that fill the chip (43 to 279 cells, 150 to 2,500 rows).
inline double xgemm_cycles(int64_t M, int K) { return (double)((M + 31) / 32) * (25000.0 + 4000.0 * ((K + 15) / 16)); }
// Rows of A against several right-hand sides in one launch: chunk c (device) is (first row, rows
// <= most <= XG_CHUNK, right-hand side); right-hand side b is B + b bstride, [K][N] at row stride ldb.
// cexp: the exponents of xgemm_colexp, ldb per right-hand side.  The phases' digits take
// xgemm_chunk_bytes per chunk; at most XG_MAXCHUNKS chunks.
constexpr int XG_CHUNK = 32, XG_MAXCHUNKS = 32768;
int64_t xgemm_chunk_bytes(int most, int K);
int xgemm_colexp(Workspace &ws, int64_t nrhs, int64_t N, int K, const double2 *B, int64_t bstride, const int **cexp,
                 cudaStream_t st);
int launch_xgemm_chunks(Workspace &ws, const int4 *chunks, int nchunks, int most, int rows, int64_t N, int K, const double2 *A,
                        int64_t lda, const double2 *B, int64_t ldb, int64_t bstride, const int *cexp, double2 *C, int64_t ldc,
                        int *err, cudaStream_t st);
// The exponents of an operand B[K][N] that its owner keeps (into e, N values), in stream order.
void launch_colexp(int64_t N, int K, const double2 *B, int *e, cudaStream_t st);

}  // namespace ephg
