// sp_solve.h -- FP64 Gram, Cholesky factorisation and triangular solves of the
// ridge readout on the FP64 tensor cores (dev_solve.cu).
//
// Matrices are row-major with a pitch of sp_solve_pad(n) doubles; the
// factorisation works on the padded matrix, whose rows and columns from n on
// sp_solve_diag sets to the identity. Everything is enqueued on the stream; no
// call allocates or waits.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>

constexpr int kSolveBlock = 64;

inline int sp_solve_pad(int n) { return (n + kSolveBlock - 1) / kSolveBlock * kSolveBlock; }

// Work area of a factorisation and its solves: the inverses of the 16 x 16
// diagonal blocks of L, then the flags.
inline size_t sp_solve_work_bytes(int n)
{
    const size_t nb = (size_t)sp_solve_pad(n) / kSolveBlock;
    return nb * 4 * 256 * sizeof(double) + (nb * nb + 2 * nb + 4) * sizeof(int);
}

// C (n x n, pitch ldc) = X^T X over rows [t0, t1) of X (rows of n doubles); the
// full matrix is written.
cudaError_t sp_solve_gram(cudaStream_t s, const double *X, int n, size_t t0, size_t t1, double *C,
                          int ldc);
// The same row range by row range, in order: `more` continues the sums in C's lower
// triangle where the rows so far (a multiple of four) ended, with the same bits as
// one call over all rows; the upper triangle comes with `last`. Only for the n and
// rows in all that sp_solve_gram sums in one part.
bool sp_solve_gram_in_ranges(int n, size_t rows);
cudaError_t sp_solve_gram_range(cudaStream_t s, const double *X, int n, size_t t0, size_t t1,
                                double *C, int ldc, bool more, bool last);
// A += lambda I, and the identity in rows and columns n .. pad(n) - 1.
cudaError_t sp_solve_diag(cudaStream_t s, double *A, int n, double lambda);
// One system: A (then its factor), its work area, right-hand sides Z (n x dout,
// dout <= 16) and an error word.
struct sp_solve_item {
    double *A;
    int n;
    void *work;
    double *Z;
    int dout;
    int *info;
};
// A = L L^T in place (lower triangle) of every item. *info (zero before) becomes
// the 1-based index of a pivot that is not positive, or -1 when a wait ran out.
cudaError_t sp_solve_factor(cudaStream_t s, const sp_solve_item *items, int count);
// L L^T Z = Z in place of every item.
cudaError_t sp_solve_apply(cudaStream_t s, const sp_solve_item *items, int count);

inline cudaError_t sp_solve_factor(cudaStream_t s, double *A, int n, void *work, int *info)
{
    const sp_solve_item it = {A, n, work, nullptr, 0, info};
    return sp_solve_factor(s, &it, 1);
}
inline cudaError_t sp_solve_apply(cudaStream_t s, double *L, int n, void *work, double *Z,
                                  int dout, int *info)
{
    const sp_solve_item it = {L, n, work, Z, dout, info};
    return sp_solve_apply(s, &it, 1);
}
