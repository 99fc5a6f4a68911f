// dev_readout.cu -- readout training on the device.
//
//   ridge  (src/reservoir.c:573-679): reset, record Phi[T][N] (no washout unless
//          asked), A = Phi^T Phi + lambda I, B = Phi^T Y, solve A W = B.
//          The reference forms A with dgemm and solves one LU (dgesv) per
//          output; here A is factored once by a blocked Cholesky in FP64 and
//          all outputs are solved together, followed by iterative refinement
//          whose residual R = Phi^T (Y - Phi W) - lambda W is formed from the
//          FP64 Phi itself. A non-positive pivot falls back to LU with partial
//          pivoting, which is what dgesv does.
//   RLS    (src/reservoir.c:681-767) and the online delta rule
//          (src/reservoir.c:244-280), with W_out and P resident on the device.
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include <mutex>
#include <cmath>
#include <chrono>
#include "sp_alloc.h"
#include "sp_stage.h"
#include "sp_dev.h"
#include "sp_kernels.cuh"
#include "sp_dev_internal.h"
#include "sp_gram.h"
#include "sp_solve.h"

using namespace sp;

#define RK(x)                                                                      \
    do {                                                                           \
        cudaError_t e_ = (x);                                                      \
        if (e_ != cudaSuccess) {                                                   \
            sp_dev_note_error(#x, e_);                                             \
            rc = (e_ == cudaErrorMemoryAllocation) ? SP_EALLOC : SP_EINTERNAL;     \
            goto out;                                                              \
        }                                                                          \
    } while (0)

namespace {

// R[i][o] = sum_{t in [t0,t1)} X[t][i] E[t][o] (- lam * W[i][o] when W != 0),
// split over `parts` contiguous t ranges reduced in a fixed order.
__global__ void k_xt_e_part(const double *__restrict__ X, int n, size_t t0, size_t t1,
                            const double *__restrict__ E, int dout, int parts,
                            double *__restrict__ part)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int pidx = blockIdx.y;
    const size_t len = t1 - t0;
    const size_t a = t0 + len * pidx / parts, b = t0 + len * (pidx + 1) / parts;
    if (i >= n)
        return;
    double acc[16];
    for (int o = 0; o < dout; ++o)
        acc[o] = 0.0;
    for (size_t t = a; t < b; ++t) {
        double x = X[t * n + i];
        for (int o = 0; o < dout; ++o)
            acc[o] = fma(x, E[t * dout + o], acc[o]);
    }
    for (int o = 0; o < dout; ++o)
        part[((size_t)pidx * n + i) * dout + o] = acc[o];
}

__global__ void k_reduce_parts(const double *__restrict__ part, int parts, int n, int dout,
                               const double *__restrict__ W, double lam, double *__restrict__ R)
{
    const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t total = (size_t)n * dout;
    if (k >= total)
        return;
    double s = 0.0;
    for (int p = 0; p < parts; ++p)
        s += part[(size_t)p * total + k];
    if (W)
        s -= lam * W[k];
    R[k] = s;
}

// E[t][o] = Y[t][o] - sum_i X[t][i] W[i][o], one warp per row t.
__global__ void k_resid_rows(const double *__restrict__ X, int n, size_t t0, size_t t1,
                             const double *__restrict__ Y, const double *__restrict__ W,
                             int dout, double *__restrict__ E)
{
    const size_t t = t0 + (size_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= t1)
        return;
    double acc[16];
    for (int o = 0; o < dout; ++o)
        acc[o] = 0.0;
    for (int i = lane; i < n; i += 32) {
        double x = X[t * n + i];
        for (int o = 0; o < dout; ++o)
            acc[o] = fma(x, W[(size_t)i * dout + o], acc[o]);
    }
    for (int o = 0; o < dout; ++o) {
        double s = acc[o];
        for (int off = 16; off; off >>= 1)
            s += __shfl_xor_sync(kFull, s, off);
        if (lane == 0)
            E[t * dout + o] = Y[t * dout + o] - s;
    }
}

// Pt[k][t - t0] = X[t][k] for rows [t0, t1) of X (T x n): 32 x 32 tiles
// through shared memory, both sides coalesced.
__global__ void k_rows_to_cols(const double *__restrict__ X, int n, size_t t0, size_t t1,
                               double *__restrict__ Pt)
{
    __shared__ double tile[32][33];
    const size_t tw = t1 - t0;
    const size_t tb = (size_t)blockIdx.y * 32, kb = (size_t)blockIdx.x * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const size_t t = tb + r, k = kb + threadIdx.x;
        tile[r][threadIdx.x] = (t < tw && k < (size_t)n) ? X[(t0 + t) * n + k] : 0.0;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const size_t k = kb + r, t = tb + threadIdx.x;
        if (k < (size_t)n && t < tw)
            Pt[k * tw + t] = tile[threadIdx.x][r];
    }
}

__global__ void k_add_diag(double *A, int n, int lda, double lam)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        A[(size_t)i * lda + i] += lam;
}

// ------------------------------------------------ LU with partial pivoting
// Unblocked right-looking LU, one column per step (fallback path only).
__global__ void k_lu_pivot(double *A, int n, int lda, int j, int *piv, int *info)
{
    __shared__ double bv[256];
    __shared__ int bi[256];
    double best = -1.0;
    int idx = j;
    for (int r = j + threadIdx.x; r < n; r += blockDim.x) {
        double v = fabs(A[(size_t)r * lda + j]);
        if (v > best) {
            best = v;
            idx = r;
        }
    }
    bv[threadIdx.x] = best;
    bi[threadIdx.x] = idx;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            double o = bv[threadIdx.x + s];
            int oi = bi[threadIdx.x + s];
            if (o > bv[threadIdx.x] || (o == bv[threadIdx.x] && oi < bi[threadIdx.x])) {
                bv[threadIdx.x] = o;
                bi[threadIdx.x] = oi;
            }
        }
        __syncthreads();
    }
    const int p = bi[0];
    if (threadIdx.x == 0) {
        piv[j] = p;
        if (A[(size_t)p * lda + j] == 0.0 && *info == 0)
            *info = j + 1;
    }
    if (p != j)
        for (int c = threadIdx.x; c < n; c += blockDim.x) {
            double t = A[(size_t)j * lda + c];
            A[(size_t)j * lda + c] = A[(size_t)p * lda + c];
            A[(size_t)p * lda + c] = t;
        }
}

__global__ void k_lu_update(double *A, int n, int lda, int j)
{
    const double pv = A[(size_t)j * lda + j];
    if (pv == 0.0)
        return;
    for (int r = j + 1 + blockIdx.x; r < n; r += gridDim.x) {
        const double l = A[(size_t)r * lda + j] / pv;
        __syncthreads();
        if (threadIdx.x == 0)
            A[(size_t)r * lda + j] = l;
        for (int c = j + 1 + threadIdx.x; c < n; c += blockDim.x)
            A[(size_t)r * lda + c] -= l * A[(size_t)j * lda + c];
    }
}

__global__ void k_lu_solve(const double *A, int n, int lda, const int *piv, double *Z, int dout)
{
    const int o = blockIdx.x;
    if (o >= dout)
        return;
    if (threadIdx.x == 0) {
        for (int j = 0; j < n; ++j) {
            int p = piv[j];
            if (p != j) {
                double t = Z[(size_t)j * dout + o];
                Z[(size_t)j * dout + o] = Z[(size_t)p * dout + o];
                Z[(size_t)p * dout + o] = t;
            }
        }
        for (int r = 0; r < n; ++r) {
            double v = Z[(size_t)r * dout + o];
            for (int c = 0; c < r; ++c)
                v -= A[(size_t)r * lda + c] * Z[(size_t)c * dout + o];
            Z[(size_t)r * dout + o] = v;
        }
        for (int r = n - 1; r >= 0; --r) {
            double v = Z[(size_t)r * dout + o];
            for (int c = r + 1; c < n; ++c)
                v -= A[(size_t)r * lda + c] * Z[(size_t)c * dout + o];
            Z[(size_t)r * dout + o] = v / A[(size_t)r * lda + r];
        }
    }
}

__global__ void k_axpy(double *y, const double *x, size_t cnt)
{
    size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < cnt)
        y[k] += x[k];
}

// W (n x dout) -> W_out (dout x n)
__global__ void k_transpose_w(const double *W, int n, int dout, double *W_out)
{
    size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < (size_t)n * dout) {
        int i = (int)(k / dout), o = (int)(k % dout);
        W_out[(size_t)o * n + i] = W[k];
    }
}

__global__ void k_sumsq(const double *x, size_t cnt, double *out)
{
    __shared__ double s[256];
    double a = 0.0;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < cnt;
         k += (size_t)gridDim.x * blockDim.x)
        a = fma(x[k], x[k], a);
    s[threadIdx.x] = a;
    __syncthreads();
    for (int st = 128; st; st >>= 1) {
        if (threadIdx.x < st)
            s[threadIdx.x] += s[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        atomicAdd(out, s[0]);
}

// ------------------------------------------------------------------- RLS
// Px = P x
__global__ void k_gemv_rows(const double *__restrict__ P, int n, const double *__restrict__ x,
                            double *__restrict__ y)
{
    const int r = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= n)
        return;
    double s = 0.0;
    for (int c = lane; c < n; c += 32)
        s = fma(P[(size_t)r * n + c], x[c], s);
    for (int off = 16; off; off >>= 1)
        s += __shfl_xor_sync(kFull, s, off);
    if (lane == 0)
        y[r] = s;
}

// scalars: denom = lambda + x.Px ; e = target - W_out x ; k = Px / denom
__global__ void k_rls_scalars(const double *x, const double *Px, int n, double lambda,
                              const double *W_out, int dout, const double *target,
                              double *scal /* [0]=denom, [1..dout]=e */)
{
    __shared__ double red[256];
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        s = fma(x[i], Px[i], s);
    red[threadIdx.x] = s;
    __syncthreads();
    for (int st = 128; st; st >>= 1) {
        if (threadIdx.x < st)
            red[threadIdx.x] += red[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        scal[0] = lambda + red[0];
    __syncthreads();
    for (int o = 0; o < dout; ++o) {
        double a = 0.0;
        for (int i = threadIdx.x; i < n; i += blockDim.x)
            a = fma(W_out[(size_t)o * n + i], x[i], a);
        red[threadIdx.x] = a;
        __syncthreads();
        for (int st = 128; st; st >>= 1) {
            if (threadIdx.x < st)
                red[threadIdx.x] += red[threadIdx.x + st];
            __syncthreads();
        }
        if (threadIdx.x == 0)
            scal[1 + o] = target[o] - red[0];
        __syncthreads();
    }
}

// W_out += e k^T ; P = (P - denom k k^T) / lambda   with k = Px / denom
__global__ void k_rls_update(double *P, int n, const double *Px, const double *scal, double lambda,
                             double *W_out, int dout)
{
    const double denom = scal[0];
    const double inv = 1.0 / denom;
    const size_t total = (size_t)n * n;
    const double sc = (lambda != 1.0) ? 1.0 / lambda : 1.0;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < total;
         q += (size_t)gridDim.x * blockDim.x) {
        const int r = (int)(q / n), c = (int)(q % n);
        const double kr = inv * Px[r], kc = inv * Px[c];
        double v = P[q] + kr * (-denom * kc);
        P[q] = (lambda != 1.0) ? sc * v : v;
    }
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < (size_t)dout * n;
         q += (size_t)gridDim.x * blockDim.x) {
        const int o = (int)(q / n), i = (int)(q % n);
        W_out[q] += (inv * Px[i]) * scal[1 + o];
    }
}

__global__ void k_diag_init(double *P, int n, double v)
{
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < (size_t)n * n;
         q += (size_t)gridDim.x * blockDim.x)
        P[q] = ((q / n) == (q % n)) ? v : 0.0;
}

// ------------------------------------------------------ fused RLS recursion
// T steps of the recursion above in one cooperative launch over recorded states
// X [T][n] (the states do not depend on the readout). CTA c owns a block of rows
// of P, in shared memory for the launch where it fits, and a step is one pass
// over them: the rank-one update with the gain of the step before and the
// product with the new state together. The products travel as the step
// kernel's spike words do, each double as two 8-byte entries that carry the
// step's number; every CTA then forms the denominator itself, and output o's
// weights are kept by CTA o % G while the products of the next step are on
// their way. Every product and sum is that of the separate kernels in their
// order, so the bits are theirs. What bounds it: the exchange, about 1 us a
// step, until P no longer fits the SMs' shared memory (about 1700 neurons)
// and streams from the L2 or HBM, read and written once a step. (N=800, 400
// steps: 4.4 us per step beside the 3.1 of a FLIF_GL, L=64 simulation; four
// launches a step took 47 together.)
struct RlsArgs {
    const double *X;           // [T][n] states
    const double *Y;           // [T][dout] targets
    double *P;                 // [n][n], or null: in shared memory only
    double *W;                 // [dout][n]
    unsigned long long *ll;    // [2][n][2] exchange entries, zero before the launch
    int *err;
    size_t T;
    long long step0;           // steps of earlier launches (error reports)
    int n, dout, rows;         // rows of P per CTA
    int resident, first, last; // P in shared memory; first / last launch of the series
    double p0, lambda;         // initial diagonal of P
};

constexpr int kRlsThreads = 256;

// the 256-term tree of k_rls_scalars: pairs 128, 64, 32 apart through shared
// memory, then 16 .. 1 within the first warp; the sum in thread 0's red[0]
__device__ __forceinline__ double rls_tree(double s, double *red)
{
    const int t = threadIdx.x;
    __syncthreads();  // readers of the last tree's red[] are done
    red[t] = s;
    __syncthreads();
    if (t < 128)
        red[t] += red[t + 128];
    __syncthreads();
    if (t < 64)
        red[t] += red[t + 64];
    __syncthreads();
    if (t < 32) {
        double v = red[t] + red[t + 32];
#pragma unroll
        for (int st = 16; st; st >>= 1)
            v += __shfl_down_sync(kFull, v, st);
        if (t == 0)
            red[0] = v;
    }
    __syncthreads();
    return red[0];
}

__global__ void __launch_bounds__(kRlsThreads, 1) k_rls(RlsArgs a)
{
    extern __shared__ __align__(16) double rls_smem[];
    const int n = a.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *s_x = rls_smem;                // [2][n] states of this step and the last
    double *s_px = s_x + 2 * (size_t)n;    // [2][n] P x of this step and the last
    double *s_k = s_px + 2 * (size_t)n;    // [n] -denom * gain of the step before
    double *red = s_k + n;                 // [256]
    double *s_P = red + kRlsThreads;       // [rows][n]
    const int r_lo = blockIdx.x * a.rows < n ? blockIdx.x * a.rows : n;
    const int r_hi = r_lo + a.rows < n ? r_lo + a.rows : n;
    double *P = a.resident ? s_P : a.P + (size_t)r_lo * n;
    const double sc = (a.lambda != 1.0) ? 1.0 / a.lambda : 1.0;

    if (a.resident || a.first)
        for (size_t q = tid; q < (size_t)(r_hi - r_lo) * n; q += kRlsThreads) {
            const int r = r_lo + (int)(q / n), c = (int)(q % n);
            P[q] = a.first ? (r == c ? a.p0 : 0.0) : a.P[(size_t)r * n + c];
        }
    double denom = 0.0, inv = 0.0;  // of the step before
    __syncthreads();
    for (size_t t = 0; t <= a.T; ++t) {
        double *x = s_x + (t & 1) * (size_t)n, *px = s_px + (t & 1) * (size_t)n;
        const double *xp = s_x + (~t & 1) * (size_t)n, *pxp = s_px + (~t & 1) * (size_t)n;
        const bool more = t < a.T;
        if (!more && a.last && (int)blockIdx.x >= a.dout)
            break;  // nothing reads P any more, and this CTA keeps no weights
        for (int i = tid; i < n; i += kRlsThreads) {
            if (more)
                x[i] = __ldg(a.X + t * n + i);
            if (t > 0) {
                const double kc = inv * pxp[i];
                s_k[i] = -denom * kc;
            }
        }
        __syncthreads();
        // rows: a warp each
        for (int r = r_lo + warp; r < r_hi; r += kRlsThreads / 32) {
            double *row = P + (size_t)(r - r_lo) * n;
            double s = 0.0;
            const double kr = t > 0 ? inv * pxp[r] : 0.0;
            // eight elements a pass, their loads ahead of the stores
            for (int c = lane; c < n; c += 256) {
                double v[8], g[8], y[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const bool in = c + 32 * u < n;
                    v[u] = in ? row[c + 32 * u] : 0.0;
                    g[u] = in && t > 0 ? s_k[c + 32 * u] : 0.0;
                    y[u] = in && more ? x[c + 32 * u] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    if (c + 32 * u >= n)
                        break;
                    if (t > 0) {
                        v[u] = v[u] + kr * g[u];
                        v[u] = (a.lambda != 1.0) ? sc * v[u] : v[u];
                        row[c + 32 * u] = v[u];
                    }
                    s = fma(v[u], y[u], s);
                }
            }
            if (!more)
                continue;
            for (int off = 16; off; off >>= 1)
                s += __shfl_xor_sync(kFull, s, off);
            if (lane < 2) {
                const unsigned long long bits = (unsigned long long)__double_as_longlong(s);
                const unsigned half = lane ? (unsigned)(bits >> 32) : (unsigned)bits;
                *(volatile unsigned long long *)(a.ll + ((t & 1) * (size_t)n + r) * 2 + lane) =
                    ((unsigned long long)(unsigned)(t + 1) << 32) | half;
            }
        }
        // output weights of the step before
        if (t > 0)
            for (int o = blockIdx.x; o < a.dout; o += gridDim.x) {
                double *w = a.W + (size_t)o * n;
                double d = 0.0;
                for (int i = tid; i < n; i += kRlsThreads)
                    d = fma(w[i], xp[i], d);
                const double e = __ldg(a.Y + (t - 1) * a.dout + o) - rls_tree(d, red);
                for (int i = tid; i < n; i += kRlsThreads)
                    w[i] += (inv * pxp[i]) * e;
            }
        if (!more)
            break;
        // all products of this step
        bool ok = true;
        const unsigned want = (unsigned)(t + 1);
        const unsigned long long *src = a.ll + (t & 1) * (size_t)n * 2;
        unsigned long long t0 = 0, polls = 0;
        for (int base = tid; base < n && ok; base += 4 * kRlsThreads) {
            unsigned pend = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (base + u * kRlsThreads < n)
                    pend |= 1u << u;
            while (pend) {
                unsigned long long v[4][2];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if ((pend >> u) & 1u) {
                        const unsigned long long *e = src + 2 * (size_t)(base + u * kRlsThreads);
                        v[u][0] = ld_volatile_u64(e);
                        v[u][1] = ld_volatile_u64(e + 1);
                    }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (((pend >> u) & 1u) && (unsigned)(v[u][0] >> 32) == want &&
                        (unsigned)(v[u][1] >> 32) == want) {
                        px[base + u * kRlsThreads] = __longlong_as_double(
                            (long long)((v[u][1] << 32) | (v[u][0] & 0xffffffffull)));
                        pend &= ~(1u << u);
                    }
                if (pend && (++polls & 63ull) == 0) {
                    const unsigned long long now = globaltimer_ns();
                    if (t0 == 0)
                        t0 = now;
                    if (ld_volatile_i32(a.err) != kErrNone || now - t0 > kBarrierTimeoutNs) {
                        if (atomicCAS(a.err, kErrNone, kErrBarrierTimeout) == kErrNone)
                            a.err[1] = (int)(a.step0 + (long long)t);
                        ok = false;
                        break;
                    }
                }
            }
        }
        if (__syncthreads_or(!ok))
            return;
        double s = 0.0;
        for (int i = tid; i < n; i += kRlsThreads)
            s = fma(x[i], px[i], s);
        denom = a.lambda + rls_tree(s, red);
        inv = 1.0 / denom;
    }
    if (a.resident && !a.last)
        for (size_t q = tid; q < (size_t)(r_hi - r_lo) * n; q += kRlsThreads)
            a.P[(size_t)r_lo * n + q] = P[q];
}

// online delta rule: W_out[o][i] += (lr * (target_o - y_o)) * x_i
__global__ void k_online(double *W_out, int n, int dout, const double *x, const double *y,
                         const double *target, double lr)
{
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < (size_t)dout * n;
         q += (size_t)gridDim.x * blockDim.x) {
        const int o = (int)(q / n), i = (int)(q % n);
        const double a = lr * (target[o] - y[o]);
        W_out[q] = __dadd_rn(W_out[q], __dmul_rn(a, x[i]));
    }
}

double ms_since(std::chrono::steady_clock::time_point t)
{
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t)
        .count();
}

}  // namespace

// per-column dot products out[o] = sum_i X[i][o] Y[i][o] (n x dout arrays),
// one block per column, fixed-order reduction
static __global__ void k_coldot(const double *__restrict__ X, const double *__restrict__ Y, int n,
                         int dout, double *__restrict__ out)
{
    __shared__ double s[256];
    const int o = blockIdx.x;
    double a = 0.0;
    for (int i = threadIdx.x; i < n; i += 256)
        a = fma(X[(size_t)i * dout + o], Y[(size_t)i * dout + o], a);
    s[threadIdx.x] = a;
    __syncthreads();
    for (int st = 128; st; st >>= 1) {
        if ((int)threadIdx.x < st)
            s[threadIdx.x] += s[threadIdx.x + st];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        out[o] = s[0];
}

// Y[i][o] += c[o] X[i][o]  (xpby = 0)  or  Y[i][o] = X[i][o] + c[o] Y[i][o]  (xpby = 1)
static __global__ void k_col_update(double *__restrict__ Y, const double *__restrict__ X,
                             const double *__restrict__ c, int n, int dout, int xpby)
{
    const size_t total = (size_t)n * dout;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < total;
         k += (size_t)gridDim.x * blockDim.x) {
        const int o = (int)(k % dout);
        Y[k] = xpby ? fma(c[o], Y[k], X[k]) : fma(c[o], X[k], Y[k]);
    }
}

// largest diagonal entry (non-negative doubles compare like their bits)
static __global__ void k_diag_max(const double *__restrict__ A, int n, int lda,
                                  unsigned long long *out)
{
    double m = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double v = A[(size_t)i * lda + i];
        if (v > m)
            m = v;
    }
    for (int off = 16; off; off >>= 1) {
        const double o = __shfl_xor_sync(kFull, m, off);
        if (o > m)
            m = o;
    }
    if ((threadIdx.x & 31) == 0 && m > 0.0)
        atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

// ------------------------------------------------------------ factor + solve
// Factor A (pitch sp_solve_pad(n)) in place and wait; *bad = 0 or the 1-based
// failing pivot.
static int cholesky(cudaStream_t s, double *A, int n, void *work, int *d_info, int *bad)
{
    int h = 0;
    if (sp_solve_factor(s, A, n, work, d_info) != cudaSuccess ||
        cudaMemcpyAsync(&h, d_info, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
        sp_dev_note_error("ridge factorisation", (int)cudaGetLastError());
        return SP_EINTERNAL;
    }
    *bad = h;
    return h < 0 ? SP_EINTERNAL : SP_OK;  // < 0: a wait ran out
}

static int lu_factor_solve(cudaStream_t s, double *A, int n, int lda, int *d_piv, int *d_info,
                           double *Z, int dout)
{
    for (int j = 0; j < n; ++j) {
        k_lu_pivot<<<1, 256, 0, s>>>(A, n, lda, j, d_piv, d_info);
        int rows = n - j - 1;
        if (rows > 0)
            k_lu_update<<<rows < 1024 ? rows : 1024, 256, 0, s>>>(A, n, lda, j);
    }
    int h = 0;
    cudaMemcpyAsync(&h, d_info, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    if (h)
        return h;
    k_lu_solve<<<dout, 32, 0, s>>>(A, n, lda, d_piv, Z, dout);
    return 0;
}

// Waits for the stream; SP_EINTERNAL when a wait of a factorisation or solve on it
// ran out (their results are then not the system's).
static int solves_done(cudaStream_t s, const int *d_info)
{
    int h = 0;
    if (cudaMemcpyAsync(&h, d_info, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess || cudaGetLastError() != cudaSuccess)
        return SP_EINTERNAL;
    return h < 0 ? SP_EINTERNAL : SP_OK;
}

// Residual R = Phi^T (Y - Phi W) - lambda W for rows [t0, t1).
static void ridge_residual(cudaStream_t s, const double *Phi, int n, size_t t0, size_t t1,
                           const double *Y, const double *W, int dout, double lambda, double *E,
                           double *part, int parts, double *R)
{
    const size_t rows = t1 - t0;
    k_resid_rows<<<(unsigned)((rows + 7) / 8), 256, 0, s>>>(Phi, n, t0, t1, Y, W, dout, E);
    dim3 g((n + 127) / 128, parts);
    k_xt_e_part<<<g, 128, 0, s>>>(Phi, n, t0, t1, E, dout, parts, part);
    const size_t tot = (size_t)n * dout;
    k_reduce_parts<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(part, parts, n, dout, W, lambda,
                                                                 R);
}

static double device_norm(cudaStream_t s, const double *x, size_t cnt, double *d_tmp)
{
    cudaMemsetAsync(d_tmp, 0, sizeof(double), s);
    k_sumsq<<<64, 256, 0, s>>>(x, cnt, d_tmp);
    double h = 0.0;
    cudaMemcpyAsync(&h, d_tmp, sizeof(double), cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    return sqrt(h);
}

// Dual-form ridge for T - w0 < n: K = Phi_w Phi_w^T + lambda I (FP64 Gram of
// the transposed rows), Cholesky (pivoted LU if it fails, as dgesv would),
// alpha = K^-1 Y_w, W = Phi_w^T alpha; B = Phi_w^T Y_w for the residual check.
// E (T x dout) is used as the right-hand side and holds alpha in rows w0..T-1.
static int ridge_dual(cudaStream_t s, const double *Phi, int n, size_t T, size_t w0,
                      const double *Y, int dout, double lambda, sp_ridge_report *rep, double *W,
                      double *B, double *E, double *part, int parts, int *info, int *piv)
{
    int rc = SP_OK;
    const size_t tw = T - w0;
    const int m = (int)tw;
    double *Pt = nullptr, *K = nullptr;
    void *work = nullptr;
    const int mp = sp_solve_pad(m);
    const size_t tot = (size_t)n * dout;
    const dim3 gp((n + 127) / 128, parts);
    auto tg = std::chrono::steady_clock::now();
    RK(sp_cuda_malloc_async(&Pt, (size_t)n * tw * sizeof(double), s));
    RK(sp_cuda_malloc_async(&K, (size_t)mp * mp * sizeof(double), s));
    RK(sp_cuda_malloc_async((char **)&work, sp_solve_work_bytes(m), s));
    {
        dim3 g((n + 31) / 32, (unsigned)((tw + 31) / 32));
        k_rows_to_cols<<<g, dim3(32, 8), 0, s>>>(Phi, n, w0, T, Pt);
        RK(sp_solve_gram(s, Pt, m, 0, (size_t)n, K, mp));
        RK(sp_solve_diag(s, K, m, lambda));
        k_xt_e_part<<<gp, 128, 0, s>>>(Phi, n, w0, T, Y, dout, parts, part);
        k_reduce_parts<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(part, parts, n, dout, nullptr,
                                                                     0.0, B);
        RK(cudaMemcpyAsync(E, Y, T * dout * sizeof(double), cudaMemcpyDeviceToDevice, s));
        RK(cudaStreamSynchronize(s));
        RK(cudaGetLastError());
        rep->gram_ms = ms_since(tg);
    }
    {
        auto tf = std::chrono::steady_clock::now();
        double *Z = E + w0 * dout;
        int bad = 0;
        rc = cholesky(s, K, m, work, info, &bad);
        if (rc)
            goto out;
        if (bad) {
            rep->factor_failed = 1;
            rep->lu_fallback = 1;
            RK(cudaMemsetAsync(info, 0, sizeof(int), s));
            RK(sp_solve_gram(s, Pt, m, 0, (size_t)n, K, mp));
            k_add_diag<<<(m + 255) / 256, 256, 0, s>>>(K, m, mp, lambda);
            if (lu_factor_solve(s, K, m, mp, piv, info, Z, dout)) {
                rc = SP_RIDGE_SINGULAR;
                goto out;
            }
        } else {
            RK(sp_solve_apply(s, K, m, work, Z, dout, info));
        }
        k_xt_e_part<<<gp, 128, 0, s>>>(Phi, n, w0, T, E, dout, parts, part);
        k_reduce_parts<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(part, parts, n, dout, nullptr,
                                                                     0.0, W);
        rc = solves_done(s, info);
        if (rc)
            goto out;
        rep->factor_ms = ms_since(tf);
    }
out:
    if (Pt)
        sp_cuda_free_async(Pt, s);
    if (K)
        sp_cuda_free_async(K, s);
    if (work)
        sp_cuda_free_async(work, s);
    cudaStreamSynchronize(s);
    return rc;
}

// Mixed-precision solve of (Phi_w^T Phi_w + lambda I) W = B given A = G + lambda I
// with G the split tensor-core Gram. The rounding error of G can exceed
// lambda, so A itself may be indefinite: the preconditioner is the FP64
// Cholesky factor of A + delta I, delta = eps * max diag (raised tenfold until
// the factorisation succeeds), and the system is solved by preconditioned
// conjugate gradients per output column whose operator p -> Phi^T (Phi p) +
// lambda p is applied in FP64 from the states themselves. So the answer is
// the FP64 ridge solution to the stated residual; the Gram's precision only
// sets how many iterations that takes.
static int ridge_mixed(cudaStream_t s, const double *Phi, int n, size_t T, size_t w0,
                       const double *Y, int dout, double lambda, int mode,
                       const sp_ridge_opts *o, sp_ridge_report *rep, double *A, double *B,
                       double *W, double *R, double *E, double *part, int parts, double *tmp,
                       void *work, int *info)
{
    int rc = SP_OK;
    const int lda = sp_solve_pad(n);
    const size_t nn = (size_t)lda * lda, tot = (size_t)n * dout;
    const unsigned gb = (unsigned)((tot + 255) / 256 < 4096 ? (tot + 255) / 256 : 4096);
    double *A0 = nullptr, *Z = nullptr, *P = nullptr, *Q = nullptr, *Yz = nullptr, *c = nullptr,
           *dots = nullptr;
    double h_rz[16], h_pq[16], h_c[16];
    auto tf = std::chrono::steady_clock::now();
    RK(sp_cuda_malloc(&A0, nn * sizeof(double)));
    RK(sp_cuda_malloc(&Z, tot * sizeof(double)));
    RK(sp_cuda_malloc(&P, tot * sizeof(double)));
    RK(sp_cuda_malloc(&Q, tot * sizeof(double)));
    RK(sp_cuda_malloc(&Yz, (T ? T : 1) * (size_t)dout * sizeof(double)));
    RK(sp_cuda_malloc(&c, 16 * sizeof(double)));
    RK(sp_cuda_malloc(&dots, 16 * sizeof(double)));
    RK(cudaMemsetAsync(Yz, 0, (T ? T : 1) * (size_t)dout * sizeof(double), s));
    RK(cudaMemcpyAsync(A0, A, nn * sizeof(double), cudaMemcpyDeviceToDevice, s));
    {
        RK(cudaMemsetAsync(tmp, 0, sizeof(double), s));
        k_diag_max<<<(n + 255) / 256, 256, 0, s>>>(A, n, lda, (unsigned long long *)tmp);
        double dmax = 0.0;
        RK(cudaMemcpyAsync(&dmax, tmp, sizeof(double), cudaMemcpyDeviceToHost, s));
        RK(cudaStreamSynchronize(s));
        double delta = (mode == 1 ? 1e-4 : 1e-5) * dmax;
        int ok = 0;
        for (int attempt = 0; attempt < 6 && !ok; ++attempt, delta *= 10.0) {
            if (attempt > 0) {
                rep->factor_failed = 1;
                RK(cudaMemcpyAsync(A, A0, nn * sizeof(double), cudaMemcpyDeviceToDevice, s));
                RK(cudaMemsetAsync(info, 0, sizeof(int), s));
            }
            RK(sp_solve_diag(s, A, n, delta));
            int bad = 0;
            rc = cholesky(s, A, n, work, info, &bad);
            if (rc)
                goto out;
            ok = bad == 0;
        }
        if (!ok) {
            rc = SP_RIDGE_SINGULAR;
            goto out;
        }
        rep->factor_ms = ms_since(tf);
    }
    {
        auto tr = std::chrono::steady_clock::now();
        const double bnorm = device_norm(s, B, tot, tmp);
        const double bden = bnorm > 0 ? bnorm : 1.0;
        // W = M^-1 B, R = B - A W (FP64 from Phi), Z = M^-1 R, P = Z
        RK(cudaMemcpyAsync(W, B, tot * sizeof(double), cudaMemcpyDeviceToDevice, s));
        RK(sp_solve_apply(s, A, n, work, W, dout, info));
        ridge_residual(s, Phi, n, w0, T, Y, W, dout, lambda, E, part, parts, R);
        RK(cudaMemcpyAsync(Z, R, tot * sizeof(double), cudaMemcpyDeviceToDevice, s));
        RK(sp_solve_apply(s, A, n, work, Z, dout, info));
        RK(cudaMemcpyAsync(P, Z, tot * sizeof(double), cudaMemcpyDeviceToDevice, s));
        k_coldot<<<dout, 256, 0, s>>>(R, Z, n, dout, dots);
        RK(cudaMemcpyAsync(h_rz, dots, dout * sizeof(double), cudaMemcpyDeviceToHost, s));
        int it = 0;
        double rel = device_norm(s, R, tot, tmp) / bden;
        while (rel > o->refine_tol && it < o->max_refine) {
            // Q = -(A P): the residual form with zero targets
            ridge_residual(s, Phi, n, w0, T, Yz, P, dout, lambda, E, part, parts, Q);
            k_coldot<<<dout, 256, 0, s>>>(P, Q, n, dout, dots);
            RK(cudaMemcpyAsync(h_pq, dots, dout * sizeof(double), cudaMemcpyDeviceToHost, s));
            RK(cudaStreamSynchronize(s));
            for (int k = 0; k < dout; ++k)
                h_c[k] = (h_pq[k] != 0.0) ? h_rz[k] / -h_pq[k] : 0.0;  // alpha
            RK(cudaMemcpyAsync(c, h_c, dout * sizeof(double), cudaMemcpyHostToDevice, s));
            k_col_update<<<gb, 256, 0, s>>>(W, P, c, n, dout, 0);  // W += alpha P
            k_col_update<<<gb, 256, 0, s>>>(R, Q, c, n, dout, 0);  // R -= alpha A P
            RK(cudaMemcpyAsync(Z, R, tot * sizeof(double), cudaMemcpyDeviceToDevice, s));
            RK(sp_solve_apply(s, A, n, work, Z, dout, info));
            k_coldot<<<dout, 256, 0, s>>>(R, Z, n, dout, dots);
            double h_rz2[16];
            RK(cudaMemcpyAsync(h_rz2, dots, dout * sizeof(double), cudaMemcpyDeviceToHost, s));
            RK(cudaStreamSynchronize(s));
            for (int k = 0; k < dout; ++k) {
                h_c[k] = (h_rz[k] != 0.0) ? h_rz2[k] / h_rz[k] : 0.0;  // beta
                h_rz[k] = h_rz2[k];
            }
            RK(cudaMemcpyAsync(c, h_c, dout * sizeof(double), cudaMemcpyHostToDevice, s));
            k_col_update<<<gb, 256, 0, s>>>(P, Z, c, n, dout, 1);  // P = Z + beta P
            ++it;
            rel = device_norm(s, R, tot, tmp) / bden;
        }
        // the reported residual is recomputed from Phi, not the recurrence
        ridge_residual(s, Phi, n, w0, T, Y, W, dout, lambda, E, part, parts, R);
        rep->rel_residual = device_norm(s, R, tot, tmp) / bden;
        rep->refine_iters = it;
        rep->refine_ms = ms_since(tr);
        rc = solves_done(s, info);
    }
out:
    cudaStreamSynchronize(s);
    void *bufs[] = {A0, Z, P, Q, Yz, c, dots};
    for (void *b : bufs)
        if (b)
            sp_cuda_free(b);
    return rc;
}

// Work buffers of the primal solve, kept across calls by a caller that fits
// many readouts in a row (the batched fits): grown to the largest sizes seen,
// freed by sp_ridge_ws_free.
struct sp_ridge_ws {
    double *A = nullptr, *B = nullptr, *W = nullptr, *R = nullptr, *E = nullptr,
           *part = nullptr, *tmp = nullptr;
    char *work = nullptr;
    int *info = nullptr, *piv = nullptr;
    size_t cap_nn = 0, cap_nd = 0, cap_td = 0, cap_n = 0;
};

extern "C" sp_ridge_ws *sp_ridge_ws_new(void) { return new sp_ridge_ws(); }

static void ws_release(sp_ridge_ws *w)
{
    void *bufs[] = {w->A, w->B, w->W, w->R, w->E, w->part, w->tmp, w->work, w->info, w->piv};
    for (void *b : bufs)
        if (b)
            sp_cuda_free(b);
    *w = sp_ridge_ws();
}

extern "C" void sp_ridge_ws_free(sp_ridge_ws *w)
{
    if (!w)
        return;
    ws_release(w);
    delete w;
}

// Buffers for n neurons, T rows and dout (<= 16) outputs, reusing what is
// large enough. The caller's stream must be idle (the batched fits wait for
// each instance before the next).
static int ws_ensure(sp_ridge_ws *w, int n, size_t T, int dout, int parts)
{
    const size_t np = (size_t)sp_solve_pad(n), nn = np * np, nd = (size_t)n * dout,
                 td = (T ? T : 1) * (size_t)dout;
    if (nn <= w->cap_nn && nd <= w->cap_nd && td <= w->cap_td && (size_t)n <= w->cap_n)
        return SP_OK;
    const size_t cnn = nn > w->cap_nn ? nn : w->cap_nn, cnd = nd > w->cap_nd ? nd : w->cap_nd,
                 ctd = td > w->cap_td ? td : w->cap_td,
                 cn = (size_t)n > w->cap_n ? (size_t)n : w->cap_n;
    ws_release(w);
    int rc = SP_OK;
    RK(sp_cuda_malloc(&w->A, cnn * sizeof(double)));
    RK(sp_cuda_malloc(&w->B, cnd * sizeof(double)));
    RK(sp_cuda_malloc(&w->W, cnd * sizeof(double)));
    RK(sp_cuda_malloc(&w->R, cnd * sizeof(double)));
    RK(sp_cuda_malloc(&w->E, ctd * sizeof(double)));
    RK(sp_cuda_malloc(&w->part, (size_t)parts * cnd * sizeof(double)));
    RK(sp_cuda_malloc(&w->tmp, 4 * sizeof(double)));
    RK(sp_cuda_malloc(&w->info, sizeof(int)));
    RK(sp_cuda_malloc(&w->piv, cn * sizeof(int)));
    RK(sp_cuda_malloc(&w->work, sp_solve_work_bytes((int)cn)));
    w->cap_nn = cnn;
    w->cap_nd = cnd;
    w->cap_td = ctd;
    w->cap_n = cn;
    return SP_OK;
out:
    ws_release(w);
    return rc;
}

// States that are still on the host when a fit starts, and the stream their copies
// take.
struct RidgeFeed {
    const double *h_phi;
    double *Phi;
    cudaStream_t copies;
};

static cudaError_t feed_all(const RidgeFeed *f, int n, size_t T)
{
    const cudaError_t e = sp_copy_in(f->Phi, f->h_phi, T * (size_t)n * sizeof(double), f->copies);
    return e == cudaSuccess ? cudaStreamSynchronize(f->copies) : e;
}

// The copy of the states with the Gram of the rows that have arrived beside it, 16
// MB and more at a time (6000 x 2000: 2.2 + 1.1 ms one after the other, 2.3 together).
static cudaError_t feed_gram(const RidgeFeed *f, cudaStream_t s, int n, size_t w0, size_t T,
                             double *A, int lda)
{
    cudaEvent_t ev = nullptr;
    cudaError_t e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (e != cudaSuccess)
        return e;
    const size_t row = (size_t)n * sizeof(double), bytes = T * row;
    size_t next = w0;  // rows [w0, next) are in the sums
    e = sp_copy_in(f->Phi, f->h_phi, bytes, f->copies, [&](size_t done) {
        const size_t have = done / row;
        size_t to = have > next ? next + (have - next) / 4 * 4 : next;
        if (done == bytes)
            to = T;
        else if ((to - next) * row < ((size_t)16 << 20))
            return cudaSuccess;
        cudaError_t r = cudaEventRecord(ev, f->copies);
        if (r == cudaSuccess)
            r = cudaStreamWaitEvent(s, ev, 0);
        if (r == cudaSuccess)
            r = sp_solve_gram_range(s, f->Phi, n, next, to, A, lda, next > w0, done == bytes);
        next = to;
        return r;
    });
    cudaEventDestroy(ev);
    return e;
}

// One group of at most 16 outputs of sp_ridge_phi (below). Work buffers come
// from `ws` when given, else are allocated for the call. With `feed` the states
// are copied to Phi here.
static int ridge_phi_group(cudaStream_t s, const double *Phi, int n, size_t T,
                           const double *Y, int dout, double lambda, const sp_ridge_opts *o,
                           sp_ridge_report *rep, double *d_W_out, sp_ridge_ws *ws,
                           const RidgeFeed *feed = nullptr)
{
    int rc = SP_OK;
    double *A = nullptr, *B = nullptr, *W = nullptr, *R = nullptr, *E = nullptr,
           *part = nullptr, *tmp = nullptr;
    char *work = nullptr;
    int *info = nullptr, *piv = nullptr;
    const int parts = 64, lda = sp_solve_pad(n);
    const size_t w0 = o->washout;
    if (dout == 0)
        return SP_OK;
    if (dout > 16)
        return SP_EINVAL; /* per-thread accumulators below hold up to 16 outputs */
    if (ws) {
        rc = ws_ensure(ws, n, T, dout, parts);
        if (rc)
            return rc;
        A = ws->A;
        B = ws->B;
        W = ws->W;
        R = ws->R;
        E = ws->E;
        part = ws->part;
        tmp = ws->tmp;
        work = ws->work;
        info = ws->info;
        piv = ws->piv;
    } else {
        RK(sp_cuda_malloc_async(&A, (size_t)lda * lda * sizeof(double), s));
        RK(sp_cuda_malloc_async(&B, (size_t)n * dout * sizeof(double), s));
        RK(sp_cuda_malloc_async(&W, (size_t)n * dout * sizeof(double), s));
        RK(sp_cuda_malloc_async(&R, (size_t)n * dout * sizeof(double), s));
        RK(sp_cuda_malloc_async(&E, (T ? T : 1) * (size_t)dout * sizeof(double), s));
        RK(sp_cuda_malloc_async(&part, (size_t)parts * n * dout * sizeof(double), s));
        RK(sp_cuda_malloc_async(&tmp, 4 * sizeof(double), s));
        RK(sp_cuda_malloc_async(&work, sp_solve_work_bytes(n), s));
        RK(sp_cuda_malloc_async(&info, sizeof(int), s));
        RK(sp_cuda_malloc_async(&piv, (size_t)n * sizeof(int), s));
    }
    RK(cudaMemsetAsync(info, 0, sizeof(int), s));
    if (feed) {
        const bool fp64 = !((o->gram_mode == SP_GRAM_BF16X3 || o->gram_mode == SP_GRAM_TF32X3 ||
                             o->gram_mode == SP_GRAM_INT8) && sp_gram_tc_available());
        if (!fp64 || (lambda > 0.0 && 2 * (T - w0) <= (size_t)n) ||
            !sp_solve_gram_in_ranges(n, T - w0)) {
            auto tc = std::chrono::steady_clock::now();
            RK(feed_all(feed, n, T));
            rep->collect_ms += ms_since(tc);
            feed = nullptr;
        }
    }

    if (lambda > 0.0 && 2 * (T - w0) <= (size_t)n) {
        // Fewer fitted rows than half the neurons: the dual form
        // W = Phi_w^T (Phi_w Phi_w^T + lambda I)^-1 Y_w, algebraically the same
        // solution, factors a (T - w0)^2 matrix instead of n^2. (lambda = 0
        // keeps the primal system, singular here, so that the call fails and
        // leaves W_out as the reference's dgesv does.)
        rc = ridge_dual(s, Phi, n, T, w0, Y, dout, lambda, rep, W, B, E, part, parts, info, piv);
        if (rc)
            goto out;
        rep->dual = 1;
        rep->gram_mode_used = 0;
        const double bnorm = device_norm(s, B, (size_t)n * dout, tmp);
        ridge_residual(s, Phi, n, w0, T, Y, W, dout, lambda, E, part, parts, R);
        rep->rel_residual = device_norm(s, R, (size_t)n * dout, tmp) / (bnorm > 0 ? bnorm : 1.0);
        rep->refine_iters = 0;
        const size_t tot = (size_t)n * dout;
        k_transpose_w<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(W, n, dout, d_W_out);
        RK(cudaStreamSynchronize(s));
        RK(cudaGetLastError());
        goto out;
    }

    {
        auto tg = std::chrono::steady_clock::now();
        int mode = o->gram_mode;
        const int slices = o->gram_slices > 0 ? o->gram_slices : SP_GRAM_INT8_SLICES;
        if ((mode == SP_GRAM_BF16X3 || mode == SP_GRAM_TF32X3 || mode == SP_GRAM_INT8) &&
            sp_gram_tc_available()) {
            rc = sp_gram_tc(s, mode, slices, Phi, n, w0, T, A, lda);
            if (rc == SP_EINVAL && mode == SP_GRAM_INT8) {
                // a state that is not finite: the FP64 Gram, as the reference
                rc = SP_OK;
                mode = 0;
                RK(sp_solve_gram(s, Phi, n, w0, T, A, lda));
            }
            if (rc)
                goto out;
        } else {
            mode = 0;
            if (feed)
                RK(feed_gram(feed, s, n, w0, T, A, lda));
            else
                RK(sp_solve_gram(s, Phi, n, w0, T, A, lda));
        }
        rep->gram_mode_used = mode;
        dim3 g((n + 127) / 128, parts);
        k_xt_e_part<<<g, 128, 0, s>>>(Phi, n, w0, T, Y, dout, parts, part);
        const size_t tot = (size_t)n * dout;
        k_reduce_parts<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(part, parts, n, dout, nullptr,
                                                                     0.0, B);
        RK(sp_solve_diag(s, A, n, lambda));
        RK(cudaStreamSynchronize(s));
        RK(cudaGetLastError());
        rep->gram_ms = ms_since(tg);
    }

    if (rep->gram_mode_used == SP_GRAM_BF16X3 || rep->gram_mode_used == SP_GRAM_TF32X3) {
        // an FP32-accumulated Gram is too coarse to factor directly at small
        // lambda: Cholesky-preconditioned CG on the FP64 operator
        rc = ridge_mixed(s, Phi, n, T, w0, Y, dout, lambda, rep->gram_mode_used, o, rep, A, B, W,
                         R, E, part, parts, tmp, work, info);
        if (rc)
            goto out;
        const size_t tot = (size_t)n * dout;
        k_transpose_w<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(W, n, dout, d_W_out);
        RK(cudaStreamSynchronize(s));
        RK(cudaGetLastError());
        goto out;
    }

    {
        auto tf = std::chrono::steady_clock::now();
        RK(cudaMemcpyAsync(W, B, (size_t)n * dout * sizeof(double), cudaMemcpyDeviceToDevice, s));
        int bad = 0;
        rc = cholesky(s, A, n, work, info, &bad);
        if (rc)
            goto out;
        if (bad) {
            // dgesv semantics: LU with partial pivoting on the original matrix
            rep->factor_failed = 1;
            rep->lu_fallback = 1;
            RK(cudaMemsetAsync(info, 0, sizeof(int), s));
            if (rep->gram_mode_used != 0) {
                rc = sp_gram_tc(s, rep->gram_mode_used,
                                o->gram_slices > 0 ? o->gram_slices : SP_GRAM_INT8_SLICES, Phi,
                                n, w0, T, A, lda);
                if (rc)
                    goto out;
            } else {
                RK(sp_solve_gram(s, Phi, n, w0, T, A, lda));
            }
            k_add_diag<<<(n + 255) / 256, 256, 0, s>>>(A, n, lda, lambda);
            int lbad = lu_factor_solve(s, A, n, lda, piv, info, W, dout);
            if (lbad) {
                rc = SP_RIDGE_SINGULAR;
                goto out;
            }
            rep->factor_ms = ms_since(tf);
        } else {
            // cholesky() has waited for the factorisation
            rep->factor_ms = ms_since(tf);
            auto ts = std::chrono::steady_clock::now();
            RK(sp_solve_apply(s, A, n, work, W, dout, info));
            RK(cudaStreamSynchronize(s));
            rep->solve_ms = ms_since(ts);
        }
        RK(cudaStreamSynchronize(s));
        RK(cudaGetLastError());
    }

    {
        // iterative refinement with FP64 residuals from Phi itself
        auto tr = std::chrono::steady_clock::now();
        const double bnorm = device_norm(s, B, (size_t)n * dout, tmp);
        int it = 0;
        double rel = 0.0;
        const int maxit = rep->lu_fallback ? 0 : o->max_refine;
        for (;;) {
            ridge_residual(s, Phi, n, w0, T, Y, W, dout, lambda, E, part, parts, R);
            rel = device_norm(s, R, (size_t)n * dout, tmp) / (bnorm > 0 ? bnorm : 1.0);
            if (rel <= o->refine_tol || it >= maxit)
                break;
            RK(sp_solve_apply(s, A, n, work, R, dout, info));
            const size_t tot = (size_t)n * dout;
            k_axpy<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(W, R, tot);
            ++it;
        }
        rep->refine_iters = it;
        rep->rel_residual = rel;
        rep->refine_ms = ms_since(tr);
    }

    {
        const size_t tot = (size_t)n * dout;
        // W (n x dout) -> W_out (dout x n)
        k_transpose_w<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(W, n, dout, d_W_out);
        rc = solves_done(s, info);
    }
out:
    if (!ws) {
        void *bufs[] = {A, B, W, R, E, part, tmp, work, info, piv};
        for (void *b : bufs)
            if (b)
                sp_cuda_free_async(b, s);
    }
    cudaStreamSynchronize(s);
    return rc;
}

extern "C" int sp_gram_fp64(cudaStream_t s, const double *X, int n, size_t t0, size_t t1,
                            double *C, int ldc)
{
    return sp_solve_gram(s, X, n, t0, t1, C, ldc) == cudaSuccess ? SP_OK : SP_EINTERNAL;
}

// Ridge on states already on the device: Phi [T x n] row-major (neuron order),
// Y [T x dout]; rows [washout, T) enter the Gram. On success d_W_out [dout x n]
// holds the solution; SP_RIDGE_SINGULAR leaves it untouched (dgesv failure in
// the reference leaves W_out as it was). The solver's per-thread accumulators
// hold 16 outputs; with more, the outputs are solved 16 at a time -- the system
// matrix is the same for all of them -- each group's targets copied to a
// contiguous block and its rows of W gathered in a work array that reaches
// d_W_out only when every group has succeeded.
extern "C" int sp_ridge_phi(cudaStream_t s, const double *Phi, int n, size_t T,
                            const double *Y, int dout, double lambda, const sp_ridge_opts *o,
                            sp_ridge_report *rep, double *d_W_out);

extern "C" int sp_ridge_phi_ws(cudaStream_t s, const double *Phi, int n, size_t T,
                               const double *Y, int dout, double lambda, const sp_ridge_opts *o,
                               sp_ridge_report *rep, double *d_W_out, sp_ridge_ws *ws)
{
    if (dout <= 16)
        return ridge_phi_group(s, Phi, n, T, Y, dout, lambda, o, rep, d_W_out, ws);
    return sp_ridge_phi(s, Phi, n, T, Y, dout, lambda, o, rep, d_W_out);
}

namespace {

size_t pad256(size_t b) { return (b + 255) & ~(size_t)255; }

// The buffers of one fit in the slab of ridge_direct_many.
struct DirectFit {
    double *A, *B, *W, *R, *E, *part;
    char *work;
};

constexpr int kManyParts = 64;

}  // namespace

extern "C" size_t sp_ridge_item_bytes(int n, size_t T, int dout)
{
    const size_t np = sp_solve_pad(n), nd = (size_t)n * dout * sizeof(double);
    return pad256(np * np * sizeof(double)) + 3 * pad256(nd) +
           pad256((T ? T : 1) * (size_t)dout * sizeof(double)) + pad256(kManyParts * nd) +
           pad256(sp_solve_work_bytes(n));
}

// The steps of ridge_phi_group's FP64 primal fit, each over every item before the
// next: one factorisation, one solve and one wait per refinement for all of them.
// An item whose Cholesky fails is left to the caller (*again). (20 fits of N 300 to
// 1600: 15.5 ms one after the other, 5 together.)
static int ridge_direct_many(cudaStream_t s, sp_ridge_item **items, int count,
                             const sp_ridge_opts *o, char *again)
{
    int rc = SP_OK;
    char *slab = nullptr;
    std::vector<DirectFit> fit(count);
    std::vector<sp_solve_item> sys, sub;
    std::vector<int> at, info(count), act;
    std::vector<double> norm(2 * (size_t)count);
    const size_t w0 = o->washout;
    size_t total = pad256(2 * (size_t)count * sizeof(double)) + pad256(count * sizeof(int));
    for (int k = 0; k < count; ++k)
        total += sp_ridge_item_bytes(items[k]->n, items[k]->T, items[k]->dout);
    RK(sp_cuda_malloc_async(&slab, total, s));
    {
        size_t off = 0;
        auto take = [&](size_t bytes) {
            char *p = slab + off;
            off += pad256(bytes);
            return p;
        };
        double *d_norm = (double *)take(2 * (size_t)count * sizeof(double));  // |B|^2, |R|^2
        int *d_info = (int *)take(count * sizeof(int));
        RK(cudaMemsetAsync(slab, 0, off, s));
        for (int k = 0; k < count; ++k) {
            const sp_ridge_item &it = *items[k];
            DirectFit &f = fit[k];
            const int n = it.n, dout = it.dout, lda = sp_solve_pad(n);
            const size_t tot = (size_t)n * dout, nd = tot * sizeof(double);
            f.A = (double *)take((size_t)lda * lda * sizeof(double));
            f.B = (double *)take(nd);
            f.W = (double *)take(nd);
            f.R = (double *)take(nd);
            f.E = (double *)take(it.T * (size_t)dout * sizeof(double));
            f.part = (double *)take(kManyParts * nd);
            f.work = take(sp_solve_work_bytes(n));
            RK(sp_solve_gram(s, it.Phi, n, w0, it.T, f.A, lda));
            k_xt_e_part<<<dim3((n + 127) / 128, kManyParts), 128, 0, s>>>(
                it.Phi, n, w0, it.T, it.Y, dout, kManyParts, f.part);
            k_reduce_parts<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(f.part, kManyParts, n, dout,
                                                                         nullptr, 0.0, f.B);
            RK(sp_solve_diag(s, f.A, n, it.lambda));
            RK(cudaMemcpyAsync(f.W, f.B, nd, cudaMemcpyDeviceToDevice, s));
            k_sumsq<<<64, 256, 0, s>>>(f.B, tot, d_norm + 2 * k);
            sys.push_back({f.A, n, f.work, f.W, dout, d_info + k});
        }
        RK(sp_solve_factor(s, sys.data(), count));
        RK(cudaMemcpyAsync(info.data(), d_info, count * sizeof(int), cudaMemcpyDeviceToHost, s));
        RK(cudaStreamSynchronize(s));
        for (int k = 0; k < count; ++k) {
            if (info[k] < 0)
                rc = SP_EINTERNAL;  // a wait ran out
            again[k] = info[k] > 0;
            if (info[k] == 0) {
                act.push_back(k);
                sub.push_back(sys[k]);
            }
        }
        if (rc)
            goto out;
        at = act;
        if (!sub.empty())
            RK(sp_solve_apply(s, sub.data(), (int)sub.size()));
        for (int it = 0; !act.empty(); ++it) {
            for (int k : act) {
                const sp_ridge_item &m = *items[k];
                const DirectFit &f = fit[k];
                ridge_residual(s, m.Phi, m.n, w0, m.T, m.Y, f.W, m.dout, m.lambda, f.E, f.part,
                               kManyParts, f.R);
                RK(cudaMemsetAsync(d_norm + 2 * k + 1, 0, sizeof(double), s));
                k_sumsq<<<64, 256, 0, s>>>(f.R, (size_t)m.n * m.dout, d_norm + 2 * k + 1);
            }
            RK(cudaMemcpyAsync(norm.data(), d_norm, norm.size() * sizeof(double),
                               cudaMemcpyDeviceToHost, s));
            RK(cudaStreamSynchronize(s));
            std::vector<int> more;
            sub.clear();
            for (int k : act) {
                const double bnorm = sqrt(norm[2 * k]);
                const double rel = sqrt(norm[2 * k + 1]) / (bnorm > 0 ? bnorm : 1.0);
                if (rel <= o->refine_tol || it >= o->max_refine)
                    continue;
                more.push_back(k);
                sub.push_back(sys[k]);
                sub.back().Z = fit[k].R;
            }
            if (!sub.empty())
                RK(sp_solve_apply(s, sub.data(), (int)sub.size()));
            for (int k : more) {
                const size_t tot = (size_t)items[k]->n * items[k]->dout;
                k_axpy<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(fit[k].W, fit[k].R, tot);
            }
            act = more;
        }
        for (int k : at) {
            const sp_ridge_item &m = *items[k];
            const size_t tot = (size_t)m.n * m.dout;
            k_transpose_w<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(fit[k].W, m.n, m.dout,
                                                                        m.d_W_out);
        }
        RK(cudaMemcpyAsync(info.data(), d_info, count * sizeof(int), cudaMemcpyDeviceToHost, s));
        RK(cudaStreamSynchronize(s));
        RK(cudaGetLastError());
        for (int k = 0; k < count; ++k)
            if (info[k] < 0)
                rc = SP_EINTERNAL;
    }
out:
    if (slab)
        sp_cuda_free_async(slab, s);
    cudaStreamSynchronize(s);
    return rc;
}

extern "C" int sp_ridge_phi_many(cudaStream_t s, sp_ridge_item *items, size_t count,
                                 const sp_ridge_opts *o, sp_ridge_ws *ws)
{
    const int mode = o->gram_mode;
    const bool fp64 = !((mode == SP_GRAM_BF16X3 || mode == SP_GRAM_TF32X3 || mode == SP_GRAM_INT8) &&
                        sp_gram_tc_available());
    std::vector<sp_ridge_item *> direct;
    std::vector<char> alone(count, 1), again;
    std::vector<size_t> index;
    for (size_t k = 0; k < count; ++k) {
        const sp_ridge_item &it = items[k];
        if (fp64 && it.dout > 0 && it.dout <= 16 && it.T > o->washout &&
            !(it.lambda > 0.0 && 2 * (it.T - o->washout) <= (size_t)it.n)) {
            direct.push_back(&items[k]);
            index.push_back(k);
        }
        items[k].rc = SP_OK;
    }
    if (direct.size() > 1) {
        again.assign(direct.size(), 0);
        const int rc = ridge_direct_many(s, direct.data(), (int)direct.size(), o, again.data());
        if (rc)
            return rc;
        for (size_t k = 0; k < direct.size(); ++k)
            alone[index[k]] = again[k];
    }
    for (size_t k = 0; k < count; ++k) {
        if (!alone[k])
            continue;
        sp_ridge_report rep;
        memset(&rep, 0, sizeof(rep));
        sp_ridge_item &it = items[k];
        it.rc = sp_ridge_phi_ws(s, it.Phi, it.n, it.T, it.Y, it.dout, it.lambda, o, &rep,
                                it.d_W_out, ws);
        if (it.rc && it.rc != SP_RIDGE_SINGULAR)
            return it.rc;
    }
    return SP_OK;
}

extern "C" int sp_ridge_phi(cudaStream_t s, const double *Phi, int n, size_t T,
                            const double *Y, int dout, double lambda, const sp_ridge_opts *o,
                            sp_ridge_report *rep, double *d_W_out)
{
    if (dout <= 16)
        return ridge_phi_group(s, Phi, n, T, Y, dout, lambda, o, rep, d_W_out, nullptr);
    int rc = SP_OK;
    double *Yg = nullptr, *Wall = nullptr;
    sp_ridge_report sum;
    memset(&sum, 0, sizeof(sum));
    RK(sp_cuda_malloc(&Yg, (T ? T : 1) * 16 * sizeof(double)));
    RK(sp_cuda_malloc(&Wall, (size_t)dout * n * sizeof(double)));
    for (int g0 = 0; g0 < dout && !rc; g0 += 16) {
        const int dg = dout - g0 < 16 ? dout - g0 : 16;
        if (T)
            RK(cudaMemcpy2DAsync(Yg, (size_t)dg * sizeof(double), Y + g0,
                                 (size_t)dout * sizeof(double), (size_t)dg * sizeof(double), T,
                                 cudaMemcpyDeviceToDevice, s));
        sp_ridge_report r1;
        memset(&r1, 0, sizeof(r1));
        rc = ridge_phi_group(s, Phi, n, T, Yg, dg, lambda, o, &r1, Wall + (size_t)g0 * n,
                             nullptr);
        sum.gram_mode_used = r1.gram_mode_used;
        sum.dual = r1.dual;
        sum.refine_iters = r1.refine_iters > sum.refine_iters ? r1.refine_iters : sum.refine_iters;
        sum.rel_residual = r1.rel_residual > sum.rel_residual ? r1.rel_residual : sum.rel_residual;
        sum.gram_ms += r1.gram_ms;
        sum.factor_ms += r1.factor_ms;
        sum.solve_ms += r1.solve_ms;
        sum.refine_ms += r1.refine_ms;
        sum.factor_failed |= r1.factor_failed;
        sum.lu_fallback |= r1.lu_fallback;
    }
    if (!rc)
        RK(cudaMemcpyAsync(d_W_out, Wall, (size_t)dout * n * sizeof(double),
                           cudaMemcpyDeviceToDevice, s));
out:
    cudaStreamSynchronize(s);
    if (Yg)
        sp_cuda_free(Yg);
    if (Wall)
        sp_cuda_free(Wall);
    sum.collect_ms = rep->collect_ms;
    *rep = sum;
    return rc;
}

// Ridge on caller-provided states (host arrays): Phi [T x n], Y [T x dout];
// writes W_out [dout x n] to the host. Same solver (and dual/split choices) as
// the reservoir readouts, on the current device and a stream of its own.
extern "C" int sp_ridge_host(const double *h_phi, size_t T, int n, const double *h_y, int dout,
                             double lambda, const sp_ridge_opts *o, sp_ridge_report *rep,
                             double *h_w_out)
{
    int rc = SP_OK;
    cudaStream_t s = nullptr, copies = nullptr;
    double *Phi = nullptr, *Y = nullptr, *Wt = nullptr;
    memset(rep, 0, sizeof(*rep));
    if (dout <= 0 || n <= 0 || T == 0 || o->washout >= T)
        return SP_EINVAL;
    auto t0 = std::chrono::steady_clock::now();
    RK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    RK(sp_cuda_malloc_async(&Phi, T * (size_t)n * sizeof(double), s));
    RK(sp_cuda_malloc_async(&Y, T * (size_t)dout * sizeof(double), s));
    RK(sp_cuda_malloc_async(&Wt, (size_t)n * dout * sizeof(double), s));
    RK(sp_copy_in(Y, h_y, T * (size_t)dout * sizeof(double), s));
    RK(cudaStreamCreateWithFlags(&copies, cudaStreamNonBlocking));
    RK(cudaStreamSynchronize(s));  // the buffers are there for the other stream
    {
        const RidgeFeed feed = {h_phi, Phi, copies};
        if (dout > 16)
            RK(feed_all(&feed, n, T));
        rep->collect_ms = ms_since(t0);
        rc = dout > 16 ? sp_ridge_phi(s, Phi, n, T, Y, dout, lambda, o, rep, Wt)
                       : ridge_phi_group(s, Phi, n, T, Y, dout, lambda, o, rep, Wt, nullptr, &feed);
    }
    if (rc)
        goto out;
    RK(cudaMemcpyAsync(h_w_out, Wt, (size_t)n * dout * sizeof(double), cudaMemcpyDeviceToHost, s));
    RK(cudaStreamSynchronize(s));
out:
    if (copies) {
        cudaStreamSynchronize(copies);
        cudaStreamDestroy(copies);
    }
    void *bufs[] = {Phi, Y, Wt};
    for (void *b : bufs)
        if (b)
            sp_cuda_free_async(b, s);
    if (s) {
        cudaStreamSynchronize(s);
        cudaStreamDestroy(s);
    }
    return rc;
}

extern "C" int sp_dev_train_ridge(sp_dev *d, const sp_host_model *m, const double *h_u,
                                  const double *h_y, size_t T, double lambda,
                                  const sp_ridge_opts *o, sp_ridge_report *rep, double *h_W_out)
{
    int rc = SP_OK;
    const int n = d->n, dout = d->dout;
    cudaStream_t s = d->stream;
    double *Phi = nullptr, *Y = nullptr, *Wt = nullptr;
    memset(rep, 0, sizeof(*rep));
    if (dout == 0)
        return SP_OK;
    auto tstart = std::chrono::steady_clock::now();

    rc = sp_dev_reset_neurons(d, m);
    if (rc)
        return rc;
    RK(sp_cuda_malloc_async(&Phi, (T ? T : 1) * (size_t)n * sizeof(double), s));
    RK(sp_cuda_malloc_async(&Y, (T ? T : 1) * (size_t)dout * sizeof(double), s));
    RK(sp_cuda_malloc_async(&Wt, (size_t)n * dout * sizeof(double), s));
    RK(cudaMemcpyAsync(Y, h_y, T * dout * sizeof(double), cudaMemcpyHostToDevice, s));
    {
        sp_run_args a;
        memset(&a, 0, sizeof(a));
        a.u = h_u;
        a.T = T;
        a.d_phi = Phi;
        a.sync = 1;
        rc = sp_dev_run(d, &a);
        if (rc)
            goto out;
    }
    rep->collect_ms = ms_since(tstart);
    rc = sp_ridge_phi(s, Phi, n, T, Y, dout, lambda, o, rep, Wt);
    if (rc == SP_RIDGE_SINGULAR) {
        // singular: the reference leaves W_out unchanged and warns
        fprintf(stderr, "Warning: Ridge regression failed (singular system).\n");
        rc = SP_OK;
        goto out;
    }
    if (rc)
        goto out;
    RK(cudaMemcpyAsync(h_W_out, Wt, (size_t)n * dout * sizeof(double), cudaMemcpyDeviceToHost, s));
    rc = sp_dev_w_out_from_nat(d, Wt);
    if (rc)
        goto out;
    RK(cudaStreamSynchronize(s));
    RK(cudaGetLastError());
out:
    void *bufs[] = {Phi, Y, Wt};
    for (void *b : bufs)
        if (b)
            sp_cuda_free_async(b, s);
    cudaStreamSynchronize(s);
    return rc;
}

// Launch shape of k_rls for n positions: CTAs, rows of P per CTA, whether P is
// kept in shared memory. Returns the shared memory, or 0 when the state vectors
// do not fit (about 5700 positions; the separate kernels then take each step:
// P is 260 MB and more, and its passes over HBM outweigh the launches).
static size_t rls_shape(const sp_dev *d, int n, int *ctas, int *rows, int *resident)
{
    if (!d->coop)
        return 0;
    const size_t room = (size_t)d->smem_max - 1024;
    const size_t base = (5 * (size_t)n + kRlsThreads) * sizeof(double);
    if (base > room)
        return 0;
    // a row per warp while the SMs last
    int G = (n + kRlsThreads / 32 - 1) / (kRlsThreads / 32);
    G = G < d->num_sms ? G : d->num_sms;
    *rows = (n + G - 1) / G;
    *ctas = (n + *rows - 1) / *rows;
    const size_t full = base + (size_t)*rows * n * sizeof(double);
    *resident = full <= room;
    return *resident ? full : base;
}

extern "C" int sp_dev_train_rls(sp_dev *d, const sp_host_model *m, const double *h_u,
                                const double *h_y, size_t T, double delta, double lambda,
                                double *h_W_out)
{
    // state, W_out and P live in position space (holes keep x = 0 and stay inert)
    int rc = SP_OK;
    const int rs = d->rs, n = d->n, dout = d->dout;
    cudaStream_t s = d->stream;
    double *P = nullptr, *Px = nullptr, *scal = nullptr, *Yd = nullptr, *Wn = nullptr;
    unsigned long long *ll = nullptr;
    int ctas = 0, rows = 0, resident = 0;
    const size_t smem = rls_shape(d, rs, &ctas, &rows, &resident);
    RK(sp_cuda_malloc(&Yd, (T ? T : 1) * (size_t)(dout ? dout : 1) * sizeof(double)));
    RK(sp_cuda_malloc(&Wn, (size_t)(dout ? dout : 1) * n * sizeof(double)));
    if (!smem || !resident || T > d->chunk)
        RK(sp_cuda_malloc(&P, (size_t)rs * rs * sizeof(double)));
    if (smem) {
        RK(sp_cuda_malloc(&ll, 4 * (size_t)rs * sizeof(unsigned long long)));
        RK(set_max_dynamic_smem((const void *)k_rls));
    } else {
        RK(sp_cuda_malloc(&Px, (size_t)rs * sizeof(double)));
        RK(sp_cuda_malloc(&scal, (size_t)(dout + 1) * sizeof(double)));
        k_diag_init<<<1024, 256, 0, s>>>(P, rs, 1.0 / delta);
    }
    RK(cudaMemsetAsync(d->W_out, 0, (size_t)rs * dout * sizeof(double), s));
    if (T && dout)
        RK(cudaMemcpyAsync(Yd, h_y, T * dout * sizeof(double), cudaMemcpyHostToDevice, s));
    rc = sp_dev_reset_neurons(d, m);
    if (rc)
        goto out;
    for (size_t t = 0; smem && t < T;) {
        // states of up to a chunk of steps in one launch, then the recursion over
        // them; the staging is the next chunk's once the stream has passed
        const size_t tc = T - t < d->chunk ? T - t : d->chunk;
        const double *u = nullptr;
        if (t)
            RK(cudaStreamSynchronize(s));
        if (h_u && d->din > 0) {
            RK(cudaMemcpyAsync(d->d_u, h_u + t * d->din, tc * d->din * sizeof(double),
                               cudaMemcpyHostToDevice, s));
            u = d->d_u;
        }
        rc = sp_dev_launch_chunk(d, u, tc, d->d_phi, nullptr);
        if (rc)
            goto out;
        RK(cudaMemsetAsync(ll, 0, 4 * (size_t)rs * sizeof(unsigned long long), s));
        RlsArgs a;
        a.X = d->d_phi;
        a.Y = Yd + t * dout;
        a.P = P;
        a.W = d->W_out;
        a.ll = ll;
        a.err = d->err;
        a.T = tc;
        a.step0 = (long long)t;
        a.n = rs;
        a.dout = dout;
        a.rows = rows;
        a.resident = resident;
        a.first = t == 0;
        a.last = t + tc == T;
        a.p0 = 1.0 / delta;
        a.lambda = lambda;
        void *args[] = {&a};
        RK(cudaLaunchCooperativeKernel((const void *)k_rls, dim3(ctas), dim3(kRlsThreads), args,
                                       smem, s));
        t += tc;
    }
    for (size_t t = 0; !smem && t < T; ++t) {
        sp_run_args a;
        memset(&a, 0, sizeof(a));
        a.u = h_u ? h_u + t * d->din : nullptr;
        a.T = 1;
        rc = sp_dev_run(d, &a);
        if (rc)
            goto out;
        k_gemv_rows<<<(rs + 7) / 8, 256, 0, s>>>(P, rs, d->V, Px);
        k_rls_scalars<<<1, 256, 0, s>>>(d->V, Px, rs, lambda, d->W_out, dout, Yd + t * dout,
                                        scal);
        k_rls_update<<<4 * d->num_sms, 256, 0, s>>>(P, rs, Px, scal, lambda, d->W_out, dout);
    }
    rc = sp_dev_w_out_to_nat(d, Wn);
    if (rc)
        goto out;
    RK(cudaMemcpyAsync(h_W_out, Wn, (size_t)n * dout * sizeof(double), cudaMemcpyDeviceToHost,
                       s));
    rc = sp_dev_sync(d);
    if (rc)
        goto out;
    RK(cudaGetLastError());
out:
    cudaStreamSynchronize(s);
    if (P) sp_cuda_free(P);
    if (Px) sp_cuda_free(Px);
    if (scal) sp_cuda_free(scal);
    if (Yd) sp_cuda_free(Yd);
    if (Wn) sp_cuda_free(Wn);
    if (ll) sp_cuda_free(ll);
    return rc;
}

extern "C" int sp_dev_train_online(sp_dev *d, const double *h_target, double lr, double *h_W_out)
{
    int rc = SP_OK;
    const int rs = d->rs, n = d->n, dout = d->dout;
    cudaStream_t s = d->stream;
    double *Wn = nullptr;
    if (dout == 0)
        return SP_OK;
    // prediction with the same readout kernel as spires_compute_output
    rc = sp_dev_readout(d, d->V, 1, d->d_y);
    if (rc)
        return rc;
    RK(sp_cuda_malloc(&Wn, (size_t)dout * n * sizeof(double)));
    RK(cudaMemcpyAsync(d->d_y + dout, h_target, (size_t)dout * sizeof(double),
                       cudaMemcpyHostToDevice, s));
    k_online<<<(unsigned)(((size_t)rs * dout + 255) / 256), 256, 0, s>>>(d->W_out, rs, dout, d->V,
                                                                        d->d_y, d->d_y + dout, lr);
    rc = sp_dev_w_out_to_nat(d, Wn);
    if (rc)
        goto out;
    RK(cudaMemcpyAsync(h_W_out, Wn, (size_t)n * dout * sizeof(double), cudaMemcpyDeviceToHost,
                       s));
    RK(cudaStreamSynchronize(s));
    RK(cudaGetLastError());
out:
    cudaStreamSynchronize(s);
    if (Wn)
        sp_cuda_free(Wn);
    return rc;
}

// ---------------------------------------------------- allocation-free solve
// Ridge readout from states the caller already holds in device memory, for
// callers that cannot allocate device memory themselves: a host framework
// that owns every device buffer through its own allocator or quota, or a
// control loop that cannot afford the implicit device-wide synchronisation of
// cudaMalloc/cudaFree. All working memory is the file-scope array below,
// sized for at most SP_NA_MAX_N neurons, SP_NA_MAX_DOUT outputs and
// SP_NA_MAX_T rows (8.7 MB); every GPU that loads this library holds it until
// the process exits. The same kernels as spires_ext_train_ridge with the FP64
// Gram run in the same order, so the two agree given the same states.
#define SP_NA_MAX_N 512
#define SP_NA_MAX_DOUT 16
#define SP_NA_MAX_T 16384
#define SP_NA_PARTS 64
/* the solver's inverted blocks and flags: sp_solve_work_bytes(512) in doubles */
#define SP_NA_WORK (8 * 4 * 256 + (8 * 8 + 2 * 8 + 4 + 1) / 2)
#define SP_NA_DOUBLES                                                                  \
    ((size_t)SP_NA_MAX_N * SP_NA_MAX_N + 3 * (size_t)SP_NA_MAX_N * SP_NA_MAX_DOUT +    \
     (size_t)SP_NA_MAX_T * SP_NA_MAX_DOUT +                                            \
     (size_t)SP_NA_PARTS * SP_NA_MAX_N * SP_NA_MAX_DOUT + 8 + SP_NA_WORK)

static __device__ __align__(256) double g_na_scratch[SP_NA_DOUBLES];
static __device__ __align__(256) int g_na_iscratch[SP_NA_MAX_N + 8];

// Device addresses of the two arrays, looked up once per device (with that
// device current) on the first call made on it, and the lock that a call holds
// until its work on them has ended: the solver's flags and hand-out counter are
// in them too, and a second call that zeroed those under a running factorisation
// would have its tiles taken before they are ready.
static double *g_na_dptr[64];
static int *g_na_iptr[64];
static std::mutex g_na_lock[64];

static int na_setup(int dev)
{
    if (g_na_dptr[dev] && g_na_iptr[dev])
        return SP_OK;
    void *pd = nullptr, *pi = nullptr;
    if (cudaGetSymbolAddress(&pd, g_na_scratch) != cudaSuccess || !pd)
        return SP_EINTERNAL;
    if (cudaGetSymbolAddress(&pi, g_na_iscratch) != cudaSuccess || !pi)
        return SP_EINTERNAL;
    g_na_dptr[dev] = (double *)pd;
    g_na_iptr[dev] = (int *)pi;
    return SP_OK;
}

// The solve, with the device's lock held.
static int na_solve(int dev, const double *d_states, const double *d_targets, size_t T, int n,
                    int dout, size_t washout, double lambda, double *d_w_out, cudaStream_t s)
{
    int rc = na_setup(dev);
    if (rc)
        return rc;
    double *A = g_na_dptr[dev];
    double *B = A + (size_t)SP_NA_MAX_N * SP_NA_MAX_N;
    double *W = B + (size_t)SP_NA_MAX_N * SP_NA_MAX_DOUT;
    double *R = W + (size_t)SP_NA_MAX_N * SP_NA_MAX_DOUT;
    double *E = R + (size_t)SP_NA_MAX_N * SP_NA_MAX_DOUT;
    double *part = E + (size_t)SP_NA_MAX_T * SP_NA_MAX_DOUT;
    double *tmp = part + (size_t)SP_NA_PARTS * SP_NA_MAX_N * SP_NA_MAX_DOUT;
    void *work = tmp + 8;
    const int lda = sp_solve_pad(n);
    int *info = g_na_iptr[dev];
    int *piv = info + 8;
    const int parts = SP_NA_PARTS;
    const size_t tot = (size_t)n * dout;
    const int maxit = 30;
    const double tol = 1e-13;

    // the work area keeps the previous call's contents: clear the flag that
    // must start at zero; every other region is fully rewritten below
    if (cudaMemsetAsync(info, 0, sizeof(int), s) != cudaSuccess)
        return SP_EINTERNAL;
    if (sp_solve_gram(s, d_states, n, washout, T, A, lda) != cudaSuccess)
        return SP_EINTERNAL;
    {
        dim3 g((n + 127) / 128, parts);
        k_xt_e_part<<<g, 128, 0, s>>>(d_states, n, washout, T, d_targets, dout, parts, part);
        k_reduce_parts<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(part, parts, n, dout,
                                                                     nullptr, 0.0, B);
    }
    if (sp_solve_diag(s, A, n, lambda) != cudaSuccess ||
        cudaMemcpyAsync(W, B, tot * sizeof(double), cudaMemcpyDeviceToDevice, s) != cudaSuccess)
        return SP_EINTERNAL;
    int bad = 0;
    if (cholesky(s, A, n, work, info, &bad) != SP_OK)
        return SP_EINTERNAL;
    bool lu = false;
    if (bad) {
        lu = true;
        cudaMemsetAsync(info, 0, sizeof(int), s);
        if (sp_solve_gram(s, d_states, n, washout, T, A, lda) != cudaSuccess)
            return SP_EINTERNAL;
        k_add_diag<<<(n + 255) / 256, 256, 0, s>>>(A, n, lda, lambda);
        if (lu_factor_solve(s, A, n, lda, piv, info, W, dout) != 0) {
            // singular system: d_w_out is not written, and the caller is told
            cudaStreamSynchronize(s);
            return SP_EINTERNAL;
        }
    } else if (sp_solve_apply(s, A, n, work, W, dout, info) != cudaSuccess) {
        return SP_EINTERNAL;
    }
    const double bnorm = device_norm(s, B, tot, tmp);
    for (int it = 0;; ++it) {
        ridge_residual(s, d_states, n, washout, T, d_targets, W, dout, lambda, E, part, parts, R);
        const double rel = device_norm(s, R, tot, tmp) / (bnorm > 0 ? bnorm : 1.0);
        if (rel <= tol || it >= (lu ? 0 : maxit))
            break;
        if (sp_solve_apply(s, A, n, work, R, dout, info) != cudaSuccess)
            return SP_EINTERNAL;
        k_axpy<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(W, R, tot);
    }
    if (solves_done(s, info) != SP_OK)
        return SP_EINTERNAL;
    k_transpose_w<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(W, n, dout, d_w_out);
    if (cudaStreamSynchronize(s) != cudaSuccess || cudaGetLastError() != cudaSuccess)
        return SP_EINTERNAL;
    return SP_OK;
}

extern "C" __attribute__((visibility("default"))) int
spires_ext_ridge_solve_noalloc(const double *d_states, const double *d_targets, size_t T,
                               size_t n_, size_t dout_, size_t washout, double lambda,
                               double *d_w_out, void *stream)
{
    if (!d_states || !d_targets || !d_w_out || T == 0 || n_ == 0 || dout_ == 0 || washout >= T)
        return SP_EINVAL;
    if (n_ > SP_NA_MAX_N || dout_ > SP_NA_MAX_DOUT || T > SP_NA_MAX_T) {
        fprintf(stderr,
                "spires_ext_ridge_solve_noalloc: size beyond the fixed work area "
                "(N=%zu > %d, outputs=%zu > %d or rows=%zu > %d)\n",
                n_, SP_NA_MAX_N, dout_, SP_NA_MAX_DOUT, T, SP_NA_MAX_T);
        return SP_EINVAL;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess)
        return SP_EINTERNAL;
    if (dev < 0 || dev >= 64)
        return SP_EINTERNAL;
    std::lock_guard<std::mutex> lock(g_na_lock[dev]);
    const int rc = na_solve(dev, d_states, d_targets, T, (int)n_, (int)dout_, washout, lambda,
                            d_w_out, (cudaStream_t)stream);
    if (rc)
        cudaStreamSynchronize((cudaStream_t)stream);  // nothing of it is left on the work area
    return rc;
}
