// dev_surrogate.cu -- the learned surrogate of the hyper-parameter search.
//
// An MLP 10 -> 128 -> 128 -> 2 with GELU (erf form) that maps a candidate's
// features (hyper-parameters plus its low-fidelity loss) to the mean and the
// log-variance of its full-fidelity log-NRMSE. Trained on the device with
// the Gaussian negative log-likelihood
//     loss = mean_s 0.5 * (v_s + (y_s - m_s)^2 * exp(-v_s))
// by Adam, all in FP32; inference can round weights and activations to BF16
// (FP32 accumulation).
//
// Every product is one of three tiled FP32 GEMM forms on 32x32 tiles staged
// in shared memory:
//     NT: C[i][j] = sum_k A[i][k] B[j][k]   (activations x weights^T)
//     NN: C[i][j] = sum_k A[i][k] B[k][j]   (output gradients x weights)
//     TN: C[i][j] = sum_k A[k][i] B[k][j]   (weight gradients over the batch)
// with fused epilogues (bias, GELU and its pre-activation store, gradient
// scaling by GELU'). The network is 18k parameters and the batches are a few
// thousand rows, so these are latency-sized launches; the layer shapes do
// not fill a tensor-core tile schedule worth its setup.
//
// Training runs a whole epoch in one launch (k_train): one cluster of 16 CTAs
// keeps the parameters in shared memory and meets twice per minibatch.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "sp_alloc.h"
#include "sp_dev.h"
#include "sp_dev_internal.h"

namespace {

constexpr int kIn = 10, kHid = 128, kOut = 2;
constexpr int kP1 = kHid * kIn, kP1b = kHid, kP2 = kHid * kHid, kP2b = kHid, kP3 = kOut * kHid,
              kP3b = kOut;
constexpr int kParams = kP1 + kP1b + kP2 + kP2b + kP3 + kP3b;
// parameter offsets: W1 [128][10], b1, W2 [128][128], b2, W3 [2][128], b3
constexpr int oW1 = 0, ob1 = oW1 + kP1, oW2 = ob1 + kP1b, ob2 = oW2 + kP2, oW3 = ob2 + kP2b,
              ob3 = oW3 + kP3;

constexpr int TILE = 32;

enum Epi : int { EPI_NONE = 0, EPI_BIAS = 1, EPI_BIAS_GELU = 2, EPI_GELU_GRAD = 3 };

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

__device__ __forceinline__ float gelu_grad(float x)
{
    // d/dx x Phi(x) = Phi(x) + x phi(x)
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

__device__ __forceinline__ float to_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// Generic tiled GEMM. FORM 0 = NT, 1 = NN, 2 = TN (see the file comment).
// C is M x N (ldc); A, B as the form reads them. Epilogues:
//   EPI_BIAS       C = acc + bias[j]
//   EPI_BIAS_GELU  Z = acc + bias[j] (stored to Zout), C = gelu(Z)
//   EPI_GELU_GRAD  C = acc * gelu'(Zin[i][j])
// bf16: round both operands to BF16 as they are staged (inference only).
template <int FORM>
__global__ void __launch_bounds__(256) k_gemm(int M, int N, int K, const float *__restrict__ A,
                                              int lda, const float *__restrict__ B, int ldb,
                                              float *__restrict__ C, int ldc,
                                              const float *__restrict__ bias, int epi,
                                              float *__restrict__ Zout, const float *__restrict__ Zin,
                                              int ldz, int bf16, int round_out)
{
    __shared__ float sA[TILE][TILE + 1];
    __shared__ float sB[TILE][TILE + 1];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8 threads
    const int i0 = blockIdx.y * TILE, j0 = blockIdx.x * TILE;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};  // rows ty, ty+8, ty+16, ty+24 of the tile; column tx
    for (int k0 = 0; k0 < K; k0 += TILE) {
        for (int r = ty; r < TILE; r += 8) {
            // sA[r][c] = A(i0 + r, k0 + c); sB[c][r'] holds B(k0 + c, j0 + r')
            const int c = tx;
            float a = 0.f, bv = 0.f;
            const int ia = i0 + r, ka = k0 + c;
            if (ia < M && ka < K)
                a = (FORM == 2) ? A[(size_t)ka * lda + ia] : A[(size_t)ia * lda + ka];
            const int jb = j0 + r, kb = k0 + c;
            if (jb < N && kb < K)
                bv = (FORM == 0) ? B[(size_t)jb * ldb + kb] : B[(size_t)kb * ldb + jb];
            if (bf16) {
                a = to_bf16(a);
                bv = to_bf16(bv);
            }
            sA[r][c] = a;
            sB[r][c] = bv;  // sB[j][k]
        }
        __syncthreads();
#pragma unroll 8
        for (int k = 0; k < TILE; ++k) {
            const float bk = sB[tx][k];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                acc[q] = fmaf(sA[ty + 8 * q][k], bk, acc[q]);
        }
        __syncthreads();
    }
    const int j = j0 + tx;
    if (j >= N)
        return;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int i = i0 + ty + 8 * q;
        if (i >= M)
            continue;
        float v = acc[q];
        if (epi == EPI_BIAS || epi == EPI_BIAS_GELU)
            v += bias[j];
        if (epi == EPI_BIAS_GELU) {
            if (Zout)
                Zout[(size_t)i * ldz + j] = v;
            v = gelu(v);
        } else if (epi == EPI_GELU_GRAD) {
            v *= gelu_grad(Zin[(size_t)i * ldz + j]);
        }
        if (round_out)
            v = to_bf16(v);
        C[(size_t)i * ldc + j] = v;
    }
}

// Column sums (bias gradients): g[j] = sum_s D[s][j], fixed order per column.
__global__ void k_colsum(const float *__restrict__ D, int B, int N, float *__restrict__ g)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= N)
        return;
    float a = 0.f;
    for (int s = 0; s < B; ++s)
        a += D[(size_t)s * N + j];
    g[j] = a;
}

// loss = sum of row terms / B (one block, fixed tree)
__global__ void k_mean(const float *__restrict__ x, int B, float *out)
{
    __shared__ float part[256];
    float a = 0.f;
    for (int s = threadIdx.x; s < B; s += 256)
        a += x[s];
    part[threadIdx.x] = a;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w)
            part[threadIdx.x] += part[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        *out = part[0] / (float)B;
}

// The rows of a minibatch, gathered by the epoch's row order.
__global__ void k_take_rows(const float *__restrict__ X, const float *__restrict__ y,
                            const int *__restrict__ perm, int B, float *__restrict__ xb,
                            float *__restrict__ yb)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= B)
        return;
    const int r = perm[s];
    for (int k = 0; k < kIn; ++k)
        xb[(size_t)s * kIn + k] = X[(size_t)r * kIn + k];
    yb[s] = y[r];
}

// Adam (Kingma & Ba 2015) with bias correction; step t >= 1.
__device__ __forceinline__ void adam_step(float &p, float gi, float &m1, float &m2, float lr,
                                          float b1, float b2, float eps, float c1, float c2)
{
    const float a = b1 * m1 + (1.0f - b1) * gi;
    const float b = b2 * m2 + (1.0f - b2) * gi * gi;
    m1 = a;
    m2 = b;
    p -= lr * (a / c1) / (sqrtf(b / c2) + eps);
}

__global__ void k_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m1,
                       float *__restrict__ m2, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        adam_step(p[i], g[i], m1[i], m2[i], lr, b1, b2, eps, c1, c2);
}

// dL/d(out) of one row (out = mean, log-variance), scaled by inv = 1/B, and the
// row's loss term.
__device__ __forceinline__ void nll_row(float m, float v, float y, float inv, float &d0, float &d1,
                                        float &loss)
{
    const float r = y - m, iv = expf(-v);
    d0 = -r * iv * inv;
    d1 = 0.5f * (1.0f - r * r * iv) * inv;
    loss = 0.5f * (v + r * r * iv);
}

// The same for rows [0, B), one thread per row.
__global__ void k_nll_grad(const float *__restrict__ out, const float *__restrict__ y, int B,
                           float *__restrict__ dout, float *__restrict__ row_loss)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < B)
        nll_row(out[2 * s], out[2 * s + 1], y[s], 1.0f / (float)B, dout[2 * s], dout[2 * s + 1],
                row_loss[s]);
}

// ------------------------------------------------------- fused training epoch
// All minibatches of one epoch in one launch: a cluster of kTC CTAs, each with
// its own copy of the parameters in shared memory. Per minibatch of B rows
//   rows     CTA q runs every kTC-th tile of 16 rows forward and back to the
//            layer gradients, 2 rows x 4 columns of a layer per thread, and
//            writes H1, H2, dZ1, dZ2 and dL/d(out) to memory
//   cluster barrier
//   weights  CTA q sums the gradients it owns over all rows in ascending order
//            (a 32 x 32 block of W2, 8 rows of W1, 8 columns of W3, the biases
//            with them) and takes their Adam step
//   cluster barrier, then every CTA reads the new parameters
// Every sum runs over the same terms in the same order as the separate kernels
// above (and so gives the same bits): only the launches between them are gone.
// What bounds it: the shared-memory reads of the two 128 x 128 products and the
// two barriers with the parameter reads behind them; 256 rows take about 20 us
// where 14 launches took 172.
constexpr int kTC = 16;           // CTAs of the cluster
constexpr int kTT = 256;          // threads
constexpr int kTR = 16;           // rows of a tile
constexpr int kTS = 256;          // rows of a staged block in the weight phase
constexpr int kW1P = kIn + 1, kHP = kHid + 4;  // padded pitches

struct TrainArgs {
    float *p, *m1, *m2;
    const float *X, *y;           // all rows
    const int *perm;              // row order of the epoch
    const float2 *corr;           // Adam's bias corrections of each minibatch
    float *H1, *H2, *dZ1, *dZ2, *dO, *rl;  // [batch][..] activations and gradients
    int n, batch, steps;
    float lr, b1, b2, eps;
};

struct TrainSmem {
    float W1[kHid * kW1P], b1[kHid], W2[kHid][kHP], b2[kHid], W3[kOut * kHid], b3[4];
    union {
        struct {
            float X[kTR][12], H1[kTR][kHP], H2[kTR][kHP], D2[kTR][kHP], dO[kTR][2];
        } r;
        struct {
            float D2[kTS][32], H1[kTS][32], D1[kTS][8], H2[kTS][8], X[kTS][kIn], dO[kTS][2];
        } w;
    };
};

// Asynchronous copies of 16 and 4 bytes through the L2 (activations and
// parameters that other CTAs have just written).
__device__ __forceinline__ void copy16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy4(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copies_done()
{
    asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;" ::: "memory");
}

__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;"
                 ::: "memory");
}

// acc[q][c] = sum_k A[q][k] W(lane + 32 c, k), k ascending: W(j, k) is W2[j][k]
// (the layer forward; 16-byte loads, conflict-free at this pitch) or W2[k][j]
// (its transpose, for the gradient).
template <bool kTrans>
__device__ __forceinline__ void layer_128(float (&acc)[2][4], const float (*A)[kHP],
                                          const float (*W)[kHP], int lane)
{
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int c = 0; c < 4; ++c)
            acc[q][c] = 0.f;
#pragma unroll 4
    for (int k = 0; k < kHid; k += 4) {
        float a[2][4], w[4][4];
#pragma unroll
        for (int q = 0; q < 2; ++q)
            *(float4 *)a[q] = *(const float4 *)&A[q][k];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (!kTrans) {
                *(float4 *)w[c] = *(const float4 *)&W[lane + 32 * c][k];
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    w[c][u] = W[k + u][lane + 32 * c];
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    acc[q][c] = fmaf(a[q][u], w[c][u], acc[q][c]);
    }
}

__global__ void __launch_bounds__(kTT, 1) k_train(TrainArgs t)
{
    extern __shared__ __align__(16) unsigned char train_smem[];
    TrainSmem &S = *(TrainSmem *)train_smem;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cta = blockIdx.x;  // the grid is one cluster

    for (int st = 0; st < t.steps; ++st) {
        const int s0 = st * t.batch;
        const int B = s0 + t.batch <= t.n ? t.batch : t.n - s0;
        const int *perm = t.perm + s0;
        // ---- the parameters (written by their owners before the last barrier;
        // read past the L1, which may hold the step before's)
        {
            float w1[kP1 / kTT];
#pragma unroll
            for (int k = 0; k < kP1 / kTT; ++k)
                w1[k] = __ldcg(t.p + oW1 + k * kTT + tid);
            const float b = __ldcg(t.p + (tid < kHid ? ob1 + tid : ob2 + tid - kHid));
            const float w3 = __ldcg(t.p + oW3 + tid);
            const float b3 = __ldcg(t.p + ob3 + (tid & 1));
#pragma unroll
            for (int k = 0; k < kP2 / 4 / kTT; ++k) {
                const int e = k * kTT + tid;
                copy16(&S.W2[e / 32][e % 32 * 4], t.p + oW2 + 4 * e);
            }
#pragma unroll
            for (int k = 0; k < kP1 / kTT; ++k) {
                const int e = k * kTT + tid;
                S.W1[e / kIn * kW1P + e % kIn] = w1[k];
            }
            (tid < kHid ? S.b1 : S.b2)[tid & (kHid - 1)] = b;
            S.W3[tid] = w3;
            if (tid < kOut)
                S.b3[tid] = b3;
            copies_done();
        }
        // ---- rows: tile g of 16 rows belongs to CTA g % kTC
        const float inv = 1.0f / (float)B;
        for (int g = cta; g * kTR < B; g += kTC) {
            const int base = g * kTR, cnt = B - base < kTR ? B - base : kTR;
            __syncthreads();
            for (int k = tid; k < kTR * kIn; k += kTT) {
                const int r = k / kIn, c = k % kIn;
                S.r.X[r][c] = r < cnt ? __ldg(t.X + (size_t)__ldg(perm + base + r) * kIn + c) : 0.f;
            }
            __syncthreads();
            // a warp takes two rows from here to their gradients by itself
            const int r0 = 2 * warp;
            const bool on[2] = {r0 < cnt, r0 + 1 < cnt};
            size_t row[2];
#pragma unroll
            for (int q = 0; q < 2; ++q)
                row[q] = (size_t)(base + r0 + q) * kHid + lane;
            float z1[2][4], z2[2][4];
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int j = lane + 32 * c;
                    float acc = 0.f;
#pragma unroll
                    for (int k = 0; k < kIn; ++k)
                        acc = fmaf(S.r.X[r0 + q][k], S.W1[j * kW1P + k], acc);
                    z1[q][c] = acc + S.b1[j];
                    const float h = gelu(z1[q][c]);
                    S.r.H1[r0 + q][j] = h;
                    if (on[q])
                        t.H1[row[q] + 32 * c] = h;
                }
            __syncwarp();
            layer_128<false>(z2, S.r.H1 + r0, S.W2, lane);
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int j = lane + 32 * c;
                    z2[q][c] += S.b2[j];
                    const float h = gelu(z2[q][c]);
                    S.r.H2[r0 + q][j] = h;
                    if (on[q])
                        t.H2[row[q] + 32 * c] = h;
                }
            __syncwarp();
            // output layer and its gradient: lane 2q + o of the warp's rows
            float o = 0.f;
            {
                const float *h = S.r.H2[r0 + ((lane >> 1) & 1)];
                const float *w = S.W3 + (lane & 1) * kHid;
#pragma unroll 4
                for (int k = 0; k < kHid; k += 4) {
                    const float4 x = *(const float4 *)(h + k), v = *(const float4 *)(w + k);
                    o = fmaf(x.x, v.x, o);
                    o = fmaf(x.y, v.y, o);
                    o = fmaf(x.z, v.z, o);
                    o = fmaf(x.w, v.w, o);
                }
                o += S.b3[lane & 1];
            }
            const float v = __shfl_sync(0xffffffffu, o, lane | 1);
            const int r = r0 + (lane >> 1);
            if (lane < 4 && !(lane & 1)) {
                float d0 = 0.f, d1 = 0.f, loss = 0.f;
                if (r < cnt) {
                    nll_row(o, v, __ldg(t.y + __ldg(perm + base + r)), inv, d0, d1, loss);
                    t.dO[2 * (base + r)] = d0;
                    t.dO[2 * (base + r) + 1] = d1;
                    t.rl[base + r] = loss;
                }
                S.r.dO[r][0] = d0;
                S.r.dO[r][1] = d1;
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int j = lane + 32 * c;
                    float d = fmaf(S.r.dO[r0 + q][0], S.W3[j], 0.f);
                    d = fmaf(S.r.dO[r0 + q][1], S.W3[kHid + j], d);
                    d *= gelu_grad(z2[q][c]);
                    S.r.D2[r0 + q][j] = d;
                    if (on[q])
                        t.dZ2[row[q] + 32 * c] = d;
                }
            __syncwarp();
            layer_128<true>(z2, S.r.D2 + r0, S.W2, lane);
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (on[q])
                        t.dZ1[row[q] + 32 * c] = z2[q][c] * gelu_grad(z1[q][c]);
        }
        cluster_barrier();
        // ---- weights: this CTA's block of W2 is rows 32 bi.., columns 32 bj..
        const int bi = cta >> 2, bj = cta & 3, c8 = 8 * cta;
        float gw[4][2] = {}, ga = 0.f, gb = 0.f;
        // what this thread owns: 8 entries of W2 (at[0] + 128 q + c), or up to two
        // others; their Adam state is loaded ahead of the sums
        int at[2] = {-1, -1};
        if (warp < 4) {
            at[0] = oW2 + (32 * bi + 4 * (tid >> 4)) * kHid + 32 * bj + 2 * (tid & 15);
        } else {
            const int q = tid - 128;
            at[0] = q < 80 ? oW1 + (c8 + q / kIn) * kIn + q % kIn
                    : q < 96 ? oW3 + ((q - 80) & 1) * kHid + c8 + ((q - 80) >> 1)
                    : bj == 0 ? ob2 + 32 * bi + q - 96
                              : -1;
            at[1] = q < 8 ? ob1 + c8 + q : (cta == 0 && q < 10 ? ob3 + q - 8 : -1);
        }
        float pv[4][2], v1[4][2], v2[4][2];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int i = warp < 4 ? at[0] + q * kHid + c : (q == 0 ? at[c] : -1);
                const bool own = i >= 0;
                pv[q][c] = own ? t.p[i] : 0.f;
                v1[q][c] = own ? t.m1[i] : 0.f;
                v2[q][c] = own ? t.m2[i] : 0.f;
            }
        for (int w0 = 0; w0 < B; w0 += kTS) {
            const int cnt = B - w0 < kTS ? B - w0 : kTS;
            __syncthreads();
            for (int k = tid; k < cnt * 8; k += kTT) {
                const int r = k >> 3, c = (k & 7) * 4;
                copy16(&S.w.D2[r][c], t.dZ2 + (size_t)(w0 + r) * kHid + 32 * bi + c);
                copy16(&S.w.H1[r][c], t.H1 + (size_t)(w0 + r) * kHid + 32 * bj + c);
            }
            for (int k = tid; k < cnt * 2; k += kTT) {
                const int r = k >> 1, c = (k & 1) * 4;
                copy16(&S.w.D1[r][c], t.dZ1 + (size_t)(w0 + r) * kHid + c8 + c);
                copy16(&S.w.H2[r][c], t.H2 + (size_t)(w0 + r) * kHid + c8 + c);
            }
            for (int k = tid; k < cnt; k += kTT) {
                const float *x = t.X + (size_t)__ldg(perm + w0 + k) * kIn;
#pragma unroll
                for (int c = 0; c < kIn; ++c)
                    copy4(&S.w.X[k][c], x + c);
                // written by another CTA: not through the L1
                const float2 d = __ldcg((const float2 *)t.dO + w0 + k);
                S.w.dO[k][0] = d.x;
                S.w.dO[k][1] = d.y;
            }
            copies_done();
            __syncthreads();
            if (warp < 4) {
                // 4 rows x 2 columns of the W2 block per thread
                const int i0 = 4 * (tid >> 4), j0 = 2 * (tid & 15);
#pragma unroll 4
                for (int r = 0; r < cnt; ++r) {
                    const float4 a = *(const float4 *)&S.w.D2[r][i0];
                    const float2 h = *(const float2 *)&S.w.H1[r][j0];
                    gw[0][0] = fmaf(a.x, h.x, gw[0][0]);
                    gw[0][1] = fmaf(a.x, h.y, gw[0][1]);
                    gw[1][0] = fmaf(a.y, h.x, gw[1][0]);
                    gw[1][1] = fmaf(a.y, h.y, gw[1][1]);
                    gw[2][0] = fmaf(a.z, h.x, gw[2][0]);
                    gw[2][1] = fmaf(a.z, h.y, gw[2][1]);
                    gw[3][0] = fmaf(a.w, h.x, gw[3][0]);
                    gw[3][1] = fmaf(a.w, h.y, gw[3][1]);
                }
            } else {
                // 80 entries of W1, 16 of W3 (threads 0..95), then the biases:
                // 8 of b1, 32 of b2 (CTAs with bj = 0), 2 of b3 (CTA 0)
                const int q = tid - 128;
                if (q < 80) {
                    const int i = q / kIn, c = q % kIn;
#pragma unroll 8
                    for (int r = 0; r < cnt; ++r)
                        ga = fmaf(S.w.D1[r][i], S.w.X[r][c], ga);
                } else if (q < 96) {
                    const int o = (q - 80) & 1, c = (q - 80) >> 1;
#pragma unroll 8
                    for (int r = 0; r < cnt; ++r)
                        ga = fmaf(S.w.dO[r][o], S.w.H2[r][c], ga);
                } else if (bj == 0) {
#pragma unroll 8
                    for (int r = 0; r < cnt; ++r)
                        ga += S.w.D2[r][q - 96];
                }
                if (q < 8) {
#pragma unroll 8
                    for (int r = 0; r < cnt; ++r)
                        gb += S.w.D1[r][q];
                } else if (cta == 0 && q < 10) {
#pragma unroll 8
                    for (int r = 0; r < cnt; ++r)
                        gb += S.w.dO[r][q - 8];
                }
            }
        }
        // ---- Adam on what this CTA owns
        const float c1 = __ldg(&t.corr[st].x), c2 = __ldg(&t.corr[st].y);
        if (warp >= 4) {
            gw[0][0] = ga;
            gw[0][1] = gb;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int i = warp < 4 ? at[0] + q * kHid + c : (q == 0 ? at[c] : -1);
                if (i < 0)
                    continue;
                adam_step(pv[q][c], gw[q][c], v1[q][c], v2[q][c], t.lr, t.b1, t.b2, t.eps, c1, c2);
                t.p[i] = pv[q][c];
                t.m1[i] = v1[q][c];
                t.m2[i] = v2[q][c];
            }
        cluster_barrier();
    }
}

// PCG32 (O'Neill 2014) for the seeded initialisation and batch shuffles.
struct Pcg {
    uint64_t s;
    uint32_t next()
    {
        const uint64_t old = s;
        s = old * 6364136223846793005ull + 1442695040888963407ull;
        const uint32_t xs = (uint32_t)(((old >> 18) ^ old) >> 27);
        const uint32_t rot = (uint32_t)(old >> 59);
        return (xs >> rot) | (xs << ((32u - rot) & 31u));
    }
    float uniform() { return (float)(next() >> 8) * (1.0f / 16777216.0f); }
};

}  // namespace

struct sp_mlp {
    cudaStream_t stream = nullptr;
    float *p = nullptr, *g = nullptr, *m1 = nullptr, *m2 = nullptr;
    int cap = 0;  // rows the work buffers hold
    float *X = nullptr, *y = nullptr, *Z1 = nullptr, *H1 = nullptr, *Z2 = nullptr, *H2 = nullptr,
          *O = nullptr, *dO = nullptr, *dH2 = nullptr, *dH1 = nullptr, *rl = nullptr,
          *loss = nullptr, *pb = nullptr;
    // training: all rows, and two epochs' row orders and bias corrections
    int cap_rows = 0, cap_steps = 0;
    float *Xall = nullptr, *yall = nullptr;
    int *d_perm = nullptr, *h_perm = nullptr;        // [2][cap_rows]
    float2 *d_corr = nullptr, *h_corr = nullptr;     // [2][cap_steps]
    cudaEvent_t epoch_done[2] = {nullptr, nullptr};
    int fused = -1;         // the cluster launch is available (-1: not asked yet)
    long long t = 0;        // Adam steps taken
    long long launches = 0; // kernels launched
};

#define MK(x)                                                                      \
    do {                                                                           \
        cudaError_t e_ = (x);                                                      \
        if (e_ != cudaSuccess) {                                                   \
            sp_dev_note_error(#x, e_);                                             \
            return (e_ == cudaErrorMemoryAllocation) ? SP_EALLOC : SP_EINTERNAL;   \
        }                                                                          \
    } while (0)

static void mlp_free_work(sp_mlp *m)
{
    float *bufs[] = {m->X, m->y, m->Z1, m->H1, m->Z2, m->H2, m->O, m->dO, m->dH2, m->dH1, m->rl};
    for (float *b : bufs)
        if (b)
            sp_cuda_free(b);
    m->X = m->y = m->Z1 = m->H1 = m->Z2 = m->H2 = m->O = m->dO = m->dH2 = m->dH1 = m->rl =
        nullptr;
    m->cap = 0;
}

static int mlp_reserve(sp_mlp *m, int rows)
{
    if (rows <= m->cap)
        return SP_OK;
    mlp_free_work(m);
    const size_t r = (size_t)rows;
    MK(sp_cuda_malloc(&m->X, r * kIn * 4));
    MK(sp_cuda_malloc(&m->y, r * 4));
    MK(sp_cuda_malloc(&m->Z1, r * kHid * 4));
    MK(sp_cuda_malloc(&m->H1, r * kHid * 4));
    MK(sp_cuda_malloc(&m->Z2, r * kHid * 4));
    MK(sp_cuda_malloc(&m->H2, r * kHid * 4));
    MK(sp_cuda_malloc(&m->O, r * kOut * 4));
    MK(sp_cuda_malloc(&m->dO, r * kOut * 4));
    MK(sp_cuda_malloc(&m->dH2, r * kHid * 4));
    MK(sp_cuda_malloc(&m->dH1, r * kHid * 4));
    MK(sp_cuda_malloc(&m->rl, r * 4));
    m->cap = rows;
    return SP_OK;
}

template <int FORM>
static void gemm(sp_mlp *m, int M, int N, int K, const float *A, int lda, const float *B, int ldb,
                 float *C, int ldc, const float *bias, int epi, float *Zout, const float *Zin,
                 int ldz, int bf16, int round_out)
{
    dim3 grid((N + TILE - 1) / TILE, (M + TILE - 1) / TILE);
    k_gemm<FORM><<<grid, 256, 0, m->stream>>>(M, N, K, A, lda, B, ldb, C, ldc, bias, epi, Zout,
                                               Zin, ldz, bf16, round_out);
    m->launches++;
}

// forward over rows [0, B) of m->X (params P), outputs in m->O
static void forward(sp_mlp *m, const float *P, int B, int bf16)
{
    gemm<0>(m, B, kHid, kIn, m->X, kIn, P + oW1, kIn, m->H1, kHid, P + ob1, EPI_BIAS_GELU, m->Z1,
            nullptr, kHid, bf16, bf16);
    gemm<0>(m, B, kHid, kHid, m->H1, kHid, P + oW2, kHid, m->H2, kHid, P + ob2, EPI_BIAS_GELU,
            m->Z2, nullptr, kHid, bf16, bf16);
    gemm<0>(m, B, kOut, kHid, m->H2, kHid, P + oW3, kHid, m->O, kOut, P + ob3, EPI_BIAS, nullptr,
            nullptr, 0, bf16, 0);
}

// loss and gradient (into m->g) for rows [0, B) of m->X / m->y
static void backward(sp_mlp *m, int B)
{
    const float *P = m->p;
    float *G = m->g;
    k_nll_grad<<<(B + 255) / 256, 256, 0, m->stream>>>(m->O, m->y, B, m->dO, m->rl);
    k_mean<<<1, 256, 0, m->stream>>>(m->rl, B, m->loss);
    m->launches += 2;
    // layer 3
    gemm<2>(m, kOut, kHid, B, m->dO, kOut, m->H2, kHid, G + oW3, kHid, nullptr, EPI_NONE, nullptr,
            nullptr, 0, 0, 0);
    k_colsum<<<1, 32, 0, m->stream>>>(m->dO, B, kOut, G + ob3);
    // dZ2 = (dO W3) * gelu'(Z2)
    gemm<1>(m, B, kHid, kOut, m->dO, kOut, P + oW3, kHid, m->dH2, kHid, nullptr, EPI_GELU_GRAD,
            nullptr, m->Z2, kHid, 0, 0);
    // layer 2
    gemm<2>(m, kHid, kHid, B, m->dH2, kHid, m->H1, kHid, G + oW2, kHid, nullptr, EPI_NONE, nullptr,
            nullptr, 0, 0, 0);
    k_colsum<<<1, kHid, 0, m->stream>>>(m->dH2, B, kHid, G + ob2);
    // dZ1 = (dZ2 W2) * gelu'(Z1)
    gemm<1>(m, B, kHid, kHid, m->dH2, kHid, P + oW2, kHid, m->dH1, kHid, nullptr, EPI_GELU_GRAD,
            nullptr, m->Z1, kHid, 0, 0);
    // layer 1
    gemm<2>(m, kHid, kIn, B, m->dH1, kHid, m->X, kIn, G + oW1, kIn, nullptr, EPI_NONE, nullptr,
            nullptr, 0, 0, 0);
    k_colsum<<<1, kHid, 0, m->stream>>>(m->dH1, B, kHid, G + ob1);
    m->launches += 3;
}

extern "C" int sp_mlp_num_params(void) { return kParams; }

static void train_free(sp_mlp *m);

extern "C" void sp_mlp_destroy(sp_mlp *m)
{
    if (!m)
        return;
    if (m->stream)
        cudaStreamSynchronize(m->stream);
    mlp_free_work(m);
    train_free(m);
    for (cudaEvent_t e : m->epoch_done)
        if (e)
            cudaEventDestroy(e);
    float *bufs[] = {m->p, m->g, m->m1, m->m2, m->loss, m->pb};
    for (float *b : bufs)
        if (b)
            sp_cuda_free(b);
    if (m->stream)
        cudaStreamDestroy(m->stream);
    delete m;
}

// Uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) weights and biases from PCG32.
extern "C" int sp_mlp_create(uint64_t seed, sp_mlp **out)
{
    *out = nullptr;
    sp_mlp *m = new sp_mlp();
    int rc = SP_OK;
    if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess ||
        sp_cuda_malloc(&m->p, kParams * 4) != cudaSuccess || sp_cuda_malloc(&m->g, kParams * 4) != cudaSuccess ||
        sp_cuda_malloc(&m->m1, kParams * 4) != cudaSuccess ||
        sp_cuda_malloc(&m->m2, kParams * 4) != cudaSuccess || sp_cuda_malloc(&m->loss, 4) != cudaSuccess ||
        sp_cuda_malloc(&m->pb, kParams * 4) != cudaSuccess)
        rc = SP_EALLOC;
    if (!rc) {
        std::vector<float> h(kParams);
        Pcg r{seed * 2862933555777941757ull + 3037000493ull};
        auto fill = [&](int off, int cnt, int fan_in) {
            const float a = 1.0f / sqrtf((float)fan_in);
            for (int k = 0; k < cnt; ++k)
                h[off + k] = (2.0f * r.uniform() - 1.0f) * a;
        };
        fill(oW1, kP1, kIn);
        fill(ob1, kP1b, kIn);
        fill(oW2, kP2, kHid);
        fill(ob2, kP2b, kHid);
        fill(oW3, kP3, kHid);
        fill(ob3, kP3b, kHid);
        if (cudaMemcpy(m->p, h.data(), kParams * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
            cudaMemset(m->m1, 0, kParams * 4) != cudaSuccess ||
            cudaMemset(m->m2, 0, kParams * 4) != cudaSuccess)
            rc = SP_EINTERNAL;
    }
    if (rc) {
        cudaGetLastError();
        sp_mlp_destroy(m);
        return rc;
    }
    *out = m;
    return SP_OK;
}

extern "C" int sp_mlp_get_params(sp_mlp *m, float *h)
{
    MK(cudaMemcpy(h, m->p, kParams * 4, cudaMemcpyDeviceToHost));
    return SP_OK;
}

extern "C" int sp_mlp_set_params(sp_mlp *m, const float *h)
{
    MK(cudaMemcpy(m->p, h, kParams * 4, cudaMemcpyHostToDevice));
    MK(cudaMemset(m->m1, 0, kParams * 4));
    MK(cudaMemset(m->m2, 0, kParams * 4));
    m->t = 0;
    return SP_OK;
}

// Loss and gradient of the NLL over n host rows (FP32, no parameter change).
extern "C" int sp_mlp_loss_grad(sp_mlp *m, const float *X, const float *y, int n, float *loss,
                                float *grad)
{
    if (n <= 0)
        return SP_EINVAL;
    int rc = mlp_reserve(m, n);
    if (rc)
        return rc;
    MK(cudaMemcpyAsync(m->X, X, (size_t)n * kIn * 4, cudaMemcpyHostToDevice, m->stream));
    MK(cudaMemcpyAsync(m->y, y, (size_t)n * 4, cudaMemcpyHostToDevice, m->stream));
    forward(m, m->p, n, 0);
    backward(m, n);
    MK(cudaGetLastError());
    MK(cudaMemcpyAsync(loss, m->loss, 4, cudaMemcpyDeviceToHost, m->stream));
    if (grad)
        MK(cudaMemcpyAsync(grad, m->g, kParams * 4, cudaMemcpyDeviceToHost, m->stream));
    MK(cudaStreamSynchronize(m->stream));
    return SP_OK;
}

static void train_free(sp_mlp *m)
{
    void *dv[] = {m->Xall, m->yall, m->d_perm, m->d_corr};
    for (void *b : dv)
        if (b)
            sp_cuda_free(b);
    if (m->h_perm)
        cudaFreeHost(m->h_perm);
    if (m->h_corr)
        cudaFreeHost(m->h_corr);
    m->Xall = m->yall = nullptr;
    m->d_perm = m->h_perm = nullptr;
    m->d_corr = m->h_corr = nullptr;
    m->cap_rows = m->cap_steps = 0;
}

// Buffers for n rows in `steps` minibatches per epoch, kept by the handle.
static int train_reserve(sp_mlp *m, int n, int steps)
{
    for (cudaEvent_t &e : m->epoch_done)
        if (!e)
            MK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    if (n <= m->cap_rows && steps <= m->cap_steps)
        return SP_OK;
    train_free(m);
    const size_t r = (size_t)n, s = (size_t)steps;
    MK(sp_cuda_malloc(&m->Xall, r * kIn * 4));
    MK(sp_cuda_malloc(&m->yall, r * 4));
    MK(sp_cuda_malloc(&m->d_perm, 2 * r * 4));
    MK(sp_cuda_malloc(&m->d_corr, 2 * s * sizeof(float2)));
    MK(cudaMallocHost(&m->h_perm, 2 * r * 4));
    MK(cudaMallocHost(&m->h_corr, 2 * s * sizeof(float2)));
    m->cap_rows = n;
    m->cap_steps = steps;
    return SP_OK;
}

// Whether k_train's cluster can be launched on this device.
static bool train_fused(sp_mlp *m)
{
    if (m->fused < 0) {
        cudaLaunchConfig_t c;
        cudaLaunchAttribute a;
        memset(&c, 0, sizeof(c));
        memset(&a, 0, sizeof(a));
        a.id = cudaLaunchAttributeClusterDimension;
        a.val.clusterDim.x = kTC;
        a.val.clusterDim.y = a.val.clusterDim.z = 1;
        c.gridDim = dim3(kTC);
        c.blockDim = dim3(kTT);
        c.dynamicSmemBytes = sizeof(TrainSmem);
        c.attrs = &a;
        c.numAttrs = 1;
        int n = 0;
        m->fused = cudaFuncSetAttribute(k_train, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)sizeof(TrainSmem)) == cudaSuccess &&
                   cudaFuncSetAttribute(k_train, cudaFuncAttributeNonPortableClusterSizeAllowed,
                                        1) == cudaSuccess &&
                   cudaOccupancyMaxActiveClusters(&n, k_train, &c) == cudaSuccess && n >= 1;
        cudaGetLastError();
    }
    return m->fused == 1;
}

static int launch_train(sp_mlp *m, const TrainArgs &t)
{
    cudaLaunchConfig_t c;
    cudaLaunchAttribute a;
    memset(&c, 0, sizeof(c));
    memset(&a, 0, sizeof(a));
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = kTC;
    a.val.clusterDim.y = a.val.clusterDim.z = 1;
    c.gridDim = dim3(kTC);
    c.blockDim = dim3(kTT);
    c.dynamicSmemBytes = sizeof(TrainSmem);
    c.stream = m->stream;
    c.attrs = &a;
    c.numAttrs = 1;
    MK(cudaLaunchKernelEx(&c, k_train, t));
    m->launches++;
    return SP_OK;
}

// Adam on minibatches of a shuffled copy of the n rows, for `epochs` passes.
// The rows are uploaded once; an epoch is one launch that gathers its
// minibatches by the epoch's row order, which the host draws while the epoch
// before runs. The separate kernels serve a device that cannot schedule the
// cluster.

extern "C" int sp_mlp_train(sp_mlp *m, const float *X, const float *y, int n, int epochs,
                            int batch, float lr, uint64_t seed, float *final_loss)
{
    if (n <= 0 || epochs < 0 || batch <= 0)
        return SP_EINVAL;
    if (batch > n)
        batch = n;
    int rc = mlp_reserve(m, batch);
    if (rc)
        return rc;
    const int steps = (int)(((long long)n + batch - 1) / batch);
    rc = train_reserve(m, n, steps);
    if (rc) {
        train_free(m);
        return rc;
    }
    std::vector<int> perm(n);
    for (int i = 0; i < n; ++i)
        perm[i] = i;
    MK(cudaMemcpyAsync(m->Xall, X, (size_t)n * kIn * 4, cudaMemcpyHostToDevice, m->stream));
    MK(cudaMemcpyAsync(m->yall, y, (size_t)n * 4, cudaMemcpyHostToDevice, m->stream));
    const bool fused = train_fused(m);
    Pcg r{seed ^ 0x5DEECE66Dull};
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    for (int ep = 0; ep < epochs && !rc; ++ep) {
        // Fisher-Yates shuffle of the row order
        for (int i = n - 1; i > 0; --i) {
            const int j = (int)(r.next() % (uint32_t)(i + 1));
            const int t = perm[i];
            perm[i] = perm[j];
            perm[j] = t;
        }
        // the staging of the epoch before the last one is free again
        const int sl = ep & 1;
        if (ep >= 2 && cudaEventSynchronize(m->epoch_done[sl]) != cudaSuccess) {
            rc = SP_EINTERNAL;
            break;
        }
        int *hp = m->h_perm + (size_t)sl * m->cap_rows, *dp = m->d_perm + (size_t)sl * m->cap_rows;
        float2 *hc = m->h_corr + (size_t)sl * m->cap_steps,
               *dc = m->d_corr + (size_t)sl * m->cap_steps;
        memcpy(hp, perm.data(), (size_t)n * 4);
        for (int st = 0; st < steps; ++st) {
            m->t++;
            hc[st] = make_float2(1.0f - powf(b1, (float)m->t), 1.0f - powf(b2, (float)m->t));
        }
        if (cudaMemcpyAsync(dp, hp, (size_t)n * 4, cudaMemcpyHostToDevice, m->stream) !=
                cudaSuccess ||
            cudaMemcpyAsync(dc, hc, (size_t)steps * sizeof(float2), cudaMemcpyHostToDevice,
                            m->stream) != cudaSuccess) {
            rc = SP_EINTERNAL;
            break;
        }
        if (fused) {
            TrainArgs t;
            t.p = m->p;
            t.m1 = m->m1;
            t.m2 = m->m2;
            t.X = m->Xall;
            t.y = m->yall;
            t.perm = dp;
            t.corr = dc;
            t.H1 = m->H1;
            t.H2 = m->H2;
            t.dZ1 = m->dH1;
            t.dZ2 = m->dH2;
            t.dO = m->dO;
            t.rl = m->rl;
            t.n = n;
            t.batch = batch;
            t.steps = steps;
            t.lr = lr;
            t.b1 = b1;
            t.b2 = b2;
            t.eps = eps;
            rc = launch_train(m, t);
        } else {
            for (int st = 0; st < steps; ++st) {
                const int s0 = st * batch;
                const int B = s0 + batch <= n ? batch : n - s0;
                k_take_rows<<<(B + 255) / 256, 256, 0, m->stream>>>(m->Xall, m->yall, dp + s0, B,
                                                                     m->X, m->y);
                forward(m, m->p, B, 0);
                backward(m, B);
                k_adam<<<(kParams + 255) / 256, 256, 0, m->stream>>>(
                    m->p, m->g, m->m1, m->m2, kParams, lr, b1, b2, eps, hc[st].x, hc[st].y);
                m->launches += 2;
            }
        }
        if (!rc && cudaEventRecord(m->epoch_done[sl], m->stream) != cudaSuccess)
            rc = SP_EINTERNAL;
    }
    if (!rc && fused && epochs > 0) {
        // the loss of the last minibatch
        const int last = n - (steps - 1) * batch;
        k_mean<<<1, 256, 0, m->stream>>>(m->rl, last, m->loss);
        m->launches++;
    }
    if (cudaStreamSynchronize(m->stream) != cudaSuccess)
        rc = SP_EINTERNAL;
    if (!rc && final_loss &&
        cudaMemcpy(final_loss, m->loss, 4, cudaMemcpyDeviceToHost) != cudaSuccess)
        rc = SP_EINTERNAL;
    if (cudaGetLastError() != cudaSuccess)
        rc = SP_EINTERNAL;
    return rc;
}

// Predicted (mean, log-variance) for n host rows; bf16 = 1 runs the BF16
// inference path (weights and activations rounded to BF16, products and sums
// in FP32 on the CUDA cores: a 10 -> 128 -> 128 -> 2 network is too small for
// tensor-core tiles to pay).
extern "C" int sp_mlp_predict(sp_mlp *m, const float *X, int n, int bf16, float *mean,
                              float *logvar)
{
    if (n <= 0)
        return SP_EINVAL;
    int rc = mlp_reserve(m, n);
    if (rc)
        return rc;
    MK(cudaMemcpyAsync(m->X, X, (size_t)n * kIn * 4, cudaMemcpyHostToDevice, m->stream));
    forward(m, m->p, n, bf16);
    MK(cudaGetLastError());
    std::vector<float> o((size_t)n * kOut);
    MK(cudaMemcpyAsync(o.data(), m->O, (size_t)n * kOut * 4, cudaMemcpyDeviceToHost, m->stream));
    MK(cudaStreamSynchronize(m->stream));
    for (int s = 0; s < n; ++s) {
        if (mean)
            mean[s] = o[2 * s];
        if (logvar)
            logvar[s] = o[2 * s + 1];
    }
    return SP_OK;
}

extern "C" long long sp_mlp_launches(const sp_mlp *m) { return m->launches; }
