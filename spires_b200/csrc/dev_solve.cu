// dev_solve.cu -- the dense FP64 work of the ridge readout (src/reservoir.c:573-679):
// Gram, Cholesky factorisation, triangular solves.
//
// All products run on the FP64 tensor cores (mma.sync m8n8k4: lane l holds
// A[l / 4][l % 4], B[l % 4][l / 4] and C[l / 4][2 (l % 4) + {0, 1}]), which here
// sustain 37 TFLOP/s, 64 multiply-adds per clock and SM -- the FP64 pipe's rate,
// but for a third of the shared-memory reads that plain FMAs from 4 x 4 register
// tiles need (those ran the Gram at 7-10 TFLOP/s, bound by them).
#include <cuda_runtime.h>
#include <cstdint>
#include "sp_kernels.cuh"
#include "sp_solve.h"

using namespace sp;

namespace {

constexpr int NB = kSolveBlock;
constexpr int kPitch = NB + 4;   // 4 mod 16: fragment loads without bank conflicts
constexpr int kThreads = 256;

__device__ __forceinline__ void mma(double (&c)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}
__device__ __forceinline__ unsigned saddr(const void *p)
{
    return (unsigned)__cvta_generic_to_shared(p);
}
// 16-byte asynchronous copy; bytes = 0 fills with zeros
__device__ __forceinline__ void copy16(void *dst, const void *src, int bytes = 16)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(saddr(dst)), "l"(src),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void copy8(void *dst, const void *src, int bytes = 8)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(saddr(dst)), "l"(src),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ int ld_acquire(const int *p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(int *p, int v)
{
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// ------------------------------------------------------------------- Gram
// Lower tiles of X^T X, BT x BT each, 16 or 32 rows of X per stage, three stages.
// The S CTAs of a cluster take one tile's rows in S contiguous parts and add their
// partial tiles in part order through each other's shared memory, so a small
// matrix with many rows still fills the device and the sum's order is fixed.
// T = 4096: N=200 0.80 -> 0.09 ms, 1000 0.80 -> 0.26, 2000 2.26 -> 0.70, 4000 6.57
// -> 2.70 (24 TFLOP/s; four waves of tiles where 3.4 would do).
template <int BT>
struct GramTile {
    static constexpr int kRows = BT == 32 ? 32 : 16, kStages = 3, kP = BT + 4;
    static constexpr int WM = BT == 128 ? 64 : BT == 64 ? 32 : 8, WN = BT == 128 ? 32 : 16;  // warp tile
    static constexpr int MT = WM / 8, NT = WN / 8;
    static constexpr size_t stage = 2 * (size_t)kRows * kP;  // doubles
    static constexpr size_t smem =
        (kStages * stage > (size_t)BT * BT ? kStages * stage : (size_t)BT * BT) * sizeof(double);
};

template <int BT>
__global__ void __launch_bounds__(kThreads, 1) k_gram(const double *__restrict__ X, int n,
                                                      size_t t0, size_t t1, double *__restrict__ C,
                                                      int ldc, int S, int wide, int more)
{
    using G = GramTile<BT>;
    extern __shared__ __align__(16) double sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tile = blockIdx.x / S, part = blockIdx.x % S;
    int bi = (int)((sqrt(8.0 * tile + 1.0) - 1.0) * 0.5);
    while ((bi + 1) * (bi + 2) / 2 <= tile) ++bi;
    while (bi * (bi + 1) / 2 > tile) --bi;
    const int bj = tile - bi * (bi + 1) / 2;
    const int i0 = bi * BT, j0 = bj * BT;
    const size_t len = t1 - t0;
    const size_t a = t0 + len * part / S, b = t0 + len * (part + 1) / S;
    const int steps = (int)((b - a + G::kRows - 1) / G::kRows);

    auto load = [&](int st) {
        if (st < steps) {
            double *dst = sm + (st % G::kStages) * G::stage;
            const size_t r0 = a + (size_t)st * G::kRows;
            if (wide) {
                constexpr int per = BT / 2;  // 16-byte pieces of a row
                for (int q = tid; q < 2 * G::kRows * per; q += kThreads) {
                    const int r = q / (2 * per), h = q / per % 2, c = q % per * 2;
                    const int col = (h ? j0 : i0) + c;
                    const bool in = r0 + r < b && col < n;
                    copy16(dst + (h * G::kRows + r) * G::kP + c, in ? X + (r0 + r) * n + col : X,
                           in ? 16 : 0);
                }
            } else {
                for (int q = tid; q < 2 * G::kRows * BT; q += kThreads) {
                    const int r = q / (2 * BT), h = q / BT % 2, c = q % BT;
                    const int col = (h ? j0 : i0) + c;
                    const bool in = r0 + r < b && col < n;
                    copy8(dst + (h * G::kRows + r) * G::kP + c, in ? X + (r0 + r) * n + col : X,
                          in ? 8 : 0);
                }
            }
        }
        copy_commit();
    };
    const int wm = warp / (BT / G::WN) * G::WM, wn = warp % (BT / G::WN) * G::WN;
    double acc[G::MT][G::NT][2] = {};
    load(0);
    load(1);
    if (more) {  // the sums over the rows before (S = 1)
#pragma unroll
        for (int m = 0; m < G::MT; ++m)
#pragma unroll
            for (int q = 0; q < G::NT; ++q)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int i = i0 + wm + 8 * m + (lane >> 2);
                    const int j = j0 + wn + 8 * q + 2 * (lane & 3) + e;
                    if (i < n && j <= i)
                        acc[m][q][e] = C[(size_t)i * ldc + j];
                }
    }
    for (int st = 0; st < steps; ++st) {
        copy_wait<1>();
        __syncthreads();
        load(st + 2);
        const double *A = sm + (st % G::kStages) * G::stage, *B = A + G::kRows * G::kP;
#pragma unroll
        for (int k = 0; k < G::kRows; k += 4) {
            double fa[G::MT], fb[G::NT];
#pragma unroll
            for (int m = 0; m < G::MT; ++m)
                fa[m] = A[(k + (lane & 3)) * G::kP + wm + 8 * m + (lane >> 2)];
#pragma unroll
            for (int q = 0; q < G::NT; ++q)
                fb[q] = B[(k + (lane & 3)) * G::kP + wn + 8 * q + (lane >> 2)];
#pragma unroll
            for (int m = 0; m < G::MT; ++m)
#pragma unroll
                for (int q = 0; q < G::NT; ++q)
                    mma(acc[m][q], fa[m], fb[q]);
        }
    }
    copy_wait<0>();
    __syncthreads();
    // the tile in shared memory, then summed over the parts and written
#pragma unroll
    for (int m = 0; m < G::MT; ++m)
#pragma unroll
        for (int q = 0; q < G::NT; ++q)
            *(double2 *)&sm[(wm + 8 * m + (lane >> 2)) * BT + wn + 8 * q + 2 * (lane & 3)] =
                make_double2(acc[m][q][0], acc[m][q][1]);
    auto cluster = [] {
        asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;"
                     ::: "memory");
    };
    if (S > 1)
        cluster();
    else
        __syncthreads();
    const int lo = BT * BT * part / S, hi = BT * BT * (part + 1) / S;
    for (int e = lo + tid; e < hi; e += kThreads) {
        double v = 0.0;
        if (S == 1) {
            v = sm[e];
        } else {
            for (int p = 0; p < S; ++p) {
                unsigned remote;
                double x;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                             : "=r"(remote)
                             : "r"(saddr(sm + e)), "r"(p));
                asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x) : "r"(remote) : "memory");
                v = p == 0 ? x : v + x;
            }
        }
        const int i = i0 + e / BT, j = j0 + e % BT;
        if (i < n && j <= i)
            C[(size_t)i * ldc + j] = v;
    }
    if (S > 1)
        cluster();  // the other CTAs may still read this one's tile
}

// the upper triangle from the lower one, 32 x 32 tiles through shared memory
__global__ void __launch_bounds__(256) k_mirror_upper(double *__restrict__ C, int n, int ldc)
{
    __shared__ double t[32][33];
    const int bi = blockIdx.y, bj = blockIdx.x;
    if (bj > bi)
        return;
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    for (int r = y; r < 32; r += 8) {
        const int i = bi * 32 + r, j = bj * 32 + x;
        t[r][x] = i < n && j < n ? C[(size_t)i * ldc + j] : 0.0;
    }
    __syncthreads();
    for (int r = y; r < 32; r += 8) {
        const int i = bj * 32 + r, j = bi * 32 + x;  // C[i][j] = C[j][i], j > i
        if (i < n && j < n && j > i)
            C[(size_t)i * ldc + j] = t[x][r];
    }
}

__global__ void k_diag_pad(double *A, int n, int np, double lam)
{
    const int i = blockIdx.x;
    if (i < n) {
        if (threadIdx.x == 0)
            A[(size_t)i * np + i] += lam;
        return;
    }
    for (int j = threadIdx.x; j <= i; j += blockDim.x)
        A[(size_t)i * np + j] = i == j ? 1.0 : 0.0;
}

// --------------------------------------------------------- factorisation
// Tile by tile, left-looking: the 64 x 64 tiles of the lower triangle are handed
// out column by column, and the CTA that takes tile (i, j) forms
// A_ij - sum_{k < j} L_ik L_jk^T as those tiles become ready, then factors it
// (i = j) or solves it against L_jj. Every tile depends on earlier ones of that
// order only, so whoever holds the earliest unfinished tile can go on. One
// launch replaces three per panel; a panel's chain (a 64 x 64 factorisation, a
// tile solve, one product, two flags) is what bounds the smaller matrices, the
// FP64 pipe the larger. (N=4000: 7.05 ms with 189 launches, now 1.49; N=1000: 1.18
// -> 0.35 ms, 22 us a panel.)
// Several matrices share a launch, column j of every one before column j + 1 of
// any: one matrix's chain leaves most of the device idle (20 of N 300 to 1600: 4.0
// ms one after the other, 0.8 together).
struct FactorItem {
    double *A;
    int np, nb;
    double *dinv;   // [nb][4][16][16] inverses of the diagonal blocks
    int *flags;     // [nb][nb] tile ready
    int *info;
};
constexpr int kItems = 32;  // matrices of a launch
struct FactorArgs {
    FactorItem item[kItems];
    int count, ntiles;
    int *counter;   // the hand-out
};

constexpr size_t kTile = (size_t)NB * kPitch;  // doubles
constexpr size_t kFactorSmem = (4 * kTile + 4 * 16 * 20 + NB) * sizeof(double);

// A tile of L (pitch np) into shared memory; commit by the caller.
__device__ __forceinline__ void load_tile(double *dst, const double *src, int np)
{
    for (int q = threadIdx.x; q < NB * NB / 2; q += kThreads) {
        const int r = q >> 5, c = (q & 31) * 2;
        copy16(dst + r * kPitch + c, src + (size_t)r * np + c);
    }
}

// Bounded wait of warp 0 for flag words: lane l watches a[l], b[l] (null = set);
// returns how many lanes from 0 on are ready (at least one), or 0 on timeout.
__device__ __forceinline__ int wait_flags(const int *a, const int *b, int *info)
{
    unsigned long long t0 = 0;
    unsigned polls = 0;
    for (;;) {
        const bool ok = (!a || ld_acquire(a)) && (!b || ld_acquire(b));
        const unsigned m = __ballot_sync(kFull, ok);
        if (m & 1u)
            return m == kFull ? 32 : __ffs(~m) - 1;
        if ((++polls & 63u) == 0) {
            const unsigned long long now = globaltimer_ns();
            if (t0 == 0)
                t0 = now;
            const int bad = now - t0 > kBarrierTimeoutNs || ld_volatile_i32(info) == -1;
            if (__any_sync(kFull, bad)) {
                if ((threadIdx.x & 31) == 0)
                    *(volatile int *)info = -1;
                return 0;
            }
        }
        __nanosleep(32);
    }
}

// Factor the 64 x 64 tile T (lower triangle, in place, pitch kPitch), four panels
// of 16 columns; s_inv gets the reciprocals of the diagonal. Returns the
// 1-based failing column in *s_bad (0 = none). All threads.
__device__ __forceinline__ void factor_tile(double *T, double *s_inv, int *s_bad)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int p = 0; p < 4; ++p) {
        const int c0 = 16 * p;
        if (warp == 0) {
            // the diagonal block: lane r < 16 holds row r
            const int r = lane & 15;
            double v[16];
#pragma unroll
            for (int c = 0; c < 16; ++c)
                v[c] = c <= r ? T[(c0 + r) * kPitch + c0 + c] : 0.0;
            double my_inv = 0.0;
            int bad = 0;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const double a = __shfl_sync(kFull, v[j], j);
                const bool ok = a > 0.0 && isfinite(a);
                if (!ok && !bad)
                    bad = c0 + j + 1;
                // sqrt(a) as a * rsqrt(a) and one Newton step for d^2 = a, d + (a - d^2)
                // / (2 d) with inv / 2 for 1 / (2 d)
                const double inv = ok ? rsqrt(a) : 1.0;
                double d = a * inv;
                d = ok ? fma(0.5 * inv, fma(-d, d, a), d) : 1.0;
                if (r == j)
                    my_inv = inv;
                v[j] = r == j ? d : v[j] * inv;
#pragma unroll
                for (int c = j + 1; c < 16; ++c) {
                    const double lc = __shfl_sync(kFull, v[j], c);
                    v[c] = fma(-v[j], lc, v[c]);
                }
            }
            if (lane < 16) {
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    if (c <= r)
                        T[(c0 + r) * kPitch + c0 + c] = v[c];
                s_inv[c0 + r] = my_inv;
            }
            if (lane == 0 && bad && *s_bad == 0)
                *s_bad = bad;
        }
        __syncthreads();
        const int rest = NB - c0 - 16;
        if (rest == 0)
            break;
        // rows below: a thread per row
        if (tid < rest) {
            double *row = T + (c0 + 16 + tid) * kPitch + c0;
            double v[16];
#pragma unroll
            for (int c = 0; c < 16; ++c)
                v[c] = row[c];
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                v[c] *= s_inv[c0 + c];
#pragma unroll
                for (int q = c + 1; q < 16; ++q)
                    v[q] = fma(-v[c], T[(c0 + q) * kPitch + c0 + c], v[q]);
            }
#pragma unroll
            for (int c = 0; c < 16; ++c)
                row[c] = v[c];
        }
        __syncthreads();
        // trailing update of the lower 8 x 8 tiles
        const int m8 = rest / 8, cnt = m8 * (m8 + 1) / 2;
        for (int q = warp; q < cnt; q += kThreads / 32) {
            int bi = 0;
            while ((bi + 1) * (bi + 2) / 2 <= q)
                ++bi;
            const int bj = q - bi * (bi + 1) / 2;
            const int ri = c0 + 16 + 8 * bi, rj = c0 + 16 + 8 * bj;
            double2 *at = (double2 *)&T[(ri + (lane >> 2)) * kPitch + rj + 2 * (lane & 3)];
            double acc[2] = {at->x, at->y};
#pragma unroll
            for (int k = 0; k < 16; k += 4)
                mma(acc, -T[(ri + (lane >> 2)) * kPitch + c0 + k + (lane & 3)],
                    T[(rj + (lane >> 2)) * kPitch + c0 + k + (lane & 3)]);
            *at = make_double2(acc[0], acc[1]);
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kThreads, 1) k_factor(const __grid_constant__ FactorArgs args)
{
    extern __shared__ __align__(16) double sm[];
    double *sA[2] = {sm, sm + kTile}, *sB[2] = {sm + 2 * kTile, sm + 3 * kTile};
    double *s_d = sm + 4 * kTile;          // [4][16][20] inverses of L_jj's blocks
    double *s_inv = s_d + 4 * 16 * 20;     // [64]
    __shared__ int s_item, s_i, s_j, s_ready, s_bad;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = 16 * (warp >> 1), wn = 32 * (warp & 1);
    int col = 0, first = 0;  // thread 0: the column of the last tile, its first tile
    for (;;) {
        if (tid == 0) {
            // column `col` holds tiles (col, col) .. (nb - 1, col) of every matrix
            int t = atomicAdd(args.counter, 1);
            s_item = -1;
            if (t < args.ntiles) {
                for (;;) {
                    int tiles = 0;
                    for (int k = 0; k < args.count; ++k)
                        tiles += args.item[k].nb > col ? args.item[k].nb - col : 0;
                    if (t < first + tiles)
                        break;
                    first += tiles;
                    ++col;
                }
                t -= first;
                int k = 0;
                for (;; ++k) {
                    const int tiles = args.item[k].nb > col ? args.item[k].nb - col : 0;
                    if (t < tiles)
                        break;
                    t -= tiles;
                }
                s_item = k;
                s_i = col + t;
                s_j = col;
            }
        }
        __syncthreads();
        if (s_item < 0)
            return;
        const FactorItem &f = args.item[s_item];
        const int i = s_i, j = s_j, nb = f.nb, np = f.np;
        const bool diag = i == j;
        const double *Li = f.A + (size_t)i * NB * np, *Lj = f.A + (size_t)j * NB * np;
        // A_ij, minus one product after the other: each is summed by itself first,
        // so a long row's rounding errors grow with its tiles, not its terms
        double sum[2][4][2];
        double *Aij = f.A + (size_t)i * NB * np + j * NB;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = wm + 8 * m + (lane >> 2), c = wn + 8 * q + 2 * (lane & 3);
                const double2 v = *(const double2 *)&Aij[(size_t)r * np + c];
                sum[m][q][0] = v.x;
                sum[m][q][1] = v.y;
            }
        int ready = 0;  // k < ready: both tiles are there
        bool dead = false;
        // waits until tiles (i, k) and (j, k) are there; all threads
        auto need = [&](int k) {
            if (k < ready)
                return;
            if (warp == 0) {
                const int kk = k + lane;
                const int got = wait_flags(kk < j ? f.flags + i * nb + kk : nullptr,
                                           kk < j ? f.flags + j * nb + kk : nullptr, f.info);
                if (lane == 0)
                    s_ready = got ? k + got : -1;
            }
            __syncthreads();
            ready = s_ready;
            __syncthreads();
            if (ready < 0)
                dead = true;
        };
        auto load = [&](int k) {
            load_tile(sA[k & 1], Li + k * NB, np);
            if (!diag)
                load_tile(sB[k & 1], Lj + k * NB, np);
            copy_commit();
        };
        if (j > 0) {
            need(0);
            if (dead)
                return;
            load(0);
        }
        for (int k = 0; k < j; ++k) {
            // the next tiles while these are multiplied, when they are known to
            // be there; else after
            const bool ahead = k + 1 < j && k + 1 < ready;
            if (ahead) {
                load(k + 1);
                copy_wait<1>();
            } else {
                copy_wait<0>();
            }
            __syncthreads();
            const double *A = sA[k & 1], *B = diag ? A : sB[k & 1];
            double acc[2][4][2] = {};
#pragma unroll 4
            for (int kk = 0; kk < NB; kk += 4) {
                double fa[2], fb[4];
#pragma unroll
                for (int m = 0; m < 2; ++m)
                    fa[m] = A[(wm + 8 * m + (lane >> 2)) * kPitch + kk + (lane & 3)];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    fb[q] = B[(wn + 8 * q + (lane >> 2)) * kPitch + kk + (lane & 3)];
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        mma(acc[m][q], fa[m], fb[q]);
            }
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    sum[m][q][0] -= acc[m][q][0];
                    sum[m][q][1] -= acc[m][q][1];
                }
            __syncthreads();  // this stage is free
            if (!ahead && k + 1 < j) {
                need(k + 1);
                if (dead)
                    return;
                load(k + 1);
            }
        }
        double *T = sA[0];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = wm + 8 * m + (lane >> 2), c = wn + 8 * q + 2 * (lane & 3);
                *(double2 *)&T[r * kPitch + c] = make_double2(sum[m][q][0], sum[m][q][1]);
            }
        double *dj = f.dinv + (size_t)j * 4 * 256;
        if (diag) {
            if (tid == 0)
                s_bad = 0;
            __syncthreads();
            factor_tile(T, s_inv, &s_bad);
            // inverses of the four diagonal blocks: lane c < 16 of warp p takes
            // column c
            if (warp < 4 && lane < 16) {
                const double *D = T + (16 * warp) * kPitch + 16 * warp;
                double y[16];
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    double s = r == lane ? 1.0 : 0.0;
#pragma unroll
                    for (int q = 0; q < r; ++q)
                        s = fma(-D[r * kPitch + q], y[q], s);
                    y[r] = s * s_inv[16 * warp + r];
                    dj[warp * 256 + r * 16 + lane] = y[r];
                }
            }
            if (tid == 0 && s_bad)
                atomicCAS(f.info, 0, j * NB + s_bad);
        } else {
            if (warp == 0) {
                const int *fl = f.flags + j * nb + j;
                const int got = wait_flags(fl, nullptr, f.info);
                if (lane == 0)
                    s_ready = got;
            }
            __syncthreads();
            if (s_ready == 0)
                return;
            load_tile(sB[0], Lj + j * NB, np);
            for (int q = tid; q < 4 * 16 * 8; q += kThreads) {
                const int r = q >> 3, c = (q & 7) * 2;
                copy16(s_d + r * 20 + c, dj + r * 16 + c);
            }
            copy_commit();
            copy_wait<0>();
            __syncthreads();
            // X L_jj^T = T, a warp per eight rows, 16 columns at a time
            const double *L = sB[0];
            double *Tw = T + 8 * warp * kPitch;
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                double x[2][2];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const double2 v =
                        *(const double2 *)&Tw[(lane >> 2) * kPitch + 16 * p + 8 * q + 2 * (lane & 3)];
                    x[q][0] = v.x;
                    x[q][1] = v.y;
                }
                for (int k = 0; k < 16 * p; k += 4) {
                    const double a = -Tw[(lane >> 2) * kPitch + k + (lane & 3)];
#pragma unroll
                    for (int q = 0; q < 2; ++q)
                        mma(x[q], a, L[(16 * p + 8 * q + (lane >> 2)) * kPitch + k + (lane & 3)]);
                }
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    *(double2 *)&Tw[(lane >> 2) * kPitch + 16 * p + 8 * q + 2 * (lane & 3)] =
                        make_double2(x[q][0], x[q][1]);
                __syncwarp();
                double y[2][2] = {};
#pragma unroll
                for (int k = 0; k < 16; k += 4) {
                    const double a = Tw[(lane >> 2) * kPitch + 16 * p + k + (lane & 3)];
#pragma unroll
                    for (int q = 0; q < 2; ++q)
                        mma(y[q], a, s_d[(16 * p + 8 * q + (lane >> 2)) * 20 + k + (lane & 3)]);
                }
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    *(double2 *)&Tw[(lane >> 2) * kPitch + 16 * p + 8 * q + 2 * (lane & 3)] =
                        make_double2(y[q][0], y[q][1]);
                __syncwarp();
            }
        }
        __syncthreads();
        for (int q = tid; q < NB * NB / 2; q += kThreads) {
            const int r = q >> 5, c = (q & 31) * 2;
            const double2 v = *(const double2 *)&T[r * kPitch + c];
            // above the diagonal the original entries stay
            if (!diag || c + 1 <= r)
                *(double2 *)&Aij[(size_t)r * np + c] = v;
            else if (c <= r)
                Aij[(size_t)r * np + c] = v.x;
        }
        __threadfence();
        __syncthreads();
        if (tid == 0)
            st_release(f.flags + i * nb + j, 1);
    }
}

// ------------------------------------------------------ triangular solves
// L z = b, then L^T x = z, in one launch: CTA c owns row blocks c, c + G, .. and
// subtracts the products with the blocks of the solution as they become ready
// (its tiles of L are fetched ahead of them), then solves against its diagonal
// block through the inverted 16 x 16 blocks. A block's chain -- a flag, a 64 x 64
// product, the diagonal solve -- is what bounds it. (N=4000, one output: 1.70 ms
// with 250 launches, now 0.57; N=1000: 0.37 -> 0.14 ms.)
struct SolveItem {
    const double *L;
    int np, nb, n, dout;
    const double *dinv;
    double *Z;          // [n][dout]
    int *flags, *info;  // [2][nb]
    int cta0, ctas;     // the launch's CTAs that work on it
};
struct SolveArgs {
    SolveItem item[kItems];
    int count;
};

constexpr int kSolveStages = 4;
constexpr size_t kSolveSmem = (kSolveStages * kTile + 4 * 16 * 20 + 3 * NB * 16) * sizeof(double);

// DO: outputs held per thread (dout <= DO).
template <bool kBack, int DO>
__device__ __forceinline__ bool solve_block(const SolveItem &a, double *sm, int i)
{
    double *s_d = sm + kSolveStages * kTile;
    double *s_z = s_d + 4 * 16 * 20;   // [64][dout] a block of the solution
    double *s_t = s_z + NB * 16;       // [64][dout] right-hand side, then the block's own
    double *s_y = s_t + NB * 16;       // [16][dout]
    __shared__ int s_ready;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = a.nb, np = a.np, dout = a.dout;
    const int r = tid >> 2, q = tid & 3;
    // terms: blocks k = 0 .. i - 1 of the solution (back: nb - 1 down to i + 1),
    // with tile (i, k) (back: (k, i), transposed), then tile (i, i)
    const int terms = kBack ? nb - 1 - i : i;
    auto blk = [&](int e) { return kBack ? nb - 1 - e : e; };
    const int *flags = a.flags + (kBack ? nb : 0);
    auto fetch = [&](int e) {
        if (e <= terms) {
            const int k = e < terms ? blk(e) : i;
            const double *src = kBack ? a.L + (size_t)k * NB * np + i * NB
                                      : a.L + (size_t)i * NB * np + k * NB;
            load_tile(sm + (e % kSolveStages) * kTile, src, np);
        }
        copy_commit();
    };
    for (int w = tid; w < 4 * 16 * 8; w += kThreads) {
        const int rr = w >> 3, c = (w & 7) * 2;
        copy16(s_d + rr * 20 + c, a.dinv + (size_t)i * 4 * 256 + rr * 16 + c);
    }
    for (int e = 0; e < kSolveStages - 1; ++e)
        fetch(e);
    double acc[DO];
#pragma unroll
    for (int o = 0; o < DO; ++o)
        acc[o] = 0.0;
    int ready = 0;
    if (kBack) {  // the block's own forward solution, maybe another CTA's
        if (warp == 0) {
            const int got = wait_flags(a.flags + i, nullptr, a.info);
            if (lane == 0)
                s_ready = got;
        }
        __syncthreads();
        if (s_ready == 0) {
            copy_wait<0>();
            return false;
        }
        __syncthreads();
    }
    for (int e = 0; e < terms; ++e) {
        if (e >= ready) {
            if (warp == 0) {
                const int ee = e + lane;
                const int got = wait_flags(ee < terms ? flags + blk(ee) : nullptr, nullptr, a.info);
                if (lane == 0)
                    s_ready = got ? e + got : -1;
            }
            __syncthreads();
            ready = s_ready;
            if (ready < 0) {
                copy_wait<0>();
                return false;
            }
        }
        fetch(e + kSolveStages - 1);
        const int k0 = blk(e) * NB;
        for (int w = tid; w < NB * dout; w += kThreads)
            s_z[w] = k0 + w / dout < a.n ? __ldcg(a.Z + (size_t)k0 * dout + w) : 0.0;
        copy_wait<kSolveStages - 1>();
        __syncthreads();
        const double *T = sm + (e % kSolveStages) * kTile;
        double term[DO];
#pragma unroll
        for (int o = 0; o < DO; ++o)
            term[o] = 0.0;
#pragma unroll 4
        for (int cc = 0; cc < 16; ++cc) {
            const int c = q + 4 * cc;
            const double l = kBack ? T[c * kPitch + r] : T[r * kPitch + c];
#pragma unroll
            for (int o = 0; o < DO; ++o)
                if (DO == 1 || o < dout)
                    term[o] = fma(l, s_z[c * dout + o], term[o]);
        }
#pragma unroll
        for (int o = 0; o < DO; ++o)
            acc[o] += term[o];
        __syncthreads();
    }
    // right-hand side minus the products
#pragma unroll
    for (int o = 0; o < DO; ++o) {
        if (o >= dout)
            break;
        double v = acc[o];
        v += __shfl_xor_sync(kFull, v, 1);
        v += __shfl_xor_sync(kFull, v, 2);
        if (q == 0)
            s_t[r * dout + o] =
                (i * NB + r < a.n ? __ldcg(a.Z + (size_t)(i * NB + r) * dout + o) : 0.0) - v;
    }
    copy_wait<0>();
    __syncthreads();
    // the diagonal block, 16 rows at a time: 4 threads per row and output
    const double *T = sm + (terms % kSolveStages) * kTile;
    for (int pp = 0; pp < 4; ++pp) {
        const int p = kBack ? 3 - pp : pp;
        for (int w = tid >> 2; w < 16 * dout; w += kThreads / 4) {
            const int rr = w / dout, o = w % dout;
            double v = 0.0;
            const int from = kBack ? 16 * (p + 1) : 0, to = kBack ? NB : 16 * p;
            for (int c = from + q; c < to; c += 4) {
                const double l = kBack ? T[c * kPitch + 16 * p + rr] : T[(16 * p + rr) * kPitch + c];
                v = fma(l, s_t[c * dout + o], v);
            }
            v += __shfl_xor_sync(kFull, v, 1);  // 16 dout is a multiple of a warp's 8
            v += __shfl_xor_sync(kFull, v, 2);
            if (q == 0)
                s_y[rr * dout + o] = s_t[(16 * p + rr) * dout + o] - v;
        }
        __syncthreads();
        for (int w = tid >> 2; w < 16 * dout; w += kThreads / 4) {
            const int rr = w / dout, o = w % dout;
            double v = 0.0;
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) {
                const int c = q + 4 * c4;
                const double d = kBack ? s_d[(16 * p + c) * 20 + rr] : s_d[(16 * p + rr) * 20 + c];
                // the inverse is lower triangular; its upper part holds zeros
                v = fma(d, s_y[c * dout + o], v);
            }
            v += __shfl_xor_sync(kFull, v, 1);  // 16 dout is a multiple of a warp's 8
            v += __shfl_xor_sync(kFull, v, 2);
            if (q == 0)
                s_t[(16 * p + rr) * dout + o] = v;
        }
        __syncthreads();
    }
    for (int w = tid; w < NB * dout; w += kThreads)
        if (i * NB + w / dout < a.n)
            a.Z[(size_t)i * NB * dout + w] = s_t[w];
    __threadfence();
    __syncthreads();
    if (tid == 0)
        st_release(const_cast<int *>(flags) + i, 1);
    return true;
}

template <int DO>
__global__ void __launch_bounds__(kThreads, 1) k_solve(const __grid_constant__ SolveArgs args)
{
    extern __shared__ __align__(16) double sm[];
    int k = 0;
    while (k + 1 < args.count && (int)blockIdx.x >= args.item[k + 1].cta0)
        ++k;
    const SolveItem &a = args.item[k];
    const int rank = blockIdx.x - a.cta0;
    for (int i = rank; i < a.nb; i += a.ctas)
        if (!solve_block<false, DO>(a, sm, i))
            return;
    // the last blocks first, each on the CTA that has the same number of blocks
    for (int c = rank; c < a.nb; c += a.ctas) {
        __syncthreads();
        if (!solve_block<true, DO>(a, sm, a.nb - 1 - c))
            return;
    }
}

int sm_count()
{
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 1;
    return v > 0 ? v : 1;
}

template <int BT>
cudaError_t launch_gram(cudaStream_t s, const double *X, int n, size_t t0, size_t t1, double *C,
                        int ldc, int S, bool more)
{
    using G = GramTile<BT>;
    const int nt = (n + BT - 1) / BT, tiles = nt * (nt + 1) / 2;
    cudaError_t e = set_max_dynamic_smem((const void *)k_gram<BT>);
    if (e != cudaSuccess)
        return e;
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute a = {};
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = (unsigned)S;
    a.val.clusterDim.y = a.val.clusterDim.z = 1;
    c.gridDim = dim3((unsigned)(tiles * S));
    c.blockDim = dim3(kThreads);
    c.dynamicSmemBytes = G::smem;
    c.stream = s;
    c.attrs = &a;
    c.numAttrs = 1;
    // 16-byte copies need even row lengths and an aligned base
    const int wide = n % 2 == 0 && ((uintptr_t)X & 15) == 0;
    return cudaLaunchKernelEx(&c, k_gram<BT>, X, n, t0, t1, C, ldc, S, wide, more ? 1 : 0);
}

}  // namespace

// The tile width for n neurons and the parts of `rows` rows.
static int gram_shape(int n, size_t rows, int *parts)
{
    // The widest tile that still fills the SMs; 32-wide ones split their rows over
    // up to 8 CTAs until they do, at least 4096 rows each (a part then takes
    // 90 us; shorter parts would win little).
    const int sms = sm_count();
    auto tiles = [&](long long bt) {
        const long long t = (n + bt - 1) / bt;
        return t * (t + 1) / 2;
    };
    *parts = 1;
    if (tiles(128) >= sms * 9 / 10)
        return 128;
    if (tiles(64) >= sms * 3 / 5)
        return 64;
    while (*parts < 8 && tiles(32) * *parts < sms && rows >= (size_t)8192 * *parts)
        *parts *= 2;
    return 32;
}

bool sp_solve_gram_in_ranges(int n, size_t rows)
{
    int parts;
    gram_shape(n, rows, &parts);
    return parts == 1;
}

cudaError_t sp_solve_gram(cudaStream_t s, const double *X, int n, size_t t0, size_t t1, double *C,
                          int ldc)
{
    return sp_solve_gram_range(s, X, n, t0, t1, C, ldc, false, true);
}

cudaError_t sp_solve_gram_range(cudaStream_t s, const double *X, int n, size_t t0, size_t t1,
                                double *C, int ldc, bool more, bool last)
{
    int S;
    const int bt = gram_shape(n, t1 - t0, &S);
    const cudaError_t e = bt == 128  ? launch_gram<128>(s, X, n, t0, t1, C, ldc, S, more)
                          : bt == 64 ? launch_gram<64>(s, X, n, t0, t1, C, ldc, S, more)
                                     : launch_gram<32>(s, X, n, t0, t1, C, ldc, S, more);
    if (e != cudaSuccess || !last)
        return e;
    const unsigned g = (unsigned)((n + 31) / 32);
    k_mirror_upper<<<dim3(g, g), 256, 0, s>>>(C, n, ldc);
    return cudaGetLastError();
}

cudaError_t sp_solve_diag(cudaStream_t s, double *A, int n, double lambda)
{
    const int np = sp_solve_pad(n);
    k_diag_pad<<<np, 128, 0, s>>>(A, n, np, lambda);
    return cudaGetLastError();
}

cudaError_t sp_solve_factor(cudaStream_t s, const sp_solve_item *items, int count)
{
    cudaError_t e = set_max_dynamic_smem((const void *)k_factor);
    for (int k0 = 0; k0 < count && e == cudaSuccess; k0 += kItems) {
        FactorArgs a;
        a.count = count - k0 < kItems ? count - k0 : kItems;
        a.ntiles = 0;
        a.counter = nullptr;
        for (int k = 0; k < a.count; ++k) {
            const sp_solve_item &it = items[k0 + k];
            FactorItem &f = a.item[k];
            f.A = it.A;
            f.np = sp_solve_pad(it.n);
            f.nb = f.np / NB;
            f.dinv = (double *)it.work;
            f.flags = (int *)(f.dinv + (size_t)f.nb * 4 * 256);
            f.info = it.info;
            a.ntiles += f.nb * (f.nb + 1) / 2;
            if (!a.counter)
                a.counter = f.flags + (size_t)f.nb * f.nb + 2 * f.nb;
            e = cudaMemsetAsync(f.flags, 0, ((size_t)f.nb * f.nb + 2 * f.nb + 4) * sizeof(int), s);
            if (e != cudaSuccess)
                return e;
        }
        const int sms = sm_count();
        void *args[] = {&a};
        e = cudaLaunchCooperativeKernel((const void *)k_factor,
                                        dim3(a.ntiles < sms ? a.ntiles : sms), dim3(kThreads), args,
                                        kFactorSmem, s);
    }
    return e;
}

cudaError_t sp_solve_apply(cudaStream_t s, const sp_solve_item *items, int count)
{
    const int sms = sm_count();
    cudaError_t e = cudaSuccess;
    // a matrix has a CTA per row block; as many matrices as the SMs hold at once
    for (int k0 = 0; k0 < count && e == cudaSuccess;) {
        SolveArgs a;
        a.count = 0;
        int grid = 0, dout = 1;
        while (k0 + a.count < count && a.count < kItems) {
            const sp_solve_item &it = items[k0 + a.count];
            SolveItem &f = a.item[a.count];
            f.L = it.A;
            f.np = sp_solve_pad(it.n);
            f.nb = f.np / NB;
            f.n = it.n;
            f.dout = it.dout;
            f.dinv = (const double *)it.work;
            f.Z = it.Z;
            f.flags = (int *)((double *)it.work + (size_t)f.nb * 4 * 256) + (size_t)f.nb * f.nb;
            f.info = it.info;
            f.cta0 = grid;
            f.ctas = f.nb < sms ? f.nb : sms;
            if (grid + f.ctas > sms)
                break;
            grid += f.ctas;
            dout = it.dout > dout ? it.dout : dout;
            ++a.count;
            e = cudaMemsetAsync(f.flags, 0, 2 * (size_t)f.nb * sizeof(int), s);
            if (e != cudaSuccess)
                return e;
        }
        const void *fn = dout == 1  ? (const void *)k_solve<1>
                         : dout <= 4 ? (const void *)k_solve<4>
                                     : (const void *)k_solve<16>;
        e = set_max_dynamic_smem(fn);
        if (e != cudaSuccess)
            return e;
        void *args[] = {&a};
        e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kThreads), args, kSolveSmem, s);
        k0 += a.count;
    }
    return e;
}
