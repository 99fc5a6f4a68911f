// sp_step_kernel.cuh -- the persistent reservoir step kernel (all neuron and
// synapse models), included by dev_reservoir.cu.
//
// Launch: a cooperative grid of G CTAs (variant 3: one cluster); CTA b owns the
// whole warps [b*nw/G, (b+1)*nw/G) of neurons (nw = ceil(n/32)); a consumer
// thread owns one neuron and keeps its state in registers for the whole launch.
//
// Variant 0: the FLIF_GL history is summed with direct loads from the
//   time-major ring (each lag is one coalesced row segment).
// Variant 1 (FLIF_GL only): one extra producer warp streams the ring rows of
//   the CTA's neuron range into a multi-stage shared-memory pipeline with
//   cp.async.bulk (bulk-copy TMA) on mbarriers; the consumers read lags from
//   shared memory. The producer runs up to one step ahead of the consumers:
//   the rows of step g are the states of steps <= g-2 (lag 1 is the register
//   copy of the previous state), so they only wait for step g-2 to finish.
//   Lags 2..33 are the thread's own last 32 states, kept in a register shift
//   register, so the producer streams lags 34.. only (3 % fewer ring bytes per
//   step at L = 1024) and the sum of a step starts as soon as its lag 1 exists.
//   The grid is sized so that each CTA streams about the same number of ring
//   columns (balanced layout, dev_reservoir.cu). A gather warp watches the
//   spike exchange and copies the words into a double-buffered shared array
//   while the consumers are still summing.
//   A ring larger than the L2 is read with cache hints: the oldest l2_pin
//   lags of a step are loaded with evict-last priority and stay L2-resident
//   from step to step (each row joins them once, when it reaches lag
//   L - l2_pin), the younger lags stream through with evict-first, so the
//   DRAM reads come first in every step and run on through the serial phase.
//
// Variant 2 (FLIF_GL whose CTAs' ring columns fit in shared memory, and
//   FLIF_CAPUTO): FLIF_GL's history is loaded into shared memory once per launch
//   and summed there (chain_pairs); the ring in global memory is still written
//   every step, as the state between launches. (N=2000, L=256: 3.4 us per step;
//   5.9 through the pipeline's stages.) FLIF_CAPUTO's registers stay in global
//   memory, read as 32-byte blocks (caputo_sum), eight in flight. A gather warp
//   as in variant 1.
// Variant 3 (2, 4, 8 or 16 CTAs as one cluster, at most 8192 neurons; SIMPLE and
//   PSC_HETEROGENEOUS): the exchange below between the CTAs' shared memories.
//   (LIF_DISCRETE N=2000: 1.1 us per step; 1.5 through the L2.)
//
// The recurrent rows of a CTA sit in shared memory for the launch where they
// fit, so the row pass after each exchange reads no global memory: rows as
// slots and tails (rowpass_lanes) or, for a dense matrix, column blocks
// (rowpass_cols).
//
// Spike exchange (SIMPLE and PSC_HETEROGENEOUS, whose recurrent input needs
// nothing of another CTA but its spike bits): a warp publishes its word as one
// 8-byte store of (sequence number, word), and a reader polls that entry until
// the number is the step's -- the word comes with its flag, so a step costs one
// store and one successful poll instead of a fence, a flag store, a flag poll,
// a fence and a second load, and no CTA-wide barrier before the store. Entries
// alternate between two buffers: a warp publishes step b + 1 only after it has
// read every word of step b, so nobody can still be reading the buffer of
// step b - 1 that it overwrites. That holds for a reader only if a warp that
// publishes waits for it: a CTA without neurons (more CTAs than warps), and in
// variant 3 a warp without, read no words and skip the steps. (LIF_DISCRETE
// N=20000: 6.7 us per step with flags and fences, 4.1 with the exchange and the
// row slots.) A gather warp starts to poll when its own CTA has published:
// polled all along, the entries' lines slowed the stores and the history stream
// (FLIF_GL N=20000, L=128: 5.9 us per step, 3.6). The other synapses publish a
// double per neuron as well and keep the flags and fences.
//
// Per micro-step, with a split-phase grid barrier:
//   history sum of step g      (overlaps the barrier wait)
//   wait barrier g             (spike words / eff of step g-1 visible)
//   recurrent input            SIMPLE: the weights of the spiking presynaptic
//                              neurons, added by the row's lane in ascending
//                              edge order; others: warp-cooperative walk, one
//                              term per edge, owner lane adds in edge order
//   neuron update, ring write, ballot -> spike word of step g
//   synapse prepare for g+1 (own spike), publish, arrive barrier g+1
#pragma once
#include <cuda.h>
#include "sp_kernels.cuh"
#include "sp_model.h"

namespace sp {

struct KP {
    int n, nwords, din, micro, G, n_macro, phase0;
    int rs;         // ring row stride in doubles (multiple of 32)
    int warps;      // consumer warps per CTA
    int R, NST;     // variant 1: ring rows per stage, stages
    int BW, NBX;    // variant 1: box width (neurons) and boxes side by side per stage
    int bal;        // balanced layout: CTA b's active positions are the first
                    // n / G (+1 for b < n % G) of its range, the rest holes
    int RB;         // variant 1: rows per box = min(R, L)
    int coef_smem;  // variant 1: coefficient table staged in shared memory
    // SIMPLE synapse, rows in shared memory for the launch (rowpass_lanes): most
    // slot groups and tail edges of a CTA; ell_cap 0 = the CSR rows are walked in
    // global memory
    int ell_cap, tail_cap;
    const int *ell_off;      // [nwords + 1] first slot group of each warp
    const uint2 *ell_col;    // [groups][32] four 16-bit column positions
    const double *ell_w;     // [groups][4][32]
    const int *tail_rp;      // [nwords][33] tails of a warp's rows, in tail_col / tail_w
    const int *tail_col;
    const double *tail_w;
    // SIMPLE synapse, column blocks of a dense matrix (see rowpass_cols): 0 = not
    // used by this launch, 1 = read from global memory, 2 = staged in shared
    // memory (col_cap: most weights of a CTA)
    int col_mode, col_cap;
    const int *col_off;      // [nwords + 1] first weight of each row word
    const uint2 *col_blk;    // [nwords][n] {row bits, weight offset from col_off}
    const double *col_w;
    int u_ring;     // input rows prefetched through shared memory, kURows deep per warp
    int win_smem;   // input weights staged in shared memory, [din][consumer thread]
    const int *nid_of;  // neuron at each position, -1 for an empty lane
    long long step0, syn_step0;
    double a, b, c, d, e, f, g, h, ci, cj, ck, cl, dt;
    int L, det_refr, diff_sto;
    const double *coef;
    double *V, *tprev, *ring;
    int *cap_pos;
    long long *refr_until;
    unsigned long long *rng;
    unsigned *spk;
    const long long *row_ptr;
    const int *col;
    const double *w;
    double *eff;
    double psc_decay, psc_omd;
    double *trace;
    const double *edge_decay, *edge_omd;
    double *edge_trace;
    int Ls;
    const double *scoef;
    double s_dta, s_tau;
    double *Iring;
    int Nc;
    const double *mx_decay, *mx_omd, *mx_c;
    double *mx_tr;
    const double *W_in;
    double gamma;
    const double *u;
    double *phi;
    unsigned *raster;
    unsigned long long *bar;  // grid-barrier arrival counter (64-bit: never wraps)
    // arrival flags, one per CTA on its own 128-byte line: CTA c stores b + 1
    // once its spike words and drive of micro-step b - 1 are published
    unsigned long long *flags;
    // spike exchange: [2][nwords] entries (sequence number << 32 | spike word);
    // the words of barrier b carry the number ll_base + b
    unsigned long long *ll;
    unsigned ll_base;
    int *err;                 // [0] error code, [1] / [2] low / high word of the micro-step
    unsigned long long tmo;   // limit of every wait, ns
    // one-shot test hook: CTA hold_cta does not arrive at the barrier that
    // opens micro-step hold_b (-1: none), so every wait on it runs out
    int hold_cta;
    long long hold_b;
    // variant 1: the oldest l2_pin lags of every step are read with L2
    // evict-last priority, younger ones and the ring writes with evict-first
    // (0: no hints)
    int l2_pin;
    // variant 1: 2-D tiled map of the ring [L rows][rs columns] of doubles,
    // box = BW columns x R rows
    alignas(64) CUtensorMap tmap;
    // variant 1, FRACTIONAL: the synapse's history passes through the same stages,
    // its coefficients staged in shared memory
    alignas(64) CUtensorMap tmap_s;
    int frac_stage;
};

// ------------------------------------------------------------ PTX helpers
__device__ __forceinline__ unsigned smem_u32(const void *p)
{
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void named_sync(int n)
{
    asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory");
}
__device__ __forceinline__ void mbar_init(unsigned long long *b, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count)
                 : "memory");
}
__device__ __forceinline__ bool mbar_test(unsigned long long *b, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n .reg .pred P;\n mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n"
        " selp.u32 %0, 1, 0, P;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *b)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *b, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)),
                 "r"(bytes)
                 : "memory");
}
// read-only load that does not allocate in L1 (per-step input weights must not
// evict the coefficient table and the CSR slice)
__device__ __forceinline__ double ldg_na(const double *ptr)
{
    double v;
    asm volatile("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(ptr));
    return v;
}

// 2-D tiled bulk-tensor load of one box at (x = column, y = row); no multicast.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y,
                                            unsigned long long *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}
// L2 eviction-priority policies for the cache-hinted ring loads and stores:
// evict-last for the slots kept resident, evict-first for the streamed ones
__device__ __forceinline__ unsigned long long l2_policy(bool keep)
{
    unsigned long long pol;
    if (keep)
        asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    else
        asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ void tma_load_2d_hint(void *dst, const CUtensorMap *map, int x, int y,
                                                 unsigned long long *bar, unsigned long long pol)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        ".L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(smem_u32(bar)),
        "l"(pol)
        : "memory");
}
__device__ __forceinline__ void st_hint_f64(double *ptr, double v, unsigned long long pol)
{
    asm volatile("st.global.L2::cache_hint.f64 [%0], %1, %2;" ::"l"(ptr), "d"(v), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void st_release_cta(volatile int *ptr, int v)
{
    asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(smem_u32((const void *)ptr)),
                 "r"(v)
                 : "memory");
}
__device__ __forceinline__ void red_release_cta(volatile int *ptr, int v)
{
    asm volatile("red.release.cta.shared::cta.add.s32 [%0], %1;" ::"r"(smem_u32((const void *)ptr)),
                 "r"(v)
                 : "memory");
}
__device__ __forceinline__ int ld_acquire_cta(volatile int *ptr)
{
    int v;
    asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];"
                 : "=r"(v)
                 : "r"(smem_u32((const void *)ptr))
                 : "memory");
    return v;
}
__device__ __forceinline__ void fence_proxy_async()
{
    asm volatile("fence.proxy.async;" ::: "memory");
}

// Bounded mbarrier wait; false on timeout or when the launch is aborting.
__device__ __forceinline__ void record_err(int *err, int code, long long step)
{
    if (atomicCAS(err, kErrNone, code) == kErrNone) {
        err[1] = (int)(unsigned)(unsigned long long)step;
        err[2] = (int)(unsigned)((unsigned long long)step >> 32);
    }
}

__device__ __forceinline__ bool mbar_wait(unsigned long long *b, unsigned parity,
                                          volatile int *s_abort, int *err,
                                          unsigned long long tmo, long long step)
{
    if (mbar_test(b, parity))
        return true;
    unsigned long long t0 = globaltimer_ns();
    unsigned polls = 0;
    while (!mbar_test(b, parity)) {
        if ((++polls & 63u) == 0) {
            if (*s_abort || ld_volatile_i32(err) != kErrNone)
                return false;
            if (globaltimer_ns() - t0 > tmo) {
                record_err(err, kErrBarrierTimeout, step);
                *s_abort = 1;
                return false;
            }
        }
    }
    return true;
}

// One chunk of 32 consecutive edges, lane l holding the weight of edge l and m
// the ballot of the spiking ones: every lane adds those of its own row, edges
// [from, to) of the chunk, in ascending order. A pass serves one edge of every
// row at once, so a chunk takes as many passes as its busiest row has spiking
// edges. (One edge a pass, found by its owner with a second ballot, took about
// 80 cycles per spiking edge.)
template <typename I>
__device__ __forceinline__ double add_chunk(double acc, double wv, unsigned m, I from, I to)
{
    if (m == 0)
        return acc;
    const int a = from <= 0 ? 0 : (from < 32 ? (int)from : 32);
    const int b = to <= 0 ? 0 : (to < 32 ? (int)to : 32);
    unsigned mine = 0;
    if (b > a)
        mine = m & (0xffffffffu >> (32 - b)) & (0xffffffffu << a);
    while (__any_sync(kFull, mine != 0)) {
        const int j = __ffs(mine) - 1;
        const double w = __shfl_sync(kFull, wv, j & 31);
        if (mine)
            acc = add(acc, w);
        mine &= mine - 1;
    }
    return acc;
}

// SIMPLE synapse, one warp: recurrent input of rows [row0, row0 + nv) for the
// lane that owns row row0 + lane. Edges are scanned 32 at a time; spiking
// presynaptic columns are found by a ballot over the spike bits and each
// weight is added by the owner lane of its row in ascending edge order, i.e.
// exactly the non-zero terms of csr_row_dot (src/sparse.c:68-76) in order.
__device__ __forceinline__ double rowpass_simple_warp(const long long *__restrict__ row_ptr,
                                                      const int *__restrict__ col,
                                                      const double *__restrict__ w,
                                                      const unsigned *s_spk, int row0, int nv,
                                                      int lane)
{
    const long long e0 = __ldg(row_ptr + row0);
    const long long e1 = __ldg(row_ptr + row0 + nv);
    const long long my_start = (lane < nv) ? __ldg(row_ptr + row0 + lane) : e1;
    const long long my_end = (lane < nv) ? __ldg(row_ptr + row0 + lane + 1) : e1;
    double acc = 0.0;
    // next chunk's column index and weight are loaded one chunk ahead
    int cn = -1;
    double wn = 0.0;
    if (e0 + lane < e1) {
        cn = __ldg(col + e0 + lane);
        wn = __ldg(w + e0 + lane);
    }
    for (long long base = e0; base < e1; base += 32) {
        const int c = cn;
        const double wv = wn;
        const long long nx = base + 32 + lane;
        cn = -1;
        if (nx < e1) {
            cn = __ldg(col + nx);
            wn = __ldg(w + nx);
        }
        const bool s = c >= 0 && ((s_spk[c >> 5] >> (c & 31)) & 1u);
        acc = add_chunk(acc, wv, __ballot_sync(kFull, s), my_start - base, my_end - base);
    }
    return acc;
}

// Per-phase timing of the last kSpStampSteps micro-steps of a launch
// (compiled in only with -DSP_PHASE_STAMPS): thread 0 of each CTA records the
// global timer at the phase boundaries of every step into g_sp_stamps
// [cta][step][phase]; spires_dbg_phase_stamps (dev_reservoir.cu) copies them
// out. Phases: 0 step start, 1 history summed, 2 barrier passed, 3 spike
// words staged, 4 row pass done (warp 0), 5 update and spike word done,
// 6 arrival made; 7 the producer issued the step's first stage.
#ifdef SP_PHASE_STAMPS
constexpr int kSpStampCtas = 160, kSpStampSteps = 32, kSpStampPhases = 8;
__device__ unsigned long long g_sp_stamps[kSpStampCtas * kSpStampSteps * kSpStampPhases];
#define SP_STAMP(cond, b, B, ph)                                                             \
    do {                                                                                    \
        if ((cond) && blockIdx.x < kSpStampCtas && (b) >= (B)-kSpStampSteps)                \
            g_sp_stamps[((size_t)blockIdx.x * kSpStampSteps + ((b) - ((B)-kSpStampSteps))) * \
                            kSpStampPhases +                                                \
                        (ph)] = globaltimer_ns();                                           \
    } while (0)
#else
#define SP_STAMP(cond, b, B, ph) \
    do {                         \
    } while (0)
#endif

// Synapses whose drive is not a spike bit (PSC and fractional: every edge
// carries a term), one warp: rows [row0, row0 + 32), lane r owns row row0 + r.
// The warp's contiguous edge range is taken 32 edges at a time, each lane
// forming one edge's term in parallel -- w_k * eff[col_k], or for
// PSC_HETEROGENEOUS the updated edge trace times w_k -- and the owner lane
// of each edge's row adds the terms in ascending edge order, the order of the
// reference's per-row loop (src/synapses/psc_heterogeneous.c:124-139,
// src/synapse.c:90-105), so the sums are the same bits as a per-row walk.
template <int ST>
__device__ __forceinline__ double rowpass_terms_warp(const KP &p, const double *ef,
                                                     const unsigned *s_spk, int row0, int lane)
{
    const long long e0 = __ldg(p.row_ptr + row0), e1 = __ldg(p.row_ptr + row0 + 32);
    const long long my_start = __ldg(p.row_ptr + row0 + lane);
    const long long my_end = __ldg(p.row_ptr + row0 + lane + 1);
    auto term_of = [&](long long k) -> double {
        if (k >= e1)
            return 0.0;
        const int c = __ldg(p.col + k);
        if (ST == SP_SYN_PSC_HET) {
            const double sv = ((s_spk[c >> 5] >> (c & 31)) & 1u) ? 1.0 : 0.0;
            const double tr = add(mul(p.edge_trace[k], __ldg(p.edge_decay + k)),
                                  mul(__ldg(p.edge_omd + k), sv));
            p.edge_trace[k] = tr;
            return mul(__ldg(p.w + k), tr);
        }
        return mul(__ldg(p.w + k), __ldcg(ef + c));
    };
    double acc = 0.0;
    // 4 chunks of 32 edges at a time: their loads in flight together, then
    // each chunk's terms added by the owner lanes in ascending edge order
    for (long long base = e0; base < e1; base += 4 * 32) {
        double t[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            t[u] = term_of(base + 32 * u + lane);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long cb = base + 32 * u;
            if (cb >= e1)
                break;
            const int cnt = e1 - cb < 32 ? (int)(e1 - cb) : 32;
            // the chunk's edges of the lane's row: from, from + 1, .. (32-bit, so that
            // an edge costs one comparison: with two of 64 bits 50 edges a row of
            // PSC_HOMOGENEOUS took 46 to 49 us a step, now 42)
            const int from = (int)min(max(my_start - cb, 0ll), 32ll);
            const unsigned len = (unsigned)((int)min(max(my_end - cb, 0ll), 32ll) - from);
#pragma unroll 8
            for (int j = 0; j < cnt; ++j) {
                const double v = __shfl_sync(kFull, t[u], j);
                if ((unsigned)(j - from) < len)
                    acc = add(acc, v);
            }
        }
    }
    return acc;
}

// SIMPLE synapse, rows in shared memory, one warp, lane r the row of position r.
// The first slots of every row are stored side by side, four to a group, and
// lane r walks its own in ascending order; a row shorter than the warp's slots
// is padded with zero weights, and a slot whose neuron did not spike adds +0.0
// (which leaves the sum's bits: it starts at +0 and never becomes -0). What a
// row has beyond the slots -- the hubs of a Barabasi-Albert graph -- follows as
// a tail that the whole warp tests 32 edges at a time, the row's lane adding
// the spiking ones in order. A warp issues in order and every addition waits
// for the one before it, so the tests of one block of eight slots are written
// between the additions of the other. (About 360 cycles for up to 8 slots and
// 27 for each more; the edge-parallel walk below takes 300 per 32 edges and 100
// for each pass that adds one edge of every row.)
__device__ __forceinline__ double rowpass_lanes(const uint2 *col, const double *w, int groups,
                                                const int *tail_rp, const int *tail_col,
                                                const double *tail_w, unsigned tails,
                                                const unsigned *s_spk, int lane)
{
    double acc = 0.0;
    const uint2 *cp = col + lane;
    const double *wp = w + lane;
    const int last = groups - 1;
    uint2 c[2];
    auto cols = [&](int q) {
#pragma unroll
        for (int e = 0; e < 2; ++e)
            c[e] = cp[(q + e < last ? q + e : last) * 32];
    };
    auto block = [&](int q, double (&v)[8]) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const double *wq = wp + (q + e < last ? q + e : last) * 128;
            const unsigned k[4] = {c[e].x & 0xffffu, c[e].x >> 16, c[e].y & 0xffffu,
                                   c[e].y >> 16};
            const unsigned live = q + e <= last ? 1u : 0u;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const double x = wq[32 * u];
                v[4 * e + u] = ((s_spk[k[u] >> 5] >> (k[u] & 31)) & live) ? x : 0.0;
            }
        }
    };
    auto sum = [&](const double (&v)[8]) {
#pragma unroll
        for (int u = 0; u < 8; ++u)
            acc = add(acc, v[u]);
    };
    if (groups > 0) {
        double va[8], vb[8];
        cols(0);
        block(0, va);
        cols(2);
        for (int q = 0; q < groups; q += 4) {
            if (q + 2 >= groups) {
                sum(va);
                break;
            }
            block(q + 2, vb);
            cols(q + 4);
            sum(va);
            block(q + 4, va);
            cols(q + 6);
            sum(vb);
        }
    }
    for (; tails; tails &= tails - 1) {
        const int row = __ffs(tails) - 1;
        const int e1 = tail_rp[row + 1];
        int base = tail_rp[row];
        auto test = [&](int at) {  // ballot of the spiking edges at .. at + 31
            const int e = at + lane < e1 ? at + lane : e1 - 1;
            const unsigned k = (unsigned)tail_col[e];
            const unsigned hit = (s_spk[k >> 5] >> (k & 31)) & (at + lane < e1 ? 1u : 0u);
            return __ballot_sync(kFull, hit != 0);
        };
        unsigned m = test(base);
        for (; base < e1; base += 32) {
            const unsigned nm = base + 32 < e1 ? test(base + 32) : 0u;
            // every lane reads the spiking edges' weights, the row's lane keeps the sum
            while (m) {
                double x[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    x[u] = m ? tail_w[base + __ffs(m) - 1] : 0.0;
                    m &= m - 1;
                }
                if (lane == row) {
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        acc = add(acc, x[u]);
                }
            }
            m = nm;
        }
    }
    return acc;
}

// SIMPLE synapse, column blocks, one warp: for row word q (rows 32q .. 32q + 31)
// and neuron j, the bits of the rows with an edge from j and where the block's
// weights, stored in row order, start. The lane of a row walks the list of
// spiking neurons in ascending order and adds w_ij where its bit is set: the
// non-zero terms of csr_row_dot (src/sparse.c:68-76) in order, at a cost that
// follows the spikes of the step and not the edges of the row. C columns are in
// flight, the next C's blocks a pass ahead: four where other warps fill the gaps,
// eight for a warp that runs alone.
template <bool kShared, int C = 4>
__device__ __forceinline__ double rowpass_cols(const uint2 *blk, const double *w,
                                               const unsigned short *s_list, int cnt, int lane)
{
    const unsigned below = (1u << lane) - 1u;
    auto fetch = [&](int t, uint2 (&c)[C]) {  // the list is padded to a multiple of C
        unsigned j[C];
#pragma unroll
        for (int u = 0; u < C; u += 4) {
            const uint2 id = *(const uint2 *)(s_list + t + u);
            j[u] = id.x & 0xffffu;
            j[u + 1] = id.x >> 16;
            j[u + 2] = id.y & 0xffffu;
            j[u + 3] = id.y >> 16;
        }
#pragma unroll
        for (int u = 0; u < C; ++u)
            c[u] = t + u >= cnt ? make_uint2(0u, 0u) : (kShared ? blk[j[u]] : __ldg(blk + j[u]));
    };
    double acc = 0.0;
    uint2 cur[C], nxt[C];
    fetch(0, cur);
    for (int t = 0; t < cnt; t += C) {
        double x[C];
#pragma unroll
        for (int u = 0; u < C; ++u) {
            const double *a = w + cur[u].y + __popc(cur[u].x & below);
            x[u] = 0.0;
            if ((cur[u].x >> lane) & 1u)
                x[u] = kShared ? *a : __ldg(a);
        }
        if (t + C < cnt)
            fetch(t + C, nxt);
#pragma unroll
        for (int u = 0; u < C; ++u) {
            acc = add(acc, x[u]);  // +0.0 where the row has no such edge
            cur[u] = nxt[u];
        }
    }
    return acc;
}

// History in shared memory: ring rows in pairs, [pair][32 lanes][2], so that one
// 16-byte load brings two lags, and two copies of the coefficients, the second
// shifted by one, so that a pair of them is a 16-byte load at either parity.
// hist + the n lags k, k + 1, ... in ascending order, lag k in row r, rows
// descending (no wrap). (A shared-memory load costs its destination registers'
// write-back, 4.8 cycles a warp for 8 bytes a lane even when all lanes read one
// word: 16.8 cycles per lag with 8-byte loads, 10.5 with pairs, against 8.5 for
// the dependent addition alone.)
__device__ __forceinline__ double chain_pairs(double hist, const double *ca, const double *cb,
                                              const double2 *ring, int k, int r, int n)
{
    if (n > 0 && !(r & 1)) {
        hist = add(hist, mul(ca[k], ring[(r >> 1) * 32].x));
        ++k;
        --r;
        --n;
    }
    const double2 *c = (const double2 *)((k & 1) ? cb + (k - 1) : ca + k);
    const double2 *v = ring + (r >> 1) * 32;
    for (; n >= 16; n -= 16, c += 8, v -= 256) {
        double x[16];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const double2 cc = c[u], vv = v[-32 * u];
            x[2 * u] = mul(cc.x, vv.y);
            x[2 * u + 1] = mul(cc.y, vv.x);
        }
#pragma unroll
        for (int u = 0; u < 16; ++u)
            hist = add(hist, x[u]);
    }
    for (; n >= 2; n -= 2, ++c, v -= 32) {
        const double2 cc = *c, vv = *v;
        hist = add(hist, mul(cc.x, vv.y));
        hist = add(hist, mul(cc.y, vv.x));
    }
    if (n > 0)
        hist = add(hist, mul(c->x, v->y));
    return hist;
}

// hist + sum of cnt products coef[j] * v[-j * stride] in ascending j, U loads
// at a time, the next U products formed while the chain of dependent additions
// runs over the current ones. ld(p) reads one value.
template <int U, typename Ld>
__device__ __forceinline__ double chain_sum(double hist, const double *coef, const double *v,
                                            size_t stride, int cnt, Ld ld)
{
    double cur[U];
    int j = 0;
    if (cnt >= U) {
#pragma unroll
        for (int u = 0; u < U; ++u)
            cur[u] = mul(coef[u], ld(v - (size_t)u * stride));
        for (; j + 2 * U <= cnt; j += U) {
            double nxt[U];
            const double *cn = coef + j + U;
            const double *vn = v - (size_t)(j + U) * stride;
#pragma unroll
            for (int u = 0; u < U; ++u)
                nxt[u] = mul(cn[u], ld(vn - (size_t)u * stride));
#pragma unroll
            for (int u = 0; u < U; ++u)
                hist = add(hist, cur[u]);
#pragma unroll
            for (int u = 0; u < U; ++u)
                cur[u] = nxt[u];
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            hist = add(hist, cur[u]);
        j += U;
    }
    for (; j < cnt; ++j)
        hist = add(hist, mul(coef[j], ld(v - (size_t)j * stride)));
    return hist;
}

// History over a time-major ring column: lags k0..lim in ascending order, lag
// k0 in row r0, rows descending and wrapping at row 0 to row L - 1.
template <int U, typename Ld>
__device__ __forceinline__ double ring_sum(double hist, const double *coef, const double *column,
                                           size_t stride, int L, int r0, int k0, int lim, Ld ld)
{
    const int cnt = lim - k0 + 1;
    if (cnt <= 0)
        return hist;
    const int n1 = cnt < r0 + 1 ? cnt : r0 + 1;
    hist = chain_sum<U>(hist, coef + k0, column + (size_t)r0 * stride, stride, n1, ld);
    if (cnt > n1)
        hist = chain_sum<U>(hist, coef + k0 + n1, column + (size_t)(L - 1) * stride, stride,
                            cnt - n1, ld);
    return hist;
}

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(smem)), "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A CTA's copy of n 8-byte words into shared memory, asynchronous, in 16-byte
// pieces where both sides are aligned; commit and wait by the caller. The start of
// a launch is these copies (67 KB of column blocks per CTA for LIF_DISCRETE N=1000,
// conn 0.1): loaded and stored, a few at a time by the CTA's few threads, they
// took most of a one-step launch (33.6 us; now 13.0, N=4000 conn 0.05 83 -> 15).
__device__ __forceinline__ void stage_words(void *dst, const void *src, int n)
{
    const bool wide = ((smem_u32(dst) | (unsigned)(uintptr_t)src) & 15u) == 0;
    int k = threadIdx.x;
    if (wide) {
        for (; k < n / 2; k += blockDim.x)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             smem_u32((char *)dst + 16 * (size_t)k)),
                         "l"((const char *)src + 16 * (size_t)k)
                         : "memory");
        k = (n & ~1) + threadIdx.x;
    }
    for (; k < n; k += blockDim.x)
        cp_async8((char *)dst + 8 * (size_t)k, (const char *)src + 8 * (size_t)k);
}

// Four consecutive doubles from a 32-byte boundary in one load.
__device__ __forceinline__ void ld_f64x4(const double *p, double (&v)[4])
{
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
                 : "l"(p));
}

// FLIF_CAPUTO memory sum of one neuron: tab[0] * newest + sum over lags
// k = 1 .. D-1, ascending, of tab[k] * row[(pos - k) mod D]; tab is readable
// three places beyond either end. Every neuron's shift register is contiguous
// with a head of its own, so the 32 lanes of a load touch 32 lines and the load
// unit's line a cycle bounds the sum (N=20000, D=510, 5 warps an SM: 150 cycles
// per lag with an 8-byte load each). Lanes therefore walk aligned 32-byte
// blocks downwards, four lags a load, Q blocks in flight while Q are summed.
// A block's elements e carry lag c0 - e; those outside the lane's run -- the
// entries before the head, then from the row's top to behind it -- add +0.0,
// which leaves the sum's bits (it starts from +0 and never becomes -0).
template <int Q>
__device__ __forceinline__ double caputo_sum(double newest, const double *tab, const double *ring,
                                             long long row, int D, int pos)
{
    double mem = add(0.0, mul(tab[0], newest));
    // the loads below stay between the stores of the steps around (ld_f64x4 does not
    // say that it reads memory, so that the sums' other loads may move past it)
    asm volatile("" ::: "memory");
    // element numbers below count from the 32-byte boundary at or under the row
    const int r0 = (int)(row & 3);
    const double *base = ring + (row - r0);
    const int top = r0 + D - 1, stop = r0 + pos + 1;  // the second run: top down to stop
    int blocks = pos > 0 ? ((r0 + pos - 1) >> 2) + 1 : 0;
    if (stop <= top)
        blocks += (top >> 2) - (stop >> 2) + 1;
    // the block to load next and the block to sum next, with their runs' ends
    int lat = pos > 0 ? (r0 + pos - 1) & ~3 : top & ~3, llo = pos > 0 ? r0 : stop;
    int at = lat, lo = llo, hi = pos > 0 ? r0 + pos - 1 : top;
    int c0 = r0 + pos + (pos > 0 ? 0 : D);
    auto load = [&](double (&v)[4]) {
        ld_f64x4(base + (lat > 0 ? lat : 0), v);
        lat -= 4;
        if (lat + 3 < llo && llo == r0) {  // the first run is loaded: on from the top
            lat = top & ~3;
            llo = stop;
        }
    };
    auto sum = [&](const double (&v)[4]) {
        const int k3 = c0 - at - 3;  // lag of the block's last element, the first to add
        const double *t = tab + (k3 < -3 ? -3 : (k3 > D - 1 ? D - 1 : k3));
        double x[4];
#pragma unroll
        for (int u = 3; u >= 0; --u) {
            const double y = mul(t[3 - u], v[u]);
            x[u] = (at + u >= lo && at + u <= hi) ? y : 0.0;
        }
#pragma unroll
        for (int u = 3; u >= 0; --u)
            mem = add(mem, x[u]);
        at -= 4;
        if (at + 3 < lo && lo == r0) {
            at = top & ~3;
            lo = stop;
            hi = top;
            c0 += D;
        }
    };
    double cur[Q][4], nxt[Q][4];
#pragma unroll
    for (int q = 0; q < Q; ++q)
        load(cur[q]);
    for (int n = 0; n < blocks; n += 2 * Q) {
#pragma unroll
        for (int q = 0; q < Q; ++q)
            load(nxt[q]);
#pragma unroll
        for (int q = 0; q < Q; ++q)
            sum(cur[q]);
        if (n + Q >= blocks)
            break;
#pragma unroll
        for (int q = 0; q < Q; ++q)
            load(cur[q]);
#pragma unroll
        for (int q = 0; q < Q; ++q)
            sum(nxt[q]);
    }
    asm volatile("" ::: "memory");
    return mem;
}

// Spike exchange between the CTAs of one cluster: the entry is written straight
// into every CTA's shared memory and polled there (VAR 3).
__device__ __forceinline__ void st_cluster_u64(const void *local, unsigned rank,
                                               unsigned long long v)
{
    unsigned remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(remote)
                 : "r"(smem_u32(local)), "r"(rank));
    asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" ::"r"(remote), "l"(v)
                 : "memory");
}
__device__ __forceinline__ unsigned long long ld_cluster_u64(const unsigned long long *local)
{
    unsigned long long v;
    asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];"
                 : "=l"(v)
                 : "r"(smem_u32(local))
                 : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;"
                 ::: "memory");
}

template <int R, typename Coef>
__device__ __forceinline__ double stage_sum(double hist, Coef coef, int k, const double *buf,
                                            int bw)
{
    double c[R], v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) {
        c[j] = coef(k + j);
        v[j] = buf[(size_t)(R - 1 - j) * bw];
    }
#pragma unroll
    for (int j = 0; j < R; ++j)
        hist = add(hist, mul(c[j], v[j]));
    return hist;
}

// Variant 1 runs at most kPipeWarps consumer warps + 1 producer warp per CTA,
// which leaves registers for a stage of lags in flight and the register lags
// per thread.
constexpr int kPipeWarps = 8;
// Variant 3: at most 16 CTAs of 16 warps, 8192 neurons.
constexpr int kClusterWarps = 16, kClusterWords = 256;

template <int VAR>
struct Bounds {
    // variant 2: consumers and the gather warp; variant 3: consumers
    static constexpr int threads = VAR == 1   ? 32 * (kPipeWarps + 2)
                                   : VAR == 2 ? 32 * (kPipeWarps + 1)
                                   : VAR == 3 ? 32 * kClusterWarps
                                              : 1024;
};

// Variant 1 keeps lags 2..kRegLags+1 of its own neuron in registers: they are
// the thread's own last states, so they are neither written to nor read back
// from the ring for the sum, and the producer streams lags kRegLags+2.. only.
constexpr int kRegLags = 32;
constexpr int kURows = 8;  // input rows in flight per warp
constexpr int kFlagStride = 16;  // u64 per CTA arrival flag (one 128-byte line)

template <int NT, int ST, int VAR>
__global__ void __launch_bounds__(Bounds<VAR>::threads, 1) k_run(const __grid_constant__ KP p)
{
    constexpr int RL = (VAR == 1 && NT == SP_FLIF_GL) ? kRegLags : 0;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_flag;
    __shared__ volatile int s_abort;
    __shared__ volatile int s_done;
    __shared__ volatile int s_gather;  // variant 1: barriers whose words are staged
    __shared__ int s_wsum[32];         // column blocks: spikes per warp of the list scan
    __shared__ volatile int s_bad[2];  // variant 0: a wait of barrier b (b & 1) ran out
    // the spike exchange carries everything another CTA needs
    constexpr bool kWords = ST == SP_SYN_SIMPLE || ST == SP_SYN_PSC_HET;

    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int NC = 32 * p.warps;  // consumer threads
    const int wb0 = (int)(((long long)blockIdx.x * p.nwords) / p.G);
    const int wb1 = (int)(((long long)(blockIdx.x + 1) * p.nwords) / p.G);
    const int L = p.L;
    const long long B = (long long)p.n_macro * p.micro;

    // spike words of the barrier, two buffers: barrier b + 1's are filled while
    // a row pass may still read barrier b's
    const size_t spk_one = (((size_t)p.nwords * 4) + 127) & ~(size_t)127;
    unsigned *s_spkb = (unsigned *)smem;
    const size_t spk_bytes0 = 2 * spk_one;
    // rows of the CTA (SIMPLE synapse): slot weights and columns, then the tails
    double *s_ell_w = (double *)(smem + spk_bytes0);
    uint2 *s_ell_col = (uint2 *)(s_ell_w + (size_t)128 * p.ell_cap);
    double *s_tail_w = (double *)(s_ell_col + (size_t)32 * p.ell_cap);
    int *s_tail_col = (int *)(s_tail_w + p.tail_cap);
    int *s_tail_rp = s_tail_col + p.tail_cap;
    const size_t csr_bytes =
        p.ell_cap > 0 ? (size_t)1280 * p.ell_cap +
                            ((size_t)12 * p.tail_cap + (size_t)132 * p.warps + 127) / 128 * 128
                      : 0;
    // column blocks: spiking neurons as a bitmap in neuron order and as a list,
    // then (staged) the CTA's weights and blocks; the input weights
    const int nwn = (p.n + 31) / 32;
    unsigned *s_bits = (unsigned *)(smem + spk_bytes0 + csr_bytes);
    unsigned short *s_list = (unsigned short *)(s_bits + (nwn + 3) / 4 * 4);
    const size_t list_bytes =
        p.col_mode ? ((size_t)(nwn + 3) / 4 * 16 + (size_t)p.n * 2 + 8 + 127) / 128 * 128 : 0;
    double *s_col_w = (double *)((char *)s_bits + list_bytes);
    uint2 *s_col_blk = (uint2 *)(s_col_w + p.col_cap);
    const size_t col_bytes =
        list_bytes +
        (p.col_mode == 2 ? ((size_t)p.col_cap * 8 + (size_t)p.warps * p.n * 8 + 127) / 128 * 128 : 0);
    double *s_win = (double *)((char *)s_bits + col_bytes);
    const size_t win_bytes = p.win_smem ? (size_t)p.din * NC * 8 : 0;
    double *s_u = (double *)((char *)s_win + win_bytes);
    const size_t u_bytes = p.u_ring ? ((size_t)p.warps * kURows * p.din * 8 + 127) / 128 * 128 : 0;
    // variant 3: the exchange entries [2][nwords]
    unsigned long long *s_ll = (unsigned long long *)((char *)s_u + u_bytes);
    const size_t ll_bytes = VAR == 3 ? ((size_t)16 * p.nwords + 127) / 128 * 128 : 0;
    const size_t spk_bytes =
        spk_bytes0 + csr_bytes + col_bytes + win_bytes + u_bytes + ll_bytes;
    // kernels with the history in shared memory: a second copy, shifted by one
    constexpr bool kPairs = VAR >= 2 && NT == SP_FLIF_GL;
    const size_t coef_one = (((size_t)L * 8 + 64) + 127) & ~(size_t)127;
    const size_t coef_bytes = p.coef_smem ? (kPairs ? 2 : 1) * coef_one : 0;
    // (FLIF_CAPUTO: four places of padding before and after the table)
    double *s_coef = (double *)(smem + spk_bytes) + (NT == SP_FLIF_CAPUTO ? 4 : 0);
    double *s_coef1 = (double *)(smem + spk_bytes + coef_one);
    double *s_scoef = (double *)(smem + spk_bytes + coef_bytes);
    const size_t scoef_bytes =
        ST == SP_SYN_FRAC && p.frac_stage ? ((size_t)p.Ls * 8 + 127) / 128 * 128 : 0;
    double *s_stage = (double *)(smem + spk_bytes + coef_bytes + scoef_bytes);
    // variants 2 and 3: the thread's column of its warp's ring block (chain_pairs)
    double2 *s_ring = (double2 *)s_stage + (size_t)warp * ((L + 1) / 2) * 32 + lane;
    auto ring_at = [&](int r) -> double & { return *((double *)(s_ring + (r >> 1) * 32) + (r & 1)); };
    const size_t STAGE = (size_t)p.NBX * p.R * p.BW;  // doubles per stage
    unsigned long long *full = (unsigned long long *)(smem + spk_bytes + coef_bytes + scoef_bytes +
                                                      (size_t)p.NST * STAGE * sizeof(double));
    unsigned long long *empty = full + p.NST;
    const int lo = wb0 * 32;
    const int S_b = 32 * (wb1 - wb0);

    if (tid == 0) {
        s_abort = 0;
        s_done = 0;
        s_gather = 0;
        s_bad[0] = s_bad[1] = 0;
    }
    if (p.coef_smem && NT == SP_FLIF_CAPUTO && tid < 8)
        s_coef[tid < 4 ? tid - 4 : L + tid - 4] = 0.0;
    if (p.coef_smem) {
        stage_words(s_coef, p.coef + (NT == SP_FLIF_CAPUTO ? 4 : 0), L);
        if (kPairs && L > 1)
            stage_words(s_coef1, p.coef + 1, L - 1);
    }
    if (scoef_bytes > 0)
        stage_words(s_scoef, p.scoef, p.Ls);
    if (ST == SP_SYN_SIMPLE && p.ell_cap > 0) {
        const int g0 = __ldg(p.ell_off + wb0), ng = __ldg(p.ell_off + wb1) - g0;  // <= ell_cap
        stage_words(s_ell_col, p.ell_col + (size_t)32 * g0, 32 * ng);
        stage_words(s_ell_w, p.ell_w + (size_t)128 * g0, 128 * ng);
        if (wb1 > wb0) {
            const int t0 = __ldg(p.tail_rp + (size_t)33 * wb0);
            const int nt = __ldg(p.tail_rp + (size_t)33 * wb1 - 1) - t0;  // <= tail_cap
            stage_words(s_tail_w, p.tail_w + t0, nt);
            for (int k = tid; k < nt; k += blockDim.x)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                                 smem_u32(s_tail_col + k)),
                             "l"(p.tail_col + t0 + k)
                             : "memory");
            for (int k = tid; k < 33 * (wb1 - wb0); k += blockDim.x)
                s_tail_rp[k] = __ldg(p.tail_rp + (size_t)33 * wb0 + k) - t0;
        }
    }
    if (ST == SP_SYN_SIMPLE && p.col_mode) {
        for (int k = tid; k < nwn; k += blockDim.x)
            s_bits[k] = 0u;
        if (p.col_mode == 2) {
            const int w0 = __ldg(p.col_off + wb0), nwt = __ldg(p.col_off + wb1) - w0;  // <= col_cap
            stage_words(s_col_w, p.col_w + w0, nwt);
            stage_words(s_col_blk, p.col_blk + (size_t)wb0 * p.n, (wb1 - wb0) * p.n);
        }
    }
    if (p.win_smem)
        for (int k = tid; k < p.din * S_b; k += blockDim.x) {
            const int q = k / p.din, j = k - q * p.din;
            cp_async8(s_win + (size_t)j * NC + q, p.W_in + (size_t)(lo + q) * p.din + j);
        }
    if (VAR == 3)  // a number that no barrier of this launch carries
        for (int k = tid; k < 2 * p.nwords; k += blockDim.x)
            s_ll[k] = (unsigned long long)p.ll_base << 32;
    if (VAR == 1) {
        if (tid == 0) {
            for (int s = 0; s < p.NST; ++s) {
                mbar_init(&full[s], 1);
                mbar_init(&empty[s], p.warps);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    if (VAR == 3)
        cluster_sync();  // every CTA's entries are set before anyone writes one

    // Entries first, first + stride, ... of barrier b (b >= 1) into dst, eight
    // polls in flight; false when the wait ran out or the launch is stopping.
    auto gather_words = [&](unsigned *dst, long long b, int first, int stride) -> bool {
        const unsigned long long *src = (VAR == 3 ? s_ll : p.ll) + (size_t)(b & 1) * p.nwords;
        const unsigned want = p.ll_base + (unsigned)b;
        unsigned long long t0 = 0;
        unsigned long long polls = 0;
        for (int base = first; base < p.nwords; base += 8 * stride) {
            unsigned pend = 0;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (base + u * stride < p.nwords)
                    pend |= 1u << u;
            while (pend) {
                unsigned long long v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    v[u] = !((pend >> u) & 1u) ? 0ull
                           : VAR == 3          ? ld_cluster_u64(src + base + u * stride)
                                               : ld_volatile_u64(src + base + u * stride);
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (((pend >> u) & 1u) && (unsigned)(v[u] >> 32) == want) {
                        dst[base + u * stride] = (unsigned)v[u];
                        pend &= ~(1u << u);
                    }
                if (VAR < 2 && pend)
                    __nanosleep(40);  // polls of all CTAs slow the stores they wait for
                if (pend && (++polls & 63ull) == 0) {
                    if (s_abort || ld_volatile_i32(p.err) != kErrNone)
                        return false;
                    const unsigned long long now = globaltimer_ns();
                    if (t0 == 0)
                        t0 = now;
                    if (now - t0 > p.tmo || polls > kBarrierMaxPolls) {
                        record_err(p.err, kErrBarrierTimeout, p.step0 + b);
                        return false;
                    }
                }
            }
        }
        return true;
    };

    // ------------------------------------------------------------ gatherer
    // Variants 1 and 2, one warp: for barrier b it collects every spike word into
    // s_spkb[b & 1] as it is published and announces the barrier in s_gather --
    // while the consumers are still summing history. Buffer b & 1 is free by
    // then: a word of barrier b is published only after its CTA has seen this
    // CTA's words of barrier b - 1, which follow the row pass of b - 2. For the
    // synapses that publish a drive it watches the arrival flags of all CTAs
    // (lane l: CTAs l, l + 32, ...) instead.
    constexpr bool kGath = VAR == 1 || VAR == 2;
    if (kGath && tid >= (VAR == 1 ? NC + 32 : NC)) {
        if (p.G <= 1 || (kWords && wb0 == wb1))
            return;
        for (long long b = 0; b < B; ++b) {
            bool ok = true;
            if (kWords) {
                unsigned *dst = s_spkb + (size_t)(b & 1) * (spk_one / 4);
                if (b == 0) {  // the previous launch's words
                    for (int wi = lane; wi < p.nwords; wi += 32)
                        dst[wi] = __ldcg(p.spk + (size_t)p.phase0 * p.nwords + wi);
                } else {
                    // nobody is much ahead of this CTA: no polls of the L2
                    // while its own warps are still at the step before
                    const unsigned need = (unsigned)b * (unsigned)(wb1 - wb0);
                    const unsigned long long t0 = globaltimer_ns();
                    unsigned polls = 0;
                    while ((int)((unsigned)ld_acquire_cta(&s_done) - need) < 0) {
                        if ((++polls & 63u) == 0 &&
                            (s_abort || ld_volatile_i32(p.err) != kErrNone ||
                             globaltimer_ns() - t0 > p.tmo))
                            break;  // the polls below have their own limit
                        __nanosleep(20);
                    }
                    ok = gather_words(dst, b, lane, 32);
                    if (!ok)
                        s_abort = 1;
                }
            } else {
                const unsigned long long want = (unsigned long long)(b + 1);
                for (int c = lane; c < p.G && ok; c += 32) {
                    const unsigned long long *f = p.flags + (size_t)c * kFlagStride;
                    if (ld_volatile_u64(f) < want) {
                        const unsigned long long t0 = globaltimer_ns();
                        unsigned long long polls = 0;
                        while (ld_volatile_u64(f) < want) {
                            if ((++polls & 255ull) == 0) {
                                if (s_abort || ld_volatile_i32(p.err) != kErrNone) {
                                    ok = false;
                                    break;
                                }
                                if (globaltimer_ns() - t0 > p.tmo || polls > kBarrierMaxPolls) {
                                    record_err(p.err, kErrBarrierTimeout, p.step0 + b);
                                    s_abort = 1;
                                    ok = false;
                                    break;
                                }
                            }
                            __nanosleep(32);
                        }
                    }
                    if (ok)
                        __threadfence();
                }
            }
            if (__any_sync(kFull, !ok))
                return;
            __syncwarp();
            if (lane == 0)
                st_release_cta(&s_gather, (int)(b + 1));
        }
        return;
    }

    // ------------------------------------------------------------ producer
    if (VAR == 1 && tid >= NC) {
        if (lane != 0 || S_b == 0)
            return;
        long long q = 0;  // stages issued
        int st = 0;       // q % NST
        long long rounds = 0;  // q / NST
        bool ok = true;
        const int S_act = p.bal ? p.n / p.G + (blockIdx.x < p.n % p.G ? 1 : 0) : S_b;
        const int nbox = (S_act + p.BW - 1) / p.BW;
        // slots [0, l2_pin) stay L2-resident, the others stream through
        const unsigned long long pol_in = l2_policy(true);
        const unsigned long long pol_out = l2_policy(false);
        int rh0 = (int)(((p.step0 - 2 - RL) % L + L) % L);  // row of the first streamed lag
        // lags k .. lim of a ring of `len` rows, lag k in row rh: a stage holds one
        // contiguous ascending row range (split at the wrap)
        auto issue = [&](const CUtensorMap *map, int k, int lim, int rh, int len, int pin,
                         long long g) {
            while (k <= lim && ok) {
                int cnt = lim - k + 1;
                if (cnt > p.RB)  // what a box holds: fewer than R when the ring is short
                    cnt = p.RB;
                if (cnt > rh + 1)
                    cnt = rh + 1;
                const int y0 = rh - cnt + 1;
                if (rounds > 0 &&
                    !mbar_wait(&empty[st], (unsigned)((rounds - 1) & 1), &s_abort, p.err,
                               p.tmo, g)) {
                    ok = false;
                    break;
                }
                mbar_expect_tx(&full[st], (unsigned)(nbox * p.RB * p.BW * 8));
                double *dst = s_stage + (size_t)st * STAGE;
                if (p.l2_pin > 0) {
                    // the oldest `pin` lags stay resident: a row is read
                    // evict-first while young and turns evict-last when it
                    // reaches lag len - pin (one row per step comes back from
                    // DRAM for that)
                    const unsigned long long pol = k + cnt > len - pin ? pol_in : pol_out;
                    for (int c = 0; c < nbox; ++c)
                        tma_load_2d_hint(dst + (size_t)c * p.R * p.BW, map, lo + c * p.BW, y0,
                                         &full[st], pol);
                } else {
                    for (int c = 0; c < nbox; ++c)
                        tma_load_2d(dst + (size_t)c * p.R * p.BW, map, lo + c * p.BW, y0,
                                    &full[st]);
                }
                ++q;
                if (++st == p.NST) {
                    st = 0;
                    ++rounds;
                }
                k += cnt;
                rh -= cnt;
                if (rh < 0)
                    rh += len;
            }
        };
        for (long long b = 0; b < B && ok; ++b, rh0 = rh0 + 1 == L ? 0 : rh0 + 1) {
            const long long g = p.step0 + b;
            const int lim = (int)(g < L ? g : L - 1);
            const long long gs = p.syn_step0 + b + 1;  // FRACTIONAL: the current formed in step b
            const int slim = ST == SP_SYN_FRAC && p.frac_stage && b + 1 < B
                                 ? (int)(gs < p.Ls ? gs : p.Ls - 1)
                                 : 0;
            if (lim < 2 + RL && slim < 2)
                continue;
            if (b >= 2 || (b == 1 && slim >= 2)) {
                // rows of step g are states of steps <= g-2; the synapse's newest
                // row is the current of step b-1, formed at the end of step b-2
                // or (b = 1) before step 0
                unsigned long long t0 = globaltimer_ns();
                unsigned polls = 0;
                // (kWords: every consumer warp counts its own steps)
                const unsigned need =
                    (unsigned)(b >= 2 ? b - 1 : 1) * (unsigned)(kWords ? wb1 - wb0 : 1);
                while ((int)((unsigned)ld_acquire_cta(&s_done) - need) < 0) {
                    if ((++polls & 63u) == 0) {
                        if (s_abort || ld_volatile_i32(p.err) != kErrNone) {
                            ok = false;
                            break;
                        }
                        if (globaltimer_ns() - t0 > p.tmo) {
                            record_err(p.err, kErrBarrierTimeout, g);
                            s_abort = 1;
                            ok = false;
                            break;
                        }
                    }
                    __nanosleep(64);
                }
                if (!ok)
                    break;
            }
            SP_STAMP(true, b, B, 7);
            if (slim >= 2)
                issue(&p.tmap_s, 2, slim, (int)((gs - 2) % p.Ls), p.Ls, 0, g);
            issue(&p.tmap, 2 + RL, lim, rh0, L, p.l2_pin, g);
        }
        // every issued copy must land before the CTA may exit
        const unsigned long long t0 = globaltimer_ns();
        for (long long qq = (q > p.NST ? q - p.NST : 0); qq < q; ++qq) {
            const int st = (int)(qq % p.NST);
            while (!mbar_test(&full[st], (unsigned)((qq / p.NST) & 1))) {
                if (globaltimer_ns() - t0 > p.tmo)
                    break;
            }
        }
        return;
    }

    // ------------------------------------------------------------ consumers
    const int gw = wb0 + warp;
    const bool wact = gw < wb1;
    const int i = gw * 32 + lane;
    const bool act = wact && __ldg(p.nid_of + i) >= 0;
    // ring writes: evict-first (a row is lag 34 when it is first read back)
    const unsigned long long c_pol_out = VAR == 1 ? l2_policy(false) : 0;

    double V = act ? p.V[i] : 0.0;
    double tprev = 0.0, vlast = 0.0;
    int cpos = 0;
    long long refr = 0;
    unsigned long long rng = 0;
    if (act) {
        if (NT == SP_FLIF_GL || NT == SP_FLIF_CAPUTO)
            tprev = p.tprev[i];
        if (NT == SP_FLIF_GL) {
            long long pr = (p.step0 - 1) % L;
            if (pr < 0)
                pr += L;
            vlast = p.ring[(size_t)pr * p.rs + i];
        }
    }
    // lag 2 + j of the next step: the state of micro-step step0 - 2 - j
    double hreg[RL > 0 ? RL : 1];
#pragma unroll
    for (int j = 0; j < (RL > 0 ? RL : 1); ++j)
        hreg[j] = 0.0;
    if (RL > 0 && act) {
#pragma unroll
        for (int j = 0; j < RL; ++j) {
            const long long pr = ((p.step0 - 2 - j) % L + L) % L;
            hreg[j] = p.ring[(size_t)pr * p.rs + i];
        }
    }
    const double coef1 = NT == SP_FLIF_GL && L > 1 ? __ldg(p.coef + 1) : 0.0;
    if (VAR >= 2 && NT == SP_FLIF_GL && wact) {
        // every thread fills and reads its own column only, the whole of it in flight
#pragma unroll 8
        for (int r = 0; r < L; ++r)
            cp_async8(&ring_at(r), p.ring + (size_t)r * p.rs + i);
        cp_async_commit();
        cp_async_wait<0>();
    }
    if (act) {
        if (NT == SP_FLIF_CAPUTO)
            cpos = p.cap_pos[i];
        if (NT == SP_FLIF_DIFFUSIVE) {
            refr = p.refr_until[i];
            rng = p.rng[i];
        }
    }
    double ptrace = (ST == SP_SYN_PSC_HOM && act) ? p.trace[i] : 0.0;
    double Ilast = 0.0;
    if (ST == SP_SYN_FRAC && act) {
        long long pr = (p.syn_step0 - 1) % p.Ls;
        if (pr < 0)
            pr += p.Ls;
        Ilast = p.Iring[(size_t)pr * p.rs + i];
    }
    // Nothing here publishes, so no other CTA waits for this one's reads of the words
    // and their entries could be overwritten before they are seen. With column
    // blocks (variant 3) a CTA's warps share one spike list: verdict() couples them.
    const bool idle = kWords && (wb0 == wb1 || (VAR == 3 && !wact && !p.col_mode));
    int cur = p.phase0;
    double sprev = 0.0;
    if (act)
        sprev = ((p.spk[cur * p.nwords + gw] >> lane) & 1u) ? 1.0 : 0.0;
    unsigned lastword = 0;
    int cst = 0, cph = 0;  // variant 1: stage consumed next and its phase parity
    double ext = 0.0;

    // this thread's column in a stage
    const int boff = VAR == 1 ? (tid / p.BW) * p.R * p.BW + (tid % p.BW) : 0;
    // Variant 1: sum + lags k .. lim of a ring of `len` rows (lag k in row rh) from
    // the stages, in ascending order; `use` false only passes the stages on. coef(k)
    // is a coefficient: a lambda, because a pointer to either memory makes every one
    // of these loads generic (FLIF_GL, scale-free graph, 128 steps: N=20000, L=1024
    // 25.7 us per step, now 22.6; N=12000, L=2000 35.1, now 27.9).
    auto stage_hist = [&](double hist, auto coef, int k, int lim, int rh, int len, bool use,
                          long long g) -> double {
        while (k <= lim && S_b > 0) {
            int cnt = lim - k + 1;
            if (cnt > p.RB)
                cnt = p.RB;
            if (cnt > rh + 1)
                cnt = rh + 1;
            // on a failed wait the launch aborts at the next barrier_wait;
            // every consumer keeps the same control flow until then
            const bool landed = mbar_wait(&full[cst], (unsigned)cph, &s_abort, p.err, p.tmo, g);
            const double *buf = s_stage + (size_t)cst * STAGE + boff;
            if (landed && use) {
                if ((cnt & 15) == 0) {
                    // full stages of 16, 32 or 64 rows: 16 lags at a time
                    // with their loads batched, still in ascending lag
                    // order (lag k + jr sits at row offset cnt-1-jr)
                    for (int h = 0; h < cnt; h += 16)
                        hist = stage_sum<16>(hist, coef, k + h,
                                             buf + (size_t)(cnt - 16 - h) * p.BW, p.BW);
                } else if ((cnt & 7) == 0) {
                    // stages of 24, 40, 48 or 56 rows: 16 at a time, then 8
                    int h = 0;
                    for (; h + 16 <= cnt; h += 16)
                        hist = stage_sum<16>(hist, coef, k + h,
                                             buf + (size_t)(cnt - 16 - h) * p.BW, p.BW);
                    for (; h < cnt; h += 8)
                        hist = stage_sum<8>(hist, coef, k + h,
                                            buf + (size_t)(cnt - 8 - h) * p.BW, p.BW);
                } else {
                    for (int jr = 0; jr < cnt; ++jr)
                        hist = add(hist, mul(coef(k + jr), buf[(size_t)(cnt - 1 - jr) * p.BW]));
                }
            }
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&empty[cst]);
            if (++cst == p.NST) {
                cst = 0;
                cph ^= 1;
            }
            k += cnt;
            rh -= cnt;
            if (rh < 0)
                rh += len;
        }
        return hist;
    };

    // FRACTIONAL: history sum of the current of micro-step b, whose row is
    // shead. It needs the currents up to step b - 1 only, not the spikes of
    // that step, so it is formed before the barrier, while the other CTAs
    // finish. Variant 1 takes it from the ring's stages where its coefficients
    // fit shared memory: the bulk copies keep more bytes in flight than the
    // threads' loads, sixteen each. (N=20000, 512 lags beside a ring of 1024: 86
    // us per step with one load in flight after the update, 69 with sixteen
    // before the barrier, 43 through the stages; the two histories are 245 MB.)
    double fhist = 0.0;
    int shead = ST == SP_SYN_FRAC ? (int)(p.syn_step0 % p.Ls) : 0;
    int srow = shead;  // its row, counted by empty lanes too
    auto frac_history = [&](long long b) {
        if (VAR == 1 && p.frac_stage && b > 0) {
            const long long gs = p.syn_step0 + b;
            const int lim = (int)(gs < p.Ls ? gs : p.Ls - 1);
            srow = srow + 1 == p.Ls ? 0 : srow + 1;
            fhist = 0.0;
            if (lim >= 1)
                fhist = add(fhist, mul(s_scoef[1], Ilast));
            fhist = stage_hist(fhist, [&](int k) { return s_scoef[k]; }, 2, lim,
                               srow >= 2 ? srow - 2 : srow - 2 + p.Ls, p.Ls, act,
                               p.step0 + b - 1);
            return;
        }
        if (!act)
            return;
        const long long gs = p.syn_step0 + b;
        const int lim = (int)(gs < p.Ls ? gs : p.Ls - 1);
        fhist = 0.0;
        if (lim >= 1)
            fhist = add(fhist, mul(__ldg(p.scoef + 1), Ilast));
        fhist = ring_sum<VAR == 0 ? 4 : 16>(fhist, p.scoef, p.Iring + i, (size_t)p.rs, p.Ls,
                                            shead >= 2 ? shead - 2 : shead - 2 + p.Ls, 2, lim,
                                            [](const double *q) { return __ldcg(q); });
    };
    // synapse prepare for the own neuron before micro-step b (src/synapse.c:145-160)
    auto prepare = [&](long long b, int buf) {
        if (!act)
            return;
        if (ST == SP_SYN_PSC_HOM) {
            ptrace = add(mul(ptrace, p.psc_decay), mul(p.psc_omd, sprev));
            p.eff[(size_t)buf * p.rs + i] = ptrace;
        } else if (ST == SP_SYN_FRAC) {
            // fhist: the history sum of this step, formed by frac_history
            const double rhs = dvd(add(-Ilast, sprev), p.s_tau);
            const double In = sub(mul(p.s_dta, rhs), fhist);
            p.Iring[(size_t)shead * p.rs + i] = In;
            shead = shead + 1 == p.Ls ? 0 : shead + 1;
            Ilast = In;
            p.eff[(size_t)buf * p.rs + i] = In;
        } else if (ST == SP_SYN_FRAC_MEXP) {
            double sum = 0.0;
            for (int c = 0; c < p.Nc; ++c) {
                double tr = p.mx_tr[(size_t)c * p.rs + i];
                tr = add(mul(tr, __ldg(p.mx_decay + c)), mul(__ldg(p.mx_omd + c), sprev));
                p.mx_tr[(size_t)c * p.rs + i] = tr;
                sum = add(sum, mul(__ldg(p.mx_c + c), tr));
            }
            p.eff[(size_t)buf * p.rs + i] = sum;
        }
    };

    // Publication of the words of barrier b (kWords): one entry per warp, or,
    // when one CTA owns every warp, the word itself in shared memory.
    auto publish = [&](long long b, unsigned word) {
        if (VAR == 3) {
            // lane r writes CTA r's copy
            if (wact && lane < p.G && !(b == p.hold_b && (int)blockIdx.x == p.hold_cta))
                st_cluster_u64(s_ll + (size_t)(b & 1) * p.nwords + gw, (unsigned)lane,
                               ((unsigned long long)(p.ll_base + (unsigned)b) << 32) | word);
            return;
        }
        if (!wact || lane != 0)
            return;
        if (p.G > 1) {
            if (b == p.hold_b && (int)blockIdx.x == p.hold_cta)
                return;
            const unsigned long long v =
                ((unsigned long long)(p.ll_base + (unsigned)b) << 32) | word;
            *(volatile unsigned long long *)(p.ll + (size_t)(b & 1) * p.nwords + gw) = v;
        } else {
            s_spkb[(size_t)(b & 1) * (spk_one / 4) + gw] = word;
        }
    };
    // Drive-publishing synapses: per-CTA arrival flags. Arriving at barrier b
    // publishes b + 1 in the CTA's own flag after its drive; waiting, consumer
    // thread t watches the flags of CTAs t, t + NC, ...
    auto barrier_arrive = [&](long long b) {
        named_sync(NC);
        if (tid == 0 && p.G > 1 && !(b == p.hold_b && (int)blockIdx.x == p.hold_cta)) {
            __threadfence();
            *(volatile unsigned long long *)(p.flags + (size_t)blockIdx.x * kFlagStride) =
                (unsigned long long)(b + 1);
        }
    };
    // waits for the gather warp's announcement of barrier b
    auto gather_wait = [&](long long b) -> bool {
        if (ld_acquire_cta(&s_gather) >= (int)(b + 1))
            return true;
        const unsigned long long t0 = globaltimer_ns();
        unsigned polls = 0;
        while (ld_acquire_cta(&s_gather) < (int)(b + 1)) {
            if ((++polls & 63u) == 0) {
                if (s_abort || ld_volatile_i32(p.err) != kErrNone)
                    return false;
                // the gather warp's own limit comes first
                if (globaltimer_ns() - t0 > 2 * p.tmo) {
                    record_err(p.err, kErrBarrierTimeout, p.step0 + b);
                    s_abort = 1;
                    return false;
                }
            }
        }
        return true;
    };
    // The warps of a CTA wait by themselves where they share nothing below;
    // with column blocks they build one spike list, so all must take the same
    // branch: s_bad[b & 1] is written before the barrier only, and for b + 2
    // only after everybody has read it.
    auto verdict = [&](long long b, bool ok) -> bool {
        ok = __all_sync(kFull, ok);
        __syncwarp();  // the vote orders no memory: the lanes' (lane 0's) words before all reads
        if (ST != SP_SYN_SIMPLE || !p.col_mode)
            return ok;
        if (!ok)
            s_bad[b & 1] = 1;
        named_sync(NC);
        return s_bad[b & 1] == 0;
    };
    // returns false when the launch must stop
    auto barrier_wait = [&](long long b) -> bool {
        if (kWords) {
            if (kGath && p.G > 1)
                return verdict(b, lane != 0 || gather_wait(b));
            unsigned *dst = s_spkb + (size_t)(b & 1) * (spk_one / 4);
            if (VAR == 3) {
                // every warp collects all words, writing the same values into the
                // CTA's buffer
                bool ok = true;
                if (!wact) {
                    // column blocks: the others' words, after verdict()
                } else if (b == 0) {
                    for (int wi = lane; wi < p.nwords; wi += 32)
                        dst[wi] = __ldcg(p.spk + (size_t)cur * p.nwords + wi);
                } else {
                    ok = gather_words(dst, b, lane, 32);
                    if (!ok)
                        s_abort = 1;
                }
                return verdict(b, ok);
            }
            if (b == 0) {  // the previous launch's words
                for (int wi = tid; wi < p.nwords; wi += NC)
                    dst[wi] = __ldcg(p.spk + (size_t)cur * p.nwords + wi);
            } else if (p.G > 1) {
                if (!gather_words(dst, b, tid, NC)) {
                    s_abort = 1;
                    s_bad[b & 1] = 1;
                }
            }
            named_sync(NC);
            if (p.G <= 1)
                return true;
            return s_bad[b & 1] == 0;  // as in verdict
        }
        if (kGath && p.G > 1) {
            if (tid == 0 && gather_wait(b))
                __threadfence();  // the drive in global memory is read next
        } else if (p.G > 1) {
            const unsigned long long want = (unsigned long long)(b + 1);
            for (int c = tid; c < p.G; c += NC) {
                const unsigned long long *f = p.flags + (size_t)c * kFlagStride;
                if (ld_volatile_u64(f) < want) {
                    const unsigned long long t0 = globaltimer_ns();
                    unsigned long long polls = 0;
                    bool ok = true;
                    while (ld_volatile_u64(f) < want) {
                        if ((++polls & 255ull) == 0) {
                            if (s_abort || ld_volatile_i32(p.err) != kErrNone) {
                                ok = false;
                                break;
                            }
                            if (globaltimer_ns() - t0 > p.tmo || polls > kBarrierMaxPolls) {
                                record_err(p.err, kErrBarrierTimeout, p.step0 + b);
                                ok = false;
                                break;
                            }
                        }
                        __nanosleep(32);
                    }
                    if (!ok) {
                        s_abort = 1;
                        break;
                    }
                }
                __threadfence();
            }
        }
        named_sync(NC);
        // one verdict for the whole CTA (another CTA may record an error at any
        // moment; every consumer must take the same branch)
        if (tid == 0)
            s_flag = (!s_abort && ld_volatile_i32(p.err) == kErrNone) ? 1 : 0;
        named_sync(NC);
        return s_flag != 0;
    };

    // prologue: drive of micro-step 0, then arrive at barrier 0 (whose spike
    // words are the previous launch's)
    if (!kWords) {
        if (ST == SP_SYN_FRAC)
            frac_history(0);
        prepare(0, cur);
        barrier_arrive(0);
    }

    // Input rows of the next kURows macro steps, in flight to shared memory
    double *s_ur = s_u + (size_t)warp * kURows * p.din;
    auto u_issue = [&](int row) {
        if (lane < p.din && row < p.n_macro)
            cp_async8(s_ur + (row & (kURows - 1)) * p.din + lane, p.u + (size_t)row * p.din + lane);
        cp_async_commit();
    };
    if (p.u_ring && !idle)
        for (int r = 0; r < kURows; ++r)
            u_issue(r);

    // step-invariant places and the counters that follow the step (64-bit
    // divisions cost hundreds of cycles each)
    // Column blocks: the spiking neurons of the barrier's words as an ascending
    // list (all consumers; returns the count). The words are in position order,
    // so the neurons' bits are collected in neuron order first; every thread then
    // takes a run of words, and a scan of their counts places its entries.
    auto spike_list = [&](const unsigned *words) -> int {
        for (int wi = tid; wi < p.nwords; wi += NC)
            for (unsigned mw = words[wi]; mw; mw &= mw - 1) {
                const int nid = __ldg(p.nid_of + wi * 32 + __ffs(mw) - 1);
                atomicOr(s_bits + (nid >> 5), 1u << (nid & 31));
            }
        named_sync(NC);
        const int per = (nwn + NC - 1) / NC;
        const int w0 = tid * per < nwn ? tid * per : nwn, w1 = w0 + per < nwn ? w0 + per : nwn;
        int c = 0;
        for (int wi = w0; wi < w1; ++wi)
            c += __popc(s_bits[wi]);
        int x = c;  // inclusive scan over the warp
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(kFull, x, off);
            if (lane >= off)
                x += y;
        }
        if (lane == 31)
            s_wsum[warp] = x;
        if (p.warps > 1)
            named_sync(NC);
        else
            __syncwarp();
        int at = x - c, total = 0;
        for (int q = 0; q < p.warps; ++q) {
            const int v = s_wsum[q];
            if (q < warp)
                at += v;
            total += v;
        }
        for (int wi = w0; wi < w1; ++wi) {
            for (unsigned mw = s_bits[wi]; mw; mw &= mw - 1)
                s_list[at++] = (unsigned short)(wi * 32 + __ffs(mw) - 1);
            s_bits[wi] = 0u;
        }
        named_sync(NC);
        return total;
    };
    int colw0 = 0;  // column blocks: the warp's first weight
    if (ST == SP_SYN_SIMPLE && p.col_mode && wact)
        colw0 = __ldg(p.col_off + gw) - (p.col_mode == 2 ? __ldg(p.col_off + wb0) : 0);
    int ell0 = 0, elln = 0;  // the warp's slot groups
    unsigned tails = 0;      // its rows with a tail
    if (ST == SP_SYN_SIMPLE && p.ell_cap > 0 && wact) {
        ell0 = __ldg(p.ell_off + gw) - __ldg(p.ell_off + wb0);
        elln = __ldg(p.ell_off + gw + 1) - __ldg(p.ell_off + gw);
        const int *rp = s_tail_rp + 33 * (gw - wb0);
        tails = __ballot_sync(kFull, rp[lane + 1] > rp[lane]);
    }
    int s = 0, m = 0;                   // macro step, micro-step within it
    int head = (int)(p.step0 % L);      // ring row of the step
    for (long long b = idle ? B : 0; b < B; ++b) {
        const long long g = p.step0 + b;
        SP_STAMP(tid == 0, b, B, 0);
        if (m == 0) {
            // ext = 0 + gamma * sum_j W_in[i][j] u[j] (netlib dgemv order)
            ext = 0.0;
            if (p.u_ring) {
                cp_async_wait<kURows - 1>();
                __syncwarp();
                if (act) {
                    const double *ur = s_ur + (s & (kURows - 1)) * p.din;
                    double t = 0.0;
                    if (p.win_smem) {
                        const double *wr = s_win + tid;
                        int j = 0;
                        for (; j + 4 <= p.din; j += 4) {
                            double x[4];
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                x[q] = mul(wr[(j + q) * NC], ur[j + q]);
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                t = add(t, x[q]);
                        }
                        if (j < p.din) {
                            const int k1 = j + 1 < p.din ? j + 1 : j, k2 = j + 2 < p.din ? j + 2 : j;
                            const double x0 = mul(wr[j * NC], ur[j]), x1 = mul(wr[k1 * NC], ur[k1]),
                                         x2 = mul(wr[k2 * NC], ur[k2]);
                            t = add(t, x0);
                            if (k1 > j)
                                t = add(t, x1);
                            if (k2 > j)
                                t = add(t, x2);
                        }
                    } else {
                        const double *wr = p.W_in + (size_t)i * p.din;
                        for (int j = 0; j < p.din; ++j)
                            t = add(t, mul(ldg_na(wr + j), ur[j]));
                    }
                    ext = add(0.0, mul(p.gamma, t));
                }
                __syncwarp();
                u_issue(s + kURows);
            } else if (act && p.din > 0 && p.gamma != 0.0 && p.u) {
                const double *ur = p.u + (size_t)s * p.din;
                const double *wr = p.W_in + (size_t)i * p.din;
                double t = 0.0;
                for (int j = 0; j < p.din; ++j)
                    t = add(t, mul(ldg_na(wr + j), ldg_na(ur + j)));
                ext = add(0.0, mul(p.gamma, t));
            }
        }

        if (ST == SP_SYN_FRAC && b + 1 < B)
            frac_history(b + 1);

        // ---- FLIF_GL history sum of step g
        bool integ = false;
        double hist = 0.0, leak = 0.0;  // what of the update does not wait for the barrier
        if (NT == SP_FLIF_GL) {
            integ = tprev > p.f;
            leak = dvd(-sub(vlast, p.c), p.d);
            const int lim = (int)(g < L ? g : L - 1);
            if (act && integ && lim >= 1)
                hist = add(hist, mul(coef1, vlast));
            if (VAR == 0) {
                if (act && integ)
                    hist = ring_sum<4>(hist, p.coef, p.ring + i, (size_t)p.rs, L,
                                       head >= 2 ? head - 2 : head - 2 + L, 2, lim,
                                       [](const double *q) { return __ldcg(q); });
            } else if (VAR >= 2) {
                // the whole history of the CTA's neurons is in shared memory
                if (act && integ && lim >= 2) {
                    const int r = head >= 2 ? head - 2 : head - 2 + L;
                    const int cnt = lim - 1, n1 = cnt < r + 1 ? cnt : r + 1;
                    hist = chain_pairs(hist, s_coef, s_coef1, s_ring, 2, r, n1);
                    if (cnt > n1)
                        hist = chain_pairs(hist, s_coef, s_coef1, s_ring, 2 + n1, L - 1, cnt - n1);
                }
            } else {
                int rh = head - 2 - RL;
                while (rh < 0)
                    rh += L;
                // lags 2 .. RL+1 from registers, in ascending order, then the stages
                auto lags = [&](auto coef) {
                    if (act && integ) {
#pragma unroll
                        for (int j = 0; j < RL; ++j)
                            if (2 + j <= lim)
                                hist = add(hist, mul(coef(2 + j), hreg[j]));
                    }
                    hist = stage_hist(hist, coef, 2 + RL, lim, rh, L, act && integ, g);
                };
                if (p.coef_smem)
                    lags([&](int k) { return s_coef[k]; });
                else
                    lags([&](int k) { return __ldg(p.coef + k); });
            }
        }

        // ---- FLIF_CAPUTO memory sum: the newest entry is V - V_0 of the last
        // step, so nothing of it waits for this step's input
        double cmem = 0.0;
        if (NT == SP_FLIF_CAPUTO) {
            integ = act && tprev > p.f;
            if (integ)
                cmem = caputo_sum<VAR == 0 ? 1 : 8>(sub(V, p.b), p.coef_smem ? s_coef : p.coef + 4,
                                                    p.ring, (long long)i * L, L, cpos);
        }

        // ---- barrier: spikes / eff of step g-1 are visible
        SP_STAMP(tid == 0, b, B, 1);
        if (!barrier_wait(b)) {
            // Input rows still on their way. Not in variant 0, where any code on this
            // way out slows the step (column blocks in global memory, N=4000: 8.1 us,
            // 8.7 with the wait); like every load, they end before the CTA's memory
            // is another's.
            if (VAR != 0)
                cp_async_wait<0>();
            if (VAR == 3)
                cluster_sync();  // the other CTAs may still write here
            return;
        }
        SP_STAMP(tid == 0, b, B, 2);
        SP_STAMP(tid == 0, b, B, 3);
        const unsigned *s_spk = s_spkb + (size_t)(b & 1) * (spk_one / 4);

        // ---- recurrent input
        double rec = 0.0;
        if (ST == SP_SYN_SIMPLE) {
            if (p.col_mode) {
                const int cnt = spike_list(s_spk);
                if (wact && cnt > 0)
                    rec = p.col_mode == 2
                              ? rowpass_cols<true>(s_col_blk + (gw - wb0) * p.n, s_col_w + colw0,
                                                   s_list, cnt, lane)
                              : rowpass_cols<false>(p.col_blk + (size_t)gw * p.n, p.col_w + colw0,
                                                    s_list, cnt, lane);
            } else if (wact) {
                // CSR rows are in position order; holes are empty rows
                if (p.ell_cap > 0)
                    rec = rowpass_lanes(s_ell_col + 32 * ell0, s_ell_w + 128 * ell0, elln,
                                        s_tail_rp + 33 * (gw - wb0), s_tail_col, s_tail_w, tails,
                                        s_spk, lane);
                else
                    rec = rowpass_simple_warp(p.row_ptr, p.col, p.w, s_spk, gw * 32, 32, lane);
            }
        } else if (wact) {
            // whole warps (holes are empty rows): every edge carries a term
            rec = rowpass_terms_warp<ST>(p, p.eff + (size_t)cur * p.rs, s_spk, gw * 32, lane);
        }

        SP_STAMP(tid == 0, b, B, 4);
        // ---- neuron update (operation order of src/neurons/<model>.c)
        bool fired = false;
        if (act) {
            const double in = add(ext, rec);
            if (NT == SP_LIF_DISCRETE) {
                V = add(add(mul(p.c, V), in), p.d);
                if (V > p.b) {
                    V = p.a;
                    fired = true;
                }
            } else if (NT == SP_LIF_BIO) {
                const double dV = dvd(add(add(-V, in), p.d), p.c);
                V = add(V, mul(dV, p.dt));
                if (V >= p.b) {
                    V = p.a;
                    fired = true;
                }
            } else if (NT == SP_FLIF_GL) {
                if (integ) {
                    const double rhs = add(add(leak, in), p.e);
                    V = sub(mul(p.g, rhs), hist);
                    if (V >= p.a) {
                        V = p.b;
                        fired = true;
                        tprev = 0.0;
                    }
                } else {
                    V = p.b;
                }
                if (VAR == 1 && p.l2_pin > 0)
                    st_hint_f64(p.ring + (size_t)head * p.rs + i, V,
                                c_pol_out);
                else
                    p.ring[(size_t)head * p.rs + i] = V;
                if (VAR >= 2)
                    ring_at(head) = V;
                if (RL > 0) {
#pragma unroll
                    for (int j = (RL > 0 ? RL : 1) - 1; j > 0; --j)
                        hreg[j] = hreg[j - 1];
                    hreg[0] = vlast;
                }
                vlast = V;
                tprev = add(tprev, p.dt);
            } else if (NT == SP_FLIF_CAPUTO) {
                if (integ) {
                    const double dV = dvd(add(mul(-p.c, sub(V, p.d)), in), p.e);
                    const double markov = mul(p.g, dV);
                    p.ring[(size_t)i * L + cpos] = sub(V, p.b);
                    cpos = (cpos + 1 == L) ? 0 : cpos + 1;
                    V = add(V, sub(markov, cmem));
                    if (V >= p.a) {
                        V = p.b;
                        fired = true;
                        tprev = 0.0;
                    }
                } else {
                    V = p.b;
                }
                tprev = add(tprev, p.dt);
            } else if (NT == SP_FLIF_DIFFUSIVE) {
                const double Vp = V;
                const double rhs = add(add(-sub(Vp, p.c), in), p.d);
                V = add(Vp, mul(p.e, rhs));
                if (g >= refr && V >= p.a) {
                    V = p.b;
                    fired = true;
                    long long steps;
                    if (p.diff_sto) {
                        double W;
                        const double u0 = u01(&rng);
                        if (u0 < p.ci) {
                            W = p.h;
                        } else {
                            const double u1 = u01(&rng);
                            const double tmin = p.f, tmax = p.g, qx = p.cj;
                            if (tmax <= tmin)
                                W = tmin;
                            else if (qx <= 1e-12)
                                W = tmin + u1 * (tmax - tmin);
                            else if (fabs(qx - 1.0) < 1e-12)
                                W = tmin * pow(tmax / tmin, u1);
                            else
                                W = pow((1.0 - u1) * p.ck + u1 * p.cl, 1.0 / (1.0 - qx));
                        }
                        steps = (W <= 0.0) ? 0 : (long long)ceil(W / p.dt);
                        if (steps < 1)
                            steps = 1;
                    } else {
                        steps = p.det_refr;
                    }
                    refr = g + steps;
                }
            }
        }
        // the ring row of step g is first read by a bulk copy as lag RL + 2,
        // RL + 2 steps later: with the register lags one proxy fence per 16
        // steps orders every row before that read (kernel boundaries order
        // the rest)
        if (VAR == 1 && (RL < 32 || (g & 15) == 15))
            fence_proxy_async();

        // ---- spike word of step g
        const unsigned word = __ballot_sync(kFull, fired);
        if (kWords && b + 1 < B)
            publish(b + 1, word);  // first: the other CTAs wait for it
        if (wact && lane == 0 && (!kWords || b + 1 == B))
            p.spk[(size_t)(cur ^ 1) * p.nwords + gw] = word;  // read by the next launch
        lastword = word;
        sprev = fired ? 1.0 : 0.0;
        SP_STAMP(tid == 0, b, B, 5);
        if (m == p.micro - 1) {
            if (act && p.phi)  // empty lanes stay 0: a recorded row is read whole
                p.phi[(size_t)s * p.rs + i] = V;
            if (wact && lane == 0 && p.raster)
                p.raster[(size_t)s * p.nwords + gw] = lastword;
        }
        if (b + 1 < B) {
            if (!kWords) {
                prepare(b + 1, cur ^ 1);
                if (VAR == 1 && ST == SP_SYN_FRAC && p.frac_stage)
                    fence_proxy_async();  // the current just written is lag 2 of a bulk copy
                barrier_arrive(b + 1);
                if (VAR == 1 && tid == 0)
                    st_release_cta(&s_done, (int)(b + 1));
            } else if (kGath) {
                __syncwarp();
                if (wact && lane == 0)
                    red_release_cta(&s_done, 1);
            }
        }
        SP_STAMP(tid == 0, b, B, 6);
        cur ^= 1;
        head = head + 1 == L ? 0 : head + 1;
        if (++m == p.micro) {
            m = 0;
            ++s;
        }
    }

    if (VAR == 3)
        cluster_sync();
    if (act) {
        p.V[i] = V;
        if (NT == SP_FLIF_GL || NT == SP_FLIF_CAPUTO)
            p.tprev[i] = tprev;
        if (NT == SP_FLIF_CAPUTO)
            p.cap_pos[i] = cpos;
        if (NT == SP_FLIF_DIFFUSIVE) {
            p.refr_until[i] = refr;
            p.rng[i] = rng;
        }
        if (ST == SP_SYN_PSC_HOM)
            p.trace[i] = ptrace;
    }
}

}  // namespace sp
