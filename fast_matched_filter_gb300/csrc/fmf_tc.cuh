// fmf_tc.cuh -- what the tensor-core kernels share: the searches of a
// persistent launch and its tile queue, tile geometry, and the PTX of
// mbarriers, bulk copies, tcgen05 and tensor memory.
#pragma once

#include "fmf_common.cuh"

namespace fmf {

constexpr int TC_Q = 128;
constexpr int TC_CB = TC_Q / 8;
constexpr int TC_TG = 16;  // templates interleaved per group of CTAs (L2 reuse of data rows)
constexpr int TC_NB_MAX = 128;  // largest tile: lag blocks, and columns of one accumulator
constexpr unsigned long long TC_WAIT_NS = 2000000000ull;  // 2 s per wait


// One search of a persistent launch (tile-queue items [item_begin, item_begin + n_tiles*T)).
struct TcProb {
    Problem P;                    // sizes, epilogue inputs, output
    const uint16_t *g_hi, *g_lo;  // bf16 (FP32 form: fp16) bits, data streams [SC][step][CB][rows_total][8]
    const uint16_t *w_hi, *w_lo;  // the same, template blocks [T][SC][step][NW][64]
    long long item_begin;         // first tile-queue item of this search
    int R;                        // data rows per stage
    int NW;                       // 128-byte template blocks per (template, channel, phase)
    int rows_total;               // rows per (channel, stream) in the data streams
    int row_front;                // rows of zero padding before sample 0
    int n_tiles;                  // output tiles of nb*128 indices
    int tg;                       // templates interleaved per group of items
    int nb;                       // lag blocks per tile (MMA N): 32, 64 or 128
    int parts;                    // k >= 1: the channels of a (tile, template) in k
                                  // ranges [j SC / k, (j + 1) SC / k) on k CTAs (items
                                  // j = 0..k-1 adjacent); their network sums go to
                                  // part_out[j][t][lag] and are added in order j after
                                  // the launch (a fixed order: deterministic results)
    float *part_out;
    // FP32 form (fmf_tc.cu): operands are fp16 pairs in units of powers of two
    const int *t_exp;             // [T][SC] exponent of each channel's template
    const int *d_exp;             // [SC] exponent of each data channel
    int chains;                   // h h chains of a channel that uses all phases, of as many
                                  // column-block pairs each as it goes; 0: one, whatever its phases
    int chain_steps;              // a pair of more K steps than this is several chains (tc_pair_chains); 0: one
    const unsigned *skip;         // nonzero: the FP32 CUDA-core kernel runs this search instead
};

struct TcLaunch {
    int n_probs;
    int split;                    // 1: hi/lo, three products; 0: single bf16 product
    uint32_t mma_types;           // operand types, in their place in the MMA's instruction descriptor
    float lo_unit;                // what a low half counts in units of the high one
    // shared memory: template buffers (2), data slots, statistics slots (2^stat_log2)
    int w_bytes, n_rows, row_bytes, stat_log2, stat_bytes;
    long long total_items;
    unsigned long long *queue;    // tile-queue head, zero before the launch
    unsigned *err;                // device error word
};

// The kernel's parameter: a lone search's is a 64th of a batch's (27 KB, which cost the
// caller 4 us more a launch).
template <int N>
struct TcBatch : TcLaunch {
    TcProb prob[N];
};

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ unsigned long long gtimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait on an mbarrier phase.  Returns false when the CTA aborted or
// when this wait gave up after `limit_ns` (then it raises the error word and
// the abort flag).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag,
                                          unsigned *err, unsigned code,
                                          unsigned long long limit_ns = TC_WAIT_NS)
{
    if (mbar_try(bar, parity))
        return true;
    unsigned long long t0 = gtimer();
#pragma unroll 1
    for (unsigned it = 1;; it++) {
        if (mbar_try(bar, parity))
            return true;
        if ((it & 63) == 0) {
            if (*abort_flag)
                return false;
            if (gtimer() - t0 > limit_ns) {
                atomicOr(err, code);
                *abort_flag = 1;
                return false;
            }
        }
    }
}

// Warp-uniform form: lane 0 waits, the result is broadcast to the warp.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag,
                                               unsigned *err, unsigned code)
{
    int ok = 0;
    if ((threadIdx.x & 31) == 0)
        ok = mbar_wait(bar, parity, abort_flag, err, code) ? 1 : 0;
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

// Before a slot that this thread has read goes back to the bulk copies: its reads are
// done (an arrival alone does not wait for loads in flight, and a copy overtook
// them while the load pipe was busy with stores).
__device__ __forceinline__ void fence_reads_before_copy()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Every lane waits; true only if all of them saw the phase complete.
__device__ __forceinline__ bool mbar_wait_all(uint32_t bar, uint32_t parity, volatile int *abort_flag,
                                              unsigned *err, unsigned code)
{
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, err, code)) != 0;
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}

// Shared-memory matrix descriptor, no swizzle (layout type 0), version 1.
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Descriptors in halves: the start address is in the low word, and only it moves
// along K, so the high words stay put.
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo,
                                        uint32_t b_hi, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n .reg .pred p;\n .reg .b64 a, b;\n setp.ne.b32 p, %6, 0;\n mov.b64 a, {%1, %2};\n"
        " mov.b64 b, {%3, %4};\n tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n}\n" ::"r"(d_tmem),
        "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     bar)
                 : "memory");
}

// One lane of a converged warp.
__device__ __forceinline__ bool elect_one()
{
    uint32_t one;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
    return one != 0;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 32 lanes x 32 bits, 16 consecutive columns per thread
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v)
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
        "[%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 16; i++)
        v[i] = __uint_as_float(r[i]);
}

// 32 lanes x 32 bits, 32 consecutive columns per thread
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float *v)
{
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 32; i++)
        v[i] = __uint_as_float(r[i]);
}

// ------------------------------------------------------------------ epilogue arithmetic
// 1/sqrt(x), one approximate MUFU operation; subnormal x is flushed to zero
// (result +inf).
__device__ __forceinline__ float rsqrt_ftz(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// atanh(y) in FP32 for the Fisher-z network sum, at most a few ulp from the
// exact value (the accuracy of the CUDA library's atanhf) with far fewer
// instructions for the common small arguments:
//  |y| <= 1/4: the Maclaurin series y + y^3/3 + ... + y^13/13 (the first
//    omitted term is below 2^-25 of the result);
//  1/4 < |y| < 1: atanh(a) = ln(q) / 2 with q = (1 + a) / (1 - a); q = 2^k m
//    with m in [sqrt(1/2), sqrt(2)) and ln(m) = 2 atanh(s), s = (m - 1) / (m + 1),
//    |s| <= 0.1716, from the same series to s^9/9;
//  |y| = 1 gives +-inf, |y| > 1 and NaN give NaN.
__device__ __forceinline__ float atanh_series(float y)
{
    const float z = y * y;
    float p = fmaf(1.0f / 13.0f, z, 1.0f / 11.0f);
    p = fmaf(p, z, 1.0f / 9.0f);
    p = fmaf(p, z, 1.0f / 7.0f);
    p = fmaf(p, z, 1.0f / 5.0f);
    p = fmaf(p, z, 1.0f / 3.0f);
    return fmaf(y * z, p, y);
}

__device__ __forceinline__ float atanh_reduced(float y)
{
    const float a = fabsf(y);
    if (!(a < 1.0f))  // 1, above 1, NaN
        return a == 1.0f ? copysignf(INFINITY, y) : __int_as_float(0x7fc00000);
    const float q = __fdividef(1.0f + a, 1.0f - a);  // in (5/3, 2^25] for a > 1/4
    const int bits = __float_as_int(q);
    const int k = (bits - 0x3f3504f3) >> 23;  // 0x3f3504f3 = sqrt(1/2)
    const float m = __int_as_float(bits - (k << 23));
    const float s = __fdividef(m - 1.0f, m + 1.0f);
    const float z = s * s;
    float p = fmaf(1.0f / 9.0f, z, 1.0f / 7.0f);
    p = fmaf(p, z, 1.0f / 5.0f);
    p = fmaf(p, z, 1.0f / 3.0f);
    float r = fmaf(s * z, p, s);                         // ln(m) / 2
    r = fmaf((float)k, 0.5f * 0.693145751953125f, r);    // + k ln2 / 2 (ln2 in two parts)
    r = fmaf((float)k, 0.5f * 1.4286068203094172e-06f, r);
    return copysignf(r, y);
}

// Called by all 32 lanes of a warp together, N values each: the series on every value,
// the reduction only when some value of the warp needs it (one vote for all; the
// common case, every |y| <= 1/4, skips it).
template <int N>
__device__ __forceinline__ void fisher_atanh(float (&y)[N])
{
    bool big = false;  // NaN included
    float r[N];
#pragma unroll
    for (int i = 0; i < N; i++) {
        big = big || !(fabsf(y[i]) <= 0.25f);
        r[i] = atanh_series(y[i]);
    }
    if (__any_sync(0xffffffffu, big)) {
#pragma unroll
        for (int i = 0; i < N; i++)
            r[i] = fabsf(y[i]) <= 0.25f ? r[i] : atanh_reduced(y[i]);
    }
#pragma unroll
    for (int i = 0; i < N; i++)
        y[i] = r[i];
}

// ------------------------------------------------------------------ tile queue
// Decodes a tile-queue item: search p, output tile, template t.  Items of one
// search are ordered so that groups of `tg` templates sweep the tiles together.
template <int N>
__device__ __forceinline__ void decode_item(const TcBatch<N> &B, long long item, int &p, int &tile, int &t,
                                            int &c_begin, int &c_end, int &part)
{
    int lo = 0, hi = N == 1 ? 0 : B.n_probs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (B.prob[mid].item_begin <= item)
            lo = mid;
        else
            hi = mid - 1;
    }
    p = lo;
    const TcProb &pr = B.prob[p];
    long long local = item - pr.item_begin;
    c_begin = 0;
    c_end = pr.P.SC;
    part = 0;
    if (pr.parts > 1) {  // the parts of a (tile, template) are adjacent items
        const int k = pr.parts;
        part = (int)(local % k);
        local /= k;
        c_begin = (int)((long long)part * pr.P.SC / k);
        c_end = (int)((long long)(part + 1) * pr.P.SC / k);
    }
    const long long per_group = (long long)pr.n_tiles * pr.tg;
    const int grp = (int)(local / per_group);
    const long long rem = local - (long long)grp * per_group;
    const int tg0 = grp * pr.tg;
    const int tgn = min(pr.tg, pr.P.T - tg0);
    tile = (int)(rem / tgn);
    t = tg0 + (int)(rem % tgn);
}

// ------------------------------------------------------------------ tile geometry
// Taps of phase phi of a channel that uses the first n of L taps.
__host__ __device__ __forceinline__ int tc_phase_taps(int L, int step, int phi, int n)
{
    const int all = (L - phi + step - 1) / step;
    const int own = n > phi ? (n - phi + step - 1) / step : 0;
    return own < all ? own : all;
}

// Phases of a channel that uses the first n taps: those past its taps hold none.
__host__ __device__ __forceinline__ int tc_phases(int step, int n) { return n < step ? (n < 1 ? 1 : n) : step; }

// End of the K range of a phase with moveout residual s (its start is s & ~15).
__host__ __device__ __forceinline__ int tc_k_end(int s, int taps) { return (s + taps + TC_Q - 1 + 15) & ~15; }

// log2 of the chains that the K steps of one column-block pair make, of a channel that uses
// the first n taps.  A pair has at least ceil(taps / 128) steps of a phase with `taps`
// taps (the last phase has the fewest), so that none of the chains is empty.
__host__ __device__ __forceinline__ int tc_pair_chains(int L, int step, int n, int chain_steps)
{
    int log2 = 0;
    if (chain_steps) {
        const int least = (tc_phase_taps(L, step, step - 1, n) + TC_Q - 1) / TC_Q;
        while (least > chain_steps << log2)
            log2++;
    }
    return log2;
}

struct TcShape {
    int k_span, R, NW;
    size_t stage;
};

inline TcShape tc_shape(int L, int step, int split, int nb)
{
    TcShape g;
    const int lphi = (L + step - 1) / step;
    g.k_span = ((2 * TC_Q - 2 + lphi) + 15) & ~15;
    g.R = nb + (g.k_span - 1) / TC_Q + 1;
    g.NW = g.k_span / 8 + 16;
    g.stage = (size_t)(split ? 2 : 1) * ((size_t)TC_CB * g.R * 16 + (size_t)g.NW * 128);
    g.stage = (g.stage + 1023) & ~(size_t)1023;
    return g;
}

// Geometry of one search in `pr` (tiles, rows, padding).
inline TcShape tc_fill_shape(const Problem &P, int split, int nb, int tg, TcProb *pr)
{
    const TcShape g = tc_shape(P.L, P.step, split, nb);
    *pr = TcProb();
    pr->P = P;
    pr->R = g.R;
    pr->NW = g.NW;
    pr->n_tiles = (int)((P.n_corr + (long long)TC_Q * nb - 1) / ((long long)TC_Q * nb));
    pr->tg = tg > 0 ? tg : TC_TG;
    pr->nb = nb;
    // Stream rows a tile can touch.  An item is processed only when its tile
    // holds a valid output k of its template, i.e. k*step + mo >= 0 and
    // k*step + mo + L <= N for every channel; hence its first row
    // r0 = (I0 + mu - s)/Q lies in [-(NB + 2), (N/step + 1)/Q + 1] whatever the
    // moveouts are, and rows [r0, r0 + R) stay inside the padded stream.
    pr->row_front = nb + 3;
    pr->rows_total = pr->row_front + (int)(((long long)P.N / P.step + 2) / TC_Q) + 2 + g.R + 1;
    pr->parts = 1;
    return g;
}

}  // namespace fmf
