// fmf_tc32.cu -- the FP32 form on the tensor cores (tcgen05 / TMEM).
//
// Same outputs as the CUDA-core kernel (fmf_plain.cu), which is bound by the
// FP32 FMA pipe; the tile geometry and the descriptor views of data and
// templates are those of fmf_tc.cu (Toeplitz x Hankel, neither built).  What
// keeps the products and sums at FP32 accuracy:
//
//   * Operands are pairs of fp16 numbers, x = s (h + 2^-11 l): s a power of two
//     (per data channel, per template channel) that brings the largest value
//     to [2^14, 2^15), h = fp16(x / s), l = fp16(2^11 (x / s - h)).  h has 11
//     significant bits and l the next 11, so the pair holds x to half a unit
//     of FP32's last place, down to 2^-50 of the channel's largest value
//     (below that l runs out of exponent).  One K step is three MMAs, h h,
//     h l and l h; the dropped l l is at most 2^-24 of |t d|.
//   * The tensor core rounds every accumulation toward zero, so a long chain
//     drifts: one accumulator over the 38 steps of a 600-tap template was
//     2.3e-8 RMS off (FP32 FMAs: 1.8e-8), 1.2e-6 at a perfect match.  So the
//     h h products run in chains of at most kChain steps, each in a fresh
//     accumulator that the epilogue adds to its registers in FP32 (rounded to
//     nearest); h l and l h, 2^-11 smaller, share one accumulator per channel.
//
// Roles of a persistent CTA (12 warps, one CTA per SM), tile queue as in
// fmf_tc.cu:
//   warp 0      producer: claims items, TMA bulk copies of one (channel, phase)
//               stage into two buffers in turn
//   warp 1      issues the h h MMAs into H0 / H1 in turn, one chain each
//   warp 2      issues the h l and l h MMAs into S0 / S1, one channel each (two
//               issuers: one thread cannot issue fast enough, and neither
//               waits for the other's accumulators)
//   warps 4-11  epilogue: chains into registers, then per channel the
//               normalisation and the network sum, both in registers (208 per
//               thread; the other four warps give theirs up)
// TMEM: H0, H1, S0, S1 of 128 columns each: all 512.
#include <cfloat>
#include <cstdlib>

#include <cuda_fp16.h>

#include "fmf_tc.cuh"

namespace fmf {

constexpr int T32_EPI_WARPS = 8;
constexpr int T32_THREADS = 32 * (4 + T32_EPI_WARPS);
constexpr int T32_MAX_ROWS = 8;     // data slots, at most
constexpr int T32_MAX_STATS = 2;    // statistics slots, at most
constexpr int kChain = 16;          // K steps of one h h chain
constexpr float kLoScale = 2048.0f;  // l is kept 2^11 up
constexpr int kTopExp = 15;          // operands are scaled to below 2^15
// data and template channels whose largest value lies outside [2^-41, 2^60) go
// to the CUDA-core kernel: the products of their scales would leave FP32
constexpr int kMinExp = -40, kMaxExp = 60;

__device__ __forceinline__ float exp2_int(int e)  // 2^e, -126 <= e <= 127
{
    return __int_as_float((e + 127) << 23);
}

// exponent e with m = f 2^e, f in [1/2, 1), from the bits of a finite m >= 0; kTopExp
// (scale 1) for 0
__device__ __forceinline__ int max_exponent(unsigned bits, bool &ok)
{
    const int e = (int)(bits >> 23) - 126;
    ok = bits == 0 || (e >= kMinExp && e <= kMaxExp);
    return bits != 0 && ok ? e : kTopExp;
}

__device__ __forceinline__ bool finite_bits(unsigned abs_bits) { return abs_bits < 0x7f800000u; }

// x / s as the pair (h, l); x that is not finite becomes 0: every window that
// holds it has a NaN energy, and its coefficient is 0 in both kernels.
__device__ __forceinline__ void split_fp16(float x, float inv_s, uint16_t &hi, uint16_t &lo)
{
    const float y = finite_bits(__float_as_uint(x) & 0x7fffffffu) ? x * inv_s : 0.0f;
    const __half h = __float2half_rn(y);
    const __half l = __float2half_rn((y - __half2float(h)) * kLoScale);
    hi = __half_as_ushort(h);
    lo = __half_as_ushort(l);
}

__device__ __forceinline__ uint4 pack8(const uint16_t *v)
{
    uint4 r;
    r.x = v[0] | ((uint32_t)v[1] << 16);
    r.y = v[2] | ((uint32_t)v[3] << 16);
    r.z = v[4] | ((uint32_t)v[5] << 16);
    r.w = v[6] | ((uint32_t)v[7] << 16);
    return r;
}

// Whether a tile of template t holds a valid output and the search runs here.
__device__ __forceinline__ bool tc32_busy(const TcProb &pr, long long I0, int t)
{
    return I0 < pr.P.k_hi[t] && I0 + (long long)TC_Q * pr.nb > pr.P.k_lo[t] && !*pr.skip;
}

// Moveout of phase phi in its stream, and the stream: m = step mu + psi.
__device__ __forceinline__ int tc32_phase(int m, int step, int &psi)
{
    if (step == 1) {
        psi = 0;
        return m;
    }
    const int mu = m >= 0 ? m / step : -((-m + step - 1) / step);
    psi = m - step * mu;
    return mu;
}

// Columns of each half tile in one statistics slot, and the bytes of that half: one
// 16-byte group more than the columns, for windows that start between two groups.
__host__ __device__ constexpr int tc32_stat_columns(bool full) { return full ? 16 : 32; }
__host__ __device__ constexpr uint32_t tc32_stat_half(bool full)
{
    return (uint32_t)(tc32_stat_columns(full) * TC_Q * (full ? 8 : 4) + 16);
}

// ------------------------------------------------------------------ operands
// Data streams as tc_data_kernel lays them out, as fp16 pairs.  The first
// thread of a channel also writes its exponent and decides whether the
// channel's values can be held: stat is the scan of prepare_problem (largest
// |x|; smallest window energy that can pass the threshold, complemented).
// The error of a coefficient from the pairs is at most 2^-51 of the largest
// value over the root of the window's energy, so windows down to 2^-42 of
// the largest value squared keep it at 1e-9.
__global__ void tc32_data_kernel(const float *__restrict__ data, int N, int SC, int step, int rows_total,
                                 int row_front, const unsigned *__restrict__ stat,
                                 uint16_t *__restrict__ g_hi, uint16_t *__restrict__ g_lo,
                                 int *__restrict__ d_exp, unsigned *skip)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long per_ch = (long long)step * TC_CB * rows_total;
    if (idx >= per_ch * SC)
        return;
    const int ch = (int)(idx / per_ch);
    long long rest = idx - ch * per_ch;
    const unsigned top = stat[ch];
    bool ok;
    const int e = max_exponent(top, ok);
    if (rest == 0) {
        d_exp[ch] = e;
        const unsigned low = ~stat[SC + ch];  // smallest energy's bits; ~0 (a NaN): none
        const float m = __uint_as_float(top);
        if (!ok || (low < 0x7f800000u && __uint_as_float(low) * 0x1p42f < m * m))
            atomicOr(skip, 1u);
    }
    const int r = (int)(rest % rows_total);
    rest /= rows_total;
    const int cb = (int)(rest % TC_CB);
    const int psi = (int)(rest / TC_CB);
    const long long x0 = (long long)TC_Q * (r - row_front) + 8 * cb;
    const float *src = data + (size_t)ch * N;
    const float inv_s = exp2_int(kTopExp - e);
    uint16_t h[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const long long pos = (long long)step * (x0 + i) + psi;
        const float v = (x0 + i >= 0 && pos < N) ? src[pos] : 0.0f;
        split_fp16(v, inv_s, h[i], l[i]);
    }
    reinterpret_cast<uint4 *>(g_hi)[idx] = pack8(h);
    reinterpret_cast<uint4 *>(g_lo)[idx] = pack8(l);
}

// Template blocks as tc_template_kernel lays them out, as fp16 pairs; one block
// per (template, channel), its taps in shared memory (read once, written 8
// times over).  Also the channel's exponent.
__global__ void __launch_bounds__(256) tc32_template_kernel(
    const float *__restrict__ tpl, const int *__restrict__ mo, int L, int step, int NW,
    uint16_t *__restrict__ w_hi, uint16_t *__restrict__ w_lo, int *__restrict__ t_exp, unsigned *skip)
{
    extern __shared__ float taps[];
    __shared__ unsigned red[8];
    __shared__ int bad;
    const long long row = blockIdx.x;  // t*SC + ch
    const float *src = tpl + row * L;
    if (threadIdx.x == 0)
        bad = 0;
    __syncthreads();
    unsigned top = 0;
    for (int j = threadIdx.x; j < L; j += blockDim.x) {
        const float v = src[j];
        taps[j] = v;
        const unsigned b = __float_as_uint(v) & 0x7fffffffu;
        if (finite_bits(b))
            top = max(top, b);
        else
            bad = 1;  // the CUDA-core kernel decides what such a template gives
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = top;
    __syncthreads();
    top = red[0];
    for (int i = 1; i < (int)(blockDim.x >> 5); i++)
        top = max(top, red[i]);
    bool ok;
    const int e = max_exponent(top, ok);
    const float inv_s = exp2_int(kTopExp - e);
    const int m0 = mo[row];
    if (threadIdx.x == 0) {
        if (!ok || bad)
            atomicOr(skip, 1u);
        t_exp[row] = e;
    }
    const int per_phase = NW * 8;
    for (int i = threadIdx.x; i < step * per_phase; i += blockDim.x) {
        const int phi = i / per_phase, ne = i - phi * per_phase;
        int psi;
        const int s = tc32_phase(m0 + phi, step, psi) & (TC_Q - 1);
        uint16_t h[8], l[8];
        const int q0 = 8 * (ne >> 3) + (ne & 7) - (TC_Q - 1 + s);
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const int q = q0 + c, j = step * q + phi;
            split_fp16(q >= 0 && j < L ? taps[j] : 0.0f, inv_s, h[c], l[c]);
        }
        const long long o = row * step * per_phase + i;
        reinterpret_cast<uint4 *>(w_hi)[o] = pack8(h);
        reinterpret_cast<uint4 *>(w_lo)[o] = pack8(l);
    }
}

// ------------------------------------------------------------------ persistent kernel
// Offsets of the barriers in the kernel's shared memory (bytes past the rings).
struct T32Bars {
    static constexpr uint32_t wfull = 0, wempty = 16, dfull = 32, dempty = dfull + 8 * T32_MAX_ROWS,
                              efull = dempty + 8 * T32_MAX_ROWS, eempty = efull + 8 * T32_MAX_STATS,
                              hfull = eempty + 8 * T32_MAX_STATS, hempty = hfull + 16, sfull = hempty + 16,
                              sempty = sfull + 16, ifull = sempty + 16, iempty = ifull + 32,
                              fin = iempty + 32, items = fin + 8, tmem = items + 32, abort = tmem + 4,
                              bytes = abort + 4;
};

// One MMA issuer's walk over the items: the h h products (SMALL false; chains of
// chain_slots data slots into H0 / H1 in turn) or the h l and l h products (into
// S0 / S1, a channel each).
template <bool VAR, bool SMALL>
__device__ __forceinline__ void tc32_issue(const TcBatch &B, const long long *ring, uint32_t bar,
                                           uint32_t w_base, uint32_t d_base, uint32_t tmem,
                                           volatile int *abort_flag, bool one)
{
    const auto uniform = [](int v) { return __shfl_sync(0xffffffffu, v, 0); };
    // the whole warp waits and keeps the books; its elected lane issues
    const auto wait = [&](uint32_t b, uint32_t parity, unsigned code) {
        return __all_sync(0xffffffffu, mbar_wait(b, parity, abort_flag, B.err, code)) != 0;
    };
    uint32_t stages = 0, slot = 0, turn = 0;
    uint32_t acc_i = 0;  // accumulators (channels or chains) begun
    const uint32_t n_rows = (uint32_t)B.n_rows;
    for (uint32_t q = 0;; q++) {
        const uint32_t is = q & 3;
        if (!wait(bar + T32Bars::ifull + 8 * is, (q >> 2) & 1, 32u))
            return;
        const long long item = ring[is];
        __syncwarp();
        if (one)
            mbar_arrive(bar + T32Bars::iempty + 8 * is);
        if (item >= B.total_items)
            return;
        int p, tile, t, c_begin, c_end, part;
        decode_item<true>(B, item, p, tile, t, c_begin, c_end, part);
        p = uniform(p);
        t = uniform(t);
        c_end = uniform(c_end);
        const TcProb &pr = B.prob[p];
        const int nb = pr.nb;
        if (!uniform(tc32_busy(pr, (long long)tile * TC_Q * nb, t)))
            continue;
        // kind::f16 descriptor: F32 accumulate, FP16 A and B, K-major, N = nb, M = 128
        const uint32_t idesc = (1u << 4) | ((uint32_t)(nb >> 3) << 17) | ((uint32_t)(TC_Q >> 4) << 24);
        const int SC = pr.P.SC, step = pr.P.step, L = pr.P.L;
        const uint32_t chain_cols = (uint32_t)pr.chain_cols;
        const uint32_t col_bytes = (uint32_t)pr.R * 16;
        // 16-byte units from a high half to its low half, and of a column-block pair
        const uint32_t a_low = (uint32_t)pr.NW * 8, b_low = 4u * (uint32_t)pr.R, b_pair = 2u * (uint32_t)pr.R;
        const uint32_t a_hi = (uint32_t)(sdesc(0, 128, 128) >> 32);
        const uint32_t b_hi = (uint32_t)(sdesc(0, col_bytes, 128) >> 32);
        const uint32_t a_base = (uint32_t)sdesc(w_base, 128, 128), b_base = (uint32_t)sdesc(d_base, col_bytes, 128);
        const uint32_t a_buf = (uint32_t)B.w_bytes >> 4, b_slot = (uint32_t)B.row_bytes >> 4;
        const size_t row0 = (size_t)t * SC;
        for (int g0 = uniform(c_begin); g0 < c_end; g0 += 32) {
            // the scalars of 32 channels, one per lane
            const int cl = min(g0 + (int)(threadIdx.x & 31), c_end - 1);
            const int mo_l = pr.P.mo[row0 + cl], n_l = VAR ? pr.P.ntap[row0 + cl] : L;
            uint32_t active = __ballot_sync(0xffffffffu, g0 + (int)(threadIdx.x & 31) < c_end && pr.P.w[row0 + cl] != 0.0f);
            for (; active; active &= active - 1) {
                const int src = __ffs(active) - 1;
                const int mo = __shfl_sync(0xffffffffu, mo_l, src), ntap = __shfl_sync(0xffffffffu, n_l, src);
                uint32_t left = 0;  // column-block pairs left to the accumulator
                uint32_t dt = 0, acc = 0;
                for (int phi = 0; phi < step; phi++, stages++) {
                    const uint32_t wb = stages & 1;
                    int psi;
                    const uint32_t sres = (uint32_t)tc32_phase(mo + phi, step, psi) & (TC_Q - 1);
                    const uint32_t k_first = sres & ~15u;
                    const uint32_t k_end = (uint32_t)tc_k_end((int)sres, step == 1 ? ntap : tc_phase_taps(L, step, phi, ntap));
                    if (!wait(bar + T32Bars::wfull + 8 * wb, (stages >> 1) & 1, 8u))
                        return;
                    const uint32_t a0 = a_base + (wb ? a_buf : 0u);
#pragma unroll 1
                    for (uint32_t j = 0; j < TC_CB / 2; j++) {
                        if (left == 0) {  // the next accumulator
                            const uint32_t empty = bar + (SMALL ? T32Bars::sempty : T32Bars::hempty) + 8 * (acc_i & 1);
                            if (acc_i >= 2 && !wait(empty, ((acc_i >> 1) - 1) & 1, 4u))
                                return;
                            tc_fence_after();
                            dt = tmem + (SMALL ? 256u : 0u) + 128u * (acc_i & 1);
                            acc = 0;
                            left = SMALL ? (uint32_t)step * (TC_CB / 2) : chain_cols;
                        }
                        // two column-block pairs per slot
                        if ((j & 1) == 0 && !wait(bar + T32Bars::dfull + 8 * slot, turn & 1, 8u))
                            return;
                        // K steps k = 16 j + 128 i: A moves 16 template blocks (2 KB), B one data
                        // row (16 bytes) per step.  The start-address field (16-byte units) of
                        // an address below 256 KB never carries out of its 14 bits.
                        const uint32_t late = 16 * j < k_first ? 1u : 0u;
                        const uint32_t n = ((k_end - 16 * j + TC_Q - 1) >> 7) - late;
                        uint32_t a = a0 + 16 * j + late * TC_Q;
                        uint32_t b = b_base + slot * b_slot + (j & 1 ? b_pair : 0u) + late;
#pragma unroll 1
                        for (uint32_t i = 0; i < n; i++) {
                            if (one) {
                                if (SMALL) {
                                    mma_f16(dt, a, a_hi, b + b_low, b_hi, idesc, acc);
                                    mma_f16(dt, a + a_low, a_hi, b, b_hi, idesc, 1);
                                } else {
                                    mma_f16(dt, a, a_hi, b, b_hi, idesc, acc);
                                }
                            }
                            acc = 1;
                            a += TC_Q;
                            b += 1;
                        }
                        const bool done = --left == 0 || (!SMALL && j == TC_CB / 2 - 1 && phi == step - 1);
                        if (one) {
                            if (j & 1)
                                mma_commit(bar + T32Bars::dempty + 8 * slot);
                            if (done)
                                mma_commit(bar + (SMALL ? T32Bars::sfull : T32Bars::hfull) + 8 * (acc_i & 1));
                        }
                        if ((j & 1) && ++slot == n_rows) {
                            slot = 0;
                            turn++;
                        }
                        if (done) {
                            acc_i++;
                            left = 0;
                        }
                    }
                    if (one)
                        mma_commit(bar + T32Bars::wempty + 8 * wb);
                }
            }
        }
    }
}

// VAR: per-channel template lengths (Fisher-z network sum); FULL: 'full'
// normalisation; NSUM: network sum.  One instantiation per mode, each with its
// own epilogue code only (the code of all roles shares the instruction cache).
template <bool VAR, bool FULL, bool NSUM>
__global__ void __launch_bounds__(T32_THREADS, 1) tc32_persistent(const __grid_constant__ TcBatch B)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int CH = tc32_stat_columns(FULL);  // columns per slot of statistics and half tile
    constexpr uint32_t kStatHalf = tc32_stat_half(FULL);

    // template blocks (2 buffers), data slots, statistics slots, barriers
    const uint32_t w_base = smem_u32(smem);
    const uint32_t d_base = w_base + 2u * B.w_bytes;
    const uint32_t e_base = d_base + (uint32_t)B.n_rows * B.row_bytes;
    uint8_t *bar_ptr = smem + 2u * B.w_bytes + (uint32_t)B.n_rows * B.row_bytes + ((uint32_t)B.stat_bytes << B.stat_log2);
    const uint32_t bar = smem_u32(bar_ptr);
    long long *ring = reinterpret_cast<long long *>(bar_ptr + T32Bars::items);  // 4 item slots
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bar_ptr + T32Bars::tmem);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(bar_ptr + T32Bars::abort);
    const int n_rows = B.n_rows, stat_log2 = B.stat_log2;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; i++) {
            mbar_init(bar + T32Bars::wfull + 8 * i, 1);
            mbar_init(bar + T32Bars::wempty + 8 * i, 2);  // one commit per MMA issuer
            mbar_init(bar + T32Bars::hfull + 8 * i, 1);
            mbar_init(bar + T32Bars::hempty + 8 * i, T32_EPI_WARPS);
            mbar_init(bar + T32Bars::sfull + 8 * i, 1);
            mbar_init(bar + T32Bars::sempty + 8 * i, T32_EPI_WARPS);
        }
        for (int i = 0; i < T32_MAX_ROWS; i++) {
            mbar_init(bar + T32Bars::dfull + 8 * i, 1);
            mbar_init(bar + T32Bars::dempty + 8 * i, 2);
        }
        for (int i = 0; i < T32_MAX_STATS; i++) {
            mbar_init(bar + T32Bars::efull + 8 * i, 1);
            mbar_init(bar + T32Bars::eempty + 8 * i, T32_EPI_WARPS);
        }
        mbar_init(bar + T32Bars::fin, 2);
        for (int i = 0; i < 4; i++) {
            mbar_init(bar + T32Bars::ifull + 8 * i, 1);
            mbar_init(bar + T32Bars::iempty + 8 * i, 3 + T32_EPI_WARPS);  // issuers, warp 3, epilogue
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    constexpr uint32_t TMEM_COLS = 512;  // H0, H1, S0, S1 at columns 0, 128, 256, 384
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_holder)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_holder;
    const long long total = B.total_items;

    if (warp < 4) {
        // registers: 384 threads x 168 at launch = 128 x 88 + 256 x 208
        asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    }
    if (warp == 0) {
        // ---------------------------------------------------------- tile queue, operands
        int stages = 0;                 // (channel, phase) stages so far; template buffer = stages & 1
        int slot = 0, turn = 0;         // data slot, times round the ring
        bool ok = true;
        for (long long q = 0; ok; q++) {
            const int is = (int)(q & 3);
            long long item = total;
            if (lane == 0) {
                const bool got = q < 4 || mbar_wait(bar + T32Bars::iempty + 8 * is, (uint32_t)(((q >> 2) - 1) & 1),
                                                    abort_flag, B.err, 1u);
                if (got && !*abort_flag)
                    item = (long long)atomicAdd(B.queue, 1ull);
                ring[is] = item;
                mbar_arrive(bar + T32Bars::ifull + 8 * is);
            }
            item = __shfl_sync(0xffffffffu, item, 0);
            if (item >= total)
                break;
            int p, tile, t, c_begin, c_end, part;
            decode_item<true>(B, item, p, tile, t, c_begin, c_end, part);
            const TcProb &pr = B.prob[p];
            const Problem &P = pr.P;
            const long long I0 = (long long)tile * TC_Q * pr.nb;
            if (!tc32_busy(pr, I0, t))
                continue;
            const int SC = P.SC, step = P.step;
            const uint32_t col_bytes = (uint32_t)pr.R * 16, wbytes = (uint32_t)pr.NW * 128;
            const size_t row0 = (size_t)t * SC;
            for (int g0 = c_begin; ok && g0 < c_end; g0 += 32) {
                // the scalars of 32 channels, one per lane
                const int cl = min(g0 + lane, c_end - 1);
                const int mo_l = P.mo[row0 + cl];
                uint32_t active = __ballot_sync(0xffffffffu, g0 + lane < c_end && P.w[row0 + cl] != 0.0f);
                for (; ok && active; active &= active - 1) {
                    const int from = __ffs(active) - 1, ch = g0 + from;
                    const int mo = __shfl_sync(0xffffffffu, mo_l, from);
                    for (int phi = 0; ok && phi < step; phi++, stages++) {
                        const int wb = stages & 1;
                        int psi;
                        const int mu = tc32_phase(mo + phi, step, psi);
                        const long long r0 = ((I0 + mu) >> 7) + pr.row_front;  // floor
                        const uint32_t wbar = bar + T32Bars::wfull + 8 * wb;
                        if (stages >= 2 && !mbar_wait_warp(bar + T32Bars::wempty + 8 * wb, ((stages >> 1) - 1) & 1,
                                                           abort_flag, B.err, 2u)) {
                            ok = false;
                            break;
                        }
                        if (lane == 0)
                            mbar_expect_tx(wbar, 2u * wbytes);
                        __syncwarp();
                        if (lane < 2)
                            bulk_g2s(w_base + wb * B.w_bytes + lane * wbytes,
                                     (lane ? pr.w_lo : pr.w_hi) + ((row0 + ch) * step + phi) * pr.NW * 64, wbytes, wbar);
                        // data: four column blocks of the R rows, both halves, per slot; lane =
                        // 4 * half + block
                        const uint16_t *src =
                            (lane & 4 ? pr.g_lo : pr.g_hi) +
                            ((((long long)ch * step + psi) * TC_CB + (lane & 3)) * pr.rows_total + r0) * 8;
                        const long long src_step = 4ll * pr.rows_total * 8;
#pragma unroll 1
                        for (int j = 0; j < TC_CB / 4; j++, src += src_step) {
                            const uint32_t dbar = bar + T32Bars::dfull + 8 * slot;
                            if (turn >= 1 && !mbar_wait_warp(bar + T32Bars::dempty + 8 * slot, (turn - 1) & 1,
                                                             abort_flag, B.err, 2u)) {
                                ok = false;
                                break;
                            }
                            if (lane == 0)
                                mbar_expect_tx(dbar, 8u * col_bytes);
                            __syncwarp();
                            if (lane < 8)
                                bulk_g2s(d_base + slot * B.row_bytes + lane * col_bytes, src, col_bytes, dbar);
                            if (++slot == n_rows) {
                                slot = 0;
                                turn++;
                            }
                        }
                    }
                }
            }
        }
        // do not leave with copies in flight: the last use of every buffer
        if (lane == 0) {
            for (int u = stages < 2 ? 0 : stages - 2; u < stages; u++)
                mbar_wait(bar + T32Bars::wfull + 8 * (u & 1), (u >> 1) & 1, abort_flag, B.err, 0u);
            for (int i = 0; i < n_rows; i++) {
                const int uses = turn + (i < slot ? 1 : 0);
                if (uses)
                    mbar_wait(bar + T32Bars::dfull + 8 * i, (uses - 1) & 1, abort_flag, B.err, 0u);
            }
        }
        __syncwarp();
    } else if (warp == 1 || warp == 2) {
        // ---------------------------------------------------------- MMA issuers
        // One thread each; the code of one instruction costs the tensor pipe as much time as
        // the instruction, so each issuer has its own short loop and moves only the low
        // words of its descriptors.
        const bool one = elect_one();
        if (warp == 1)
            tc32_issue<VAR, false>(B, ring, bar, w_base, d_base, tmem, abort_flag, one);
        else
            tc32_issue<VAR, true>(B, ring, bar, w_base, d_base, tmem, abort_flag, one);
        __syncwarp();
        if (one) {
            mma_commit(bar + T32Bars::fin);
            mbar_wait(bar + T32Bars::fin, 0, abort_flag, B.err, 0u);
        }
        __syncwarp();
    } else if (warp == 3) {
        // ---------------------------------------------------------- window statistics
        // Slot e: CH columns of each half of the tile (a column is 128 windows, contiguous
        // in the statistics of the channel's stream), copied from a 16-byte boundary.
        {
            int ec = 0;
            bool ok = true;
            for (long long q = 0; ok; q++) {
                const int is = (int)(q & 3);
                if (!mbar_wait_warp(bar + T32Bars::ifull + 8 * is, (uint32_t)((q >> 2) & 1), abort_flag, B.err, 32u))
                    break;
                const long long item = ring[is];
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(bar + T32Bars::iempty + 8 * is);
                if (item >= total)
                    break;
                if (VAR)
                    continue;
                int p, tile, t, c_begin, c_end, part;
                decode_item<true>(B, item, p, tile, t, c_begin, c_end, part);
                const TcProb &pr = B.prob[p];
                const Problem &P = pr.P;
                const long long I0 = (long long)tile * TC_Q * pr.nb;
                if (!tc32_busy(pr, I0, t))
                    continue;
                const int nc = pr.nb / 2;
                const size_t row0 = (size_t)t * P.SC;
                for (int g0 = c_begin; ok && g0 < c_end; g0 += 32) {
                    const int cl = min(g0 + lane, c_end - 1);
                    const int mo_l = P.mo[row0 + cl];
                    uint32_t active = __ballot_sync(0xffffffffu, g0 + lane < c_end && P.w[row0 + cl] != 0.0f);
                    for (; ok && active; active &= active - 1) {
                        const int from = __ffs(active) - 1, ch = g0 + from;
                        int psi;  // phase 0: the moveout's own stream
                        const int mu = tc32_phase(__shfl_sync(0xffffffffu, mo_l, from), P.step, psi);
                        constexpr int kAlign = FULL ? 1 : 3;
                        const long long x0 = (I0 + mu) & ~(long long)kAlign;
                        const char *src = reinterpret_cast<const char *>(P.stat_e) +
                                          (ch * P.stat_ch + psi * P.stat_ps + x0) * (FULL ? 8 : 4);
                        for (int c0 = 0; c0 < nc; c0 += CH, ec++) {
                            const int es = ec & ((1 << stat_log2) - 1);
                            const uint32_t ebar = bar + T32Bars::efull + 8 * es;
                            if ((ec >> stat_log2) >= 1 &&
                                !mbar_wait_warp(bar + T32Bars::eempty + 8 * es, ((ec >> stat_log2) - 1) & 1,
                                                abort_flag, B.err, 2u)) {
                                ok = false;
                                break;
                            }
                            const uint32_t bytes = min(CH, nc) * TC_Q * (FULL ? 8 : 4) + 16;
                            if (lane == 0)
                                mbar_expect_tx(ebar, 2u * bytes);
                            __syncwarp();
                            if (lane < 2)  // the two halves of the tile
                                bulk_g2s(e_base + es * (uint32_t)B.stat_bytes + lane * kStatHalf,
                                         src + (size_t)(lane * nc + c0) * TC_Q * (FULL ? 8 : 4), bytes, ebar);
                        }
                    }
                }
            }
            for (int i = 0; i < (1 << stat_log2); i++) {  // the last use of every slot
                const int uses = (ec >> stat_log2) + (i < (ec & ((1 << stat_log2) - 1)) ? 1 : 0);
                if (uses && lane == 0)
                    mbar_wait(bar + T32Bars::efull + 8 * i, (uses - 1) & 1, abort_flag, B.err, 0u);
            }
        }
        __syncwarp();
    } else {
        // ---------------------------------------------------------- epilogue
        // Warp w reads TMEM lane quarter w % 4 (rows 32*(w%4) + lane) and its half of the
        // columns; numerators and network sums of its outputs live in registers.
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        constexpr int NCM = TC_NB_MAX / 2;  // columns per thread, at most
        const int quarter = warp & 3;
        const int cgroup = (warp - 4) >> 2;
        const int b = TC_Q - 1 - (32 * quarter + lane);  // phase of this thread's row
        const uint32_t lane_base = tmem + ((uint32_t)(32 * quarter) << 16);
        int c = 0, hc = 0, ec = 0;  // channels, chains and statistics slots used
        for (long long q = 0;; q++) {
            const int is = (int)(q & 3);
            long long item = total;
            if (lane == 0) {
                if (mbar_wait(bar + T32Bars::ifull + 8 * is, (uint32_t)((q >> 2) & 1), abort_flag, B.err, 64u)) {
                    item = ring[is];
                    mbar_arrive(bar + T32Bars::iempty + 8 * is);
                }
            }
            item = __shfl_sync(0xffffffffu, item, 0);
            if (item >= total)
                break;
            int p, tile, t, c_begin, c_end, part;
            decode_item<true>(B, item, p, tile, t, c_begin, c_end, part);
            const TcProb &pr = B.prob[p];
            if (*pr.skip)
                continue;
            const int nb = pr.nb;
            const int NC = nb / 2;  // columns of this thread (16, 32 or 64)
            const int a0 = cgroup * NC;
            const int SC = pr.P.SC, step = pr.P.step, n_corr = pr.P.n_corr;
            const long long I0 = (long long)tile * TC_Q * nb;
            const int klo = pr.P.k_lo[t], khi = pr.P.k_hi[t];
            const bool busy = I0 < khi && I0 + (long long)TC_Q * nb > klo;
            // valid lag blocks of this thread: klo <= I0 + Q*a + b < khi
            const long long kb = I0 + b;
            const int a_lo = (int)max(0LL, (klo - kb + TC_Q - 1) / TC_Q) - a0;
            const int a_hi = (int)min((long long)nb, (khi - kb + TC_Q - 1) / TC_Q) - a0;
            const long long k0 = kb + (long long)TC_Q * a0;  // this thread's first output
            float sum[NCM];
#pragma unroll
            for (int i = 0; i < NCM; i++)
                sum[i] = 0.0f;
            const size_t row0 = (size_t)t * SC;
            const int n_chains = (step * (TC_CB / 2) + pr.chain_cols - 1) / pr.chain_cols;
            for (int g0 = c_begin; busy && g0 < c_end; g0 += 32) {
                // the scalars of 32 channels, one per lane
                const int cl = min(g0 + lane, c_end - 1);
                const float w_l = g0 + lane < c_end ? pr.P.w[row0 + cl] : 0.0f, sst_l = pr.P.sst[row0 + cl];
                const int mo_l = pr.P.mo[row0 + cl];
                // 2^unit: the product of the operands' scales
                const int unit_l = pr.t_exp[row0 + cl] + pr.d_exp[cl] - 2 * kTopExp;
                const float ts_l = FULL ? pr.P.tsum[row0 + cl] * exp2_int(-unit_l) : 0.0f;
                uint32_t active = __ballot_sync(0xffffffffu, w_l != 0.0f);
#pragma unroll 1
                for (; active; active &= active - 1) {
                    const int from = __ffs(active) - 1, ch = g0 + from;
                    [[maybe_unused]] const size_t row = row0 + ch;
                    const float wc = __shfl_sync(0xffffffffu, w_l, from), sst = __shfl_sync(0xffffffffu, sst_l, from);
                    const float unit = exp2_int(__shfl_sync(0xffffffffu, unit_l, from));
                    const float ts = FULL ? __shfl_sync(0xffffffffu, ts_l, from) : 0.0f;
                    const int mo = __shfl_sync(0xffffffffu, mo_l, from);
                    float num[NCM];
#pragma unroll
                    for (int i = 0; i < NCM; i++)
                        num[i] = 0.0f;
                    // numerators: the chains' sums, then S 2^-11
#pragma unroll 1
                    for (int j = 0; j <= n_chains; j++) {
                        const bool last = j == n_chains;
                        const int u = last ? c : hc;
                        if (!mbar_wait_all(bar + (last ? T32Bars::sfull : T32Bars::hfull) + 8 * (u & 1), (u >> 1) & 1,
                                           abort_flag, B.err, 16u))
                            goto epilogue_done;
                        tc_fence_after();
                        const uint32_t h = lane_base + (last ? 256u : 0u) + 128u * (u & 1) + a0;
                        const float f = last ? 1.0f / kLoScale : 1.0f;  // powers of two: exact products
#pragma unroll
                        for (int c0 = 0; c0 < NCM; c0 += 32) {  // a tile of 16 columns reads 16 too many
                            if (c0 < NC) {
                                float x[32];
                                tmem_ld32(h + c0, x);
                                tmem_wait_ld();
#pragma unroll
                                for (int i = 0; i < 32; i++)
                                    num[c0 + i] = fmaf(x[i], f, num[c0 + i]);
                            }
                        }
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0)
                            mbar_arrive(bar + (last ? T32Bars::sempty : T32Bars::hempty) + 8 * (u & 1));
                        if (!last)
                            hc++;
                    }
                    const float wu = wc * unit;  // a power of two: cc * wc rounds the same
                    float *oc = pr.P.out + ((size_t)t * n_corr + k0) * SC + ch;
                    if constexpr (VAR) {
                        // window sums of the channel's own length from its running sums, the
                        // threshold on the square root, atanh(cc - 10 eps) * z
                        const bool any = a_hi > a_lo;
                        const int qs32 = TC_Q * step;
                        const long long u0 = k0 * step + mo;
                        const int ntap = pr.P.ntap[row];
                        const float zw = pr.P.zweight[row], u2 = pr.P.unit2[ch];
                        const float nf = (float)ntap, inv_n = 1.0f / nf;
                        const long long *__restrict__ pf = pr.P.pre2q + (size_t)ch * (pr.P.N + 1) + u0;
                        const float2 *__restrict__ pg =
                            FULL ? pr.P.pre1f + (size_t)ch * (pr.P.N + 1) + u0 : nullptr;
#pragma unroll
                        for (int h4 = 0; h4 < NCM; h4 += 4) {  // loads of 4 values, then their use
                            if (h4 < NC) {
                                long long lo[4], hi[4];
                                float2 lo1[4], hi1[4];
#pragma unroll
                                for (int j = 0; j < 4; j++) {
                                    const int o = min(max(h4 + j, a_lo), a_hi - 1) * qs32;  // a valid lag
                                    lo[j] = any ? pf[o] : 0;
                                    hi[j] = any ? pf[o + ntap] : 0;
                                    if constexpr (FULL) {
                                        lo1[j] = any ? pg[o] : make_float2(0.0f, 0.0f);
                                        hi1[j] = any ? pg[o + ntap] : make_float2(0.0f, 0.0f);
                                    }
                                }
#pragma unroll
                                for (int j = 0; j < 4; j++) {
                                    const int a = h4 + j;
                                    float ssd, num1 = num[a];
                                    if constexpr (FULL) {
                                        float mean;
                                        window_centred(lo[j], hi[j], u2, lo1[j], hi1[j], nf, inv_n, ssd, mean);
                                        num1 = fmaf(-mean, ts, num1);
                                    } else {
                                        ssd = window_energy(lo[j], hi[j], u2);
                                    }
                                    const float pe = sst * ssd, r = rsqrt_ftz(pe);
                                    const float cc = pe * r > kThreshold ? num1 * (r * unit) : 0.0f;
                                    sum[a] = fmaf(fisher_atanh(cc - 10.0f * FLT_EPSILON), zw, sum[a]);
                                }
                            }
                        }
                    } else {
                        int psi;
                        const int mu = tc32_phase(mo, step, psi);
                        const int head = (int)((I0 + mu) & (FULL ? 1 : 3));  // past the 16-byte boundary
#pragma unroll
                        for (int c0 = 0; c0 < NCM; c0 += CH) {
                            if (c0 < NC) {
                                const int es = ec & ((1 << stat_log2) - 1);
                                if (!mbar_wait_all(bar + T32Bars::efull + 8 * es, (ec >> stat_log2) & 1, abort_flag,
                                                   B.err, 16u))
                                    goto epilogue_done;
                                const uint8_t *at = smem + (e_base - w_base) + es * (uint32_t)B.stat_bytes +
                                                    cgroup * kStatHalf + (head + b) * (FULL ? 8 : 4);
                                constexpr int CB = 16;  // values in flight
#pragma unroll
                                for (int h0 = 0; h0 < CH; h0 += CB) {
                                    if (c0 + h0 < NC) {
                                        float e[CB], mm[CB];
#pragma unroll
                                        for (int i = 0; i < CB; i++) {
                                            if constexpr (FULL) {
                                                const float2 v = *reinterpret_cast<const float2 *>(at + (h0 + i) * TC_Q * 8);
                                                e[i] = v.x;
                                                mm[i] = v.y;
                                            } else {
                                                e[i] = *reinterpret_cast<const float *>(at + (h0 + i) * TC_Q * 4);
                                            }
                                        }
                                        if (h0 + CB >= CH || c0 + h0 + CB >= NC) {  // the slot is read
                                            fence_reads_before_copy();
                                            __syncwarp();
                                            if (lane == 0)
                                                mbar_arrive(bar + T32Bars::eempty + 8 * es);
                                        }
#pragma unroll
                                        for (int i = 0; i < CB; i++) {
                                            const int a = c0 + h0 + i;
                                            const float num1 = FULL ? fmaf(-mm[i], ts, num[a]) : num[a];
                                            const float den = sst * e[i];
                                            // den is normal where it passes; outside the valid lags the
                                            // statistics, and with them cc, are anything
                                            const float cc = den > kThreshold ? num1 * rsqrt_ftz(den) : 0.0f;
                                            if (NSUM)
                                                sum[a] = fmaf(cc, wu, sum[a]);
                                            else if (a >= a_lo && a < a_hi)
                                                oc[(size_t)a * TC_Q * SC] = cc * unit;
                                        }
                                    }
                                }
                                ec++;
                            }
                        }
                    }
                    c++;
                }
            }
            if (NSUM) {
                // a channel part writes its partial sums to its own plane of part_out
                const bool parts = pr.parts > 1;
                float *o = (parts ? pr.part_out + (size_t)part * pr.P.T * n_corr : pr.P.out) +
                           (size_t)t * n_corr + k0;
                const long long lim = n_corr - k0;
                float zn = 1.0f, zb = 0.0f, zs = 1.0f;
                if (VAR && !parts) {
                    zn = pr.P.vp_norm[t];
                    zb = pr.P.vp_bias[t];
                    zs = pr.P.vp_scale[t];
                }
#pragma unroll
                for (int a = 0; a < NCM; a++) {
                    if (a < NC && (long long)a * TC_Q < lim) {
                        float v = busy && a >= a_lo && a < a_hi ? sum[a] : 0.0f;
                        if (VAR && !parts)  // the Fisher-z transform of every output
                            v = (tanhf(v / zn) + zb) * zs;
                        o[(size_t)a * TC_Q] = v;
                    }
                }
            }
        }
    epilogue_done:;
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS)
                     : "memory");
    }
}

// ------------------------------------------------------------------ host side
struct Tc32Search {
    TcProb pr;        // of all templates; w_* hold `room` templates
    int room, parts;
    uint16_t *w;
    size_t w_elems;   // of one half, all room templates
};

size_t tc32_search_size() { return sizeof(Tc32Search); }

// Operand blocks of one chunk of templates take at most this much memory.
constexpr size_t kMaxTemplateBytes = (size_t)4 << 30;

// Lag blocks per tile of an FP32 search on the tensor cores, or 0: the CUDA cores.
int tc32_choose_nb(size_t T, size_t SC, size_t L, size_t step, size_t n_corr)
{
    if (const char *env = getenv("FMF_TC32")) {
        if (atoi(env) == 0)
            return 0;
        if (atoi(env) > 1)
            return tc_choose_nb((int)L, (int)step, 1, atoi(env));
    }
    // CUDA cores: microseconds of the busiest SM, a tile of 4,096 outputs at a time
    const double taps = (double)step * (double)((((L + step - 1) / step + 19) / 20) * 20);
    const double tiles = (double)T * (double)((n_corr + 4095) / 4096);
    const double waves = tiles <= 304.0 ? 1.0 : tiles / 304.0;
    const double plain_us = waves * (double)SC * (taps * 0.02 + (double)step * 0.5 + 0.5);
    if (plain_us < 60.0)
        return 0;
    const int want = n_corr > 8192 ? 128 : (n_corr > 4096 ? 64 : 32);
    for (int nb = want; nb >= 32; nb >>= 1) {
        const int fit = tc_choose_nb((int)L, (int)step, 1, nb);
        if (fit)
            return fit;
    }
    return 0;
}

// Data streams and room for the operand blocks of P's templates (or of a part
// of them, taken in turn).  P.scan must be set.
int tc32_begin(const Problem &P, int nb, int tg, int max_templates, Scratch &ws, cudaStream_t s,
               Tc32Search *out)
{
    int rc;
    const int step = P.step, SC = P.SC;
    TcProb &pr = out->pr;
    const TcShape g = tc_fill_shape(P, 1, nb, tg, &pr);
    const size_t per_template = (size_t)SC * step * g.NW * 64;  // one half
    size_t room = kMaxTemplateBytes / (4 * per_template);
    room = room < 1 ? 1 : room;
    room = room < (size_t)max_templates ? room : (size_t)max_templates;
    const size_t g_elems = (size_t)SC * step * TC_CB * pr.rows_total * 8;
    const size_t n_rows = (size_t)P.T * SC;
    out->room = (int)room;
    out->w_elems = room * per_template;
    out->parts = tc_choose_parts(&pr);
    uint16_t *g_hi = nullptr;
    int *meta = nullptr;
    if ((rc = ws.get(&g_hi, 2 * g_elems, "fp16 data streams")) ||
        (rc = ws.get(&out->w, 2 * out->w_elems, "fp16 template blocks")) ||
        (rc = ws.get(&meta, n_rows + SC, "operand exponents")))
        return rc;
    pr.g_hi = g_hi;
    pr.g_lo = g_hi + g_elems;
    pr.w_hi = out->w;
    pr.w_lo = out->w + out->w_elems;
    pr.t_exp = meta;
    pr.d_exp = pr.t_exp + n_rows;
    // chains of whole column-block pairs, at most kChain K steps where a pair has no more
    const int most = (g.k_span + TC_Q - 1) / TC_Q;  // K steps of one pair
    pr.chain_cols = kChain / most > 1 ? kChain / most : 1;
    pr.skip = P.scan + 3 * SC;
    const long long n = (long long)SC * step * TC_CB * pr.rows_total;
    tc32_data_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(
        P.data, P.N, SC, step, pr.rows_total, pr.row_front, P.scan, g_hi, g_hi + g_elems,
        const_cast<int *>(pr.d_exp), P.scan + 3 * SC);
    count_launch();
    return check_launch("FP32 tensor-core data streams");
}

// Operand blocks of templates [t0, t0 + nt), nt <= room, into the search's
// buffer; *sub is that part of the search.
int tc32_templates(const Tc32Search *full, int t0, int nt, cudaStream_t s, TcProb *sub)
{
    const Problem &P = full->pr.P;
    tc_subset(&full->pr, t0, nt, sub);
    sub->w_hi = full->w;
    sub->w_lo = full->w + full->w_elems;
    cudaError_t e = cudaFuncSetAttribute(tc32_template_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kMaxDynamicSmem - 1024);
    if (e != cudaSuccess)
        return set_error(FMF_ERR_CUDA, "tc32_template_kernel shared memory: %s", cudaGetErrorString(e));
    tc32_template_kernel<<<(unsigned)((size_t)nt * P.SC), 256, (size_t)P.L * sizeof(float), s>>>(
        sub->P.tpl, sub->P.mo, P.L, P.step, sub->NW, full->w, full->w + full->w_elems,
        const_cast<int *>(sub->t_exp),
        P.scan + 3 * P.SC);
    count_launch();
    return check_launch("FP32 tensor-core templates");
}

// Templates [t0, t0 + nt) of a begun search: their operand blocks and the
// persistent launch, a roomful at a time.
int tc32_run(const Tc32Search *full, int t0, int nt, unsigned *err, Scratch &ws, cudaStream_t s)
{
    int rc;
    for (int a = t0; a < t0 + nt; a += full->room) {
        const int n = t0 + nt - a < full->room ? t0 + nt - a : full->room;
        TcProb sub;
        unsigned long long *queue = nullptr;
        if ((rc = tc32_templates(full, a, n, s, &sub)) || (rc = ws.get(&queue, 1, "tile queue")) ||
            (rc = tc_run(&sub, 1, TC_FORM_FP32, full->parts, queue, err, s)))
            return rc;
    }
    return FMF_OK;
}

const unsigned *tc32_flag(const Tc32Search *full) { return full->pr.skip; }

// One search of a batch: all its operands; *out is ready for a shared launch.
int tc32_prepare(const Problem &P, int nb, int tg, Scratch &ws, cudaStream_t s, TcProb *out)
{
    Tc32Search st;
    int rc = tc32_begin(P, nb, tg, P.T, ws, s, &st);
    if (rc)
        return rc;
    if (st.room < P.T)
        return set_error(FMF_ERR_OOM, "template blocks of a batched search exceed %zu bytes", kMaxTemplateBytes);
    return tc32_templates(&st, 0, P.T, s, out);
}

// Shared memory of one launch: two template buffers, two statistics slots (32 KB
// each: half a channel of a full tile) and as many data slots as fit (a channel
// has 4); long templates give up a statistics slot first.
size_t tc32_layout(TcBatch *B, bool var, bool full)
{
    const size_t fixed = 2 * (size_t)B->w_bytes + T32Bars::bytes;
    B->stat_bytes = 2 * (int)tc32_stat_half(full);
    for (int least = 3; least >= 2; least--)
        for (int k = 1; k >= 0; k--) {
            B->stat_log2 = var ? 0 : k;
            const size_t stats = var ? 0 : (size_t)B->stat_bytes << B->stat_log2;
            if (fixed + stats > (size_t)kMaxDynamicSmem)
                continue;
            const size_t rows = (kMaxDynamicSmem - fixed - stats) / B->row_bytes;
            B->n_rows = rows < (size_t)T32_MAX_ROWS ? (int)rows : T32_MAX_ROWS;
            if (B->n_rows >= least) {
                if (var)
                    B->stat_bytes = 0;
                const size_t smem = fixed + stats + (size_t)B->n_rows * B->row_bytes;
                return smem < 120 * 1024 ? 120 * 1024 : smem;  // one CTA per SM: its TMEM is all there is
            }
        }
    return 0;
}

int tc32_launch(const TcBatch &B, bool var, bool full, unsigned grid, size_t smem, cudaStream_t s)
{
    void (*kern)(const TcBatch);
    if (var)
        kern = full ? tc32_persistent<true, true, true> : tc32_persistent<true, false, true>;
    else if (B.prob[0].P.network_sum)
        kern = full ? tc32_persistent<false, true, true> : tc32_persistent<false, false, true>;
    else
        kern = full ? tc32_persistent<false, true, false> : tc32_persistent<false, false, false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
    if (e != cudaSuccess)
        return set_error(FMF_ERR_CUDA, "tc32_persistent shared memory (%zu bytes): %s", smem,
                         cudaGetErrorString(e));
    kern<<<grid, T32_THREADS, smem, s>>>(B);
    count_launch();
    return check_launch("tc32_persistent");
}

}  // namespace fmf
