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
// times over).  Also the phases' moveouts and streams, the channel's exponent
// and its K steps.
__global__ void __launch_bounds__(256) tc32_template_kernel(
    const float *__restrict__ tpl, const int *__restrict__ mo, const int *__restrict__ ntap, int L,
    int step, int NW, uint16_t *__restrict__ w_hi, uint16_t *__restrict__ w_lo, int *__restrict__ mu_out,
    int *__restrict__ psi_out, int *__restrict__ t_exp, int *__restrict__ k_steps, unsigned *skip)
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
        int steps = 0;
        for (int phi = 0; phi < step; phi++) {
            const int m = m0 + phi;
            const int mu = m >= 0 ? m / step : -((-m + step - 1) / step);
            const int s = ((mu % TC_Q) + TC_Q) % TC_Q;
            mu_out[row * step + phi] = mu;
            psi_out[row * step + phi] = m - step * mu;
            steps += tc_k_end(s, tc_phase_taps(L, step, phi, ntap ? ntap[row] : L)) - (s & ~15);
        }
        k_steps[row] = steps >> 4;
    }
    const int per_phase = NW * 8;
    for (int i = threadIdx.x; i < step * per_phase; i += blockDim.x) {
        const int phi = i / per_phase, ne = i - phi * per_phase;
        const int m = m0 + phi;
        const int mu = m >= 0 ? m / step : -((-m + step - 1) / step);
        const int s = ((mu % TC_Q) + TC_Q) % TC_Q;
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
// VAR: per-channel template lengths (Fisher-z network sum); FULL: 'full'
// normalisation; one instantiation per mode, each with its own epilogue code.
template <bool VAR, bool FULL>
__global__ void __launch_bounds__(T32_THREADS, 1) tc32_persistent(const __grid_constant__ TcBatch B)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    uint8_t *bar_base = smem + 2 * (size_t)B.stage_bytes;
    const uint32_t full0 = smem_u32(bar_base), empty0 = full0 + 16, hfull0 = full0 + 32, hempty0 = full0 + 48,
                   sfull0 = full0 + 64, sempty0 = full0 + 80, ifull0 = full0 + 96, iempty0 = full0 + 128,
                   fin = full0 + 160;
    long long *ring = reinterpret_cast<long long *>(bar_base + 168);  // 4 item slots
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bar_base + 200);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(bar_base + 204);

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; i++) {
            mbar_init(full0 + 8 * i, 1);
            mbar_init(empty0 + 8 * i, 2);  // one commit per MMA issuer
            mbar_init(hfull0 + 8 * i, 1);
            mbar_init(hempty0 + 8 * i, T32_EPI_WARPS);
            mbar_init(sfull0 + 8 * i, 1);
            mbar_init(sempty0 + 8 * i, T32_EPI_WARPS);
        }
        mbar_init(fin, 2);
        for (int i = 0; i < 4; i++) {
            mbar_init(ifull0 + 8 * i, 1);
            mbar_init(iempty0 + 8 * i, 2 + T32_EPI_WARPS);
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
        // registers: 384 threads x 168 at launch = 128 x 72 + 256 x 216
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    }
    if (warp == 0) {
        // ---------------------------------------------------------- producer + tile queue
        int uses = 0;  // stages loaded so far; buffer = uses & 1
        bool ok = true;
        for (long long q = 0; ok; q++) {
            const int slot = (int)(q & 3);
            long long item = total;
            if (lane == 0) {
                const bool got = q < 4 || mbar_wait(iempty0 + 8 * slot, (uint32_t)(((q >> 2) - 1) & 1),
                                                    abort_flag, B.err, 1u);
                if (got && !*abort_flag)
                    item = (long long)atomicAdd(B.queue, 1ull);
                ring[slot] = item;
                mbar_arrive(ifull0 + 8 * slot);
            }
            item = __shfl_sync(0xffffffffu, item, 0);
            if (item >= total)
                break;
            int p, tile, t, c_begin, c_end, part;
            decode_item<true>(B, item, p, tile, t, c_begin, c_end, part);
            const TcProb &pr = B.prob[p];
            const Problem &P = pr.P;
            const int nb = pr.nb;
            const long long I0 = (long long)tile * TC_Q * nb;
            if (!(I0 < P.k_hi[t] && I0 + (long long)TC_Q * nb > P.k_lo[t]) || *pr.skip)
                continue;
            const int SC = P.SC, step = P.step, R = pr.R, NW = pr.NW;
            const uint32_t data_bytes = (uint32_t)TC_CB * R * 16, wbytes = (uint32_t)NW * 128;
            const float *w = P.w + (size_t)t * SC;
            for (int ch = c_begin; ok && ch < c_end; ch++) {
                if (w[ch] == 0.0f)
                    continue;
                for (int phi = 0; phi < step; phi++) {
                    const int b = uses & 1;
                    const long long meta = ((long long)t * SC + ch) * step + phi;
                    const int mu = pr.mu[meta], psi = pr.psi[meta];
                    const int sres = ((mu % TC_Q) + TC_Q) % TC_Q;
                    const long long r0 = (I0 + mu - sres) / TC_Q + pr.row_front;
                    if (uses >= 2 &&
                        !mbar_wait_warp(empty0 + 8 * b, ((uses >> 1) - 1) & 1, abort_flag, B.err, 2u)) {
                        ok = false;
                        break;
                    }
                    const uint32_t st = smem_u32(smem + (size_t)b * B.stage_bytes);
                    if (lane == 0)
                        mbar_expect_tx(full0 + 8 * b, 2u * (data_bytes + wbytes));
                    __syncwarp();
                    const int cb = lane & 15, hl = lane >> 4;
                    const uint16_t *src = (hl ? pr.g_lo : pr.g_hi) +
                                          ((((long long)ch * step + psi) * TC_CB + cb) * pr.rows_total + r0) * 8;
                    bulk_g2s(st + hl * data_bytes + cb * (uint32_t)R * 16, src, (uint32_t)R * 16,
                             full0 + 8 * b);
                    if (lane < 2) {
                        const uint16_t *wsrc = (lane ? pr.w_lo : pr.w_hi) + meta * NW * 64;
                        bulk_g2s(st + 2 * data_bytes + lane * wbytes, wsrc, wbytes, full0 + 8 * b);
                    }
                    uses++;
                }
            }
        }
        // do not leave with copies in flight
        if (lane == 0)
            for (int u = uses < 2 ? 0 : uses - 2; u < uses; u++)
                mbar_wait(full0 + 8 * (u & 1), (u >> 1) & 1, abort_flag, B.err, 0u);
        __syncwarp();
    } else if (warp == 1 || warp == 2) {
        // ---------------------------------------------------------- MMA issuers
        const bool small = warp == 2;  // the h l and l h products
        if (lane == 0) {
            int used = 0;       // stages consumed
            int c = 0, hc = 0;  // channels and h h chains begun
            for (long long q = 0;; q++) {
                const int slot = (int)(q & 3);
                if (!mbar_wait(ifull0 + 8 * slot, (uint32_t)((q >> 2) & 1), abort_flag, B.err, 32u))
                    goto mma_done;
                const long long item = ring[slot];
                mbar_arrive(iempty0 + 8 * slot);
                if (item >= total)
                    break;
                int p, tile, t, c_begin, c_end, part;
                decode_item<true>(B, item, p, tile, t, c_begin, c_end, part);
                const TcProb &pr = B.prob[p];
                const Problem &P = pr.P;
                const int nb = pr.nb;
                const long long I0 = (long long)tile * TC_Q * nb;
                if (!(I0 < P.k_hi[t] && I0 + (long long)TC_Q * nb > P.k_lo[t]) || *pr.skip)
                    continue;
                // kind::f16 descriptor: F32 accumulate, FP16 A and B, K-major, N = nb, M = 128
                const uint32_t idesc = (1u << 4) | ((uint32_t)(nb >> 3) << 17) | ((uint32_t)(TC_Q >> 4) << 24);
                const int SC = P.SC, step = P.step;
                const uint32_t data_bytes = (uint32_t)TC_CB * pr.R * 16, wbytes = (uint32_t)pr.NW * 128;
                const uint32_t lbo_b = (uint32_t)pr.R * 16;
                const uint64_t a_lo = wbytes >> 4, b_lo = data_bytes >> 4;
                const uint64_t b_step = (2u * lbo_b) >> 4;
                const float *w = P.w + (size_t)t * SC;
                for (int ch = c_begin; ch < c_end; ch++) {
                    if (w[ch] == 0.0f)
                        continue;
                    uint32_t acc = 0, dt = 0;
                    int left = 0;  // K steps left in the current chain
                    if (small) {
                        if (c >= 2 &&
                            !mbar_wait(sempty0 + 8 * (c & 1), ((c >> 1) - 1) & 1, abort_flag, B.err, 4u))
                            goto mma_done;
                        tc_fence_after();
                        dt = tmem + 256u + 128u * (c & 1);
                    }
                    for (int phi = 0; phi < step; phi++, used++) {
                        const int s = used & 1;
                        if (!mbar_wait(full0 + 8 * s, (used >> 1) & 1, abort_flag, B.err, 8u))
                            goto mma_done;
                        tc_fence_after();
                        const long long meta = ((long long)t * SC + ch) * step + phi;
                        const int mu = pr.mu[meta];
                        const int sres = ((mu % TC_Q) + TC_Q) % TC_Q;
                        const int taps = tc_phase_taps(P.L, step, phi, VAR ? P.ntap[(size_t)t * SC + ch] : P.L);
                        const int k_first = sres & ~15, k_end = tc_k_end(sres, taps);
                        const uint32_t zhi = smem_u32(smem + (size_t)s * B.stage_bytes);
                        const uint32_t whi = zhi + 2u * data_bytes;
                        // descriptors advance by additions, as in fmf_tc.cu
                        uint64_t ah = sdesc(whi + (uint32_t)(k_first >> 3) * 128u, 128, 128);
                        const uint64_t b0 = sdesc(zhi, lbo_b, 128);
                        int k = k_first;
                        while (k < k_end) {
                            const int blk_end = min(k_end, (k & ~(TC_Q - 1)) + TC_Q);
                            uint64_t bh = b0 + (((uint32_t)((k & (TC_Q - 1)) >> 3) * lbo_b +
                                                 (uint32_t)(k / TC_Q) * 16u) >> 4);
                            for (; k < blk_end; k += 16) {
                                if (small) {
                                    mma_bf16(dt, ah, bh + b_lo, idesc, acc);
                                    acc = 1;
                                    mma_bf16(dt, ah + a_lo, bh, idesc, 1);
                                } else {
                                    if (left == 0) {  // a chain begins, in the other H accumulator
                                        if (hc >= 2 && !mbar_wait(hempty0 + 8 * (hc & 1), ((hc >> 1) - 1) & 1,
                                                                  abort_flag, B.err, 4u))
                                            goto mma_done;
                                        tc_fence_after();
                                        dt = tmem + 128u * (hc & 1);
                                        acc = 0;
                                        left = kChain;
                                    }
                                    mma_bf16(dt, ah, bh, idesc, acc);
                                    acc = 1;
                                    if (--left == 0) {
                                        mma_commit(hfull0 + 8 * (hc & 1));
                                        hc++;
                                    }
                                }
                                ah += 16;
                                bh += b_step;
                            }
                        }
                        mma_commit(empty0 + 8 * s);
                    }
                    if (small) {
                        mma_commit(sfull0 + 8 * (c & 1));
                    } else if (left > 0) {
                        mma_commit(hfull0 + 8 * (hc & 1));
                        hc++;
                    }
                    c++;
                }
            }
        mma_done:
            mma_commit(fin);
            mbar_wait(fin, 0, abort_flag, B.err, 0u);
        }
        __syncwarp();
    } else if (warp >= 4) {
        // ---------------------------------------------------------- epilogue
        // Warp w reads TMEM lane quarter w % 4 (rows 32*(w%4) + lane) and its half of the
        // columns; numerators and network sums of its outputs live in registers.
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        constexpr int NCM = TC_NB_MAX / 2;  // columns per thread, at most
        constexpr int CH = 16;              // columns per batch of statistics loads
        const int quarter = warp & 3;
        const int cgroup = (warp - 4) >> 2;
        const int b = TC_Q - 1 - (32 * quarter + lane);  // phase of this thread's row
        const uint32_t lane_base = tmem + ((uint32_t)(32 * quarter) << 16);
        int c = 0, hc = 0;  // channels and chains drained
        for (long long q = 0;; q++) {
            const int slot = (int)(q & 3);
            long long item = total;
            if (lane == 0) {
                if (mbar_wait(ifull0 + 8 * slot, (uint32_t)((q >> 2) & 1), abort_flag, B.err, 64u)) {
                    item = ring[slot];
                    mbar_arrive(iempty0 + 8 * slot);
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
            const int SC = pr.P.SC, step = pr.P.step, n_corr = pr.P.n_corr, N = pr.P.N;
            const bool nsum = VAR || pr.P.network_sum != 0;
            const long long I0 = (long long)tile * TC_Q * nb;
            const int klo = pr.P.k_lo[t], khi = pr.P.k_hi[t];
            const bool busy = I0 < khi && I0 + (long long)TC_Q * nb > klo;
            // valid lag blocks of this thread: klo <= I0 + Q*a + b < khi
            const long long kb = I0 + b;
            const int a_lo = (int)max(0LL, (klo - kb + TC_Q - 1) / TC_Q) - a0;
            const int a_hi = (int)min((long long)nb, (khi - kb + TC_Q - 1) / TC_Q) - a0;
            const bool any = busy && a_hi > a_lo;
            const bool interior = __all_sync(0xffffffffu, a_lo <= 0 && a_hi >= NC);
            const int qs32 = TC_Q * step;
            const long long k0 = kb + (long long)TC_Q * a0;  // this thread's first output
            float sum[NCM];
#pragma unroll
            for (int i = 0; i < NCM; i++)
                sum[i] = 0.0f;
            for (int ch = c_begin; busy && ch < c_end; ch++) {
                const size_t row = (size_t)t * SC + ch;
                const float wc = pr.P.w[row];
                if (wc == 0.0f)
                    continue;
                const float sst = pr.P.sst[row];
                const int n_chains = (pr.k_steps[row] + kChain - 1) / kChain;
                // 2^unit: the product of the operands' scales
                const int unit_e = pr.t_exp[row] + pr.d_exp[ch] - 2 * kTopExp;
                const float unit = exp2_int(unit_e);
                const float ts = FULL ? pr.P.tsum[row] * exp2_int(-unit_e) : 0.0f;
                const long long u0 = k0 * step + pr.P.mo[row];
                const float *__restrict__ se = VAR || FULL ? nullptr : pr.P.stat_e + (size_t)ch * N + u0;
                const float2 *__restrict__ sem =
                    VAR || !FULL ? nullptr
                                 : reinterpret_cast<const float2 *>(pr.P.stat_e) + (size_t)ch * N + u0;
                float e[CH], mm[CH];
                auto load_stats = [&](int c0) {  // indices clamped into the valid range
#pragma unroll
                    for (int i = 0; i < CH; i++) {
                        const int o = (interior ? c0 + i : min(max(c0 + i, a_lo), a_hi - 1)) * qs32;
                        if (FULL) {
                            const float2 em = any ? __ldg(sem + o) : make_float2(0.0f, 0.0f);
                            e[i] = em.x;
                            mm[i] = em.y;
                        } else {
                            e[i] = any ? __ldg(se + o) : 0.0f;
                        }
                    }
                };
                float num[NCM];
                for (int j = 0; j < n_chains; j++, hc++) {
                    const uint32_t h = lane_base + 128u * (hc & 1) + a0;
                    if (!mbar_wait_warp(hfull0 + 8 * (hc & 1), (hc >> 1) & 1, abort_flag, B.err, 16u))
                        goto epilogue_done;
                    tc_fence_after();
                    float x[32];
                    if (NC >= 32) {
#pragma unroll
                        for (int c0 = 0; c0 < NCM; c0 += 32) {
                            if (c0 < NC) {
                                tmem_ld32(h + c0, x);
                                tmem_wait_ld();
#pragma unroll
                                for (int i = 0; i < 32; i++)
                                    num[c0 + i] = j == 0 ? x[i] : num[c0 + i] + x[i];
                            }
                        }
                    } else {
                        tmem_ld16(h, x);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; i++)
                            num[i] = j == 0 ? x[i] : num[i] + x[i];
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(hempty0 + 8 * (hc & 1));
                }
                if (!VAR)
                    load_stats(0);
                const uint32_t sc = lane_base + 256u + 128u * (c & 1) + a0;
                if (!mbar_wait_warp(sfull0 + 8 * (c & 1), (c >> 1) & 1, abort_flag, B.err, 16u))
                    goto epilogue_done;
                tc_fence_after();
                const float wu = wc * unit;  // a power of two: cc * wc rounds the same
                float *oc = pr.P.out + ((size_t)t * n_corr + k0) * SC + ch;
#pragma unroll
                for (int c0 = 0; c0 < NCM; c0 += CH) {
                    if (c0 < NC) {
                        float x[CH];
                        tmem_ld16(sc + c0, x);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < CH; i++)
                            x[i] = fmaf(x[i], 1.0f / kLoScale, num[c0 + i]);
                        if (c0 + CH >= NC) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0)
                                mbar_arrive(sempty0 + 8 * (c & 1));
                        }
                        if constexpr (VAR) {
                            // window sums of the channel's own length from its running sums, the
                            // threshold on the square root, atanh(cc - 10 eps) * z
                            const int ntap = pr.P.ntap[row];
                            const float zw = pr.P.zweight[row], u2 = pr.P.unit2[ch];
                            const float nf = (float)ntap, inv_n = 1.0f / nf;
                            const long long *__restrict__ pf = pr.P.pre2q + (size_t)ch * (N + 1) + u0;
                            const float2 *__restrict__ pg =
                                FULL ? pr.P.pre1f + (size_t)ch * (N + 1) + u0 : nullptr;
#pragma unroll
                            for (int h4 = 0; h4 < CH; h4 += 4) {  // loads of 4 values, then their use
                                long long lo[4], hi[4];
                                float2 lo1[4], hi1[4];
#pragma unroll
                                for (int j = 0; j < 4; j++) {
                                    const int o = min(max(c0 + h4 + j, a_lo), a_hi - 1) * qs32;
                                    lo[j] = any ? pf[o] : 0;
                                    hi[j] = any ? pf[o + ntap] : 0;
                                    if constexpr (FULL) {
                                        lo1[j] = any ? pg[o] : make_float2(0.0f, 0.0f);
                                        hi1[j] = any ? pg[o + ntap] : make_float2(0.0f, 0.0f);
                                    }
                                }
#pragma unroll
                                for (int j = 0; j < 4; j++) {
                                    const int a = c0 + h4 + j;
                                    float ssd, num1 = x[h4 + j];
                                    if constexpr (FULL) {
                                        float mean;
                                        window_centred(lo[j], hi[j], u2, lo1[j], hi1[j], nf, inv_n, ssd, mean);
                                        num1 = fmaf(-mean, ts, num1);
                                    } else {
                                        ssd = window_energy(lo[j], hi[j], u2);
                                    }
                                    const float pe = sst * ssd, r = rsqrt_ftz(pe);
                                    const float cc = pe * r > kThreshold ? num1 * (r * unit) : 0.0f;
                                    const float z =
                                        fmaf(fisher_atanh(cc - 10.0f * FLT_EPSILON), zw, sum[a]);
                                    sum[a] = (a >= a_lo && a < a_hi) ? z : sum[a];
                                }
                            }
                        } else {
                            float ec[CH], mc[CH];
#pragma unroll
                            for (int i = 0; i < CH; i++) {
                                ec[i] = e[i];
                                mc[i] = mm[i];
                            }
                            if (c0 + CH < NC)
                                load_stats(c0 + CH);  // the next batch, before this one's use
                            if (nsum && interior) {
#pragma unroll
                                for (int i = 0; i < CH; i++) {
                                    const float num1 = FULL ? fmaf(-mc[i], ts, x[i]) : x[i];
                                    const float den = sst * ec[i];
                                    const float cc = den > kThreshold ? num1 * rsqrtf(den) : 0.0f;
                                    sum[c0 + i] = fmaf(cc, wu, sum[c0 + i]);
                                }
                            } else {
#pragma unroll
                                for (int i = 0; i < CH; i++) {
                                    const int a = c0 + i;
                                    const float num1 = FULL ? fmaf(-mc[i], ts, x[i]) : x[i];
                                    const float den = sst * ec[i];
                                    const float cc = den > kThreshold ? num1 * rsqrtf(den) : 0.0f;
                                    const bool valid = a >= a_lo && a < a_hi;
                                    if (nsum)
                                        sum[a] = valid ? fmaf(cc, wu, sum[a]) : sum[a];
                                    else if (valid)
                                        oc[(size_t)a * TC_Q * SC] = cc * unit;
                                }
                            }
                        }
                    }
                }
                c++;
            }
            if (nsum) {
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
                        float v = sum[a];  // 0 outside the valid lags
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
    const size_t n_rows = (size_t)P.T * SC, n_meta = n_rows * step;
    out->room = (int)room;
    out->w_elems = room * per_template;
    out->parts = tc_choose_parts(&pr);
    uint16_t *g_hi = nullptr;
    int *meta = nullptr;
    if ((rc = ws.get(&g_hi, 2 * g_elems, "fp16 data streams")) ||
        (rc = ws.get(&out->w, 2 * out->w_elems, "fp16 template blocks")) ||
        (rc = ws.get(&meta, 2 * n_meta + 2 * n_rows + SC, "phase moveouts")))
        return rc;
    pr.g_hi = g_hi;
    pr.g_lo = g_hi + g_elems;
    pr.w_hi = out->w;
    pr.w_lo = out->w + out->w_elems;
    pr.mu = meta;
    pr.psi = meta + n_meta;
    pr.t_exp = meta + 2 * n_meta;
    pr.k_steps = pr.t_exp + n_rows;
    pr.d_exp = pr.k_steps + n_rows;
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
        sub->P.tpl, sub->P.mo, sub->P.ntap, P.L, P.step, sub->NW, full->w, full->w + full->w_elems,
        const_cast<int *>(sub->mu), const_cast<int *>(sub->psi), const_cast<int *>(sub->t_exp),
        const_cast<int *>(sub->k_steps), P.scan + 3 * P.SC);
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

TcKernel tc32_kernel(bool var, bool full)
{
    return var ? (full ? tc32_persistent<true, true> : tc32_persistent<true, false>)
               : (full ? tc32_persistent<false, true> : tc32_persistent<false, false>);
}

int tc32_threads() { return T32_THREADS; }

}  // namespace fmf
