// fmf_tc.cu -- the numerators on the tensor cores (tcgen05 / TMEM): the FP32 form
// of searches large enough for it, and the bf16 forms.
//
// Same outputs as the CUDA-core kernel (fmf_plain.cu), which is bound by the
// FP32 FMA pipe; the numerator sum_j t[j]*d[k*step+mo+j] is a Toeplitz x Hankel
// product per channel, laid out so that neither matrix is built in full:
//
//   Output index i = I0 + Q*a + b of one template and channel (I0 a multiple
//   of Q = 128, a = lag block, b = phase in [0, Q)) needs data samples
//   p + Q*a + b + j with p = I0 + mo.  Writing p = Q*r0 + s (0 <= s < Q) and
//   k = s + b + j,
//       X[i] = sum_k A[Q-1-b][k] * B[a][k],
//       A[m][k] = t[k + m - (Q-1+s)]          (template Toeplitz, M = 128 rows)
//       B[a][k] = d[Q*(r0 + a) + k]            (data Hankel, N = NB lag blocks)
//   with K = s + L + Q - 1 (rounded to 16; the leading s & ~15 columns are
//   skipped because they multiply zeros).
//
//   * B is a view of the data stored "column-blocked": per channel, for each
//     16-byte column block cb of a Q-sample row, all rows are contiguous,
//     G[cb][row][8].  In the canonical no-swizzle K-major layout (8-row x
//     16-byte core matrices) rows are then 16 bytes apart, so B for any row
//     offset and any K step is a descriptor (start = cb*R*16 + row*16,
//     leading-dimension offset R*16, stride offset 128) -- no Hankel copy.
//   * A is a view of 8 shifted copies of the template interleaved in
//     128-byte blocks, W[n][e][c] = t[8n + e + c - (Q-1+s)]: core matrix
//     (row group g, K group k') of A is block W[g + k'], so both descriptor
//     offsets are 128 bytes.  W is 8/Q of the Toeplitz matrix.
//   * step > 1: taps j = step*q + phi read the decimated stream
//     d_psi[x] = d[step*x + psi]; each phase is a unit-step correlation with
//     its own template taps and moveout, accumulated into the same sums.
//
// Operands are pairs, high h and low l, and one K step is three MMAs: h h, h l
// and l h (the dropped l l is the square of the pair's rounding).
//   * split bf16: h = bf16(x), l = bf16(x - h): 2^-16 of a product at most.
//   * FP32: x = s (h + 2^-11 l) in fp16, s a power of two (per data channel, per
//     template channel) that brings the largest value to [2^14, 2^15), h =
//     fp16(x / s), l = fp16(2^11 (x / s - h)).  h has 11 significant bits and l
//     the next 11, so the pair holds x to half a unit of FP32's last place,
//     down to 2^-50 of the channel's largest value (below that l runs out of
//     exponent), and the dropped l l is at most 2^-24 of |t d|.
//   * single bf16: h alone, one MMA.
// The tensor core rounds every accumulation toward zero, so a long chain drifts, most of
// all at a match, where every product adds: a chain of m steps that add something to the
// output is some 0.6e-7 m low at a perfect match.  So the h h products run in chains of a
// few steps (tc_chains), each in a fresh accumulator that the epilogue adds to its
// registers in FP32 (rounded to nearest); h l and l h, smaller by the pair's rounding,
// share one accumulator per channel.  RMS error at perfect matches of Hann-tapered noise,
// FP32 multiply-adds and here: 56 taps 1.34 and 1.36e-7, 112 taps 1.74 and 1.21e-7, 300
// taps 2.80 and 2.50e-7, 600 taps 4.1 and 3.5e-7, 1,200 taps 6.0 and 3.8e-7 (with chains of
// 16 steps 2.1, 2.8, 4.7, 7.2, 7.3e-7); away from matches it is further below.
//
// What bounds it: the tensor pipe, and with it the power limit, from some 500
// taps (40 templates x 60 channels x 1.08M lags x 600 taps in 6.3 ms: 1.8
// PFLOP/s of MMAs, 1.74 is what cuBLAS sustains under the limit); the issuing
// threads and the epilogue below, which takes some 400 cycles per chain (with the
// preparation 300 taps 5.2 ms, 60 taps 4.3 ms; in chains of 16 steps 4.7 and 3.5 ms).
// An issuing thread's code costs as much as its MMAs: a branchy loop took 500 cycles
// per MMA of 64.
//
// Roles of a persistent CTA (12 warps, one CTA per SM), which takes items (one
// template x NB*Q consecutive outputs, all channels or a part of them) from a
// tile queue:
//   warp 0      claims items; TMA bulk copies of the template blocks of a (channel,
//               phase) stage (two buffers) and of its data, four column blocks
//               per slot
//   warp 1      issues the h h MMAs into H0 / H1 in turn, one chain each
//   warp 2      issues the h l and l h MMAs into S0 / S1, one channel each (two
//               issuers: one thread cannot issue fast enough, and neither
//               waits for the other's accumulators)
//   warp 3      bulk copies of the window statistics
//   warps 4-11  epilogue: chains into registers, then per channel the
//               normalisation and the network sum, both in registers (208 per
//               thread; the other four warps give theirs up)
// TMEM: H0, H1, S0, S1 of 128 columns each: all 512.
// Every wait is bounded (globaltimer); on timeout the CTA raises an error
// word, stops issuing, waits for its own copies/MMAs (bounded) and frees TMEM.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdlib>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "fmf_tc.cuh"

namespace fmf {

// Epilogue warps, a quarter of them on each TMEM lane quarter: 8 with 64 columns of a
// full tile each; 16 with 32 for per-channel lengths, whose epilogue does four
// times the arithmetic per output and waits for it (40 templates x 60 channels x
// 300,000 lags: 7.2 ms with 8).
constexpr int tc_epi_warps(bool var) { return var ? 16 : 8; }
constexpr int tc_threads(bool var) { return 32 * (4 + tc_epi_warps(var)); }
constexpr int tc_groups(bool var) { return tc_epi_warps(var) / 4; }  // column groups of a tile
constexpr int TC_MAX_ROWS = 8;     // data slots, at most
constexpr int TC_MAX_PARTS = 32;   // channel parts of an item, at most
constexpr int TC_MAX_STATS = 2;    // statistics slots, at most
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

// x / s as the pair (h, l); x that is not finite becomes 0.  With a common length every
// window that holds it has a NaN energy, and its coefficient is 0 in both kernels;
// with per-channel lengths, whose energies are integers, such a channel raises the
// search's flag.
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

// Whether the CUDA cores run this search instead.
__device__ __forceinline__ bool tc_skipped(const TcProb &pr) { return pr.skip && *pr.skip; }

// Whether the tile at I0 holds a valid output.  The range of a template without any is
// empty, wherever it lies: its moveouts may point anywhere.
__device__ __forceinline__ bool tc_holds(int k_lo, int k_hi, long long I0, int nb)
{
    return k_lo < k_hi && I0 < k_hi && I0 + (long long)TC_Q * nb > k_lo;
}

// Whether a tile of template t holds a valid output and the search runs here.
__device__ __forceinline__ bool tc_busy(const TcProb &pr, long long I0, int t)
{
    return tc_holds(pr.P.k_lo[t], pr.P.k_hi[t], I0, pr.nb) && !tc_skipped(pr);
}

// Moveout of phase phi in its stream, and the stream: m = step mu + psi.
__device__ __forceinline__ int tc_phase(int m, int step, int &psi)
{
    if (step == 1) {
        psi = 0;
        return m;
    }
    const int mu = m >= 0 ? m / step : -((-m + step - 1) / step);
    psi = m - step * mu;
    return mu;
}

// A statistics slot: `columns` lag blocks of each column group of the tile from each of
// `streams` arrays, copied from the 16-byte boundary before the first window.
// Fixed lengths: window energies, or (energy, mean) pairs.  Per-channel lengths:
// running sums of d^2 at a window's start and end; for 'full' there are no slots (the
// epilogue reads those, and those of d, itself).
struct StatSlot {
    int columns, streams, elem, groups;
    __host__ __device__ constexpr StatSlot(bool var, bool full)
        : columns(var ? 4 : (full ? 16 : 32)), streams(var ? (full ? 0 : 2) : 1),
          elem(var || full ? 8 : 4), groups(var ? 4 : 2)
    {
    }
    __host__ __device__ constexpr uint32_t part() const { return (uint32_t)(columns * TC_Q * elem + 16); }
    __host__ __device__ constexpr uint32_t bytes() const { return (uint32_t)(groups * streams) * part(); }
    __host__ __device__ constexpr int align() const { return 16 / elem - 1; }  // mask of elements
};

// The same as a bf16 pair in the data's own units: l is bf16(x - h).  keep: x that is not
// finite stays so.
__device__ __forceinline__ void split_bf16(float x, bool keep, uint16_t &hi, uint16_t &lo)
{
    const float y = keep || finite_bits(__float_as_uint(x) & 0x7fffffffu) ? x : 0.0f;
    const __nv_bfloat16 h = __float2bfloat16_rn(y);
    const __nv_bfloat16 l = __float2bfloat16_rn(y - __bfloat162float(h));
    hi = __bfloat16_as_ushort(h);
    lo = __bfloat16_as_ushort(l);
}

template <bool FP32>
__device__ __forceinline__ void split_pair(float x, float inv_s, bool keep, uint16_t &hi, uint16_t &lo)
{
    if constexpr (FP32)
        split_fp16(x, inv_s, hi, lo);
    else
        split_bf16(x, keep, hi, lo);
}

// ------------------------------------------------------------------ operands
// FP32: the scale of a data channel from the scan of prepare_problem, stat (largest
// |x|; smallest window energy that can pass the threshold, complemented).  The
// caller that is `first` also writes the channel's exponent and decides whether
// the pairs hold its values.  A sample is off by 2^-51 of the largest value M at most, a
// coefficient so by sqrt(L) 2^-51 M over the root of the window's energy (Cauchy-Schwarz):
// windows down to 2^-42 M^2 keep it at sqrt(L) 2^-30, 2.3e-8 at 600 taps, and near 1e-9
// where the samples' errors are independent.
__device__ __forceinline__ float tc_channel_scale(const unsigned *stat, int ch, int SC, bool first, int *d_exp,
                                                  unsigned *skip)
{
    const unsigned top = stat[ch];
    bool ok;
    const int e = max_exponent(top, ok);
    if (first) {
        d_exp[ch] = e;
        const unsigned low = ~stat[SC + ch];  // smallest energy's bits; ~0 (a NaN): none
        const float m = __uint_as_float(top);
        if (!ok || (low < 0x7f800000u && __uint_as_float(low) * 0x1p42f < m * m))
            atomicOr(skip, 1u);
    }
    return exp2_int(kTopExp - e);
}

// G[ch][psi][cb][r][e] = pair of d[ch][step*(Q*(r - row_front) + 8*cb + e) + psi], zero outside [0, N).
// A block turns the samples of `rows` rows of every phase through shared memory:
// loads of consecutive samples, stores of consecutive rows of a column block (a
// thread per 16 bytes, reading its own 8 samples, kept the L1 at 98 %: 60
// channels x 1.08M samples 231 us, 93 us here).  A block of `tiles` per channel, 256
// threads, dynamic shared memory tc_turn_bytes.
constexpr int TC_TURN_PITCH = TC_Q + 8;  // halves per row: 16-byte reads of 8 rows hit distinct banks
constexpr int TC_TURN_STEP = 64;         // the largest step with a row of every phase
__host__ __device__ __forceinline__ int tc_turn_rows(int step)
{
    int rows = 32;
    while (rows > 1 && rows * step > TC_TURN_STEP)
        rows >>= 1;
    return rows;
}
static size_t tc_turn_bytes(int step, bool pairs)
{
    return (size_t)(pairs ? 2 : 1) * step * tc_turn_rows(step) * TC_TURN_PITCH * sizeof(uint16_t);
}

struct TcDataWork {
    const float *data;
    int N, SC, step, tiles, rows_total, row_front;
    const unsigned *stat;
    uint16_t *g_hi, *g_lo;
    int *d_exp;
    unsigned *skip;
    // bf16 forms: samples that are not finite stay so, and with them the numerators of the
    // windows round them ('short' with per-channel lengths: no energy tells of them)
    bool keep;
};

template <bool FP32>
__device__ __forceinline__ void tc_data_block(const TcDataWork &d, int block, uint4 *turn_smem)
{
    const int step = d.step, N = d.N, rows_total = d.rows_total, row_front = d.row_front;
    const float *__restrict__ data = d.data;
    uint16_t *__restrict__ g_hi = d.g_hi, *__restrict__ g_lo = d.g_lo;
    const int rows = tc_turn_rows(step), ch = block / d.tiles, tile = block - ch * d.tiles, row0 = tile * rows;
    uint16_t *hi = reinterpret_cast<uint16_t *>(turn_smem), *lo = hi + step * rows * TC_TURN_PITCH;
    float inv_s = 1.0f;
    if constexpr (FP32)
        inv_s = tc_channel_scale(d.stat, ch, d.SC, tile == 0 && threadIdx.x == 0, d.d_exp, d.skip);
    const float *src = data + (size_t)ch * N;
    const long long pos0 = (long long)step * TC_Q * (row0 - row_front);
    const int count = step * TC_Q * rows;
    constexpr int kLoads = 8;  // in flight per thread; count is a multiple of 128
    // sample i is sample q of phase psi; a thread's next one, without a division, 256 on
    const int dq = 256 / step, dpsi = 256 - dq * step;
    int q = (int)threadIdx.x / step, psi = (int)threadIdx.x - q * step;
    const bool one = step == 1;
    for (int i0 = threadIdx.x; i0 < count; i0 += kLoads * 256) {
        float x[kLoads];
#pragma unroll
        for (int j = 0; j < kLoads; j++) {
            const int i = i0 + 256 * j;
            const long long pos = pos0 + i;
            x[j] = i < count && pos >= 0 && pos < N ? __ldg(src + pos) : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < kLoads; j++) {
            const int i = i0 + 256 * j;
            if (i < count) {
                const int at = one ? (i >> 7) * TC_TURN_PITCH + (i & (TC_Q - 1))
                                   : (psi * rows + (q >> 7)) * TC_TURN_PITCH + (q & (TC_Q - 1));
                uint16_t h, l;
                split_pair<FP32>(x[j], inv_s, d.keep, h, l);
                hi[at] = h;
                if (g_lo)
                    lo[at] = l;
            }
            if (!one) {
                q += dq;
                psi += dpsi;
                if (psi >= step) {
                    psi -= step;
                    q++;
                }
            }
        }
    }
    __syncthreads();
    const int n = min(rows, rows_total - row0), rows_log2 = 31 - __clz(rows);
    for (int i = threadIdx.x; i < step * TC_CB * rows; i += 256) {
        const int r = i & (rows - 1), rest = i >> rows_log2, cb = rest & (TC_CB - 1), psi = rest / TC_CB;
        if (r < n) {
            const int at = (psi * rows + r) * TC_TURN_PITCH + 8 * cb;
            const size_t o = (((size_t)ch * step + psi) * TC_CB + cb) * rows_total + row0 + r;
            reinterpret_cast<uint4 *>(g_hi)[o] = *reinterpret_cast<const uint4 *>(hi + at);
            if (g_lo)
                reinterpret_cast<uint4 *>(g_lo)[o] = *reinterpret_cast<const uint4 *>(lo + at);
        }
    }
}

// The same for larger steps, whose phases do not share a block: one thread per
// 16-byte row chunk.
template <bool FP32>
__global__ void tc_data_sparse_kernel(const float *__restrict__ data, int N, int SC, int step, int rows_total,
                                      int row_front, const unsigned *__restrict__ stat,
                                      uint16_t *__restrict__ g_hi, uint16_t *__restrict__ g_lo,
                                      int *__restrict__ d_exp, unsigned *skip, bool keep)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long per_ch = (long long)step * TC_CB * rows_total;
    if (idx >= per_ch * SC)
        return;
    const int ch = (int)(idx / per_ch);
    long long rest = idx - ch * per_ch;
    float inv_s = 1.0f;
    if constexpr (FP32)
        inv_s = tc_channel_scale(stat, ch, SC, rest == 0, d_exp, skip);
    const int r = (int)(rest % rows_total);
    rest /= rows_total;
    const int cb = (int)(rest % TC_CB);
    const int psi = (int)(rest / TC_CB);
    const long long x0 = (long long)TC_Q * (r - row_front) + 8 * cb;
    const float *src = data + (size_t)ch * N;
    uint16_t h[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const long long pos = (long long)step * (x0 + i) + psi;
        const float v = (x0 + i >= 0 && pos < N) ? src[pos] : 0.0f;
        split_pair<FP32>(v, inv_s, keep, h[i], l[i]);
    }
    reinterpret_cast<uint4 *>(g_hi)[idx] = pack8(h);
    if (g_lo)
        reinterpret_cast<uint4 *>(g_lo)[idx] = pack8(l);
}

// W[t][ch][phi][n][e][c] = pair of tphi[8n + e + c - (Q-1+s)], tphi[q] = tpl[step*q + phi],
// s = mu mod Q, mu = floor((mo + phi) / step); one block per (template,
// channel), its taps in shared memory (read once, written 8 times over), or several where
// that would leave SMs idle over the phases of a large step (4 templates x 3 channels,
// step 439: 256 us with one block each, 20 us here).
// FP32: also the channel's exponent, and the search's flag where a tap is not finite; the
// bf16 forms keep such a tap.  queue: the tile queue of the persistent launch that
// follows, cleared here (a memset costs 2 us).
struct TcTemplateWork {
    const float *tpl;
    const int *mo;
    int L, step, NW;
    uint16_t *w_hi, *w_lo;
    int *t_exp;
    unsigned *skip;
    unsigned long long *queue;
    int parts;  // blocks per (template, channel)
};

template <bool FP32>
__device__ __forceinline__ void tc_template_block(const TcTemplateWork &w, unsigned block, float *taps)
{
    const unsigned part = block % (unsigned)w.parts;
    const long long row = block / (unsigned)w.parts;  // t*SC + ch
    const float *__restrict__ tpl = w.tpl;
    uint16_t *__restrict__ w_hi = w.w_hi, *__restrict__ w_lo = w.w_lo;
    const int L = w.L, step = w.step, NW = w.NW;
    int *t_exp = w.t_exp;
    unsigned *skip = w.skip;
    if (w.queue && block == 0 && threadIdx.x == 0)
        *w.queue = 0;
    const float *src = tpl + row * L;
    float inv_s = 1.0f;
    if constexpr (FP32) {
        __shared__ unsigned red[8];
        __shared__ int bad;
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
        inv_s = exp2_int(kTopExp - e);
        if (threadIdx.x == 0) {
            if (!ok || bad)
                atomicOr(skip, 1u);
            t_exp[row] = e;
        }
    } else {
        for (int j = threadIdx.x; j < L; j += blockDim.x)
            taps[j] = src[j];
        __syncthreads();
    }
    const int m0 = w.mo[row];
    const int per_phase = NW * 8, used = tc_phases(step, L) * per_phase;
    const int end = (int)((long long)used * (part + 1) / w.parts);
    for (int i = (int)((long long)used * part / w.parts) + threadIdx.x; i < end; i += blockDim.x) {
        const int phi = i / per_phase, ne = i - phi * per_phase;
        int psi;
        const int s = tc_phase(m0 + phi, step, psi) & (TC_Q - 1);
        uint16_t h[8], l[8];
        const int q0 = 8 * (ne >> 3) + (ne & 7) - (TC_Q - 1 + s);
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const int q = q0 + c, j = step * q + phi;
            split_pair<FP32>(q >= 0 && j < L ? taps[j] : 0.0f, inv_s, true, h[c], l[c]);
        }
        const long long o = row * step * per_phase + i;
        reinterpret_cast<uint4 *>(w_hi)[o] = pack8(h);
        if (w_lo)
            reinterpret_cast<uint4 *>(w_lo)[o] = pack8(l);
    }
}

// FP32: raises the flag where pairs cannot hold a template, as tc_template_block does, for
// searches whose operands are made in parts: the first parts run before the others'
// operands are made, and the flag is the whole search's.  A block per (template, channel).
__global__ void __launch_bounds__(128) tc_template_check_kernel(const float *__restrict__ tpl, int L, unsigned *skip)
{
    const float *src = tpl + (size_t)blockIdx.x * L;
    unsigned top = 0;
    for (int j = threadIdx.x; j < L; j += blockDim.x)
        top = max(top, __float_as_uint(src[j]) & 0x7fffffffu);
    top = __reduce_max_sync(0xffffffffu, top);
    __shared__ unsigned red[4];
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = top;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 4; i++)
            top = max(top, red[i]);
        bool ok;
        max_exponent(top, ok);  // (a value that is not finite is above them all)
        if (!ok)
            atomicOr(skip, 1u);
    }
}

// Both in one launch: blocks [0, n_data) turn data, the others make template blocks.
template <bool FP32>
__global__ void __launch_bounds__(256) tc_operand_kernel(const TcDataWork d, unsigned n_data, const TcTemplateWork w)
{
    extern __shared__ uint4 operand_smem[];
    if (blockIdx.x < n_data)
        tc_data_block<FP32>(d, (int)blockIdx.x, operand_smem);
    else
        tc_template_block<FP32>(w, blockIdx.x - n_data, reinterpret_cast<float *>(operand_smem));
}

// ------------------------------------------------------------------ persistent kernel
// Offsets of the barriers in the kernel's shared memory (bytes past the rings).
struct TcBars {
    static constexpr uint32_t wfull = 0, wempty = 16, dfull = 32, dempty = dfull + 8 * TC_MAX_ROWS,
                              efull = dempty + 8 * TC_MAX_ROWS, eempty = efull + 8 * TC_MAX_STATS,
                              hfull = eempty + 8 * TC_MAX_STATS, hempty = hfull + 16, sfull = hempty + 16,
                              sempty = sfull + 16, ifull = sempty + 16, iempty = ifull + 32,
                              fin = iempty + 32, items = fin + 8, tmem = items + 32, abort = tmem + 4,
                              bytes = abort + 4;
};

// One MMA issuer's walk over the items: the h h products (SMALL false; chains of
// chain_slots data slots into H0 / H1 in turn) or the h l and l h products (into
// S0 / S1, a channel each).
template <bool VAR, bool SMALL, int N>
__device__ __forceinline__ void tc_issue(const TcBatch<N> &B, const long long *ring, uint32_t bar,
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
        if (!wait(bar + TcBars::ifull + 8 * is, (q >> 2) & 1, 32u))
            return;
        const long long item = ring[is];
        __syncwarp();
        if (one)
            mbar_arrive(bar + TcBars::iempty + 8 * is);
        if (item >= B.total_items)
            return;
        int p, tile, t, c_begin, c_end, part;
        decode_item(B, item, p, tile, t, c_begin, c_end, part);
        p = uniform(p);
        t = uniform(t);
        c_end = uniform(c_end);
        const TcProb &pr = B.prob[p];
        const int nb = pr.nb;
        const long long I0 = (long long)tile * TC_Q * nb;
        if (!uniform(tc_busy(pr, I0, t)))
            continue;
        // the template's lag blocks in this tile, in steps of 16: the other accumulator
        // columns stay as they are, and their outputs are not used
        const int cols = uniform((int)min((long long)nb, (pr.P.k_hi[t] - I0 + 16 * TC_Q - 1) / (16 * TC_Q) * 16));
        // kind::f16 descriptor: F32 accumulate, A and B both FP16 or both BF16, K-major, N = cols, M = 128
        const uint32_t idesc = (1u << 4) | B.mma_types | ((uint32_t)(cols >> 3) << 17) | ((uint32_t)(TC_Q >> 4) << 24);
        const int SC = pr.P.SC, step = pr.P.step, L = pr.P.L;
        const uint32_t all_pairs = (uint32_t)uniform(tc_phases(step, L)) * (TC_CB / 2);
        const uint32_t chains = SMALL ? 0u : (uint32_t)pr.chains;
        const uint32_t col_bytes = (uint32_t)pr.R * 16;
        // 16-byte units from a high half to its low half, and of a column-block pair
        const uint32_t a_low = (uint32_t)pr.NW * 8, b_low = 4u * (uint32_t)pr.R, b_pair = 2u * (uint32_t)pr.R;
        const uint32_t a_hi = (uint32_t)(sdesc(0, 128, 128) >> 32);
        const uint32_t b_hi = (uint32_t)(sdesc(0, col_bytes, 128) >> 32);
        const uint32_t a_base = (uint32_t)sdesc(w_base, 128, 128), b_base = (uint32_t)sdesc(d_base, col_bytes, 128);
        const uint32_t a_buf = (uint32_t)B.w_bytes >> 4, b_slot = (uint32_t)B.row_bytes >> 4;
        const size_t row0 = (size_t)t * SC;
        const int chain_steps = SMALL ? 0 : pr.chain_steps;
        int phases = uniform(tc_phases(step, L));
        uint32_t parts_log2 = (uint32_t)uniform(tc_pair_chains(L, step, L, chain_steps));
        for (int g0 = uniform(c_begin); g0 < c_end; g0 += 32) {
            // the scalars of 32 channels, one per lane
            const int cl = min(g0 + (int)(threadIdx.x & 31), c_end - 1);
            const int mo_l = pr.P.mo[row0 + cl], n_l = VAR ? pr.P.ntap[row0 + cl] : L;
            uint32_t active = __ballot_sync(0xffffffffu, g0 + (int)(threadIdx.x & 31) < c_end && pr.P.w[row0 + cl] != 0.0f);
            for (; active; active &= active - 1) {
                const int src = __ffs(active) - 1;
                const int mo = __shfl_sync(0xffffffffu, mo_l, src), ntap = __shfl_sync(0xffffffffu, n_l, src);
                if (VAR)
                    phases = tc_phases(step, ntap);
                if (VAR && chain_steps)
                    parts_log2 = (uint32_t)tc_pair_chains(L, step, ntap, chain_steps);
                // a chain ends where `chains` of them spread over all pairs do, and at the last pair
                uint32_t credit = 0;
                bool fresh = true;
                uint32_t dt = 0, acc = 0;
                const auto next_acc = [&]() {
                    const uint32_t empty = bar + (SMALL ? TcBars::sempty : TcBars::hempty) + 8 * (acc_i & 1);
                    if (acc_i >= 2 && !wait(empty, ((acc_i >> 1) - 1) & 1, 4u))
                        return false;
                    tc_fence_after();
                    dt = tmem + (SMALL ? 256u : 0u) + 128u * (acc_i & 1);
                    acc = 0;
                    return true;
                };
                for (int phi = 0; phi < phases; phi++, stages++) {
                    const uint32_t wb = stages & 1;
                    int psi;
                    const uint32_t sres = (uint32_t)tc_phase(mo + phi, step, psi) & (TC_Q - 1);
                    const uint32_t k_first = sres & ~15u;
                    const uint32_t k_end = (uint32_t)tc_k_end((int)sres, step == 1 ? ntap : tc_phase_taps(L, step, phi, ntap));
                    if (!wait(bar + TcBars::wfull + 8 * wb, (stages >> 1) & 1, 8u))
                        return;
                    const uint32_t a0 = a_base + (wb ? a_buf : 0u);
#pragma unroll 1
                    for (uint32_t j = 0; j < TC_CB / 2; j++) {
                        if (fresh && !next_acc())
                            return;
                        // two column-block pairs per slot
                        if ((j & 1) == 0 && !wait(bar + TcBars::dfull + 8 * slot, turn & 1, 8u))
                            return;
                        // K steps k = 16 j + 128 i: A moves 16 template blocks (2 KB), B one data
                        // row (16 bytes) per step.  The start-address field (16-byte units) of
                        // an address below 256 KB never carries out of its 14 bits.
                        const uint32_t late = 16 * j < k_first ? 1u : 0u;
                        uint32_t n = ((k_end - 16 * j + TC_Q - 1) >> 7) - late;
                        uint32_t a = a0 + 16 * j + late * TC_Q;
                        uint32_t b = b_base + slot * b_slot + (j & 1 ? b_pair : 0u) + late;
                        const auto issue = [&](uint32_t steps) {
#pragma unroll 1
                            for (uint32_t i = 0; i < steps; i++) {
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
                        };
                        if (!SMALL && parts_log2) {  // all chains of this pair but the last
                            const uint32_t all = n;
                            for (uint32_t part = 1; part >> parts_log2 == 0; part++) {
                                const uint32_t rest = all - ((all * part) >> parts_log2);
                                issue(n - rest);
                                n = rest;
                                if (one)
                                    mma_commit(bar + TcBars::hfull + 8 * (acc_i & 1));
                                acc_i++;
                                if (!next_acc())
                                    return;
                            }
                        }
                        issue(n);
                        credit += chains;
                        const bool done = credit >= all_pairs || (!SMALL && parts_log2) ||
                                          (j == TC_CB / 2 - 1 && phi == phases - 1);
                        if (credit >= all_pairs)
                            credit -= all_pairs;
                        if (one) {
                            if (j & 1)
                                mma_commit(bar + TcBars::dempty + 8 * slot);
                            if (done)
                                mma_commit(bar + (SMALL ? TcBars::sfull : TcBars::hfull) + 8 * (acc_i & 1));
                        }
                        if ((j & 1) && ++slot == n_rows) {
                            slot = 0;
                            turn++;
                        }
                        fresh = done;
                        if (done)
                            acc_i++;
                    }
                    if (one)
                        mma_commit(bar + TcBars::wempty + 8 * wb);
                }
            }
        }
    }
}

// VAR: per-channel template lengths (Fisher-z network sum); FULL: 'full'
// normalisation; NSUM: network sum.  One instantiation per mode, each with its
// own epilogue code only (the code of all roles shares the instruction cache).
// ONE (per-channel lengths): every channel is one chain (the bf16 forms), whose
// numerators go from the accumulators to the sums without a stop in registers; with
// that stop 16 epilogue warps spill.
template <bool VAR, bool FULL, bool NSUM, bool ONE, int N>
__global__ void __launch_bounds__(tc_threads(VAR), 1) tc_persistent(const __grid_constant__ TcBatch<N> B)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr StatSlot kStat(VAR, FULL);
    constexpr int CH = kStat.columns;
    constexpr uint32_t kStatPart = kStat.part();
    constexpr int TC_EPI_WARPS = tc_epi_warps(VAR), G = tc_groups(VAR);
    static_assert(kStat.groups == G, "statistics slots hold the epilogue's column groups");
    const bool pairs = B.split != 0;

    // template blocks (2 buffers), data slots, statistics slots, barriers
    const uint32_t w_base = smem_u32(smem);
    const uint32_t d_base = w_base + 2u * B.w_bytes;
    const uint32_t e_base = d_base + (uint32_t)B.n_rows * B.row_bytes;
    uint8_t *bar_ptr = smem + 2u * B.w_bytes + (uint32_t)B.n_rows * B.row_bytes + ((uint32_t)B.stat_bytes << B.stat_log2);
    const uint32_t bar = smem_u32(bar_ptr);
    long long *ring = reinterpret_cast<long long *>(bar_ptr + TcBars::items);  // 4 item slots
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bar_ptr + TcBars::tmem);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(bar_ptr + TcBars::abort);
    const int n_rows = B.n_rows, stat_log2 = B.stat_log2;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; i++) {
            mbar_init(bar + TcBars::wfull + 8 * i, 1);
            mbar_init(bar + TcBars::wempty + 8 * i, pairs ? 2 : 1);  // one commit per MMA issuer
            mbar_init(bar + TcBars::hfull + 8 * i, 1);
            mbar_init(bar + TcBars::hempty + 8 * i, TC_EPI_WARPS);
            mbar_init(bar + TcBars::sfull + 8 * i, 1);
            mbar_init(bar + TcBars::sempty + 8 * i, TC_EPI_WARPS);
        }
        for (int i = 0; i < TC_MAX_ROWS; i++) {
            mbar_init(bar + TcBars::dfull + 8 * i, 1);
            mbar_init(bar + TcBars::dempty + 8 * i, pairs ? 2 : 1);
        }
        for (int i = 0; i < TC_MAX_STATS; i++) {
            mbar_init(bar + TcBars::efull + 8 * i, 1);
            mbar_init(bar + TcBars::eempty + 8 * i, TC_EPI_WARPS);
        }
        mbar_init(bar + TcBars::fin, 2);
        for (int i = 0; i < 4; i++) {
            mbar_init(bar + TcBars::ifull + 8 * i, 1);
            mbar_init(bar + TcBars::iempty + 8 * i, (pairs ? 3 : 2) + TC_EPI_WARPS);  // issuers, warp 3, epilogue
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
        // registers: 384 threads x 168 at launch = 128 x 88 + 256 x 208; 640 x 96 =
        // 128 x 64 + 512 x 104 ('full' only: 1,432 -> 1,375 us below, 'short' 757 -> 830 us)
        if (VAR && FULL)
            asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        else if (!VAR)
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
                const bool got = q < 4 || mbar_wait(bar + TcBars::iempty + 8 * is, (uint32_t)(((q >> 2) - 1) & 1),
                                                    abort_flag, B.err, 1u);
                if (got && !*abort_flag)
                    item = (long long)atomicAdd(B.queue, 1ull);
                ring[is] = item;
                mbar_arrive(bar + TcBars::ifull + 8 * is);
            }
            item = __shfl_sync(0xffffffffu, item, 0);
            if (item >= total)
                break;
            int p, tile, t, c_begin, c_end, part;
            decode_item(B, item, p, tile, t, c_begin, c_end, part);
            const TcProb &pr = B.prob[p];
            const Problem &P = pr.P;
            const long long I0 = (long long)tile * TC_Q * pr.nb;
            if (!tc_busy(pr, I0, t))
                continue;
            const int SC = P.SC, step = P.step, all_phases = tc_phases(P.step, P.L);
            const uint32_t col_bytes = (uint32_t)pr.R * 16, wbytes = (uint32_t)pr.NW * 128;
            const size_t row0 = (size_t)t * SC;
            for (int g0 = c_begin; ok && g0 < c_end; g0 += 32) {
                // the scalars of 32 channels, one per lane
                const int cl = min(g0 + lane, c_end - 1);
                const int mo_l = P.mo[row0 + cl], n_l = VAR ? P.ntap[row0 + cl] : 0;
                uint32_t active = __ballot_sync(0xffffffffu, g0 + lane < c_end && P.w[row0 + cl] != 0.0f);
                for (; ok && active; active &= active - 1) {
                    const int from = __ffs(active) - 1, ch = g0 + from;
                    const int mo = __shfl_sync(0xffffffffu, mo_l, from);
                    const int phases = VAR ? tc_phases(step, __shfl_sync(0xffffffffu, n_l, from)) : all_phases;
                    for (int phi = 0; ok && phi < phases; phi++, stages++) {
                        const int wb = stages & 1;
                        int psi;
                        const int mu = tc_phase(mo + phi, step, psi);
                        const long long r0 = ((I0 + mu) >> 7) + pr.row_front;  // floor
                        const uint32_t wbar = bar + TcBars::wfull + 8 * wb;
                        if (stages >= 2 && !mbar_wait_warp(bar + TcBars::wempty + 8 * wb, ((stages >> 1) - 1) & 1,
                                                           abort_flag, B.err, 2u)) {
                            ok = false;
                            break;
                        }
                        if (lane == 0)
                            mbar_expect_tx(wbar, pairs ? 2u * wbytes : wbytes);
                        __syncwarp();
                        if (lane < (pairs ? 2 : 1))
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
                            const uint32_t dbar = bar + TcBars::dfull + 8 * slot;
                            if (turn >= 1 && !mbar_wait_warp(bar + TcBars::dempty + 8 * slot, (turn - 1) & 1,
                                                             abort_flag, B.err, 2u)) {
                                ok = false;
                                break;
                            }
                            if (lane == 0)
                                mbar_expect_tx(dbar, pairs ? 8u * col_bytes : 4u * col_bytes);
                            __syncwarp();
                            if (lane < (pairs ? 8 : 4))
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
                mbar_wait(bar + TcBars::wfull + 8 * (u & 1), (u >> 1) & 1, abort_flag, B.err, 0u);
            for (int i = 0; i < n_rows; i++) {
                const int uses = turn + (i < slot ? 1 : 0);
                if (uses)
                    mbar_wait(bar + TcBars::dfull + 8 * i, (uses - 1) & 1, abort_flag, B.err, 0u);
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
            tc_issue<VAR, false>(B, ring, bar, w_base, d_base, tmem, abort_flag, one);
        else if (pairs)
            tc_issue<VAR, true>(B, ring, bar, w_base, d_base, tmem, abort_flag, one);
        __syncwarp();
        if (one) {
            mma_commit(bar + TcBars::fin);
            mbar_wait(bar + TcBars::fin, 0, abort_flag, B.err, 0u);
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
                if (!mbar_wait_warp(bar + TcBars::ifull + 8 * is, (uint32_t)((q >> 2) & 1), abort_flag, B.err, 32u))
                    break;
                const long long item = ring[is];
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(bar + TcBars::iempty + 8 * is);
                if (item >= total)
                    break;
                int p, tile, t, c_begin, c_end, part;
                decode_item(B, item, p, tile, t, c_begin, c_end, part);
                const TcProb &pr = B.prob[p];
                const Problem &P = pr.P;
                const long long I0 = (long long)tile * TC_Q * pr.nb;
                if (kStat.streams == 0 || !tc_busy(pr, I0, t))
                    continue;
                const int nc = pr.nb / G;
                const size_t row0 = (size_t)t * P.SC;
                for (int g0 = c_begin; ok && g0 < c_end; g0 += 32) {
                    const int cl = min(g0 + lane, c_end - 1);
                    const int mo_l = P.mo[row0 + cl], n_l = VAR ? P.ntap[row0 + cl] : 0;
                    uint32_t active = __ballot_sync(0xffffffffu, g0 + lane < c_end && P.w[row0 + cl] != 0.0f);
                    for (; ok && active; active &= active - 1) {
                        const int from = __ffs(active) - 1, ch = g0 + from;
                        int psi;  // phase 0: the moveout's own stream
                        const int mu = tc_phase(__shfl_sync(0xffffffffu, mo_l, from), P.step, psi);
                        // lane = G * array + column group
                        const char *src;
                        if constexpr (VAR) {
                            int psi2;  // the windows' ends
                            const int far = tc_phase(psi + __shfl_sync(0xffffffffu, n_l, from), P.step, psi2);
                            const long long x = I0 + mu + (lane & G ? far : 0);
                            src = reinterpret_cast<const char *>(P.pre2q) + (ch * P.pre_ch + (lane & G ? psi2 : psi) * P.pre_ps +
                                          (x & ~(long long)kStat.align())) * kStat.elem;
                        } else {
                            src = reinterpret_cast<const char *>(P.stat_e) +
                                  (ch * P.stat_ch + psi * P.stat_ps + ((I0 + mu) & ~(long long)kStat.align())) *
                                      kStat.elem;
                        }
                        src += (size_t)(lane & (G - 1)) * nc * TC_Q * kStat.elem;
                        for (int c0 = 0; c0 < nc; c0 += CH, ec++) {
                            const int es = ec & ((1 << stat_log2) - 1);
                            const uint32_t ebar = bar + TcBars::efull + 8 * es;
                            if ((ec >> stat_log2) >= 1 &&
                                !mbar_wait_warp(bar + TcBars::eempty + 8 * es, ((ec >> stat_log2) - 1) & 1,
                                                abort_flag, B.err, 2u)) {
                                ok = false;
                                break;
                            }
                            const uint32_t bytes = min(CH, nc) * TC_Q * kStat.elem + 16;
                            if (lane == 0)
                                mbar_expect_tx(ebar, (uint32_t)(G * kStat.streams) * bytes);
                            __syncwarp();
                            if (lane < G * kStat.streams)
                                bulk_g2s(e_base + es * (uint32_t)B.stat_bytes + lane * kStatPart,
                                         src + (size_t)c0 * TC_Q * kStat.elem, bytes, ebar);
                        }
                    }
                }
            }
            for (int i = 0; i < (1 << stat_log2); i++) {  // the last use of every slot
                const int uses = (ec >> stat_log2) + (i < (ec & ((1 << stat_log2) - 1)) ? 1 : 0);
                if (uses && lane == 0)
                    mbar_wait(bar + TcBars::efull + 8 * i, (uses - 1) & 1, abort_flag, B.err, 0u);
            }
        }
        __syncwarp();
    } else {
        // ---------------------------------------------------------- epilogue
        // Warp w reads TMEM lane quarter w % 4 (rows 32*(w%4) + lane) and its half of the
        // columns; numerators and network sums of its outputs live in registers.
        if (VAR && FULL)
            asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        else if (!VAR)
            asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        constexpr int NCM = TC_NB_MAX / G;  // columns per thread, at most
        const int quarter = warp & 3;
        const int cgroup = (warp - 4) >> 2;
        const int b = TC_Q - 1 - (32 * quarter + lane);  // phase of this thread's row
        const uint32_t lane_base = tmem + ((uint32_t)(32 * quarter) << 16);
        int c = 0, hc = 0, ec = 0;  // channels, chains and statistics slots used
        for (long long q = 0;; q++) {
            const int is = (int)(q & 3);
            long long item = total;
            if (lane == 0) {
                if (mbar_wait(bar + TcBars::ifull + 8 * is, (uint32_t)((q >> 2) & 1), abort_flag, B.err, 64u)) {
                    item = ring[is];
                    mbar_arrive(bar + TcBars::iempty + 8 * is);
                }
            }
            item = __shfl_sync(0xffffffffu, item, 0);
            if (item >= total)
                break;
            int p, tile, t, c_begin, c_end, part;
            decode_item(B, item, p, tile, t, c_begin, c_end, part);
            const TcProb &pr = B.prob[p];
            if (tc_skipped(pr))
                continue;
            const int nb = pr.nb;
            const int NC = nb / G;  // columns of this thread
            const int a0 = cgroup * NC;
            const int SC = pr.P.SC, step = pr.P.step, n_corr = pr.P.n_corr;
            const long long I0 = (long long)tile * TC_Q * nb;
            const int klo = pr.P.k_lo[t], khi = pr.P.k_hi[t];
            const bool busy = tc_holds(klo, khi, I0, nb);
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
            // h h chains of a channel: of whole pairs, or several of each
            const auto chains_of = [&](int n) {
                const int log2 = tc_pair_chains(pr.P.L, step, n, pr.chain_steps), cols = tc_phases(step, n) * (TC_CB / 2);
                const long long all = tc_phases(step, pr.P.L) * (TC_CB / 2);
                // (the last pair ends one, whether or not the chains before it come out even)
                return log2 ? cols << log2 : (int)((cols - 1) * (long long)pr.chains / all) + 1;
            };
            const int chains = ONE || VAR ? 1 : chains_of(pr.P.L);
            for (int g0 = c_begin; busy && g0 < c_end; g0 += 32) {
                // the scalars of 32 channels, one per lane
                const int cl = min(g0 + lane, c_end - 1);
                const float w_l = g0 + lane < c_end ? pr.P.w[row0 + cl] : 0.0f, sst_l = pr.P.sst[row0 + cl];
                const int mo_l = pr.P.mo[row0 + cl];
                // 2^unit: the product of the operands' scales
                const int unit_l = pr.t_exp ? pr.t_exp[row0 + cl] + pr.d_exp[cl] - 2 * kTopExp : 0;
                const int n_l = VAR ? pr.P.ntap[row0 + cl] : 0;
                const float z_l = VAR ? pr.P.zweight[row0 + cl] : 0.0f, u2_l = VAR ? pr.P.unit2[cl] : 0.0f;
                const float ts_l = FULL ? pr.P.tsum[row0 + cl] * exp2_int(-unit_l) : 0.0f;
                const int chains_l = VAR && !ONE ? chains_of(n_l) : 0;
                uint32_t active = __ballot_sync(0xffffffffu, w_l != 0.0f);
#pragma unroll 1
                for (; active; active &= active - 1) {
                    const int from = __ffs(active) - 1, ch = g0 + from;
                    const float wc = __shfl_sync(0xffffffffu, w_l, from), sst = __shfl_sync(0xffffffffu, sst_l, from);
                    const float unit = exp2_int(__shfl_sync(0xffffffffu, unit_l, from));
                    const float ts = FULL ? __shfl_sync(0xffffffffu, ts_l, from) : 0.0f;
                    const int mo = __shfl_sync(0xffffffffu, mo_l, from);
                    float num[ONE ? 1 : NCM];
#pragma unroll
                    for (int i = 0; i < NCM; i++)
                        if constexpr (!ONE)
                            num[i] = 0.0f;
                    if constexpr (ONE) {  // both sums are awaited here and read below
                        if (!mbar_wait_all(bar + TcBars::hfull + 8 * (hc & 1), (hc >> 1) & 1, abort_flag, B.err, 16u) ||
                            (pairs && !mbar_wait_all(bar + TcBars::sfull + 8 * (c & 1), (c >> 1) & 1, abort_flag,
                                                     B.err, 16u)))
                            goto epilogue_done;
                        tc_fence_after();
                    }
                    const int n_chains = VAR && !ONE ? __shfl_sync(0xffffffffu, chains_l, from) : chains;
                    const int n_sums = n_chains + (pairs ? 1 : 0);
                    // numerators: the chains' sums, then S (FP32: times 2^-11)
#pragma unroll 1
                    for (int j = 0; !ONE && j < n_sums; j++) {
                        const bool last = j == n_chains;
                        const int u = last ? c : hc;
                        if (!mbar_wait_all(bar + (last ? TcBars::sfull : TcBars::hfull) + 8 * (u & 1), (u >> 1) & 1,
                                           abort_flag, B.err, 16u))
                            goto epilogue_done;
                        tc_fence_after();
                        const uint32_t h = lane_base + (last ? 256u : 0u) + 128u * (u & 1) + a0;
                        const float f = last ? B.lo_unit : 1.0f;  // powers of two: exact products
                        constexpr int LD = VAR ? 16 : 32;  // columns per load; a small tile reads too many
#pragma unroll
                        for (int c0 = 0; c0 < NCM; c0 += LD) {
                            if (c0 < NC) {
                                float x[LD];
                                if constexpr (VAR)
                                    tmem_ld16(h + c0, x);
                                else
                                    tmem_ld32(h + c0, x);
                                tmem_wait_ld();
#pragma unroll
                                for (int i = 0; i < LD; i++)
                                    if constexpr (!ONE)
                                        num[c0 + i] = fmaf(x[i], f, num[c0 + i]);
                            }
                        }
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0)
                            mbar_arrive(bar + (last ? TcBars::sempty : TcBars::hempty) + 8 * (u & 1));
                        if (!last)
                            hc++;
                    }
                    const float wu = wc * unit;  // a power of two: cc * wc rounds the same
                    // per-channel outputs: this channel's, one lag block after the other
                    float *oc = pr.P.by_channel ? pr.P.by_channel + (row0 + ch) * n_corr + k0
                                                : pr.P.out + ((size_t)t * n_corr + k0) * SC + ch;
                    const size_t oc_step = (size_t)TC_Q * (pr.P.by_channel ? 1 : SC);
                    int psi;
                    const int mu = tc_phase(mo, step, psi);
                    const int head = (int)((I0 + mu) & kStat.align());  // past the 16-byte boundary
                    if constexpr (VAR) {
                        // window sums of the channel's own length from its running sums, the
                        // threshold on the square root, atanh(cc - 10 eps) * z
                        const int ntap = __shfl_sync(0xffffffffu, n_l, from);
                        const float zw = __shfl_sync(0xffffffffu, z_l, from), u2 = __shfl_sync(0xffffffffu, u2_l, from);
                        const float nf = (float)ntap, inv_n = 1.0f / nf;
                        int psi2;
                        const int far = tc_phase(psi + ntap, step, psi2);
                        const int head2 = (int)((I0 + mu + far) & kStat.align());
                        // 'full' reads its four running sums per output, 32 bytes, from global memory
                        // (L2): in slots of two columns they took 16 waits a channel (12 stations x
                        // 3 channels x 598 taps x 7 templates x 959,372 samples: 1,651 us, 1,375 here)
                        const long long g1 = ch * pr.P.pre_ch + (long long)psi * pr.P.pre_ps + k0 + mu;
                        const long long g2 = ch * pr.P.pre_ch + (long long)psi2 * pr.P.pre_ps + k0 + mu + far;
                        float x[16];  // ONE: the numerators of 16 columns
#pragma unroll
                        for (int c0 = 0; c0 < NCM; c0 += CH) {
                            if (c0 < NC) {
                                if constexpr (ONE) {
                                    if (c0 % 16 == 0) {  // (a tile of 32 lag blocks reads 8 columns too many)
                                        tmem_ld16(lane_base + 128u * (hc & 1) + a0 + c0, x);
                                        float small[16];
                                        if (pairs)
                                            tmem_ld16(lane_base + 256u + 128u * (c & 1) + a0 + c0, small);
                                        tmem_wait_ld();
                                        if (pairs) {
#pragma unroll
                                            for (int i = 0; i < 16; i++)
                                                x[i] = fmaf(small[i], B.lo_unit, x[i]);
                                        }
                                        if (c0 + 16 >= NC) {  // the accumulators are read
                                            tc_fence_before();
                                            __syncwarp();
                                            if (lane == 0) {
                                                mbar_arrive(bar + TcBars::hempty + 8 * (hc & 1));
                                                if (pairs)
                                                    mbar_arrive(bar + TcBars::sempty + 8 * (c & 1));
                                            }
                                        }
                                    }
                                }
                                long long lo[CH], hi[CH];
                                float2 lo1[CH], hi1[CH];
                                if constexpr (FULL) {
#pragma unroll
                                    for (int j = 0; j < CH; j++) {
                                        lo[j] = __ldg(pr.P.pre2q + g1 + (c0 + j) * TC_Q);
                                        hi[j] = __ldg(pr.P.pre2q + g2 + (c0 + j) * TC_Q);
                                        lo1[j] = __ldg(pr.P.pre1f + g1 + (c0 + j) * TC_Q);
                                        hi1[j] = __ldg(pr.P.pre1f + g2 + (c0 + j) * TC_Q);
                                    }
                                } else {
                                    const int es = ec & ((1 << stat_log2) - 1);
                                    if (!mbar_wait_all(bar + TcBars::efull + 8 * es, (ec >> stat_log2) & 1,
                                                       abort_flag, B.err, 16u))
                                        goto epilogue_done;
                                    const uint8_t *slot = smem + (e_base - w_base) + es * (uint32_t)B.stat_bytes +
                                                          cgroup * kStatPart;
                                    const uint8_t *at = slot + (head + b) * 8,
                                                  *at2 = slot + G * kStatPart + (head2 + b) * 8;
#pragma unroll
                                    for (int j = 0; j < CH; j++) {
                                        lo[j] = *reinterpret_cast<const long long *>(at + j * TC_Q * 8);
                                        hi[j] = *reinterpret_cast<const long long *>(at2 + j * TC_Q * 8);
                                    }
                                    fence_reads_before_copy();
                                    __syncwarp();
                                    if (lane == 0)
                                        mbar_arrive(bar + TcBars::eempty + 8 * es);
                                    ec++;
                                }
                                // (outside the valid lags the sums are anything, and are not used)
                                float y[CH];
#pragma unroll
                                for (int j = 0; j < CH; j++) {
                                    float ssd, num1;
                                    if constexpr (ONE)
                                        num1 = x[(c0 + j) % 16];
                                    else
                                        num1 = num[c0 + j];
                                    if constexpr (FULL) {
                                        float mean;
                                        window_centred(lo[j], hi[j], u2, lo1[j], hi1[j], nf, inv_n, ssd, mean);
                                        num1 = fmaf(-mean, ts, num1);
                                    } else {
                                        ssd = window_energy(lo[j], hi[j], u2);
                                    }
                                    const float pe = sst * ssd, r = rsqrt_ftz(pe);
                                    y[j] = (pe * r > kThreshold ? num1 * (r * unit) : 0.0f) - 10.0f * FLT_EPSILON;
                                }
                                fisher_atanh<CH>(y);
#pragma unroll
                                for (int j = 0; j < CH; j++)
                                    sum[c0 + j] = fmaf(y[j], zw, sum[c0 + j]);
                            }
                        }
                    } else {
#pragma unroll
                        for (int c0 = 0; c0 < NCM; c0 += CH) {
                            if (c0 < NC) {
                                const int es = ec & ((1 << stat_log2) - 1);
                                if (!mbar_wait_all(bar + TcBars::efull + 8 * es, (ec >> stat_log2) & 1, abort_flag,
                                                   B.err, 16u))
                                    goto epilogue_done;
                                const uint8_t *at = smem + (e_base - w_base) + es * (uint32_t)B.stat_bytes +
                                                    cgroup * kStatPart + (head + b) * (FULL ? 8 : 4);
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
                                                mbar_arrive(bar + TcBars::eempty + 8 * es);
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
                                                oc[a * oc_step] = cc * unit;
                                        }
                                    }
                                }
                                ec++;
                            }
                        }
                    }
                    if (ONE)
                        hc++;
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

// ------------------------------------------------------------------ self-tests
// every lane of every warp takes part (the tail reads a dummy value)
__global__ void fisher_atanh_kernel(const float *__restrict__ y, float *__restrict__ out, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float r[1] = {i < n ? y[i] : 0.0f};
    fisher_atanh<1>(r);
    if (i < n)
        out[i] = r[0];
}

int launch_fisher_atanh(const float *y, float *out, long long n, cudaStream_t s)
{
    if (n <= 0)
        return FMF_OK;
    fisher_atanh_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(y, out, n);
    count_launch();
    return check_launch("fisher_atanh_kernel");
}

// Self-test of the bounded waits: one CTA waits on an mbarrier that nothing
// ever arrives on; the wait must give up after `limit_ns`, raise code 128 in
// the error word and return, leaving the context usable.
__global__ void wait_selftest_kernel(unsigned *err, unsigned long long limit_ns)
{
    __shared__ __align__(8) unsigned long long bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0)
        mbar_wait(smem_u32(&bar), 0, &abort_flag, err, 128u, limit_ns);
    __syncthreads();
}

int launch_wait_selftest(unsigned *err, unsigned ms, cudaStream_t s)
{
    wait_selftest_kernel<<<1, 32, 0, s>>>(err, (unsigned long long)ms * 1000000ull);
    count_launch();
    return check_launch("wait_selftest_kernel");
}

// ------------------------------------------------------------------ host side
// Largest tile (lag blocks per CTA tile) whose channel operands, twice over, fit in
// shared memory; 0: none.
int tc_choose_nb(int L, int step, int pairs, int forced)
{
    const int cands[3] = {128, 64, 32};
    for (int i = 0; i < 3; i++) {
        if (forced && cands[i] != forced)
            continue;
        if (2 * tc_shape(L, step, pairs, cands[i]).stage + 256 <= 227 * 1024)
            return cands[i];
    }
    return 0;
}

static int n_sms()
{
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
        n = 148;
    cudaGetLastError();
    return n;
}

// out[i] = sum over parts j = 0..k-1 of part[j][i], in that order; with
// per-channel lengths (norm set) the Fisher-z transform of that sum,
// (tanh(v / norm[t]) + bias[t]) * scale[t] for row t = i / n_corr.  Bound by the loads'
// latency: eight parts' values are in flight (one after the other: 12 us for 13 x 115,115
// outputs, 8 us here).  Added by whichever part came last in the persistent kernel
// itself, they held up its end instead: 0.27 -> 0.39 ms of the search.
__global__ void tc_parts_sum_kernel(const float *__restrict__ part, int k, long long m, int n_corr,
                                    const float *__restrict__ norm, const float *__restrict__ bias,
                                    const float *__restrict__ scale, float *__restrict__ out)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m)
        return;
    constexpr int kLoads = 8;
    float v = 0.0f;
    for (int j0 = 0; j0 < k; j0 += kLoads) {
        float x[kLoads];
#pragma unroll
        for (int j = 0; j < kLoads; j++)
            if (j0 + j < k)
                x[j] = __ldg(part + (size_t)(j0 + j) * m + i);
#pragma unroll
        for (int j = 0; j < kLoads; j++)
            if (j0 + j < k)
                v = j0 + j == 0 ? x[j] : v + x[j];
    }
    if (norm) {
        const int t = (int)(i / n_corr);
        v = (tanhf(v / norm[t]) + bias[t]) * scale[t];
    }
    out[i] = v;
}

// Channel parts k (1..32, at most SC) for a search of `items` (tile, template)
// items: the k that minimises the busiest SM's work, ceil(k items / SMs)
// rounds of (1/k + 0.05) item each (0.05: an item's fixed pipeline fill and
// output write), within 5 % of the best k in thirteen searches of 6 to 400 items.  (One
// template x 60 channels x 300 taps x 3,000 samples: 70 us in 8 parts, 56 in 16, 50 in
// 32.)  FMF_TC_PARTS=k forces a value.
static int choose_parts(long long items, int SC)
{
    const int sms = n_sms(), kmax = SC < TC_MAX_PARTS ? SC : TC_MAX_PARTS;
    if (const char *env = getenv("FMF_TC_PARTS")) {
        const int k = atoi(env);
        if (k >= 1)
            return k < kmax ? k : kmax;
    }
    int best = 1;
    double best_cost = 1e300;
    for (int k = 1; k <= kmax; k++) {
        const long long rounds = (k * items + sms - 1) / sms;
        const double cost = (double)rounds * (1.0 / k + 0.05);
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best = k;
        }
    }
    return best;
}

// Shared memory of one launch: two template buffers, two statistics slots (32 KB
// each: half a channel of a full tile) and as many data slots as fit (a channel
// has 4); long templates give up a statistics slot first.
static size_t tc_layout(TcLaunch *B, int nb, bool var, bool full)
{
    const StatSlot slot(var, full);
    const size_t fixed = 2 * (size_t)B->w_bytes + TcBars::bytes;
    B->stat_bytes = (int)slot.bytes();
    if (slot.streams == 1 && nb / 2 < slot.columns)  // (the second group lies part() bytes on)
        B->stat_bytes = (int)(slot.part() + nb / 2 * TC_Q * slot.elem + 16);
    for (int least = 3; least >= 1; least--)
        for (B->stat_log2 = 1; B->stat_log2 >= 0; B->stat_log2--) {
            const size_t stats = (size_t)B->stat_bytes << B->stat_log2;
            if (fixed + stats > (size_t)kMaxDynamicSmem)
                continue;
            const size_t rows = (kMaxDynamicSmem - fixed - stats) / B->row_bytes;
            B->n_rows = rows < (size_t)TC_MAX_ROWS ? (int)rows : TC_MAX_ROWS;
            if (B->n_rows >= least) {
                const size_t smem = fixed + stats + (size_t)B->n_rows * B->row_bytes;
                return smem < 120 * 1024 ? 120 * 1024 : smem;  // one CTA per SM: its TMEM is all there is
            }
        }
    return 0;
}

// What a search asks of the shared memory of a launch it is in.
static void tc_add_needs(TcLaunch *B, int *nb, const TcProb &pr, int form)
{
    const int halves = form != TC_FORM_BF16 ? 2 : 1;
    B->w_bytes = max(B->w_bytes, halves * pr.NW * 128);
    B->row_bytes = max(B->row_bytes, halves * 4 * pr.R * 16);
    *nb = max(*nb, pr.nb);
}

// The members of the next launch among n searches of one mode: the first that is not
// `taken` yet and those after it, in order, that share a launch with it -- at most
// TC_MAX_PROBS.  The buffers are as large as the largest member's, so a search stays out
// that would leave fewer than three data slots (a long template beside a large tile: a
// bf16 search of 5,600 taps and one of 600 leave none).
int tc_group(const TcProb *probs, int n, int form, unsigned char *taken, int *members)
{
    TcLaunch B = {};
    int nb = 0, count = 0;
    for (int i = 0; i < n && count < TC_MAX_PROBS; i++) {
        if (taken[i])
            continue;
        TcLaunch with = B;
        int with_nb = nb;
        tc_add_needs(&with, &with_nb, probs[i], form);
        const Problem &P = probs[i].P;
        if (count && (tc_layout(&with, with_nb, P.ntap != nullptr, P.normalize != 0) == 0 || with.n_rows < 3))
            continue;
        B = with;
        nb = with_nb;
        taken[i] = 1;
        members[count++] = i;
    }
    return count;
}

// Channel parts of a prepared search run by itself (tc_run).  A lone search with
// fewer (tile, template) items than SMs runs each item as k channel parts
// (network sum only; with per-channel lengths the parts add raw Fisher-z sums
// and the transform follows the addition), k chosen to shorten the busiest
// SM's queue.  FMF_TC_PARTS=k overrides the choice where parts are allowed.
int tc_choose_parts(const TcProb *prob)
{
    const Problem &P = prob->P;
    return P.SC >= 2 ? choose_parts((long long)prob->n_tiles * P.T, P.SC) : 1;
}

template <int N>
static void (*tc_kernel(int form, bool var, bool full, bool nsum))(const TcBatch<N>)
{
    if constexpr (N == 1) {  // (no batch holds searches of per-channel lengths)
        if (var && form == TC_FORM_FP32)
            return full ? tc_persistent<true, true, true, false, 1> : tc_persistent<true, false, true, false, 1>;
        if (var)
            return full ? tc_persistent<true, true, true, true, 1> : tc_persistent<true, false, true, true, 1>;
    }
    if (nsum)
        return full ? tc_persistent<false, true, true, false, N> : tc_persistent<false, false, true, false, N>;
    return full ? tc_persistent<false, true, false, false, N> : tc_persistent<false, false, false, false, N>;
}

// One persistent launch over the tile queue of `n` prepared searches (n <= N).
// `form`: the operands they were prepared with.  `queue`: a device counter, zero before
// the launch.  `parts`: channel parts of every item (n = 1 only).
template <int N>
static int tc_run_n(const TcProb *probs, int n, int form, int parts, unsigned long long *queue, unsigned *err,
                    cudaStream_t s)
{
    static thread_local TcBatch<N> Bh;  // large; built on the host for the launch only
    TcBatch<N> &B = Bh;
    const Problem &P0 = probs[0].P;
    const bool var = P0.ntap != nullptr, full = P0.normalize != 0, nsum = P0.network_sum != 0;
    Scratch pws(s);
    float *part_out = nullptr;
    if (parts > 1 && nsum && pws.get(&part_out, (size_t)parts * P0.T * P0.n_corr, "channel-part sums")) {
        set_error(FMF_OK, "");  // no memory: in one part
        part_out = nullptr;
        parts = 1;
    }
    B.split = form != TC_FORM_BF16;  // operand pairs
    B.mma_types = form == TC_FORM_FP32 ? 0u : (1u << 7) | (1u << 10);
    B.lo_unit = form == TC_FORM_FP32 ? 1.0f / kLoScale : 1.0f;
    B.w_bytes = B.row_bytes = 0;
    int nb = 0;
    long long items = 0;
    for (int i = 0; i < n; i++) {
        const Problem &P = probs[i].P;
        if ((P.ntap != nullptr) != var || (P.normalize != 0) != full || (P.network_sum != 0) != nsum)
            return set_error(FMF_ERR_ARG, "a persistent launch mixes kinds of search");
        B.prob[i] = probs[i];
        B.prob[i].item_begin = items;
        B.prob[i].parts = parts;
        B.prob[i].part_out = part_out;
        items += (long long)probs[i].n_tiles * P.T * parts;
        tc_add_needs(&B, &nb, probs[i], form);
    }
    B.n_probs = n;
    B.total_items = items;
    B.queue = queue;
    B.err = err;
    const size_t smem = tc_layout(&B, nb, var, full);
    if (smem == 0)
        return set_error(FMF_ERR_SMEM, "tensor-core buffers do not fit shared memory");
    if (N > 1 && var)
        return set_error(FMF_ERR_ARG, "a batch of searches of per-channel lengths");
    void (*kern)(const TcBatch<N>) = tc_kernel<N>(form, var, full, nsum);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
    if (e != cudaSuccess)
        return set_error(FMF_ERR_CUDA, "tc_persistent shared memory (%zu bytes): %s", smem,
                         cudaGetErrorString(e));
    const unsigned grid = (unsigned)(items < n_sms() ? (items > 0 ? items : 1) : n_sms());
    kern<<<grid, tc_threads(var), smem, s>>>(B);
    count_launch();
    note_bounded_waits();
    int rc = check_launch("tc_persistent");
    if (rc || !part_out)
        return rc;
    const long long m = (long long)P0.T * P0.n_corr;
    tc_parts_sum_kernel<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(part_out, parts, m, P0.n_corr,
                                                                     var ? P0.vp_norm : nullptr,
                                                                     P0.vp_bias, P0.vp_scale, P0.out);
    count_launch();
    return check_launch("tc_parts_sum_kernel");
}

int tc_run(const TcProb *probs, int n, int form, int parts, unsigned long long *queue, unsigned *err, cudaStream_t s)
{
    if (n < 1 || n > TC_MAX_PROBS)
        return set_error(FMF_ERR_ARG, "a persistent launch takes 1..%d searches", TC_MAX_PROBS);
    return n == 1 ? tc_run_n<1>(probs, n, form, parts, queue, err, s)
                  : tc_run_n<TC_MAX_PROBS>(probs, n, form, parts, queue, err, s);
}

size_t tc_prob_size() { return sizeof(TcProb); }

// Templates [t0, t0 + nt) of a search, as a search of its own (every
// template-indexed pointer offset but the operand blocks; data streams shared).
static void tc_subset(const TcProb *full, int t0, int nt, TcProb *out)
{
    TcProb q = *full;
    const size_t SC = q.P.SC;
    const size_t o = (size_t)t0 * SC;
    q.P.tpl += o * q.P.L;
    q.P.sst += o;
    if (q.P.tsum)
        q.P.tsum += o;
    q.P.mo += o;
    q.P.w += o;
    q.P.k_lo += t0;
    q.P.k_hi += t0;
    if (q.P.ntap)
        q.P.ntap += o;
    if (q.P.zweight)
        q.P.zweight += o;
    if (q.P.vp_norm) {
        q.P.vp_norm += t0;
        q.P.vp_bias += t0;
        q.P.vp_scale += t0;
    }
    q.P.out += (size_t)t0 * q.P.n_corr * (q.P.network_sum ? 1 : SC);
    q.P.T = nt;
    if (q.t_exp)
        q.t_exp += o;
    *out = q;
}

struct TcSearch {
    TcProb pr;       // of all templates; the operand blocks hold `room` of them
    int form, room, parts;
    TcDataWork data;
    bool data_due;   // the data streams are made with the first templates
    unsigned long long *queue;
    uint16_t *w;
    size_t w_elems;  // of one half, all room templates
};

constexpr size_t kOneLaunchTaps = 24 * 1024;  // bytes: 8 blocks of 256 threads per SM

size_t tc_search_size() { return sizeof(TcSearch); }

// Operand blocks of one part of the templates take at most this much memory, and so do
// their per-channel outputs on the way to the caller's layout.
constexpr size_t kMaxTemplateBytes = (size_t)4 << 30, kMaxChannelBytes = (size_t)1 << 30;

size_t tc_template_bytes(const Problem &P, int nb)
{
    return (size_t)P.T * P.SC * P.step * tc_shape(P.L, P.step, 1, nb).NW * 256;
}

// Lag blocks per tile of an FP32 search on the tensor cores, or 0: the CUDA cores.
// The latter take 21 us and what plain_us says (10 % off, over 288 searches of 1 to 64
// templates, 1 to 15 channels, 50 to 800 taps, 2,000 to 120,000 samples, step 1 and 3);
// the tensor cores' further kernels take 40 to 50 us however small the search.  They
// cross near 25 (16 templates x 1 channel x 200 taps x 30,000 samples: 30 us here, 39 us
// there) and the line is at 50, where the tensor cores are up to 1.5 times faster (16
// templates x 15 channels x 50 taps x 8,000: 89 us and 48 us; 64 templates: 230 us and
// 85 us): searches below it run the very kernels of the entry point without
// allocations, and launch as many.  Taken by this rule the 288 are within 2 % of the
// faster side on average.  The tile: one of 64 or
// 32 where the outputs would leave most of a larger one empty (4 templates x 15
// channels x 50 taps, 651 outputs: 55, 56, 58 us with 32, 64, 128; 39,984 outputs: 86,
// 75, 70 us).
//
// Below kFp32LeastTaps the pairs' 22 bits show: the RMS error against 64 bits is 1.4 of the
// FMAs' at 10 taps, 1.08 at 40, 1.00 at 44 to 52 and falls to 0.4 at 300 (random searches; at
// matches tc_chains keeps it below theirs).
int tc_fp32_nb(size_t T, size_t SC, size_t L, size_t step, size_t n_corr)
{
    if (const char *env = getenv("FMF_TC32")) {  // 0: the CUDA cores; 32, 64, 128: this tile
        if (atoi(env) == 0)
            return 0;
        if (atoi(env) > 1)
            return tc_choose_nb((int)L, (int)step, 1, atoi(env));
    }
    if (L < kFp32LeastTaps)
        return 0;
    // a tile of 4,096 outputs per block, two blocks per SM, groups of 20 taps per phase
    const double taps = (double)step * (double)((((L + step - 1) / step + 19) / 20) * 20);
    const double tiles = (double)T * (double)((n_corr + 4095) / 4096) / 304.0;
    const double outputs = (double)T * (double)n_corr / (304.0 * 4096.0);
    // a phase's loads and barriers: 1.45 us in full tiles, 1.14 in nearly empty ones
    const double fill = std::min(1.0, (double)n_corr / 4096.0), full = (double)step * 1.45 + 1.9;
    const double phases = fill * full + (1.0 - fill) * std::min(full, (double)step * 1.14 + 3.6);
    const double plain_us = (double)SC * ((taps * 0.0165 + phases) * (tiles < 1.0 ? 1.0 : tiles) +
                                          taps * 0.03 * (step > 3 ? outputs : tiles));
    if (plain_us < 50.0)
        return 0;
    const int want = n_corr > 8192 ? 128 : (n_corr > 4096 ? 64 : 32);
    int nb = 0;
    for (int i = want; i >= 32 && !nb; i >>= 1)
        nb = tc_choose_nb((int)L, (int)step, 1, i);
    if (!nb)
        return 0;
    // Many templates of few lags: a tile holds little, and each costs 2.7 us and more per
    // channel and phase.  (100 templates x 9 channels x 300 lags, step 20, 300 taps: 319 us
    // on the CUDA cores, 397 here; 10 templates x 3 channels 128 and 114; the line is within
    // 10 % of the faster side in 240 searches of steps 3 to 200.)
    // Rounds of whole items on the busiest SM, in the channel parts of all templates, a
    // roomful of templates at a time (few at large steps, whose operand blocks are large).
    const size_t per_template = SC * step * (size_t)tc_shape((int)L, (int)step, 1, nb).NW * 256;
    const long long room = std::min((long long)T, std::max(1ll, (long long)(kMaxTemplateBytes / per_template)));
    const long long n_tiles = (long long)((n_corr + 128 * (size_t)nb - 1) / (128 * (size_t)nb));
    const long long k = choose_parts((long long)T * n_tiles, (int)SC);
    const double rounds = (double)((T + room - 1) / room) * (double)((k * room * n_tiles + 151) / 152) / (double)k;
    const double used = (double)std::min(step, L), tc_us = 50.0 + rounds * (double)SC * used * (2.7 + 0.0066 * (double)L / used);
    return plain_us + 21.0 < tc_us ? 0 : nb;
}

// h h chains of a channel of an FP32 search, and the K steps (least of the pairs') past
// which a column-block pair is several.  Of a pair's steps, (taps + 15) / 128 add something
// to an output, and chains of m such steps are off by some 0.6e-7 m at a perfect match (the
// header of this file; of unequal ones m is the mean over the steps); multiply-adds of L
// taps in a row by 1.65e-8 sqrt(L), RMS.  m up to 0.24 sqrt(L) - 0.35 keeps the former below
// the latter.
static int tc_chains(int L, int step, int *chain_steps)
{
    const double most = 0.24 * std::sqrt((double)L) - 0.35, per_pair = ((L + step - 1) / step + 15) / 128.0;
    *chain_steps = (int)std::ceil(most < 1.0 ? 1.0 : most);
    const long long pairs = (long long)tc_phases(step, L) * (TC_CB / 2);
    for (long long n = 1; n < pairs; n++) {  // n chains: `longer` of them have a pair more
        const long long each = pairs / n, longer = pairs - each * n;
        const double mean = (double)(longer * (each + 1) * (each + 1) + (n - longer) * each * each) / (double)pairs;
        if (mean * per_pair <= most)
            return (int)n;
    }
    return (int)pairs;
}

// Per-channel outputs of at least so many channels go through an array of their own and
// are turned; of fewer, the caller's array takes them with little waste, as the lags beside
// one another fill its sectors.  Turned and in place, 20 templates, 40M outputs in all, 60
// taps, FP32: 1 channel 938 and 223 us, 3 channels 574 and 251, 8 channels 379 and 326, 10
// channels 340 and 361, 36 channels 288 and 420; the bf16 forms and 4M outputs cross there
// too.
constexpr int kTurnLeast = 10;

// Begins a search: data streams of `form`, and room for the operand blocks of up to
// max_templates templates at a time.  The statistics of P (running sums, with
// per-channel lengths) have a tile of padding round them; FP32 needs P.scan.  turn:
// per-channel outputs go through an array of their own (channel_outputs_kernel).
int tc_begin(const Problem &P, int form, int nb, int tg, int max_templates, Scratch &ws, cudaStream_t s,
             TcSearch *out, bool turn)
{
    int rc;
    const int step = P.step, SC = P.SC;
    const bool pairs = form != TC_FORM_BF16, fp32 = form == TC_FORM_FP32;
    const size_t halves = pairs ? 2 : 1;
    TcProb &pr = out->pr;
    const TcShape g = tc_fill_shape(P, pairs, nb, tg, &pr);
    const size_t per_template = (size_t)SC * step * g.NW * 64;  // one half
    size_t room = kMaxTemplateBytes / (2 * halves * per_template);
    room = room < 1 ? 1 : room;
    room = room < (size_t)max_templates ? room : (size_t)max_templates;
    const size_t turned = P.network_sum || !turn || SC < kTurnLeast ? 0 : (size_t)SC * P.n_corr;  // of a template
    if (turned) {
        const size_t most = kMaxChannelBytes / (turned * sizeof(float));
        room = most < 1 ? 1 : (most < room ? most : room);
    }
    const size_t g_elems = (size_t)SC * step * TC_CB * pr.rows_total * 8;
    const size_t n_rows = (size_t)P.T * SC;
    out->form = form;
    out->room = (int)room;
    out->w_elems = room * per_template;
    out->parts = tc_choose_parts(&pr);
    uint16_t *g_hi = nullptr;
    int *exps = nullptr;
    if ((rc = ws.get(&g_hi, halves * g_elems, "tensor-core data streams")) ||
        (rc = ws.get(&out->w, halves * out->w_elems, "tensor-core template blocks")) ||
        (fp32 && (rc = ws.get(&exps, n_rows + SC, "operand exponents"))) ||
        (rc = ws.get(&out->queue, 1, "tile queue")))
        return rc;
    if (turned && ws.get(&pr.P.by_channel, room * turned, "per-channel outputs")) {
        set_error(FMF_OK, "");  // no room for them: written in place
        pr.P.by_channel = nullptr;
    }
    uint16_t *g_lo = pairs ? g_hi + g_elems : nullptr;
    pr.g_hi = g_hi;
    pr.g_lo = g_lo;
    pr.w_hi = out->w;
    pr.w_lo = pairs ? out->w + out->w_elems : nullptr;
    if (fp32) {
        pr.t_exp = exps;
        pr.d_exp = exps + n_rows;
        pr.skip = P.scan + 3 * SC;
        if (out->room < P.T) {
            tc_template_check_kernel<<<(unsigned)n_rows, 128, 0, s>>>(P.tpl, P.L, P.scan + 3 * SC);
            count_launch();
            if ((rc = check_launch("tc_template_check_kernel")))
                return rc;
        }
    }
    // The bf16 pairs' own rounding (4.4e-6 of a product) is far above a channel-long chain's
    pr.chains = fp32 ? tc_chains(P.L, step, &pr.chain_steps) : 0;
    TcDataWork &d = out->data;
    d = TcDataWork{P.data, P.N, SC, step, 0, pr.rows_total, pr.row_front, fp32 ? P.scan : nullptr, g_hi, g_lo,
                   fp32 ? exps + n_rows : nullptr, fp32 ? P.scan + 3 * SC : nullptr, P.ntap && P.normalize == 0};
    const int rows = tc_turn_rows(step);
    d.tiles = (pr.rows_total + rows - 1) / rows;
    out->data_due = step <= TC_TURN_STEP && (long long)d.tiles * SC < (1ll << 30);
    if (out->data_due)  // with the first templates
        return FMF_OK;
    const long long n = (long long)SC * step * TC_CB * pr.rows_total;
    auto kern = fp32 ? tc_data_sparse_kernel<true> : tc_data_sparse_kernel<false>;
    kern<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(P.data, P.N, SC, step, pr.rows_total, pr.row_front, d.stat,
                                                     g_hi, g_lo, d.d_exp, d.skip, d.keep);
    count_launch();
    return check_launch("tensor-core data streams");
}

// Operand blocks of templates [t0, t0 + nt), nt <= room, into the search's
// buffer; *sub is that part of the search.
static int tc_templates(TcSearch *full, int t0, int nt, unsigned long long *queue, cudaStream_t s, TcProb *sub)
{
    const Problem &P = full->pr.P;
    tc_subset(&full->pr, t0, nt, sub);
    const bool fp32 = full->form == TC_FORM_FP32;
    auto kern = fp32 ? tc_operand_kernel<true> : tc_operand_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem - 1024);
    if (e != cudaSuccess)
        return set_error(FMF_ERR_CUDA, "tc_operand_kernel shared memory: %s", cudaGetErrorString(e));
    // blocks of 2,048 16-byte pairs at least, until there are eight per SM
    const size_t rows = (size_t)nt * P.SC, most = (size_t)tc_phases(P.step, P.L) * sub->NW * 8 / 2048;
    const unsigned parts = rows >= 1216 || most < 2 ? 1u : (unsigned)std::min(most, (1216 + rows - 1) / rows);
    const TcTemplateWork w{sub->P.tpl, sub->P.mo, P.L, P.step, sub->NW, full->w,
                           const_cast<uint16_t *>(full->pr.w_lo), const_cast<int *>(sub->t_exp),
                           const_cast<unsigned *>(full->pr.skip), queue, (int)parts};
    unsigned n_data = full->data_due ? (unsigned)full->data.tiles * full->data.SC : 0;
    const unsigned n_templates = (unsigned)rows * parts;
    const size_t turn = tc_turn_bytes(P.step, full->pr.g_lo != nullptr), taps = (size_t)P.L * sizeof(float);
    // one launch (4 us less than two in a search of 50 us), unless the templates' shared
    // memory would leave room for fewer of the data's blocks
    if (n_data && (taps > kOneLaunchTaps || n_templates > (1u << 30))) {
        kern<<<n_data, 256, turn, s>>>(full->data, n_data, w);
        count_launch();
        n_data = 0;
    }
    kern<<<n_data + n_templates, 256, n_data && turn > taps ? turn : taps, s>>>(full->data, n_data, w);
    full->data_due = false;
    count_launch();
    return check_launch("tensor-core operands");
}

// Templates [t0, t0 + nt) of a begun search: their operand blocks and the
// persistent launch, a roomful at a time.  The channel parts of an FP32 search and its
// flag are those of all its templates, so that its results do not depend on how they
// are parted (a call with host arrays runs them in parts); the bf16 forms choose them
// for each launch, which keeps the SMs busier through the last few templates.
int tc_run_templates(TcSearch *full, int t0, int nt, unsigned *err, cudaStream_t s)
{
    int rc;
    for (int a = t0; a < t0 + nt; a += full->room) {
        const int n = t0 + nt - a < full->room ? t0 + nt - a : full->room;
        TcProb sub;
        if ((rc = tc_templates(full, a, n, full->queue, s, &sub)) ||
            (!sub.P.by_channel && (rc = clear_outputs(sub.P, s))) ||
            (rc = tc_run(&sub, 1, full->form, full->form == TC_FORM_FP32 ? full->parts : tc_choose_parts(&sub),
                         full->queue, err, s)) ||
            (sub.P.by_channel && (rc = launch_channel_outputs(sub.P, sub.skip, s))))
            return rc;
    }
    return FMF_OK;
}

// FP32: nonzero afterwards if the CUDA cores have to run the search.
const unsigned *tc_flag(const TcSearch *full) { return full->pr.skip; }

// One search of a batch: all its operands; *out is ready for a shared launch.
int tc_prepare(const Problem &P, int form, int nb, int tg, Scratch &ws, cudaStream_t s, TcProb *out)
{
    TcSearch st;
    int rc = tc_begin(P, form, nb, tg, P.T, ws, s, &st, false);
    if (rc)
        return rc;
    if (st.room < P.T) {  // a shared launch needs them all at once
        const size_t halves = form != TC_FORM_BF16 ? 2 : 1;
        st.w_elems = st.w_elems / st.room * P.T;
        st.room = P.T;
        if ((rc = ws.get(&st.w, halves * st.w_elems, "tensor-core template blocks")))
            return rc;
        st.pr.w_hi = st.w;
        st.pr.w_lo = halves == 2 ? st.w + st.w_elems : nullptr;
    }
    return tc_templates(&st, 0, P.T, nullptr, s, out);
}

}  // namespace fmf
