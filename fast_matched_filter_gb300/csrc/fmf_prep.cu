// fmf_prep.cu -- per-call preprocessing kernels.
//
//  * template_scalars_kernel : valid output range [k_lo, k_hi) of each template
//    (reference: matched_filter.c:53-76 start/stop, matched_filter.cu:302-308
//    n_corr_t), and the template energies sum(t^2) when the caller
//    passes none, computed as the reference wrapper computes them for
//    float32 templates (numpy.sum(templates**2, axis=-1),
//    fast_matched_filter.py:256-261): float32 squares summed in numpy's
//    pairwise order, so the values are bit-identical.
//  * template_center_kernel: "full" only -- template minus its FP64 mean and
//    the FP64 sum of the centred values.  sum(t*(d-m)) equals
//    sum((t-tbar)*(d-m)) exactly, so centring changes no result; it removes
//    the template's DC term from the products the numerator sums.
//  * channel_centre_kernel : "full" only -- the constant subtracted from each
//    data channel, the median of evenly spaced samples (robust to transients).
//  * window_stats_kernel   : sliding-window statistics of every channel for
//    windows of L samples starting at each sample index:
//      short: E = sum d^2                      (matched_filter.c:622)
//      full : m = sum d'/L, V = sum d'^2 - (sum d')^2/L   (d' = d - mu)
//    each window's sums composed from parts inside the window (the end of
//    its first 32-sample chunk, whole chunks, the start of its last chunk) in
//    double-float FP32 arithmetic, so that no window sum is the difference of
//    running sums and a large transient before a quiet window costs it no
//    digits (the reference's FP64 running sums lose 2^-53 of everything summed
//    before the window, matched_filter.c:29-31, 660-705).
#include "fmf_common.cuh"

namespace fmf {

__device__ __forceinline__ double block_sum_f64(double v, double *red)
{
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, o);
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0)
        red[wid] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0) {
        for (int i = 0; i < (int)(blockDim.x >> 5); i++)
            s += red[i];
        red[32] = s;
    }
    __syncthreads();
    return red[32];
}

// numpy's float32 pairwise sum of the squares of a[0:n) (the reduction
// numpy.sum applies along a contiguous axis): fewer than 8 values -- a running
// sum from -0; up to 128 -- eight interleaved partial sums, combined as
// ((r0 + r1) + (r2 + r3)) + ((r4 + r5) + (r6 + r7)), then the values past the
// last multiple of 8 in order; more -- the sum of the two halves split at n/2
// rounded down to a multiple of 8.  Explicit round-to-nearest operations: no
// fused multiply-add may change a rounding.
//
// One warp per row.  The eight partial sums of a block of up to 128 values are
// eight lanes, combined by exchanges in the same order, so a warp sums four
// blocks at a time; lane 0 then adds the blocks up the split tree.  (A thread
// per row walked the whole row: 7.6 us for rows of 100 values, against 3 us.)
constexpr int kEnergyLeaves = 256;  // blocks of one round; a block has at least 57 values

// numpy's recursion over n values as a walk: the leaves in order, and after each how many
// finished pairs to add (bits of its path).
struct PairwiseWalk {
    int off[32], len[32];   // right halves still to come, the innermost last
    int n_off = 0, o, m;    // the next node, none if m is 0
    unsigned in_right = 0;  // whether it lies in the right half of its parent (bit 0), of that one's, ...
    __device__ explicit PairwiseWalk(int n) : o(0), m(n) {}
    // The next leaf; false after the last.
    __device__ bool next(int &leaf, int &size, int &adds)
    {
        if (m == 0)
            return false;
        while (m > 128) {
            const int half = m / 2 - m / 2 % 8;
            off[n_off] = o + half;
            len[n_off++] = m - half;
            m = half;
            in_right <<= 1;
        }
        leaf = o;
        size = m;
        adds = __ffs(~in_right) - 1;  // halves that this leaf ends
        in_right >>= adds;
        m = 0;
        if (n_off) {
            o = off[--n_off];
            m = len[n_off];
            in_right |= 1;
        }
        return true;
    }
};

// The squares of a[0:n), n <= 128, by 8 lanes (k = 0..7) of a warp.
__device__ __forceinline__ float pairwise_leaf_sq(const float *a, int n, int k)
{
    if (n < 8) {
        float r = -0.0f;
        for (int i = 0; i < n; i++)
            r = __fadd_rn(r, __fmul_rn(a[i], a[i]));
        return r;
    }
    const int whole = n - (n % 8);
    float r = __fmul_rn(a[k], a[k]);
#pragma unroll 4
    for (int i = 8; i < whole; i += 8)
        r = __fadd_rn(r, __fmul_rn(a[i + k], a[i + k]));
    const unsigned group = 0xffu << (threadIdx.x & 24);
    for (int o = 1; o < 8; o <<= 1)  // addition commutes: every lane ends with lane 0's sum
        r = __fadd_rn(r, __shfl_xor_sync(group, r, o));
    for (int i = whole; i < n; i++)
        r = __fadd_rn(r, __fmul_rn(a[i], a[i]));
    return r;
}

// One warp: the energy of row r of L values, in lane 0.
__device__ __forceinline__ float row_energy(const float *a, int L)
{
    __shared__ float leaf[4][kEnergyLeaves];
    __shared__ int at[4][kEnergyLeaves];              // first value of the block
    __shared__ unsigned char size[4][kEnergyLeaves];  // and how many: 128 at most
    __shared__ unsigned char ends[4][kEnergyLeaves];  // pairs to add after the block
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float stack[32];
    int sp = 0, here;
    PairwiseWalk walk(L);
    do {  // a round of blocks
        int n = 0;
        if (lane == 0) {
            int o, m, adds;
            for (; n < kEnergyLeaves && walk.next(o, m, adds); n++) {
                at[w][n] = o;
                size[w][n] = (unsigned char)m;
                ends[w][n] = (unsigned char)adds;
            }
        }
        here = __shfl_sync(0xffffffffu, n, 0);
        __syncwarp();
        for (int j = lane >> 3; j < here; j += 4) {
            const float v = pairwise_leaf_sq(a + at[w][j], size[w][j], lane & 7);
            if ((lane & 7) == 0)
                leaf[w][j] = v;
        }
        __syncwarp();
        if (lane == 0)
            for (int j = 0; j < here; j++) {
                float v = leaf[w][j];
                for (int q = ends[w][j]; q > 0; q--)
                    v = __fadd_rn(stack[--sp], v);
                stack[sp++] = v;
            }
        __syncwarp();
    } while (here == kEnergyLeaves);
    return stack[0];
}

// Everything that is made of the templates' scalars, in one launch of 128 threads per
// block.  The first blocks, if rows > 0: a warp per row (template, channel), its
// energy into sst (tpl set) and the largest one of each channel into scan (if
// set).  The other blocks, if T > 0: a thread per template, its valid lags.
__global__ void __launch_bounds__(128) template_scalars_kernel(
    const float *__restrict__ tpl, float *__restrict__ sst, int rows, int L, unsigned *__restrict__ scan,
    const int *__restrict__ mo, int T, int SC, int N, int step, int n_corr, int *__restrict__ k_lo,
    int *__restrict__ k_hi)
{
    const int row_blocks = (int)((rows + 3ll) / 4);
    if ((int)blockIdx.x < row_blocks) {
        const int r = blockIdx.x * 4 + (threadIdx.x >> 5);
        if (r >= rows)
            return;
        const float e = tpl ? row_energy(tpl + (size_t)r * L, L) : sst[r];
        if ((threadIdx.x & 31) == 0) {
            if (tpl)
                sst[r] = e;
            if (scan && e > 0.0f)  // NaN left out: such a channel's coefficients are all 0
                atomicMax(scan + 2 * SC + r % SC, __float_as_uint(e));
        }
        return;
    }
    const int t = (blockIdx.x - row_blocks) * blockDim.x + threadIdx.x;
    if (t >= T)
        return;
    int lo = 0, hi = 0;
    const int *m = mo + (size_t)t * SC;
    for (int ch = 0; ch < SC; ch++) {
        lo = min(lo, m[ch]);
        hi = max(hi, m[ch]);
    }
    long long first = lo < 0 ? ((long long)(-lo) + step - 1) / step : 0;
    long long last = (long long)N - L - hi;
    long long a = 0, b = 0;
    if (last >= 0) {
        b = last / step + 1;
        if (b > n_corr)
            b = n_corr;
        a = first < b ? first : b;
    }
    k_lo[t] = (int)a;
    k_hi[t] = (int)b;
}

void launch_template_scalars(const float *tpl, float *sst, int rows, int L, unsigned *scan, const int *mo,
                             int T, int SC, int N, int step, int n_corr, int *k_lo, int *k_hi, cudaStream_t s)
{
    const unsigned blocks = (unsigned)((rows + 3ll) / 4 + (T + 127) / 128);
    template_scalars_kernel<<<blocks, 128, 0, s>>>(tpl, sst, rows, L, scan, mo, T, SC, N, step, n_corr, k_lo, k_hi);
    count_launch();
}

// check_zeros count of the reference wrapper (fast_matched_filter.py:322-361)
// on the device: counts[t] += number of zeros among out[t][i] with
// i % last_axis < stop, over a row of row_len values.  Grid (blocks, T).
__global__ void zero_count_kernel(const float *__restrict__ out, long long row_len, long long last_axis,
                                  long long stop, unsigned long long *__restrict__ counts)
{
    const int t = blockIdx.y;
    const float *row = out + (size_t)t * row_len;
    const long long span = last_axis == row_len ? stop : row_len;  // network sum: lags < stop
    const bool all = last_axis == row_len;
    const long long stride = (long long)gridDim.x * blockDim.x;
    unsigned c = 0;
    constexpr int kLoads = 8;  // in flight (one at a time: 1 TB/s)
    for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; i0 < span; i0 += kLoads * stride) {
        float x[kLoads];
#pragma unroll
        for (int j = 0; j < kLoads; j++)
            x[j] = i0 + j * stride < span ? __ldg(row + i0 + j * stride) : 1.0f;
#pragma unroll
        for (int j = 0; j < kLoads; j++)
            c += x[j] == 0.0f && (all || (i0 + j * stride) % last_axis < stop) ? 1u : 0u;
    }
    for (int o = 16; o > 0; o >>= 1)
        c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c)
        atomicAdd(counts + t, (unsigned long long)c);
}

// Per-channel outputs (T, n_corr, SC) from the (T, SC, n_corr) array that the tensor
// cores' epilogue writes in runs of 32 lags: tiles of 64 lags x up to 64 channels
// through shared memory.  Zeros outside the valid lags and on channels of weight 0; all
// zeros if the flag leaves the search to the CUDA cores.  (Written in place, 4
// bytes per 32-byte sector, the coefficients of 8 templates x 36 channels x
// 119,601 lags took 712 us; now 119 us and 75 us here.)
constexpr int kTurnLags = 64, kTurnChannels = 64;
__global__ void __launch_bounds__(256) channel_outputs_kernel(
    const float *__restrict__ by_channel, const float *__restrict__ w, const int *__restrict__ k_lo,
    const int *__restrict__ k_hi, int T, int SC, int n_corr, const unsigned *__restrict__ flag,
    float *__restrict__ out)
{
    __shared__ float tile[kTurnChannels][kTurnLags + 1];
    const int c_tiles = (SC + kTurnChannels - 1) / kTurnChannels;
    const int k0 = (int)(blockIdx.x / c_tiles) * kTurnLags, c0 = (int)(blockIdx.x % c_tiles) * kTurnChannels;
    const int nk = min(kTurnLags, n_corr - k0), nc = min(kTurnChannels, SC - c0);
    const bool zero = flag && *flag;
    const int dk = 256 / nc, dc = 256 % nc;  // from one of a thread's elements to the next
    for (int t = blockIdx.y; t < T; t += gridDim.y) {
        const int lo = k_lo[t] - k0, hi = k_hi[t] - k0;
        __syncthreads();
        const int k = threadIdx.x & 63;
        const bool lag = !zero && k >= lo && k < hi;
        const float *src = by_channel + ((size_t)t * SC + c0) * n_corr + k0 + k;
        constexpr int kLoads = 8;  // in flight
        for (int b = threadIdx.x >> 6; b < nc; b += 4 * kLoads) {
            float x[kLoads];
#pragma unroll
            for (int j = 0; j < kLoads; j++) {
                const int c = b + 4 * j;
                x[j] = lag && c < nc && w[(size_t)t * SC + c0 + c] != 0.0f ? src[(size_t)c * n_corr] : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < kLoads; j++)
                if (b + 4 * j < nc)
                    tile[b + 4 * j][k] = x[j];
        }
        __syncthreads();
        float *o = out + ((size_t)t * n_corr + k0) * SC + c0;
        int kk = threadIdx.x / nc, cc = threadIdx.x % nc;
        for (int i = threadIdx.x; i < nk * nc; i += 256) {
            o[(size_t)kk * SC + cc] = tile[cc][kk];
            kk += dk;
            cc += dc;
            if (cc >= nc) {
                cc -= nc;
                kk++;
            }
        }
    }
}

int launch_channel_outputs(const Problem &P, const unsigned *flag, cudaStream_t s)
{
    const long long tiles = (long long)((P.n_corr + kTurnLags - 1) / kTurnLags) *
                            ((P.SC + kTurnChannels - 1) / kTurnChannels);
    if (tiles > 0x7fffffffLL)
        return set_error(FMF_ERR_ARG, "too many tiles of per-channel outputs");
    channel_outputs_kernel<<<dim3((unsigned)tiles, (unsigned)(P.T < 65535 ? P.T : 65535)), 256, 0, s>>>(
        P.by_channel, P.w, P.k_lo, P.k_hi, P.T, P.SC, P.n_corr, flag, P.out);
    count_launch();
    return check_launch("channel_outputs_kernel");
}

// grid = T*SC blocks of 128 threads
__global__ void template_center_kernel(const float *__restrict__ tpl, int L,
                                       float *__restrict__ tcen,
                                       float *__restrict__ tsum)
{
    __shared__ double red[33];
    size_t row = blockIdx.x;
    const float *src = tpl + row * L;
    float *dst = tcen + row * L;
    double s = 0.0;
    for (int j = threadIdx.x; j < L; j += blockDim.x)
        s += (double)src[j];
    double mean = block_sum_f64(s, red) / (double)L;
    float mf = (float)mean;
    double s2 = 0.0;
    for (int j = threadIdx.x; j < L; j += blockDim.x) {
        float v = src[j] - mf;
        dst[j] = v;
        s2 += (double)v;
    }
    double tot = block_sum_f64(s2, red);
    if (threadIdx.x == 0)
        tsum[row] = (float)tot;
}

// grid = SC blocks of 1024 threads: the centre c[ch] that 'full' subtracts
// from each data channel.  Any constant gives the same coefficients (the
// centred templates sum to zero, so sum t'(d - m) = sum t'(d - c - (m - c))),
// but the size of d - c sets the rounding of the numerator's products, of the
// tensor-core split most of all (2^-16 of each operand).  The channel mean
// moves with a large transient (a 1,000-sample burst at 1e3 shifts a 40,000-
// sample channel's mean by ~80 times a 1e-2 noise); the median of 8192
// evenly spaced samples stays at the level of the quiet data.  It is one of
// the samples, so d - c is exact in FP32 wherever c/2 <= d <= 2c.
//
// The sample stays in registers (8 values a thread) and its median is found by
// radix selection, 11 + 11 + 10 bits of the values' order-preserving keys; the
// first pass's bins split a binade in four, so that few lanes of a warp meet in
// one.  (A bitonic sort in shared memory took 70 us, whatever N.)
constexpr int kCentreSample = 8192;
constexpr int kCentreThreads = 1024;
__global__ void __launch_bounds__(kCentreThreads) channel_centre_kernel(const float *__restrict__ data, int N,
                                                                        float *__restrict__ centre)
{
    constexpr int PER = kCentreSample / kCentreThreads, BINS = 2048;
    __shared__ unsigned hist[BINS];
    __shared__ unsigned warp_sum[32];
    __shared__ unsigned found[2];  // bin and the rank inside it
    const float *src = data + (size_t)blockIdx.x * N;
    const int S = min(N, kCentreSample), lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned key[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const int k = threadIdx.x + j * kCentreThreads;
        const unsigned u = k < S ? __float_as_uint(src[(long long)k * N / S]) : 0x7f800000u;  // padding: +inf
        key[j] = u & 0x80000000u ? ~u : u | 0x80000000u;
    }
    unsigned rank = (unsigned)(S - 1) / 2, prefix = 0;
    const int shifts[3] = {21, 10, 0}, widths[3] = {11, 11, 10};
#pragma unroll
    for (int pass = 0; pass < 3; pass++) {
        const int shift = shifts[pass];
        const unsigned mask = (1u << widths[pass]) - 1, above = pass == 0 ? 0u : ~0u << (shift + widths[pass]);
        for (int i = threadIdx.x; i < BINS; i += kCentreThreads)
            hist[i] = 0;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < PER; j++)
            if ((key[j] & above) == (prefix & above))
                atomicAdd(&hist[(key[j] >> shift) & mask], 1u);
        __syncthreads();
        // each thread two bins: exclusive scan, then the bin that holds the rank
        const unsigned c0 = hist[2 * threadIdx.x], c1 = hist[2 * threadIdx.x + 1];
        unsigned x = c0 + c1;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            x += lane >= o ? y : 0;
        }
        if (lane == 31)
            warp_sum[wid] = x;
        __syncthreads();
        unsigned w = warp_sum[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, w, o);
            w += lane >= o ? y : 0;
        }
        const unsigned before_warp = __shfl_sync(0xffffffffu, w, wid) - warp_sum[wid];
        const unsigned before = before_warp + x - (c0 + c1);
        if (rank >= before && rank < before + c0) {
            found[0] = 2 * threadIdx.x;
            found[1] = rank - before;
        } else if (rank >= before + c0 && rank < before + c0 + c1) {
            found[0] = 2 * threadIdx.x + 1;
            found[1] = rank - before - c0;
        }
        __syncthreads();
        prefix |= found[0] << shift;
        rank = found[1];
    }
    if (threadIdx.x == 0)
        centre[blockIdx.x] = __uint_as_float(prefix & 0x80000000u ? prefix & 0x7fffffffu : ~prefix);
}

// ---------------------------------------------------------------- window statistics
// Each window's sums are composed from parts that all lie inside the window,
// never taken as the difference of running sums: with samples in 32-sample
// chunks, the window [u, u + L) is
//     (u to the end of u's chunk) + (whole chunks) + (start of the last chunk to u + L),
// each part summed in double-float FP32 arithmetic (squares split exactly by
// FMA, TwoSum additions with the rounding errors carried in the low word).
// A difference of running sums loses the digits of everything summed before
// the window -- after a large transient, a quiet window holds 1e-10 of the
// running energy -- whereas here the sums of d^2 have only non-negative parts
// (about 44 significant bits whatever came before) and the sums of d' are
// accurate to 2^-44 of the window's own sum of |d'|.

constexpr int kStatThreads = 256;
constexpr int kStatGroup = 16;  // consecutive windows per thread
static_assert(kStatWindows == kStatThreads * kStatGroup, "one group of windows per thread");

// padded shared-memory index: one spare slot per 32, so that threads 16 or 32
// samples apart hit different banks
__device__ __forceinline__ int stat_pad(int i) { return i + (i >> 5); }

// Staged samples per block: the windows' span plus a zero tail read by the last
// group's loops, a multiple of the 32-sample chunk.
__host__ __device__ __forceinline__ int stat_span(int L) { return (kStatWindows + L + 63) & ~31; }

// Shared-memory carve (in floats, each part 16-byte aligned): squares, values
// ('full'), chunk sums of both, staged outputs.
struct StatLayout {
    int s2, s1, q2, q1, out, total;
    __host__ __device__ StatLayout(int L, bool full)
    {
        const int span = stat_span(L), padded = span + (span >> 5);
        const int nq = span >> 5, pw = kStatWindows + (kStatWindows >> 5);
        auto al = [](int x) { return (x + 3) & ~3; };
        s2 = 0;
        s1 = al(s2 + 2 * padded);
        q2 = al(s1 + (full ? padded : 0));
        q1 = al(q2 + 2 * nq);
        out = al(q1 + (full ? 2 * nq : 0));
        total = al(out + (full ? 2 : 1) * pw);
    }
};

size_t window_stats_smem(int L, bool full) { return (size_t)StatLayout(L, full).total * sizeof(float); }

// A thread's windows of a block's for coalesced stores where step > 1: row by row, the
// r-th row from window 0's, its j-th window, with one division at the start instead of
// one per window.
struct WindowWalk {
    const StatPlace place;
    int per, rows, head, x0, r, j, dr, dj;
    __device__ WindowWalk(const StatPlace &p, int c0, int nwin) : place(p)
    {
        const int n = (int)blockDim.x, i = (int)threadIdx.x;
        per = nwin > 0 ? (nwin - 1) / p.step + 1 : 1;  // windows of a row
        rows = min(p.step, nwin);
        head = c0 % p.step;                          // row of window 0
        x0 = c0 / p.step;                            // and its place there
        r = i / per;
        j = i - r * per;
        dr = n / per;
        dj = n - dr * per;
    }
    __device__ bool in() const { return r < rows; }
    __device__ int window() const { return r + j * place.step; }
    __device__ long long at() const
    {
        const int wrap = head + r >= place.step, psi = head + r - (wrap ? place.step : 0);
        return psi * place.ps + min(psi, place.rem) + x0 + j + wrap;
    }
    __device__ void next()
    {
        r += dr;
        j += dj;
        if (j >= per) {
            j -= per;
            r++;
        }
    }
};

// f(u, o) for this thread's windows u of the block's nwin; o: its place in the channel
// past first_place().
__device__ __forceinline__ long long first_place(const StatPlace &place, long long c0) { return place.step == 1 ? c0 : 0; }
template <int THREADS, class F>
__device__ __forceinline__ void each_window(const StatPlace &place, long long c0, int nwin, F f)
{
    if (place.step == 1) {
        for (int u = threadIdx.x; u < nwin; u += THREADS)
            f(u, (long long)u);
    } else {
        for (WindowWalk at(place, (int)c0, nwin); at.in(); at.next())
            if (at.window() < nwin)
                f(at.window(), at.at());
    }
}

// Problem::dc of a window (u-th of its channel): every kDcStride-th one counts.
__device__ __forceinline__ float window_dc(float mx, unsigned u, float Lf, float en, float mean)
{
    return u % kDcStride == 0 && en > 0.0f ? fmaxf(mx, Lf * mean * mean / en) : mx;
}

__device__ __forceinline__ void block_dc(float mx, unsigned *word)
{
    const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
    if ((threadIdx.x & 31) == 0 && top > *(volatile unsigned *)word)
        atomicMax(word, top);
}

// A block's part of Problem::scan: one atomic per block, and only where it changes the
// channel's value.  `mem`: shared memory that is not read any more after the first
// barrier here.
__device__ __forceinline__ void scan_block(unsigned top, unsigned low, float *mem, unsigned *scan, int ch, int SC)
{
    __syncthreads();
    unsigned *red = reinterpret_cast<unsigned *>(mem);
    const int warps = blockDim.x >> 5;
    top = __reduce_max_sync(0xffffffffu, top);
    low = __reduce_max_sync(0xffffffffu, low);
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = top;
        red[32 + (threadIdx.x >> 5)] = low;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        unsigned v = 0;
        for (int i = 0; i < warps; i++)
            v = max(v, red[32 * threadIdx.x + i]);
        unsigned *word = scan + threadIdx.x * SC + ch;
        if (v > *(volatile unsigned *)word)
            atomicMax(word, v);
    }
}

// Blocks of kStatWindows windows of a channel, channel by channel (any grid): all of
// them, or those of `list` (their count, then their numbers); kStatThreads threads,
// dynamic smem = window_stats_smem(L, FULL).  short: stat_e[ch][u] = sum of d^2 over
// [u, u + L); FULL: (centred energy, mean) of d' = d - mu[ch] as float pairs,
// and the centred data into dcen.  Windows past N - L are not written.  One
// instantiation per mode: the 'short' one keeps no sums of d' in registers,
// so three blocks share an SM.
template <bool FULL, bool SCAN>
__global__ void __launch_bounds__(kStatThreads, FULL ? 2 : 3)
window_stats_kernel(const float *__restrict__ data, int N, int L, int SC, const float *__restrict__ mu,
                    float *__restrict__ dcen, float *__restrict__ stat_e, const StatPlace place,
                    unsigned *__restrict__ scan, unsigned *__restrict__ dc, const unsigned *__restrict__ list)
{
    extern __shared__ float4 stat_smem[];
    constexpr bool full = FULL;
    const StatLayout lay(L, full);
    float *base = reinterpret_cast<float *>(stat_smem);
    float2 *s2 = reinterpret_cast<float2 *>(base + lay.s2);
    float *s1 = base + lay.s1;
    float2 *q2 = reinterpret_cast<float2 *>(base + lay.q2);
    float2 *q1 = reinterpret_cast<float2 *>(base + lay.q1);
    float *out1 = base + lay.out;
    float2 *out2 = reinterpret_cast<float2 *>(base + lay.out);

    const int per_ch = (N + kStatWindows - 1) / kStatWindows;
    const unsigned n_blocks = list ? list[0] : (unsigned)per_ch * SC;
    for (unsigned item = blockIdx.x; item < n_blocks; item += gridDim.x) {
        const unsigned blk = list ? list[1 + item] : item;
        const int ch = (int)(blk / per_ch);
        const long long c0 = (long long)(blk % per_ch) * kStatWindows;
        const int len = (int)min((long long)kStatWindows + L - 1, (long long)N - c0);
        const int nwin = min(kStatWindows, len - L + 1);
        const int span = stat_span(L), nq = span >> 5;
        const float m = full ? mu[ch] : 0.0f;
        const float *src = data + (size_t)ch * N + c0;
        constexpr int kLoads = 4;  // loads in flight per thread before their use
        unsigned top = 0;          // bits of the largest finite |v|
        for (int i0 = threadIdx.x; i0 < span; i0 += kLoads * kStatThreads) {
            float x[kLoads];
#pragma unroll
            for (int j = 0; j < kLoads; j++) {
                const int i = i0 + j * kStatThreads;
                x[j] = i < len ? __ldg(src + i) : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < kLoads; j++) {
                const int i = i0 + j * kStatThreads;
                if (i < span) {
                    const float v = i < len ? x[j] - m : 0.0f;
                    if (full && i < kStatWindows && i < len)
                        dcen[(size_t)ch * N + c0 + i] = v;
                    const float sq = v * v;
                    s2[stat_pad(i)] = make_float2(sq, fmaf(v, v, -sq));  // v^2 exactly
                    if (SCAN) {
                        const unsigned av = __float_as_uint(v) & 0x7fffffffu;
                        top = av < 0x7f800000u ? max(top, av) : top;
                    }
                    if (full)
                        s1[stat_pad(i)] = v;
                }
            }
        }
        __syncthreads();
        for (int k = threadIdx.x; k < nq; k += kStatThreads) {  // chunk sums
            float h2 = 0.0f, l2 = 0.0f, h1 = 0.0f, l1 = 0.0f;
#pragma unroll 8
            for (int j = 0; j < 32; j++) {
                const float2 x = s2[stat_pad(32 * k + j)];
                pair_add(h2, l2, x.x, x.y);
                if (full)
                    pair_add(h1, l1, s1[stat_pad(32 * k + j)], 0.0f);
            }
            q2[k] = make_float2(h2, l2);
            if (full)
                q1[k] = make_float2(h1, l1);
        }
        __syncthreads();

        const float Lf = (float)L, invL = 1.0f / Lf;
        auto emit = [&](int u, float h2, float l2, float h1, float l1) {
            if (full) {
                float v, mean;
                window_centred_sums(h2, l2, h1, l1, Lf, invL, v, mean);
                out2[stat_pad(u)] = make_float2(v, mean);
            } else {
                out1[stat_pad(u)] = h2 + l2;
            }
        };
        if (L >= 32) {
            // windows u0 .. u0 + 15 of this thread: all start in chunk a and end
            // past it, so suffix (in chunk a) + whole chunks + tail never overlap
            const int u0 = threadIdx.x * kStatGroup;
            if (u0 < nwin) {
                const int a = u0 >> 5;
                float sh2[kStatGroup], sl2[kStatGroup], sh1[kStatGroup], sl1[kStatGroup];
                float h2 = 0.0f, l2 = 0.0f, h1 = 0.0f, l1 = 0.0f;
                for (int j = u0 + kStatGroup; j < 32 * a + 32; j++) {
                    const float2 x = s2[stat_pad(j)];
                    pair_add(h2, l2, x.x, x.y);
                    if (full)
                        pair_add(h1, l1, s1[stat_pad(j)], 0.0f);
                }
#pragma unroll
                for (int r = kStatGroup - 1; r >= 0; r--) {  // suffix sums, last start first
                    const float2 x = s2[stat_pad(u0 + r)];
                    pair_add(h2, l2, x.x, x.y);
                    sh2[r] = h2;
                    sl2[r] = l2;
                    if (full) {
                        pair_add(h1, l1, s1[stat_pad(u0 + r)], 0.0f);
                        sh1[r] = h1;
                        sl1[r] = l1;
                    }
                }
                const int e0 = u0 + L;  // end (exclusive) of window u0
                float mh2 = 0.0f, ml2 = 0.0f, mh1 = 0.0f, ml1 = 0.0f;  // whole chunks
                for (int k = a + 1; k < (e0 >> 5); k++) {
                    pair_add(mh2, ml2, q2[k].x, q2[k].y);
                    if (full)
                        pair_add(mh1, ml1, q1[k].x, q1[k].y);
                }
                float rh2 = 0.0f, rl2 = 0.0f, rh1 = 0.0f, rl1 = 0.0f;  // tail in the last chunk
                for (int j = e0 & ~31; j < e0; j++) {
                    const float2 x = s2[stat_pad(j)];
                    pair_add(rh2, rl2, x.x, x.y);
                    if (full)
                        pair_add(rh1, rl1, s1[stat_pad(j)], 0.0f);
                }
#pragma unroll
                for (int r = 0; r < kStatGroup; r++) {
                    const int e = e0 + r;
                    if (r > 0 && (e & 31) == 0) {  // the tail's chunk is whole: move it to the middle
                        const int k = (e >> 5) - 1;
                        pair_add(mh2, ml2, q2[k].x, q2[k].y);
                        rh2 = rl2 = 0.0f;
                        if (full) {
                            pair_add(mh1, ml1, q1[k].x, q1[k].y);
                            rh1 = rl1 = 0.0f;
                        }
                    }
                    if (u0 + r < nwin) {
                        float th2 = sh2[r], tl2 = sl2[r], th1 = 0.0f, tl1 = 0.0f;
                        pair_add(th2, tl2, mh2, ml2);
                        pair_add(th2, tl2, rh2, rl2);
                        if (full) {
                            th1 = sh1[r];
                            tl1 = sl1[r];
                            pair_add(th1, tl1, mh1, ml1);
                            pair_add(th1, tl1, rh1, rl1);
                        }
                        emit(u0 + r, th2, tl2, th1, tl1);
                    }
                    const float2 x = s2[stat_pad(e)];
                    pair_add(rh2, rl2, x.x, x.y);
                    if (full)
                        pair_add(rh1, rl1, s1[stat_pad(e)], 0.0f);
                }
            }
        } else {  // windows shorter than a chunk: direct sums
            for (int u = threadIdx.x; u < nwin; u += kStatThreads) {
                float h2 = 0.0f, l2 = 0.0f, h1 = 0.0f, l1 = 0.0f;
                for (int j = u; j < u + L; j++) {
                    const float2 x = s2[stat_pad(j)];
                    pair_add(h2, l2, x.x, x.y);
                    if (full)
                        pair_add(h1, l1, s1[stat_pad(j)], 0.0f);
                }
                emit(u, h2, l2, h1, l1);
            }
        }
        __syncthreads();
        // energies at or below this pass no template's threshold
        const float dead = SCAN ? kThreshold / __uint_as_float(scan[2 * SC + ch]) * 0.999f : 0.0f;
        unsigned low = 0;  // the smallest energy above it, bits complemented
        float mx = 0.0f;
        float *row = stat_e + (ch * place.ch + first_place(place, c0)) * (full ? 2 : 1);
        each_window<kStatThreads>(place, c0, nwin, [&](int u, long long o) {
            float en;
            if (full) {
                const float2 v = out2[stat_pad(u)];
                reinterpret_cast<float2 *>(row)[o] = v;
                en = v.x;
                if (dc)
                    mx = window_dc(mx, (unsigned)c0 + u, Lf, v.x, v.y);
            } else {
                en = out1[stat_pad(u)];
                row[o] = en;
            }
            if (SCAN && en > dead)
                low = max(low, ~__float_as_uint(en));
        });
        if (full && dc)
            block_dc(mx, dc + ch);
        if (SCAN)
            scan_block(top, low, base, scan, ch, SC);
        __syncthreads();  // shared memory is free for the next block
    }
}

// ---------------------------------------------------------------- the usual blocks
// The same statistics from exact running sums in fixed point, which take a third of
// the instructions, for blocks of windows whose values lie close enough together;
// the others go on the list for window_stats_kernel.
//
// A block's squares are rounded to the unit 2^(2e - 40), all its |v| below 2^e; the sums
// of a window's squares are exact, so only the squares' own rounding remains, half
// a unit each ('full': with the squares' exact remainders and the mean's rounding, two
// units).  The block stays here if every window's energy is at least L 2^27 units (or,
// for 'short', exactly zero), so that rounding is at most 2^-26 (2^-28) of it, half of
// its float's own rounding: windows down to 1/90 of the block's largest value in
// amplitude.  A transient on quiet noise, a value that is not finite, a level shift
// or a window that ends in a gap send their block to the list.
//
// A number in units is two 20-bit digits, which magic-number additions take from
// floats without conversion instructions (64-bit conversions run on the FP64 pipe:
// 322 us below); the digits' running sums are 32-bit integers that wrap, and the
// differences of one window fit them (L <= 2,048).  Chunks of 16 samples, a thread
// each: running sums inside the chunk, then a scan of the chunks' sums.
//
// What bounds it: the instructions, mostly integer ones.  60 channels x 1.08M samples x
// 600 taps: 354 us with window_stats_kernel alone, 233 us here and 3 us for the second
// launch; 'full', 30 channels x 8.6M: 1,161 us and 903 + 3 us.
constexpr int kFixThreads = 512;
constexpr int kFixChunk = 16;
constexpr int kFixBits = 40, kFixDigit = 20;
constexpr int kFixLongest = 2048;
// Windows of fewer samples are too quiet now and then by themselves, and every block of
// noise would go on the list: 1 to 3 samples ('full': 4) in a block of 4,096 windows.
constexpr int kFixShortest = 8;
// Fewer blocks than this are one or two rounds of the SMs either way, and the second
// launch would cost more than it saves.
constexpr int kFixLeastBlocks = 608;
static_assert((kStatWindows + kFixLongest + kFixChunk) / kFixChunk <= kFixThreads, "a thread per chunk");

struct FixLayout {  // in 4-byte words: samples, running sums of d^2 and d, chunk offsets of both
    int chunks, padded, p2, p1, o2, o1, total;
    __host__ __device__ FixLayout(int L, bool full)
    {
        chunks = (kStatWindows + L + kFixChunk) / kFixChunk;
        padded = chunks * (kFixChunk + 1);
        p2 = (padded + 3) & ~3;
        p1 = p2 + 2 * padded;
        o2 = p1 + (full ? 2 * padded : 0);
        o1 = o2 + 2 * chunks;
        total = o1 + (full ? 2 * chunks : 0);
    }
    size_t bytes() const { return (size_t)total * 4; }
};

// x in units, |x| < 2^40, as digits: adds them to hi and lo.  (1.5 * 2^23 + integer:
// the integer, rounded to nearest, is in the low bits.)
__device__ __forceinline__ void fix_add(float x, unsigned &hi, unsigned &lo)
{
    const float magic = 12582912.0f;  // 1.5 * 2^23 = 0x4b400000
    const float t = fmaf(x, 1.0f / (1 << kFixDigit), magic);
    const float rest = fmaf(-(t - magic), (float)(1 << kFixDigit), x);  // exact, at most 2^19
    hi += __float_as_uint(t) - 0x4b400000u;
    lo += __float_as_uint(rest + magic) - 0x4b400000u;
}

// hi 2^20 + lo as a float pair (hi in [-2^31, 2^31), |lo| <= 2^30): three exact parts.
__device__ __forceinline__ void fix_pair(int hi, int lo, float &h, float &l)
{
    const float f1 = (float)(hi >> 8) * 268435456.0f;                       // 2^28
    const float f2 = (float)(((hi & 255) << 12) + (lo >> 8)) * 256.0f;
    float e;
    h = two_diff(f1, -f2, e);
    l = e + (float)(lo & 255);
}

// grid = (ceil(N / kStatWindows), SC), kFixThreads threads, dynamic smem FixLayout.
template <bool FULL, bool SCAN>
__global__ void __launch_bounds__(kFixThreads, FULL ? 2 : 3)
window_fixed_kernel(const float *__restrict__ data, int N, int L, const float *__restrict__ mu,
                    float *__restrict__ dcen, float *__restrict__ stat_e, const StatPlace place,
                    unsigned *__restrict__ scan, unsigned *__restrict__ dc, unsigned *__restrict__ list)
{
    extern __shared__ float4 stat_smem[];
    __shared__ uint2 warp_sums[2][kFixThreads / 32];
    __shared__ unsigned shared_top;
    __shared__ int odd;  // the block goes on the list
    const FixLayout lay(L, FULL);
    float *raw = reinterpret_cast<float *>(stat_smem);
    uint2 *p2 = reinterpret_cast<uint2 *>(raw + lay.p2), *p1 = reinterpret_cast<uint2 *>(raw + lay.p1);
    uint2 *o2 = reinterpret_cast<uint2 *>(raw + lay.o2), *o1 = reinterpret_cast<uint2 *>(raw + lay.o1);
    const int chunks = lay.chunks, span = chunks * kFixChunk;
    const auto pad = [](int i) { return i + (i >> 4); };

    const int ch = blockIdx.y, SC = gridDim.y;
    const long long c0 = (long long)blockIdx.x * kStatWindows;
    const int len = (int)min((long long)kStatWindows + L - 1, (long long)N - c0);
    const int nwin = min(kStatWindows, len - L + 1);
    const float m = FULL ? mu[ch] : 0.0f;
    const float *src = data + (size_t)ch * N + c0;
    if (threadIdx.x == 0) {
        shared_top = 0;
        odd = 0;
    }
    unsigned top = 0;   // bits of the largest |v|; of a value that is not finite, too
    unsigned most = 0;  // bits of the largest finite one
    float *dst = FULL ? dcen + (size_t)ch * N + c0 : nullptr;
    constexpr int kLoads = 5;
    for (int i0 = threadIdx.x; i0 < span; i0 += kLoads * kFixThreads) {
        float x[kLoads];
#pragma unroll
        for (int j = 0; j < kLoads; j++) {
            const int i = i0 + j * kFixThreads;
            x[j] = i < len ? __ldg(src + i) : m;
        }
#pragma unroll
        for (int j = 0; j < kLoads; j++) {
            const int i = i0 + j * kFixThreads;
            if (i < span) {
                const float v = FULL ? x[j] - m : x[j];
                if (FULL && i < kStatWindows && i < len)
                    dst[i] = v;
                const unsigned av = __float_as_uint(v) & 0x7fffffffu;
                top = max(top, av);
                if (SCAN)
                    most = av < 0x7f800000u ? max(most, av) : most;
                raw[pad(i)] = v;
            }
        }
    }
    __syncthreads();
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0)
        atomicMax(&shared_top, top);
    __syncthreads();
    top = shared_top;
    const int e = top ? (int)(top >> 23) - 126 : 0;  // every |v| < 2^e
    const bool bad = e < -38 || e > 60;              // (infinities and NaN have the largest e)
    bool lost = false;  // some square is not zero but less than half a unit ('short')
    const auto pow2 = [](int k) { return __int_as_float((k + 127) << 23); };
    if (!bad) {
        const float s = pow2(kFixBits / 2 - e);  // squares of s v are in units
        uint2 t2 = make_uint2(0, 0), t1 = make_uint2(0, 0);
        const int c = threadIdx.x;
        if (c < chunks) {
            const int at = c * (kFixChunk + 1);
#pragma unroll
            for (int j = 0; j < kFixChunk; j++) {
                const float v = raw[at + j] * s, sq = v * v;
                p2[at + j] = t2;
                fix_add(sq, t2.x, t2.y);
                if (FULL) {  // the square's remainder, at most 2^16 units
                    t2.y += __float_as_uint(fmaf(v, v, -sq) + 12582912.0f) - 0x4b400000u;
                    p1[at + j] = t1;
                    fix_add(v * (float)(1 << kFixBits / 2), t1.x, t1.y);
                } else {
                    lost = lost || (sq < 0.5f && v != 0.0f);
                }
            }
        }
        // exclusive scan of the chunks' sums
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        const auto scan_chunks = [&](uint2 t, uint2 *sums, uint2 *to) {
            uint2 y = t;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned a = __shfl_up_sync(0xffffffffu, y.x, o), b = __shfl_up_sync(0xffffffffu, y.y, o);
                if (lane >= o) {
                    y.x += a;
                    y.y += b;
                }
            }
            if (lane == 31)
                sums[wid] = y;
            __syncthreads();
            unsigned hx = 0, lx = 0;
            for (int i = 0; i < wid; i++) {
                hx += sums[i].x;
                lx += sums[i].y;
            }
            if (c < chunks)
                to[c] = make_uint2(hx + y.x - t.x, lx + y.y - t.y);
        };
        scan_chunks(t2, warp_sums[0], o2);
        if (FULL)
            scan_chunks(t1, warp_sums[1], o1);
        lost = __syncthreads_or(lost) != 0;
    }
    const float Lf = (float)L, invL = 1.0f / Lf;
    const float u2 = pow2(bad ? 0 : 2 * e - kFixBits), u1 = pow2(bad ? 0 : e - kFixBits);
    const float least = Lf * 0x1p27f * u2;  // energy below which the unit is too coarse
    // energies at or below this pass no template's threshold
    const float dead = SCAN ? kThreshold / __uint_as_float(scan[2 * SC + ch]) * 0.999f : 0.0f;
    unsigned low = 0;  // the smallest energy above it, bits complemented
    float mx = 0.0f;
    float *row = stat_e + (ch * place.ch + first_place(place, c0)) * (FULL ? 2 : 1);
    bool far = false;  // a window too quiet for the block's unit
    each_window<kFixThreads>(place, c0, bad ? 0 : nwin, [&](int u, long long o) {
        const int a = pad(u), b = pad(u + L), ca = u >> 4, cb = (u + L) >> 4;
        const uint2 pa2 = p2[a], pb2 = p2[b], qa2 = o2[ca], qb2 = o2[cb];
        const unsigned hi2 = pb2.x + qb2.x - (pa2.x + qa2.x);
        const int lo2 = (int)(pb2.y + qb2.y - (pa2.y + qa2.y));
        float en;
        if constexpr (FULL) {
            const uint2 pa1 = p1[a], pb1 = p1[b], qa1 = o1[ca], qb1 = o1[cb];
            float h2, l2, h1, l1, mean;
            fix_pair((int)hi2, lo2, h2, l2);
            fix_pair((int)(pb1.x + qb1.x - (pa1.x + qa1.x)), (int)(pb1.y + qb1.y - (pa1.y + qa1.y)), h1, l1);
            window_centred_sums(h2 * u2, l2 * u2, h1 * u1, l1 * u1, Lf, invL, en, mean);
            far = far || !(en >= least);
            reinterpret_cast<float2 *>(row)[o] = make_float2(en, mean);
            if (dc)
                mx = window_dc(mx, (unsigned)c0 + u, Lf, en, mean);
        } else {
            // the top 24 bits and the rest, added with one rounding
            const float f = fmaf((float)(hi2 >> 8), 268435456.0f, (float)((int)((hi2 & 255) << 20) + lo2));
            en = f * u2;
            far = far || (en < least && (en != 0.0f || lost));
            row[o] = en;
        }
        if (SCAN && en > dead)
            low = max(low, ~__float_as_uint(en));
    });
    if (far || bad)
        odd = 1;  // (any thread's)
    __syncthreads();
    if (odd && threadIdx.x == 0 && nwin > 0)
        list[1 + atomicAdd(list, 1u)] = blockIdx.y * gridDim.x + blockIdx.x;
    if (FULL && dc && !odd)
        block_dc(mx, dc + ch);
    // the largest value counts in any case; the smallest energy of a listed block is made there
    if (SCAN)
        scan_block(most, odd ? 0u : low, raw, scan, ch, SC);
}

StatPlace stat_rows(int SC, int N, int step, int pad, size_t *elems)
{
    StatPlace p;
    p.step = step;
    p.rem = 0;
    p.ps = ((long long)(N + step - 1) / step + 2ll * pad + 3) & ~3ll;
    p.ch = p.ps * step;
    *elems = (size_t)SC * (size_t)p.ch;
    return p;
}

StatPlace stat_rows_packed(int N, int step) { return StatPlace{(long long)N, N / step, N % step, step}; }

size_t window_list_words(int N, int SC)
{
    const long long blocks = (long long)((N + kStatWindows - 1) / kStatWindows) * SC;
    return blocks >= kFixLeastBlocks && blocks < 0x7fffffffLL ? (size_t)blocks + 1 : 0;
}

int launch_window_stats(const float *data, int N, int L, int SC, const float *mu, float *dcen,
                        float *stat_e, const StatPlace &place, unsigned *scan, unsigned *dc, unsigned *list,
                        cudaStream_t s)
{
    const bool full = mu != nullptr;
    const int per_ch = (N + kStatWindows - 1) / kStatWindows;
    unsigned grid = (unsigned)per_ch * SC;
    cudaError_t e;
    const size_t fixed = FixLayout(L, full).bytes();
    if (fixed > (size_t)kMaxDynamicSmem - 1024 || L > kFixLongest || L < kFixShortest || SC > 65535)
        list = nullptr;
    if (list) {
        auto kern = scan ? (full ? window_fixed_kernel<true, true> : window_fixed_kernel<false, true>)
                         : (full ? window_fixed_kernel<true, false> : window_fixed_kernel<false, false>);
        e = cudaMemsetAsync(list, 0, sizeof(unsigned), s);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem - 1024);
        if (e != cudaSuccess)
            return set_error(FMF_ERR_CUDA, "window statistics: %s", cudaGetErrorString(e));
        kern<<<dim3(per_ch, SC), kFixThreads, fixed, s>>>(data, N, L, mu, dcen, stat_e, place, scan, dc, list);
        count_launch();
        grid = grid < 608 ? grid : 608;  // the listed blocks, few or none
    }
    auto kern = scan ? (full ? window_stats_kernel<true, true> : window_stats_kernel<false, true>)
                     : (full ? window_stats_kernel<true, false> : window_stats_kernel<false, false>);
    const size_t smem = window_stats_smem(L, full);
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmem);
    if (e != cudaSuccess)
        return set_error(FMF_ERR_CUDA, "window statistics shared memory (%zu bytes): %s", smem,
                         cudaGetErrorString(e));
    kern<<<grid, kStatThreads, smem, s>>>(data, N, L, SC, mu, dcen, stat_e, place, scan, dc, list);
    count_launch();
    return FMF_OK;
}

}  // namespace fmf
