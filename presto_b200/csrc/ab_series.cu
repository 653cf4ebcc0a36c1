// ab_series.cu -- the time-series input path of the search on the device:
// create_accelobs' .dat branch (src/accel_utils.c:1516-1563), i.e. the
// forward realfft (src/fastffts.c:163-246) and deredden(fft, n/2, 6, 200,
// 0.5/dt, n dt) (src/misc_utils.c:912-1067).
//
// realfft: the n/2-point complex FFT of the samples taken in pairs, then the
// untangling pass into n/2 bins with bin 0 = (DC, Nyquist).  For a
// power-of-two M = n/2 the complex FFT is one radix-16 Stockham transform in
// shared memory up to 8192 points, and above that a four-step transform
// M = M1 M2 in two passes over memory: strided columns with the inter-step
// twiddles, then rows written in their transposed places.  Any other even n
// (dedispersed series are usually 2^a 3^b 5^c 7^d samples long) goes through
// Bluestein's chirp-z transform on power-of-two transforms of length
// >= 2M - 1, its products fused into their four passes.
//
// deredden: the block partition depends only on bin indices (lengths
// startwidth ln(bin) up to endwidth), so the host plans it as runs of equal
// blocks (some hundred); one warp per block takes the exact median of its
// powers, then every bin is scaled by the reference's interpolated
// normalisation with its fast inverse square root, in float with explicit
// rounding, so the same input gives the reference's bits.
#include <cuda_runtime.h>
#include <math.h>

#include "ab_fft.cuh"
#include "ab_kernels.h"
#include "ab_norm.cuh"

namespace ab {
namespace {

// W_M^j = exp(-2 pi i j / M), 0 <= j < M
__device__ __forceinline__ double2 root(long long j, double invM)
{
    double s, c;
    sincospi(-2.0 * ((double) j * invM), &s, &c);
    return make_double2(c, s);
}

// v[m] *= W_M^{a (t + NT m)}, m = 0..15 (a, t + NT m < 2^13, M a power of
// two: a (t + NT m) / M is exact): two FP64 roots and their products instead
// of sixteen roots; fifteen FP64 products stay far below the FP32 rounding.
__device__ __forceinline__ void step_twiddles(float2 (&v)[16], int a, int t, int NT, long long M)
{
    const double inv = 1.0 / (double) M;
    double2 w = root((long long) a * t, inv);
    const double2 q = root((long long) a * NT, inv);
#pragma unroll
    for (int m = 0; m < 16; m++) {
        const float cr = (float) w.x, ci = (float) w.y;
        v[m] = make_float2(v[m].x * cr - v[m].y * ci, v[m].x * ci + v[m].y * cr);
        w = dmul(w, q);
    }
}

// Bluestein's chirp-z transform for any length M: with c_j = exp(i pi j^2 / M),
// X_k = conj(c_k) sum_j (x_j conj(c_j)) c_{k-j}, a linear convolution done as
// a circular one of power-of-two length L >= 2M - 1.  Chirps are evaluated in
// FP64 from j^2 mod 2M (exact: j < 2^25, so j^2 and the multiple of 2M taken
// from it stay below 2^53), the products with them in FP64; the transforms of
// length L are the FP32 power-of-two FFT.
struct Chirp {
    long long M, L;
    double twoM, inv2M;
};

Chirp make_chirp(long long M, long long L)
{
    return Chirp{M, L, 2.0 * (double) M, 1.0 / (2.0 * (double) M)};
}

__device__ __forceinline__ double2 chirp(long long j, const Chirp &c)
{
    const double sq = (double) j * (double) j;
    double r = fma(-floor(sq * c.inv2M), c.twoM, sq);      // the quotient is off by one at most
    if (r < 0.0) r += c.twoM;
    if (r >= c.twoM) r -= c.twoM;
    double s, co;
    sincospi(r / (double) c.M, &s, &co);
    return make_double2(co, s);
}

// x_j conj(c_j), zero from M on
__device__ __forceinline__ float2 blu_in(const float2 *z, long long j, const Chirp &c)
{
    if (j >= c.M) return make_float2(0.f, 0.f);
    const double2 h = chirp(j, c);
    const double xr = z[j].x, xi = z[j].y;
    return make_float2((float) (xr * h.x + xi * h.y), (float) (xi * h.x - xr * h.y));
}

// the convolution's kernel c_{|j|}, circular in L
__device__ __forceinline__ float2 blu_kernel(long long j, const Chirp &c)
{
    const long long m = j < c.M ? j : (j > c.L - c.M ? c.L - j : -1);
    if (m < 0) return make_float2(0.f, 0.f);
    const double2 h = chirp(m, c);
    return make_float2((float) h.x, (float) h.y);
}

// conj(c_k) conj(v_k) / L: the inverse transform is taken as a forward one of
// the conjugate
__device__ __forceinline__ float2 blu_out(float2 v, long long k, const Chirp &c)
{
    const double2 h = chirp(k, c);
    const double inv = 1.0 / (double) c.L;
    const double yr = (double) v.x * inv, yi = -(double) v.y * inv;
    return make_float2((float) (yr * h.x + yi * h.y), (float) (yi * h.x - yr * h.y));
}

// Transforms of more than 8192 points go as M = M1 M2 in two passes over
// memory, points n = n1 M2 + n2, bins k = k1 + M1 k2:
//   columns   the M2 transforms over n1 (stride M2), times W_M^{n2 k1}, in
//             the same places;
//   rows      the M1 transforms over n2 (contiguous).
// A column CTA takes C neighbouring columns, so that its reads and writes
// are whole C float2 runs; its threads are ordered column fastest, and the
// C shared-memory buffers lie 16 / C float2 off each other's banks.  512
// threads (16 points each, 128 registers) whatever the length: C = 4 at 2048
// points fills 32-byte sectors, C = 2 at 4096 half of one (the neighbouring
// CTA's half comes from L2).  At M = 2^22 the two passes take 30 + 27 us; three
// transposes, two row passes with a root per point and a copy took 120 us.
template <int L> struct ColShape {
    static constexpr int NT = L / 16;
    static constexpr int CTA = NT >= 512 ? 1024 : 512;
    static constexpr int C = CTA / NT;
    static constexpr int STRIDE = FftShape<L>::SMEM + (C >= 16 ? 1 : 16 / C);
    static constexpr size_t SMEM = (size_t) C * STRIDE * sizeof(float2);
};

enum { COL_PLAIN, COL_BLU_IN, COL_BLU_KERNEL };

// MODE: where the points come from (an array, Bluestein's chirped input or
// its kernel).
template <int L, int MODE>
__global__ void __launch_bounds__(ColShape<L>::CTA) k_fft_cols(const float2 *in, float2 *out, int M2,
                                                               long long M, Chirp ch)
{
    using CS = ColShape<L>;
    extern __shared__ float2 fsm[];
    const int c = threadIdx.x % CS::C, t = threadIdx.x / CS::C;
    const int n2 = blockIdx.x * CS::C + c;
    float2 v[16];
#pragma unroll
    for (int m = 0; m < 16; m++) {
        const long long j = (long long) (t + CS::NT * m) * M2 + n2;
        if constexpr (MODE == COL_BLU_IN) v[m] = blu_in(in, j, ch);
        else if constexpr (MODE == COL_BLU_KERNEL) v[m] = blu_kernel(j, ch);
        else v[m] = in[j];
    }
    FftTw<L, -1> tw;
    tw.init(t);
    fft_run<L, -1>(v, fsm + c * CS::STRIDE, t, tw);
    step_twiddles(v, n2, t, CS::NT, M);
#pragma unroll
    for (int m = 0; m < 16; m++) out[(long long) (t + CS::NT * m) * M2 + n2] = v[m];
}

enum { ROW_PLAIN, ROW_CONV, ROW_BLU_OUT };

// What becomes of bin k of a transform: kept, the convolution's product
// conj(v B[k]) (the next transform's input), or the chirped result.
template <int MODE>
__device__ __forceinline__ void put_bin(float2 *out, long long k, float2 v, const float2 *B, const Chirp &ch)
{
    if constexpr (MODE == ROW_CONV) {
        const float2 y = B[k];
        out[k] = make_float2(v.x * y.x - v.y * y.y, -(v.x * y.y + v.y * y.x));
    } else if constexpr (MODE == ROW_BLU_OUT) {
        if (k < ch.M) out[k] = blu_out(v, k, ch);
    } else {
        out[k] = v;
    }
}

// The rows' transforms with bin k1 + M1 k2 written to its natural place: the
// same shape, a CTA's C rows giving runs of C bins.
template <int L, int MODE>
__global__ void __launch_bounds__(ColShape<L>::CTA) k_fft_rows_out(const float2 *in, float2 *out, int M1,
                                                                   const float2 *B, Chirp ch)
{
    using CS = ColShape<L>;
    extern __shared__ float2 fsm[];
    const int r0 = blockIdx.x * CS::C;
    float2 v[16];
    {
        // read along the rows, hand over in shared memory to the threads that
        // are ordered row fastest for the writes
        const int c = threadIdx.x / CS::NT, t = threadIdx.x % CS::NT;
#pragma unroll
        for (int m = 0; m < 16; m++) v[m] = in[(long long) (r0 + c) * L + t + CS::NT * m];
#pragma unroll
        for (int m = 0; m < 16; m++) fsm[c * CS::STRIDE + pad16(t + CS::NT * m)] = v[m];
    }
    __syncthreads();
    const int c = threadIdx.x % CS::C, t = threadIdx.x / CS::C;
    float2 *sm = fsm + c * CS::STRIDE;
#pragma unroll
    for (int m = 0; m < 16; m++) v[m] = sm[pad16(t + CS::NT * m)];
    FftTw<L, -1> tw;
    tw.init(t);
    __syncthreads();
    fft_run<L, -1>(v, sm, t, tw);
#pragma unroll
    for (int m = 0; m < 16; m++)
        put_bin<MODE>(out, (long long) (t + CS::NT * m) * M1 + r0 + c, v[m], B, ch);
}

// A transform of L <= 8192 points in one CTA.
template <int L, bool BLU_IN, int MODE>
__global__ void __launch_bounds__(FftShape<L>::CTA) k_fft_one(const float2 *in, float2 *out, const float2 *B, Chirp ch)
{
    using SH = FftShape<L>;
    extern __shared__ float2 fsm[];
    const int grp = threadIdx.x / SH::NT, t = threadIdx.x - grp * SH::NT;
    float2 v[16];
#pragma unroll
    for (int m = 0; m < 16; m++) {
        const int k = t + SH::NT * m;
        v[m] = BLU_IN ? blu_in(in, k, ch) : in[k];
    }
    FftTw<L, -1> tw;
    tw.init(t);
    __syncthreads();                        // out may be in: every group has read it
    fft_run<L, -1>(v, fsm + grp * SH::SMEM, t, tw);
    if (grp) return;                        // the CTA's other groups did the same
#pragma unroll
    for (int m = 0; m < 16; m++) put_bin<MODE>(out, t + SH::NT * m, v[m], B, ch);
}

// Bluestein's kernel for a transform in one CTA
__global__ void k_blu_kernel(float2 *b, Chirp ch)
{
    const long long j = (long long) blockIdx.x * blockDim.x + threadIdx.x;
    if (j < ch.L) b[j] = blu_kernel(j, ch);
}

// realfft's untangling (src/fastffts.c:195-229, forward): pair (il, n/2 - il)
// per thread, sums of the float inputs in float as the reference, products
// in FP64 without contraction, twiddles exp(-2 pi i il / n) computed directly.
__global__ void k_untangle(float2 *c, long long n)
{
    const long long il = (long long) blockIdx.x * blockDim.x + threadIdx.x;
    const long long nby2 = n >> 1, nby4 = n >> 2;
    if (il == 0) {
        const float t = c[0].x;
        c[0] = make_float2(__fadd_rn(t, c[0].y), __fsub_rn(t, c[0].y));
        return;
    }
    if (il > nby4) return;
    const long long ih = nby2 - il;
    const float2 a = c[il], b = c[ih];
    double wi, wr;
    sincospi(-2.0 * (double) il / (double) n, &wi, &wr);
    const double h1r = 0.5 * (double) __fadd_rn(a.x, b.x), h1i = 0.5 * (double) __fsub_rn(a.y, b.y);
    const double h2r = 0.5 * (double) __fadd_rn(a.y, b.y), h2i = -0.5 * (double) __fsub_rn(a.x, b.x);
    const double h2rwr = __dmul_rn(h2r, wr), h2rwi = __dmul_rn(h2r, wi);
    const double h2iwr = __dmul_rn(h2i, wr), h2iwi = __dmul_rn(h2i, wi);
    const float2 lo = make_float2((float) __dsub_rn(__dadd_rn(h1r, h2rwr), h2iwi),
                                  (float) __dadd_rn(__dadd_rn(h1i, h2iwr), h2rwi));
    const float2 hi = make_float2((float) __dadd_rn(__dsub_rn(h1r, h2rwr), h2iwi),
                                  (float) __dadd_rn(__dadd_rn(-h1i, h2iwr), h2rwi));
    c[il] = lo;
    c[ih] = hi;
}


// Run i of the block partition (equal blocks one behind the other): first
// bin, block length, index of the first block, block count.  runs[nruns] is
// a sentinel: the bin and the block behind the last.
__device__ __forceinline__ int run_of_block(const int4 *runs, int nruns, int block)
{
    int lo = 0, hi = nruns - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (runs[mid].z <= block) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Median of each block's powers / ln 2 (the block "mean" of deredden), one
// warp per block of at most 32 NV bins, held in registers: the k-th smallest
// by building its bits from the top (one warp-wide count a bit; powers are
// not negative, so their bits order as they do), and the (k+1)-th as the
// smallest above it unless it is equal.  2^22 bins in 49645 blocks: 160 us as
// 32-thread CTAs with 4-pass radix selects through shared memory, 42 us so
// (some 350 warp instructions a block; issue-bound).
template <int NV>
__global__ void __launch_bounds__(256) k_dered_means(const float2 *fft, const int4 *runs, int nruns, int nb,
                                                     float *means)
{
    const int block = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (block >= nb) return;
    const int4 r = runs[run_of_block(runs, nruns, block)];
    const int n = r.y;
    const float2 *x = fft + r.x + (long long) (block - r.z) * n;
    unsigned u[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) {
        u[q] = 0xFFFFFFFFu;                                 // above every power
        if (lane + 32 * q < n) {
            const float2 v = x[lane + 32 * q];
            u[q] = __float_as_uint(__fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y)));
        }
    }
    const unsigned k = (unsigned) (n - 1) / 2;
    unsigned pre = 0;
    for (int bit = 30; bit >= 0; bit--) {
        const unsigned trial = pre | (1u << bit);
        unsigned below = 0;
#pragma unroll
        for (int q = 0; q < NV; q++) below += u[q] < trial;
        if (__reduce_add_sync(0xffffffffu, below) <= k) pre = trial;
    }
    float med = __uint_as_float(pre);
    if (!(n & 1)) {
        unsigned upto = 0, next = 0xFFFFFFFFu;
#pragma unroll
        for (int q = 0; q < NV; q++) {
            upto += u[q] <= pre;
            if (u[q] > pre) next = min(next, u[q]);
        }
        upto = __reduce_add_sync(0xffffffffu, upto);
        next = __reduce_min_sync(0xffffffffu, next);
        const float hi = upto > k + 1 ? med : __uint_as_float(next);
        med = (float) (0.5 * ((double) med + (double) hi));
    }
    if (lane == 0) means[block] = (float) ((double) med / 0.69314718055994530942);
}

// Every bin by its own thread: from the middle of block b - 1 to the middle
// of block b the line between their means, the first half of block 0 its own
// mean, the second half of the last block the line before it carried on
// (slope 1 when there is one block).  Bin 0 becomes (1, 0).  (One CTA per
// segment of some 90 bins took 62 us at 2^22 bins, this 31 us.)
__global__ void __launch_bounds__(256) k_dered_apply(float2 *fft, const int4 *runs, int nruns, int nb,
                                                    const float *means)
{
    const int last = runs[nruns].x;                         // first bin behind the blocks
    const long long bin0 = (long long) blockIdx.x * 1024;
    // the run of the CTA's first bin, then forward
    int ri;
    {
        int lo = 0, hi = nruns - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (runs[mid].x <= bin0) lo = mid;
            else hi = mid - 1;
        }
        ri = lo;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const long long bin = bin0 + threadIdx.x + 256 * q;
        if (bin == 0) fft[0] = make_float2(1.0f, 0.0f);
        if (bin == 0 || bin >= last) continue;
        while (bin >= runs[ri + 1].x) ri++;
        const int4 r = runs[ri];
        const int in = (int) bin - r.x, k = in / r.y, off = in - k * r.y;
        const int b = r.z + k;                              // the bin's block
        // segment s = 0: before block 0's middle; else behind block s - 1's
        const int s = off < r.y / 2 ? b : b + 1;
        float norm;
        if (s == 0) {
            norm = fast_invsqrtf(means[0]);
        } else {
            const int kk = s < nb ? s : nb - 1;             // slope of blocks kk - 1, kk
            // lengths of block b and of the neighbours the segment involves
            const int4 rp = (k == 0 && ri > 0) ? runs[ri - 1] : r;
            const int4 rn = (k == r.w - 1 && ri + 1 < nruns) ? runs[ri + 1] : r;
            const int len_prev = rp.y, len_next = rn.y;     // of blocks b - 1 and b + 1
            long long start;
            if (s == b) start = (long long) r.x + (long long) k * r.y - len_prev + len_prev / 2;
            else start = (long long) r.x + (long long) k * r.y + r.y / 2;
            float dslope = 1.0f;
            if (kk >= 1) {
                const int sum = kk == b ? len_prev + r.y : r.y + len_next;
                dslope = (float) ((double) __fsub_rn(means[kk], means[kk - 1]) / (0.5 * (double) sum));
            }
            const float ii = (float) (bin - start);
            norm = fast_invsqrtf(__fadd_rn(means[s - 1], __fmul_rn(dslope, ii)));
        }
        const float2 v = fft[bin];
        fft[bin] = make_float2(__fmul_rn(v.x, norm), __fmul_rn(v.y, norm));
    }
}

template <int L, int MODE>
cudaError_t cols_L(const float2 *in, float2 *out, int M2, long long M, const Chirp &ch, cudaStream_t st)
{
    using CS = ColShape<L>;
    cudaError_t e = cudaFuncSetAttribute(k_fft_cols<L, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int) CS::SMEM);
    if (e != cudaSuccess) return e;
    k_fft_cols<L, MODE><<<(unsigned) (M2 / CS::C), CS::CTA, CS::SMEM, st>>>(in, out, M2, M, ch);
    return cudaGetLastError();
}

template <int MODE>
cudaError_t cols(int L, const float2 *in, float2 *out, int M2, long long M, const Chirp &ch, cudaStream_t st)
{
    switch (L) {
        case 256: return cols_L<256, MODE>(in, out, M2, M, ch, st);
        case 512: return cols_L<512, MODE>(in, out, M2, M, ch, st);
        case 1024: return cols_L<1024, MODE>(in, out, M2, M, ch, st);
        case 2048: return cols_L<2048, MODE>(in, out, M2, M, ch, st);
        case 4096: return cols_L<4096, MODE>(in, out, M2, M, ch, st);
        case 8192: return cols_L<8192, MODE>(in, out, M2, M, ch, st);
        default: return cudaErrorInvalidValue;
    }
}

template <int L, int MODE>
cudaError_t rows_out_L(const float2 *in, float2 *out, int M1, const float2 *B, const Chirp &ch, cudaStream_t st)
{
    using CS = ColShape<L>;
    cudaError_t e = cudaFuncSetAttribute(k_fft_rows_out<L, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int) CS::SMEM);
    if (e != cudaSuccess) return e;
    k_fft_rows_out<L, MODE><<<(unsigned) (M1 / CS::C), CS::CTA, CS::SMEM, st>>>(in, out, M1, B, ch);
    return cudaGetLastError();
}

template <int MODE>
cudaError_t rows_out(int L, const float2 *in, float2 *out, int M1, const float2 *B, const Chirp &ch,
                     cudaStream_t st)
{
    switch (L) {
        case 256: return rows_out_L<256, MODE>(in, out, M1, B, ch, st);
        case 512: return rows_out_L<512, MODE>(in, out, M1, B, ch, st);
        case 1024: return rows_out_L<1024, MODE>(in, out, M1, B, ch, st);
        case 2048: return rows_out_L<2048, MODE>(in, out, M1, B, ch, st);
        case 4096: return rows_out_L<4096, MODE>(in, out, M1, B, ch, st);
        case 8192: return rows_out_L<8192, MODE>(in, out, M1, B, ch, st);
        default: return cudaErrorInvalidValue;
    }
}

template <int L, bool BLU_IN, int MODE>
cudaError_t one_L(const float2 *in, float2 *out, const float2 *B, const Chirp &ch, cudaStream_t st)
{
    using SH = FftShape<L>;
    const size_t smem = (size_t) SH::G * SH::SMEM * sizeof(float2);
    cudaError_t e = cudaFuncSetAttribute(k_fft_one<L, BLU_IN, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int) smem);
    if (e != cudaSuccess) return e;
    k_fft_one<L, BLU_IN, MODE><<<1, SH::CTA, smem, st>>>(in, out, B, ch);
    return cudaGetLastError();
}

template <bool BLU_IN, int MODE>
cudaError_t fft_one(int L, const float2 *in, float2 *out, const float2 *B, const Chirp &ch, cudaStream_t st)
{
    switch (L) {
        case 512: return one_L<512, BLU_IN, MODE>(in, out, B, ch, st);
        case 1024: return one_L<1024, BLU_IN, MODE>(in, out, B, ch, st);
        case 2048: return one_L<2048, BLU_IN, MODE>(in, out, B, ch, st);
        case 4096: return one_L<4096, BLU_IN, MODE>(in, out, B, ch, st);
        case 8192: return one_L<8192, BLU_IN, MODE>(in, out, B, ch, st);
        default: return cudaErrorInvalidValue;
    }
}

// M = M1 M2 of a transform above 8192 points
void split_len(long long M, int *M1, int *M2)
{
    int m = 0;
    while ((1LL << m) < M) m++;
    *M1 = 1 << (m / 2);
    *M2 = (int) (M / *M1);
}

}  // namespace

bool pow2_fft_supported(long long M)
{
    if (M & (M - 1)) return false;
    return (M >= 512 && M <= 8192) || (M >= (1 << 16) && M <= (1LL << 26));
}

long long bluestein_len(long long M)
{
    long long L = 1;
    while (L < 2 * M - 1) L <<= 1;
    if (L < 512) L = 512;
    if (L > 8192 && L < (1 << 16)) L = 1 << 16;       // the four-step's shortest
    return L;
}

bool realfft_supported(long long n)
{
    if (n < 1024 || n % 2) return false;
    const long long M = n / 2;
    return pow2_fft_supported(M) || M <= (1LL << 25);
}

cudaError_t launch_realfft(const float *series, float2 *out, float2 *scratch, long long n, cudaStream_t st)
{
    const long long M = n / 2;
    if (n % 2 || !pow2_fft_supported(M)) return cudaErrorInvalidValue;
    const float2 *x = reinterpret_cast<const float2 *>(series);
    cudaError_t e;
    if (M <= 8192) {
        e = fft_one<false, ROW_PLAIN>((int) M, x, out, nullptr, Chirp{}, st);
    } else {
        int M1, M2;
        split_len(M, &M1, &M2);
        e = cols<COL_PLAIN>(M1, x, scratch, M2, M, Chirp{}, st);
        if (e == cudaSuccess) e = rows_out<ROW_PLAIN>(M2, scratch, out, M1, nullptr, Chirp{}, st);
    }
    if (e != cudaSuccess) return e;
    const long long nthr = M / 2 + 1;
    k_untangle<<<(unsigned) ((nthr + 255) / 256), 256, 0, st>>>(out, n);
    return cudaGetLastError();
}

// Four passes over memory: the chirped input's columns, the rows with the
// convolution's product, the second transform's columns, its rows with the
// chirped output.  (As separate transforms with their transposes and products
// they were 27 passes: 480 us and two copies at M = 3024000, L = 2^23.
// Leaving the bins in the first transform's order and going back by rows,
// then columns, saves a pass and 70 us more, but sums the second transform in
// another order: where a large mean dominates the series, as in counts off a
// filterbank, that alone moves the other bins by 1e-5.)
cudaError_t launch_realfft_bluestein(const float *series, float2 *out, float2 *a, float2 *scratch, float2 *B,
                                     bool build_B, long long n, cudaStream_t st)
{
    const long long M = n / 2, L = bluestein_len(M);
    if (n % 2 || n < 1024 || M > (1LL << 25)) return cudaErrorInvalidValue;
    const Chirp ch = make_chirp(M, L);
    const float2 *x = reinterpret_cast<const float2 *>(series);
    cudaError_t e = cudaSuccess;
    if (L <= 8192) {
        if (build_B) {                               // FFT of the chirp kernel, kept per M
            k_blu_kernel<<<(unsigned) ((L + 255) / 256), 256, 0, st>>>(B, ch);
            e = fft_one<false, ROW_PLAIN>((int) L, B, B, nullptr, ch, st);
        }
        if (e == cudaSuccess) e = fft_one<true, ROW_CONV>((int) L, x, a, B, ch, st);
        if (e == cudaSuccess) e = fft_one<false, ROW_BLU_OUT>((int) L, a, out, nullptr, ch, st);
    } else {
        int M1, M2;
        split_len(L, &M1, &M2);
        if (build_B) {
            e = cols<COL_BLU_KERNEL>(M1, nullptr, scratch, M2, L, ch, st);
            if (e == cudaSuccess) e = rows_out<ROW_PLAIN>(M2, scratch, B, M1, nullptr, ch, st);
        }
        if (e == cudaSuccess) e = cols<COL_BLU_IN>(M1, x, scratch, M2, L, ch, st);
        if (e == cudaSuccess) e = rows_out<ROW_CONV>(M2, scratch, a, M1, B, ch, st);
        if (e == cudaSuccess) e = cols<COL_PLAIN>(M1, a, scratch, M2, L, ch, st);
        if (e == cudaSuccess) e = rows_out<ROW_BLU_OUT>(M2, scratch, out, M1, nullptr, ch, st);
    }
    if (e != cudaSuccess) return e;
    const long long nthr = M / 2 + 1;
    k_untangle<<<(unsigned) ((nthr + 255) / 256), 256, 0, st>>>(out, n);
    return cudaGetLastError();
}

cudaError_t launch_deredden(float2 *fft, const int4 *runs, int nruns, int nb, int maxlen, long long numbins,
                            float *means, cudaStream_t st)
{
    if (nb <= 0 || nruns <= 0 || maxlen > AB_DERED_MAXW) return cudaErrorInvalidValue;
    const unsigned grid = (unsigned) ((nb + 7) / 8);
    if (maxlen <= 128) k_dered_means<4><<<grid, 256, 0, st>>>(fft, runs, nruns, nb, means);
    else if (maxlen <= 256) k_dered_means<8><<<grid, 256, 0, st>>>(fft, runs, nruns, nb, means);
    else k_dered_means<AB_DERED_MAXW / 32><<<grid, 256, 0, st>>>(fft, runs, nruns, nb, means);
    k_dered_apply<<<(unsigned) ((numbins + 1023) / 1024), 256, 0, st>>>(fft, runs, nruns, nb, means);
    return cudaGetLastError();
}

}  // namespace ab
