// ab_corr.cu -- template correlation of the searches and plane calls: the
// f-fdot planes of subharm_fderivs_vol (src/accel_utils.c:1025-1210) as a
// sliding correlation over segments of the spectrum.
//
// A bank's sub-planes of consecutive blocks lie side by side on one half-bin
// column grid, and a cell depends on the bins within its template's half
// width only, so the columns need not be correlated block by block.  They are
// cut into segments of V = 2048 - 4 hw columns, whatever the blocks, each from
// one 1024-bin window of the spectrum, hw being the widest half width of a
// class of templates: wide templates get short segments, narrow ones long
// ones.  (Transforms over one block or a few whole ones spend a third to a
// half of their length on overlap: all templates pay for the widest one's, and
// block lengths do not fit the transform's.  zmax = 600 with 16 harmonics at
// N = 2^23: 12.5 million transforms of 4096 points, 134 ms; now 22 million
// pairs of 1024 points, 105 ms.  zmax = 200, wmax = 300 with 8 at 2^22: 317 and
// 200 ms.)  Each block keeps its own normalisation: a segment
// is transformed with its first block's and a column's powers are scaled by
// its own block's over that, squared.  Where blocks of one segment differ so
// much that FP32 would carry one's values into another's cells (SEG_RANGE),
// they are correlated one by one (k_corr_apart).
//
// Banks whose reference transform wraps into valid cells, and the local-power
// normalisation (a factor per bin and block), need every block's own data:
// their segments are cut from one block's window, periodic as in the
// reference's circular correlation.
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>

#include "ab_fft.cuh"
#include "ab_index.h"
#include "ab_kernels.h"
#include "ab_norm.cuh"

namespace ab {

constexpr int SEG_H = AB_SEG_BINS;          // bins of a segment's window
constexpr int SEG_WARPS = 8;                // warps per CTA, two to a template
constexpr int SEG_MAXBLK = 256;             // blocks that share one segment
constexpr int SEG_TILE = AB_SEG_TILE;       // templates of a CTA at most
constexpr int SEG_P = 34;                   // exchange row stride (points): 16-byte rows, no conflicts
// What a segment over several blocks may hold: no bin brighter than this
// against the normalisation of a block whose own window does not hold it, and
// block normalisations within this factor of each other.  A bin of amplitude A
// leaves FP32 rounding of some 3e-7 A / 32 in every column of its segment (its
// power spreads over the transform): 1e-5 at 1024, below 1e-5 of any power
// a search keeps.  Other segments are correlated block by block, each block's
// data cut to its own window.
constexpr float SEG_RANGE = 1024.0f;

// ---------------------------------------------------------------------------
// radix 32 in registers
// ---------------------------------------------------------------------------
// a exp(2 pi i M / 32)
template <int M> __device__ __forceinline__ float2 tw32(float2 a)
{
    constexpr int m = M & 31;
    if constexpr (m == 0) {
        return a;
    } else if constexpr (m % 8 == 0) {
        return m == 8 ? mul_i<1>(a) : m == 16 ? make_float2(-a.x, -a.y) : mul_i<-1>(a);
    } else {
        // cos and sin of pi k / 16
        constexpr double C[9] = {1.0, 0.98078528040323044913, 0.92387953251128675613,
                                 0.83146961230254523708, 0.70710678118654752440,
                                 0.55557023301960222474, 0.38268343236508977173,
                                 0.19509032201612826785, 0.0};
        constexpr int q = m / 8, k = m % 8;
        constexpr double c0 = C[k], s0 = C[8 - k];
        constexpr float c = (float) (q == 0 ? c0 : q == 1 ? -s0 : q == 2 ? -c0 : s0);
        constexpr float s = (float) (q == 0 ? s0 : q == 1 ? c0 : q == 2 ? -s0 : -c0);
        return cmul(a, make_float2(c, s));
    }
}

// x[n2 + 8 K1] *= w32^(n2 K1)
template <int K1> __device__ __forceinline__ void tw32_row(float2 (&x)[32])
{
    x[8 * K1 + 1] = tw32<1 * K1>(x[8 * K1 + 1]);
    x[8 * K1 + 2] = tw32<2 * K1>(x[8 * K1 + 2]);
    x[8 * K1 + 3] = tw32<3 * K1>(x[8 * K1 + 3]);
    x[8 * K1 + 4] = tw32<4 * K1>(x[8 * K1 + 4]);
    x[8 * K1 + 5] = tw32<5 * K1>(x[8 * K1 + 5]);
    x[8 * K1 + 6] = tw32<6 * K1>(x[8 * K1 + 6]);
    x[8 * K1 + 7] = tw32<7 * K1>(x[8 * K1 + 7]);
}

// Inverse (+i) DFT of 32 points in place: n = 8 n1 + n2, k = k1 + 4 k2; bin k
// is left in x[bin32(k)].
__device__ __forceinline__ void dft32(float2 (&x)[32])
{
#pragma unroll
    for (int n2 = 0; n2 < 8; n2++) dft4v<1>(x[n2], x[8 + n2], x[16 + n2], x[24 + n2]);
    tw32_row<1>(x);
    tw32_row<2>(x);
    tw32_row<3>(x);
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) dft8<1>(x + 8 * k1);
}
__host__ __device__ constexpr int bin32(int k) { return 8 * (k & 3) + (k >> 2); }

// Spectra, twiddles and templates are laid out for lanes that hold points
// l + 32 m of 1024: points 64 p + l and 64 p + 32 + l side by side, 16 bytes a
// lane.
__host__ __device__ constexpr int seg_place(int k) { return (k & ~63) + 2 * (k & 31) + ((k >> 5) & 1); }

// ---------------------------------------------------------------------------
// columns and normalisations
// ---------------------------------------------------------------------------
__device__ __forceinline__ ab_hgeom seg_geom(const SearchConsts &sc, const ab_bank &b, double startr)
{
    return ab_harm_geom(startr, startr + sc.rstep - AB_DR, b.numharm, b.harmnum, sc.obs_zlo, sc.obs_wlo,
                        sc.corr_uselen);
}

// Per (bank, block): the block's columns and its normalisation (1 / sqrt of
// the median power / ln 2 of its own window, or photon counts).  A window
// with a value that is not finite, or a median of zero, makes every cell of
// the block NaN in the block's own transform: its normalisation is NaN, and
// the bad bins count as zero for the blocks beside it (k_seg_fwd), whose
// windows do not hold them.  Also the largest part of a value in the window
// (SEG_RANGE).  Blocks of banks correlated by their own data get their
// normalisation from k_prep_time.
__global__ void __launch_bounds__(256) k_seg_cols(const ab_bank *banks, SearchConsts sc, BlockBatch bb,
                                                  const float2 *fft, SegCols *cols, double *norms, int *apart)
{
    extern __shared__ float spw[];
    __shared__ double s_norm;
    __shared__ unsigned s_loud;
    const ab_bank b = banks[blockIdx.y];
    const int j = blockIdx.x;
    const ab_hgeom g = seg_geom(sc, b, bb.startr[j]);
    const long long at = (long long) blockIdx.y * bb.nblk + j;
    if (threadIdx.x == 0) {
        long long lim = sc.inmem ? g.numrs : min(g.numrs, b.numrs_max);
        if (sc.inmem && j >= bb.npre0) lim = min(lim, sc.clip_col - g.rlo * AB_RDR);
        cols[at].c0 = g.rlo * AB_RDR;
        cols[at].lim = (int) max(lim, 0ll);
        s_loud = 0u;
        if (blockIdx.x == 0 && blockIdx.y == 0) apart[0] = 0;
    }
    if (b.own_data) return;
    __syncthreads();
    const long long lobin = g.rlo - b.hw0;
    const int numdata = b.fftlen_ref / AB_NUMBETWEEN;
    bool bad = false;
    float loud = 0.f;
    for (int i = threadIdx.x; i < numdata; i += blockDim.x) {
        const long long bin = lobin + i - sc.obs_lobin;
        if (bin >= 0 && bin < sc.numbins) {
            const float2 v = fft[bin];
            if (isfinite(v.x) && isfinite(v.y)) loud = fmaxf(loud, fmaxf(fabsf(v.x), fabsf(v.y)));
            else bad = true;
        }
    }
    // (not negative: the bits order as the values do)
    const unsigned lb = __reduce_max_sync(0xffffffffu, __float_as_uint(loud));
    if ((threadIdx.x & 31) == 0) atomicMax(&s_loud, lb);
    bad = __syncthreads_or(bad);
    const double n = block_norm(sc, lobin, numdata, fft, spw, &s_norm);
    if (threadIdx.x == 0) {
        cols[at].loud = __uint_as_float(s_loud);
        norms[at] = (bad || !isfinite(n)) ? (double) NAN : n;
    }
}

__device__ __forceinline__ const SegGroup &group_of_unit(const SegGroup *g, int ng, int unit)
{
    int lo = 0, hi = ng - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (g[mid].unit0 <= unit) lo = mid;
        else hi = mid - 1;
    }
    return g[lo];
}

__device__ __forceinline__ const SegGroup &group_of_cta(const SegGroup *g, int ng, int cta)
{
    int lo = 0, hi = ng - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (g[mid].cta0 <= cta) lo = mid;
        else hi = mid - 1;
    }
    return g[lo];
}

// first block of [0, n) whose columns reach past column q
__device__ __forceinline__ int first_block(const SegCols *c, int n, long long q)
{
    int lo = 0, hi = n - 1;                     // last block that starts at or before q
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (c[mid].c0 <= q) lo = mid;
        else hi = mid - 1;
    }
    while (lo > 0 && c[lo - 1].c0 + c[lo - 1].lim > q) lo--;
    return lo;
}

// The normalisation a unit's data carry: of its first block, or of the first
// one after it that has one.
__device__ __forceinline__ double unit_norm(const double *nm, int j0, int n)
{
    for (int j = j0; j < n && j < j0 + SEG_MAXBLK; j++)
        if (nm[j] > 0.0 && isfinite(nm[j])) return nm[j];
    return 1.0;
}

// Blocks of [j0, n) whose columns a unit of V columns from column q holds; all
// lanes of a warp.
__device__ __forceinline__ int unit_blocks(const SegCols *c, int j0, int n, long long q, int V)
{
    n = min(n, j0 + SEG_MAXBLK);
    int nj = 1;
    for (;;) {
        const int j = j0 + nj + (int) (threadIdx.x & 31);
        const unsigned in = __ballot_sync(0xffffffffu, j < n && c[j].c0 < q + V);
        nj += __popc(in);
        if (in != 0xffffffffu) return nj;
    }
}

// Block j's own window, as points [lo, hi) of a segment whose window starts at bin0.
__device__ __forceinline__ void block_window(const SearchConsts &sc, const ab_bank &b, const SegCols &c, long long bin0,
                                             int &lo, int &hi)
{
    const long long a = c.c0 / 2 - b.hw0 - sc.obs_lobin, e = min(a + b.fftlen_ref / AB_NUMBETWEEN, sc.numbins);
    lo = (int) min(max(max(a, 0ll) - bin0, 0ll), (long long) SEG_H);
    hi = (int) max(min(e - bin0, (long long) SEG_H), 0ll);
}

// The points t + 64 m of a window (x: its point 0) times norm, zero outside
// points [lo, hi) and where not finite.
__device__ __forceinline__ void load_window(float2 (&v)[16], const float2 *x, int lo, int hi, int t, double norm)
{
#pragma unroll
    for (int m = 0; m < 16; m++) {
        const int k = t + FftShape<SEG_H>::NT * m;
        v[m] = make_float2(0.f, 0.f);
        if (k >= lo && k < hi) {
            const float2 a = x[k];
            if (isfinite(a.x) && isfinite(a.y))
                v[m] = make_float2((float) ((double) a.x * norm), (float) ((double) a.y * norm));
        }
    }
}

// Whether blocks [j0, j0 + nj) of one unit are to be kept apart (SEG_RANGE), as
// far as this warp's points of the window (k0, k0 + 64, ... below k1) tell.
__device__ __forceinline__ bool keep_apart(const SearchConsts &sc, const ab_bank &b, const SegCols *c, const double *nm,
                                           int j0, int nj, const float2 *x0, long long bin0, int k0, int k1)
{
    const int lane = threadIdx.x & 31;
    float n = 0.f, i = 0.f, a = 0.f;            // largest norm, 1 / norm and part of a value
    for (int j = j0 + lane; j < j0 + nj; j += 32) {
        const double x = nm[j];
        a = fmaxf(a, c[j].loud);
        if (!(x > 0.0 && isfinite(x))) continue;
        n = fmaxf(n, (float) x);
        i = fmaxf(i, (float) (1.0 / x));
    }
    n = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(n)));
    i = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(i)));
    a = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(a)));
    if (!(n * i <= SEG_RANGE)) return true;
    if (n * a <= SEG_RANGE) return false;
    // which values, against which blocks
    bool far = false;
    for (int j = j0; j < j0 + nj; j++) {
        const double x = nm[j];
        if (!(x > 0.0 && isfinite(x))) continue;
        int lo, hi;
        block_window(sc, b, c[j], bin0, lo, hi);
        for (int k = k0; k < k1; k += FftShape<SEG_H>::NT) {
            if ((k >= lo && k < hi) || bin0 + k < 0) continue;
            const float2 v = x0[k];
            far |= isfinite(v.x) && isfinite(v.y) && (double) fmaxf(fabsf(v.x), fabsf(v.y)) * x > (double) SEG_RANGE;
        }
    }
    return __any_sync(0xffffffffu, far);
}

// Forward transforms of the units' windows, four per CTA, and what the
// correlation needs to know of a unit.  apart: units whose blocks are kept
// apart, apart[0] of them in any order from apart[1] on.
__global__ void __launch_bounds__(256) k_seg_fwd(const ab_bank *banks, SearchConsts sc, BlockBatch bb,
                                                 const SegGroup *groups, int ngroups, int nunits,
                                                 const SegCols *cols, const double *norms, const float2 *fft,
                                                 const float2 *dtime, long long dt_per_block, float2 *xhat,
                                                 SegUnit *units, int *apart)
{
    using SH = FftShape<SEG_H>;
    extern __shared__ float2 fsm[];
    __shared__ int s_apart[SH::CTA / 32];
    const int grp = threadIdx.x / SH::NT, t = threadIdx.x - grp * SH::NT;
    const int unit = blockIdx.x * SH::G + grp;
    const bool ok = unit < nunits;
    const SegGroup g = group_of_unit(groups, ngroups, ok ? unit : nunits - 1);
    const ab_bank b = banks[g.bank];
    const int u = (ok ? unit : nunits - 1) - g.unit0;
    float2 v[16];
    if (g.nsub) {
        const int j = g.blk0 + u / g.nsub, off = u % g.nsub * (g.V / 2) + b.hw0 - g.hw;
        const int numdata = b.fftlen_ref / AB_NUMBETWEEN;
        const float2 *d = dtime + j * dt_per_block + b.dtime_off;
#pragma unroll
        for (int m = 0; m < 16; m++) v[m] = d[(off + t + SH::NT * m) % numdata];
        if (t == 0 && ok) units[unit] = SegUnit{1.0, u / g.nsub, 1};
        if (t == 0) s_apart[2 * grp] = s_apart[2 * grp + 1] = 0;
    } else {
        const SegCols *c = cols + (long long) g.bank * bb.nblk + g.blk0;
        const double *nm = norms + (long long) g.bank * bb.nblk + g.blk0;
        const long long q = c[0].c0 + (long long) u * g.V, bin0 = q / 2 - g.hw - sc.obs_lobin;
        const int j0 = first_block(c, g.nblk, q), nj = unit_blocks(c, j0, g.nblk, q, g.V);
        const double norm = unit_norm(nm, j0, g.nblk);
        // the windows of its blocks: nothing else is read
        int lo, hi, lo1, hi0;
        block_window(sc, b, c[j0], bin0, lo, hi0);
        block_window(sc, b, c[j0 + nj - 1], bin0, lo1, hi);
        const bool far = nj > 1 && keep_apart(sc, b, c, nm, j0, nj, fft + bin0, bin0, t, hi);
        if ((t & 31) == 0) s_apart[threadIdx.x >> 5] = far;
        if (t == 0 && ok) units[unit] = SegUnit{norm, j0, nj};
        load_window(v, fft + bin0, lo, hi, t, norm);
    }
    FftTw<SEG_H, -1> tw;
    tw.init(t);
    fft_run<SEG_H, -1>(v, fsm + grp * SH::SMEM, t, tw);     // (its barriers order s_apart)
    if (!ok) return;
    if (t == 0 && (s_apart[2 * grp] | s_apart[2 * grp + 1])) {
        units[unit].nj = -units[unit].nj;
        apart[1 + atomicAdd(apart, 1)] = unit;
    }
    float2 *o = xhat + (long long) unit * SEG_H;
#pragma unroll
    for (int m = 0; m < 16; m++) {
        const int k = t + SH::NT * m;
        o[seg_place(k)] = v[m];
    }
}

// ---------------------------------------------------------------------------
// correlation
// ---------------------------------------------------------------------------
constexpr int TW_OFF = SEG_H;                                   // float2
constexpr int EX_OFF = 2 * SEG_H;
constexpr size_t SEG_SMEM = sizeof(float2) * (EX_OFF + SEG_WARPS * 32 * SEG_P);

struct SegMap {
    int4 blk[SEG_MAXBLK];                       // first column, columns, offset, scale of a block here
    int4 first[32];                             // the first block of each group of 64 columns
    unsigned char jlo[32], more[32];
    float *row[SEG_TILE];                       // the templates' rows in the first block's plane
    unsigned any;                               // bit k: group k of 64 columns has further blocks
};

// exp(2 pi i l s / 1024) of lane l, bin s
__device__ __forceinline__ void fill_twiddles(float2 *tw)
{
    for (int i = threadIdx.x; i < SEG_H; i += blockDim.x) {
        double s, c;
        sincospi((double) (((i & 31) * (i >> 5)) & (SEG_H - 1)) * (2.0 / SEG_H), &s, &c);
        tw[seg_place(i)] = make_float2((float) c, (float) s);
    }
}

// One CTA: one unit (segment) and a tile of its class's templates.  A warp
// takes one of a template's two 1024-point inverse transforms (even or odd
// columns), 32 points a lane: radix 32 over the points 32 apart, the twiddles,
// one exchange through the warp's own shared memory, radix 32 again -- no
// barrier between warps and 8 bytes of exchange each way per point, where
// radix 16 needs two exchanges behind CTA barriers at 4096 points.
// Measured (B200): 4.8 to 5.1 ns per template and segment (5.3 to 5.7 before the
// powers were stored past L1, which they had swept of the templates, and with
// half the templates to a CTA).  At that stage shared memory and L1 data path
// were 58 % busy, the FP32 pipe 38 %, issue 47 %: held by latencies at the 16
// warps that 128 registers leave an SM.  Both transforms
// of a template in one warp's paired FP32 instructions halve the issue but
// leave 8 warps: 20 % slower.  Prefetching the next template into L1: 4 % slower;
// loads and butterflies interleaved by hand, or one body for both passes: the
// same.  Segments of 2048 bins with 4096-point transforms by a whole CTA (radix
// 16): 14.2 ns each, 16 % slower over the jerk search than this then was.
// The blocks of a unit are looked up once, by k_seg_fwd, and not by each of its
// CTAs: 107.4 -> 105.0 ms and 201.9 -> 199.6 (the two searches above).
//
// Here: tile `tile` of the group's templates against the data spectrum in fsm,
// normalised with ref, whose columns from q belong to nj blocks (c and nm: the
// first one's; blk0: its index in the batch).  All threads of the CTA.
__device__ __forceinline__ void corr_tile(const SegGroup &g, const ab_bank &b, const SearchConsts &sc, const SegCols *c,
                                          const double *nm, int blk0, int nj, long long q, double ref, int tile,
                                          const float2 *tmpl, const int *perm, float *planes,
                                          long long plane_per_block, float2 *fsm, SegMap &m)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int j = threadIdx.x; j < nj; j += blockDim.x) {
        const int tc0 = (int) (c[j].c0 - q) + 2 * g.hw;
        const int lo = max(tc0, 2 * g.hw), hi = min(tc0 + c[j].lim, 2 * g.hw + g.V);
        // element of this block's transform column 0, from the first block's (in
        // 32 bits: launch_corr_seg)
        const long long off = sc.inmem ? c[j].c0 - c[0].c0 - tc0 : (long long) j * plane_per_block - tc0;
        const double r = nm[j] / ref;
        m.blk[j] = make_int4(lo, max(hi - lo, 0), (int) off,
                             __float_as_int((float) (r * r) * (1.0f / ((float) SEG_H * SEG_H))));
    }
    for (int i = threadIdx.x; i < g.tile && tile * g.tile + i < g.nt; i += blockDim.x)
        m.row[i] = planes + (sc.inmem ? c[0].c0 : (long long) blk0 * plane_per_block + b.plane_off) +
                   perm[g.t_lo + tile * g.tile + i] * (sc.inmem ? sc.rlen : (long long) b.numrs_max);
    __syncthreads();
    if (threadIdx.x < 32) {
        const int k0 = 64 * threadIdx.x;
        int a = 0, n = 0;
        for (int j = 0; j < nj; j++) {
            const int4 e = m.blk[j];
            if (e.y > 0 && e.x < k0 + 64 && e.x + e.y > k0) {
                if (n == 0) a = j;
                n = j - a + 1;
            }
        }
        m.first[threadIdx.x] = n ? m.blk[a] : make_int4(0, 0, 0, 0);
        m.jlo[threadIdx.x] = (unsigned char) a;
        m.more[threadIdx.x] = (unsigned char) (n > 1 ? n - 1 : 0);
        const unsigned any = __ballot_sync(0xffffffffu, n > 1);
        if (threadIdx.x == 0) m.any = any;
    }
    __syncthreads();
    const float4 *xs = reinterpret_cast<const float4 *>(fsm) + lane;
    const float4 *tws = reinterpret_cast<const float4 *>(fsm + TW_OFF) + lane;
    float2 *ex = fsm + EX_OFF + warp * 32 * SEG_P;
    const float4 *ex4 = reinterpret_cast<const float4 *>(ex + lane * SEG_P);
    const int par = warp & 1;
    // (templates lie in the order of perm)
    const int nt = min(g.nt - tile * g.tile, g.tile);
    const float4 *kp = reinterpret_cast<const float4 *>(tmpl + b.seg_tmpl_off + par * SEG_H) + lane +
                       (long long) (g.t_lo - b.perm_off + tile * g.tile + (warp >> 1)) * SEG_H;
    for (int ti = warp >> 1; ti < nt; ti += SEG_WARPS / 2, kp += SEG_WARPS / 2 * SEG_H) {
        float2 v[32];
#pragma unroll
        for (int p = 0; p < 16; p++) {
            const float4 k = __ldg(kp + 32 * p);
            v[2 * p] = make_float2(k.x, k.y);
            v[2 * p + 1] = make_float2(k.z, k.w);
        }
#pragma unroll
        for (int p = 0; p < 16; p++) {
            const float4 x = xs[32 * p];
            v[2 * p] = cmulc(make_float2(x.x, x.y), v[2 * p]);
            v[2 * p + 1] = cmulc(make_float2(x.z, x.w), v[2 * p + 1]);
        }
        dft32(v);
#pragma unroll
        for (int p = 0; p < 16; p++) {
            const float4 w = tws[32 * p];
            const float2 y = v[bin32(2 * p)];
            ex[(2 * p) * SEG_P + lane] = p ? cmul(y, make_float2(w.x, w.y)) : y;
            ex[(2 * p + 1) * SEG_P + lane] = cmul(v[bin32(2 * p + 1)], make_float2(w.z, w.w));
        }
        __syncwarp();
#pragma unroll
        for (int p = 0; p < 16; p++) {
            const float4 y = ex4[p];
            v[2 * p] = make_float2(y.x, y.y);
            v[2 * p + 1] = make_float2(y.z, y.w);
        }
        __syncwarp();
        dft32(v);
        float *row = m.row[ti];
#pragma unroll
        for (int k = 0; k < 32; k++) {
            float2 &y = v[bin32(k)];
            y.x = fmaf(y.x, y.x, y.y * y.y);
            const int col = 64 * k + 2 * lane + par;
            const int4 e = m.first[k];
            if ((unsigned) (col - e.x) < (unsigned) e.y) __stcs(row + (e.z + col), y.x * __int_as_float(e.w));
        }
        if (const unsigned more = m.any) {
#pragma unroll
            for (int k = 0; k < 32; k++) {
                if (!((more >> k) & 1u)) continue;
                const int col = 64 * k + 2 * lane + par;
                for (int j = m.jlo[k] + 1, n = m.more[k]; n > 0; n--, j++) {
                    const int4 f = m.blk[j];
                    if ((unsigned) (col - f.x) < (unsigned) f.y)
                        __stcs(row + (f.z + col), v[bin32(k)].x * __int_as_float(f.w));
                }
            }
        }
    }
}

__global__ void __launch_bounds__(32 * SEG_WARPS, 2)
    k_corr_seg(const ab_bank *banks, SearchConsts sc, BlockBatch bb, const SegGroup *groups, int ngroups,
               const SegCols *cols, const double *norms, const float2 *xhat, const float2 *tmpl,
               const int *perm, const SegUnit *units, float *planes, long long plane_per_block)
{
    extern __shared__ __align__(16) float2 fsm[];
    __shared__ SegMap s_map;
    const SegGroup g = group_of_cta(groups, ngroups, blockIdx.x);
    const int r0 = blockIdx.x - g.cta0, u = r0 % g.nunits, tile = r0 / g.nunits;
    const SegUnit w = units[g.unit0 + u];
    if (w.nj < 0) return;                       // k_corr_apart's
    const ab_bank b = banks[g.bank];
    {
        const float4 *src = reinterpret_cast<const float4 *>(xhat + (long long) (g.unit0 + u) * SEG_H);
        float4 *dst = reinterpret_cast<float4 *>(fsm);
        for (int i = threadIdx.x; i < SEG_H / 2; i += blockDim.x) dst[i] = src[i];
        fill_twiddles(fsm + TW_OFF);
    }
    const long long at = (long long) g.bank * bb.nblk + g.blk0;
    const SegCols *c = cols + at;
    const long long q = g.nsub ? c[w.j0].c0 + (long long) (u % g.nsub) * g.V : c[0].c0 + (long long) u * g.V;
    corr_tile(g, b, sc, c + w.j0, norms + at + w.j0, g.blk0 + w.j0, w.nj, q, w.norm, tile, tmpl, perm, planes,
              plane_per_block, fsm, s_map);
}

// The units whose blocks are kept apart (SEG_RANGE), one block and tile of
// templates at a time: the block's data cut to its own window, transformed
// here.  One CTA per SM shares the list, which is all but always empty.
__global__ void __launch_bounds__(32 * SEG_WARPS, 1)
    k_corr_apart(const ab_bank *banks, SearchConsts sc, BlockBatch bb, const SegGroup *groups, int ngroups,
                 const SegCols *cols, const double *norms, const float2 *fft, const float2 *tmpl, const int *perm,
                 const SegUnit *units, const int *apart, float *planes, long long plane_per_block)
{
    using SH = FftShape<SEG_H>;
    extern __shared__ __align__(16) float2 fsm[];
    __shared__ SegMap s_map;
    const int n = apart[0];
    if (n == 0) return;
    fill_twiddles(fsm + TW_OFF);
    long long base = 0;                         // items of the units before this one
    for (int i = 0; i < n; i++) {
        const int unit = apart[1 + i];
        const SegGroup g = group_of_unit(groups, ngroups, unit);
        const SegUnit w = units[unit];
        const ab_bank b = banks[g.bank];
        const long long at = (long long) g.bank * bb.nblk + g.blk0;
        const long long q = cols[at].c0 + (long long) (unit - g.unit0) * g.V;
        const long long bin0 = q / 2 - g.hw - sc.obs_lobin;
        const int ntile = (g.nt + g.tile - 1) / g.tile, items = -w.nj * ntile;
        for (int k = (int) ((blockIdx.x + gridDim.x - base % gridDim.x) % gridDim.x); k < items; k += (int) gridDim.x) {
            const int j = w.j0 + k / ntile, tile = k % ntile;
            const SegCols *c = cols + at + j;
            const double *nm = norms + at + j;
            const double ref = unit_norm(nm, 0, 1);
            __syncthreads();                    // every warp has done with the last item
            {
                const int grp = threadIdx.x / SH::NT, t = threadIdx.x - grp * SH::NT;
                int lo, hi;
                block_window(sc, b, *c, bin0, lo, hi);
                float2 v[16];
                load_window(v, fft + bin0, lo, hi, t, ref);
                FftTw<SEG_H, -1> tw;
                tw.init(t);
                fft_run<SEG_H, -1>(v, fsm + EX_OFF + grp * SH::SMEM, t, tw);
                if (grp == 0) {                 // (the other groups did the same)
#pragma unroll
                    for (int m = 0; m < 16; m++) fsm[seg_place(t + SH::NT * m)] = v[m];
                }
            }
            corr_tile(g, b, sc, c, nm, g.blk0 + j, 1, q, ref, tile, tmpl, perm, planes, plane_per_block, fsm, s_map);
        }
        base += items;
    }
}

cudaError_t launch_seg_cols(const ab_bank *banks_dev, int nbanks, const SearchConsts &sc, const BlockBatch &bb,
                            const float2 *fft, int numdata_max, SegCols *cols, double *norms, int *apart, cudaStream_t st)
{
    const size_t smem = sizeof(float) * (size_t) numdata_max;
    if (smem > 48 * 1024) return cudaErrorInvalidValue;
    k_seg_cols<<<dim3((unsigned) bb.nblk, (unsigned) nbanks), 256, smem, st>>>(banks_dev, sc, bb, fft, cols, norms, apart);
    return cudaGetLastError();
}

cudaError_t launch_seg_fwd(const ab_bank *banks_dev, const SearchConsts &sc, const BlockBatch &bb,
                           const SegGroup *groups, int ngroups, int nunits, const SegCols *cols,
                           const double *norms, const float2 *fft, const float2 *dtime, long long dt_per_block,
                           float2 *xhat, SegUnit *units, int *apart, cudaStream_t st)
{
    using SH = FftShape<SEG_H>;
    if (nunits <= 0) return cudaSuccess;
    k_seg_fwd<<<(unsigned) ((nunits + SH::G - 1) / SH::G), SH::CTA, (size_t) SH::G * SH::SMEM * sizeof(float2), st>>>(
        banks_dev, sc, bb, groups, ngroups, nunits, cols, norms, fft, dtime, dt_per_block, xhat, units, apart);
    return cudaGetLastError();
}

cudaError_t launch_corr_seg(const ab_bank *banks_dev, const SearchConsts &sc, const BlockBatch &bb,
                            const SegGroup *groups, int ngroups, int nctas, const SegCols *cols,
                            const double *norms, const float2 *xhat, const float2 *tmpl, const int *perm,
                            const SegUnit *units, float *planes, long long plane_per_block, cudaStream_t st)
{
    if (nctas <= 0) return cudaSuccess;
    // corr_tile's offsets between blocks (ab_batch_blocks keeps to this)
    if (!sc.inmem && bb.nblk > 1 && bb.nblk * plane_per_block > INT_MAX) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(k_corr_seg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) SEG_SMEM);
    if (e != cudaSuccess) return e;
    k_corr_seg<<<(unsigned) nctas, 32 * SEG_WARPS, SEG_SMEM, st>>>(banks_dev, sc, bb, groups, ngroups, cols, norms,
                                                                  xhat, tmpl, perm, units, planes, plane_per_block);
    return cudaGetLastError();
}

cudaError_t launch_corr_apart(const ab_bank *banks_dev, const SearchConsts &sc, const BlockBatch &bb,
                              const SegGroup *groups, int ngroups, int nctas, const SegCols *cols,
                              const double *norms, const float2 *fft, const float2 *tmpl, const int *perm,
                              const SegUnit *units, const int *apart, float *planes, long long plane_per_block,
                              cudaStream_t st)
{
    if (nctas <= 0) return cudaSuccess;
    static_assert(4 * FftShape<SEG_H>::SMEM <= SEG_WARPS * 32 * SEG_P, "the transforms' exchange");
    cudaError_t e = cudaFuncSetAttribute(k_corr_apart, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) SEG_SMEM);
    if (e != cudaSuccess) return e;
    const unsigned grid = (unsigned) (nctas < 148 ? nctas : 148);
    k_corr_apart<<<grid, 32 * SEG_WARPS, SEG_SMEM, st>>>(banks_dev, sc, bb, groups, ngroups, cols, norms, fft, tmpl,
                                                        perm, units, apart, planes, plane_per_block);
    return cudaGetLastError();
}

}  // namespace ab
