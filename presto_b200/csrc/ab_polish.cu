// ab_polish.cu -- candidate polishing on the device: optimize_accelcand
// (src/accel_utils.c:552-626) for acceleration searches with harmonic
// polishing, the reference's default, every candidate of a search at once.
//
// A cluster of 1 to 8 CTAs of 512 threads per candidate runs
// max_rz_arr_harmonics (src/maximize_rz.c:173-228): local powers of the
// harmonics, two Nelder-Mead stages over (r, z / 4) maximising the sum of the
// harmonics' locally normalised powers (LOWACC kernels, step 0.4, size
// tolerance 1e-4; then HIGHACC kernels, step 0.01, 1e-7), then each harmonic's
// power, local power and derivatives (get_localpower3d, get_derivs3d,
// src/characteristics.c:79-193).  Complex amplitudes at fractional (r, z)
// come from rz_interp (src/rzinterp.c:144-232): a warp correlates the data
// with the FP64 response generated at the fractional offset, lanes splitting
// the kernel points.  The simplex bookkeeping runs identically in every
// thread; each function value is summed by one warp in the reference's
// harmonic order and broadcast through shared memory, so control flow stays
// uniform.  Iterations are bounded (5000 per stage, as the reference).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>

#include "ab_kernels.h"
#include "ab_resp.cuh"

namespace cg = cooperative_groups;

namespace ab {
namespace {

constexpr int PL_THREADS = 512;
constexpr int PL_WARPS = PL_THREADS / 32;
constexpr int PL_MAXH = AB_POLISH_MAX_HARM;
constexpr int PL_LOCPOW = 20;                 // NUMLOCPOWAVG, include/presto.h:99
constexpr int PL_DELTA = 5;                   // DELTAAVGBINS, include/presto.h:103
constexpr double PL_ZSCALE = 4.0;             // src/maximize_rz.c:6
constexpr int PL_ITEMS = PL_MAXH * PL_LOCPOW;

__device__ __forceinline__ int z_halfwidth(double z, bool highacc)   // src/responses.c:27-47
{
    return (int) (0.5 * 1.1 * fabs(z)) + (highacc ? 48 : 16);
}

// |z| below the fast points' range (out of line: its registers are not the
// loop's)
__device__ __noinline__ double2 slow_point(double frac, double z, int numkern, int c)
{
    return z_resp_point(frac, 1, z, numkern, c);
}

// rz_interp (src/rzinterp.c:144-232) at (r, z) with kernel half-width hw,
// shared by P warps: this lane of warp part sums kernel points lane + 32 (part
// + P k) in FP64.  The lanes' and parts' sums add up to the amplitude; the
// exact-bin cases come from lane 0 of part 0 alone.
__device__ __noinline__ double2 rz_interp_part(const float2 *data, long long numdata, double r, double z, int hw,
                                  int part, int P, int lane, const double2 *tab)
{
    if (r > numdata - 1.0 || r < 0.0) return make_double2(0.0, 0.0);
    double dint;
    const double frac = modf(r, &dint);
    const long long intfreq = (long long) dint;
    if (fabs(z) < 1E-4) {
        const bool first = part == 0 && lane == 0;
        if (frac < 1E-5) {
            const float2 v = data[intfreq];
            return first ? make_double2(v.x, v.y) : make_double2(0.0, 0.0);
        }
        if ((1.0 - frac) < 1E-5) {
            const float2 v = data[intfreq + 1];
            return first ? make_double2(v.x, v.y) : make_double2(0.0, 0.0);
        }
    }
    const int numkern = 2 * hw;
    long long lodata = intfreq - hw, loresp = 0;
    if (lodata < 0) {
        loresp = -lodata;
        lodata = 0;
    }
    const long long hidata = intfreq + hw - 1;
    const long long hiresp = (hidata > numdata - 1) ? numkern - hidata + numdata - 1 : numkern;
    const long long nsum = hiresp - loresp;
    double ar = 0.0, ai = 0.0;
    const bool fast = fabs(z) >= 1e-3;
    ZResp zr;
    if (fast) zr.init(frac, z, numkern);
    for (long long ii = lane + 32 * part; ii < nsum; ii += 32 * P) {
        const double2 pv = fast ? zr.point((int) (loresp + ii), tab)
                                : slow_point(frac, z, numkern, (int) (loresp + ii));
        const float pr = (float) pv.x, pim = (float) pv.y;      // the reference's response is float
        const float2 d = data[lodata + ii];
        ar += (double) d.x * (double) pr + (double) __fmul_rn(d.y, pim);
        ai += (double) d.y * (double) pr - (double) pim * (double) d.x;
    }
    return make_double2(ar, ai);
}

__device__ __forceinline__ double2 warp_sum(double2 v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    return v;
}

// rz_interp by one warp.
__device__ float2 warp_rz_interp(const float2 *data, long long numdata, double r, double z, int hw,
                                 int lane, const double2 *tab)
{
    const double2 v = warp_sum(rz_interp_part(data, numdata, r, z, hw, 0, 1, lane, tab));
    return make_float2((float) v.x, (float) v.y);
}

__device__ __forceinline__ double powerf2(float2 a) { return (double) a.x * a.x + (double) a.y * a.y; }

constexpr int PL_MAXK = 8;                    // CTAs (one cluster) per candidate at most
constexpr int PL_PARTS = PL_MAXK * PL_WARPS;

struct PolishSmem {
    double2 tab[FRESNEL_TAB];
    double r[PL_ITEMS], z[PL_ITEMS];
    int hw[PL_ITEMS];
    float2 amp[PL_ITEMS];
    int cnt[PL_MAXH];
    float locpow[PL_MAXH];
    double2 part[2][PL_PARTS];  // partial amplitudes of one evaluation, by turns
    double val;
    int nitem;
    int raw;                    // max_rz_arr: one harmonic, raw power (-noharmpolish)
};

// The cluster's CTAs run the same simplex: each keeps all the partial sums
// and amplitudes, its own and those that the others' warps store into its
// shared memory, adds them in the same order and so takes the same turns.  One
// cluster barrier per evaluation: the partial sums alternate between two
// buffers, and a CTA passes the barrier behind evaluation n + 1 only after
// every CTA has read those of evaluation n.
struct Team {
    int k, rank, gwarp, nwarps, lane, turn;
    __device__ __forceinline__ void init()
    {
        k = (int) cg::this_cluster().num_blocks();
        rank = (int) cg::this_cluster().block_rank();
        gwarp = rank * PL_WARPS + (threadIdx.x >> 5);
        nwarps = k * PL_WARPS;
        lane = threadIdx.x & 31;
        turn = 0;
    }
    __device__ __forceinline__ void sync() const
    {
        if (k > 1) cg::this_cluster().sync();
        else __syncthreads();
    }
    // *at = v in every CTA's shared memory (lanes of the warp, one CTA each)
    template <class T> __device__ __forceinline__ void store(T *at, T v) const
    {
        if (k == 1) {
            if (lane == 0) *at = v;
        } else if (lane < k) {
            *cg::this_cluster().map_shared_rank(at, lane) = v;
        }
    }
};

// Amplitudes of items [0, n) but those in [skip0, skip1) (all threads of the
// cluster).
__device__ void interp_items(const float2 *data, long long numdata, int n, int skip0, int skip1, PolishSmem &s,
                             const Team &tm)
{
    for (int it = tm.gwarp; it < n; it += tm.nwarps) {
        if (it >= skip0 && it < skip1) continue;
        const float2 a = warp_rz_interp(data, numdata, s.r[it], s.z[it], s.hw[it], tm.lane, s.tab);
        tm.store(&s.amp[it], a);
    }
    tm.sync();
}

// get_localpower3d (w = 0) of harmonic n = 1..nh at (r n, z n) into s.locpow
// (float, as max_rz_arr_harmonics keeps them).
__device__ void local_powers(const float2 *data, long long numdata, double r, double z, int nh,
                             PolishSmem &s, const Team &tm)
{
    if (threadIdx.x == 0) {
        int k = 0;
        for (int ii = 0; ii < nh; ii++) {
            const double rh = r * (ii + 1), zh = z * (ii + 1);
            const int hw = z_halfwidth(zh, false);
            double lo1 = rh - PL_DELTA - PL_LOCPOW / 2, hi1 = lo1 + PL_LOCPOW / 2;
            double lo2 = rh + PL_DELTA, hi2 = lo2 + PL_LOCPOW / 2;
            double *b[4] = {&lo1, &lo2, &hi1, &hi2};
            for (int q = 0; q < 4; q++) {
                if (*b[q] < 0.0) *b[q] = 0.0;
                if (*b[q] > numdata) *b[q] = (double) numdata;
            }
            int c = 0;
            for (double f = lo1; f < hi1 && k < PL_ITEMS; f += 1.0, c++, k++) {
                s.r[k] = f;
                s.z[k] = zh;
                s.hw[k] = hw;
            }
            for (double f = lo2; f < hi2 && k < PL_ITEMS; f += 1.0, c++, k++) {
                s.r[k] = f;
                s.z[k] = zh;
                s.hw[k] = hw;
            }
            s.cnt[ii] = c;
        }
        s.nitem = k;
    }
    tm.sync();                                  // and every CTA is done with its last amplitudes
    interp_items(data, numdata, s.nitem, 0, 0, s, tm);
    if (threadIdx.x == 0) {
        int k = 0;
        for (int ii = 0; ii < nh; ii++) {
            double sum = 0.0;
            for (int c = 0; c < s.cnt[ii]; c++, k++) sum += powerf2(s.amp[k]);
            s.locpow[ii] = (float) (sum / (double) PL_LOCPOW);
        }
    }
    __syncthreads();
}

// Minus the summed normalised power of the harmonics at (r, zs * ZSCALE)
// (power_call_rz_harmonics_gsl, src/maximize_rz.c:42-62); all threads.
__device__ __noinline__ double eval_harmonics(const float2 *data, long long numdata, int nh, int kernhw, double r,
                                 double zs, PolishSmem &s, Team &tm)
{
    // P warps per harmonic (all warps of the cluster busy for few harmonics)
    const int P = nh >= tm.nwarps ? 1 : tm.nwarps / nh;
    double2 *part = s.part[tm.turn];
    tm.turn ^= 1;
    for (int w = tm.gwarp; w < nh * P; w += tm.nwarps) {
        const int ii = w / P, n = ii + 1;
        const double2 v = warp_sum(rz_interp_part(data, numdata, r * n, zs * PL_ZSCALE * n, kernhw,
                                                  w - ii * P, P, tm.lane, s.tab));
        tm.store(&part[w], v);
    }
    tm.sync();
    // one warp: a lane per harmonic, the sum over harmonics in order
    if (threadIdx.x < 32) {
        double term = 0.0;
        if (tm.lane < nh) {
            double ar = 0.0, ai = 0.0;
            for (int q = 0; q < P; q++) {
                ar += part[tm.lane * P + q].x;
                ai += part[tm.lane * P + q].y;
            }
            const float2 a = make_float2((float) ar, (float) ai);
            term = s.raw ? powerf2(a) : powerf2(a) / (double) s.locpow[tm.lane];
        }
        double total = 0.0;
        for (int ii = 0; ii < nh; ii++) total += __shfl_sync(0xffffffffu, term, ii);
        // power_call_rz (src/maximize_rz.c:10-23) for one raw power
        if (tm.lane == 0) s.val = s.raw ? -total : (isfinite(total) ? -total : 0.0);
    }
    __syncthreads();
    const double v = s.val;
    __syncthreads();
    return v;
}

// Nelder-Mead over (r, zs), the oracle's orc_nm_minimize step for step.
__device__ double nm_minimize(const float2 *data, long long numdata, int nh, int kernhw, double *x,
                              double step, double tol, PolishSmem &s, Team &tm)
{
    double v[3][2], fv[3], xt[2], xt2[2];
    for (int i = 0; i < 3; i++) {
        v[i][0] = x[0];
        v[i][1] = x[1];
        if (i > 0) v[i][i - 1] += step;
        fv[i] = eval_harmonics(data, numdata, nh, kernhw, v[i][0], v[i][1], s, tm);
    }
    for (int iter = 0; iter < 5000; iter++) {
        int hi = 0, lo = 0;
        for (int i = 1; i < 3; i++) {
            if (fv[i] > fv[hi]) hi = i;
            if (fv[i] < fv[lo]) lo = i;
        }
        int shi = (hi == 0) ? 1 : 0;
        for (int i = 0; i < 3; i++)
            if (i != hi && fv[i] > fv[shi]) shi = i;
        double c[2] = {0.0, 0.0};
        for (int i = 0; i < 3; i++)
            if (i != hi) {
                c[0] += v[i][0];
                c[1] += v[i][1];
            }
        c[0] /= 2;
        c[1] /= 2;
        // x(t) = (1 - t) c + t x_worst
        xt[0] = 2.0 * c[0] - v[hi][0];
        xt[1] = 2.0 * c[1] - v[hi][1];
        const double fr = eval_harmonics(data, numdata, nh, kernhw, xt[0], xt[1], s, tm);
        if (fr < fv[lo]) {
            xt2[0] = 3.0 * c[0] - 2.0 * v[hi][0];
            xt2[1] = 3.0 * c[1] - 2.0 * v[hi][1];
            const double fe = eval_harmonics(data, numdata, nh, kernhw, xt2[0], xt2[1], s, tm);
            if (fe < fv[lo]) {
                v[hi][0] = xt2[0];
                v[hi][1] = xt2[1];
                fv[hi] = fe;
            } else {
                v[hi][0] = xt[0];
                v[hi][1] = xt[1];
                fv[hi] = fr;
            }
        } else if (fr > fv[shi]) {
            if (fr <= fv[hi]) {
                v[hi][0] = xt[0];
                v[hi][1] = xt[1];
                fv[hi] = fr;
            }
            xt2[0] = 0.5 * c[0] + 0.5 * v[hi][0];
            xt2[1] = 0.5 * c[1] + 0.5 * v[hi][1];
            const double fc = eval_harmonics(data, numdata, nh, kernhw, xt2[0], xt2[1], s, tm);
            if (fc <= fv[hi]) {
                v[hi][0] = xt2[0];
                v[hi][1] = xt2[1];
                fv[hi] = fc;
            } else {
                for (int i = 0; i < 3; i++) {
                    if (i == lo) continue;
                    v[i][0] = 0.5 * (v[i][0] + v[lo][0]);
                    v[i][1] = 0.5 * (v[i][1] + v[lo][1]);
                    fv[i] = eval_harmonics(data, numdata, nh, kernhw, v[i][0], v[i][1], s, tm);
                }
            }
        } else {
            v[hi][0] = xt[0];
            v[hi][1] = xt[1];
            fv[hi] = fr;
        }
        double m0 = 0.0, m1 = 0.0, s2 = 0.0;
        for (int i = 0; i < 3; i++) {
            m0 += v[i][0] / 3;
            m1 += v[i][1] / 3;
        }
        for (int i = 0; i < 3; i++) {
            s2 += (v[i][0] - m0) * (v[i][0] - m0);
            s2 += (v[i][1] - m1) * (v[i][1] - m1);
        }
        if (sqrt(s2 / 3) < tol) break;
    }
    int lo = 0;
    for (int i = 1; i < 3; i++)
        if (fv[i] < fv[lo]) lo = i;
    x[0] = v[lo][0];
    x[1] = v[lo][1];
    return fv[lo];
}

__global__ void __launch_bounds__(PL_THREADS) k_polish_rz(const float2 *data, long long numdata,
                                                          long long lobin, const PolishIn *in,
                                                          const double2 *fresnel_tab, ab_polished *out)
{
    __shared__ PolishSmem s;
    Team tm;
    tm.init();
    const PolishIn c = in[blockIdx.x / tm.k];
    ab_polished &o = out[blockIdx.x / tm.k];
    for (int i = threadIdx.x; i < FRESNEL_TAB; i += blockDim.x) s.tab[i] = fresnel_tab[i];
    const int nh = c.mode == 1 ? 1 : (c.numharm < 1 ? 1 : (c.numharm > PL_MAXH ? PL_MAXH : c.numharm));
    if (threadIdx.x == 0) s.raw = c.mode == 1;
    const double rin = c.r - (double) lobin, zin = c.z;
    local_powers(data, numdata, rin, zin, nh, s, tm);
    double x[2] = {rin, zin / PL_ZSCALE};
    int kernhw = z_halfwidth(fabs(zin * nh) + 4.0, false);
    nm_minimize(data, numdata, nh, kernhw, x, 0.4, 1.0e-4, s, tm);
    kernhw = z_halfwidth(fabs(x[1] * nh) + 4.0, true);
    nm_minimize(data, numdata, nh, kernhw, x, 0.01, 1.0e-7, s, tm);
    const double rout = x[0], zout = x[1] * PL_ZSCALE;
    local_powers(data, numdata, rout, zout, nh, s, tm);
    // harmonic powers (HIGHACC kernel of the second stage) and the five
    // derivative points r n - 0.006 .. + 0.006 (get_derivs3d) per harmonic
    if (threadIdx.x == 0) {
        for (int ii = 0; ii < nh; ii++) {
            const int n = ii + 1;
            const double zs = zout / PL_ZSCALE * n;
            s.r[ii] = rout * n;
            s.z[ii] = zs * PL_ZSCALE;
            s.hw[ii] = kernhw;
            const int hwd = z_halfwidth(zout * n, true);
            double f = rout * n - 0.006;
            for (int q = 0; q < 5; q++, f += 0.003) {
                const int k = PL_MAXH + 5 * ii + q;
                s.r[k] = f;
                s.z[k] = zout * n;
                s.hw[k] = hwd;
            }
        }
    }
    tm.sync();
    // items: [0, nh) powers, [PL_MAXH, PL_MAXH + 5 nh) derivative points
    interp_items(data, numdata, PL_MAXH + 5 * nh, nh, PL_MAXH, s, tm);
    tm.sync();                                  // no CTA leaves while another may store into it
    if (threadIdx.x == 0 && tm.rank == 0) {
        const double pi = 3.14159265358979323846, twopi = 6.28318530717958647692;
        o.numharm = nh;
        for (int ii = 0; ii < nh; ii++) {
            const int n = ii + 1;
            o.hirs[ii] = (rout + (double) lobin) * n;
            o.hizs[ii] = zout * n;
            o.hiws[ii] = 0.0;
            o.pows[ii] = powerf2(s.amp[ii]);
            double pwr[5], phs[5];
            for (int q = 0; q < 5; q++) {
                const float2 a = s.amp[PL_MAXH + 5 * ii + q];
                pwr[q] = powerf2(a);
                const double t = atan2((double) a.y, (double) a.x);
                phs[q] = t > 0.0 ? t : t + twopi;
            }
            for (int q = 0; q < 4; q++)
                if (fabs(phs[q + 1] - phs[q]) > pi) phs[q + 1] -= twopi;
            ab_rderivs &d = o.derivs[ii];
            d.pow = pwr[2];
            d.phs = phs[2];
            d.dpow = (pwr[3] - pwr[1]) / 0.006;
            d.dphs = (phs[3] - phs[1]) / 0.006;
            d.d2pow = (pwr[4] - 2.0 * pwr[2] + pwr[0]) / 0.000036;
            d.d2phs = (phs[4] - 2.0 * phs[2] + phs[0]) / 0.000036;
            d.locpow = (double) s.locpow[ii];
        }
    }
}

}  // namespace

static_assert(FRESNEL_TAB == POLISH_FRESNEL_TAB, "table length");

// f and g at k / FRESNEL_STEPS: the system f' = -pi x g, g' = pi x f - 1 is
// neutrally stable, so Taylor steps in extended precision carry the asymptotic
// values at x = 9 (terms below 1e-21) down to 0 with their accuracy.
void fresnel_table(double2 *out)
{
    const long double pi = 3.14159265358979323846264338327950288L;
    const int k0 = 9 * FRESNEL_STEPS;
    long double x = 9.0L, h = 1.0L / (pi * x * x), f = 1.0L, g = 1.0L;
    for (int m = 14; m >= 1; m--) {
        f = 1.0L - (long double) ((4 * m - 3) * (4 * m - 1)) * h * h * f;
        g = 1.0L - (long double) ((4 * m - 1) * (4 * m + 1)) * h * h * g;
    }
    f *= h * x;
    g *= h * h * x;
    const long double d = -1.0L / FRESNEL_STEPS;
    for (int k = k0; k >= 0; k--) {
        if (k < FRESNEL_TAB) out[k] = make_double2((double) f, (double) g);
        x = (long double) k / FRESNEL_STEPS;
        long double a0 = f, b0 = g, a1 = -pi * x * g, b1 = pi * x * f - 1.0L, p = d;
        f += a1 * p;
        g += b1 * p;
        for (int n = 1; n < 24; n++) {
            const long double a2 = -pi * (x * b1 + b0) / (n + 1), b2 = pi * (x * a1 + a0) / (n + 1);
            p *= d;
            f += a2 * p;
            g += b2 * p;
            a0 = a1;
            b0 = b1;
            a1 = a2;
            b1 = b2;
        }
    }
}

// CTAs per candidate.  Its evaluations follow one another, so a candidate's
// time is a chain: a cluster of up to 8 CTAs (one per SM) shares each evaluation's
// kernel points while that leaves a thread four of them, which also evens
// out lists whose candidates differ in length; very long lists fill the SMs
// on their own.
static int polish_cluster(const PolishIn *in, int n)
{
    double most = 0.0;
    for (int i = 0; i < n; i++) {
        const int nh = in[i].mode == 1 ? 1 : in[i].numharm;
        most = fmax(most, nh * 2.0 * (0.55 * (fabs(in[i].z * nh) + 4.0) + 48.0));
    }
    int k = 1;
    while (k < PL_MAXK && most >= 4.0 * PL_THREADS * k && 2LL * k * n <= 16 * 148) k *= 2;
    return k;
}

cudaError_t launch_polish(const float2 *data, long long numdata, long long lobin, const PolishIn *in_host,
                          const PolishIn *in, int n, const double2 *fresnel_tab, ab_polished *out, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    const int k = polish_cluster(in_host, n);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned) n * k);
    cfg.blockDim = dim3(PL_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned) k;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_polish_rz, data, numdata, lobin, in, fresnel_tab, out);
}

}  // namespace ab
