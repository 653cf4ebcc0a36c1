// ab_norm.cuh -- spectrum normalisation helpers shared by the search's block
// preparation and the time-series path.
#pragma once
#include <cuda_runtime.h>

#include "ab_kernels.h"
#include "ab_select.cuh"

namespace ab {

// invsqrtf (src/misc_utils.c:291-302): the published fast inverse square
// root, one Newton step, in float with explicit rounding.
__device__ __forceinline__ float fast_invsqrtf(float x)
{
    const float y = __int_as_float(0x5f3759df - (__float_as_int(x) >> 1));
    const float t = __fmul_rn(__fmul_rn(__fmul_rn(0.5f, x), y), y);
    return __fmul_rn(y, __fsub_rn(1.5f, t));
}

// -locpow: the factor invsqrtf(local power) that scales bin i of a block's
// window of numdata powers pw (src/accel_utils.c:1100-1113).  corr_loc_pow
// (src/corr_routines.c:309-366) correlates the powers with a double top-hat
// of 20 taps at offsets +-6..+-15 bins, each (numdata / 2) / NUMLOCPOWAVG in
// integer arithmetic, through real FFTs whose round trip carries 2 / numdata:
//   local[i] = (2 / numdata) floor(numdata / 40) sum_{6 <= |j| <= 15} pw[i + j],
// and the first and last 15 bins take the value of the nearest bin 15 from
// the edge.  The sum is formed exactly here (the reference's FP32 FFTs round
// it); no tap wraps, since every bin used lies 15 or more from the edges.
__device__ __forceinline__ float locpow_invsqrt(const float *pw, int numdata, int i)
{
    constexpr int khw = 20 / 2 + 5;                    // NUMLOCPOWAVG / 2 + DELTAAVGBINS
    const int c = i < khw ? khw : (i > numdata - 1 - khw ? numdata - 1 - khw : i);
    double s = 0.0;
#pragma unroll
    for (int j = 6; j <= khw; j++) s += (double) pw[c - j] + (double) pw[c + j];
    const double normal = (double) ((numdata / 2) / 20);
    const float local = (float) (s * normal * (2.0 / (double) numdata));
    return fast_invsqrtf(local);
}

// Block normalisation 1/sqrt(median(|X|^2)/ln 2) of the numdata bins from
// lobin (zero outside the spectrum), or 1/sqrt(nph) when nph is given
// (src/accel_utils.c:1079-1099).  The median is taken over float POWER()
// values without FMA, sorted exactly; even counts average the two central
// values (GSL semantics).  pw: shared scratch of numdata floats.
// Called by every thread of the CTA.
// The block's normalisation (src/accel_utils.c:1079-1113): 1/sqrt(nph) with
// -photon, else 1/sqrt(median/ln 2) of the window's powers.  With -locpow
// (sc.norm_type 1) it leaves the window's powers in pw for locpow_invsqrt
// and returns 0 (the factor is per bin).
__device__ __forceinline__ double block_norm(const SearchConsts &sc, long long lobin, int numdata, const float2 *fft,
                             float *pw, double *s_norm)
{
    if (sc.nph > 0.0f) {
        if (threadIdx.x == 0) *s_norm = 1.0 / sqrt((double) sc.nph);
    } else if (sc.norm_type == 1) {
        for (int i = threadIdx.x; i < numdata; i += blockDim.x) {
            long long bin = lobin + i - sc.obs_lobin;
            float2 v = (bin >= 0 && bin < sc.numbins) ? fft[bin] : make_float2(0.f, 0.f);
            pw[i] = __fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y));
        }
        if (threadIdx.x == 0) *s_norm = 0.0;
    } else {
        // block median of |X|^2 in float (POWER(), no FMA), src/accel_utils.c:1087-1099
        for (int i = threadIdx.x; i < numdata; i += blockDim.x) {
            long long bin = lobin + i - sc.obs_lobin;
            float2 v = (bin >= 0 && bin < sc.numbins) ? fft[bin] : make_float2(0.f, 0.f);
            pw[i] = __fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y));
        }
        __syncthreads();
        // the two central order statistics (equal for odd counts), as a sort gives them
        __shared__ unsigned s_hist[256], s_res[2];
        const float lo = select_rank(pw, numdata, (numdata - 1) / 2, s_hist, s_res);
        const float hi = (numdata & 1) ? lo : next_rank(pw, numdata, (numdata - 1) / 2, lo, s_res);
        if (threadIdx.x == 0) {
            double m = (numdata & 1) ? (double) lo : 0.5 * ((double) lo + (double) hi);
            float med = (float) m;
            *s_norm = 1.0 / sqrt((double) med / 0.69314718055994530942);
        }
    }
    __syncthreads();
    return *s_norm;
}

}  // namespace ab
