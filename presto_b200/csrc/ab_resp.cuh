// ab_resp.cuh -- FP64 response generators shared by the template kernels and
// the candidate polisher: Fresnel integrals and the r / z response points.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace ab {

// ======================================================================
// FP64 Fresnel integrals: power series for x <= 1.8, Lentz continued
// fraction for erfc((1-i) sqrt(pi)/2 x) up to 5.5 (Numerical Recipes 2ed
// section 6.9), and above that the auxiliary functions' asymptotic series
// (Abramowitz & Stegun 7.3.27-28; C and S from f and g by 7.3.9-10), whose
// terms fall below 1e-18 within about a dozen steps there (3.6e-14 absolute
// against Cephes' fresnl over 5.5..40).
// ======================================================================
__device__ __forceinline__ void fresnel64(double xin, double *s, double *c)
{
    double x = fabs(xin), S, C;
    if (x < 1e-300) {
        S = 0.0;
        C = 0.0;
    } else if (x <= 1.8) {
        double t = 0.5 * M_PI * x * x, term = x, sc = 0.0, ss = 0.0;
        for (int k = 0; k < 200; k++) {
            double contrib = term / (2 * k + 1);
            switch (k & 3) {
                case 0: sc += contrib; break;
                case 1: ss += contrib; break;
                case 2: sc -= contrib; break;
                default: ss -= contrib; break;
            }
            term *= t / (k + 1);
            if (k > 4 && fabs(term) < 1e-18 * (fabs(sc) + fabs(ss))) break;
        }
        C = sc;
        S = ss;
    } else if (x >= 5.5) {
        const double px2 = M_PI * x * x, t = 1.0 / (px2 * px2);
        double f = 1.0, g = 1.0, c = 1.0, d = 1.0;
        for (int m = 1; m < 40; m++) {
            c *= -(double) ((4 * m - 3) * (4 * m - 1)) * t;
            d *= -(double) ((4 * m - 1) * (4 * m + 1)) * t;
            f += c;
            g += d;
            if (fabs(c) < 1e-18 && fabs(d) < 1e-18) break;
        }
        f /= M_PI * x;
        g /= M_PI * M_PI * x * x * x;
        double sp, cp;
        sincospi(0.5 * x * x, &sp, &cp);           // sin, cos(pi x^2 / 2)
        C = 0.5 + f * sp - g * cp;
        S = 0.5 - f * cp - g * sp;
    } else {
        const double fpmin = 1e-300;
        double px2 = M_PI * x * x;
        double br = 1.0, bi = -px2, cr = 1.0 / fpmin, ci = 0.0;
        double den = br * br + bi * bi;
        double dr = br / den, di = -bi / den, hr = dr, hi = di;
        for (int n = 1; n < 100000; n++) {
            double an = -(double) (2 * n - 1) * (double) (2 * n);
            br += 4.0;
            double tr = an * dr + br, ti = an * di + bi;
            den = tr * tr + ti * ti;
            dr = tr / den;
            di = -ti / den;
            den = cr * cr + ci * ci;
            cr = br + an * cr / den;
            ci = bi - an * ci / den;
            double delr = cr * dr - ci * di, deli = cr * di + ci * dr;
            double nhr = hr * delr - hi * deli, nhi = hr * deli + hi * delr;
            hr = nhr;
            hi = nhi;
            if (fabs(delr - 1.0) + fabs(deli) < 1e-16) break;
        }
        double sp, cp;
        sincospi(0.5 * x * x, &sp, &cp);             // e^{i pi x^2 / 2}
        double ar = x * (cp + sp), ai = x * (sp - cp);
        double fr = ar * hr - ai * hi, fi = ar * hi + ai * hr;
        double gr = 1.0 - fr, gi = -fi;
        C = 0.5 * (gr - gi);
        S = 0.5 * (gr + gi);
    }
    if (xin < 0.0) {
        C = -C;
        S = -S;
    }
    *s = S;
    *c = C;
}

// gen_r_response point c (src/responses.c:159-225), written with direct
// sin/cos of the exact argument instead of the trig recursion.
__device__ __forceinline__ double2 r_resp_point(double roffset, int numbetween, int numkern, int c)
{
    double rbypi = numkern / (double) (2 * numbetween) + roffset - (double) c / numbetween;
    double s, co;
    sincospi(rbypi, &s, &co);
    double r = M_PI * rbypi;
    double sinc = (r == 0.0) ? 1.0 : s / r;
    double2 v = make_double2(co * sinc, s * sinc);
    if (roffset < 1E-3 && c == numkern / 2) {
        double t = roffset * roffset;
        v = make_double2(1 - 6.579736267392905746 * t, roffset * (M_PI - 10.335425560099940058 * t));
    }
    return v;
}

// gen_z_response point c (src/responses.c:228-316)
__device__ __forceinline__ double2 z_resp_point(double roffset, int numbetween, double z, int numkern, int c)
{
    double absz = fabs(z);
    if (absz < 1E-4) return r_resp_point(roffset, numbetween, numkern, c);
    double startr = roffset - (0.5 * z), ip;
    double startroffset = (startr < 0) ? 1.0 + modf(startr, &ip) : modf(startr, &ip);
    int signz = (z < 0.0) ? -1 : 1;
    double zd = signz * M_SQRT2 / sqrt(absz);
    double cons = zd / 2.0;
    double pibyz = M_PI / z;
    startr += numkern / (double) (2 * numbetween);
    double r = startr + c * (-1.0 / numbetween);
    double yy = r * zd;
    double zz = yy + z * zd;
    double xx = pibyz * r * r;
    double sx, cx;
    sincos(xx, &sx, &cx);
    double fsy, fcy, fsz, fcz;
    fresnel64(yy, &fsy, &fcy);
    fresnel64(zz, &fsz, &fcz);
    double tr = signz * (fcz - fcy), ti = fsy - fsz;
    double2 v = make_double2((tr * cx - ti * sx) * cons, -(tr * sx + ti * cx) * cons);
    if (startroffset < 1E-3 && absz < 1E-3 && c == numkern / 2) {
        double z2 = z * z, x2 = startroffset * startroffset;
        v.x = 1.0 - 0.16449340668482264365 * z2;
        v.y = -0.5235987755982988731 * z;
        v.x += startroffset * 1.6449340668482264365 * z;
        v.y += startroffset * (M_PI - 0.5167712780049970029 * z2);
        v.x += x2 * (-6.579736267392905746 + 0.9277056288952613070 * z2);
        v.y += x2 * (3.1006276680299820175 * z);
    }
    return v;
}

// ======================================================================
// Fast response points (candidate polishing).  With the auxiliary functions
// f and g (Abramowitz & Stegun 7.3.5-6), C + iS at x > 0 is
//   (1 + i) / 2 - (g + i f) exp(i pi x^2 / 2),
// and along a response both Fresnel arguments have the phase of the point's
// own factor exp(-i pi r^2 / z), up to a constant: only the points between the
// two ends of the drift need a sine and a cosine at all, and f and g vary
// slowly.  About 170 FP64 operations a point; three sines and cosines, two
// series term by term and, for 1.8 < x < 5.5, continued fractions of some
// thirty divisions each took several times that (with up to 8 CTAs a
// candidate, 160 candidates of a zmax = 600 search with 16 harmonics went from
// 104 to 39 ms and from 302 to 64 ms; B200).
// ======================================================================
constexpr int FRESNEL_STEPS = 64;               // table points per unit of x
constexpr int FRESNEL_TAB = 353;                // x = 0 .. 5.5

// f and g at x >= 0.  Up to 5.5 the Taylor series about the nearest table
// point, |d| <= 1/128, its coefficients from f' = -pi x g and g' = pi x f - 1:
// the first left out is below 1e-18 (f and g are smooth: coefficient n falls
// like x^-n, and like pi^(n/2) / (n/2)! at 0).  Above, the asymptotic series
// (7.3.27-28) to m = 11, whose next term is below 1e-18 at 5.5.
__device__ __forceinline__ void fresnel_fg(double x, const double2 *tab, double &f, double &g)
{
    if (x < 5.5) {
        const int k = __double2int_rn(x * FRESNEL_STEPS);
        const double x0 = (double) k * (1.0 / FRESNEL_STEPS), d = x - x0;
        const double2 t = tab[k];
        double a0 = t.x, b0 = t.y, p = d;
        double a1 = -M_PI * (x0 * b0), b1 = fma(M_PI, x0 * a0, -1.0);
        f = fma(a1, p, a0);
        g = fma(b1, p, b0);
#pragma unroll
        for (int n = 1; n < 9; n++) {
            const double c = M_PI / (n + 1);
            const double a2 = -c * fma(x0, b1, b0), b2 = c * fma(x0, a1, a0);
            p *= d;
            f = fma(a2, p, f);
            g = fma(b2, p, g);
            a0 = a1;
            b0 = b1;
            a1 = a2;
            b1 = b2;
        }
    } else {
        const double h = 1.0 / (M_PI * x * x), t = h * h;
        // f: 1 - 1.3 t + 1.3.5.7 t^2 - ..., g: 1 - 3.5 t + 3.5.7.9 t^2 - ...
        f = 1.0;
        g = 1.0;
#pragma unroll
        for (int m = 11; m >= 1; m--) {
            f = fma(-(double) ((4 * m - 3) * (4 * m - 1)) * t, f, 1.0);
            g = fma(-(double) ((4 * m - 1) * (4 * m + 1)) * t, g, 1.0);
        }
        f *= h * x;
        g *= t * x;
    }
}

// What the points of one z response share: gen_z_response at roffset, one
// point per bin, numkern (even) points.
struct ZResp {
    double start, z, zd, cons, pibyz, ec, es;
    double sgn;
    __device__ __forceinline__ void init(double roffset, double zz, int numkern)
    {
        z = zz;
        sgn = z < 0.0 ? -1.0 : 1.0;
        zd = sgn * M_SQRT2 / sqrt(fabs(z));
        cons = 0.5 * fabs(zd);
        pibyz = M_PI / z;
        start = roffset - 0.5 * z + 0.5 * numkern;
        // the second argument's phase over the first's: 2 pi r + pi z, r = start - c
        sincospi(2.0 * roffset, &es, &ec);
    }
    // |z| >= 1e-3; agrees with z_resp_point to the rounding of its phases
    __device__ __forceinline__ double2 point(int c, const double2 *tab) const
    {
        const double r = start - c, yy = r * zd, zz = yy + z * zd;
        double fy, gy, fz, gz;
        fresnel_fg(fabs(yy), tab, fy, gy);
        fresnel_fg(fabs(zz), tab, fz, gz);
        fy *= sgn;
        fz *= sgn;
        const double wr = gz * ec - fz * es, wi = gz * es + fz * ec;
        double vr = yy < 0.0 ? -gy : gy, vi = yy < 0.0 ? -fy : fy;
        if (zz < 0.0) {
            vr += wr;
            vi += wi;
        } else {
            vr -= wr;
            vi -= wi;
        }
        if (yy < 0.0 && zz >= 0.0) {
            double sx, cx;
            sincos(pibyz * r * r, &sx, &cx);
            vr += cx + sgn * sx;
            vi += sgn * cx - sx;
        }
        return make_double2(cons * vr, cons * vi);
    }
};

}  // namespace ab
