// H0^(2) and H1^(2) of a real positive argument in FP64, both from one evaluation.
//
// The 2-D Green's function needs J0, Y0, J1 and Y1 of the same argument at every quadrature
// point.  Four separate library calls repeat the argument reduction, the square root and the
// sine / cosine four times (and take their slowest paths at the small arguments of close
// pairs: 2.7 us a point on one thread); here they share everything.  With x = sqrt(u):
//   x >= 3: H_nu^(2)(x) = sqrt(2/(pi x)) (P_nu - j Q_nu) e^{-j(x - nu pi/2 - pi/4)} (DLMF
//     10.17.1), P_nu and x Q_nu smooth in 1/x^2: Chebyshev interpolants on x >= 80, [25, 80),
//     [8, 25), [4.5, 8) and [3, 4.5) (degrees 3, 5, 10, 12 and 12, interpolation error below
//     1e-16 of the modulus), computed at start-up from Hankel's integral
//       P - j Q = 1/Gamma(nu + 1/2) int_0^inf e^{-t} t^{nu - 1/2} (1 - j t/(2x))^{nu - 1/2} dt
//     (DLMF 10.9.30 rotated) by the trapezoidal rule in sqrt(t), long double;
//   x < 3: J0, J1/x and the regular parts of Y0, Y1 (DLMF 10.2.2, 10.8.1) as Chebyshev
//     interpolants of their power series in x^2, degree 12, plus one logarithm.
// x^{-1/2} comes from one FP32 estimate of u^{-1/4} and a third-order correction, so no
// division or square root is left; the phase is reduced by multiples of pi/4 in two parts
// (exact difference, then the tail), sine and cosine are Taylor polynomials on +-pi/4.
#pragma once
#include <cuda_runtime.h>

#include <complex>
#include <vector>

#define GH_XZ 80.0
#define GH_XA 25.0
#define GH_XB 8.0
#define GH_XC 4.5
#define GH_XD 3.0
#define GH_DEG_Z 3
#define GH_DEG_A 5
#define GH_DEG_B 10
#define GH_DEG_C 12  // both intervals below GH_XB
#define GH_DEG_E 12  // x < GH_XD

// Coefficients in the variable s in [-1, 1] of each interval: P0, x Q0, P1, x Q1, or
// J0, J1/x and the regular parts of Y0 and Y1/x.
struct HankelTab {
    double z[4][GH_DEG_Z + 1], a[4][GH_DEG_A + 1], b[4][GH_DEG_B + 1], c[4][GH_DEG_C + 1], d[4][GH_DEG_C + 1],
        e[4][GH_DEG_E + 1];
};
__constant__ HankelTab c_hankel;
static HankelTab h_hankel;  // computed here, uploaded to every device

// ------------------------------------------------------------------ host: the coefficients
static void hankel_pq(long double x, int nu, long double &P, long double &Q) {
    // trapezoidal rule in v = sqrt(t): 2 e^{-v^2} v^{2 nu} (1 - j v^2/(2x))^{nu - 1/2}; the
    // nearest branch point is sqrt(x) off the real axis, so the step 1/16 is exact at x >= 3
    const long double h = 1.0L / 16;
    std::complex<long double> sum = nu == 0 ? 0.5L : 0.0L;
    for (int i = 1; i < 160; ++i) {
        const long double v = i * h, v2 = v * v;
        const std::complex<long double> r = std::sqrt(std::complex<long double>(1.0L, -v2 / (2 * x)));
        sum += std::exp(-v2) * (nu == 0 ? 1.0L / r : v2 * r);
    }
    const long double spi = std::sqrt(std::acos(-1.0L));  // Gamma(1/2); Gamma(3/2) is half of it
    sum *= 2 * h / (nu == 0 ? spi : spi / 2);
    P = sum.real();
    Q = -sum.imag();
}

// Power series in q = x^2/4 of the four functions of the interval x < GH_XD.
static void hankel_low(long double u, long double f[4]) {
    const long double q = u / 4, pi = std::acos(-1.0L), gamma = 0.577215664901532860606512090082402431L;
    long double t0 = 1, t1 = 1, hk = 0, s[4] = {0, 0, 0, 0};
    for (int k = 0; k < 40; ++k) {
        if (k > 0) {
            t0 *= -q / ((long double)k * k);
            t1 *= -q / ((long double)k * (k + 1));
            hk += 1.0L / k;
        }
        s[0] += t0;
        s[1] += t1;
        s[2] += hk * t0;
        s[3] += (2 * hk + 1.0L / (k + 1) - 2 * gamma) * t1;
    }
    f[0] = s[0];
    f[1] = s[1] / 2;
    f[2] = 2 / pi * (gamma * s[0] - s[2]);
    f[3] = -s[3] / (2 * pi);
}

// Degree-d interpolants (Chebyshev nodes of s in [-1, 1]) of the four functions f(s), as
// power coefficients in s.
template <typename F>
static void hankel_fit(int deg, double *out, F f) {
    const int n = deg + 1;
    const long double pi = std::acos(-1.0L);
    std::vector<long double> val(4 * n);
    for (int i = 0; i < n; ++i) {
        long double v[4];
        f(std::cos(pi * (i + 0.5L) / n), v);
        for (int ch = 0; ch < 4; ++ch) val[ch * n + i] = v[ch];
    }
    for (int ch = 0; ch < 4; ++ch) {
        std::vector<long double> pow(n, 0.0L), t0(n, 0.0L), t1(n, 0.0L), t2(n, 0.0L);
        t0[0] = 1;
        t1[1] = 1;
        for (int j = 0; j < n; ++j) {
            long double c = 0;
            for (int i = 0; i < n; ++i) c += val[ch * n + i] * std::cos(pi * j * (i + 0.5L) / n);
            c *= (j == 0 ? 1.0L : 2.0L) / n;
            const std::vector<long double> &t = j == 0 ? t0 : t1;  // T_j (t1 holds it for j >= 1)
            for (int i = 0; i < n; ++i) pow[i] += c * t[i];
            if (j >= 1) {
                for (int i = 0; i < n; ++i) t2[i] = (i > 0 ? 2 * t1[i - 1] : 0.0L) - t0[i];
                t0 = t1;
                t1 = t2;
            }
        }
        for (int i = 0; i < n; ++i) out[ch * n + i] = (double)pow[i];
    }
}

static void hankel_tables() {
    auto range = [](long double y0, long double y1) {  // y = 1/x^2 in [y0, y1]
        return [=](long double s, long double v[4]) {
            const long double x = 1 / std::sqrt(0.5L * (y0 + y1) + 0.5L * (y1 - y0) * s);
            for (int nu = 0; nu < 2; ++nu) {
                hankel_pq(x, nu, v[2 * nu], v[2 * nu + 1]);
                v[2 * nu + 1] *= x;
            }
        };
    };
    const long double yz = 1 / ((long double)GH_XZ * GH_XZ), ya = 1 / ((long double)GH_XA * GH_XA), yb = 1 / ((long double)GH_XB * GH_XB),
                      yc = 1 / ((long double)GH_XC * GH_XC), yd = 1 / ((long double)GH_XD * GH_XD);
    hankel_fit(GH_DEG_Z, &h_hankel.z[0][0], range(0.0L, yz));
    hankel_fit(GH_DEG_A, &h_hankel.a[0][0], range(yz, ya));
    hankel_fit(GH_DEG_B, &h_hankel.b[0][0], range(ya, yb));
    hankel_fit(GH_DEG_C, &h_hankel.c[0][0], range(yb, yc));
    hankel_fit(GH_DEG_C, &h_hankel.d[0][0], range(yc, yd));
    hankel_fit(GH_DEG_E, &h_hankel.e[0][0], [](long double s, long double v[4]) {
        hankel_low(0.5L * GH_XD * GH_XD * (s + 1), v);
    });
}

// ------------------------------------------------------------------ device
__device__ __forceinline__ double gh_fourth_root_estimate(double u) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"((float)u));
    asm("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(y));
    return (double)y;
}

// The four polynomials of one interval at s, degree DEG.
template <int DEG>
__device__ __forceinline__ void gh_poly(const double (&t)[4][DEG + 1], double s, double (&v)[4]) {
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) v[ch] = t[ch][DEG];
#pragma unroll
    for (int i = DEG - 1; i >= 0; --i)
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) v[ch] = fma(v[ch], s, t[ch][i]);
}

// Sine and cosine on [-pi/4, pi/4] (Taylor, truncation below 7e-17), turned by n pi/2.
__device__ __forceinline__ void gh_sincos_quadrant(double r, int n, double &sn, double &cs) {
    const double z = r * r;
    double ps = -1.0 / 1307674368000.0, pc = 1.0 / 20922789888000.0;
    ps = fma(ps, z, 1.0 / 6227020800.0);
    pc = fma(pc, z, -1.0 / 87178291200.0);
    ps = fma(ps, z, -1.0 / 39916800.0);
    pc = fma(pc, z, 1.0 / 479001600.0);
    ps = fma(ps, z, 1.0 / 362880.0);
    pc = fma(pc, z, -1.0 / 3628800.0);
    ps = fma(ps, z, -1.0 / 5040.0);
    pc = fma(pc, z, 1.0 / 40320.0);
    ps = fma(ps, z, 1.0 / 120.0);
    pc = fma(pc, z, -1.0 / 720.0);
    ps = fma(ps, z, -1.0 / 6.0);
    pc = fma(pc, z, 1.0 / 24.0);
    pc = fma(pc, z, -0.5);
    const double s0 = fma(ps, r * z, r), c0 = fma(pc, z, 1.0);
    const double a = (n & 1) ? c0 : s0, b = (n & 1) ? s0 : c0;
    sn = (n & 2) ? -a : a;
    cs = ((n + 1) & 2) ? -b : b;
}

// High words of the interval bounds (u is compared by them: no FP64 comparison per point; a
// bound's low word is 0, so the comparisons are exact).
#define GH_HI_MIN 0x39b00000  // 2^-100
#define GH_HI_MAX 0x45c00000  // 2^93
#define GH_HI_Z 0x40b90000    // 80^2
#define GH_HI_A 0x40838800    // 25^2
#define GH_HI_B 0x40500000    // 8^2
#define GH_HI_C 0x40344000    // 4.5^2
#define GH_HI_D 0x40220000    // 3^2

// s = u^{-1/4}, inv = 1/x, x = sqrt(u).
__device__ __forceinline__ void gh_roots(double u, double &s, double &inv, double &x) {
    // e = 1 - u s^4 of the estimate (below 1e-6), then (1 - e)^{-1/4} to e^2
    s = gh_fourth_root_estimate(u);
    const double s2 = s * s;
    const double e = fma(-u * s2, s2, 1.0);
    s = fma(s * e, fma(e, 5.0 / 32.0, 0.25), s);
    inv = s * s;
    x = u * inv;
    x = fma(0.5 * inv, fma(-x, x, u), x);
}

// Phase x - pi/4 = n pi/2 + r: n rounded by the 1.5 2^52 shift, r = x - (2n + 1) pi/4.
__device__ __forceinline__ void gh_phase(double x, double &sn, double &cs) {
    const double shift = 6755399441055744.0;
    const double t = fma(x, 0.63661977236758134308, -0.5) + shift;
    const double m = fma(2.0, t - shift, 1.0);
    double r = fma(-m, 0.78539816339744830962, x);
    r = fma(-m, 3.0616169978683829431e-17, r);
    gh_sincos_quadrant(r, __double2loint(t), sn, cs);
}

// The Hankel pair from modulus polynomials v, s = x^{-1/2}, inv = 1/x and the phase.
__device__ __forceinline__ void gh_combine(const double (&v)[4], double s, double inv, double sn, double cs,
                                                    double2 &g, double2 &h) {
    // g = (j/4) sqrt(2/(pi x)) (cos - j sin)(P0 - j Q0); H1 carries another factor j
    const double A = 0.19947114020071633897 * s;  // sqrt(2/pi)/4
    const double As = A * sn, Ac = A * cs, q0 = v[1] * inv, q1 = v[3] * inv;
    g = make_double2(fma(As, v[0], Ac * q0), fma(Ac, v[0], -As * q0));
    const double Bs = As * inv, Bc = Ac * inv;
    h = make_double2(fma(Bs, q1, -Bc * v[2]), fma(Bs, v[2], Bc * q1));
}

// Sine and cosine of x, |x| < 2^30: x = n pi/2 + r in two parts, then the polynomials.
__device__ __forceinline__ void gh_sincos(double x, double &sn, double &cs) {
    const double shift = 6755399441055744.0;
    const double t = fma(x, 0.63661977236758134308, shift), m = t - shift;
    double r = fma(-m, 1.57079632679489661923, x);
    r = fma(-m, 6.1232339957367658862e-17, r);
    gh_sincos_quadrant(r, __double2loint(t), sn, cs);
}

__device__ __noinline__ static void hankel_pair_library(double u, double2 &g, double2 &h) {
    const double x = sqrt(u);
    g = make_double2(0.25 * y0(x), 0.25 * j0(x));
    h = make_double2(0.25 * y1(x) / x, 0.25 * j1(x) / x);
}

// g = (j/4) H0^(2)(x), h = (j/4) H1^(2)(x) / x, x = sqrt(u).  Outside 2^-100 <= u < 2^93 (the
// FP32 range of the root estimate, exact phase multiples) the library functions.
__device__ __forceinline__ void hankel_pair(double u, double2 &g, double2 &h) {
    const int hi = __double2hiint(u);
    if (hi < GH_HI_MIN || hi >= GH_HI_MAX) {
        hankel_pair_library(u, g, h);
        return;
    }
    double s, inv, x, v[4];
    gh_roots(u, s, inv, x);
    if (hi >= GH_HI_D) {
        const double y = inv * inv;
        constexpr double yz = 1.0 / (GH_XZ * GH_XZ), ya = 1.0 / (GH_XA * GH_XA), yb = 1.0 / (GH_XB * GH_XB),
                         yc = 1.0 / (GH_XC * GH_XC), yd = 1.0 / (GH_XD * GH_XD);
        if (hi >= GH_HI_Z) gh_poly<GH_DEG_Z>(c_hankel.z, fma(y, 2.0 / yz, -1.0), v);
        else if (hi >= GH_HI_A) gh_poly<GH_DEG_A>(c_hankel.a, fma(y, 2.0 / (ya - yz), -(ya + yz) / (ya - yz)), v);
        else if (hi >= GH_HI_B) gh_poly<GH_DEG_B>(c_hankel.b, fma(y, 2.0 / (yb - ya), -(yb + ya) / (yb - ya)), v);
        else if (hi >= GH_HI_C) gh_poly<GH_DEG_C>(c_hankel.c, fma(y, 2.0 / (yc - yb), -(yc + yb) / (yc - yb)), v);
        else gh_poly<GH_DEG_C>(c_hankel.d, fma(y, 2.0 / (yd - yc), -(yd + yc) / (yd - yc)), v);
        double sn, cs;
        gh_phase(x, sn, cs);
        gh_combine(v, s, inv, sn, cs, g, h);
    } else {
        gh_poly<GH_DEG_E>(c_hankel.e, fma(u, 2.0 / (GH_XD * GH_XD), -1.0), v);
        const double l = 0.31830988618379067154 * log(0.25 * u);  // (2/pi) ln(x/2)
        g = make_double2(0.25 * fma(l, v[0], v[2]), 0.25 * v[0]);
        h = make_double2(0.25 * (fma(l, v[1], v[3]) - 0.63661977236758134308 * (inv * inv)), 0.25 * v[1]);
    }
}

// Two arguments at once: where both lie at x >= 25 (most points of a large body) the two
// evaluations run interleaved and share every coefficient load; else one after the other.
__device__ __forceinline__ void hankel_pair2(const double (&u)[2], double2 (&g)[2], double2 (&h)[2]) {
    const int hi0 = __double2hiint(u[0]), hi1 = __double2hiint(u[1]);
    const int lo = min(hi0, hi1), top = max(hi0, hi1);
    if (lo >= GH_HI_A && top < GH_HI_MAX) {
        double s[2], inv[2], x[2], v[2][4], sn[2], cs[2];
        constexpr double yz = 1.0 / (GH_XZ * GH_XZ), ya = 1.0 / (GH_XA * GH_XA);
#pragma unroll
        for (int i = 0; i < 2; ++i) gh_roots(u[i], s[i], inv[i], x[i]);
        const bool far = lo >= GH_HI_Z;
        if (far || top < GH_HI_Z) {
            const double m = far ? 2.0 / yz : 2.0 / (ya - yz), c = far ? -1.0 : -(ya + yz) / (ya - yz);
            double w[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) w[i] = fma(inv[i] * inv[i], m, c);
            if (far) {
#pragma unroll
                for (int i = 0; i < 2; ++i) gh_poly<GH_DEG_Z>(c_hankel.z, w[i], v[i]);
            } else {
#pragma unroll
                for (int i = 0; i < 2; ++i) gh_poly<GH_DEG_A>(c_hankel.a, w[i], v[i]);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const double y = inv[i] * inv[i];
                if ((i == 0 ? hi0 : hi1) >= GH_HI_Z) gh_poly<GH_DEG_Z>(c_hankel.z, fma(y, 2.0 / yz, -1.0), v[i]);
                else gh_poly<GH_DEG_A>(c_hankel.a, fma(y, 2.0 / (ya - yz), -(ya + yz) / (ya - yz)), v[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) gh_phase(x[i], sn[i], cs[i]);
#pragma unroll
        for (int i = 0; i < 2; ++i) gh_combine(v[i], s[i], inv[i], sn[i], cs[i], g[i], h[i]);
    } else {
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
            double2 gi, hi;
            hankel_pair(i == 0 ? u[0] : u[1], gi, hi);
            if (i == 0) {
                g[0] = gi;
                h[0] = hi;
            } else {
                g[1] = gi;
                h[1] = hi;
            }
        }
    }
}
