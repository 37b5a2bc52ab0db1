// specfun.cuh -- device special functions for the secondary-emission model
// and the counter-based random numbers.
//
// Reference: specFun.pyx (binom :34, betainc :37, gammainc :40, betaincinv
// :53-253, gammaincinv :268-341), randomGen.pyx (uniform/normal draws).
//  * P(a,x) and I_x(a,b) use the power series / continued fractions of
//    Abramowitz & Stegun 6.5.29, 6.5.31 and 26.5.8 (modified Lentz).
//  * betaincinv and gammaincinv follow the reference's own algorithms: Temme's
//    asymptotic inversion with Halley refinement, and the Numerical-Recipes
//    style Halley iteration with bisection fallback -- same branches, same
//    expansion coefficients, same iteration limits.
//  * Random numbers: Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11), keyed
//    by the run seed, counted by (particle, step, draw): every draw of every
//    absorbed particle is reproducible regardless of thread scheduling.
#pragma once

#include <math.h>
#include <stdint.h>

namespace oec {
namespace sf {

constexpr double kPi = 3.141592653589793;
constexpr double kMachEps = 2.220446049250313e-16;
constexpr double kTiny = 1e-300;
constexpr double kCfEps = 1e-16;

__device__ inline double lgam(double a) { return lgamma(a); }

// Regularised lower incomplete gamma P(a, x), a > 0, with lga = lgamma(a)
// given (an inverse evaluates it many times for one a).
__device__ inline double gammainc_lg(double a, double x, double lga) {
    if (!(x > 0.0)) return 0.0;
    if (isinf(x)) return 1.0;
    double lpref = -x + a * log(x) - lga;
    if (x < a + 1.0) {
        double term = 1.0 / a, sum = term, an = a;
        for (int n = 0; n < 100000; ++n) {
            an += 1.0;
            term *= x / an;
            sum += term;
            if (fabs(term) <= fabs(sum) * kCfEps) break;
        }
        double p = sum * exp(lpref);
        return p > 1.0 ? 1.0 : p;
    }
    // continued fraction f = 1/(b0 + a1/(b1 + a2/(b2 + ...))), b_i = x+1-a+2i,
    // a_i = -i(i-a), by the forward recurrence of its convergents (one fused
    // multiply-add per term on the dependency chain; a division only at the
    // convergence checks, every 4 terms, which also renormalise A and B)
    const double b0 = x + 1.0 - a;
    double A2 = 0.0, B2 = 1.0, A1 = 1.0, B1 = b0;  // convergents n-2, n-1
    double f = A1 / B1;
    for (int i = 1; i < 100000; ++i) {
        const double an = -i * (i - a), bn = b0 + 2.0 * i;
        const double A = bn * A1 + an * A2, B = bn * B1 + an * B2;
        A2 = A1;
        B2 = B1;
        A1 = A;
        B1 = B;
        if ((i & 3) == 0) {
            const double r = 1.0 / B1, fn = A1 * r;
            A1 *= r;
            A2 *= r;
            B2 *= r;
            B1 = 1.0;
            const bool done = fabs(fn - f) <= 4.0 * kCfEps * fabs(fn);
            f = fn;
            if (done) break;
        }
    }
    double p = 1.0 - exp(lpref) * f;
    return p < 0.0 ? 0.0 : p;
}

// Regularised lower incomplete gamma P(a, x), a > 0.
__device__ inline double gammainc(double a, double x) { return gammainc_lg(a, x, lgam(a)); }

// Continued fraction of I_x(a, b): 1/(1 + d1/(1 + d2/(1 + ...))) with
// d1 = -(a+b)x/(a+1), d_{2m} = m(b-m)x/((a+2m-1)(a+2m)),
// d_{2m+1} = -(a+m)(a+b+m)x/((a+2m)(a+2m+1)), by the forward recurrence of
// its convergents (one fused multiply-add per term on the dependency chain;
// a division only at the convergence checks, which also renormalise).
__device__ inline double beta_cf(double a, double b, double x) {
    const double qab = a + b, qap = a + 1.0, qam = a - 1.0;
    double A2 = 1.0, B2 = 1.0, A1 = 1.0, B1 = 1.0 - qab * x / qap;  // convergents 1 and 2
    double h = A1 / B1;
    for (int m = 1; m < 100000; ++m) {
        const int m2 = 2 * m;
        const double de = m * (b - m) * x / ((qam + m2) * (a + m2));
        const double dodd = -(a + m) * (qab + m) * x / ((a + m2) * (qap + m2));
        double A = A1 + de * A2, B = B1 + de * B2;
        A2 = A1;
        B2 = B1;
        A1 = A;
        B1 = B;
        A = A1 + dodd * A2;
        B = B1 + dodd * B2;
        A2 = A1;
        B2 = B1;
        A1 = A;
        B1 = B;
        if ((m & 1) == 0) {
            const double r = 1.0 / B1, hn = A1 * r;
            A1 *= r;
            A2 *= r;
            B2 *= r;
            B1 = 1.0;
            const bool done = fabs(hn - h) <= 4.0 * kCfEps * fabs(hn);
            h = hn;
            if (done) break;
        }
    }
    return h;
}

// Regularised incomplete beta I_x(a, b) with lb = lgamma(a+b) - lgamma(a) -
// lgamma(b) given (the same value, computed once per inverse).
__device__ inline double betainc_lb(double a, double b, double x, double lb) {
    if (x <= 0.0) return 0.0;
    if (x >= 1.0) return 1.0;
    double bt = exp(lb + a * log(x) + b * log1p(-x));
    if (x < (a + 1.0) / (a + b + 2.0)) return bt * beta_cf(a, b, x) / a;
    return 1.0 - bt * beta_cf(b, a, 1.0 - x) / b;
}

__device__ inline double lbeta_inv(double a, double b) { return lgam(a + b) - lgam(a) - lgam(b); }

// Regularised incomplete beta I_x(a, b).
__device__ inline double betainc(double a, double b, double x) { return betainc_lb(a, b, x, lbeta_inv(a, b)); }

__device__ inline double beta(double a, double b) { return exp(lgam(a) + lgam(b) - lgam(a + b)); }

__device__ inline double binom_pdf(unsigned k, double p, unsigned n) {
    if (k > n) return 0.0;
    if (p == 0.0) return k == 0 ? 1.0 : 0.0;
    if (p == 1.0) return k == n ? 1.0 : 0.0;
    double lc = lgam((double)n + 1.0) - lgam((double)k + 1.0) - lgam((double)(n - k) + 1.0);
    return exp(lc + k * log(p) + (double)(n - k) * log1p(-p));
}

// x with 1 - Phi(x) = q.
__device__ inline double gauss_qinv(double q) { return -normcdfinv(q); }

// Student-t quantile by bisection on its CDF through I_x(nu/2, 1/2).
__device__ inline double tdist_pinv(double p, double nu) {
    if (p <= 0.0) return -INFINITY;
    if (p >= 1.0) return INFINITY;
    if (p == 0.5) return 0.0;
    double sign = 1.0;
    if (p < 0.5) {
        p = 1.0 - p;
        sign = -1.0;
    }
    double lo = 0.0, hi = 1.0;
    for (int i = 0; i < 2000 && 1.0 - 0.5 * betainc(0.5 * nu, 0.5, nu / (nu + hi * hi)) < p; ++i) hi *= 2.0;
    for (int i = 0; i < 200; ++i) {
        double mid = 0.5 * (lo + hi);
        if (1.0 - 0.5 * betainc(0.5 * nu, 0.5, nu / (nu + mid * mid)) < p)
            lo = mid;
        else
            hi = mid;
        if (hi - lo <= 1e-15 * hi) break;
    }
    return sign * 0.5 * (lo + hi);
}

// Inverse of P(a, .): specFun.pyx:268-341 (Halley steps, bisection fallback).
__device__ inline double gammaincinv(double a, double p, double acc = 1.e-9) {
    const double a1 = a - 1.0;
    double eps = sqrt(acc);
    if (!(a > 0.0)) return NAN;
    if (p >= 1.0) return fmax(100.0, a + 100.0 * sqrt(a));
    if (p <= 0.0) return 0.0;
    const double gln = lgam(a);
    double x, t, lna1 = 0.0, afac = 0.0;
    if (a > 1.0) {
        lna1 = log(a1);
        afac = exp(a1 * (lna1 - 1.0) - gln);
        double pp = p < 0.5 ? p : 1.0 - p;
        t = sqrt(-2.0 * log(pp));
        x = (2.30753 + t * 0.27061) / (1.0 + t * (0.99229 + t * 0.04481)) - t;
        if (p < 0.5) x = -x;
        x = fmax(1.e-3, a * pow(1.0 - 1.0 / (9.0 * a) - x / (3.0 * sqrt(a)), 3));
    } else {
        t = 1.0 - a * (0.253 + a * 0.12);
        if (p < t)
            x = pow(p / t, 1.0 / a);
        else
            x = 1.0 - log(1.0 - (p - t) / (1.0 - t));
    }
    int j;
    for (j = 0; j < 20; ++j) {
        if (x <= 0.0) return 0.0;
        double err = gammainc_lg(a, x, gln) - p;
        if (a > 1.0)
            t = afac * exp(-(x - a1) + a1 * (log(x) - lna1));
        else
            t = exp(-x + a1 * log(x) - gln);
        double u = err / t;
        t = u / (1.0 - 0.5 * fmin(1.0, u * ((a - 1.0) / x - 1.0)));
        x -= t;
        if (x <= 0.0) x = 0.5 * (x + t);
        if (fabs(t) < eps * x) {
            j = 0;
            break;
        }
    }
    if (j == 20) j = 19;  // the reference's loop variable ends at 19 when no break
    if (j == 19 && x < a) {
        eps = eps * eps;
        double err = gammainc_lg(a, x, gln) - p;
        double xr = x;
        for (int guard = 0; err <= 0 && guard < 2000; ++guard) {
            xr *= 2.0;
            err = gammainc_lg(a, xr, gln) - p;
        }
        double xl = 0.0;
        x = 0.5 * (xr + xl);
        for (int k = 0; k < 100; ++k) {
            err = gammainc_lg(a, x, gln) - p;
            if (err <= 0.0)
                xl = x;
            else
                xr = x;
            x = 0.5 * (xr + xl);
            if (0.5 * (xr - x) < eps * x) break;
            if (x < eps * a) {
                x = 0.0;
                break;
            }
        }
    }
    return x;
}

// Inverse of I_x(a, b): specFun.pyx:53-253.
__device__ inline double betaincinv(double a, double b, double p, double acc = 1.e-12) {
    double q = 1.0 - p;
    const double sqrt2 = sqrt(2.0);
    const double EPS = sqrt(acc);
    const unsigned n_halley = (unsigned)((-log(acc) / log(10.0)) + 1.0);
    double x = 0.0;
    bool swapped = false;
    if (q <= kMachEps) return 1.0;
    if (p <= kMachEps) return 0.0;
    if (a == 1 && b == 1) return p;
    if (a == 0.5 && b == 0.5) return sin(p * 0.5 * kPi);
    if (a == 0.5 && b >= 0.5) {
        x = tdist_pinv(0.5 * q, 2. * b);
        return 1 - 2. * b / (2. * b + x * x);
    }
    if (a >= 0.5 && b == 0.5) {
        x = tdist_pinv(0.5 * p, 2. * a);
        return 2. * a / (2. * a + x * x);
    }
    if (a > b) {
        double t = a; a = b; b = t;
        t = p; p = q; q = t;
        swapped = true;
    }
    if (a + b >= 5) {
        if ((b - a) <= sqrt(a)) {
            // Temme, section 2: a and b close.
            double eta0 = -1. / sqrt(a) * gauss_qinv(p);
            double be = b - a;
            double e2 = eta0 * eta0, e3 = e2 * eta0, e4 = e3 * eta0, e5 = e4 * eta0, e6 = e5 * eta0;
            double eps1 = (-0.5 * be * sqrt2 + 0.125 * (1. - 2. * be) * eta0 - 1. / 48. * be * sqrt2 * e2 -
                           1. / 192. * e3 - 1. / 3840. * be * sqrt2 * e4);
            double eps2 = (1. / 12. * be * sqrt2 * (3. * be - 2.) + 1. / 128. * (20. * be * be - 12 * be + 1.) * eta0 +
                           1. / 960. * be * sqrt2 * (20. * be - 1.) * e2 +
                           1. / 4608. * (16. * be * be + 30. * be - 15.) * e3 +
                           1. / 53760. * be * sqrt2 * (21. * be + 32.) * e4 + 1. / 368640. * (-32. * be * be + 63.) * e5 +
                           1. / 25804480 * be * sqrt2 * (120. * be + 17.) * e6);
            double eps3 = (1. / 480. * be * sqrt2 * (-75. * be * be + 80. * be - 16.) +
                           1. / 9216. * (-1080. * be * be * be + 868. * be * be - 90. * be * be - 45.) * eta0 +
                           1. / 53760 * be * sqrt2 * (-1190. * be * be + 84. * be + 373.) * e2 +
                           1. / 368640. * (-2240. * be * be * be - 2508. * be * be + 2100. * be - 165.) * e3);
            double eta = eta0 + (eps1 / a + eps2 / (a * a) + eps3 / (a * a * a));
            double r = sqrt(0.25 - 0.25 * exp(-0.5 * eta * eta));
            x = eta > 0 ? 0.5 + r : 0.5 - r;
        } else if (0.2 <= a / (a + b) && a / (a + b) <= 0.8) {
            if (pow(p, 1. / a) < 0.0025) {
                x = pow(a * p * beta(a, b), 1. / a);
            } else if (pow(q, 1. / b) < 0.0025) {
                x = 1 - pow(b * q * beta(a, b), 1. / b);
            } else {
                // Temme, section 3: a/(a+b) in [0.2, 0.8].
                double r = a + b, s2 = a / r, c2 = b / r, s = sqrt(s2), c = sqrt(c2);
                double eta0 = -1. / sqrt(r) * gauss_qinv(p);
                double e2 = eta0 * eta0, e3 = e2 * eta0, e4 = e3 * eta0;
                double s4 = s2 * s2, s6 = s4 * s2, s8 = s6 * s2, s10 = s8 * s2, s12 = s10 * s2, s14 = s12 * s2;
                double c4 = c2 * c2, c6 = c4 * c2;
                double eps1 = ((2. * s2 - 1) / (2 * s * c) - (5. * s4 - 5. * s2 - 1) / (36. * s2 * c2) * eta0 +
                               (46. * s6 - 69. * s4 + 21. * s2 + 1) / (1620. * s2 * s * c2 * c) * e2 -
                               (-2. * s2 - 62. * s6 + 31. * s8 + 33. * s4 + 7.) / (6480. * s4 * pow(c, 4)) * e3 +
                               (88. * s6 - 52. * s2 - 115. * s8 + 46. * s10 - 17. * s4 + 25.) /
                                   (90720. * s4 * s * c4 * c) * e4);
                double eps2 = (-(52. * s6 - 78. * s4 + 12. * s2 + 7.) / (405. * s2 * s * c2 * c) +
                               (2. * s2 - 370. * s6 + 185. * s8 + 183. * s4 - 7.) / (2592. * s4 * pow(c, 4)) * eta0 -
                               (776. * s2 + 10240. * s6 - 13525. * s8 - 533. + 5410. * s10 - 1835. * s4) /
                                   (204120. * s4 * s * c4 * c) * e2 +
                               (3747. * s2 + 15071. * s12 - 15821. * s6 + 45588. * s8 - 45213. * s10 - 3372. * s4 -
                                1579.) /
                                   (2099520. * s6 * c6) * e3);
                double eps3 = ((3704. * s10 - 9620. * s8 + 6686. * s6 - 769. * s4 - 1259. * s2 + 449.) /
                                   (102060. * s4 * s * c4 * c) -
                               (750479. * s12 - 151557. * s2 - 727469. * s6 + 2239932. * s8 - 2251437. * s10 +
                                140052. * s4 + 63149.) /
                                   (20995200. * s6 * c6) * eta0 +
                               (729754. * s14 - 78755. * s2 - 2554139. * s12 + 146879. * s6 - 1602610. * s8 +
                                3195183. * s10 + 105222. * s4 + 29233.) /
                                   (36741600. * s6 * s * c6 * c) * e2);
                double eta = eta0 + (eps1 / r + eps2 / (r * r) + eps3 / (r * r * r));
                if (eta * eta < 0.49) {
                    x = (s2 + s * c * eta + (1. - 2. * s2) / 3. * eta * eta +
                         (13. * s4 - 13. * s2 + 1.) / (36. * s * c) * eta * eta * eta +
                         (46. * s6 - 69. * s4 + 21. * s2 + 1.) / (270. * s2 * c2) * eta * eta * eta * eta);
                } else {
                    double al, u;
                    if (eta < 0) {
                        al = c2 / s2;
                        u = exp(1. / s2 * (-0.5 * eta * eta + s2 * log(s2) + c2 * log(c2)));
                    } else {
                        al = s2 / c2;
                        u = exp(1. / c2 * (-0.5 * eta * eta + s2 * log(s2) + c2 * log(c2)));
                    }
                    x = (u + al * u * u + 3. * al * (3. * al + 1.) / 6. * u * u * u +
                         4. * al * (4. * al + 1.) * (4. * al + 2.) / 24. * u * u * u * u +
                         5 * al * (5. * al + 1.) * (5. * al + 2.) * (5. * al + 3.) / 120. * u * u * u * u * u);
                    if (eta >= 0) x = 1 - x;
                }
            }
        } else {
            // Temme, section 4: a much smaller than b (a and b swapped so a <= b).
            double eta0 = 1. / b * gammaincinv(a, p);
            double mu = a / b;
            double w = sqrt(1. + mu);
            double w2 = w * w, w3 = w * w2, w4 = w3 * w, w5 = w4 * w, w6 = w5 * w, w7 = w6 * w, w8 = w7 * w,
                   w9 = w8 * w, w10 = w9 * w;
            double wa1 = w + 1, wa1p2 = wa1 * wa1, wa1p3 = wa1p2 * wa1, wa1p4 = wa1p3 * wa1;
            double d1 = eta0 - mu, d2 = d1 * d1, d3 = d2 * d1, d4 = d3 * d1;
            double eps1 = ((w + 2.) * (w - 1.) / (3. * w) + (w3 + 9. * w2 + 21. * w + 5.) / (36. * w2 * wa1) * d1 -
                           (w4 - 13. * w3 + 69. * w2 + 167. * w + 46.) / (1620. * wa1p2 * w3) * d2 -
                           (7. * w5 + 21. * w4 + 70. * w3 + 26. * w2 - 93. * w - 31.) / (6480. * wa1p3 * w4) * d3 -
                           (75. * w6 + 202. * w5 + 188. * w4 - 888. * w3 - 1345. * w2 + 118. * w + 138.) /
                               (272160. * wa1p4 * w5) * d4);
            double eps2 = ((28. * w4 + 131. * w3 + 402. * w2 + 581. * w + 208.) * (w - 1.) / (1620. * wa1 * w3) -
                           (35. * w6 - 154. * w5 - 623. * w4 - 1636. * w3 - 3983. * w2 - 3514. * w - 925.) /
                               (12960. * wa1p2 * w4) * d1 -
                           (2132. * w7 + 7915. * w6 + 16821. * w5 + 35066. * w4 + 87490. * w3 + 141183. * w2 +
                            95993. * w + 21640.) /
                               (816480. * w5 * wa1p3) * d2 -
                           (11053. * w8 + 53308. * w7 + 117010. * w6 + 163924. * w5 + 116188. * w4 - 258428. * w3 -
                            677042. * w2 - 481940. * w - 105497.) /
                               (14696640. * wa1p4 * w6) * d3);
            double eps3 = (-((3592. * w7 + 8375. * w6 - 1323. * w5 - 29198. * w4 - 89578. * w3 - 154413. * w2 -
                              116063. * w - 29632.) *
                             (w - 1.)) /
                               (816480. * w5 * wa1p2) -
                           (442043. * w9 + 2054169. * w8 + 3803094. * w7 + 3470754. * w6 + 2141568. * w5 -
                            2393568. * w4 - 19904934. * w3 - 34714674. * w2 - 23128299. * w - 5253353.) /
                               (146966400. * w6 * wa1p3) * d1 -
                           (116932. * w10 + 819281. * w9 + 2378172. * w8 + 4341330. * w7 + 6806004. * w6 +
                            10622748. * w5 + 18739500. * w4 + 30651894. * w3 + 30869976. * w2 + 15431867. * w +
                            2919016.) /
                               (146966400. * wa1p4 * w7) * d2);
            double eta = eta0 + (eps1 / b + eps2 / (b * b) + eps3 / (b * b * b));
            double u = exp(-eta + mu * log(eta) - (1 + mu) * log(1 + mu) + mu);
            if (eta == mu) {
                x = 1. / (1. + mu);
            } else {
                x = eta < mu ? 0.5 * (1. / (1. + mu) + 1.) : 0.5 / (1. + mu);
                for (unsigned j = 0; j < n_halley; ++j) {
                    if (x <= 0.0) return 0.0;
                    if (x >= 1.) return 1.0;
                    double err = x * pow(1 - x, mu) - u;
                    double y = 1. - x;
                    double der1 = pow(y, mu) - mu * x * pow(y, mu - 1);
                    double der2 = mu * (mu - 1.) * x * pow(y, mu - 2.);
                    double t = 2 * err * der1 / (2. * der1 * der1 - err * der2);
                    x -= t;
                    if (fabs(t) < 0.1 * x) break;
                }
            }
            x = 1 - x;
        }
    } else if (a < 1. && b < 1.) {
        if (p > betainc(a, b, (1. - a) / (2. - a - b))) {
            double t = pow(b * q * beta(b, a), 1. / b);
            x = 1 - t / (1 + t);
        } else {
            double t = pow(a * p * beta(a, b), 1. / a);
            x = t / (1 + t);
        }
    } else if (a > 1. && b > 1.) {
        if (p > betainc(b, a, (1. - b) / (2. - b - a))) {
            double t = pow(b * q * beta(b, a), 1. / b);
            x = 1. - t + (a - 1.) / (b + 1.) * t * t +
                (a - 1.) * (b * b + 3. * a * b - b + 5. * a - 4.) / (2. * pow(b + 1., 2) * (b + 2.)) * t * t * t;
        } else {
            double t = pow(a * p * beta(a, b), 1. / a);
            x = t + (b - 1.) / (a + 1.) * t * t +
                (b - 1.) * (a * a + 3. * b * a - a + 5. * b - 4.) / (2. * pow(a + 1., 2) * (a + 2.)) * t * t * t;
        }
    } else if (a <= 1. && b > 1.) {
        x = pow(1 - pow(q, a * beta(b, a)), 1. / a);
    }
    if (x <= 0)
        x = 0.;
    else if (x >= 1.)
        x = 1.;
    // Halley refinement on I_x(a,b) - p.
    const double bfi = 1. / beta(a, b);
    const double a1 = a - 1., a2 = a1 - 1., b1 = b - 1., b2 = b1 - 1.;
    const double lb = lbeta_inv(a, b);
    for (unsigned j = 0; j < n_halley; ++j) {
        // as in the reference, these early exits ignore the a<->b swap
        if (x <= 0.0) return 0.0;
        if (x >= 1.) return 1.0;
        double err = betainc_lb(a, b, x, lb) - p;
        double y = 1. - x;
        double xa1 = pow(x, a1), xa2 = pow(x, a2), yb1 = pow(y, b1), yb2 = pow(y, b2);
        double der1 = xa1 * yb1 * bfi;
        double der2 = bfi * (xa2 * yb1 - xa1 * yb2);
        double t = 2 * err * der1 / (2. * der1 * der1 - err * der2);
        x -= t;
        if (fabs(t) < EPS * x) break;
    }
    return swapped ? 1 - x : x;
}

// ------------------------------------- inverses with the constants laid out
// An emission inverts I_x(a, b) and P(a, .) for a few dozen fixed (a, b) only,
// so what depends on them alone (logs of gamma, the expansion coefficients of
// the starting guess, the terms of the continued fraction without x, the
// reciprocals of the series) is laid out once per launch and the inverse of one
// draw reads it.  Same branches, limits and iterations as betaincinv and
// gammaincinv above; the derivatives come from the incomplete function's own
// prefactor x^a (1-x)^b / B = x (1-x) I' (and x^a e^-x / Gamma = x P') instead
// of four powers, so an iteration costs two logarithms and one exponential.

constexpr int kBetaTerms = 12;    // tabulated steps of the continued fraction
constexpr int kGammaTerms = 40;   // tabulated reciprocals of the series

struct GammaConst {
    double a, lga, i9, i3;          // lgamma(a), 1/(9a), 1/(3 sqrt a)
    double rec[kGammaTerms];        // 1 / (a + 1 + n)
};

// The constants of a, by the threads of a block together (at least 32 +
// kGammaTerms of them).
__device__ inline void gamma_const(double a, GammaConst &C) {
    const int n = (int)threadIdx.x - 32;
    if (n >= 0 && n < kGammaTerms) C.rec[n] = 1.0 / (a + 1.0 + n);
    if (threadIdx.x != 0) return;
    C.a = a;
    C.lga = lgam(a);
    C.i9 = 1.0 / (9.0 * a);
    C.i3 = 1.0 / (3.0 * sqrt(a));
}

// P(a, x) for finite x > 0 and its prefactor x^a e^-x / Gamma(a); gammainc_lg
// with the series' divisions replaced by the tabulated reciprocals.
__device__ inline double gammainc_t(const GammaConst &C, double x, double *e) {
    const double a = C.a;
    *e = exp(-x + a * log(x) - C.lga);
    if (x < a + 1.0) {
        double term = 1.0 / a, sum = term;
        int n = 0;
        for (; n < kGammaTerms; ++n) {
            term *= x * C.rec[n];
            sum += term;
            if (fabs(term) <= fabs(sum) * kCfEps) break;
        }
        if (n == kGammaTerms)
            for (double an = a + kGammaTerms; n < 100000; ++n) {
                an += 1.0;
                term *= x / an;
                sum += term;
                if (fabs(term) <= fabs(sum) * kCfEps) break;
            }
        const double p = sum * *e;
        return p > 1.0 ? 1.0 : p;
    }
    const double b0 = x + 1.0 - a;
    double A2 = 0.0, B2 = 1.0, A1 = 1.0, B1 = b0;
    double f = A1 / B1;
    for (int i = 1; i < 100000; ++i) {
        const double an = -i * (i - a), bn = b0 + 2.0 * i;
        const double A = bn * A1 + an * A2, B = bn * B1 + an * B2;
        A2 = A1;
        B2 = B1;
        A1 = A;
        B1 = B;
        if ((i & 3) == 0) {
            const double r = 1.0 / B1, fn = A1 * r;
            A1 *= r;
            A2 *= r;
            B2 *= r;
            B1 = 1.0;
            const bool done = fabs(fn - f) <= 4.0 * kCfEps * fabs(fn);
            f = fn;
            if (done) break;
        }
    }
    const double p = 1.0 - *e * f;
    return p < 0.0 ? 0.0 : p;
}

__device__ inline double gammainc_of(const GammaConst &C, double x) {
    if (!(x > 0.0)) return 0.0;
    if (isinf(x)) return 1.0;
    double e;
    return gammainc_t(C, x, &e);
}

// gammaincinv for the normal course of the iteration; the cases that end in
// its bisection go to it.
__device__ inline double gammaincinv_t(const GammaConst &C, double p) {
    const double a = C.a, eps = sqrt(1.e-9);
    if (!(a > 0.0) || p >= 1.0 || p <= 0.0) return gammaincinv(a, p);
    double x, t;
    if (a > 1.0) {
        const double pp = p < 0.5 ? p : 1.0 - p;
        t = sqrt(-2.0 * log(pp));
        x = (2.30753 + t * 0.27061) / (1.0 + t * (0.99229 + t * 0.04481)) - t;
        if (p < 0.5) x = -x;
        const double r = 1.0 - C.i9 - x * C.i3;
        x = fmax(1.e-3, a * (r * r * r));
    } else {
        t = 1.0 - a * (0.253 + a * 0.12);
        if (p < t)
            x = pow(p / t, 1.0 / a);
        else
            x = 1.0 - log(1.0 - (p - t) / (1.0 - t));
    }
    for (int j = 0; j < 20; ++j) {
        if (x <= 0.0) return 0.0;
        if (isinf(x)) break;
        double e;
        const double err = gammainc_t(C, x, &e) - p;
        const double u = err * x / e;
        t = u / (1.0 - 0.5 * fmin(1.0, u * ((a - 1.0) / x - 1.0)));
        x -= t;
        if (x <= 0.0) x = 0.5 * (x + t);
        if (fabs(t) < eps * x) return x;
    }
    return gammaincinv(a, p);
}

enum BetaKind { kBetaGeneric = 0, kBetaOne, kBetaClose, kBetaMiddle, kBetaFar, kBetaSmall, kBetaLow };

struct BetaConst {
    double a0, b0;                  // as given
    double a, b, ia, ib;            // a <= b and their reciprocals
    double lb, xt;                  // log 1/B, the switch to 1 - I_1-x(b, a)
    double q1[2];                   // (a+b)/(a+1), (a+b)/(b+1)
    double2 cf[2][kBetaTerms];      // d_2m, d_2m+1 without x for (a, b), (b, a)
    double beta, scale, thr, pa, pb;
    double c[7], g[6];              // eta(eta0); x(eta) or the coefficients of small a, b
    int kind, swapped;
};

__device__ inline double2 beta_cf_term(double a, double b, int m) {
    const double qab = a + b, qap = a + 1.0, qam = a - 1.0;
    const int m2 = 2 * m;
    return make_double2(m * (b - m) / ((qam + m2) * (a + m2)), -(a + m) * (qab + m) / ((a + m2) * (qap + m2)));
}

// beta_cf with the tabulated terms (the rest formed on the spot).
__device__ inline double beta_cf_t(double a, double b, double x, const double2 *__restrict__ cf, double q1) {
    double A2 = 1.0, B2 = 1.0, A1 = 1.0, B1 = 1.0 - q1 * x;
    double h = A1 / B1;
    for (int m = 1; m < 100000; ++m) {
        double de, dodd;
        if (m <= kBetaTerms) {
            const double2 d = cf[m - 1];
            de = d.x * x;
            dodd = d.y * x;
        } else {
            const int m2 = 2 * m;
            const double qab = a + b, qap = a + 1.0, qam = a - 1.0;
            de = m * (b - m) * x / ((qam + m2) * (a + m2));
            dodd = -(a + m) * (qab + m) * x / ((a + m2) * (qap + m2));
        }
        double A = A1 + de * A2, B = B1 + de * B2;
        A2 = A1;
        B2 = B1;
        A1 = A;
        B1 = B;
        A = A1 + dodd * A2;
        B = B1 + dodd * B2;
        A2 = A1;
        B2 = B1;
        A1 = A;
        B1 = B;
        if ((m & 1) == 0) {
            const double r = 1.0 / B1, hn = A1 * r;
            A1 *= r;
            A2 *= r;
            B2 *= r;
            B1 = 1.0;
            const bool done = fabs(hn - h) <= 4.0 * kCfEps * fabs(hn);
            h = hn;
            if (done) break;
        }
    }
    return h;
}

// I_x(a, b) for 0 < x < 1 and its prefactor x^a (1-x)^b / B.
__device__ inline double betainc_t(const BetaConst &C, double x, double *bt) {
    *bt = exp(C.lb + C.a * log(x) + C.b * log1p(-x));
    if (x < C.xt) return *bt * beta_cf_t(C.a, C.b, x, C.cf[0], C.q1[0]) * C.ia;
    return 1.0 - *bt * beta_cf_t(C.b, C.a, 1.0 - x, C.cf[1], C.q1[1]) * C.ib;
}

// The constants of (a, b), by the first 96 threads of a block together.
__device__ inline void beta_const(double a, double b, BetaConst &C) {
    const int tid = threadIdx.x, m = tid & 31;
    if (tid >= 96) return;
    if (tid >= 32) {  // the continued fractions' terms, one thread each
        const double lo = a > b ? b : a, hi = a > b ? a : b;
        const bool first = tid < 64;
        if (m < kBetaTerms) C.cf[first ? 0 : 1][m] = first ? beta_cf_term(lo, hi, m + 1) : beta_cf_term(hi, lo, m + 1);
        if (m == kBetaTerms) C.q1[first ? 0 : 1] = (a + b) / ((first ? lo : hi) + 1.0);
        return;
    }
    if (m > 0) return;
    C.a0 = a;
    C.b0 = b;
    C.swapped = 0;
    C.kind = kBetaGeneric;
    if (a == 1 && b == 1) {
        C.kind = kBetaOne;
        return;
    }
    if (!(a > 0.0) || !(b > 0.0) || a == 0.5 || b == 0.5) return;
    if (a > b) {
        const double t = a;
        a = b;
        b = t;
        C.swapped = 1;
    }
    C.a = a;
    C.b = b;
    C.ia = 1.0 / a;
    C.ib = 1.0 / b;
    const double sqrt2 = sqrt(2.0);
    if (a + b >= 5 && b - a <= sqrt(a)) {
        C.kind = kBetaClose;
        const double be = b - a, a2 = a * a, a3 = a * a * a;
        C.scale = 1. / sqrt(a);
        C.c[0] = -0.5 * be * sqrt2 / a + 1. / 12. * be * sqrt2 * (3. * be - 2.) / a2 +
                 1. / 480. * be * sqrt2 * (-75. * be * be + 80. * be - 16.) / a3;
        C.c[1] = 0.125 * (1. - 2. * be) / a + 1. / 128. * (20. * be * be - 12 * be + 1.) / a2 +
                 1. / 9216. * (-1080. * be * be * be + 868. * be * be - 90. * be * be - 45.) / a3;
        C.c[2] = -1. / 48. * be * sqrt2 / a + 1. / 960. * be * sqrt2 * (20. * be - 1.) / a2 +
                 1. / 53760 * be * sqrt2 * (-1190. * be * be + 84. * be + 373.) / a3;
        C.c[3] = -1. / 192. / a + 1. / 4608. * (16. * be * be + 30. * be - 15.) / a2 +
                 1. / 368640. * (-2240. * be * be * be - 2508. * be * be + 2100. * be - 165.) / a3;
        C.c[4] = -1. / 3840. * be * sqrt2 / a + 1. / 53760. * be * sqrt2 * (21. * be + 32.) / a2;
        C.c[5] = 1. / 368640. * (-32. * be * be + 63.) / a2;
        C.c[6] = 1. / 25804480 * be * sqrt2 * (120. * be + 17.) / a2;
    } else if (a + b >= 5 && 0.2 <= a / (a + b) && a / (a + b) <= 0.8) {
        C.kind = kBetaMiddle;
        const double r = a + b, r2 = r * r, r3 = r2 * r, s2 = a / r, c2 = b / r, s = sqrt(s2), c = sqrt(c2);
        const double s4 = s2 * s2, s6 = s4 * s2, s8 = s6 * s2, s10 = s8 * s2, s12 = s10 * s2, s14 = s12 * s2;
        const double c4 = c2 * c2, c6 = c4 * c2;
        C.scale = 1. / sqrt(r);
        C.c[0] = (2. * s2 - 1) / (2 * s * c) / r -
                 (52. * s6 - 78. * s4 + 12. * s2 + 7.) / (405. * s2 * s * c2 * c) / r2 +
                 (3704. * s10 - 9620. * s8 + 6686. * s6 - 769. * s4 - 1259. * s2 + 449.) /
                     (102060. * s4 * s * c4 * c) / r3;
        C.c[1] = -(5. * s4 - 5. * s2 - 1) / (36. * s2 * c2) / r +
                 (2. * s2 - 370. * s6 + 185. * s8 + 183. * s4 - 7.) / (2592. * s4 * c4) / r2 -
                 (750479. * s12 - 151557. * s2 - 727469. * s6 + 2239932. * s8 - 2251437. * s10 + 140052. * s4 +
                  63149.) / (20995200. * s6 * c6) / r3;
        C.c[2] = (46. * s6 - 69. * s4 + 21. * s2 + 1) / (1620. * s2 * s * c2 * c) / r -
                 (776. * s2 + 10240. * s6 - 13525. * s8 - 533. + 5410. * s10 - 1835. * s4) /
                     (204120. * s4 * s * c4 * c) / r2 +
                 (729754. * s14 - 78755. * s2 - 2554139. * s12 + 146879. * s6 - 1602610. * s8 + 3195183. * s10 +
                  105222. * s4 + 29233.) / (36741600. * s6 * s * c6 * c) / r3;
        C.c[3] = -(-2. * s2 - 62. * s6 + 31. * s8 + 33. * s4 + 7.) / (6480. * s4 * c4) / r +
                 (3747. * s2 + 15071. * s12 - 15821. * s6 + 45588. * s8 - 45213. * s10 - 3372. * s4 - 1579.) /
                     (2099520. * s6 * c6) / r2;
        C.c[4] = (88. * s6 - 52. * s2 - 115. * s8 + 46. * s10 - 17. * s4 + 25.) / (90720. * s4 * s * c4 * c) / r;
        C.c[5] = C.c[6] = 0.0;
        C.g[0] = s2;
        C.g[1] = s * c;
        C.g[2] = (1. - 2. * s2) / 3.;
        C.g[3] = (13. * s4 - 13. * s2 + 1.) / (36. * s * c);
        C.g[4] = (46. * s6 - 69. * s4 + 21. * s2 + 1.) / (270. * s2 * c2);
        C.g[5] = s2 * log(s2) + c2 * log(c2);
        C.pa = pow(0.0025, a);
        C.pb = pow(0.0025, b);
    } else if (a + b >= 5) {
        // Temme, section 4: eta as a polynomial in eta0 - mu
        C.kind = kBetaFar;
        const double mu = a / b, w = sqrt(1. + mu), b2 = b * b, b3 = b2 * b;
        const double w2 = w * w, w3 = w * w2, w4 = w3 * w, w5 = w4 * w, w6 = w5 * w, w7 = w6 * w, w8 = w7 * w,
                     w9 = w8 * w, w10 = w9 * w;
        const double wa1 = w + 1, wa1p2 = wa1 * wa1, wa1p3 = wa1p2 * wa1, wa1p4 = wa1p3 * wa1;
        C.scale = 1. / b;
        C.c[0] = (w + 2.) * (w - 1.) / (3. * w) / b +
                 (28. * w4 + 131. * w3 + 402. * w2 + 581. * w + 208.) * (w - 1.) / (1620. * wa1 * w3) / b2 -
                 (3592. * w7 + 8375. * w6 - 1323. * w5 - 29198. * w4 - 89578. * w3 - 154413. * w2 - 116063. * w -
                  29632.) * (w - 1.) / (816480. * w5 * wa1p2) / b3;
        C.c[1] = (w3 + 9. * w2 + 21. * w + 5.) / (36. * w2 * wa1) / b -
                 (35. * w6 - 154. * w5 - 623. * w4 - 1636. * w3 - 3983. * w2 - 3514. * w - 925.) /
                     (12960. * wa1p2 * w4) / b2 -
                 (442043. * w9 + 2054169. * w8 + 3803094. * w7 + 3470754. * w6 + 2141568. * w5 - 2393568. * w4 -
                  19904934. * w3 - 34714674. * w2 - 23128299. * w - 5253353.) / (146966400. * w6 * wa1p3) / b3;
        C.c[2] = -(w4 - 13. * w3 + 69. * w2 + 167. * w + 46.) / (1620. * wa1p2 * w3) / b -
                 (2132. * w7 + 7915. * w6 + 16821. * w5 + 35066. * w4 + 87490. * w3 + 141183. * w2 + 95993. * w +
                  21640.) / (816480. * w5 * wa1p3) / b2 -
                 (116932. * w10 + 819281. * w9 + 2378172. * w8 + 4341330. * w7 + 6806004. * w6 + 10622748. * w5 +
                  18739500. * w4 + 30651894. * w3 + 30869976. * w2 + 15431867. * w + 2919016.) /
                     (146966400. * wa1p4 * w7) / b3;
        C.c[3] = -(7. * w5 + 21. * w4 + 70. * w3 + 26. * w2 - 93. * w - 31.) / (6480. * wa1p3 * w4) / b -
                 (11053. * w8 + 53308. * w7 + 117010. * w6 + 163924. * w5 + 116188. * w4 - 258428. * w3 -
                  677042. * w2 - 481940. * w - 105497.) / (14696640. * wa1p4 * w6) / b2;
        C.c[4] = -(75. * w6 + 202. * w5 + 188. * w4 - 888. * w3 - 1345. * w2 + 118. * w + 138.) /
                 (272160. * wa1p4 * w5) / b;
        C.g[0] = mu;
        C.g[1] = (1. + mu) * log(1. + mu) - mu;
        C.g[2] = 1. / (1. + mu);
    } else if (a > 1. && b > 1.) {
        C.kind = kBetaSmall;
        C.g[0] = (a - 1.) / (b + 1.);
        C.g[1] = (a - 1.) * (b * b + 3. * a * b - b + 5. * a - 4.) / (2. * (b + 1.) * (b + 1.) * (b + 2.));
        C.g[2] = (b - 1.) / (a + 1.);
        C.g[3] = (b - 1.) * (a * a + 3. * b * a - a + 5. * b - 4.) / (2. * (a + 1.) * (a + 1.) * (a + 2.));
        C.thr = betainc(b, a, (1. - b) / (2. - b - a));
    } else if (a <= 1. && b > 1.) {
        C.kind = kBetaLow;
    } else {
        return;
    }
    C.beta = beta(a, b);
    C.lb = lbeta_inv(a, b);
    C.xt = (a + 1.0) / (a + b + 2.0);
}

// G holds the constants of P(min(a, b), .).
__device__ inline double betaincinv_t(const BetaConst &C, const GammaConst &G, double p) {
    constexpr double EPS = 1.e-6;       // sqrt of the accuracy 1e-12
    constexpr unsigned n_halley = 13;   // -log10(1e-12) + 1
    double q = 1.0 - p;
    if (q <= kMachEps) return 1.0;
    if (p <= kMachEps) return 0.0;
    if (C.kind == kBetaOne) return p;
    if (C.kind == kBetaGeneric) return betaincinv(C.a0, C.b0, p);
    const double a = C.a, b = C.b;
    if (C.swapped) {
        const double t = p;
        p = q;
        q = t;
    }
    double x;
    if (C.kind == kBetaClose || (C.kind == kBetaMiddle && p >= C.pa && q >= C.pb)) {
        const double e0 = -C.scale * gauss_qinv(p);
        const double eta =
            e0 + (C.c[0] + e0 * (C.c[1] + e0 * (C.c[2] + e0 * (C.c[3] + e0 * (C.c[4] + e0 * (C.c[5] + e0 * C.c[6]))))));
        if (C.kind == kBetaClose) {
            const double r = sqrt(0.25 - 0.25 * exp(-0.5 * eta * eta));
            x = eta > 0 ? 0.5 + r : 0.5 - r;
        } else if (eta * eta < 0.49) {
            x = C.g[0] + eta * (C.g[1] + eta * (C.g[2] + eta * (C.g[3] + eta * C.g[4])));
        } else {
            const double s2 = C.g[0], c2 = 1.0 - s2;
            const double al = eta < 0 ? c2 / s2 : s2 / c2;
            const double u = exp((C.g[5] - 0.5 * eta * eta) / (eta < 0 ? s2 : c2));
            x = (u + al * u * u + 3. * al * (3. * al + 1.) / 6. * u * u * u +
                 4. * al * (4. * al + 1.) * (4. * al + 2.) / 24. * u * u * u * u +
                 5 * al * (5. * al + 1.) * (5. * al + 2.) * (5. * al + 3.) / 120. * u * u * u * u * u);
            if (eta >= 0) x = 1 - x;
        }
    } else if (C.kind == kBetaFar) {
        const double mu = C.g[0], e0 = C.scale * gammaincinv_t(G, p), d = e0 - mu;
        const double eta = e0 + (C.c[0] + d * (C.c[1] + d * (C.c[2] + d * (C.c[3] + d * C.c[4]))));
        const double u = exp(-eta + mu * log(eta) - C.g[1]);
        if (eta == mu) {
            x = C.g[2];
        } else {
            x = eta < mu ? 0.5 * (C.g[2] + 1.) : 0.5 * C.g[2];
            for (unsigned j = 0; j < n_halley; ++j) {
                if (x <= 0.0) return 0.0;
                if (x >= 1.) return 1.0;
                const double y = 1. - x, iy = 1. / y, ym = exp(mu * log(y));
                const double err = x * ym - u;
                const double der1 = ym - mu * x * ym * iy;
                const double der2 = mu * (mu - 1.) * x * ym * iy * iy;
                const double t = 2 * err * der1 / (2. * der1 * der1 - err * der2);
                x -= t;
                if (fabs(t) < 0.1 * x) break;
            }
        }
        x = 1 - x;
    } else if (C.kind == kBetaLow) {
        x = pow(1 - pow(q, a * C.beta), C.ia);
    } else {
        const bool middle = C.kind == kBetaMiddle;
        const bool upper = middle ? p >= C.pa : p > C.thr;
        const double t = upper ? pow(b * q * C.beta, C.ib) : pow(a * p * C.beta, C.ia);
        if (middle)
            x = upper ? 1 - t : t;
        else
            x = upper ? 1. - t + t * t * (C.g[0] + t * C.g[1]) : t + t * t * (C.g[2] + t * C.g[3]);
    }
    if (x <= 0)
        x = 0.;
    else if (x >= 1.)
        x = 1.;
    for (unsigned j = 0; j < n_halley; ++j) {
        // as in the reference, these early exits ignore the a<->b swap
        if (x <= 0.0) return 0.0;
        if (x >= 1.) return 1.0;
        // Halley's step 2 e I' / (2 I'^2 - e I'') with I' = bt / (x y) and the
        // reference's I'' = I' (1/x - 1/y)
        double bt;
        const double err = betainc_t(C, x, &bt) - p, y = 1. - x;
        const double t = 2 * err * (x * y) / (2. * bt - err * (y - x));
        x -= t;
        if (fabs(t) < EPS * x) break;
    }
    return C.swapped ? 1 - x : x;
}

// ------------------------------------------------------------- Philox

__device__ __forceinline__ uint4 philox4x32_10(uint4 ctr, uint2 key) {
    const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        uint32_t hi0 = __umulhi(M0, ctr.x), lo0 = M0 * ctr.x;
        uint32_t hi1 = __umulhi(M1, ctr.z), lo1 = M1 * ctr.z;
        ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
        key.x += W0;
        key.y += W1;
    }
    return ctr;
}

// Uniform [0,1) doubles for one absorbed particle: draw d of particle `id`
// at `step`; or, in replay mode, uniforms[row*stride + d].
struct Draws {
    uint2 key;
    uint32_t id, step;
    const double *replay;
    int d = 0;
    __device__ double next() {
        int k = d++;
        if (replay) return replay[k];
        uint4 r = philox4x32_10(make_uint4(id, step, (uint32_t)(k >> 1), 0x0ecu), key);
        uint32_t a = (k & 1) ? r.z : r.x, b = (k & 1) ? r.w : r.y;
        return ((double)(a >> 5) * 67108864.0 + (double)(b >> 6)) * (1.0 / 9007199254740992.0);
    }
    // Standard normal by Box-Muller from two draws.
    __device__ double normal() {
        double u1 = 1.0 - next(), u2 = next();
        return sqrt(-2.0 * log(u1)) * cos(2.0 * kPi * u2);
    }
};

}  // namespace sf
}  // namespace oec
