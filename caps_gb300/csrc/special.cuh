// special.cuh -- modified Bessel functions of half-integer order and the Mie
// coefficients a_l, b_l (log-magnitudes), FP64 device code.
//
// Algorithms (the same as CaPS v0.5):
//  * K_{n+1/2}(x): upward recurrence K_{l+1/2} = (2l-1)/x K_{l-1/2} + K_{l-3/2}
//    from K_{1/2}, K_{3/2}, rescaled by 2^-600 on growth (bessel.c:781-821);
//    for n >= 100 the uniform asymptotic expansion DLMF 10.41.4 (bessel.c:706).
//  * I_{n+1/2}(x): Wronskian I_nu K_{nu+1} + I_{nu+1} K_nu = 1/x with the ratio
//    I_nu/I_{nu+1} from the continued fraction DLMF 10.33.1 (bessel.c:635,831), one per (l, x);
//    for n >= 100 the uniform expansion DLMF 10.41.3 (bessel.c:673).
//  * Mie coefficients: perfect reflector (libcaps.c:485) and Drude-type metal
//    (libcaps.c:557), both as log|a_l|, log|b_l|.
#pragma once
#include "common.cuh"

namespace capsgpu {

// I_nu(x)/I_{nu+1}(x) by the continued fraction b_1 + 1/(b_2 + 1/(...)), b_k = 2(nu+k)/x (DLMF 10.33.1), its N-th
// convergent as y_0 / y_1 of the backward recurrence y_{k-1} = b_k y_k + y_{k+1}: all terms are positive, so
// nothing cancels, and a step takes about two operations (a Lentz step takes two divisions, the forward recurrence of
// numerator and denominator three operations and a test).  Convergents differ by 1/(B_k B_{k-1}) relative, B_k the
// denominators, which grow by e^{asinh((nu+k)/x)} or more per step: below 2^-60 after 21 / asinh(nu/x) steps, and
// after sqrt(42 x) whatever nu where steps are small against x (16 more cover those that are not).
// The b_k of four steps come from one exact nu + k, so that their rounding stays that of the largest of the four.
CAPS_DEV double ratioI(double nu, double x)
{
    const double t = 2.0 / x;
    if ((nu + 1) * t > 0x1p60) return (nu + 1) * t; // the rest is below 2^-120
    const float z = (float)(0.5 * nu * t); // nu / x
    const float n1 = 21.0f / asinhf(z) + 3.0f, n2 = sqrtf(42.0f * (float)x) + 17.0f;
    const int N4 = (int)fminf(n1, n2) / 4 + 1; // (fminf passes over a NaN)
    double c = nu + 4 * N4, y = 1.0, y1 = 0.0;
    for (int g = 0; g < N4; g++, c -= 4.0) {
        const double b0 = c * t, b1 = b0 - t, b2 = fma(-2.0, t, b0), b3 = fma(-3.0, t, b0);
        const double p = fma(b0, y, y1), q = fma(b1, p, y);
        y1 = fma(b2, q, p);
        y = fma(b3, y1, q);
    }
    return y / y1;
}

// Debye polynomials of DLMF 10.41.10 as polynomials in p^2 (p^k taken out),
// summed as log1p(sum_k U_k y^k)
CAPS_DEV double debye_sum(double p2, double y)
{
    const double U1 = (3 - 5 * p2) / 24;
    const double U2 = (81 + p2 * (-462 + 385 * p2)) / 1152;
    const double U3 = (30375 + p2 * (-369603 + p2 * (765765 - 425425 * p2))) / 414720;
    const double U4 = (4465125 + p2 * (-94121676 + p2 * (349922430 + p2 * (-446185740 + 185910725 * p2)))) / 39813120;
    const double U5 = (1519035525. + p2 * (-49286948607. + p2 * (284499769554. + p2 * (-614135872350. + p2 * (566098157625. - 188699385875. * p2))))) / 6688604160.;
    return log1p(y * (U1 + y * (U2 + y * (U3 + y * (U4 + y * U5)))));
}

CAPS_DEV double logI_asymp(double nu, double x)
{
    const double z = x / nu, a = sqrt(1 + z * z), p2 = 1 / (1 + z * z);
    const double s = debye_sum(p2, 1 / (nu * a));
    const double eta = a + log(z / (1 + a));
    return nu * eta - 0.5 * log(2 * PI * nu * a) + s;
}

CAPS_DEV double logK_asymp(double nu, double x)
{
    const double z = x / nu, a = sqrt(1 + z * z), p2 = 1 / (1 + z * z);
    const double s = debye_sum(p2, -1 / (nu * a));
    const double eta = a + log(z / (1 + a));
    return -nu * eta - 0.5 * log(a) + 0.5 * log(0.5 * PI / nu) + s;
}

// log I_{n+1/2}(x), log K_{n+1/2}(x); rho = I_{n+1/2}(x) / I_{n+3/2}(x)
CAPS_DEV void logIK_half(int n, double x, double rho, double *logI, double *logK)
{
    if (n >= 100) {
        *logK = logK_asymp(n + 0.5, x);
        *logI = logI_asymp(n + 0.5, x);
        return;
    }
    const double logx = log(x), invx = 1.0 / x;
    double k0 = 1, k1 = 1 + invx;
    int sc = 0;
    double odd = 3.0; // 2 l - 1
    for (int l = 2; l <= n + 1; l++, odd += 2.0) { // tests on exponents: an FP64 comparison costs what an addition does
        const double kn = fma(odd * invx, k1, k0);
        k0 = k1; k1 = kn;
        if (expo(k0) >= 600) { k0 = shift2(k0, -600); k1 = shift2(k1, -600); sc += 600; }
    }
    const double pre = -x + 0.5 * (log(PI / 2) - logx) + sc * LN2;
    const double lk = pre + log(k0), lkp = pre + log(k1);
    *logK = lk;
    *logI = -logx - lkp - log1p(exp(lk - lkp - log(rho)));
}

CAPS_DEV double logadd(double a, double b)
{
    if (isinf(a) && a < 0) return b;
    if (isinf(b) && b < 0) return a;
    return a > b ? a + log1p(exp(b - a)) : b + log1p(exp(a - b));
}

// log|a_l|, log|b_l| at chi = xi_/(1+L/R); epsm1 = +inf selects perfect reflectors.  Four lanes share one l
// (all 32 lanes of the warp call): lane j of the four takes the functions of order l + 1/2 (j even) or l - 1/2 at chi
// (j < 2) or, for a metal, at n chi; all four end with the same values.
CAPS_DEV void mie(double LbyR, double xi_, int l, double epsm1, double *lna, double *lnb)
{
    const int j = threadIdx.x & 3;
    const bool pr = isinf(epsm1); // uniform: one frequency per warp
    const double chi = xi_ / (1 + LbyR);
    const double ln_chi = log(xi_) - log1p(LbyR);
    const double ln_n = pr ? 0.0 : log1p(epsm1) / 2, nr = pr ? 1.0 : exp(ln_n);
    const double x = j < 2 ? chi : nr * chi;
    // I_{l+1/2} / I_{l+3/2} by the continued fraction, I_{l-1/2} / I_{l+1/2} from it
    const double rho = ratioI(l + 0.5, x), my_ratio = (2 * l + 1) / x + 1.0 / rho;
    double lI, lK;
    logIK_half(j & 1 ? l - 1 : l, x, j & 1 ? my_ratio : rho, &lI, &lK);
    auto of = [&](double v, int k) { return __shfl_sync(0xffffffffu, v, (threadIdx.x & 28) | k); };
    const double ratio = of(my_ratio, 0), lIp = of(lI, 0), lKp = of(lK, 0), lKm = of(lK, 1);
    if (pr) {
        *lnb = LOGPI - LN2 + lIp - lKp;
        const double num = LOGPI - LN2 + lIp + log(chi * ratio - l);
        const double den = logadd(log((double)l) + lKp, ln_chi + lKm);
        *lna = num - den;
        return;
    }
    const double ln_l = log((double)l);
    const double ratio_n = of(my_ratio, 2), lIp_n = of(lI, 2), lIm_n = of(lI, 3);
    const double ln_gB = lIp_n + lIp + ln_chi + log(nr * ratio_n - ratio);
    const double ln_gC = log(epsm1) + lIp_n + logadd(ln_chi + lKm, ln_l + lKp);
    const double ln_gD = ln_chi + logadd(lIp_n + lKm, ln_n + lKp + lIm_n);
    const double num = lIp_n + lIp + log(-l * epsm1 + nr * chi * (nr * ratio - ratio_n));
    *lnb = LOGPI - LN2 + ln_gB - ln_gD;
    *lna = LOGPI - LN2 + num - logadd(ln_gC, ln_gD);
}

} // namespace capsgpu
