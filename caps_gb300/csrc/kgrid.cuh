// kgrid.cuh -- quadrature nodes for the K integrals of one (xi, m) matrix.
//
// K_{nu,p}^{(m)}(alpha) = int_1^inf r_p(x) e^{-alpha x} P_nu^mu(x) (x^2-1)^{-s} dx,
// mu = 2 max(m,1), s = (m>0)  (integration.c:257-286).  All degrees nu = mu..nu_max share one set of
// nodes, so that the K kernel obtains all P_nu^mu(x_k) from one forward recurrence per node.
//
// With x = 1 + u^2 / (4 alpha) the exponential is a Gaussian, e^{-alpha} e^{-u^2/4}, and
// (x^2-1)^{-s} P_nu^mu(x) is a polynomial in u^2 with zeros on the imaginary axis only.  For every
// degree the logarithm of the integrand then has a curvature between 1/2 and 1 at its peak and
// grows by at most e^{v^2/2} at u + iv, so the trapezoidal rule in u of step h has the error
// e^{-2 pi^2 / h^2} (h = 0.6: 2e-24) for all degrees at once, at 1.7 nodes per unit of the peak's
// width; panels of Gauss-Legendre nodes take 5 to 8 for the same integrals, and their edges a serial
// walk.  At u = 0 the integrand ends as u^{2 m' + 1} (even powers times dx): the map
//   u = c log(1 + e^{w / c})
// makes it decay like e^{(k+1) w / c}, k = mu + 1 - 2s, on the left and is linear on the right; its
// poles lie at w = +- i pi c.  The Fresnel coefficients are singular at x = +- i sqrt(eps), at a
// distance d = sqrt(2 alpha (1 + sqrt(1 + eps))) from the real u axis, where the integrand may have grown by
// e^{d^2/2}: the error is about e^{-2 pi d / h + d^2 / 2}, 2e-15 at d = 4 (in 40 digits 3.5e-15 for nu = mu, K_TM, the largest
// seen, 4e-16 for K_TE), the end of the range d >= 4 that dominates, with c = 1.5; closer ones are resolved in log u,
// c = 8 h, since their angle is at least pi / 4.
//
// The range: on the left the lowest degree's integrand, at most p (log y + (1 - y^2) / 2) below its
// peak in log at u = sqrt(2 p) y, p = k + 1 (exact for x - 1 << 1, an upper bound otherwise); on
// the right 14.5 past the peak of the highest degree (e^{-52}; the curvature is at least 1/2).
// Closed forms, evaluated on the host: 30 ns per matrix.
#pragma once
#include <cmath>

namespace capsgpu {

constexpr double KG_H = 0.6;          // step in w
constexpr double KG_LEFT = 42.0;      // e-folds below the lowest peak where the nodes start
constexpr double KG_RIGHT = 14.5;

struct KGrid { double w0, c; int n; }; // nodes w0 + j KG_H, j = 0 .. n - 1

// y < 1 with p (log y + (1 - y^2) / 2) = -KG_LEFT, by bisection in log y; it depends on m alone
inline double kgrid_left(int mu, int s)
{
    const double p = mu + 2 - 2 * s, e = KG_LEFT / p;
    double lo = -(e + 0.5), hi = 0.0; // log y >= -(e + 1/2)
    for (int it = 0; it < 50; it++) {
        const double z = 0.5 * (lo + hi);
        if (z + 0.5 * (1.0 - std::exp(2.0 * z)) < -e) lo = z;
        else hi = z;
    }
    return std::sqrt(2.0 * p) * std::exp(lo);
}

inline KGrid kgrid(double alpha, int mu, int nu_max, double epsm1, double left)
{
    // peak of the highest degree: alpha sinh t <= sqrt(nu'^2 + mu'^2 / sinh^2 t) bounds q = sinh^2 t
    const double nu = nu_max + 2.0, m2 = (mu + 2.0) * (mu + 2.0), b = nu * nu;
    const double a2q = 0.5 * (b + std::sqrt(b * b + 4.0 * alpha * alpha * m2)), q = a2q / (alpha * alpha);
    // u^2 = 4 alpha (cosh t - 1)
    const double u1 = std::sqrt(q < 1e16 ? 4.0 * alpha * (q / (std::sqrt(1.0 + q) + 1.0)) : 4.0 * std::sqrt(a2q)) + KG_RIGHT;
    const bool wide = std::isinf(epsm1) || !(2.0 * alpha * (1.0 + std::sqrt(1.0 + epsm1)) < 16.0);
    const double c = wide ? 1.5 : 8.0 * KG_H;
    auto W = [&](double u) { return u > 30.0 * c ? u : c * std::log(std::expm1(u / c)); };
    const double w0 = W(left);
    return KGrid{w0, c, (int)((W(u1) - w0) / KG_H) + 2};
}

} // namespace capsgpu
