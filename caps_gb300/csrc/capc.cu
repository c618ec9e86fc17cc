// capc.cu -- the cylinder-plane geometry at T = 0 (the reference's capc.cpp:20-177).
//
// A cylinder of radius R at distance d from a plane, both perfect reflectors: scalar
// Dirichlet (D) and Neumann (N) modes decouple, and at wave number q along the axis the
// reference writes (capc.cpp:47-127, :155-177)
//   log det(1 - M(q)) = log(1 - M_00) + log det(1 - (U - V)) + log det(1 - (U + V + alpha v v^T))
// for mu1, mu2 = 1 .. lmax, with
//   U = r(mu1)^1/2 r(mu2)^1/2 K_{mu1+mu2}(2 calL q),  V = the same with K_{|mu1-mu2|},
//   v_mu = r(0)^1/2 r(mu)^1/2 K_mu(2 calL q),  M_00 = r(0) K_0(2 calL q),  alpha = 2/(1 - M_00),
// calL = R + d, r(n) = I_n(Rq)/K_n(Rq) (D) or I'_n(Rq)/|K'_n(Rq)| (N).  The energy per
// length is E/(hbar c) = 1/(8 pi d) int_0^inf dx q logdet(q), q = x/(2d), by QUADPACK qagi
// (capc.cpp:129-153).
//
// GPU form: per q one block builds three short tables as scaled doubles -- sqrt r(mu),
// K_k(2 calL q) for k <= 2 lmax, and sqrt(alpha r(0)) sqrt r(mu) K_mu(2 calL q) -- and one
// kernel writes 1 - M of both matrices of every q of a batch in fixed point, each element a product of
// table entries (no exp or log per element); the batched Cholesky with
// kernel_logdet's rules (matrix.c:57-149) gives the log dets.  A batch is every node of
// one qagi step.
//
// Integer-order Bessel functions, own method (the reference evaluates Cephes Chebyshev
// fits for orders 0 and 1, bessel.c:283-461, and per-order recurrences or Debye
// asymptotics above, bessel.c:506-633):
//   * K_0, K_1: trapezoidal rule on K_nu(x) = int_0^inf exp(-x cosh t) cosh(nu t) dt
//     (DLMF 10.32.9), geometrically convergent in the step;
//   * I_0: trapezoidal rule on I_0(x) = (1/pi) int_0^pi exp(x cos th) dth (DLMF 10.32.3),
//     exact up to aliasing terms I_{2N}(x), and Hankel's expansion (DLMF 10.40.1) for
//     large x;
//   * K_n, n >= 2: upward recurrence K_{n+1} = K_{n-1} + (2n/x) K_n (all terms positive);
//   * I_{n+1}/I_n: backward recurrence of the ratio started high enough above the largest
//     order that the starting error has decayed (Miller's algorithm); on the GPU that of I_n itself,
//     I_{n-1} = I_{n+1} + (2n/x) I_n, which takes no divisions, scaled to I_0.
// Values are kept as mantissa x 2^exponent, so nothing overflows and no logarithm is
// taken: table entries are accurate to a few ulps, where exp(sum of logs) loses |log| ulps.
#include <algorithm>
#include <cctype>
#include <cmath>
#include <mutex>
#include <type_traits>
#include <vector>

#include "../../include/libcaps.h"
#include "../../include/capc.h"
#include "../../include/bessel.h"
#include "fix.cuh"
#include "internal.h"

namespace capsgpu {

namespace {

constexpr double H_LN2 = 0.69314718055994530942;
constexpr double H_INV_LN2 = 1.4426950408889634074;
constexpr double H_LN2_TAIL = 2.3190468138462996e-17; // ln 2 - (double)(ln 2)
constexpr double H_PI = 3.14159265358979323846;

// (not inlined: k_capc_tab runs through its code once, and fetching it from the L2 cache is what it would wait for)
#define HX_FN __host__ __device__ __noinline__
struct hx { double m; long long e; }; // m 2^e with m in [0.5, 1), or m = 0

// m 2^k, on the GPU by integer work alone (an FP64 operation of a warp holds its scheduler's unit for 64 clocks)
__host__ __device__ double hscale(double m, int k)
{
#ifdef __CUDA_ARCH__
    return shift2(m, k);
#else
    return std::ldexp(m, k);
#endif
}
HX_FN hx hnorm(double m, long long e)
{
    if (m == 0.0 || !isfinite(m)) return hx{m, 0};
#ifdef __CUDA_ARCH__
    const int k = expo(m) + 1;
    return hx{shift2(m, -k), e + k};
#else
    int k;
    const double f = std::frexp(m, &k);
    return hx{f, e + k};
#endif
}
HX_FN hx hmul(hx a, hx b) { return hnorm(a.m * b.m, a.e + b.e); }
HX_FN hx hdiv(hx a, hx b) { return hnorm(a.m / b.m, a.e - b.e); }
HX_FN hx hadd(hx a, hx b) // a, b >= 0
{
    if (a.m == 0.0) return b;
    if (b.m == 0.0) return a;
    if (a.e < b.e) { const hx t = a; a = b; b = t; }
    const long long d = b.e - a.e;
    return hnorm(a.m + (d < -1100 ? 0.0 : hscale(b.m, (int)d)), a.e);
}
HX_FN hx hsqrt(hx a)
{
    if (a.e & 1) { a.m *= 2.0; a.e -= 1; }
    return hnorm(sqrt(a.m), a.e / 2);
}
double hlog(hx a) { return std::log(a.m) + (double)a.e * H_LN2; }
__host__ __device__ double hval(hx a)
{
    if (a.m == 0.0 || !isfinite(a.m)) return a.m;
    if (a.e > 1100) return INFINITY;
    if (a.e < -1100) return 0.0;
    return hscale(a.m, (int)a.e);
}
// e^y for any finite y: y = n ln2 + r, with n ln2 carried exactly (fma) so that r keeps
// full relative accuracy however large n is
HX_FN hx hexp(double y)
{
    const double n = floor(y * H_INV_LN2);
    const double p = n * H_LN2, perr = fma(n, H_LN2, -p);
    const double r = ((y - p) - perr) - n * H_LN2_TAIL;
    return hnorm(exp(r), (long long)n);
}

// e^x K_0(x) and e^x K_1(x): trapezoidal rule in t with step h.  The integrand is analytic
// in |Im t| < pi/2; the step keeps the discretisation error below e^-40 relative both for
// small x (strip error ~ e^{-pi^2/h} / x) and large x (Gaussian of width x^-1/2).
void k01_scaled(double x, double &S0, double &S1)
{
    const double h = std::min(9.8696044010893586 / (42.0 + std::max(0.0, -std::log(x))), 0.6 / std::sqrt(x));
    double s0 = 0.5, s1 = 0.5, prev = 1.0;
    for (int k = 1; k < 1000000; k++) {
        const double t = k * h, sh = std::sinh(0.5 * t);
        const double g = std::exp(-2.0 * x * sh * sh); // exp(-x (cosh t - 1))
        const double f1 = g * std::cosh(t);
        s0 += g;
        s1 += f1;
        if (f1 < 1e-18 * s1 && f1 <= prev) break; // past the peak and negligible
        prev = f1;
    }
    S0 = h * s0;
    S1 = h * s1;
}

// e^-x I_0(x)
double i0_scaled(double x)
{
    if (x > 2000.0) {
        // Hankel: sum_k a_k / x^k, a_k = a_{k-1} (2k-1)^2 / (8k), all terms positive
        double term = 1.0, sum = 1.0;
        for (int k = 1; k < 60; k++) {
            term *= (2.0 * k - 1) * (2.0 * k - 1) / (8.0 * k * x);
            sum += term;
            if (term < 1e-18 * sum) break;
        }
        return sum / std::sqrt(2.0 * H_PI * x);
    }
    // N intervals on [0, pi]: the rule adds I_{2N}(x) + I_{2N+2}... relative to I_0, which
    // is below e^-50 once (2N)^2 >= 100 x (large x) or 2N >= 40 (small x)
    const int N = 20 + (int)std::ceil(std::sqrt(25.0 * x));
    double s = 0.5 * (1.0 + std::exp(-2.0 * x));
    for (int k = 1; k < N; k++) {
        const double sh = std::sin(0.5 * H_PI * k / N);
        s += std::exp(-2.0 * x * sh * sh); // exp(x (cos th - 1))
    }
    return s / N;
}

// K_0 .. K_J at x > 0
void k_table(double x, int J, hx *K)
{
    double S0, S1;
    k01_scaled(x, S0, S1);
    const hx ex = hexp(-x);
    K[0] = hmul(ex, hnorm(S0, 0));
    if (J >= 1) K[1] = hmul(ex, hnorm(S1, 0));
    double a = S0, b = S1; // K_{j-1}, K_j in units of 2^e e^-x
    long long e = 0;
    for (int j = 1; j < J; j++) {
        const double c = a + (2.0 * j / x) * b;
        a = b;
        b = c;
        if (b > 0x1p500) { a = std::ldexp(a, -500); b = std::ldexp(b, -500); e += 500; }
        K[j + 1] = hmul(ex, hnorm(b, e));
    }
}

// I_0 .. I_J at x > 0
void i_table(double x, int J, hx *I)
{
    I[0] = hmul(hexp(x), hnorm(i0_scaled(x), 0));
    if (J < 1) return;
    // start of the ratio recurrence: the error of r_M = 0 reaches order j damped by
    // I_M K_j / (K_M I_j) < e^-50 for M^2 >= j^2 + 50 x
    const int M = (int)std::ceil(std::sqrt((double)J * J + 50.0 * x)) + 30;
    std::vector<double> r(J);
    double rr = 0.0; // I_{j+1}/I_j
    for (int j = M - 1; j >= 0; j--) {
        rr = 1.0 / (2.0 * (j + 1) / x + rr);
        if (j < J) r[j] = rr;
    }
    for (int j = 0; j < J; j++) I[j + 1] = hmul(I[j], hnorm(r[j], 0));
}

// ---- tables and batch ----

// device-side table of one q: S[0..n), KQ[0..2n], W[0..n) as scaled doubles (m 2^e)
int tab_stride(int n) { return 4 * n + 1; }
// its scratch: KQ[0..2n+1], KR[0..n+1], IR[0..n+1] as computed
int raw_stride(int n) { return 4 * n + 6; }

__host__ __device__ sd to_sd(hx a)
{
    if (a.m == 0.0 || !isfinite(a.m)) return sd{a.m, 0};
    const long long e = a.e < -(1LL << 29) ? -(1LL << 29) : a.e > 1LL << 29 ? 1LL << 29 : a.e;
    return sd{a.m, (int)e};
}

std::mutex g_capc_mu;
struct Buf {
    void *p = nullptr;
    size_t bytes = 0;
    void *get(size_t need)
    {
        if (need > bytes) {
            if (p) CK(cudaFree(p));
            bytes = std::max(need, bytes + bytes / 4);
            CK(cudaMalloc(&p, bytes));
        }
        return p;
    }
};
Buf b_tab, b_raw, b_rho, b_A, b_md, b_ld, b_tr, b_res, b_st, b_fro, b_work;

} // namespace

// y_{j+1} = y_{j-1} + (2 j / x) y_j, j = j0, j0 + step, ... for count steps from a = y_{j0-step}, b = y_{j0}, raw values
// (b 2^e) stored for orders 0 .. J by one warp: 32 coefficients at a time, one per lane, and 32 values, so that a step of
// the chain is a multiply-add; the exponent is tested every eighth step where coefficients allow it
CAPS_DEV void bessel_chain(double x, double a, double b, int j0, int step, int count, int J, hx *out)
{
    const int lane = threadIdx.x & 31;
    int e = 0;
    for (int i0 = 0; i0 < count; i0 += 32) {
        const double cl = 2.0 * (j0 + step * (i0 + lane)) / x; // past the end: finite and unused
        const bool small = __all_sync(0xffffffffu, expo(cl) < 60); // eight steps: below 2^500 2^(61 * 8)
        double mine = 0.0;
        int emine = 0;
        auto steps = [&](auto ns, int i) {
            constexpr int NS = decltype(ns)::value;
            double cf[NS];
#pragma unroll
            for (int u = 0; u < NS; u++) cf[u] = __shfl_sync(0xffffffffu, cl, i + u);
#pragma unroll
            for (int u = 0; u < NS; u++) {
                const double c = fma(cf[u], b, a);
                a = b;
                b = c;
                if (lane == i + u) mine = b;
            }
            if (lane >= i && lane < i + NS) emine = e;
            if (expo(b) >= 500) {
                a = shift2(a, -500);
                b = shift2(b, -500);
                e += 500;
            }
        };
        if (small)
#pragma unroll 1
            for (int i = 0; i < 32; i += 8) steps(std::integral_constant<int, 8>(), i);
        else
#pragma unroll 1
            for (int i = 0; i < 32; i++) steps(std::integral_constant<int, 1>(), i);
        const int j = j0 + step * (i0 + lane + 1);
        if (i0 + lane < count && j <= J) out[j] = hx{mine, emine};
    }
}

// the tables of one q (grid nq; the first three warps take the chains of K(2 calL q), K(R q), I(R q)), M_ii of its two
// matrices, log(1 - M_00) (NaN: not below 1).  Bound by the chains of 2 n steps; on the host the tables
// of one q took 17 us, one after the other (30 of them 500 us; the kernel 52).
constexpr int CT_NT = 256;
__global__ void __launch_bounds__(CT_NT) k_capc_tab(int nq, double R, double d, int n, const double *qs, bool dirichlet, hx *raw, int rstride, sd *tab,
                                                 int tstride, double *mdiag, double *rho)
{
    const int iq = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (iq >= nq) return;
    const double q = qs[iq], xK = 2.0 * (R + d) * q, xR = R * q;
    hx *KQ = raw + (size_t)iq * rstride, *KR = KQ + 2 * n + 2, *IR = KR + n + 2;
    auto total = [](double v) {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };
    __shared__ hx scale[3]; // what the raw values of each table are multiplied by
    if (warp < 2) {
        // K_0, K_1 as k01_scaled, 32 terms at a time; K_j in units of e^-x
        const double x = warp ? xR : xK;
        const int J = warp ? n + 1 : 2 * n + 1;
        hx *K = warp ? KR : KQ;
        const double h = fmin(9.8696044010893586 / (42.0 + fmax(0.0, -log(x))), 0.6 / sqrt(x));
        double s0 = 0.5, s1 = 0.5;
        for (int k = 0; k < 1000000; k += 32) {
            const double t = (k + lane + 1) * h, sh = sinh(0.5 * t);
            const double g = exp(-2.0 * x * sh * sh), f1 = g * cosh(t);
            s0 += total(g);
            s1 += total(f1);
            const double last = __shfl_sync(0xffffffffu, f1, 31), prev = __shfl_sync(0xffffffffu, f1, 30);
            if (last < 1e-18 * s1 && last <= prev) break;
        }
        s0 *= h;
        s1 *= h;
        if (lane == 0) {
            K[0] = hx{s0, 0};
            K[1] = hx{s1, 0};
            scale[warp] = hexp(-x);
        }
        bessel_chain(x, s0, s1, 1, 1, J - 1, J, K);
    } else if (warp == 2) {
        // I_0 as i0_scaled; the orders downwards from M
        const double x = xR;
        const int J = n + 1, M = (int)ceil(sqrt((double)J * J + 50.0 * x)) + 30;
        bessel_chain(x, 0.0, 1.0, M, -1, M, J, IR);
        double i0;
        if (x > 2000.0) {
            double term = 1.0, sum = 1.0;
            for (int k = 1; k < 60; k++) {
                term *= (2.0 * k - 1) * (2.0 * k - 1) / (8.0 * k * x);
                sum += term;
                if (term < 1e-18 * sum) break;
            }
            i0 = sum / sqrt(2.0 * H_PI * x);
        } else {
            const int N = 20 + (int)ceil(sqrt(25.0 * x));
            double s = 0.0;
            for (int k = lane + 1; k < N; k += 32) {
                const double sh = sin(0.5 * H_PI * k / N);
                s += exp(-2.0 * x * sh * sh);
            }
            i0 = (total(s) + 0.5 * (1.0 + exp(-2.0 * x))) / N;
        }
        __syncwarp();
        if (lane == 0) scale[2] = hdiv(hmul(hexp(x), hnorm(i0, 0)), IR[0]);
    }
    __syncthreads();
    // the three tables lie one after the other
    for (int j = tid; j < 4 * n + 6; j += CT_NT) KQ[j] = hmul(scale[j < 2 * n + 2 ? 0 : j < 3 * n + 4 ? 1 : 2], KQ[j]);
    __syncthreads();
    // r(j): I'_0 / |K'_0| = I_1 / K_1;  I'_j / |K'_j| = (I_{j-1} + I_{j+1}) / (K_{j-1} + K_{j+1})
    auto rat = [&](int j) {
        hx a = IR[j], b = KR[j];
        if (!dirichlet) {
            a = IR[j + 1];
            b = KR[j + 1];
            if (j > 0) {
                a = hadd(IR[j - 1], a);
                b = hadd(KR[j - 1], b);
            }
        }
        return hdiv(a, b);
    };
    const hx r0 = rat(0);
    const double M00 = hval(hmul(r0, KQ[0]));
    const bool ok = M00 < 1.0 && isfinite(M00);
    const hx c1 = hsqrt(hmul(hnorm(ok ? 2.0 / (1.0 - M00) : 1.0, 0), r0));
    if (tid == 0) rho[iq] = ok ? log1p(-M00) : NAN;
    sd *T = tab + (size_t)iq * tstride;
    double *md = mdiag + (size_t)2 * iq * n;
    for (int mu = 1 + tid; mu <= n; mu += CT_NT) {
        const hx s = hsqrt(rat(mu));
        const sd S = to_sd(s), W = to_sd(hmul(c1, hmul(s, KQ[mu])));
        T[mu - 1] = S;
        T[3 * n + mu] = W;
        const sd P = sd_mul(S, S);
        const double U = sd_to_double(sd_mul(P, to_sd(KQ[2 * mu]))), V = sd_to_double(sd_mul(P, to_sd(KQ[0])));
        md[mu - 1] = U - V;
        md[n + mu - 1] = U + V + sd_to_double(sd_mul(W, W));
    }
    for (int k = tid; k <= 2 * n; k += CT_NT) T[n + k] = to_sd(KQ[k]);
}

// 1 - M of matrix `task` = 2 iq + type in fixed point (lower triangle, column-major) and sums of squares of M, one per
// block.  grid (ceil(n/64), ceil(n/16), 2 nq): thread r walks 16 columns c <= r.  Bound by the FP64 pipe (about
// eight operations per element); an FP64 matrix converted afterwards took 154 us for 60 matrices of
// dimension 300, this 64.
constexpr int CE_X = 64, CE_Y = 16;
__global__ void __launch_bounds__(CE_X) k_capc_elem(int ntask, int n, const sd *__restrict__ tab, int tstride, const int *info, long long *A,
                                                    size_t mstride, const double *mdiag, double *fro_out, int *status)
{
    const int task = blockIdx.z, r = blockIdx.x * CE_X + threadIdx.x, c0 = blockIdx.y * CE_Y;
    if (task >= ntask) return;
    double fro = 0.0;
    if (c0 < (int)(blockIdx.x + 1) * CE_X) { // uniform: the block has elements
        const sd *T = tab + (size_t)(task >> 1) * tstride;
        const sd *S = T, *KQ = T + n, *W = T + 3 * n + 1;
        const bool type = task & 1;
        const int fq = FQ - info[2 * task];
        const long long one = fq >= 0 ? 1LL << fq : 0;
        int err = 0;
        if (r < n) {
            const sd Sr = S[r], Wr = W[r];
            // m 2^e of products of three mantissas in [0.5, 1)
            auto val = [](double m, int e) { return e > 1000 ? m * INFINITY : e < -1020 ? 0.0 : shift2(m, e); };
            const int c1 = min(c0 + CE_Y, r);
#pragma unroll 4
            for (int c = c0; c < c1; c++) {
                const sd Sc = S[c], Ku = KQ[r + c + 2], Kv = KQ[r - c];
                const double P = Sr.m * Sc.m, U = val(P * Ku.m, Sr.e + Sc.e + Ku.e), V = val(P * Kv.m, Sr.e + Sc.e + Kv.e);
                double M = U - V;
                if (type) {
                    const sd Wc = W[c];
                    M = U + V + val(Wr.m * Wc.m, Wr.e + Wc.e);
                }
                A[(size_t)task * mstride + (size_t)c * n + r] = -to_fix(M, fq, err);
                fro = fma(M, M, fro);
            }
            fro *= 2.0;
            if (r >= c0 && r < c0 + CE_Y) {
                const double M = mdiag[(size_t)task * n + r];
                A[(size_t)task * mstride + (size_t)r * n + r] = one - to_fix(M, fq, err);
                fro = fma(M, M, fro);
            }
        }
        if (err) atomicOr(status + task, err);
    }
    __shared__ double red[CE_X / 32];
    for (int o = 16; o > 0; o >>= 1) fro += __shfl_xor_sync(0xffffffffu, fro, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = fro;
    __syncthreads();
    if (threadIdx.x == 0) fro_out[((size_t)task * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = red[0] + red[1];
}

// log det of the cylinder-plane round trip for nq wave numbers; returns the number of
// results that are NaN because of a numerical failure
int capc_batch(double R, double d, int n, const double *q, int nq, char DN, int mode, double *out)
{
    std::lock_guard<std::mutex> lk(g_capc_mu);
    const size_t mstride = (size_t)n * n;
    const int ts = tab_stride(n);
    // chunks of at most 4 GB of matrices, 4 GB of the factorisation's workspace (250 KB for the smallest matrices) and
    // 16384 wave numbers (grid z = 2 per q)
    const int chunk = (int)std::max<size_t>(1, std::min({(size_t)nq, (size_t)16384, ((size_t)4 << 30) / (2 * mstride * sizeof(double)),
                                                         ((size_t)4 << 30) / cholesky_work_bytes(2, n)}));
    const int rs = raw_stride(n);
    const dim3 ge((n + CE_X - 1) / CE_X, (n + CE_Y - 1) / CE_Y);
    const int nfro = ge.x * ge.y;
    std::vector<double> rho(chunk), res(2 * (size_t)chunk);
    std::vector<int> hst(2 * (size_t)chunk);
    int nbad = 0;
    const cudaStream_t st = 0;
    for (int q0 = 0; q0 < nq; q0 += chunk) {
        const int nc = std::min(chunk, nq - q0), nt = 2 * nc;
        sd *d_tab = (sd *)b_tab.get((size_t)nc * ts * sizeof(sd));
        double *d_A = (double *)b_A.get((size_t)nt * mstride * sizeof(double));
        double *d_md = (double *)b_md.get((size_t)nt * n * sizeof(double));
        double *d_ld = (double *)b_ld.get((size_t)nt * n * sizeof(double));
        double *d_tr = (double *)b_tr.get((size_t)nt * sizeof(double));
        double *d_res = (double *)b_res.get((size_t)nt * sizeof(double));
        int *d_st = (int *)b_st.get((size_t)nt * sizeof(int));
        hx *d_raw = (hx *)b_raw.get((size_t)nc * rs * sizeof(hx));
        double *d_q = (double *)b_rho.get((size_t)2 * nc * sizeof(double)), *d_rho = d_q + nc;
        double *d_fro = (double *)b_fro.get((size_t)nt * nfro * sizeof(double));
        void *d_work = b_work.get(cholesky_work_bytes(nt, n));
        CK(cudaMemcpyAsync(d_q, q + q0, (size_t)nc * sizeof(double), cudaMemcpyHostToDevice, st));
        g_counters.h2d += (long long)nc * sizeof(double);
        CK(cudaMemsetAsync(d_st, 0, (size_t)nt * sizeof(int), st));
        k_capc_tab<<<nc, CT_NT, 0, st>>>(nc, R, d, n, d_q, DN == 'D', d_raw, rs, d_tab, ts, d_md, d_rho);
        launch_fix_scale(nullptr, nt, n, d_md, d_work, st);
        k_capc_elem<<<dim3(ge.x, ge.y, nt), CE_X, 0, st>>>(nt, n, d_tab, ts, (const int *)d_work, (long long *)d_A, mstride, d_md, d_fro, d_st);
        COUNT_LAUNCH(2);
        CK(cudaGetLastError());
        launch_stats(nullptr, nt, n, d_A, n, mstride, d_md, mode, d_tr, d_res, d_st, st, d_fro, nfro);
        launch_cholesky(nt, n, d_A, n, mstride, d_st, d_md, d_ld, d_work, st, true);
        launch_final(nt, n, d_ld, d_work, d_tr, d_st, d_res, mode, st);
        CK(cudaMemcpyAsync(rho.data(), d_rho, (size_t)nc * sizeof(double), cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(res.data(), d_res, (size_t)nt * sizeof(double), cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(hst.data(), d_st, (size_t)nt * sizeof(int), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        g_counters.d2h += (long long)nt * (sizeof(double) + sizeof(int)) + (long long)nc * sizeof(double);
        g_counters.nmat += nt;
        for (int k = 0; k < nc; k++) {
            const bool bad = std::isnan(rho[k]) || (hst[2 * k] & ~0xF) || (hst[2 * k + 1] & ~0xF);
            out[q0 + k] = bad ? NAN : rho[k] + res[2 * k] + res[2 * k + 1];
            nbad += bad;
        }
    }
    return nbad;
}

} // namespace capsgpu

using namespace capsgpu;

namespace {
char norm_dn(char DN) { return std::toupper((unsigned char)DN) == 'D' ? 'D' : 'N'; } // capc.cpp:51-53
int norm_lmax(double R, double d, int lmax) { return lmax > 0 ? lmax : std::max(25, (int)(5 * R / d)); } // capc.cpp:28
} // namespace

extern "C" int caps_capc_lmax(double R, double d, double eta)
{
    TERMINATE(!(R > 0) || !(d > 0) || !(eta > 0), "capc: R, d and eta must be positive");
    return std::max(25, (int)std::ceil(eta / d * R));
}

extern "C" double caps_capc_pfa(double R, double d)
{
    return -H_PI * H_PI * H_PI / 1920 * std::sqrt(R / (2 * d)) / (d * d);
}

extern "C" int caps_capc_logdet_batch(double R, double d, int lmax, const double *q, int nq, char DN, detalg_t detalg, double *out)
{
    TERMINATE(!(R > 0) || !(d > 0), "capc: R and d must be positive");
    if (nq <= 0) return 0;
    for (int k = 0; k < nq; k++) TERMINATE(!(q[k] > 0) || !std::isfinite(q[k]), "capc: wave number q must be positive and finite");
    return capc_batch(R, d, norm_lmax(R, d, lmax), q, nq, norm_dn(DN), detalg == DETALG_HODLR ? 1 : 0, out);
}

extern "C" double caps_capc_logdet(double R, double d, int lmax, double q, char DN, detalg_t detalg)
{
    double r = NAN;
    caps_capc_logdet_batch(R, d, lmax, &q, 1, DN, detalg, &r);
    return r;
}

extern "C" double caps_capc_energy_T0(double R, double d, int lmax, char p, double epsrel, detalg_t detalg, int *neval_out,
                                      int *ier_out)
{
    TERMINATE(!(R > 0) || !(d > 0), "capc: R and d must be positive");
    TERMINATE(!(epsrel > 0), "capc: epsrel must be positive");
    const int n = norm_lmax(R, d, lmax);
    const char DN = norm_dn(p);
    const int mode = detalg == DETALG_HODLR ? 1 : 0;
    // integrand x -> q logdet(q), q = x/(2d) (capc.cpp:180-194), every node of a qagi step in one batch
    const BatchFn F = [&](const double *x, int k, double *y) {
        std::vector<double> qs(k);
        for (int i = 0; i < k; i++) qs[i] = x[i] / (2 * d);
        capc_batch(R, d, n, qs.data(), k, DN, mode, y);
        for (int i = 0; i < k; i++) y[i] *= qs[i];
    };
    double abserr = 0;
    int neval = 0, ier = 0;
    const double integral = qagi_batched(F, 0, 1, 0, epsrel, &abserr, &neval, &ier);
    if (neval_out) *neval_out = neval;
    if (ier_out) *ier_out = ier;
    return integral / (4 * H_PI * 2 * d);
}

// ---- integer-order modified Bessel functions (the reference's bessel.h names) ----

extern "C" double bessel_logI0(double x)
{
    if (x < 0) return NAN;
    if (x == 0) return 0.0;
    std::vector<hx> I(1);
    i_table(x, 0, I.data());
    return hlog(I[0]);
}

extern "C" double bessel_logI1(double x)
{
    if (!(x > 0)) return NAN;
    std::vector<hx> I(2);
    i_table(x, 1, I.data());
    return hlog(I[1]);
}

extern "C" double bessel_logK0(double x)
{
    if (!(x > 0)) return NAN;
    hx K;
    k_table(x, 0, &K);
    return hlog(K);
}

extern "C" double bessel_logK1(double x)
{
    if (!(x > 0)) return NAN;
    hx K[2];
    k_table(x, 1, K);
    return hlog(K[1]);
}

extern "C" double bessel_logIn(int n, double x)
{
    if (n < 0) n = -n;
    if (n == 0) return bessel_logI0(x);
    if (n == 1) return bessel_logI1(x);
    if (x == 0) return -INFINITY;
    if (!(x > 0)) return NAN;
    std::vector<hx> I(n + 1);
    i_table(x, n, I.data());
    return hlog(I[n]);
}

extern "C" double bessel_logKn(int n, double x)
{
    if (n < 0) n = -n;
    if (!(x > 0)) return NAN;
    std::vector<hx> K(n + 1);
    k_table(x, n, K.data());
    return hlog(K[n]);
}
