// sweep.cu -- the mixed form's round-trip matrix from a band of q-sums and a three-term
// recurrence of the I integrals: a kernel that fills the table of I row by row and one that forms
// the elements from its tiles.
//
// The q-sum of every (l1, l2) pair (integration.c:491-609) costs O(l) terms, O(ldim^3) per
// matrix.  The I integrals also obey the three-term recurrence of the associated Legendre
// functions in either degree, (2l+1) x P_l^m = (l-m+1) P_{l+1}^m + (l+m) P_{l-1}^m, which,
// applied once in each degree of I_{l1 l2} = int w(x) P_{l1}^{m'} P_{l2}^{m'} (m' = max(m,1)),
// links four neighbours:
//   (l1-m'+1) I(l1+1, l2) = (2l1+1)/(2l2+1) [(l2-m'+1) I(l1, l2+1) + (l2+m') I(l1, l2-1)]
//                           - (l1+m') I(l1-1, l2).
// Seeded with q-sums on the diagonal (l1 = l2), the first subdiagonal (l1 = l2 + 1) and the
// first column of the window, it fills the lower triangle row by row, moving away from the
// diagonal.  Against the q-sums of the reference's algorithm the filled values agree to ~1e-11
// relative (also 1000 rows from the seeds, from xi = 0.1 to 1119, m = 0 to 400), and
// log det(1 - M) built from them moves by <= 5e-14 relative in float-float arithmetic -- far
// below the FP32 storage of M, which dominates the mixed form's error.  The recurrence costs
// O(1) per pair: the q-sums shrink to 4 L pairs per matrix (two of which the trace rule's
// diagonal reads anyway).
//
// Scaling.  The table is held as T(w1, w2) = I(w1, w2) 2^{k(w1) + k(w2)} (w: index into the
// window [lmin-1, lmin+ldim]) with k(w) = -floor(log2 I_TM(w, w) / 2), so that T_TM(w, w) lies in
// [1, 4).  For a plate of real dielectric function the weight w(x) of the integral has one sign
// per polarisation, so I_p is a signed Gram matrix and |T(w1, w2)| <= sqrt(T(w1,w1) T(w2,w2)) < 4:
// every value sits in one fixed float-float frame (no per-entry exponent); far entries that
// fall below 2^-121 of that frame flush to zero, as they do in the FP32 matrix.  The powers of
// two enter the recurrence coefficients exactly.
//
// Elements (libcaps.c:761-831, integration.c:762-888) in this frame.  With
// Um(w) = u(w) 2^{k(w) - k(w-1)}, Vp(w) = v(w) 2^{k(w) - k(w+1)} (u, v the coefficients of the
// B, C, D combinations), dA(w) = Sa(w) 2^{-k(w)}, dB(w) = Sb(w) 2^{-k(w)} (Sa, Sb the symmetric
// Mie and normalisation factors), and per polarisation
//   J(x, y) = Um(x) T(x-1, y) - Vp(x) T(x+1, y)      (B, C, D differentiate in l1 ...)
//   H(x, y) = Um(y) T(x, y-1) - Vp(y) T(x, y+1)      (... and in l2)
//   B(x, y) = Um(y) J(x, y-1) - Vp(y) J(x, y+1),
// the 2x2 block at window row x, column y is
//   EE = dA(x) dA(y) [B_TM - m^2 T_TE],          MM = dB(x) dB(y) [m^2 T_TM - B_TE],
//   EM = m dA(x) dB(y) [H_TE - J_TM],            ME = m dB(x) dA(y) [J_TE - H_TM]
// (m = 0: EE = dA dA T_TM, MM = -dB dB T_TE).  Um = (l+1) Cm and Vp = l Cp for m >= 1, Cp and Cm
// the column coefficients of the recurrence, so one pair of tables serves both.
//
// Two kernels behind a table of coefficients (k_sweep_tab).  k_rec_ff fills T row by row, one CTA per matrix and
// polarisation; k_elem_sweep forms the elements of all pairs from tiles of T, with the row factors dA, dB
// folded into the row's coefficients and the column factors into the column's.  The elements go
// straight into the FP32 delta matrix (-M, lower triangle, column-major), with sums
// of squares for the reference's Mercator bound where they are wanted; the FP64 diagonal comes from the band
// (k_diag_ff).  One kernel for both, one CTA per matrix with producer warps for the rows and consumer warps for
// the elements, was bound by its 10 warps' latencies and by stores 2 n rows apart from lane to lane: 547 matrices of
// ldim 1050 8.9 ms, now 2.1 (rows) + 4.0 (elements).
#include "common.cuh"
#include "ff.cuh"
#include "internal.h"
#include "qsum_ff.cuh"

namespace capsgpu {

// window index of the first l with I != 0: l = max(lmin - 1, m')
CAPS_DEV int seed_col(const Task &T)
{
    const int mm = T.m > 0 ? T.m : 1;
    return T.lmin - 1 >= mm ? 0 : 1;
}

// ranges of rows of T: part q of P forms rows (row(q), row(q + 1)], row(0) = -1, of about equal numbers of pairs; parts
// q >= 1 start from the q-sums of rows row(q) - 1 and row(q).  The number depends on ldim alone, so that a matrix has the
// same value in every batch.  Few matrices leave SMs idle behind the chain of rows; parts of 512 rows against one part, ms of
// seeds, table and elements: ldim 1050, 1 matrix 0.77 -> 0.55, 6 0.86 -> 0.63, 48 1.30 -> 1.12, 547 6.42 -> 6.40; 1500, 1
// 1.23 -> 0.81, 48 2.20 -> 1.81, 200 4.80 -> 4.73; 2000, 1 1.90 -> 0.91, 48 3.40 -> 2.44, 150 6.27 -> 5.95; 3000, 6
// 5.22 -> 1.58.  No batch loses, so the line is where there is a second part
__host__ __device__ inline int recf_row(int q, int P, int L) { return q <= 0 ? -1 : q >= P ? L - 1 : (int)(L * sqrt((double)q / P)); }
__host__ __device__ inline int recf_parts(int ldim) { return ldim < 1024 ? 1 : ldim / 512; }

// ---------------------------------------------------------------------------
// seeds: q-sums of the pairs of two kinds per window index w
// ---------------------------------------------------------------------------
// grid (np ceil(L/128), ngroups): the first block row computes kind0, the second kind1
// (so that a warp runs sums of one kind and similar length), two more per part q = 1 .. the pairs (row(q) - 1, w) and
// (row(q), w), rows[((((list entry) (P - 1) + q - 1) * 2 + i) * 2 + pol) * L + w].  groups as in launch_itab_grp; a_0,
// a_1, a_2 come from the per-m tables (a012f_pair), so no pair table is formed.  seed[((task *
// 2 + pol) * SEED_KINDS + kind) * L + w] receives the pair's value as float-float with exponent;
// pairs outside the window are not written (nothing reads them).
template <int G>
__global__ void __launch_bounds__(128, 7) k_seed_ff(const Task *tasks, const int *tlist, const int4 *groups, int ngroups, int ldim,
                                                    const float4 *__restrict__ KP, const int *__restrict__ KPe, int nu_stride,
                                                    const float4 *__restrict__ ptabf, int pstride, const A12L *__restrict__ tl,
                                                    const A12J *__restrict__ tj, int kind0, int kind1, ffe *seed, int P, ffe *rows, int *status,
                                                    int stop_bits)
{
    const int L = ldim + 2, NJ = 2 * L - 1, nbw = (L + 127) / 128;
    const int gi = blockIdx.y;
    if (gi >= ngroups) return;
    const int bp = (int)blockIdx.x / nbw, kind = bp == 0 ? kind0 : bp == 1 ? kind1 : SEED_KINDS; // SEED_KINDS: a row
    const int rq = (bp - 2) / 2 + 1, ri = bp & 1;
    const int w = ((int)blockIdx.x % nbw) * 128 + threadIdx.x;
    if (w >= L) return;
    const int4 grp = groups[gi];
    const int ng = grp.y;
    int tk[G];
#pragma unroll
    for (int g = 0; g < G; g++) tk[g] = g < ng ? (tlist ? tlist[grp.x + g] : grp.x + g) : 0;
    const Task &T = tasks[tk[0]];
    int a1 = w, a2 = w;
    if (kind == SEED_D1) a1 = w + 1;
    else if (kind == SEED_D2) a1 = w + 2;
    else if (kind == SEED_COL) a2 = seed_col(T);
    else if (kind == SEED_KINDS) a1 = recf_row(rq, P, L) - 1 + ri;
    if (a1 >= L || (kind == SEED_KINDS && w > a1)) return;
    auto store = [&](int g, int pol, float h, float l, int e) {
        ffe *o = kind == SEED_KINDS ? rows + ((((size_t)(grp.x + g) * (P - 1) + rq - 1) * 2 + ri) * 2 + pol) * L
                                    : seed + ((size_t)(tk[g] * 2 + pol) * SEED_KINDS + kind) * L;
        o[w] = ffe{h, l, e, 0};
    };
    const int mm = T.m > 0 ? T.m : 1, l1 = T.lmin - 1 + a1, l2 = T.lmin - 1 + a2;
    if (a1 < a2 || l2 < mm || l2 < T.m || l1 < 1) { // I = 0 for l < m (integration.c:631)
        for (int g = 0; g < ng; g++) { store(g, 1, 0.0f, 0.0f, FFE_ZERO_E); store(g, 0, 0.0f, 0.0f, FFE_ZERO_E); }
        return;
    }
    const A012F A12 = a012f_pair(T.m, T.lmin, a1, a2, tl + (size_t)grp.z * L, tj + (size_t)grp.z * NJ);
    const unsigned bad = qsum_ff_pair<G>(T, tk, ng, l1, l2, A12, KP, KPe, nu_stride, ptabf + (size_t)grp.z * 2 * pstride * 2,
                                          pstride, stop_bits, store);
#pragma unroll
    for (int g = 0; g < G; g++)
        if (g < ng && (bad & (1u << g))) atomicOr(status + tk[g], ST_ERR_NONFINITE);
}

// ---------------------------------------------------------------------------
// the sweep
// ---------------------------------------------------------------------------
CAPS_DEV ff ff_sub(ff x, ff y) { return ff_add(x, ff_neg(y)); }
// x c for c exactly representable in FP32 (small integers)
CAPS_DEV ff ff_mulf(ff x, float c)
{
    const float p = x.h * c;
    float e = fmaf(x.h, c, -p);
    e = fmaf(x.l, c, e);
    return ff_fast2(p, e);
}
// a x + b y: the two products with their rounding errors (fmaf), one exact sum of the leading
// parts and one renormalisation (the float-float error of ff_add(ff_mul, ff_mul), fewer steps)
CAPS_DEV ff ff_dot2(ff a, ff x, ff b, ff y)
{
    const float p = a.h * x.h, q = b.h * y.h;
    float ep = fmaf(a.h, x.h, -p);
    ep = fmaf(a.h, x.l, ep);
    ep = fmaf(a.l, x.h, ep);
    float eq = fmaf(b.h, y.h, -q);
    eq = fmaf(b.h, y.l, eq);
    eq = fmaf(b.l, y.h, eq);
    const float s = p + q, bb = s - p;
    const float t = (p - (s - bb)) + (q - bb);
    return ff_fast2(s, t + (ep + eq));
}
// FP32 of a x + b y + c z: float-float products and sums, one rounding at the end
CAPS_DEV float ff_dot3(ff a, ff x, ff b, ff y, ff c, ff z)
{
    const float p = a.h * x.h, q = b.h * y.h, u = c.h * z.h;
    float ep = fmaf(a.h, x.h, -p);
    ep = fmaf(a.h, x.l, ep);
    ep = fmaf(a.l, x.h, ep);
    float eq = fmaf(b.h, y.h, -q);
    eq = fmaf(b.h, y.l, eq);
    eq = fmaf(b.l, y.h, eq);
    float eu = fmaf(c.h, z.h, -u);
    eu = fmaf(c.h, z.l, eu);
    eu = fmaf(c.l, z.h, eu);
    const float s1 = p + q, b1 = s1 - p, t1 = (p - (s1 - b1)) + (q - b1);
    const float s2 = s1 + u, b2 = s2 - s1, t2 = (s1 - (s2 - b2)) + (u - b2);
    return s2 + ((t1 + t2) + (ep + (eq + eu)));
}

// 1 / y in float-float: the hardware reciprocal and two corrections (relative error ~2^-48)
CAPS_DEV ff ff_rcp(ff y)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y.h));
    ff q{r, 0.0f};
#pragma unroll
    for (int it = 0; it < 2; it++) {
        const ff e = ff_sub(ff{1.0f, 0.0f}, ff_mul(q, y));
        q = ff_add(q, ff_mul(q, e));
    }
    return q;
}

// k(w) of the scaling: I_TM(w, w) 2^{2 k(w)} in [1, 4).  Window indices below the first
// column (zero rows) take the first column's k.
CAPS_DEV int sw_k(const ffe *__restrict__ d0tm, int w, int c)
{
    const ffe v = d0tm[w < c ? c : w];
    return v.h == 0.0f ? 0 : -(v.e >> 1);
}

// a seed (h + l) 2^e in the frame: times 2^{k1 + k2}
CAPS_DEV ff sw_seed(const ffe &v, int k12) { return v.h == 0.0f ? ff{0.0f, 0.0f} : ff_shift(ff{v.h, v.l}, v.e + k12); }

// FP32 of h 2^e; below 2^-120 -> 0, non-finite or above 2^125 sets bad
CAPS_DEV float sw_out(float h, int e, bool &bad)
{
    const int k = fexpo(h);
    if (k == -127) return 0.0f;
    if (k == 128 || k + e > 125) { bad = true; return h; }
    return fshift(h, e);
}

// per listed task and window index w, tab[(b * SWF_FIELDS + field) * L + w]: pairs of float-float numbers --
// Cp, Cm of the recurrence; R1 = 1 / Cp(w - 1), -R1 Cm(w - 1) of row w; the mantissas of Um dA, -Vp dA; m dA, dA; Um dB, -Vp dB;
// m dB, dB; the scaled seeds (TE, TM) of row w, T(w, w), T(w, w - 1), T(w, c); the exponents of dA, dB as two
// integers, a bound of the exponents of the six factors times theirs, and k(w)
enum { SWF_C, SWF_R, SWF_UA, SWF_A, SWF_UB, SWF_B, SWF_D0, SWF_D1, SWF_COL, SWF_E, SWF_FIELDS };

// grid nlist, 256 threads
__global__ void __launch_bounds__(256) k_sweep_tab(const Task *tasks, const int *tlist, int nlist, int ldim, const ffe *__restrict__ seed,
                                                   const ffe *__restrict__ Saf, const ffe *__restrict__ Sbf, float4 *tab)
{
    const int L = ldim + 2;
    if ((int)blockIdx.x >= nlist) return;
    const int task = tlist ? tlist[blockIdx.x] : (int)blockIdx.x;
    const Task &T = tasks[task];
    const int mt = T.m, mm = mt > 0 ? mt : 1, lm1 = T.lmin - 1, c = seed_col(T);
    auto sp = [&](int pol, int kind) { return seed + ((size_t)(task * 2 + pol) * SEED_KINDS + kind) * L; };
    const ffe *d0tm = sp(1, SEED_D0);
    auto CP = [&](int w) {
        const int l = lm1 + w;
        return w >= c && w + 1 < L ? ff_shift(ff_from_d((double)(l - mm + 1) / (2.0 * l + 1)), sw_k(d0tm, w, c) - sw_k(d0tm, w + 1, c))
                                   : ff{0.0f, 0.0f};
    };
    auto CM = [&](int w) {
        const int l = lm1 + w;
        return w >= c + 1 ? ff_shift(ff_from_d((double)(l + mm) / (2.0 * l + 1)), sw_k(d0tm, w, c) - sw_k(d0tm, w - 1, c)) : ff{0.0f, 0.0f};
    };
    auto pair = [](ff a, ff b) { return make_float4(a.h, a.l, b.h, b.l); };
    for (int w = threadIdx.x; w < L; w += blockDim.x) {
        float4 *t = tab + (size_t)blockIdx.x * SWF_FIELDS * L + w;
        auto put = [&](int field, float4 v) { t[(size_t)field * L] = v; };
        const int l = lm1 + w, kw = sw_k(d0tm, w, c);
        const ff cp = CP(w), cm = CM(w);
        put(SWF_C, pair(cp, cm));
        ff r1{0.0f, 0.0f}, r2{0.0f, 0.0f};
        if (w >= c + 3) {
            r1 = ff_rcp(CP(w - 1));
            r2 = ff_neg(ff_mul(r1, CM(w - 1)));
        }
        put(SWF_R, pair(r1, r2));
        const ff um = ff_mulf(cm, (float)(l + 1)), vp = ff_neg(ff_mulf(cp, (float)l));
        const ffe a = Saf[(size_t)task * L + w], b = Sbf[(size_t)task * L + w];
        const ff dA{a.h, a.l}, dB{b.h, b.l};
        const int ea = a.h == 0.0f ? 0 : min(max(a.e - kw, -30000), 30000), eb = b.h == 0.0f ? 0 : min(max(b.e - kw, -30000), 30000);
        const float4 f[4] = {pair(ff_mul(um, dA), ff_mul(vp, dA)), pair(ff_mulf(dA, (float)mt), dA), pair(ff_mul(um, dB), ff_mul(vp, dB)),
                             pair(ff_mulf(dB, (float)mt), dB)};
        put(SWF_UA, f[0]);
        put(SWF_A, f[1]);
        put(SWF_UB, f[2]);
        put(SWF_B, f[3]);
        const int xa = max(max(fexpo(f[0].x), fexpo(f[0].z)), max(fexpo(f[1].x), fexpo(f[1].z))) + ea; // not finite: 128
        const int xb = max(max(fexpo(f[2].x), fexpo(f[2].z)), max(fexpo(f[3].x), fexpo(f[3].z))) + eb;
        put(SWF_E, make_float4(__int_as_float(ea), __int_as_float(eb), __int_as_float(max(xa, xb)), __int_as_float(kw)));
        auto seeds = [&](int kind, int y, int wi) {
            ff v[2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
            if (y >= c && wi >= 0)
                for (int pol = 0; pol < 2; pol++) v[pol] = sw_seed(sp(pol, kind)[wi], kw + sw_k(d0tm, y, c));
            return pair(v[0], v[1]);
        };
        put(SWF_D0, seeds(SEED_D0, w, w));
        put(SWF_D1, seeds(SEED_D1, w - 1, w - 1));
        put(SWF_COL, seeds(SEED_COL, c, w));
    }
}

// T(r, y), y <= r, of listed task b at tt[((b * 2 + pol) * L + r) * L + y].  Grid nlist * P * 2: a part of the rows and one
// polarisation (TE, TM) per CTA, the ring of three rows in shared memory (r and the two before it), one barrier per row; a thread keeps the coefficients of its first
// columns in registers and the next row's seeds and factors are loaded a row ahead, so that the row's chain
// is two float-float sums and the barrier.  Bound by that chain and by issue (about 95 instructions per column).
constexpr int RF_NT = 256, RF_RING = 3, RF_KEEP = 4;
__global__ void __launch_bounds__(RF_NT) k_rec_ff(const Task *tasks, const int *tlist, int nlist, int ldim, int P, const ffe *__restrict__ rows,
                                                  const float4 *__restrict__ tab, float2 *tt,
                                                  const int *status)
{
    extern __shared__ __align__(16) float2 rf_sm[];
    const int L = ldim + 2;
    const int pol = blockIdx.x & 1, part = blockIdx.x >> 1, b = part / P, q = part % P, tid = threadIdx.x;
    if (b >= nlist) return;
    const int task = tlist ? tlist[b] : b;
    if (status[task] & ~0xF) return; // no status changes in this launch: uniform
    const int c = seed_col(tasks[task]), r0 = recf_row(q, P, L) + 1, r1 = recf_row(q + 1, P, L);
    const float4 *W = tab + (size_t)b * SWF_FIELDS * L;
    float2 *t = tt + (((size_t)b * 2 + pol) * L + r0) * L;
    __shared__ float4 s_r[2];       // of the next row: R1, -R2
    __shared__ float2 s_seed[2][3]; // and its seeds
    auto fetch = [&](int row) {
        if (tid < 4 && row < L) {
            const float4 v = __ldg(W + (size_t)(tid < 3 ? SWF_D0 + tid : SWF_R) * L + row);
            if (tid < 3) s_seed[row & 1][tid] = pol ? make_float2(v.z, v.w) : make_float2(v.x, v.y);
            else s_r[row & 1] = v;
        }
    };
    float4 keep[RF_KEEP];
#pragma unroll
    for (int i = 0; i < RF_KEEP; i++) keep[i] = tid + i * RF_NT < L ? __ldg(W + (size_t)SWF_C * L + tid + i * RF_NT) : make_float4(0, 0, 0, 0);
    fetch(r0);
    // rows r, r - 1, r - 2; rows before the first are never read: y >= c + 1 and y <= r - 2 need r >= 3
    float2 *D = rf_sm, *P1 = rf_sm + L, *P2 = rf_sm + 2 * L;
    if (q > 0) // the two rows before the part, from their q-sums
        for (int i = 0; i < 2; i++) {
            const int rr = r0 - 2 + i;
            const ffe *src = rows + ((((size_t)b * (P - 1) + q - 1) * 2 + i) * 2 + pol) * L;
            const int kr = __float_as_int(__ldg(W + (size_t)SWF_E * L + rr).w);
            for (int y = tid; y <= rr; y += RF_NT) {
                const ff v = y < c ? ff{0.0f, 0.0f} : sw_seed(src[y], kr + __float_as_int(__ldg(W + (size_t)SWF_E * L + y).w));
                (i ? P1 : P2)[y] = make_float2(v.h, v.l);
            }
        }
    __syncthreads();
    for (int r = r0; r <= r1; r++) {
        fetch(r + 1);
        const float4 R = s_r[r & 1];
        const float2 *seeds = s_seed[r & 1];
        auto column = [&](int y, const float4 &C) {
            float2 v = make_float2(0.0f, 0.0f);
            if (y >= c) {
                if (y == r || y == r - 1 || y == c) v = seeds[y == r ? 0 : y == r - 1 ? 1 : 2];
                else {
                    auto ld = [](const float2 &u) { return ff{u.x, u.y}; };
                    const ff s = ff_dot2(ff{R.x, R.y}, ff_dot2(ff{C.x, C.y}, ld(P1[y + 1]), ff{C.z, C.w}, ld(P1[y - 1])), ff{R.z, R.w}, ld(P2[y]));
                    v = make_float2(s.h, s.l);
                }
            }
            D[y] = v;
            t[y] = v;
        };
#pragma unroll
        for (int i = 0; i < RF_KEEP; i++)
            if (tid + i * RF_NT <= r) column(tid + i * RF_NT, keep[i]);
        for (int y = tid + RF_KEEP * RF_NT; y <= r; y += RF_NT) column(y, __ldg(W + (size_t)SWF_C * L + y));
        __syncthreads();
        float2 *next = P2;
        P2 = P1;
        P1 = D;
        D = next;
        t += L;
    }
}

// Elements from the table.  Grid (ceil(ldim / EL_X), ceil(ldim / EL_Y), nlist), EL_X threads: thread x walks EL_Y columns y <= x of
// a tile of T in shared memory, with J(x, v) = Um(x) T(x-1, v) - Vp(x) T(x+1, v) of the columns y - 1, y, y + 1 in
// registers; consecutive threads write consecutive rows of the column-major matrix.  S receives -M; sums (FRO) the sum
// of squares of M (both triangles), one per block.
//
// Pairs whose four elements are all below 2^-62 of the matrix (the FP64 form's last digit; the panel solves take
// what is below 2^-52 as zero) are stored as zeros where a whole warp's are, unless the sums are wanted.  Bound by
// issue and shared-memory latency at 11 CTAs per SM (256 instructions per pair); the next column read one step ahead
// cost more in registers' moves than it hid (4.4 ms against 4.0).
constexpr int EL_X = 64, EL_Y = 16, EL_LD = EL_Y + 3; // odd row length: consecutive rows in distinct banks
template <bool FRO>
__global__ void __launch_bounds__(EL_X) k_elem_sweep(const Task *tasks, const int *tlist, int nlist, int ldim, const float2 *__restrict__ tt,
                                                     const float4 *__restrict__ tab, float *S, size_t sstride, float *sums, int *status)
{
    const int L = ldim + 2, n = 2 * ldim, b = blockIdx.z, tid = threadIdx.x;
    if (b >= nlist) return;
    const int task = tlist ? tlist[b] : b;
    const int X0 = blockIdx.x * EL_X + 1, x = X0 + tid, y0 = blockIdx.y * EL_Y + 1;
    __shared__ float2 sT[2][EL_X + 2][EL_LD];
    __shared__ float red[EL_X / 32];
    float fro = 0.0f;
    if (y0 <= min(X0 + EL_X - 1, ldim)) { // uniform: the block has elements
        bool bad = false;
        const int mt = tasks[task].m;
        // T(u, v) of rows X0 - 1 .. X0 + EL_X and columns y0 - 1 .. y0 + EL_Y, any order of u and v
        constexpr int ROWS = EL_X / (EL_Y + 2); // rows at a time
        const int ti = tid / (EL_Y + 2), tj = tid % (EL_Y + 2), v = min(y0 - 1 + tj, L - 1);
        if (ti < ROWS) {
            const float2 *t0 = tt + (size_t)b * 2 * L * L, *t1 = t0 + (size_t)L * L;
#pragma unroll 4
            for (int i = ti; i < EL_X + 2; i += ROWS) {
                const int u = min(X0 - 1 + i, L - 1);
                const size_t o = u >= v ? (size_t)u * L + v : (size_t)v * L + u;
                sT[0][i][tj] = t0[o];
                sT[1][i][tj] = t1[o];
            }
        }
        __syncthreads();
        const float4 *W = tab + (size_t)b * SWF_FIELDS * L;
        auto F = [&](int f, int w) { return __ldg(W + (size_t)f * L + w); };
        auto lo = [](const float4 &v) { return ff{v.x, v.y}; };
        auto hi = [](const float4 &v) { return ff{v.z, v.w}; };
        const int xx = min(x, ldim);
        auto TV = [&](int pol, int i, int v) { const float2 q = sT[pol][tid + i][v - y0 + 1]; return ff{q.x, q.y}; };
        const float4 xE = F(SWF_E, xx);
        const int eA = __float_as_int(xE.x), eB = __float_as_int(xE.y), exr = __float_as_int(xE.z);
        float *Sp = S + (size_t)task * sstride + (size_t)2 * (y0 - 1) * n + 2 * (x - 1);
        const int y1 = min(y0 + EL_Y - 1, ldim); // uniform; lanes with x < y are idle
        auto store = [&](int y, float ee, float mm, float em, float me) {
            *reinterpret_cast<float2 *>(Sp) = make_float2(-ee, -me);
            if (y != x) {
                *reinterpret_cast<float2 *>(Sp + n) = make_float2(-em, -mm);
                if (FRO) fro += 2.0f * (ee * ee + me * me + mm * mm + em * em);
            } else {
                Sp[n + 1] = -mm;
                if (FRO) fro += ee * ee + mm * mm + 2.0f * me * me;
            }
        };
        if (mt == 0) {
            const ff dA = hi(F(SWF_A, xx)), dB = hi(F(SWF_B, xx));
            for (int y = y0; y <= min(y1, x) && x <= ldim; y++, Sp += 2 * (size_t)n) {
                const float4 yE = F(SWF_E, y);
                const ff z{0.0f, 0.0f};
                const ff a = ff_mul(dA, hi(F(SWF_A, y))), bb = ff_mul(dB, hi(F(SWF_B, y)));
                store(y, sw_out(ff_dot3(a, TV(1, 1, y), z, z, z, z), eA + __float_as_int(yE.x), bad),
                      sw_out(-ff_dot3(bb, TV(0, 1, y), z, z, z, z), eB + __float_as_int(yE.y), bad), 0.0f, 0.0f);
            }
        } else {
            const float4 fUA = F(SWF_UA, xx), fUB = F(SWF_UB, xx);
            const ff UA = lo(fUA), VA = hi(fUA), UB = lo(fUB), VB = hi(fUB), mA = lo(F(SWF_A, xx)), mB = lo(F(SWF_B, xx));
            // of column v: dA(x) J_TM, dB(x) J_TE, m dB(x) T_TM, m dA(x) T_TE (mantissas)
            struct Col { ff JT, JE, mT, mE; };
            struct Raw { ff a, t, d, ea, e, ed; }; // T_TM and T_TE at x - 1, x, x + 1
            auto raw = [&](int v) { return Raw{TV(1, 0, v), TV(1, 1, v), TV(1, 2, v), TV(0, 0, v), TV(0, 1, v), TV(0, 2, v)}; };
            auto form = [&](const Raw &q) {
                return Col{ff_dot2(UA, q.a, VA, q.d), ff_dot2(UB, q.ea, VB, q.ed), ff_mul(mB, q.t), ff_mul(mA, q.e)};
            };
            // exponent of the largest of a column's values, from the magnitudes' bits
            auto top = [&](const Raw &q) {
                auto m = [](ff x) { return __float_as_int(x.h) & 0x7fffffff; };
                return (max(max(max(m(q.a), m(q.t)), max(m(q.d), m(q.ea))), max(m(q.e), m(q.ed))) >> 23) - 127;
            };
            Col cm{}, c0{};
            int em_ = top(raw(y0 - 1)), e0_ = top(raw(y0));
            bool have = false; // cm and c0 are formed (uniform over the warp)
            for (int y = y0; y <= y1; y++, Sp += 2 * (size_t)n) {
                const bool act = x <= ldim && y <= x;
                const float4 yE = F(SWF_E, y);
                const Raw qp = raw(y + 1);
                const int ep_ = top(qp);
                // five products of three factors, each below 2^(sum of exponents + 3)
                const bool zero = !FRO && y != x && exr + __float_as_int(yE.z) + max(max(em_, e0_), ep_) + 6 < -62;
                em_ = e0_;
                e0_ = ep_;
                if (__all_sync(0xffffffffu, !act || zero)) {
                    if (act) store(y, 0.0f, 0.0f, 0.0f, 0.0f);
                    have = false;
                    continue;
                }
                if (!have) {
                    cm = form(raw(y - 1));
                    c0 = form(raw(y));
                    have = true;
                }
                const Col cp = form(qp);
                // EE = dA dA [B_TM - m^2 T_TE], MM = dB dB [m^2 T_TM - B_TE], B(x, y) = Um(y) J(x, y-1) - Vp(y) J(x, y+1);
                // EM = m dA(x) dB(y) [H_TE - J_TM], ME = m dB(x) dA(y) [J_TE - H_TM], H(x, y) = Um(y) T(x, y-1) - Vp(y) T(x, y+1)
                const float4 gUA = F(SWF_UA, y), gUB = F(SWF_UB, y);
                const ff yUA = lo(gUA), yVA = hi(gUA), yUB = lo(gUB), yVB = hi(gUB), yA = lo(F(SWF_A, y)), yB = lo(F(SWF_B, y));
                const float ee = ff_dot3(yUA, cm.JT, yVA, cp.JT, ff_neg(yA), c0.mE);
                const float mm = -ff_dot3(yUB, cm.JE, yVB, cp.JE, ff_neg(yB), c0.mT);
                const float em = ff_dot3(yUB, cm.mE, yVB, cp.mE, ff_neg(yB), c0.JT);
                const float me = -ff_dot3(yUA, cm.mT, yVA, cp.mT, ff_neg(yA), c0.JE);
                const int fA = __float_as_int(yE.x), fB = __float_as_int(yE.y);
                bool wrong = false;
                const float oee = sw_out(ee, eA + fA, wrong), omm = sw_out(mm, eB + fB, wrong), oem = sw_out(em, eA + fB, wrong),
                            ome = sw_out(me, eB + fA, wrong);
                if (act) {
                    bad |= wrong;
                    store(y, oee, omm, oem, ome);
                }
                cm = c0;
                c0 = cp;
            }
        }
        if (__syncthreads_or(bad) && tid == 0) atomicOr(status + task, ST_ERR_NONFINITE);
    }
    if (FRO) { // per-block sums, added by the statistics kernel in order
        for (int o = 16; o > 0; o >>= 1) fro += __shfl_xor_sync(0xffffffffu, fro, o);
        if ((tid & 31) == 0) red[tid >> 5] = fro;
        __syncthreads();
        if (tid == 0) sums[((size_t)task * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = red[0] + red[1];
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
size_t seed_bytes(int ldim, int ntask) { return (size_t)ntask * 2 * SEED_KINDS * (ldim + 2) * sizeof(ffe); }

static size_t sweep_smem_bytes(int ldim) { return (size_t)RF_RING * (ldim + 2) * sizeof(float2); }

// windows up to this take the recurrence (its ring of rows fits in shared memory), larger ones the q-sums of every pair
constexpr int SWEEP_MAX = 7000;
bool sweep_fits(int ldim) { return ldim <= SWEEP_MAX; }
int sweep_nsum(int ldim) { return ((ldim + EL_X - 1) / EL_X) * ((ldim + EL_Y - 1) / EL_Y); }
size_t sweep_work_bytes(int ldim, int nlist)
{
    const size_t L = ldim + 2;
    return (size_t)nlist * L * (SWF_FIELDS * sizeof(float4) + 2 * L * sizeof(float2) + (recf_parts(ldim) - 1) * 4 * sizeof(ffe));
}
static ffe *sweep_rows(void *work, int ldim, int nlist)
{
    const size_t L = ldim + 2;
    return (ffe *)((char *)work + (size_t)nlist * L * (SWF_FIELDS * sizeof(float4) + 2 * L * sizeof(float2)));
}

void launch_seed_ff(const Task *tasks, const int *tlist, const int4 *groups, int ngroups, int ldim, const float4 *KP, const int *KPe,
                    int nu_stride, const float4 *ptabf, int pstride, const void *a12t, int ngroup_all, void *seed, bool band,
                    void *work, int nlist, int *status, cudaStream_t st)
{
    if (ngroups <= 0) return;
    const int L = ldim + 2;
    const A12L *tl = (const A12L *)a12t;
    const A12J *tj = (const A12J *)((const char *)a12t + (size_t)L * ngroup_all * sizeof(A12L));
    const int P = band ? 1 : recf_parts(ldim);
    dim3 g(2 * P * ((L + 127) / 128), ngroups);
    k_seed_ff<3><<<g, 128, 0, st>>>(tasks, tlist, groups, ngroups, ldim, KP, KPe, nu_stride, ptabf, pstride, tl, tj,
                                    band ? SEED_D0 : SEED_D1, band ? SEED_D2 : SEED_COL, (ffe *)seed, P, P > 1 ? sweep_rows(work, ldim, nlist) : nullptr,
                                    status, QSUM_FF_STOP_BITS);
    COUNT_LAUNCH(1);
    CK(cudaGetLastError());
}

void launch_sweep_ff(const Task *tasks, const int *tlist, int nlist, int ldim, const void *seed, const void *Saf, const void *Sbf,
                     void *work, float *S, size_t sstride, float *sums, int *status, cudaStream_t st)
{
    if (nlist <= 0) return;
    static size_t attr = 0;
    const size_t smem = sweep_smem_bytes(ldim), L = ldim + 2;
    if (smem > attr) {
        CK(cudaFuncSetAttribute(k_rec_ff, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr = smem;
    }
    float4 *tab = (float4 *)work;
    float2 *tt = (float2 *)(tab + nlist * SWF_FIELDS * L);
    k_sweep_tab<<<nlist, 256, 0, st>>>(tasks, tlist, nlist, ldim, (const ffe *)seed, (const ffe *)Saf, (const ffe *)Sbf, tab);
    const int P = recf_parts(ldim);
    k_rec_ff<<<nlist * P * 2, RF_NT, smem, st>>>(tasks, tlist, nlist, ldim, P, sweep_rows(work, ldim, nlist), tab, tt, status);
    const dim3 g((ldim + EL_X - 1) / EL_X, (ldim + EL_Y - 1) / EL_Y, nlist);
    if (sums) k_elem_sweep<true><<<g, EL_X, 0, st>>>(tasks, tlist, nlist, ldim, tt, tab, S, sstride, sums, status);
    else k_elem_sweep<false><<<g, EL_X, 0, st>>>(tasks, tlist, nlist, ldim, tt, tab, S, sstride, nullptr, status);
    COUNT_LAUNCH(3);
    CK(cudaGetLastError());
}

} // namespace capsgpu
