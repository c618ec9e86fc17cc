// sweep64.cu -- the FP64 form's round-trip matrix from a few q-sums per row and the three-term
// recurrence of the I integrals, straight into the fixed-point matrix 1 - M.
//
// The recurrence, its scaling T(w1, w2) = I(w1, w2) 2^{k(w1) + k(w2)} and the element formulas are
// those of sweep.cu, here in FP64: the q-sum of every pair costs O(ldim^3) per matrix, the
// recurrence O(1) per pair from q-sums on the diagonal, the first subdiagonal and the first
// column.  The recurrence links values of one accuracy by positive coefficients of order one,
// moving away from the diagonal; against q-sums of every pair log det changes by 1e-13 relative
// at most (tests/test_gpu_sweep64.py), the size of the q-sums' own rounding.
//
// Two kernels behind the seeds and a table of coefficients, both bound by the FP64 pipe (two operations per clock and
// SM).  k_rec64 fills the table T row by row, 4 operations per entry and polarisation, one CTA per
// matrix, range of rows and polarisation: a range but the first starts from the q-sums of two whole
// rows, and the number of ranges depends on ldim alone, so that a matrix has the same value in every
// batch.  k_elem64 forms the elements of all pairs at once: the row factors dA, dB are folded into the
// coefficients of their row (J' = dA J costs what J does) and the column factors into tables, 18 operations for
// the four elements of a pair; conversion to fixed point is integer work.  For a perfectly
// reflecting plate T_TE = -T_TM, and only T_TM is formed.
#include "fix.cuh"
#include "internal.h"
#include "qsum64.cuh"

namespace capsgpu {

// window index of the first l with I != 0: l = max(lmin - 1, m')
CAPS_DEV int col64(const Task &T)
{
    const int mm = T.m > 0 ? T.m : 1;
    return T.lmin - 1 >= mm ? 0 : 1;
}

// ranges of rows of T: part q of P forms rows (row(q), row(q + 1)], row(0) = -1, of about equal
// numbers of pairs; parts q >= 1 start from the q-sums of rows row(q) - 1 and row(q)
__host__ __device__ inline int rec64_row(int q, int P, int L) { return q <= 0 ? -1 : q >= P ? L - 1 : (int)(L * sqrt((double)q / P)); }
// A part of 512 rows takes 0.25 ms at row 512 and 1 ms at row 2048 of a matrix; its two rows of
// q-sums cost about as much as 100 rows
__host__ __device__ inline int rec64_parts(int ldim) { return ldim < 1024 ? 1 : ldim / 512; }

// ---------------------------------------------------------------------------
// seeds
// ---------------------------------------------------------------------------
// seed[((task * 2 + pol) * SEED_KINDS + kind) * L + w]: the pair (w, w), (w+1, w), (w+2, w) or (w, c);
// rows[(((b * (P - 1) + q - 1) * 2 + i) * 2 + pol) * L + y]: row(q) - 1 + i of listed task b, y <= row
// grid (ceil(L / 32) * (2 + 2 (P - 1)), nlist), one pair per thread; kind0 and kind1 first.  One warp per CTA: a
// step of the q recurrence takes about 20 FP64 operations, 16 clocks of the SM's pipe each and warp, so that the
// warps of one CTA would wait for each other while other SMs have none (free energy at R/L = 20: four warps per
// CTA 0.68 ms, one 0.55; R/L = 100 3.18 and 3.05)
constexpr int SEED_NT = 32;
__global__ void __launch_bounds__(SEED_NT) k_seed64(const Task *tasks, const int *tlist, int nlist, int ldim, int P, int kind0, int kind1,
                                                const sd *__restrict__ K, int nu_stride, const double *__restrict__ lft,
                                                const double4 *__restrict__ ptab, int pstride, sd *seed, sd *rows, int *status)
{
    const int L = ldim + 2, nbw = (L + SEED_NT - 1) / SEED_NT;
    if ((int)blockIdx.y >= nlist) return;
    const int task = tlist ? tlist[blockIdx.y] : (int)blockIdx.y;
    const Task &T = tasks[task];
    const int part = blockIdx.x / nbw, w = ((int)blockIdx.x % nbw) * SEED_NT + threadIdx.x;
    if (w >= L) return;
    int a1 = w, a2 = w;
    sd *oT, *oE;
    if (part < 2) {
        const int kind = part ? kind1 : kind0;
        if (kind == SEED_D1) a1 = w + 1;
        else if (kind == SEED_D2) a1 = w + 2;
        else if (kind == SEED_COL) a2 = col64(T);
        oT = seed + ((size_t)(task * 2 + 1) * SEED_KINDS + kind) * L + w;
        oE = seed + ((size_t)(task * 2 + 0) * SEED_KINDS + kind) * L + w;
    } else {
        const int q = (part - 2) / 2 + 1, i = (part - 2) & 1;
        a1 = rec64_row(q, P, L) - 1 + i;
        const size_t o = ((((size_t)blockIdx.y * (P - 1) + q - 1) * 2 + i) * 2) * L + w;
        oT = rows + o + L;
        oE = rows + o;
    }
    if (a1 >= L || a1 < a2) return; // outside the triangle: nothing reads it
    const int mm = T.m > 0 ? T.m : 1, l1 = T.lmin - 1 + a1, l2 = T.lmin - 1 + a2;
    if (l2 < mm || l2 < T.m || l1 < 1) { // I = 0 for l < m (integration.c:631)
        *oT = *oE = sd{0, 0};
        return;
    }
    sd rT, rE;
    if (qsum_pair(T, l1, l2, a012_pair(T.m, T.lmin, a1, a2, lft), K + (size_t)(task * 2 + 1) * nu_stride - T.mu,
                  K + (size_t)(task * 2 + 0) * nu_stride - T.mu, ptab + (size_t)task * 2 * pstride, pstride, rT, rE))
        atomicOr(status + task, ST_ERR_NONFINITE);
    *oT = rT;
    *oE = rE;
}

// M_ii alone, from the band seeds (the arithmetic of the full assembly); grid (ceil(ldim / 128), ntask)
__global__ void k_diag64(const Task *tasks, int ntask, int ldim, const sd *__restrict__ seed, const sd *Sa, const sd *Sb, const double2 *uv,
                         double *mdiag, int *status)
{
    const int L = ldim + 2, a = blockIdx.x * blockDim.x + threadIdx.x, task = blockIdx.y;
    if (a >= ldim || task >= ntask) return;
    const Task &T = tasks[task];
    const size_t so = (size_t)task * L + a + 1;
    auto Iv = [&](int p, int x, int y) { // the diagonal block reads I at |x - y| in {0, 2} only
        return seed[((size_t)(task * 2 + p) * SEED_KINDS + (x == y ? SEED_D0 : SEED_D2)) * L + min(x, y)];
    };
    sd EE, MM, EM, ME;
    elem_block<true>(T.m, a + 1, a + 1, Sa[so], Sa[so], Sb[so], Sb[so], uv[so], uv[so], Iv, EE, MM, EM, ME);
    const double ee = sd_to_double(EE), mm = sd_to_double(MM);
    if (!isfinite(ee) || !isfinite(mm)) atomicOr(status + task, ST_ERR_NONFINITE);
    mdiag[(size_t)task * 2 * ldim + 2 * a] = ee;
    mdiag[(size_t)task * 2 * ldim + 2 * a + 1] = mm;
}

// ---------------------------------------------------------------------------
// per-window tables
// ---------------------------------------------------------------------------
// per listed task and window index: Cp, Cm of the recurrence; R1 = 1 / Cp(w - 1), R2 = -Cm(w - 1) R1
// of row w; UA = Um dA, VA = -Vp dA, A = m dA and the same with dB; dA, dB; the largest of the six; the scaled seeds of row w:
// T(w, w), T(w, w - 1), T(w, c), TE and TM each.  tab[(b * W_FIELDS + field) * L + w], so that consecutive lanes read
// consecutive entries
enum { W_CP, W_CM, W_R1, W_R2, W_UA, W_VA, W_A, W_UB, W_VB, W_B, W_DA, W_DB, W_MX, W_SEED, W_FIELDS = W_SEED + 7 }; // even

// m 2^e as a double; below the normal range 0, above it infinite
CAPS_DEV double sd_scaled(sd v, int k)
{
    if (v.m == 0.0 || v.e + k < -1000) return 0.0;
    if (v.e + k > 1000) return INFINITY;
    return shift2(v.m, v.e + k);
}
// k(w): I_TM(w, w) 2^{2k} in [1, 4); below the first column that column's
CAPS_DEV int k64(const sd *__restrict__ d0tm, int w, int c)
{
    const sd v = d0tm[w < c ? c : w];
    return v.m == 0.0 ? 0 : -(v.e >> 1);
}

// grid nlist, 256 threads; also the matrix's scale exponent (see k_fix_convert)
__global__ void __launch_bounds__(256) k_sweep64_tab(const Task *tasks, const int *tlist, int nlist, int ldim, const sd *__restrict__ seed,
                                                     const sd *__restrict__ Sa, const sd *__restrict__ Sb, double *tab, int *ktab)
{
    const int L = ldim + 2;
    if ((int)blockIdx.x >= nlist) return;
    const int task = tlist ? tlist[blockIdx.x] : (int)blockIdx.x;
    const Task &T = tasks[task];
    const int c = col64(T), mm = T.m > 0 ? T.m : 1, lm1 = T.lmin - 1;
    const sd *d0 = seed + ((size_t)(task * 2 + 1) * SEED_KINDS + SEED_D0) * L;
    for (int w = threadIdx.x; w < L; w += blockDim.x) {
        const int kw = k64(d0, w, c), l = lm1 + w;
        auto CP = [&](int v, int kv) { // Cp(v), k(v) = kv
            return v >= c && v + 1 < L ? (double)(lm1 + v - mm + 1) / (2.0 * (lm1 + v) + 1) * pow2i(max(min(kv - k64(d0, v + 1, c), 1000), -1000)) : 0.0;
        };
        auto CM = [&](int v, int kv) {
            return v >= c + 1 ? (double)(lm1 + v + mm) / (2.0 * (lm1 + v) + 1) * pow2i(max(min(kv - k64(d0, v - 1, c), 1000), -1000)) : 0.0;
        };
        double *t = tab + (size_t)blockIdx.x * W_FIELDS * L + w;
        const double cp = CP(w, kw), cm = CM(w, kw);
        double r1 = 0.0, r2 = 0.0;
        if (w >= c + 1) {
            const int k1 = k64(d0, w - 1, c);
            const double p = CP(w - 1, k1);
            if (p != 0.0) {
                r1 = 1.0 / p;
                r2 = -CM(w - 1, k1) / p;
            }
        }
        const double um = (l + 1.0) * cm, vp = l * cp, m = T.m;
        const double dA = sd_scaled(Sa[(size_t)task * L + w], -kw), dB = sd_scaled(Sb[(size_t)task * L + w], -kw);
        double f[W_FIELDS] = {cp, cm, r1, r2, um * dA, -vp * dA, m * dA, um * dB, -vp * dB, m * dB, dA, dB};
        int top = 0; // by the high words, so that a NaN is largest
#pragma unroll
        for (int i = W_UA; i <= W_B; i++) top = max(top, __double2hiint(f[i]) & 0x7fffffff);
        f[W_MX] = __hiloint2double(top, 0);
#pragma unroll
        for (int pol = 0; pol < 2; pol++) {
            const sd *sp = seed + (size_t)(task * 2 + pol) * SEED_KINDS * L;
            f[W_SEED + pol] = w >= c ? sd_scaled(sp[SEED_D0 * L + w], 2 * kw) : 0.0;
            f[W_SEED + 2 + pol] = w > c ? sd_scaled(sp[SEED_D1 * L + w - 1], kw + k64(d0, w - 1, c)) : 0.0;
            f[W_SEED + 4 + pol] = w >= c ? sd_scaled(sp[SEED_COL * L + w], kw + k64(d0, c, c)) : 0.0;
        }
#pragma unroll
        for (int i = 0; i < W_FIELDS; i++) t[(size_t)i * L] = f[i];
        ktab[(size_t)blockIdx.x * L + w] = kw;
    }
}

// ---------------------------------------------------------------------------
// the table
// ---------------------------------------------------------------------------
// T(r, y), y <= r, of listed task b at tt[((b * 2 + pol) * L + y) * L + r] (column y of the triangle
// contiguous, the order in which k_elem64 reads it)
constexpr int R64_NT = 256, R64_RING = 4;

// grid nlist * P * 2: one polarisation (TE, TM) per CTA, none for the TE of a perfect reflector.  The ring of
// four rows (L + 2 values each) is in shared memory, or in global memory (ring != nullptr) where it does
// not fit; one barrier per row.  Rows are a serial chain, so nothing but the ring, three dependent FP64
// operations and the barrier stands in it: a thread keeps the coefficients of its first columns in
// registers, and the next row's seeds and factors are loaded a row ahead (with all of them loaded in
// the row, 2 us a row).  Both polarisations in one CTA hold one SM's FP64 pipe for 2800 clocks per
// row of 700 columns while others have no matrix (24 matrices of ldim 1050 0.98 ms, one polarisation per CTA 0.52;
// 4 of ldim 2500 2.4 and 1.3).  A row of ldim 140 takes 0.45 us.
constexpr int R64_KEEP = 3; // columns per thread with coefficients in registers
__global__ void __launch_bounds__(R64_NT) k_rec64(const Task *tasks, const int *tlist, int nlist, int ldim, int P,
                                                  const sd *__restrict__ rows, const double *__restrict__ tab,
                                                  const int *__restrict__ ktab, double *tt, const int *status, double *ring)
{
    extern __shared__ __align__(16) double r64_sm[];
    const int L = ldim + 2, LP = L + 2;
    const int pol = blockIdx.x & 1, part = blockIdx.x >> 1, b = part / P, q = P - 1 - part % P;
    if (b >= nlist) return;
    const int task = tlist ? tlist[b] : b;
    if (status[task] & ~0xF) return; // no status changes in this launch: uniform
    const Task &T = tasks[task];
    if (T.is_pr && pol == 0) return;
    const int c = col64(T), r1 = rec64_row(q + 1, P, L);
    double *R = ring ? ring + (size_t)blockIdx.x * R64_RING * LP : r64_sm;
    auto rowp = [&](int r) { return R + (size_t)(r & 3) * LP; };
    const double *W = tab + (size_t)b * W_FIELDS * L;
    auto F = [&](int f, int w) { return __ldg(W + (size_t)f * L + w); };
    const int *kt = ktab + (size_t)b * L;
    double *t = tt + ((size_t)b * 2 + pol) * L * L;
    const int tid = threadIdx.x;
    int r = 0;
    if (q > 0) { // the two rows before the range, from their q-sums
        r = rec64_row(q, P, L) + 1;
        for (int i = 0; i < 2; i++) {
            const int rr = r - 2 + i;
            const sd *src = rows + ((((size_t)b * (P - 1) + q - 1) * 2 + i) * 2 + pol) * L;
            double *D = rowp(rr);
            for (int y = tid; y <= rr; y += R64_NT) D[y] = y < c ? 0.0 : sd_scaled(src[y], kt[rr] + kt[y]);
        }
        __syncthreads();
    }
    __shared__ double ahead[2][5]; // of the next row: its seeds (W_SEED ..), R1, R2
    auto fetch = [&](int row) {
        if (tid < 5 && row < L) ahead[row & 1][tid] = F(tid < 3 ? W_SEED + 2 * tid + pol : W_R1 + tid - 3, row);
    };
    double cp[R64_KEEP], cm[R64_KEEP];
#pragma unroll
    for (int i = 0; i < R64_KEEP; i++) {
        const int y = tid + i * R64_NT;
        cp[i] = y < L ? F(W_CP, y) : 0.0;
        cm[i] = y < L ? F(W_CM, y) : 0.0;
    }
    fetch(r);
    __syncthreads();
    for (; r <= r1; r++) {
        fetch(r + 1);
        double *D = rowp(r);
        // rows before the first are never read: y >= c + 1 and y <= r - 2 need r >= 3
        const double *P1 = rowp(r + 3), *P2 = rowp(r + 2); // rows r - 1, r - 2
        const double *sr = ahead[r & 1];
        const double R1 = sr[3], R2 = sr[4];
        auto column = [&](int y, double Cp, double Cm) {
            double v = 0.0;
            if (y >= c) {
                if (y == r || y == r - 1 || y == c) v = sr[y == r ? 0 : y == r - 1 ? 1 : 2];
                else v = fma(R1, fma(Cp, P1[y + 1], Cm * P1[y - 1]), R2 * P2[y]);
            }
            D[y] = v;
            t[(size_t)y * L + r] = v;
        };
#pragma unroll
        for (int i = 0; i < R64_KEEP; i++)
            if (tid + i * R64_NT <= r) column(tid + i * R64_NT, cp[i], cm[i]);
        for (int y = tid + R64_KEEP * R64_NT; y <= r; y += R64_NT) column(y, F(W_CP, y), F(W_CM, y));
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// elements
// ---------------------------------------------------------------------------
// grid (ceil(ldim / E64_X), ceil(ldim / ny), nlist), E64_X threads: thread x (window index 1 ..
// ldim, a row of 2x2 blocks) walks ny columns y <= x with T and J of the columns y - 1, y, y + 1 in
// registers; consecutive threads write consecutive rows of the column-major matrix.
//
// Bound by the FP64 pipe: 18 operations per pair.  Far from the diagonal T is so small that all four
// elements round to zero (a third of the pairs of a free energy's matrices at R/L = 50); a warp whose pairs all
// do, by the exponents of T and of the largest factors, stores zeros and forms nothing: 441 matrices of ldim 700
// 5.0 ms with every element formed and 20 operations, 3.1 so; 24 of ldim 1050 0.62 and 0.34.  Where
// the sums of squares are wanted, too, every element is formed.
constexpr int E64_X = 64, E64_Y = 16;
template <bool FRO>
__global__ void __launch_bounds__(E64_X) k_elem64(const Task *tasks, const int *tlist, int nlist, int ldim, int ny, const double *__restrict__ tt,
                                                  const double *__restrict__ tab, const double *__restrict__ mdiag, const int *info,
                                                  long long *A, size_t mstride, double *fro_out, int *status)
{
    const int L = ldim + 2, n = 2 * ldim;
    const int b = blockIdx.z;
    if (b >= nlist) return;
    const int task = tlist ? tlist[b] : b;
    const int x = blockIdx.x * E64_X + threadIdx.x + 1, y0 = blockIdx.y * ny + 1;
    double fro = 0.0;
    if (y0 <= min((int)(blockIdx.x + 1) * E64_X, ldim)) { // uniform: some thread of the block has y0 <= x
        int err = 0;
        const Task &T = tasks[task];
        const int mt = T.m;
        const bool pr = T.is_pr;
        const double *W = tab + (size_t)b * W_FIELDS * L;
        auto F = [&](int f, int w) { return __ldg(W + (size_t)f * L + w); };
        const double *tE = tt + (size_t)b * 2 * L * L, *tT = tE + (size_t)L * L;
        const int xx = min(x, ldim); // lanes past the end repeat the last row's loads
        // T(u, v) for any order of u and v
        auto TV = [&](const double *t, int u, int v) { return u >= v ? t[(size_t)v * L + u] : t[(size_t)u * L + v]; };
        const int fq = 60 - info[2 * task];
        const long long one = fq >= 0 ? 1LL << fq : 0;
        long long *Am = A + (size_t)task * mstride + (size_t)2 * (y0 - 1) * n + 2 * (x - 1);
        auto store = [&](int y, double ee, double mm, double em, double me) {
            if (y != x) {
                *reinterpret_cast<longlong2 *>(Am) = make_longlong2(-to_fix(ee, fq, err), -to_fix(me, fq, err));
                *reinterpret_cast<longlong2 *>(Am + n) = make_longlong2(-to_fix(em, fq, err), -to_fix(mm, fq, err));
                if (FRO) fro += 2.0 * (fma(ee, ee, me * me) + fma(mm, mm, em * em));
            } else {
                // the diagonal from M_ii, which the trace is taken from too
                const double dee = mdiag[(size_t)task * n + 2 * (x - 1)], dmm = mdiag[(size_t)task * n + 2 * (x - 1) + 1];
                *reinterpret_cast<longlong2 *>(Am) = make_longlong2(one - to_fix(dee, fq, err), -to_fix(me, fq, err));
                Am[n + 1] = one - to_fix(dmm, fq, err);
                if (FRO) fro += fma(dee, dee, dmm * dmm) + 2.0 * me * me;
            }
        };
        const int y1 = min(y0 + ny - 1, ldim); // uniform; lanes with x < y are idle
        if (mt == 0) {
            const double dA = F(W_DA, xx), dB = F(W_DB, xx);
            for (int y = y0; y <= min(y1, x); y++, Am += 2 * (size_t)n) {
                if (x > ldim) break;
                const double t = tT[(size_t)y * L + xx], e = pr ? -t : tE[(size_t)y * L + xx];
                store(y, dA * F(W_DA, y) * t, -(dB * F(W_DB, y) * e), 0.0, 0.0);
            }
        } else {
            const double mA = F(W_A, xx), mB = F(W_B, xx);
            const double UxA = F(W_UA, xx), VxA = F(W_VA, xx), UxB = F(W_UB, xx), VxB = F(W_VB, xx);
            // of column v, with J(x, v) = Um(x) T(x-1, v) - Vp(x) T(x+1, v): J'_TM = dA(x) J_TM, J'_TE = dB(x) J_TE, m dB(x) T_TM and
            // m dA(x) T_TE
            struct Col { double JT, JE, mT, mE; };
            struct Raw { double a, t, d, ea, e, ed; };
            auto raw = [&](int v) {
                Raw q{TV(tT, xx - 1, v), TV(tT, xx, v), TV(tT, xx + 1, v), 0.0, 0.0, 0.0};
                if (!pr) {
                    q.ea = TV(tE, xx - 1, v);
                    q.e = TV(tE, xx, v);
                    q.ed = TV(tE, xx + 1, v);
                }
                return q;
            };
            auto form = [&](const Raw &q) {
                Col r;
                r.JT = fma(UxA, q.a, VxA * q.d);
                r.mT = mB * q.t;
                if (pr) {
                    r.JE = -fma(UxB, q.a, VxB * q.d);
                    r.mE = -(mA * q.t);
                } else {
                    r.JE = fma(UxB, q.ea, VxB * q.ed);
                    r.mE = mA * q.e;
                }
                return r;
            };
            // biased exponents: of the largest of a column's values (0: all zero)
            auto ex = [](double v) { return __double2hiint(v) >> 20 & 0x7ff; };
            auto top = [&](const Raw &q) { return max(max(max(ex(q.a), ex(q.t)), max(ex(q.d), ex(q.ea))), max(ex(q.e), ex(q.ed))); };
            const int exr = ex(F(W_MX, xx));
            Raw qm = raw(y0 - 1), q0 = raw(y0);
            Col cm{}, c0{};
            int em = top(qm), e0 = top(q0);
            bool have = false; // cm and c0 are formed (uniform over the warp)
            Raw next = raw(y0 + 1);
            for (int y = y0; y <= y1; y++, Am += 2 * (size_t)n) {
                const Raw qp = next;
                next = raw(min(y + 2, ldim + 1)); // a column ahead, for where few warps hide the loads
                const int ep = top(qp);
                const bool act = x <= ldim && y <= x;
                // five products of three factors, each below 2^(sum of exponents + 3): zero below half a unit of 2^-fq
                const bool zero = !FRO && y != x && exr + ex(F(W_MX, y)) + max(max(em, e0), ep) - 3 * 1023 + 6 + fq < -1;
                if (__all_sync(0xffffffffu, !act || zero)) {
                    if (act) {
                        *reinterpret_cast<longlong2 *>(Am) = make_longlong2(0, 0);
                        *reinterpret_cast<longlong2 *>(Am + n) = make_longlong2(0, 0);
                    }
                    have = false;
                } else {
                    if (!have) {
                        if (y > y0) { // (rare: the values were dropped)
                            qm = raw(y - 1);
                            q0 = raw(y);
                        }
                        cm = form(qm);
                        c0 = form(q0);
                        have = true;
                    }
                    const Col cp = form(qp);
                    // EE = dA dA [B_TM - m^2 T_TE], MM = dB dB [m^2 T_TM - B_TE], B(x, y) = Um(y) J(x, y-1) - Vp(y) J(x, y+1)
                    // EM = m dA(x) dB(y) [H_TE - J_TM], ME = m dB(x) dA(y) [J_TE - H_TM], H(x, y) = Um(y) T(x, y-1) - Vp(y) T(x, y+1)
                    const double yUA = F(W_UA, y), yVA = F(W_VA, y), yA = F(W_A, y), yUB = F(W_UB, y), yVB = F(W_VB, y), yB = F(W_B, y);
                    const double ee = fma(yUA, cm.JT, fma(yVA, cp.JT, -(yA * c0.mE)));
                    const double mm = fma(yB, c0.mT, -fma(yUB, cm.JE, yVB * cp.JE));
                    const double me2 = fma(yUA, cm.mT, yVA * cp.mT);
                    const double eem = fma(yUB, cm.mE, fma(yVB, cp.mE, -(yB * c0.JT))), mee = fma(yA, c0.JE, -me2);
                    if (act) store(y, ee, mm, eem, mee);
                    cm = c0;
                    c0 = cp;
                }
                em = e0;
                e0 = ep;
            }
        }
        if (err) atomicOr(status + task, err);
    }
    if (FRO) { // per-block sums, added by the statistics kernel in order
        __shared__ double red[E64_X / 32];
        for (int o = 16; o > 0; o >>= 1) fro += __shfl_xor_sync(0xffffffffu, fro, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = fro;
        __syncthreads();
        if (threadIdx.x == 0) fro_out[((size_t)task * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = red[0] + red[1];
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static size_t r64_ring_bytes(int ldim) { return (size_t)R64_RING * (ldim + 4) * sizeof(double); }
static bool r64_ring_fits(int ldim) { return r64_ring_bytes(ldim) <= 220 * 1024; }

size_t seed64_bytes(int ldim, int ntask) { return (size_t)ntask * 2 * SEED_KINDS * (ldim + 2) * sizeof(sd); }

int sweep64_nfro(int ldim) { return ((ldim + E64_X - 1) / E64_X) * ((ldim + E64_Y - 1) / E64_Y); }

// T, the column tables, rows of q-sums, k, the ring
size_t sweep64_work_bytes(int ldim, int nlist)
{
    const size_t L = ldim + 2, P = rec64_parts(ldim);
    size_t b = (size_t)nlist * L * (2 * L * sizeof(double) + W_FIELDS * sizeof(double) + (P - 1) * 4 * sizeof(sd) + sizeof(int)) + 512;
    if (!r64_ring_fits(ldim)) b += (size_t)nlist * P * 2 * r64_ring_bytes(ldim);
    return b;
}

static void seed64(const Task *tasks, const int *tlist, int nlist, int ldim, int P, int k0, int k1, const sd *K, int nu_stride,
                   const double *lft, const double4 *ptab, int pstride, void *seed, sd *rows, int *status, cudaStream_t st)
{
    const int nbw = (ldim + 2 + SEED_NT - 1) / SEED_NT;
    k_seed64<<<dim3(nbw * (2 + 2 * (P - 1)), nlist), SEED_NT, 0, st>>>(tasks, tlist, nlist, ldim, P, k0, k1, K, nu_stride, lft, ptab, pstride,
                                                                  (sd *)seed, rows, status);
    COUNT_LAUNCH(1);
}

void launch_diag64(const Task *tasks, int ntask, int ldim, const sd *K, int nu_stride, const double *lft, const double4 *ptab, int pstride,
                   const sd *Sa, const sd *Sb, const double2 *uv, void *seed, double *mdiag, int *status, cudaStream_t st)
{
    seed64(tasks, nullptr, ntask, ldim, 1, SEED_D0, SEED_D2, K, nu_stride, lft, ptab, pstride, seed, nullptr, status, st);
    k_diag64<<<dim3((ldim + 127) / 128, ntask), 128, 0, st>>>(tasks, ntask, ldim, (const sd *)seed, Sa, Sb, uv, mdiag, status);
    COUNT_LAUNCH(1);
    CK(cudaGetLastError());
}

void launch_sweep64(const Task *tasks, const int *tlist, int nlist, int ldim, const sd *K, int nu_stride, const double *lft,
                    const double4 *ptab, int pstride, const sd *Sa, const sd *Sb, void *seed, const double *mdiag, const int *info,
                    void *work, long long *A, size_t mstride, double *fro, int *status, cudaStream_t st)
{
    if (nlist <= 0) return;
    const size_t L = ldim + 2;
    const int P = rec64_parts(ldim);
    double *tt = (double *)work, *tab = tt + (size_t)nlist * 2 * L * L; // 16-byte multiples: W_FIELDS is even
    sd *rows = (sd *)(tab + nlist * W_FIELDS * L);
    int *kt = (int *)(rows + (size_t)nlist * (P - 1) * 4 * L);
    const size_t ring_off = ((char *)(kt + nlist * L) - (char *)work + 255) & ~(size_t)255;
    const bool fits = r64_ring_fits(ldim);
    double *ring = fits ? nullptr : (double *)((char *)work + ring_off);
    const size_t sm = fits ? r64_ring_bytes(ldim) : 0;
    static size_t attr = 0;
    if (sm > attr) {
        CK(cudaFuncSetAttribute(k_rec64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        attr = sm;
    }
    seed64(tasks, tlist, nlist, ldim, P, SEED_D1, SEED_COL, K, nu_stride, lft, ptab, pstride, seed, rows, status, st);
    k_sweep64_tab<<<nlist, 256, 0, st>>>(tasks, tlist, nlist, ldim, (const sd *)seed, Sa, Sb, tab, kt);
    k_rec64<<<nlist * P * 2, R64_NT, sm, st>>>(tasks, tlist, nlist, ldim, P, rows, tab, kt, tt, status, ring);
    // A step to the next column is a chain of loads and 18 operations, 1200 clocks: 4 columns where 16 leave SMs
    // without a CTA (one matrix of ldim 140 24 us with 16, 9 with 4), elsewhere 4 would be one in twelve more operations
    // (32 of ldim 350: 93 us).  The elements are the same bits, the sums of squares come in the order of E64_Y.
    const int nx = (ldim + E64_X - 1) / E64_X;
    const int ny = !fro && (long long)nx * ((ldim + E64_Y - 1) / E64_Y) * nlist < device_sms() ? 4 : E64_Y;
    const dim3 g(nx, (ldim + ny - 1) / ny, nlist);
    if (fro) k_elem64<true><<<g, E64_X, 0, st>>>(tasks, tlist, nlist, ldim, ny, tt, tab, mdiag, info, A, mstride, fro, status);
    else k_elem64<false><<<g, E64_X, 0, st>>>(tasks, tlist, nlist, ldim, ny, tt, tab, mdiag, info, A, mstride, fro, status);
    COUNT_LAUNCH(3);
    CK(cudaGetLastError());
}

} // namespace capsgpu
