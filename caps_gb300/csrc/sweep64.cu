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
// One CTA takes a range of rows of one matrix.  Where a batch has fewer matrices than the
// chip has SMs, the rows are split over P CTAs of about equal numbers of pairs; each but the first
// starts from the q-sums of two whole rows (ldim more q-sums per CTA).
//
// What bounds it: the FP64 pipe, two operations per clock and SM.  The row factors dA, dB of
// the elements are folded into the coefficients of their row (J' = dA J costs what J does) and
// the column factors into tables, so that a pair takes 8 operations in the recurrence and 20 in
// its four elements; conversion to fixed point is integer work.
#include "common.cuh"
#include "internal.h"
#include "qsum64.cuh"
#include "umma.cuh"

namespace capsgpu {

// window index of the first l with I != 0: l = max(lmin - 1, m')
CAPS_DEV int col64(const Task &T)
{
    const int mm = T.m > 0 ? T.m : 1;
    return T.lmin - 1 >= mm ? 0 : 1;
}

// first element row (1 .. ldim) of part q of P: equal numbers of pairs
__host__ __device__ inline int sweep64_row(int q, int P, int ldim)
{
    if (q <= 0) return 1;
    if (q >= P) return ldim + 1;
    const int x = 1 + (int)(ldim * sqrt((double)q / P));
    return x < 5 ? 5 : x;
}

// ---------------------------------------------------------------------------
// seeds
// ---------------------------------------------------------------------------
// seed[((task * 2 + pol) * SEED_KINDS + kind) * L + w]: the pair (w, w), (w+1, w), (w+2, w) or (w, c);
// rows[(((b * (P - 1) + q - 1) * 2 + i) * 2 + pol) * L + y]: T rows x_q - 1 + i of listed task b, y <= row
// grid (ceil(L / 128) * (2 + 2 (P - 1)), nlist), one pair per thread; kind0 and kind1 first
__global__ void __launch_bounds__(128) k_seed64(const Task *tasks, const int *tlist, int nlist, int ldim, int P, int kind0, int kind1,
                                                const sd *__restrict__ K, int nu_stride, const double *__restrict__ lft,
                                                const double4 *__restrict__ ptab, int pstride, sd *seed, sd *rows, int *status)
{
    const int L = ldim + 2, nbw = (L + 127) / 128;
    if ((int)blockIdx.y >= nlist) return;
    const int task = tlist ? tlist[blockIdx.y] : (int)blockIdx.y;
    const Task &T = tasks[task];
    const int part = blockIdx.x / nbw, w = ((int)blockIdx.x % nbw) * 128 + threadIdx.x;
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
        a1 = sweep64_row(q, P, ldim) - 1 + i;
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

// M_ii alone, from the band seeds (the arithmetic of k_elem<true>); grid (ceil(ldim / 128), ntask)
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
// of row w; UA = Um dA, VA = -Vp dA, A = m dA and the same with dB; dA, dB.  tab[(b * W_FIELDS + field) * L + w], so that consecutive lanes read
// consecutive entries
enum { W_CP, W_CM, W_R1, W_R2, W_UA, W_VA, W_A, W_UB, W_VB, W_B, W_DA, W_DB, W_FIELDS };

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
        const double f[W_FIELDS] = {cp, cm, r1, r2, um * dA, -vp * dA, m * dA, um * dB, -vp * dB, m * dB, dA, dB};
#pragma unroll
        for (int i = 0; i < W_FIELDS; i++) t[(size_t)i * L] = f[i];
        ktab[(size_t)blockIdx.x * L + w] = kw;
    }
}

// ---------------------------------------------------------------------------
// the sweep
// ---------------------------------------------------------------------------
constexpr int S64_NT = 256, S64_NW = S64_NT / 32, S64_CH = 30, S64_RING = 4;

// v in units of 2^-q, rounded, saturated at +-2^62 (integer work only)
CAPS_DEV long long to_fix(double v, int q, bool &bad)
{
    const long long b = __double_as_longlong(v);
    const int ex = (int)((b >> 52) & 0x7ff);
    bad |= ex == 0x7ff;
    const int sh = ex - 1075 + q;
    long long mnt = (b & 0xfffffffffffffLL) | (1LL << 52);
    if (sh >= 10) mnt = 1LL << 62;
    else if (sh >= 0) mnt <<= sh;
    else mnt = sh < -54 ? 0 : (mnt + (1LL << (-sh - 1))) >> -sh;
    return b < 0 ? -mnt : mnt;
}

// grid nlist * P.  The ring of four rows (TE then TM, L + 2 values each) is in shared memory, or
// in global memory (ring != nullptr) where it does not fit.  Row r of T, a barrier, the elements
// of row r - 1: 30 columns per pass of 32 lanes, J of the neighbours by shuffles.
template <bool FRO>
__global__ void __launch_bounds__(S64_NT) k_sweep64(const Task *tasks, const int *tlist, int nlist, int ldim, int P,
                                                    const sd *__restrict__ seed, const sd *__restrict__ rows, const double *__restrict__ tab,
                                                    const int *__restrict__ ktab, const double *__restrict__ mdiag, const int *info,
                                                    long long *A, size_t mstride, double *fro_out, int *status, double *ring)
{
    extern __shared__ __align__(16) double s64_sm[];
    const int L = ldim + 2, n = 2 * ldim, LP = L + 2;
    const int b = blockIdx.x / P, q = P - 1 - (int)blockIdx.x % P;
    if (b >= nlist) return;
    const int task = tlist ? tlist[b] : b;
    __shared__ int s_st;
    if (threadIdx.x == 0) s_st = status[task];
    __syncthreads();
    if (s_st & ~0xF) return;
    const Task &T = tasks[task];
    const int mt = T.m, c = col64(T);
    const int x0 = sweep64_row(q, P, ldim), x1 = sweep64_row(q + 1, P, ldim);
    double *R = ring ? ring + (size_t)blockIdx.x * S64_RING * 2 * LP : s64_sm;
    auto rowp = [&](int r) { return R + (size_t)((r & 3) * 2) * LP; };
    const double *W = tab + (size_t)b * W_FIELDS * L;
    auto F = [&](int f, int w) { return __ldg(W + (size_t)f * L + w); };
    const int *kt = ktab + (size_t)b * L;
    auto sp = [&](int pol, int kind) { return seed + ((size_t)(task * 2 + pol) * SEED_KINDS + kind) * L; };
    const int fq = 60 - info[2 * task];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    long long *Am = A + (size_t)task * mstride;
    const double *md = mdiag + (size_t)task * n;
    bool bad = false;
    double fro = 0.0;
    int r = 0;
    if (q > 0) { // rows x0 - 1 and x0 from their q-sums
        for (int i = 0; i < 2; i++) {
            const int rr = x0 - 1 + i;
            const sd *src = rows + ((((size_t)b * (P - 1) + q - 1) * 2 + i) * 2) * L;
            double *D = rowp(rr), *D1 = rowp(rr - 1);
            for (int y = tid; y <= rr; y += S64_NT) {
                const int k = kt[rr] + kt[y];
                const double vE = y < c ? 0.0 : sd_scaled(src[y], k), vT = y < c ? 0.0 : sd_scaled(src[L + y], k);
                D[y] = vE;
                D[LP + y] = vT;
                if (i == 1 && y == rr - 1) { D1[rr] = vE; D1[LP + rr] = vT; }
            }
        }
        r = x0 + 1;
        __syncthreads();
    }
    for (; r <= x1 && r < L; r++) {
        double *D = rowp(r);
        // rows before the first are never read: y >= c + 1 and y <= r - 2 need r >= 3
        double *P1 = rowp(r + 3), *P2 = rowp(r + 2); // rows r - 1, r - 2
        const double R1 = F(W_R1, r), R2 = F(W_R2, r);
        for (int y = tid; y <= r; y += S64_NT) {
            double vE = 0.0, vT = 0.0;
            if (y >= c) {
                if (y == r || y == r - 1 || y == c) {
                    const int kind = y == r ? SEED_D0 : (y == r - 1 ? SEED_D1 : SEED_COL), wi = kind == SEED_COL ? r : y;
                    const int k = kt[r] + kt[y];
                    vE = sd_scaled(sp(0, kind)[wi], k);
                    vT = sd_scaled(sp(1, kind)[wi], k);
                } else {
                    const double Cp = F(W_CP, y), Cm = F(W_CM, y);
                    vE = fma(R1, fma(Cp, P1[y + 1], Cm * P1[y - 1]), R2 * P2[y]);
                    vT = fma(R1, fma(Cp, P1[LP + y + 1], Cm * P1[LP + y - 1]), R2 * P2[LP + y]);
                }
            }
            D[y] = vE;
            D[LP + y] = vT;
            // T(r, r-1) and T(r, r-2) past the diagonals of rows r-1 and r-2
            if (y == r - 1) { P1[r] = vE; P1[LP + r] = vT; }
            if (y == r - 2) { P2[r] = vE; P2[LP + r] = vT; }
        }
        __syncthreads();
        const int x = r - 1;
        if (x < x0) continue; // uniform
        const double *Rm = rowp(x + 3), *R0 = rowp(x), *Rp = rowp(x + 1);
        const double dA = F(W_DA, x), dB = F(W_DB, x), mA = F(W_A, x), mB = F(W_B, x);
        const double UxA = F(W_UA, x), VxA = F(W_VA, x), UxB = F(W_UB, x), VxB = F(W_VB, x);
        const int r0 = 2 * (x - 1);
        for (int k = warp; k * S64_CH <= x; k += S64_NW) {
            const int y = k * S64_CH - 1 + lane;
            // J'_TM = dA(x) J_TM, J'_TE = dB(x) J_TE with J(x, y) = Um(x) T(x-1, y) - Vp(x) T(x+1, y)
            double JT = 0.0, JE = 0.0;
            if (mt > 0 && y >= 0 && y <= x + 1) {
                JT = fma(UxA, Rm[LP + y], VxA * Rp[LP + y]);
                JE = fma(UxB, Rm[y], VxB * Rp[y]);
            }
            const double JTm = __shfl_up_sync(0xffffffffu, JT, 1), JTp = __shfl_down_sync(0xffffffffu, JT, 1);
            const double JEm = __shfl_up_sync(0xffffffffu, JE, 1), JEp = __shfl_down_sync(0xffffffffu, JE, 1);
            if (lane == 0 || lane == 31 || y < 1 || y > x) continue;
            const double tT = R0[LP + y], tE = R0[y];
            double ee, mm, em = 0.0, me = 0.0;
            if (mt == 0) {
                ee = dA * F(W_DA, y) * tT;
                mm = -(dB * F(W_DB, y) * tE);
            } else {
                // EE = dA dA [B_TM - m^2 T_TE], MM = dB dB [m^2 T_TM - B_TE], B(x, y) = Um(y) J(x, y-1) - Vp(y) J(x, y+1)
                const double yUA = F(W_UA, y), yVA = F(W_VA, y), yA = F(W_A, y), yUB = F(W_UB, y), yVB = F(W_VB, y), yB = F(W_B, y);
                const double hE = fma(yUB, R0[y - 1], yVB * R0[y + 1]), hT = fma(yUA, R0[LP + y - 1], yVA * R0[LP + y + 1]);
                ee = fma(yUA, JTm, fma(yVA, JTp, -(mA * (yA * tE))));
                mm = fma(mB, yB * tT, -fma(yUB, JEm, yVB * JEp));
                em = fma(mA, hE, -(yB * JT)); // m dA(x) dB(y) [H_TE - J_TM]
                me = fma(-mB, hT, yA * JE);   // m dB(x) dA(y) [J_TE - H_TM]
            }
            const int c0 = 2 * (y - 1);
            long long *col = Am + (size_t)c0 * n + r0;
            if (y != x) {
                *reinterpret_cast<longlong2 *>(col) = make_longlong2(-to_fix(ee, fq, bad), -to_fix(me, fq, bad));
                *reinterpret_cast<longlong2 *>(col + n) = make_longlong2(-to_fix(em, fq, bad), -to_fix(mm, fq, bad));
                if (FRO) fro += 2.0 * (fma(ee, ee, me * me) + fma(mm, mm, em * em));
            } else {
                // the diagonal from M_ii, which the trace is taken from too
                const double dee = md[r0], dmm = md[r0 + 1];
                const long long one = 1LL << fq;
                *reinterpret_cast<longlong2 *>(col) = make_longlong2(one - to_fix(dee, fq, bad), -to_fix(me, fq, bad));
                col[n + 1] = one - to_fix(dmm, fq, bad);
                if (FRO) fro += fma(dee, dee, dmm * dmm) + 2.0 * me * me;
            }
        }
    }
    if (FRO) { // per-CTA sums, added by the statistics kernel in order
        __shared__ double red[S64_NW];
        for (int o = 16; o > 0; o >>= 1) fro += __shfl_xor_sync(0xffffffffu, fro, o);
        if (lane == 0) red[warp] = fro;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int w = 0; w < S64_NW; w++) s += red[w];
            fro_out[(size_t)task * P + q] = s;
        }
    }
    if (__syncthreads_or(bad) && tid == 0) atomicOr(status + task, ST_ERR_NONFINITE);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static size_t s64_ring_bytes(int ldim) { return (size_t)S64_RING * 2 * (ldim + 4) * sizeof(double); }
static bool s64_ring_fits(int ldim) { return s64_ring_bytes(ldim) <= 220 * 1024; }

size_t seed64_bytes(int ldim, int ntask) { return (size_t)ntask * 2 * SEED_KINDS * (ldim + 2) * sizeof(sd); }

size_t sweep64_work_bytes(int ldim, int nlist, int P)
{
    const size_t L = ldim + 2;
    size_t b = (size_t)nlist * (P - 1) * 4 * L * sizeof(sd) + (size_t)nlist * L * (W_FIELDS * sizeof(double) + sizeof(int)) + 512;
    if (!s64_ring_fits(ldim)) b += (size_t)nlist * P * s64_ring_bytes(ldim);
    return b;
}

// CTAs per matrix: about one per SM in all, at least 16 rows per part and at most 16 parts (each
// starts from the q-sums of two rows).  One matrix of ldim 140: 2 parts 0.36 ms for seeds and
// sweep, 8 parts 0.15, the q-sums and elements of every pair 0.15; 32 matrices of ldim 350: 4 parts
// 0.6, every pair 2.3 ms
int sweep64_parts(int ldim, int nlist)
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        CK(cudaGetDevice(&dev));
        CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    }
    return max(1, min(min(16, ldim / 16), sms / max(nlist, 1)));
}

static void seed64(const Task *tasks, const int *tlist, int nlist, int ldim, int P, int k0, int k1, const sd *K, int nu_stride,
                   const double *lft, const double4 *ptab, int pstride, void *seed, sd *rows, int *status, cudaStream_t st)
{
    const int nbw = (ldim + 2 + 127) / 128;
    k_seed64<<<dim3(nbw * (2 + 2 * (P - 1)), nlist), 128, 0, st>>>(tasks, tlist, nlist, ldim, P, k0, k1, K, nu_stride, lft, ptab, pstride,
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

void launch_sweep64(const Task *tasks, const int *tlist, int nlist, int ldim, int P, const sd *K, int nu_stride, const double *lft,
                    const double4 *ptab, int pstride, const sd *Sa, const sd *Sb, void *seed, const double *mdiag, const int *info,
                    void *work, long long *A, size_t mstride, double *fro, int *status, cudaStream_t st)
{
    if (nlist <= 0) return;
    const size_t L = ldim + 2;
    double *tab = (double *)work; // 16-byte multiples: W_FIELDS is even
    sd *rows = (sd *)(tab + nlist * W_FIELDS * L);
    int *kt = (int *)(rows + (size_t)nlist * (P - 1) * 4 * L);
    const size_t ring_off = ((char *)(kt + nlist * L) - (char *)work + 255) & ~(size_t)255;
    const bool fits = s64_ring_fits(ldim);
    double *ring = fits ? nullptr : (double *)((char *)work + ring_off);
    const size_t sm = fits ? s64_ring_bytes(ldim) : 0;
    static size_t attr = 0;
    if (sm > attr) {
        CK(cudaFuncSetAttribute(k_sweep64<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        CK(cudaFuncSetAttribute(k_sweep64<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        attr = sm;
    }
    seed64(tasks, tlist, nlist, ldim, P, SEED_D1, SEED_COL, K, nu_stride, lft, ptab, pstride, seed, rows, status, st);
    k_sweep64_tab<<<nlist, 256, 0, st>>>(tasks, tlist, nlist, ldim, (const sd *)seed, Sa, Sb, tab, kt);
    if (fro)
        k_sweep64<true><<<nlist * P, S64_NT, sm, st>>>(tasks, tlist, nlist, ldim, P, (const sd *)seed, rows, tab, kt, mdiag, info, A,
                                                       mstride, fro, status, ring);
    else
        k_sweep64<false><<<nlist * P, S64_NT, sm, st>>>(tasks, tlist, nlist, ldim, P, (const sd *)seed, rows, tab, kt, mdiag, info, A,
                                                        mstride, fro, status, ring);
    COUNT_LAUNCH(2);
    CK(cudaGetLastError());
}

} // namespace capsgpu
