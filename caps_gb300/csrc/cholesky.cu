// cholesky.cu -- batched blocked Cholesky of the FP64 form and the log-det, in fixed point on
// the tensor cores.
//
// A = 1 - M is symmetric positive definite (the reference calls kernel_logdet with sym_spd=2,
// libcaps.c:954, and its HODLR path factors LL^T) and its diagonal is at most about 1, so every
// entry of A, of its Schur complements and of its Cholesky factor L lies in a fixed range:
// |A_ij| <= sqrt(A_ii A_jj) and sum_k L_ik^2 <= A_ii.  All of them are therefore held as 64-bit
// integers in units of 2^-60 (an FP64 number near 1 has units of 2^-53), and the FP64 pipe --
// two fused multiply-adds per clock and SM on this GPU, 1.05 TFLOP/s in all -- is left out:
//
//  * products with 64 columns (panel solve, trailing update) run on the tensor cores, split into exact
//    products of digits (Ozaki's scheme, with a common scale instead of one per row).  A factor x
//    is split into six signed 9-bit digits, x = sum_i d_i 2^(-8-9i), exact as FP16; the MMAs
//    (kind::f16, FP32 accumulators) form sum_k d_i(k) d_j(k) as exact integers in one accumulator
//    per i + j = 0..6, and the epilogue adds the accumulators up as 64-bit integers.  Digit
//    products with i + j > 6 are below 2^-60 and left out, so the error of a product is that
//    of the last digit, 2^-54 per factor -- an FP64 sum of 64 products has 2^-53 of its
//    partial sums at every step.
//  * the 64 x 64 diagonal blocks (factor and inverse) are taken in FP32 and corrected to 2^-54 by a
//    few such products (k_fix_potf2); blocks where that fails run on the integer pipes: a number is
//    h 2^30 + l, and a product needs three 32 x 32 -> 64 bit multiply-adds (h h, h l, l h).
//
// Per 64 columns three launches over the batch: k_fix_potf2 (diagonal block, W = L_kk^-1 as digit
// images, log det), k_fix_trsm (X = S W^T for the rows below, stored as digit images only),
// k_fix_syrk (S -= X X^T).  log det A = 2 sum_j log L_jj.  A non-positive pivot marks the task
// (ST_ERR_PIVOT) and its result becomes NaN; nothing traps.  A matrix whose diagonal exceeds 2
// (M with large negative diagonal entries) is scaled by a power of four on conversion.
//
// A matrix that is not positive definite keeps none of these bounds, and integers that wrap could end as
// positive pivots.  So what the bounds say is checked, and a matrix that breaks them is marked like one with a
// non-positive pivot: entries below 2 (on conversion, in the panel solve and in potf2_limbs), and the squares of
// a row of the factor, summed over all panels so far in FP32, below 2 (FIX_ROW).  While both hold nothing wraps,
// and the pivots are what they are.
#include "common.cuh"
#include "fix.cuh"
#include "internal.h"
#include "umma.cuh"
#include <algorithm>

namespace capsgpu {

// the digit products of one 128 x 64 tile, K = 64, of groups G0 .. G1 - 1, accumulator g at tmem + 64 g: NA
// digits of A (ASTEP bytes apart) and NBD digits of B (one block apart); alo, blo: low descriptor
// words of digit 0.  Unrolled, so that every descriptor is a sum with a constant.  Two parts, groups
// 0..SY_G0 - 1 and the rest, are handed to the folding warps one after the other.
template <int NA, int NBD, int ASTEP, int G0, int G1> CAPS_DEV void mma_groups(uint32_t tmem, uint32_t alo, uint32_t blo)
{
    constexpr uint32_t idesc = umma::idesc_f16(128, 64), hi = umma::desc_hi(1024);
#pragma unroll
    for (int g = G0; g < G1; g++) {
        const int i0 = g > NBD - 1 ? g - NBD + 1 : 0, i1 = g < NA - 1 ? g : NA - 1;
#pragma unroll
        for (int i = 0; i < NA; i++)
            if (i >= i0 && i <= i1) {
#pragma unroll
                for (int ks = 0; ks < 4; ks++) {
                    const uint32_t d = tmem + g * NB, a = alo + i * (ASTEP / 16) + ks * 16, b = blo + (g - i) * (IMG_BLK / 16) + ks * 16;
                    if (i == i0 && ks == 0) umma::mma_f16_lo<0>(d, a, b, hi, idesc);
                    else umma::mma_f16_lo<1>(d, a, b, hi, idesc);
                }
            }
    }
}

// the same for groups g0 .. g1 - 1 and ND x ND digits of which the first fa of A and fb of B are zero: their
// products are left out, and groups below fa + fb have none.  Entries of the factor fall off so fast
// away from the diagonal that of all products in the trailing updates of a free energy's matrices
// (R/L = 50) 5 % are left, and a third of the tiles have any.
CAPS_DEV void mma_nonzero(uint32_t tmem, uint32_t alo, uint32_t blo, int fa, int fb, int g0, int g1)
{
    constexpr uint32_t idesc = umma::idesc_f16(128, 64), hi = umma::desc_hi(1024);
    for (int g = max(g0, fa + fb); g < g1; g++) {
        const int i0 = max(fa, g - (ND - 1)), i1 = min(ND - 1, g - fb);
        uint32_t a = alo + i0 * (2 * IMG_BLK / 16), b = blo + (g - i0) * (IMG_BLK / 16);
        const uint32_t d = tmem + g * NB;
        umma::mma_f16_lo<0>(d, a, b, hi, idesc);
#pragma unroll
        for (int ks = 1; ks < 4; ks++) umma::mma_f16_lo<1>(d, a + ks * 16, b + ks * 16, hi, idesc);
#pragma unroll 1
        for (int i = i0 + 1; i <= i1; i++) {
            a += 2 * IMG_BLK / 16;
            b -= IMG_BLK / 16;
#pragma unroll
            for (int ks = 0; ks < 4; ks++) umma::mma_f16_lo<1>(d, a + ks * 16, b + ks * 16, hi, idesc);
        }
    }
}

// 16 columns of group s of this warp's lanes folded into v: groups come in the order s = s0, ..., 6 and
// each weighs 2^-9 of the one before, v = 512 v + g up to s = 5 (units of 2^-61; |v| < 2), then
// units of 2^-60.  One piece of code for all groups: unrolled, its first pass through the instruction cache
// cost more than the work.  A sum (an integer below 2^25) is read as the bits of g + 1.5 2^23 and the
// constant taken out at the end; a warp with one of 2^22 or more converts (19 clocks a number and warp where
// this takes about 7).
CAPS_DEV void fold_group(uint32_t taddr, int s, int s0, long long (&v)[16])
{
    float f[16];
    unsigned t[16], over = 0;
    umma::ld16(taddr, f);
#pragma unroll
    for (int c = 0; c < 16; c++) {
        t[c] = __float_as_uint(f[c] + FX_MAGIC);
        over |= t[c] ^ 0x4B000000u;
    }
    if (__any_sync(0xffffffffu, over >> 23)) {
#pragma unroll
        for (int c = 0; c < 16; c++) t[c] = FX_MBITS + (unsigned)__float2int_rn(f[c]);
    }
    if (s < 6) { // uniform
#pragma unroll
        for (int c = 0; c < 16; c++) v[c] = (long long)((unsigned long long)v[c] * 512 + t[c]);
    } else {
        unsigned long long k = 0;
        for (int i = s0; i < 6; i++) k = k * 512 + FX_MBITS;
#pragma unroll
        for (int c = 0; c < 16; c++) v[c] = ((long long)((unsigned long long)v[c] - k) + (((int)(t[c] - FX_MBITS) + 256) >> 9) + 1) >> 1;
    }
}

// ---------------------------------------------------------------------------
// FP64 -> fixed point, in place (lower triangle)
// ---------------------------------------------------------------------------
// scale exponent of a matrix whose largest diagonal entry is mx: none below 2, else a power of four
CAPS_DEV int fix_sexp(double mx) { return mx >= 2.0 ? 2 * ((min(ilogb(mx), 1023) + 2) / 2) : 0; }
// a diagonal entry is below 2, and so are the squares of a row of the factor; their FP32 sum stays below this
constexpr float FIX_ROW = 2.25f;

// for producers that write fixed point themselves: the exponents alone, one warp per task
__global__ void k_fix_scale(const int *tlist, int nlist, int n, const double *mdiag, FixInfo *info)
{
    const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (b >= nlist) return;
    const int task = tlist ? tlist[b] : b;
    double mx = 0.0;
    for (int i = lane; i < n; i += 32) mx = fmax(mx, 1.0 - mdiag[(size_t)task * n + i]);
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) info[task].sexp = fix_sexp(mx);
}

// grid (ceil(n / 8), ntask), 256 threads: 8 columns per block
__global__ void __launch_bounds__(256) k_fix_convert(int ntask, int n, double *A, size_t lda, size_t mstride, int *status,
                                                     const double *mdiag, FixInfo *info)
{
    const int task = blockIdx.y;
    if (task >= ntask || (status[task] & 0xF) != ST_FACTOR) return; // error bits may be set by this launch: not read
    __shared__ double red[8];
    double mx = 0.0;
    for (int i = threadIdx.x; i < n; i += 256) mx = fmax(mx, 1.0 - mdiag[(size_t)task * n + i]);
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    for (int w = 0; w < 8; w++) mx = fmax(mx, red[w]);
    const int sexp = fix_sexp(mx);
    if (blockIdx.x == 0 && threadIdx.x == 0) info[task].sexp = sexp;
    const double sc = ldexp(1.0, FQ - sexp);
    bool over = false;
    for (int c = blockIdx.x * 8; c < min(n, (int)blockIdx.x * 8 + 8); c++) {
        double *col = A + (size_t)task * mstride + (size_t)c * lda;
        for (int r = c + threadIdx.x; r < n; r += 256) {
            const double x = col[r] * sc, v = fmin(fmax(x, -0x1.fp61), 0x1.fp61);
            over |= !(fabs(x) < 0x1p61);
            reinterpret_cast<long long *>(col)[r] = __double2ll_rn(v);
        }
    }
    if (over) atomicOr(status + task, ST_ERR_PIVOT);
}

// ---------------------------------------------------------------------------
// diagonal block
// ---------------------------------------------------------------------------
// x = h 2^30 + l, |l| <= 2^29
CAPS_DEV int2 limbs(long long x)
{
    const int l = (int)((unsigned)x << 2) >> 2;
    return make_int2(l, (int)((x - l) >> 30));
}
// running sum of products of limbs: a sum over h h plus 2^-30 b (the l l terms, below one unit,
// are left out); units of the product of the two factors' units times 2^60
struct LAcc {
    long long a = 0, b = 0;
    CAPS_DEV void add(int2 x, int2 y)
    {
        a += (long long)x.y * y.y;
        b += (long long)x.y * y.x;
        b += (long long)x.x * y.y;
    }
    CAPS_DEV void add3(int2 x, int2 y) // with the l l term
    {
        add(x, y);
        b += ((long long)x.x * y.x) >> 30;
    }
    CAPS_DEV long long q60() const { return a + ((b + (1 << 29)) >> 30); } // units 2^-60 times 2^-q -> 2^-q
    // product of two numbers in units of 2^-w, in the same units
    CAPS_DEV long long q(int w) const { return (a << (60 - w)) + ((b + (1LL << (w - 31))) >> (w - 30)); }
};

// 1 / sqrt(d 2^-60), d > 0, as r 2^(k - 60) with r in (2^59, 2^60]: the FP32 reciprocal square
// root of the normalised value and one third-order Newton step in integers (error a few 2^-60)
CAPS_DEV long long fix_rsqrt(long long d, int &k)
{
    const int sh = (__clzll(d) - 2) & ~1;          // d 2^sh in [2^60, 2^62)
    const unsigned long long f = sh >= 0 ? (unsigned long long)d << sh : (unsigned long long)d >> -sh;
    k = sh >> 1;
    const float v = (float)(unsigned)(f >> 32) * 0x1p-28f;
    const unsigned R = min((unsigned)(rsqrtf(v) * 0x1p31f), 0x7fffffffu);
    const unsigned long long R2 = (unsigned long long)R * R;                  // 2^-62
    const long long e = (1LL << 58) - (long long)__umul64hi(f, R2);           // 1 - v r^2, 2^-58
    const float ef = (float)e * 0x1p-58f;
    const long long c = 2 * e + (long long)(int)(0.375f * ef * ef * 0x1p60f); // e / 2 + 3 e^2 / 8, 2^-60
    return ((long long)R << 29) + (__mul64hi((long long)((unsigned long long)R << 32), c << 4) >> 3);
}

constexpr int PP = NB + 1;
constexpr int PF_NT = 512;

// The block in limbs throughout, for blocks that k_fix_potf2 cannot take (ill conditioned beyond FP32, or
// not positive definite): L_kk by 16-column sub-panels, then W; about 80 us.  T, W: [64][PP] integers, Y:
// 3 x [16][17] limb pairs; on return W holds L_kk^-1 in units of 2^-wq (returned), *logs the sum of log
// L_jj over the first nb columns, *bad whether a pivot was not positive.  All threads.
//
// Warps 0..2: every warp holds the sub-panel's 16 diagonal rows in lanes 0..15 (all three compute
// them alike, so no warp waits for another) and 16 of the up to 48 rows below in lanes 16..31.
// Then all warps apply the rank-16 update to the rest of the triangle, in 2 x 2 tiles.  W: the
// four 16 x 16 diagonal blocks by substitution, one lane per column, then X_ij = -X_ii sum_k L_ik
// X_kj by distance from the diagonal.
__device__ __noinline__ int potf2_limbs(const long long *Sm, size_t lda, int nb, long long *T, long long *W, int2 *Y, double *logs, bool *isbad)
{
    __shared__ long long piv[NB], inv[NB];
    __shared__ int invk[NB];
    __shared__ double slog[2];
    __shared__ float rown[NB]; // squares of each row's entries so far
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    bool bad = false;
    if (tid < NB) rown[tid] = 0.0f;
    __syncthreads(); // the shared memory is free
    {
        long long v[NB * NB / PF_NT];
#pragma unroll
        for (int u = 0; u < NB * NB / PF_NT; u++) {
            const int e = tid + PF_NT * u, c = e >> 6, r = e & 63;
            v[u] = (r >= c && r < nb && c < nb) ? Sm[(size_t)c * lda + r] : (r == c ? 1LL << FQ : 0LL);
        }
#pragma unroll
        for (int u = 0; u < NB * NB / PF_NT; u++) {
            const int e = tid + PF_NT * u, c = e >> 6, r = e & 63;
            T[r * PP + c] = v[u];
            bad |= v[u] >= 1LL << (FQ + 1) || v[u] <= -(1LL << (FQ + 1));
        }
    }
    __syncthreads();
    int2 *Lm = reinterpret_cast<int2 *>(T);
    constexpr int PB = 16;
#pragma unroll 1
    for (int o = 0; o < NB; o += PB) {
        if (warp < 3) {
            const int row = lane < 16 ? o + lane : o + 16 * (warp + 1) + lane - 16;
            const bool live = row < NB;
            long long s[PB], b[PB];
#pragma unroll
            for (int c = 0; c < PB; c++) {
                s[c] = live && o + c <= row ? T[row * PP + o + c] : 0;
                b[c] = 0;
            }
            asm volatile("bar.sync 1, 96;" ::: "memory"); // the three warps have read the diagonal rows
            const bool mine = live && (warp == 0 || lane >= 16);
            float sq = 0.0f;
#pragma unroll
            for (int j = 0; j < PB; j++) {
                const long long sj = s[j] + ((b[j] + (1 << 29)) >> 30);
                long long d = __shfl_sync(0xffffffffu, sj, j);
                bad |= d <= 0;
                d = d > 0 ? d : 1LL << FQ;
                int k;
                const long long r = fix_rsqrt(d, k);
                if (warp == 0 && lane == 0) { piv[o + j] = d; inv[o + j] = r; invk[o + j] = k; }
                // x = s r 2^k
                const int2 sl = limbs(sj), rl = limbs(r);
                const long long ll = (long long)sl.x * rl.x, bb = (long long)sl.y * rl.x + (long long)sl.x * rl.y + (ll >> 30);
                const long long x = (((long long)sl.y * rl.y) << k) + (k < 30 ? bb >> (30 - k) : bb << (k - 30));
                const int2 xl = limbs(x);
                if (mine && row > o + j) {
                    const float xf = (float)sj * 0x1p-60f * ((float)r * 0x1p-60f) * ldexpf(1.0f, k);
                    sq = fmaf(xf, xf, sq);
                    Lm[row * PP + o + j] = xl;
                }
                const int nh = -xl.y, nl = -xl.x;
#pragma unroll
                for (int c = j + 1; c < PB; c++) {
                    const int cl = __shfl_sync(0xffffffffu, xl.x, c), ch = __shfl_sync(0xffffffffu, xl.y, c);
                    s[c] += (long long)nh * ch;
                    b[c] += (long long)nh * cl;
                    b[c] += (long long)nl * ch;
                }
            }
            if (mine) {
                sq += rown[row];
                rown[row] = sq;
                bad |= !(sq < FIX_ROW);
            }
        }
        __syncthreads();
        const int c0 = o + PB, t2 = (NB - c0) / 2; // 2 x 2 tiles: rows and columns c0 + i, c0 + i + t2
        for (int e = tid; e < t2 * (t2 + 1) / 2; e += PF_NT) {
            int ti = (int)((sqrtf(8.0f * e + 1.0f) - 1.0f) * 0.5f);
            while ((ti + 1) * (ti + 2) / 2 <= e) ti++;
            while (ti * (ti + 1) / 2 > e) ti--;
            const int tj = e - ti * (ti + 1) / 2;
            const int r0 = c0 + 2 * ti, q0 = c0 + 2 * tj;
            LAcc a00, a01, a10, a11;
#pragma unroll
            for (int k = 0; k < PB; k++) {
                const int2 x0 = Lm[r0 * PP + o + k], x1 = Lm[(r0 + 1) * PP + o + k];
                const int2 y0 = Lm[q0 * PP + o + k], y1 = Lm[(q0 + 1) * PP + o + k];
                a00.add(x0, y0);
                a01.add(x0, y1);
                a10.add(x1, y0);
                a11.add(x1, y1);
            }
            T[r0 * PP + q0] -= a00.q60();
            if (ti != tj) T[r0 * PP + q0 + 1] -= a01.q60();
            T[(r0 + 1) * PP + q0] -= a10.q60();
            T[(r0 + 1) * PP + q0 + 1] -= a11.q60();
        }
        __syncthreads();
    }
    // sum of log L_jj = 1/2 sum of log pivot (1 + (d - 1) where d is near 1: the difference is exact)
    if (tid < NB) {
        const long long d = piv[tid];
        double lg = 0.0;
        if (tid < nb) lg = d > (1LL << (FQ - 1)) ? log1p((double)(d - (1LL << FQ)) * 0x1p-60) : log((double)d * 0x1p-60);
        for (int o = 16; o > 0; o >>= 1) lg += __shfl_xor_sync(0xffffffffu, lg, o);
        if (lane == 0) slog[warp] = lg;
    }
    // W in units of 2^-wq: 57 holds entries up to 16; a worse conditioned block takes coarser units
    int wq = 57;
#pragma unroll 1
    for (;; wq -= 12) {
        __syncthreads();
        const float lim = ldexpf(1.0f, 61 - wq - 1); // limbs need |w| < 2^(61 - wq)
        bool over = false;
        auto put = [&](int r, int c, long long v, float approx) {
            over |= !(fabsf(approx) < lim);
            W[r * PP + c] = v;
        };
        if (tid < NB) {
            const int o = tid & ~15, c = tid & 15;
            int2 w[16];
#pragma unroll
            for (int r = 0; r < 16; r++) {
                LAcc t;
#pragma unroll
                for (int k = 0; k < r; k++) t.add(Lm[(o + r) * PP + o + k], w[k]); // w = 0 above the diagonal
                const long long rv = inv[o + r];
                const int k = invk[o + r];
                // 2^k inv, units 2^-60: times -t (units 2^-wq), or itself
                const long long y = r == c ? -(1LL << wq) : (r < c ? 0 : t.q60());
                const int2 yl = limbs(y), rl = limbs(rv);
                const long long ll = (long long)yl.x * rl.x, bb = (long long)yl.y * rl.x + (long long)yl.x * rl.y + (ll >> 30);
                const long long v = -((((long long)yl.y * rl.y) << k) + (k < 30 ? bb >> (30 - k) : bb << (k - 30)));
                w[r] = limbs(v);
                put(o + r, o + c, v, (float)y * ldexpf(1.0f, k - wq));
            }
        }
        __syncthreads();
        for (int dl = 1; dl < 4; dl++) {
            const int np = 4 - dl;
            for (int e = tid; e < np * 256; e += PF_NT) {
                const int p = e >> 8, r = (e >> 4) & 15, c = e & 15, i = p + dl;
                long long sum = 0;
                for (int k = p; k < i; k++) {
                    LAcc t;
#pragma unroll
                    for (int q = 0; q < 16; q++) t.add(Lm[(i * 16 + r) * PP + k * 16 + q], limbs(W[(k * 16 + q) * PP + p * 16 + c]));
                    sum += t.q60();
                }
                over |= !(fabsf((float)sum) < 0x1p59f);
                Y[(p * 16 + r) * 17 + c] = limbs(sum);
            }
            __syncthreads();
            for (int e = tid; e < np * 256; e += PF_NT) {
                const int p = e >> 8, r = (e >> 4) & 15, c = e & 15, i = p + dl;
                LAcc t;
                float ap = 0.0f;
#pragma unroll
                for (int q = 0; q < 16; q++)
                    if (q <= r) {
                        const int2 x = limbs(W[(i * 16 + r) * PP + i * 16 + q]), y = Y[(p * 16 + q) * 17 + c];
                        t.add3(x, y);
                        ap = fmaf((float)x.y, (float)y.y, ap);
                    }
                put(i * 16 + r, p * 16 + c, -t.q(wq), ap * ldexpf(1.0f, 60 - 2 * wq));
            }
            __syncthreads();
        }
        if (!__syncthreads_or(over) || wq <= 33) break;
    }
    __syncthreads();
    *logs = 0.5 * (slog[0] + slog[1]);
    *isbad = __syncthreads_or(bad) != 0;
    return wq;
}

// ---- the block in FP32 and one correction ----
// L_kk and W = L_kk^-1 of the 64 x 64 block at k0 (past the matrix: the identity), W as digit images in
// the operand layout, sum of log L_jj into logdet[task * nbk + block]; one CTA per matrix.
//
// A factor in 64-bit arithmetic is a chain of 64 long steps (about 1000 clocks each in limbs, more on
// the FP64 pipe).  Instead W0 ~ L^-1 is taken from an FP32 Cholesky (a chain of 64 steps of about 90
// clocks) and corrected by products that the tensor cores form to 2^-54:
//   E = W0 S W0^T - I                             (|E| ~ 1e-6),
//   I + E = (I + Y)(I + Y)^T, Y = F(E) - F(P P^T), P = F(E) the lower triangle with half the diagonal
//                                                 (left out: third order in E),
//   L^-1 = (I + Y)^-1 W0 = W0 - Z W0, Z = Y - P^2,
//   log L_jj = log(1 + Y_jj) - log W0_jj.
// W0 has three digits (27 bits), so that the products take 17 MMAs per 16 columns instead of 26; P P^T
// and P^2 are of second order and FP32 suffices.  Where E is not small (|E| > 2^-18, beyond which its third
// order shows; a block of condition above about 50) or FP32 finds no factor, potf2_limbs takes the
// block.
//
// A block that is near the identity needs no first factor: with |S - 1| < 2^-19 (Frobenius) W0 = 1, E = S - 1
// as it stands, third order is below 2^-57 and W = 1 - Z; below 2^-33 second order is too; up to 2^-10 W0 = 1 - F(S - 1)
// leaves an E below 2^-19, and no FP32 factor is needed (8 us).  Two thirds to
// four fifths of the blocks of a free energy's matrices are such (all but the first few of a
// matrix), and the blocks of one launch tend to be so together: a launch of such blocks takes about 14 us
// instead of 40 (factorisation of a free energy at R/L = 100 11.0 -> 9.2 ms, of the 5500 small matrices of
// a T = 0 energy 6.3 -> 4.3).
//
// 512 threads.  The FP32 part runs on the block augmented by the identity in panels of 8 columns (three
// warps hold a panel's 8 diagonal rows and 24 of the others each; two barriers per panel), so that its
// code is short: fully unrolled 32 x 32 steps spent most of their time fetching instructions (50 us a
// block; 82 us with the 64-bit limbs).  64 rows use lanes 0..63 of tensor memory, so the warps of lane
// quadrants 0 and 1 fold, 16 columns each; warps 2 and 3 take the logarithms of W0_jj meanwhile.
constexpr int PF_W0 = ND * IMG_BLK, PF_WT = PF_W0 + 3 * IMG_BLK, PF_F = PF_WT + 3 * IMG_BLK, PF_SMEM = PF_F + 2 * NB * PP * 4; // 130 KB
static_assert(NB * PP * 16 + 3 * 16 * 17 * 8 <= PF_SMEM, "potf2_limbs fits");

// F: the block (lower triangle) in FP32, replaced by L; X: W0 = L^-1, all 64 x 64; rinv: scratch of 64.  Begins
// and ends with a barrier; false where a pivot is not above 1e-6 (in the three panel warps).
CAPS_DEV bool pf_factor32(float *F, float *X, float *rinv)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    bool ok = true;
    for (int e = tid; e < NB * NB; e += PF_NT) X[(e >> 6) * PP + (e & 63)] = (e >> 6) == (e & 63) ? 1.0f : 0.0f;
    __syncthreads();
#pragma unroll 1
    for (int p = 0; p <= 8; p++) {
        const int o = p * 8, q = o - 8;
        if (warp < 3 && p < 8) {
            const int row = lane < 8 ? o + lane : o + warp * 24 + lane;
            const bool live = row < NB;
            float a[8];
#pragma unroll
            for (int c = 0; c < 8; c++) a[c] = live ? F[row * PP + o + c] : 0.0f;
            asm volatile("bar.sync 1, 96;" ::: "memory"); // the three warps have read the diagonal rows
            // every lane keeps the panel's pivots, so that none is broadcast: the chain of a column is a
            // reciprocal square root (2^-22, as good as the factor needs), a product, a shuffle and an fma
            float rv = 0.0f, d[8];
#pragma unroll
            for (int j = 0; j < 8; j++) d[j] = __shfl_sync(0xffffffffu, a[j], j);
#pragma unroll
            for (int j = 0; j < 8; j++) {
                ok &= d[j] > 1e-6f;
                float r;
                asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fmaxf(d[j], 1e-6f)));
                if (lane == j) rv = r;
                a[j] *= r;
#pragma unroll
                for (int c = j + 1; c < 8; c++) {
                    const float y = __shfl_sync(0xffffffffu, a[j], c);
                    a[c] = fmaf(-a[j], y, a[c]);
                    d[c] = fmaf(-y, y, d[c]);
                }
            }
            if (live && (warp == 0 || lane >= 8))
#pragma unroll
                for (int c = 0; c < 8; c++) F[row * PP + o + c] = a[c];
            if (warp == 0 && lane < 8) rinv[o + lane] = rv;
        } else if (warp >= 4 && warp < 6 && p > 0) { // rows q .. q + 7 of X, one column per thread
            const int c = tid - 128;
            float x[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                float t = X[(q + i) * PP + c];
#pragma unroll
                for (int k = 0; k < i; k++) t = fmaf(-F[(q + i) * PP + q + k], x[k], t);
                x[i] = t * rinv[q + i];
            }
#pragma unroll
            for (int i = 0; i < 8; i++) X[(q + i) * PP + c] = x[i];
        }
        __syncthreads();
        // 2 x 2 tiles: of the block's rest with panel p, then of X below row o with panel p - 1
        const int ts = p < 8 ? (56 - o) / 2 : 0, ns = ts * (ts + 1) / 2;
        // (two loops with constant strides: one loop over both kinds took twice as long)
        for (int e = tid; e < ns; e += PF_NT) {
            int ti = (int)((sqrtf(8.0f * e + 1.0f) - 1.0f) * 0.5f);
            ti += (ti + 1) * (ti + 2) / 2 <= e;
            ti -= ti * (ti + 1) / 2 > e;
            const int tj = e - ti * (ti + 1) / 2, rr = o + 8 + 2 * ti, cc = o + 8 + 2 * tj;
            const float *x0 = F + rr * PP + o, *y0 = F + cc * PP + o;
            float *out = F + rr * PP + cc, s00 = 0, s01 = 0, s10 = 0, s11 = 0;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                s00 = fmaf(x0[k], y0[k], s00);
                s01 = fmaf(x0[k], y0[PP + k], s01);
                s10 = fmaf(x0[PP + k], y0[k], s10);
                s11 = fmaf(x0[PP + k], y0[PP + k], s11);
            }
            out[0] -= s00;
            if (ti != tj) out[1] -= s01;
            out[PP] -= s10;
            out[PP + 1] -= s11;
        }
        // columns in pairs by lane, rows by warp, from the last warp on (the first have the block's tiles)
        const int cc = 2 * lane;
        if (cc < o)
            for (int rr = o + 2 * (PF_NT / 32 - 1 - warp); rr < NB; rr += PF_NT / 16) {
                const float *x0 = F + rr * PP + q, *y0 = X + q * PP + cc;
                float *out = X + rr * PP + cc, s00 = 0, s01 = 0, s10 = 0, s11 = 0;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const float w0 = y0[k * PP], w1 = y0[k * PP + 1];
                    s00 = fmaf(x0[k], w0, s00);
                    s01 = fmaf(x0[k], w1, s01);
                    s10 = fmaf(x0[PP + k], w0, s10);
                    s11 = fmaf(x0[PP + k], w1, s11);
                }
                out[0] -= s00;
                out[1] -= s01;
                out[PP] -= s10;
                out[PP + 1] -= s11;
            }
        __syncthreads();
    }
    return ok;
}

// eight FP32 numbers times 2^18 as FP16 high and low parts
CAPS_DEV void split_half(const float (&x)[8], uint4 &h, uint4 &l)
{
    unsigned hw[4], lw[4];
#pragma unroll
    for (int p = 0; p < 4; p++) {
        const float a = x[2 * p] * 0x1p18f, b = x[2 * p + 1] * 0x1p18f;
        const __half2 hh = __floats2half2_rn(a, b);
        const __half2 ll = __floats2half2_rn(a - __low2float(hh), b - __high2float(hh));
        hw[p] = *reinterpret_cast<const unsigned *>(&hh);
        lw[p] = *reinterpret_cast<const unsigned *>(&ll);
    }
    h = make_uint4(hw[0], hw[1], hw[2], hw[3]);
    l = make_uint4(lw[0], lw[1], lw[2], lw[3]);
}

// one thread of warp 15 issues, warps of quadrants 0 and 1 fold; see k_fix_potf2
struct PfCtx {
    uint64_t *sfull; // two mbarriers
    uint32_t tmem;
    int n0, n1;      // their completed phases
    bool live;       // no wait has run out
};
// D = A B^T of 64 x 64 blocks with NA and NBD digits into v (folding warps: row quad * 32 + lane, columns part * 16
// + c).  Begins with a barrier: the digits are written, the accumulators free.
template <int NA, int NBD> CAPS_DEV void pf_product(uint32_t a, uint32_t b, long long (&v)[16], PfCtx &C)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3, part = warp >> 2;
    umma::fence_smem_async();
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    if (warp == 15) {
        if (lane == 0) {
            mma_groups<NA, NBD, IMG_BLK, 0, SY_G0>(C.tmem, umma::desc_lo(a, 128), umma::desc_lo(b, 128));
            umma::commit(&C.sfull[0]);
            mma_groups<NA, NBD, IMG_BLK, SY_G0, NG>(C.tmem, umma::desc_lo(a, 128), umma::desc_lo(b, 128));
            umma::commit(&C.sfull[1]);
        }
        __syncwarp();
    } else if (quad < 2) {
#pragma unroll
        for (int c = 0; c < 16; c++) v[c] = 0;
#pragma unroll 1
        for (int g = 0; g < NG; g++) {
            if (g == 0 || g == SY_G0) {
                C.live = C.live && umma::mbar_wait(&C.sfull[g ? 1 : 0], (g ? C.n1 : C.n0) & 1, FIX_WAIT_ITERS);
                C.live = __all_sync(0xffffffffu, C.live);
                umma::fence_after();
            }
            if (C.live) fold_group(C.tmem + ((uint32_t)(quad * 32) << 16) + g * NB + part * 16, g, 0, v);
        }
        umma::fence_before();
    }
    C.n0++;
    C.n1++;
}

// digits of this warp's 16 columns of a folded product into an image
CAPS_DEV void pf_store(const long long (&v)[16], unsigned char *img)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3, part = warp >> 2;
#pragma unroll
    for (int q = 0; q < 2; q++) {
        long long x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = v[q * 8 + u];
        uint4 d[ND];
        split8(x, d);
#pragma unroll
        for (int i = 0; i < ND; i++) *reinterpret_cast<uint4 *>(img + i * IMG_BLK + img_off(quad * 32 + lane, part * 2 + q)) = d[i];
    }
}

__global__ void __launch_bounds__(PF_NT, 1) k_fix_potf2(int ntask, int n, int k0, const long long *S, size_t lda, size_t mstride, int *status,
                                                        FixWork wk, double *logdet)
{
    const int task = blockIdx.x;
    // (an update on another stream may set a wait error meanwhile: one decision for the block)
    if (task >= ntask || !__syncthreads_and(status[task] == ST_FACTOR)) return;
    extern __shared__ __align__(1024) unsigned char pf_sm[];
    float *F = reinterpret_cast<float *>(pf_sm + PF_F), *X = F + NB * PP;
    int *W27 = reinterpret_cast<int *>(X); // W0 2^-wexp in units of 2^-26
    __shared__ float rinv[NB];
    __shared__ uint64_t sfull[2], drain;
    __shared__ uint32_t tslot;
    __shared__ int s_ok, s_max, s_emax;
    __shared__ float s_fro[PF_NT / 32];
    __shared__ double slog[2];
    __shared__ long long sy[8];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = warp & 3, part = warp >> 2;
    const bool folds = quad < 2;
    const int nb = min(NB, n - k0);
    const long long *Sm = S + (size_t)task * mstride + (size_t)k0 * lda + k0;
    const int er = tid & 63, ek = tid >> 6; // this thread's row and chunk of 8 columns of an image
    long long *tmp = reinterpret_cast<long long *>(pf_sm + PF_W0); // [64][PP]
    // the lower triangle (the identity past the matrix), mirrored in shared memory, and |S - 1|^2
    {
        long long x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int c = ek * 8 + u;
            x[u] = c <= er && er < nb ? Sm[(size_t)c * lda + er] : (er == c ? 1LL << FQ : 0LL);
        }
        if (tid == 0) {
            umma::mbar_init(&sfull[0], 1);
            umma::mbar_init(&sfull[1], 1);
            umma::mbar_init(&drain, 1);
            s_ok = 1;
            s_max = s_emax = 0;
        }
        if (tid < 2) slog[tid] = 0.0;
        if (warp == 15) umma::alloc(&tslot, 512);
        float fro = 0.0f;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int c = ek * 8 + u;
            if (c <= er) {
                const float e = fx_value(x[u] - (er == c ? 1LL << FQ : 0LL));
                fro = fmaf(e, e, fro);
                F[er * PP + c] = e;
                tmp[er * PP + c] = x[u];
                tmp[c * PP + er] = x[u];
            }
        }
        for (int o = 16; o > 0; o >>= 1) fro += __shfl_xor_sync(0xffffffffu, fro, o);
        if (lane == 0) s_fro[warp] = fro;
    }
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    float fro = 0.0f;
    for (int w = 0; w < PF_NT / 32; w++) fro += s_fro[w];
    fro *= 2.0f; // both triangles (the diagonal counts twice)
    const bool near1 = fro < 0x1p-38f;     // W0 = 1
    const bool second = !(fro < 0x1p-66f); // PP^T and P^2 reach the last digit
    const uint32_t base = umma::smem_u32(pf_sm);
    const int row = quad * 32 + lane, c0 = part * 16;
    PfCtx C{sfull, tslot, 0, 0, true};
    bool ok = true;
    int wexp = 0;
    long long v[16];
    if (near1) {
        // E = S - 1
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int c = ek * 8 + u;
            if (c >= er) F[er * PP + c] = c == er ? 0.5f * F[er * PP + c] : 0.0f;
        }
        if (folds)
#pragma unroll
            for (int c = 0; c < 16; c++) v[c] = tmp[row * PP + c0 + c] - (row == c0 + c ? 1LL << FQ : 0LL);
    } else {
        long long x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = tmp[er * PP + ek * 8 + u];
        uint4 d[ND];
        split8(x, d);
#pragma unroll
        for (int i = 0; i < ND; i++) *reinterpret_cast<uint4 *>(pf_sm + i * IMG_BLK + img_off(er, ek)) = d[i];
        if (fro < 0x1p-20f) {
            // W0 = 1 - F(S - 1)
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int c = ek * 8 + u;
                X[er * PP + c] = c > er ? 0.0f : c == er ? 1.0f - 0.5f * F[er * PP + c] : -F[er * PP + c];
            }
        } else {
            if (er >= ek * 8 && er < ek * 8 + 8) F[er * PP + er] += 1.0f;
            if (!pf_factor32(F, X, rinv)) s_ok = 0; // its barriers stand between this and the reads below
        }
        float mx = 0.0f;
#pragma unroll
        for (int u = 0; u < 8; u++) mx = fmaxf(mx, fabsf(X[er * PP + ek * 8 + u]));
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) atomicMax(&s_max, __float_as_int(mx)); // non-negative floats order as integers; NaN is large
        __syncthreads();
        const float w0max = __int_as_float(s_max);
        ok = s_ok && w0max < 1e6f; // uniform
        while (wexp < 24 && w0max > 3.9f * (float)(1 << wexp)) wexp++;
    }
    if (ok && !near1) {
        const float sc = (float)(1 << 26) / (float)(1 << wexp);
        // W0 in place as integers of 27 bits, then its digits, by rows and by columns
#pragma unroll
        for (int u = 0; u < 8; u++) W27[er * PP + ek * 8 + u] = fx_f2i(X[er * PP + ek * 8 + u] * sc);
        __syncthreads();
#pragma unroll
        for (int t = 0; t < 2; t++) {
            long long x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) x[u] = (long long)(t ? W27[(ek * 8 + u) * PP + er] : W27[er * PP + ek * 8 + u]) << (FQ - 26);
            uint4 d[ND];
            split8(x, d); // the last three digits are zero
#pragma unroll
            for (int i = 0; i < 3; i++) *reinterpret_cast<uint4 *>(pf_sm + (t ? PF_WT : PF_W0) + i * IMG_BLK + img_off(er, ek)) = d[i];
        }
        // T = W0 S, in the digits' place afterwards
        pf_product<3, ND>(base + PF_W0, base, v, C);
        if (folds) pf_store(v, pf_sm);
        if (warp == 2 || warp == 3) { // logarithms of W0_jj on warps that neither fold nor issue
            const int j = (warp - 2) * 32 + lane;
            const double w = (double)W27[j * PP + j] * pow2i(wexp - 26);
            double lw = j < nb ? (w > 0.5 && w < 2.0 ? log1p(w - 1.0) : log(w)) : 0.0;
            for (int o = 16; o > 0; o >>= 1) lw += __shfl_xor_sync(0xffffffffu, lw, o);
            if (lane == 0) slog[warp - 2] = lw;
        }
        // E = T W0^T - I; P = F(E) in FP32 in place of L
        pf_product<ND, 3>(base, base + PF_W0, v, C);
        if (folds) {
            int mx = 0;
#pragma unroll
            for (int c = 0; c < 16; c++) {
                v[c] = (v[c] << (2 * wexp)) - (row == c0 + c ? 1LL << FQ : 0LL);
                const float e = fx_value(v[c]);
                F[row * PP + c0 + c] = row > c0 + c ? e : row == c0 + c ? 0.5f * e : 0.0f;
                mx = max(mx, __float_as_int(fabsf(e)));
            }
            for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            if (lane == 0) atomicMax(&s_emax, mx);
        }
    }
    if (ok) {
        __syncthreads(); // the MMAs have read T: P's parts take its place (rows high, low, columns high, low)
        if (second) {
#pragma unroll
            for (int t = 0; t < 2; t++) {
                float x[8];
#pragma unroll
                for (int u = 0; u < 8; u++) x[u] = t ? F[(ek * 8 + u) * PP + er] : F[er * PP + ek * 8 + u];
                uint4 h, l;
                split_half(x, h, l);
                *reinterpret_cast<uint4 *>(pf_sm + (2 * t) * IMG_BLK + img_off(er, ek)) = h;
                *reinterpret_cast<uint4 *>(pf_sm + (2 * t + 1) * IMG_BLK + img_off(er, ek)) = l;
            }
        }
        const float emax = __int_as_float(s_emax);
        // P P^T and P^2, scaled by 2^36: high high + high low + low high
        if (second) {
            umma::fence_smem_async();
            umma::fence_before();
            __syncthreads();
            umma::fence_after();
        }
        if (warp == 15 && second) {
            if (lane == 0) {
                constexpr uint32_t idesc = umma::idesc_f16(128, 64), hi = umma::desc_hi(1024);
                const uint32_t ph = umma::desc_lo(base, 128), pl = ph + IMG_BLK / 16;
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    const uint32_t qh = ph + t * 2 * IMG_BLK / 16, ql = qh + IMG_BLK / 16, d = C.tmem + t * NB;
#pragma unroll
                    for (int ks = 0; ks < 4; ks++) {
                        if (ks == 0) umma::mma_f16_lo<0>(d, ph, ql, hi, idesc);
                        else umma::mma_f16_lo<1>(d, ph + ks * 16, ql + ks * 16, hi, idesc);
                        umma::mma_f16_lo<1>(d, pl + ks * 16, qh + ks * 16, hi, idesc);
                        umma::mma_f16_lo<1>(d, ph + ks * 16, qh + ks * 16, hi, idesc);
                    }
                }
                umma::commit(&sfull[0]);
            }
            __syncwarp();
        } else if (folds) {
            float gg[16], pp[16];
#pragma unroll
            for (int c = 0; c < 16; c++) gg[c] = pp[c] = 0.0f;
            if (second) {
                C.live = C.live && umma::mbar_wait(&sfull[0], C.n0 & 1, FIX_WAIT_ITERS);
                C.live = __all_sync(0xffffffffu, C.live);
                umma::fence_after();
                if (C.live) {
                    umma::ld16(C.tmem + ((uint32_t)(quad * 32) << 16) + c0, gg);
                    umma::ld16(C.tmem + ((uint32_t)(quad * 32) << 16) + NB + c0, pp);
                }
            }
            if (C.live) {
                long long ydiag = 0;
                float gdiag = 0.0f;
#pragma unroll
                for (int c = 0; c < 16; c++) {
                    // Z = F(E) - F(P P^T) - P^2
                    const bool dg = row == c0 + c;
                    const long long e = dg ? v[c] >> 1 : v[c];
                    const float g = dg ? 0.5f * gg[c] : gg[c];
                    if (dg) {
                        ydiag = e;
                        gdiag = g;
                    }
                    v[c] = row >= c0 + c ? e - fx_f2i((g + pp[c]) * 0x1p24f) : 0; // below 2^30 for |E| < 2^-18
                }
                // log(1 + y) = y - y^2 / 2 + y^3 / 3 of Y's diagonal
                const float y = fx_value(ydiag);
                long long ysum = row < nb ? ydiag - fx_f2i(gdiag * 0x1p24f + y * y * (0.5f - 0.33333333f * y) * 0x1p60f) : 0;
                // (64 atomic additions to one word of shared memory took 3 us)
                for (int o = 16; o > 0; o >>= 1) ysum += __shfl_xor_sync(0xffffffffu, ysum, o);
                if (lane == 0) sy[part * 2 + quad] = ysum;
                if (!near1) pf_store(v, pf_sm); // Z's digits; every MMA so far has completed
            }
            umma::fence_before();
        }
        if (second) C.n0++;
        // W = W0 - Z W0, its digits straight to the image (below 4: the top digit stays below 1024)
        if (!near1) pf_product<ND, 3>(base, base + PF_WT, v, C);
        if (folds) {
#pragma unroll
            for (int c = 0; c < 16; c++)
                v[c] = (near1 ? (row == c0 + c ? 1LL << FQ : 0LL) : (long long)W27[row * PP + c0 + c] << (FQ - 26)) - v[c];
            if (C.live) pf_store(v, wk.wimg(task, n));
        }
        ok = emax < 0x1p-18f;
    }
    if (!__syncthreads_and(C.live)) {
        if (tid == 0) atomicOr(status + task, ST_ERR_WAIT);
        if (tid == 15 * 32) { // the MMAs issued before the failure complete before the tensor memory goes
            umma::commit(&drain);
            umma::mbar_wait(&drain, 0, FIX_WAIT_ITERS);
        }
    } else if (ok) {
        if (tid == 0) {
            wk.info[task].wexp = wexp;
            logdet[(size_t)task * fix_nbk(n) + k0 / NB] = (double)(((sy[0] + sy[1]) + (sy[2] + sy[3])) + ((sy[4] + sy[5]) + (sy[6] + sy[7]))) * 0x1p-60 - (slog[0] + slog[1]);
        }
    } else {
        double lg;
        bool bad;
        long long *T = reinterpret_cast<long long *>(pf_sm), *W = T + NB * PP;
        const int wq = potf2_limbs(Sm, lda, nb, T, W, reinterpret_cast<int2 *>(W + NB * PP), &lg, &bad);
        __shared__ unsigned long long smax;
        if (tid == 0) smax = 0;
        __syncthreads();
        unsigned long long mx = 0;
        for (int e = tid; e < NB * NB; e += PF_NT) {
            const int r = e >> 6, c = e & 63;
            if (c <= r) {
                const long long w = W[r * PP + c];
                mx = max(mx, (unsigned long long)(w < 0 ? -w : w));
            }
        }
        atomicMax(&smax, mx);
        __syncthreads();
        int we = 0;
        while (we < 40 && (float)smax * exp2f((float)(-wq - we)) > 3.9f) we++;
        unsigned char *img = wk.wimg(task, n);
        const int sh = FQ - wq - we;
        for (int e = tid; e < NB * 8; e += PF_NT) {
            const int j = e & 63, kc = e >> 6;
            long long x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int c = kc * 8 + u;
                const long long w = c <= j ? W[j * PP + c] : 0;
                x[u] = sh >= 0 ? w << sh : (w + (1LL << (-sh - 1))) >> -sh;
            }
            uint4 d[ND];
            split8(x, d);
#pragma unroll
            for (int i = 0; i < ND; i++) *reinterpret_cast<uint4 *>(img + i * IMG_BLK + img_off(j, kc)) = d[i];
        }
        if (tid == 0) {
            wk.info[task].wexp = we;
            logdet[(size_t)task * fix_nbk(n) + k0 / NB] = lg;
            if (bad) atomicOr(status + task, ST_ERR_PIVOT);
        }
    }
    umma::fence_before();
    __syncthreads();
    if (warp == 15) {
        umma::fence_after();
        umma::dealloc(C.tmem, 512);
    }
}

// ---------------------------------------------------------------------------
// panel solve: X = S W^T for 128 rows below the diagonal block
// ---------------------------------------------------------------------------
// grid (ceil(rows / 128), ntask), 512 threads, 144 KB of shared memory.  The threads split the
// rows of S into digits while the digits of W arrive by bulk copies; one thread issues the
// MMAs of each group, and all warps fold the accumulators (lane quadrant warp mod 4, 16 of
// the 64 columns), split X and store its images.  Rows past n are zero.  Bound by its latencies (loads, 104
// MMAs, fold): with 256 threads and the loads in four rounds 45 us for 336 CTAs.
constexpr int TR_NT = 512;
constexpr int TR_A = ND * 2 * IMG_BLK, TR_B = ND * IMG_BLK; // 96 KB, 48 KB
constexpr int TR_SMEM = TR_A + TR_B;
__global__ void __launch_bounds__(TR_NT) k_fix_trsm(int ntask, int n, int k0, const long long *S, size_t lda, size_t mstride, int *status,
                                                    FixWork wk)
{
    const int task = blockIdx.y;
    if (task >= ntask || !__syncthreads_and((status[task] & ~ST_ERR_WAIT) == ST_FACTOR)) return; // as in k_fix_potf2
    extern __shared__ __align__(1024) unsigned char tr_sm[];
    __shared__ uint64_t wfull, gfull[2];
    __shared__ uint32_t tslot, s_any[2][3]; // or of the magnitudes' low and high words: S, X of both row blocks
    __shared__ float s_rn[4][128];          // squares of X, 16 columns each
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row0 = k0 + NB + blockIdx.x * 128;
    int *first = wk.first + (size_t)task * (fix_nbk(n) + 1) + blockIdx.x * 2;
    const long long *Sm = S + (size_t)task * mstride;
    {
        const int r = tid & 127, R = row0 + r, kc = tid >> 7; // chunks kc and kc + 4 of 8 columns
        long long x[16];
#pragma unroll
        for (int u = 0; u < 16; u++) x[u] = R < n ? Sm[(size_t)(k0 + (kc + (u >> 3) * 4) * 8 + (u & 7)) * lda + R] : 0;
        if (tid < 6) s_any[tid & 1][tid >> 1] = 0;
        __syncthreads();
        unsigned long long any = 0;
#pragma unroll
        for (int u = 0; u < 16; u++) any |= digit_mag(x[u]);
        const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)any), hi = __reduce_or_sync(0xffffffffu, (unsigned)(any >> 32));
        if (lane == 0 && (lo | hi)) {
            atomicOr(&s_any[0][0], lo);
            atomicOr(&s_any[1][0], hi);
        }
        __syncthreads();
        if ((s_any[0][0] | s_any[1][0]) == 0) { // S has no digit here: X = 0
            if (tid < 2) first[tid] = NG;
            if (k0 == 0 && tid < 128 && R < n) wk.rn[(size_t)task * n + R] = 0.0f;
            return;
        }
        if (warp == 0) umma::alloc(&tslot, 512);
        if (tid == 0) {
            umma::mbar_init(&wfull, 1);
            for (int g = 0; g < 2; g++) umma::mbar_init(&gfull[g], 1);
            umma::mbar_arrive_tx(&wfull, TR_B);
            umma::bulk_g2s(tr_sm + TR_A, wk.wimg(task, n), TR_B, &wfull);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            long long y[8];
#pragma unroll
            for (int u = 0; u < 8; u++) y[u] = x[h * 8 + u];
            uint4 d[ND];
            split8(y, d);
#pragma unroll
            for (int i = 0; i < ND; i++) *reinterpret_cast<uint4 *>(tr_sm + i * 2 * IMG_BLK + img_off(r, kc + h * 4)) = d[i];
        }
    }
    umma::fence_smem_async();
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tslot, 0);
    const bool have = umma::mbar_wait(&wfull, 0, FIX_WAIT_ITERS);
    if (!have && tid == 0) atomicOr(status + task, ST_ERR_WAIT);
    bool ok = have;
    const int fa = first_digit((unsigned long long)s_any[1][0] << 32 | s_any[0][0]);
    if (warp == 0 && have) {
        const uint32_t a = umma::desc_lo(umma::smem_u32(tr_sm), 128), b = a + TR_A / 16;
        if (lane == 0) {
            mma_nonzero(tmem, a, b, fa, 0, 0, SY_G0);
            umma::commit(&gfull[0]);
            mma_nonzero(tmem, a, b, fa, 0, SY_G0, NG);
            umma::commit(&gfull[1]);
        }
        __syncwarp();
    }
    const int quad = warp & 3, part = warp >> 2;
    bool over = s_any[1][0] >> 22; // an entry of S is 2 or more (2^54 units of 2^-53)
    long long v[16];
#pragma unroll
    for (int c = 0; c < 16; c++) v[c] = 0;
#pragma unroll 1
    for (int g = 0; g < NG; g++) {
        if (g == 0 || g == SY_G0) {
            ok = ok && umma::mbar_wait(&gfull[g ? 1 : 0], 0, FIX_WAIT_ITERS);
            ok = __all_sync(0xffffffffu, ok);
            umma::fence_after();
        }
        if (ok && g >= fa) fold_group(tmem + ((uint32_t)(quad * 32) << 16) + g * NB + part * 16, g, fa, v);
        if (g == 0 && fa == 0) {
            // The fold holds sums below 4.  Of X 2^-wexp, below sqrt 2, the later groups are at most 1.01 (64 products of
            // top digits, 1023 at most, with second ones, 256), so the first is below 2.75, and a sum with such a first group
            // is below 4.  Without top digits of S the sum is below 64 * 2^-8 * 4 = 1
#pragma unroll
            for (int c = 0; c < 16; c++) over |= (unsigned)v[c] - (FX_MBITS - (11 << 14)) > 2u * (11 << 14);
        }
    }
    const int wexp = wk.info[task].wexp, rb = quad >> 1; // rb: row block of the pair
    {
        if (wexp) // uniform
#pragma unroll
            for (int c = 0; c < 16; c++) over |= (unsigned long long)(v[c] + (1LL << (FQ + 1 - wexp))) >> (FQ + 2 - wexp) != 0;
        unsigned long long any = 0;
        float sq = 0.0f;
#pragma unroll
        for (int c = 0; c < 16; c++) {
            v[c] <<= wexp;
            any |= digit_mag(v[c]);
            // in units of 2^-20, |X| < 2
            const float f = __int_as_float((int)FX_MBITS + ((int)(v[c] >> 32) >> 8)) - FX_MAGIC;
            sq = fmaf(f, f, sq);
        }
        s_rn[part][quad * 32 + lane] = sq;
        const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)any), hi = __reduce_or_sync(0xffffffffu, (unsigned)(any >> 32));
        if (lane == 0 && (lo | hi)) {
            atomicOr(&s_any[0][1 + rb], lo);
            atomicOr(&s_any[1][1 + rb], hi);
        }
    }
    umma::fence_before();
    __syncthreads();
    if (tid < 2) first[tid] = first_digit((unsigned long long)s_any[1][1 + tid] << 32 | s_any[0][1 + tid]);
    if (tid < 128 && row0 + tid < n) {
        float *t = wk.rn + (size_t)task * n + row0 + tid;
        const float s = fmaf((s_rn[0][tid] + s_rn[1][tid]) + (s_rn[2][tid] + s_rn[3][tid]), 0x1p-40f, k0 ? *t : 0.0f);
        *t = s;
        over |= s > FIX_ROW || (s_any[1][1] | s_any[1][2]) >> 22;
    }
    if (over) atomicOr(status + task, ST_ERR_PIVOT);
    if (ok) {
        const int r = quad * 32 + lane, blk = blockIdx.x * 2 + rb; // row block below the diagonal block
        // digits that are zero in both blocks of the pair are not read
        const int f = first_digit((unsigned long long)(s_any[1][1] | s_any[1][2]) << 32 | (s_any[0][1] | s_any[0][2]));
        const size_t dst = (size_t)(fix_nbk(n) + 1) * IMG_BLK;          // digit to digit
        unsigned char *img = wk.ximg(task, n) + (size_t)blk * IMG_BLK;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            long long x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) x[u] = v[q * 8 + u];
            uint4 d[ND];
            split8(x, d);
#pragma unroll
            for (int i = 0; i < ND; i++)
                if (i >= f) *reinterpret_cast<uint4 *>(img + i * dst + img_off(r & 63, part * 2 + q)) = d[i];
        }
    } else if (lane == 0)
        atomicOr(status + task, ST_ERR_WAIT);
    // a wait that ran out leaves MMAs in flight: wait for the last of them (bounded)
    // before the tensor memory goes
    if (tid == 0 && have && !ok) umma::mbar_wait(&gfull[1], 0, FIX_WAIT_ITERS);
    if (warp == 0) { // every warp has read its accumulators (the barrier above)
        umma::fence_after();
        umma::dealloc(tmem, 512);
    }
}

// ---------------------------------------------------------------------------
// trailing update: S -= X X^T
// ---------------------------------------------------------------------------
// A CTA takes one pair of row blocks (128 rows) against up to `chunk` 64-column blocks: the rows'
// digits (96 KB) stay in shared memory, the columns' (48 KB) come in two stages.  Warp 16 copies,
// warp 17 issues the MMAs (104 of 128 x 64 x 16 per tile), warps 0..15 fold and update S (lane
// quadrant warp mod 4, 16 of the 64 columns).  The accumulators are handed over in two parts, groups 0..3 (40
// MMAs) and 4..6 (64), each folded while the MMAs of the other run (with a hand-over per group and a
// ring of eight accumulators the hand-overs alone took 2.6 us per tile).
constexpr int SY_EPI = 16, SY_THREADS = (SY_EPI + 2) * 32;
constexpr int SY_SMEM = TR_A + 2 * TR_B; // 192 KB
__global__ void __launch_bounds__(SY_THREADS, 1) k_fix_syrk(int ntask, int n, int t0, int jlo, int jhi, int chunk, long long *S, size_t lda, size_t mstride,
                                                            int *status, FixWork wk)
{
    const int task = blockIdx.y;
    // (the next diagonal block, on another stream, may mark the matrix meanwhile: one decision for the block)
    if (task >= ntask || !__syncthreads_and((status[task] & ~ST_ERR_WAIT) == ST_FACTOR)) return;
    // item -> row pair p (largest first) and its column blocks [j0, j1)
    const int nbt = (n - t0 + NB - 1) / NB, np = (nbt + 1) / 2;
    int p = np - 1, it = blockIdx.x;
    for (; p >= 0; p--) {
        const int items = (max(min(min(2 * p + 2, nbt), jhi) - jlo, 0) + chunk - 1) / chunk;
        if (it < items) break;
        it -= items;
    }
    if (p < 0) return;
    const int j0 = jlo + it * chunk, j1 = min(j0 + chunk, min(min(2 * p + 2, nbt), jhi));
    // first nonzero digits of the rows and of column block j; tiles without a product are skipped
    const int *first = wk.first + (size_t)task * (fix_nbk(n) + 1);
    const int fa = 2 * p + 1 < nbt ? min(first[2 * p], first[2 * p + 1]) : first[2 * p];
    bool any = false;
    for (int j = j0; j < j1; j++) any |= fa + first[j] < NG;
    if (!any) return; // uniform: nothing writes first in this launch
    extern __shared__ __align__(1024) unsigned char sy_sm[];
    __shared__ uint64_t afull, bfull[2], bempty[2], sfull[2], sempty[2], drain;
    __shared__ uint32_t tslot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) umma::alloc(&tslot, 512);
    if (tid == 0) {
        umma::mbar_init(&afull, 1);
        for (int i = 0; i < 2; i++) {
            umma::mbar_init(&bfull[i], 1);
            umma::mbar_init(&bempty[i], 1);
            umma::mbar_init(&sfull[i], 1);
            umma::mbar_init(&sempty[i], SY_EPI);
        }
        umma::mbar_init(&drain, 1);
    }
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tslot, 0);
    if (warp < SY_EPI) {
        const int quad = warp & 3, part = warp >> 2;
        const int R = t0 + p * 128 + quad * 32 + lane;
        long long *Sm = S + (size_t)task * mstride + R;
        int q = 0; // tiles so far
        for (int j = j0; j < j1; j++) {
            const int s0 = fa + first[j];
            if (s0 >= NG) continue;
            const int c0 = t0 + j * NB + part * 16;
            const int jm = R < n ? min(n - c0, R - c0 + 1) : 0; // columns c0 .. c0 + jm - 1 of this row
            unsigned long long *dst = reinterpret_cast<unsigned long long *>(Sm + (size_t)c0 * lda);
            long long v[16];
#pragma unroll
            for (int c = 0; c < 16; c++) v[c] = 0;
            bool ok = true;
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                ok = ok && umma::mbar_wait(&sfull[h], q & 1, FIX_WAIT_ITERS);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                umma::fence_after();
#pragma unroll 1
                for (int g = max(s0, h ? SY_G0 : 0); g < (h ? NG : SY_G0); g++)
                    fold_group(tmem + ((uint32_t)(quad * 32) << 16) + g * NB + part * 16, g, s0, v);
                umma::fence_before();
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::smem_u32(&sempty[h])) : "memory");
            }
            if (!ok) {
                if (lane == 0) atomicOr(status + task, ST_ERR_WAIT);
                break;
            }
            // the subtraction as an atomic add at the L2 cache: exact in integers, and no load's latency
            // stands between the accumulators and the next tile (loads and stores: 287 us for the second
            // panel of 24 matrices of dimension 2100)
#pragma unroll
            for (int c = 0; c < 16; c++)
                if (c < jm) atomicAdd(dst + (size_t)c * lda, 0ULL - (unsigned long long)v[c]);
            q++;
        }
    } else if (warp == SY_EPI) {
        if (lane == 0) {
            const unsigned char *img = wk.ximg(task, n);
            const size_t dstep = (size_t)(fix_nbk(n) + 1) * IMG_BLK;
            umma::mbar_arrive_tx(&afull, (ND - fa) * 2 * IMG_BLK);
            for (int i = fa; i < ND; i++) umma::bulk_g2s(sy_sm + i * 2 * IMG_BLK, img + i * dstep + (size_t)2 * p * IMG_BLK, 2 * IMG_BLK, &afull);
            int last[2] = {-1, -1}, q = 0;
            for (int j = j0; j < j1; j++) {
                const int fb = first[j];
                if (fa + fb >= NG) continue;
                const int s = q & 1, u = q >> 1;
                if (u > 0 && !umma::mbar_wait(&bempty[s], (u - 1) & 1, FIX_WAIT_ITERS)) {
                    atomicOr(status + task, ST_ERR_WAIT);
                    break;
                }
                umma::mbar_arrive_tx(&bfull[s], (ND - fb) * IMG_BLK);
                for (int i = fb; i < ND; i++)
                    umma::bulk_g2s(sy_sm + TR_A + s * TR_B + i * IMG_BLK, img + i * dstep + (size_t)j * IMG_BLK, IMG_BLK, &bfull[s]);
                last[s] = u;
                q++;
            }
            // no copy may be in flight when the CTA leaves
            umma::mbar_wait(&afull, 0, FIX_WAIT_ITERS);
            for (int s = 0; s < 2; s++)
                if (last[s] >= 0) umma::mbar_wait(&bfull[s], last[s] & 1, FIX_WAIT_ITERS);
        }
    } else if (lane == 0) {
        const uint32_t a = umma::desc_lo(umma::smem_u32(sy_sm), 128);
        bool ok = umma::mbar_wait(&afull, 0, FIX_WAIT_ITERS);
        for (int j = j0, q = 0; ok && j < j1; j++) {
            const int fb = first[j], s = q & 1, u = q >> 1;
            if (fa + fb >= NG) continue;
            ok = umma::mbar_wait(&bfull[s], u & 1, FIX_WAIT_ITERS);
            umma::fence_after();
            for (int h = 0; ok && h < 2; h++) {
                if (q > 0) ok = umma::mbar_wait(&sempty[h], (q - 1) & 1, FIX_WAIT_ITERS);
                if (!ok) break;
                umma::fence_after();
                const uint32_t b = a + (TR_A + s * TR_B) / 16;
                mma_nonzero(tmem, a, b, fa, fb, h ? SY_G0 : 0, h ? NG : SY_G0);
                umma::commit(&sfull[h]);
            }
            umma::commit(&bempty[s]);
            q++;
        }
        if (!ok) atomicOr(status + task, ST_ERR_WAIT);
        // every MMA this thread issued completes before the CTA frees tensor memory
        umma::commit(&drain);
        umma::mbar_wait(&drain, 0, FIX_WAIT_ITERS);
    }
    umma::fence_before();
    __syncthreads();
    if (warp == 0) {
        umma::fence_after();
        umma::dealloc(tmem, 512);
    }
}

// log det and the post-checks of kernel_logdet (matrix.c:78-82, :144-145): one warp per task adds
// the diagonal blocks' sums (Kahan per lane, then the lanes in order)
__global__ void k_final(int ntask, int n, const double *logdet, const FixInfo *info, const double *trace, int *status, double *result,
                        int mode)
{
    const int task = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (task >= ntask) return;
    const int st = status[task];
    if (st & ~0xF) { if (lane == 0) result[task] = NAN; return; }
    if (st != ST_FACTOR) return; // trace or Mercator result already stored
    const int nbk = fix_nbk(n);
    double s = 0.0, c = 0.0;
    for (int j = lane; j < nbk; j += 32) {
        const double y = logdet[(size_t)task * nbk + j] - c;
        const double t = s + y;
        c = (t - s) - y;
        s = t;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane != 0) return;
    double ld = 2.0 * s + n * (LN2 * info[task].sexp);
    if (mode == 1 && fabs(trace[task]) > fabs(ld)) ld = -trace[task];
    result[task] = ld;
}

// the exponents first (launch_fix_scale), then the digit table, the rows' squares, the images
static size_t fix_info_bytes(int ntask) { return ((size_t)ntask * sizeof(FixInfo) + 255) & ~(size_t)255; }
static size_t fix_first_bytes(int ntask, int n) { return ((size_t)2 * ntask * (fix_nbk(n) + 1) * sizeof(int) + 255) & ~(size_t)255; }
static size_t fix_rn_bytes(int ntask, int n) { return ((size_t)ntask * n * sizeof(float) + 255) & ~(size_t)255; }

size_t cholesky_work_bytes(int ntask, int n)
{
    return fix_info_bytes(ntask) + fix_first_bytes(ntask, n) + fix_rn_bytes(ntask, n) + (size_t)ntask * fix_task_bytes(n);
}

FixWork fix_work(int ntask, int n, void *work)
{
    unsigned char *w = (unsigned char *)work, *first = w + fix_info_bytes(ntask), *rn = first + fix_first_bytes(ntask, n);
    return FixWork{rn + fix_rn_bytes(ntask, n), (FixInfo *)w, (int *)first, (float *)rn, 0};
}

static int fix_sms()
{
    static int sms = 0;
    if (!sms) {
        CK(cudaFuncSetAttribute(k_fix_potf2, cudaFuncAttributeMaxDynamicSharedMemorySize, PF_SMEM));
        CK(cudaFuncSetAttribute(k_fix_trsm, cudaFuncAttributeMaxDynamicSharedMemorySize, TR_SMEM));
        CK(cudaFuncSetAttribute(k_fix_syrk, cudaFuncAttributeMaxDynamicSharedMemorySize, SY_SMEM));
        sms = device_sms();
    }
    return sms;
}

void fix_convert(int ntask, int n, double *A, size_t lda, size_t mstride, int *status, const double *mdiag, const FixWork &wk,
                 cudaStream_t st)
{
    k_fix_convert<<<dim3((n + 7) / 8, ntask), 256, 0, st>>>(ntask, n, A, lda, mstride, status, mdiag, wk.info);
    COUNT_LAUNCH(1);
}

void fix_syrk(int ntask, int n, int t0, long long *S, size_t lda, size_t mstride, int *status, const FixWork &wk, cudaStream_t st, int jlo,
              int jhi)
{
    // tiles per CTA: about three CTAs per SM where the batch is small, at most 8 tiles
    const int nbt = (n - t0 + NB - 1) / NB, np = (nbt + 1) / 2;
    auto cols = [&](int p) { return std::max(std::min({2 * p + 2, nbt, jhi}) - jlo, 0); };
    long long tiles = 0;
    for (int p = 0; p < np; p++) tiles += cols(p);
    const int chunk = (int)std::max(1LL, std::min(8LL, tiles * ntask / (3LL * fix_sms())));
    int items = 0;
    for (int p = 0; p < np; p++) items += (cols(p) + chunk - 1) / chunk;
    if (items == 0) return;
    k_fix_syrk<<<dim3(items, ntask), SY_THREADS, SY_SMEM, st>>>(ntask, n, t0, jlo, jhi, chunk, S, lda, mstride, status, wk);
    COUNT_LAUNCH(1);
}

void launch_cholesky(int ntask, int n, double *A, size_t lda, size_t mstride, int *status, const double *mdiag, double *logdet, void *work,
                     cudaStream_t st, bool fixed, const TwoStreams *two)
{
    fix_sms();
    FixWork wk = fix_work(ntask, n, work);
    int *const first = wk.first;
    long long *S = reinterpret_cast<long long *>(A);
    // grid y is at most 65535: every caller's chunk is
    if (!fixed) fix_convert(ntask, n, A, lda, mstride, status, mdiag, wk, st);
    // The next diagonal block and panel need the first column block of an update only.  With a second stream, of high
    // priority, they go on there, and the rest of the update follows on the caller's beside them, up to the panel
    // after the next: factorisation of 24 matrices of dimension 2100 2.32 -> 2.02 ms, 4 of 5000 5.16 -> 4.45, of the free
    // energy at R/L = 100 8.87 -> 8.51, 32 of 700 0.66 -> 0.63.  Where an update is a few tiles the split and the
    // events cost more (one of 280 0.23 -> 0.25), so it takes more than eight blocks.  Integer additions
    // commute: the values are the same either way.
    const bool ahead = two && n > 8 * NB;
    const cudaStream_t cs = ahead ? two->stream : st;
    if (ahead) {
        CK(cudaEventRecord(two->ev[2], st));
        CK(cudaStreamWaitEvent(cs, two->ev[2], 0));
    }
    for (int k0 = 0, k = 0; k0 < n; k0 += NB, k++) {
        wk.par = k & 1;
        wk.first = first + (size_t)wk.par * ntask * (fix_nbk(n) + 1);
        // the update before the last has written this column
        if (ahead && k >= 2) CK(cudaStreamWaitEvent(cs, two->ev[wk.par], 0));
        k_fix_potf2<<<ntask, PF_NT, PF_SMEM, cs>>>(ntask, n, k0, S, lda, mstride, status, wk, logdet);
        COUNT_LAUNCH(1);
        const int t0 = k0 + NB, rest = n - t0;
        if (rest <= 0) break;
        k_fix_trsm<<<dim3((rest + 127) / 128, ntask), TR_NT, TR_SMEM, cs>>>(ntask, n, k0, S, lda, mstride, status, wk);
        COUNT_LAUNCH(1);
        if (!ahead) {
            fix_syrk(ntask, n, t0, S, lda, mstride, status, wk, cs);
            continue;
        }
        CK(cudaEventRecord(two->ev[2], cs));
        CK(cudaStreamWaitEvent(st, two->ev[2], 0));
        fix_syrk(ntask, n, t0, S, lda, mstride, status, wk, cs, 0, 1);
        fix_syrk(ntask, n, t0, S, lda, mstride, status, wk, st, 1);
        CK(cudaEventRecord(two->ev[wk.par], st));
    }
    if (ahead) {
        CK(cudaEventRecord(two->ev[2], cs));
        CK(cudaStreamWaitEvent(st, two->ev[2], 0));
    }
    CK(cudaGetLastError());
}

void launch_fix_scale(const int *tlist, int nlist, int n, const double *mdiag, void *work, cudaStream_t st)
{
    if (nlist <= 0) return;
    k_fix_scale<<<(nlist + 3) / 4, 128, 0, st>>>(tlist, nlist, n, mdiag, (FixInfo *)work);
    COUNT_LAUNCH(1);
    CK(cudaGetLastError());
}

void launch_final(int ntask, int n, const double *logdet, const void *work, const double *trace, int *status, double *result, int mode,
                  cudaStream_t st)
{
    k_final<<<(ntask + 3) / 4, 128, 0, st>>>(ntask, n, logdet, (const FixInfo *)work, trace, status, result, mode);
    COUNT_LAUNCH(1);
    CK(cudaGetLastError());
}

} // namespace capsgpu
