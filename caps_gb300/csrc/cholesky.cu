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
//  * products with 64 columns (panel solve, trailing update) run on the tensor cores.  A factor x
//    is split into six signed 9-bit digits, x = sum_i d_i 2^(-8-9i), exact as FP16; the MMAs
//    (kind::f16, FP32 accumulators) form sum_k d_i(k) d_j(k) as exact integers in one accumulator
//    per i + j = 0..6, and the epilogue adds the accumulators up as 64-bit integers.  Digit
//    products with i + j > 6 are below 2^-60 and left out, so the error of a product is that
//    of the last digit, 2^-54 per factor -- an FP64 sum of 64 products has 2^-53 of its
//    partial sums at every step.
//  * the 64 x 64 diagonal blocks (factor and inverse) run on the integer pipes: a number is
//    h 2^30 + l, and a product needs three 32 x 32 -> 64 bit multiply-adds (h h, h l, l h).
//
// Per 64 columns three launches over the batch: k_fix_potf2 (diagonal block, W = L_kk^-1 as digit
// images, log det), k_fix_trsm (X = S W^T for the rows below, stored as digit images only),
// k_fix_syrk (S -= X X^T).  log det A = 2 sum_j log L_jj.  A non-positive pivot marks the task
// (ST_ERR_PIVOT) and its result becomes NaN; nothing traps.  A matrix whose diagonal exceeds 2
// (M with large negative diagonal entries) is scaled by a power of four on conversion.
#include "common.cuh"
#include "internal.h"
#include "umma.cuh"
#include <algorithm>
#include <cuda_fp16.h>

namespace capsgpu {

constexpr int NB = 64;
constexpr int FQ = 60;                       // fixed point: value = integer 2^-60
constexpr int ND = 6, NG = 7;                // digits of a factor, accumulators (i + j = 0..6)
constexpr int IMG_BLK = NB * NB * 2;         // bytes of one digit of one 64 x 64 block
constexpr int FIX_WAIT_ITERS = 1 << 22;      // polls of a bounded mbarrier wait

// per-task workspace: W image, X image (one digit after the other, a spare row block so that a
// pair of row blocks can always be read), exponents
__host__ __device__ inline int fix_nbk(int n) { return (n + NB - 1) / NB; }
__host__ __device__ inline size_t fix_ximg_bytes(int n) { return (size_t)(fix_nbk(n) + 1) * ND * IMG_BLK; }
__host__ __device__ inline size_t fix_task_bytes(int n) { return (size_t)ND * IMG_BLK + fix_ximg_bytes(n); }
struct FixInfo { int sexp, wexp; };          // A 2^-sexp is factored; W 2^-wexp is in the image
struct FixWork {
    unsigned char *img;
    FixInfo *info;
    __host__ __device__ unsigned char *wimg(int task, int n) const { return img + (size_t)task * fix_task_bytes(n); }
    __host__ __device__ unsigned char *ximg(int task, int n) const { return wimg(task, n) + (size_t)ND * IMG_BLK; }
};

// byte offset of element (row, k) inside one digit of a 64-row block: the operand layout of
// umma.cuh (8 x 16-byte core matrices), k innermost, 1024 bytes per 8 rows
CAPS_DEV int img_off(int row, int kcore) { return (row >> 3) * 1024 + kcore * 128 + (row & 7) * 16; }

// ---- digits ----
// eight numbers (units of 2^-60, |x| < 4) to six 16-byte vectors of FP16 digits
CAPS_DEV void split8(const long long (&x)[8], uint4 (&d)[ND])
{
    const __half2 off = __half2half2(__ushort_as_half(0x6500)); // 1280
    unsigned w[ND][4];
#pragma unroll
    for (int p = 0; p < 4; p++) {
        unsigned f[2][ND];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            // round to units of 2^-53 and bias the five low digits by 256, so that they are plain bit fields
            constexpr long long BIAS = 256LL * (1 + (1LL << 9) + (1LL << 18) + (1LL << 27) + (1LL << 36));
            const long long t = ((x[2 * p + u] + 64) >> 7) + BIAS;
#pragma unroll
            for (int i = 1; i < ND; i++) f[u][i] = (unsigned)(t >> (9 * (5 - i))) & 511u;
            const int top = (int)(t >> 45);
            f[u][0] = __half_as_ushort(__int2half_rn(min(max(top, -2047), 2047)));
        }
        w[0][p] = f[0][0] | f[1][0] << 16;
#pragma unroll
        for (int i = 1; i < ND; i++) {
            // 0x6400 | u is 1024 + u in FP16
            const unsigned raw = (f[0][i] | f[1][i] << 16) | 0x64006400u;
            const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&raw), off);
            w[i][p] = *reinterpret_cast<const unsigned *>(&h);
        }
    }
#pragma unroll
    for (int i = 0; i < ND; i++) d[i] = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
}

// the MMAs of group s = i + j of one 128 x 64 tile, K = 64: A digits 16 KB apart, B digits 8 KB
CAPS_DEV void mma_group(uint32_t acc, uint32_t a, uint32_t b, int s)
{
    constexpr uint32_t idesc = umma::idesc_f16(128, 64);
    bool first = true;
    for (int i = s > ND - 1 ? s - ND + 1 : 0; i <= s && i < ND; i++) {
        const uint32_t ai = a + i * 2 * IMG_BLK, bj = b + (s - i) * IMG_BLK;
#pragma unroll
        for (int ks = 0; ks < 4; ks++) {
            umma::mma_f16(acc, umma::desc_kmajor(ai + ks * 256, 128, 1024), umma::desc_kmajor(bj + ks * 256, 128, 1024), idesc, !first);
            first = false;
        }
    }
}

// NC columns of group s of this warp's lanes folded into v (units of 2^-60 once s = 0 is in);
// groups come in the order s = 6, 5, ..., 0, of weight 2^(44 - 9 s)
template <int NC> CAPS_DEV void fold_group(uint32_t taddr, int s, long long (&v)[NC])
{
#pragma unroll
    for (int h = 0; h < NC / 16; h++) {
        float f[16];
        umma::ld16(taddr + h * 16, f);
#pragma unroll
        for (int c = 0; c < 16; c++) {
            const int g = __float2int_rn(f[c]);
            long long &a = v[h * 16 + c];
            switch (s) { // uniform, constant after unrolling
            case 6: a = g; break;
            case 5: a += (long long)g * 512; break;
            case 4: a = (a + (long long)g * 262144 + 512) >> 10; break;
            case 3: a += (long long)g * (1 << 17); break;
            case 2: a += (long long)g * (1 << 26); break;
            case 1: a += (long long)((unsigned long long)(unsigned)(g * 8) << 32); break;
            default: a += (long long)((unsigned long long)(unsigned)(g * 4096) << 32); break;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// FP64 -> fixed point, in place (lower triangle)
// ---------------------------------------------------------------------------
// scale exponent of a matrix whose largest diagonal entry is mx: none below 2, else a power of four
CAPS_DEV int fix_sexp(double mx) { return mx >= 2.0 ? min(2 * ((ilogb(mx) + 2) / 2), 400) : 0; }

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
__global__ void __launch_bounds__(256) k_fix_convert(int ntask, int n, double *A, size_t lda, size_t mstride, const int *status,
                                                     const double *mdiag, FixInfo *info)
{
    const int task = blockIdx.y;
    if (task >= ntask || status[task] != ST_FACTOR) return;
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
    for (int c = blockIdx.x * 8; c < min(n, (int)blockIdx.x * 8 + 8); c++) {
        double *col = A + (size_t)task * mstride + (size_t)c * lda;
        for (int r = c + threadIdx.x; r < n; r += 256) {
            const double v = fmin(fmax(col[r] * sc, -0x1.fp61), 0x1.fp61);
            reinterpret_cast<long long *>(col)[r] = __double2ll_rn(v);
        }
    }
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

// one CTA of 256 threads per matrix.  L_kk and W = L_kk^-1 of the 64 x 64 block at k0 (past the
// matrix: the identity), W as digit images in the operand layout, sum of log L_jj into
// logdet[task * nbk + block].
//
// In 16-column sub-panels.  Warps 0..2: every warp holds the sub-panel's 16 diagonal rows in
// lanes 0..15 (all three compute them alike, so no warp waits for another) and 16 of the up to 48
// rows below in lanes 16..31, a row of 16 entries in registers; column j's entries reach the
// warp by shuffles.  Then all warps apply the rank-16 update to the rest of the triangle, in
// 2 x 2 tiles.  W: the four 16 x 16 diagonal blocks by substitution, one lane per column, then
// X_ij = -X_ii sum_k L_ik X_kj by distance from the diagonal.  Bound by the pivot chain (about
// 200 clocks per column: reciprocal square root, product, shuffle, multiply-add) and the
// 32-bit multipliers.
constexpr int PP = NB + 1;
__global__ void __launch_bounds__(256) k_fix_potf2(int ntask, int n, int k0, const long long *S, size_t lda, size_t mstride, int *status,
                                                   FixWork wk, double *logdet)
{
    const int task = blockIdx.x;
    if (task >= ntask || status[task] != ST_FACTOR) return;
    extern __shared__ __align__(16) unsigned char pf_sm[];
    long long *T = reinterpret_cast<long long *>(pf_sm);   // [64][PP]: the block, then L as limbs (int2)
    long long *W = T + NB * PP;                            // [64][PP]: W, units of 2^-wq
    int2 *Y = reinterpret_cast<int2 *>(W + NB * PP);       // [48][17] x 3 blocks: sums of a distance, as limbs
    __shared__ long long piv[NB], inv[NB];
    __shared__ int invk[NB];
    __shared__ unsigned long long smax;
    __shared__ double slog[2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nb = min(NB, n - k0);
    const long long *Sm = S + (size_t)task * mstride + (size_t)k0 * lda + k0;
    {
        long long v[16];
#pragma unroll
        for (int u = 0; u < 16; u++) {
            const int e = tid + 256 * u, c = e >> 6, r = e & 63;
            v[u] = (r >= c && r < nb && c < nb) ? Sm[(size_t)c * lda + r] : (r == c ? 1LL << FQ : 0LL);
        }
#pragma unroll
        for (int u = 0; u < 16; u++) {
            const int e = tid + 256 * u, c = e >> 6, r = e & 63;
            T[r * PP + c] = v[u];
        }
    }
    __syncthreads();
    int2 *Lm = reinterpret_cast<int2 *>(T);
    bool bad = false;
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
                if (live && row > o + j && (warp == 0 || lane >= 16)) Lm[row * PP + o + j] = xl;
                const int nh = -xl.y, nl = -xl.x;
#pragma unroll
                for (int c = j + 1; c < PB; c++) {
                    const int cl = __shfl_sync(0xffffffffu, xl.x, c), ch = __shfl_sync(0xffffffffu, xl.y, c);
                    s[c] += (long long)nh * ch;
                    b[c] += (long long)nh * cl;
                    b[c] += (long long)nl * ch;
                }
            }
        }
        __syncthreads();
        const int c0 = o + PB, t2 = (NB - c0) / 2; // 2 x 2 tiles: rows and columns c0 + i, c0 + i + t2
        for (int e = tid; e < t2 * (t2 + 1) / 2; e += 256) {
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
        if (tid == 0) smax = 0;
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
            for (int e = tid; e < np * 256; e += 256) {
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
            for (int e = tid; e < np * 256; e += 256) {
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
    unsigned long long mx = 0;
    for (int e = tid; e < NB * NB; e += 256) {
        const int r = e >> 6, c = e & 63;
        if (c <= r) {
            const long long v = W[r * PP + c];
            mx = max(mx, (unsigned long long)(v < 0 ? -v : v));
        }
    }
    atomicMax(&smax, mx);
    __syncthreads();
    // image: W 2^-wexp in units of 2^-60, below 3.9 (the top digit stays below 1024)
    int wexp = 0;
    while (wexp < 40 && ldexp((double)smax, -wq - wexp) > 3.9) wexp++;
    unsigned char *img = wk.wimg(task, n);
    const int sh = FQ - wq - wexp;
    for (int e = tid; e < NB * 8; e += 256) {
        const int j = e & 63, kc = e >> 6;
        long long x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int c = kc * 8 + u;
            const long long v = c <= j ? W[j * PP + c] : 0;
            x[u] = sh >= 0 ? v << sh : (v + (1LL << (-sh - 1))) >> -sh;
        }
        uint4 d[ND];
        split8(x, d);
#pragma unroll
        for (int i = 0; i < ND; i++) *reinterpret_cast<uint4 *>(img + i * IMG_BLK + img_off(j, kc)) = d[i];
    }
    const int anybad = __syncthreads_or(bad);
    if (tid == 0) {
        wk.info[task].wexp = wexp;
        logdet[(size_t)task * fix_nbk(n) + k0 / NB] = 0.5 * (slog[0] + slog[1]);
        if (anybad) atomicOr(status + task, ST_ERR_PIVOT);
    }
}
constexpr int POTF2_SMEM = NB * PP * 16 + 3 * 16 * 17 * 8;

// ---------------------------------------------------------------------------
// panel solve: X = S W^T for 128 rows below the diagonal block
// ---------------------------------------------------------------------------
// grid (ceil(rows / 128), ntask), 256 threads, 144 KB of shared memory.  The threads split the
// rows of S into digits while the digits of W arrive by bulk copies; one thread issues the
// MMAs of each group, and all warps fold the accumulators (lane quadrant warp mod 4, 32 of
// the 64 columns), split X and store its images.  Rows past n are zero.
constexpr int TR_A = ND * 2 * IMG_BLK, TR_B = ND * IMG_BLK; // 96 KB, 48 KB
constexpr int TR_SMEM = TR_A + TR_B;
__global__ void __launch_bounds__(256) k_fix_trsm(int ntask, int n, int k0, const long long *S, size_t lda, size_t mstride, int *status,
                                                  FixWork wk)
{
    const int task = blockIdx.y;
    if (task >= ntask || (status[task] & ~ST_ERR_WAIT) != ST_FACTOR) return; // a wait error of this launch is masked: uniform per block
    extern __shared__ __align__(1024) unsigned char tr_sm[];
    __shared__ uint64_t wfull, gfull[NG];
    __shared__ uint32_t tslot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row0 = k0 + NB + blockIdx.x * 128;
    if (warp == 0) umma::alloc(&tslot, 512);
    if (tid == 0) {
        umma::mbar_init(&wfull, 1);
        for (int g = 0; g < NG; g++) umma::mbar_init(&gfull[g], 1);
        umma::mbar_arrive_tx(&wfull, TR_B);
        umma::bulk_g2s(tr_sm + TR_A, wk.wimg(task, n), TR_B, &wfull);
    }
    const long long *Sm = S + (size_t)task * mstride;
    {
        const int r = tid & 127, R = row0 + r;
        for (int kc = tid >> 7; kc < 8; kc += 2) {
            long long x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) x[u] = R < n ? Sm[(size_t)(k0 + kc * 8 + u) * lda + R] : 0;
            uint4 d[ND];
            split8(x, d);
#pragma unroll
            for (int i = 0; i < ND; i++) *reinterpret_cast<uint4 *>(tr_sm + i * 2 * IMG_BLK + img_off(r, kc)) = d[i];
        }
    }
    umma::fence_smem_async();
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = tslot;
    const bool have = umma::mbar_wait(&wfull, 0, FIX_WAIT_ITERS);
    if (!have && tid == 0) atomicOr(status + task, ST_ERR_WAIT);
    bool ok = have;
    if (warp == 0 && have) {
        if (lane == 0) {
            const uint32_t a = umma::smem_u32(tr_sm), b = a + TR_A;
            for (int g = 0; g < NG; g++) {
                mma_group(tmem + g * NB, a, b, NG - 1 - g);
                umma::commit(&gfull[g]);
            }
        }
        __syncwarp();
    }
    const int quad = warp & 3, half = warp >> 2;
    long long v[32];
#pragma unroll
    for (int g = 0; g < NG; g++) {
        ok = ok && umma::mbar_wait(&gfull[g], 0, FIX_WAIT_ITERS);
        ok = __all_sync(0xffffffffu, ok);
        umma::fence_after();
        if (ok) fold_group(tmem + ((uint32_t)(quad * 32) << 16) + g * NB + half * 32, NG - 1 - g, v);
    }
    if (ok) {
        const int wexp = wk.info[task].wexp;
        const int r = quad * 32 + lane, blk = blockIdx.x * 2 + (r >> 6); // row block below the diagonal block
        const size_t dst = (size_t)(fix_nbk(n) + 1) * IMG_BLK;          // digit to digit
        unsigned char *img = wk.ximg(task, n) + (size_t)blk * IMG_BLK;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            long long x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) x[u] = v[q * 8 + u] << wexp;
            uint4 d[ND];
            split8(x, d);
#pragma unroll
            for (int i = 0; i < ND; i++) *reinterpret_cast<uint4 *>(img + i * dst + img_off(r & 63, half * 4 + q)) = d[i];
        }
    } else if (lane == 0)
        atomicOr(status + task, ST_ERR_WAIT);
    // a group's wait that ran out leaves its MMAs in flight: wait for the last of them (bounded)
    // before the tensor memory goes
    if (tid == 0 && have && !ok) umma::mbar_wait(&gfull[NG - 1], 0, FIX_WAIT_ITERS);
    umma::fence_before();
    __syncthreads();
    if (warp == 0) {
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
// quadrant warp mod 4, 16 of the 64 columns).  The 512
// columns of tensor memory are a ring of eight 64-column slots; a tile takes seven in turn, one
// per group, and a slot is free again once the epilogue has folded it, so that the MMAs of the
// next tile run under the epilogue of this one.
constexpr int SY_EPI = 16, SY_THREADS = (SY_EPI + 2) * 32, SY_SLOTS = 8;
constexpr int SY_SMEM = TR_A + 2 * TR_B; // 192 KB
__global__ void __launch_bounds__(SY_THREADS, 1) k_fix_syrk(int ntask, int n, int t0, int chunk, long long *S, size_t lda, size_t mstride,
                                                            int *status, FixWork wk)
{
    const int task = blockIdx.y;
    if (task >= ntask || (status[task] & ~ST_ERR_WAIT) != ST_FACTOR) return;
    // item -> row pair p (largest first) and its column blocks [j0, j1)
    const int nbt = (n - t0 + NB - 1) / NB, np = (nbt + 1) / 2;
    int p = np - 1, it = blockIdx.x;
    for (; p >= 0; p--) {
        const int items = (min(2 * p + 2, nbt) + chunk - 1) / chunk;
        if (it < items) break;
        it -= items;
    }
    if (p < 0) return;
    const int j0 = it * chunk, j1 = min(j0 + chunk, min(2 * p + 2, nbt));
    extern __shared__ __align__(1024) unsigned char sy_sm[];
    __shared__ uint64_t afull, bfull[2], bempty[2], sfull[SY_SLOTS], sempty[SY_SLOTS], drain;
    __shared__ uint32_t tslot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) umma::alloc(&tslot, 512);
    if (tid == 0) {
        umma::mbar_init(&afull, 1);
        for (int i = 0; i < 2; i++) {
            umma::mbar_init(&bfull[i], 1);
            umma::mbar_init(&bempty[i], 1);
        }
        for (int i = 0; i < SY_SLOTS; i++) {
            umma::mbar_init(&sfull[i], 1);
            umma::mbar_init(&sempty[i], SY_EPI);
        }
        umma::mbar_init(&drain, 1);
    }
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = tslot;
    if (warp < SY_EPI) {
        const int quad = warp & 3, part = warp >> 2;
        const int R = t0 + p * 128 + quad * 32 + lane;
        long long *Sm = S + (size_t)task * mstride + R;
        int use = 0;
        for (int j = j0; j < j1; j++) {
            const int c0 = t0 + j * NB + part * 16;
            const int jm = R < n ? min(n - c0, R - c0 + 1) : 0; // columns c0 .. c0 + jm - 1 of this row
            long long *dst = Sm + (size_t)c0 * lda;
            long long v[16];
            bool ok = true;
#pragma unroll
            for (int g = 0; g < NG; g++, use++) {
                const int slot = use % SY_SLOTS;
                ok = ok && umma::mbar_wait(&sfull[slot], (use / SY_SLOTS) & 1, FIX_WAIT_ITERS);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                umma::fence_after();
                fold_group(tmem + ((uint32_t)(quad * 32) << 16) + slot * NB + part * 16, NG - 1 - g, v);
                umma::fence_before();
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::smem_u32(&sempty[slot])) : "memory");
            }
            if (!ok) {
                if (lane == 0) atomicOr(status + task, ST_ERR_WAIT);
                break;
            }
            // the accumulators are free: these loads and stores run under the next tile's MMAs
#pragma unroll
            for (int h = 0; h < 2; h++) {
                long long cur[8];
#pragma unroll
                for (int c = 0; c < 8; c++) cur[c] = h * 8 + c < jm ? dst[(size_t)(h * 8 + c) * lda] : 0;
#pragma unroll
                for (int c = 0; c < 8; c++)
                    if (h * 8 + c < jm) dst[(size_t)(h * 8 + c) * lda] = cur[c] - v[h * 8 + c];
            }
        }
    } else if (warp == SY_EPI) {
        if (lane == 0) {
            const unsigned char *img = wk.ximg(task, n);
            const size_t dstep = (size_t)(fix_nbk(n) + 1) * IMG_BLK;
            umma::mbar_arrive_tx(&afull, TR_A);
            for (int i = 0; i < ND; i++) umma::bulk_g2s(sy_sm + i * 2 * IMG_BLK, img + i * dstep + (size_t)2 * p * IMG_BLK, 2 * IMG_BLK, &afull);
            int last[2] = {-1, -1};
            for (int j = j0; j < j1; j++) {
                const int q = j - j0, s = q & 1, u = q >> 1;
                if (u > 0 && !umma::mbar_wait(&bempty[s], (u - 1) & 1, FIX_WAIT_ITERS)) {
                    atomicOr(status + task, ST_ERR_WAIT);
                    break;
                }
                umma::mbar_arrive_tx(&bfull[s], TR_B);
                for (int i = 0; i < ND; i++)
                    umma::bulk_g2s(sy_sm + TR_A + s * TR_B + i * IMG_BLK, img + i * dstep + (size_t)j * IMG_BLK, IMG_BLK, &bfull[s]);
                last[s] = u;
            }
            // no copy may be in flight when the CTA leaves
            umma::mbar_wait(&afull, 0, FIX_WAIT_ITERS);
            for (int s = 0; s < 2; s++)
                if (last[s] >= 0) umma::mbar_wait(&bfull[s], last[s] & 1, FIX_WAIT_ITERS);
        }
    } else if (lane == 0) {
        const uint32_t a = umma::smem_u32(sy_sm);
        bool ok = umma::mbar_wait(&afull, 0, FIX_WAIT_ITERS);
        int use = 0;
        for (int j = j0; ok && j < j1; j++) {
            const int q = j - j0, s = q & 1, u = q >> 1;
            ok = umma::mbar_wait(&bfull[s], u & 1, FIX_WAIT_ITERS);
            umma::fence_after();
            for (int g = 0; ok && g < NG; g++, use++) {
                const int slot = use % SY_SLOTS;
                if (use >= SY_SLOTS) ok = umma::mbar_wait(&sempty[slot], (use / SY_SLOTS - 1) & 1, FIX_WAIT_ITERS);
                if (!ok) break;
                umma::fence_after();
                mma_group(tmem + slot * NB, a, a + TR_A + s * TR_B, NG - 1 - g);
                umma::commit(&sfull[slot]);
            }
            umma::commit(&bempty[s]);
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

size_t cholesky_work_bytes(int ntask, int n)
{
    const size_t info = ((size_t)ntask * sizeof(FixInfo) + 255) & ~(size_t)255;
    return info + (size_t)ntask * fix_task_bytes(n);
}

static FixWork fix_work(int ntask, void *work)
{
    const size_t info = ((size_t)ntask * sizeof(FixInfo) + 255) & ~(size_t)255;
    return FixWork{(unsigned char *)work + info, (FixInfo *)work};
}

void launch_cholesky(int ntask, int n, double *A, size_t lda, size_t mstride, int *status, const double *mdiag, double *logdet, void *work,
                     cudaStream_t st, bool fixed)
{
    static bool attr = false;
    static int sms = 148;
    if (!attr) {
        CK(cudaFuncSetAttribute(k_fix_potf2, cudaFuncAttributeMaxDynamicSharedMemorySize, POTF2_SMEM));
        CK(cudaFuncSetAttribute(k_fix_trsm, cudaFuncAttributeMaxDynamicSharedMemorySize, TR_SMEM));
        CK(cudaFuncSetAttribute(k_fix_syrk, cudaFuncAttributeMaxDynamicSharedMemorySize, SY_SMEM));
        int dev = 0;
        CK(cudaGetDevice(&dev));
        CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        attr = true;
    }
    const FixWork wk = fix_work(ntask, work);
    long long *S = reinterpret_cast<long long *>(A);
    // grid y is at most 65535: every caller's chunk is
    if (!fixed) {
        k_fix_convert<<<dim3((n + 7) / 8, ntask), 256, 0, st>>>(ntask, n, A, lda, mstride, status, mdiag, wk.info);
        COUNT_LAUNCH(1);
    }
    for (int k0 = 0; k0 < n; k0 += NB) {
        k_fix_potf2<<<ntask, 256, POTF2_SMEM, st>>>(ntask, n, k0, S, lda, mstride, status, wk, logdet);
        COUNT_LAUNCH(1);
        const int t0 = k0 + NB, rest = n - t0;
        if (rest <= 0) break;
        k_fix_trsm<<<dim3((rest + 127) / 128, ntask), 256, TR_SMEM, st>>>(ntask, n, k0, S, lda, mstride, status, wk);
        COUNT_LAUNCH(1);
        // tiles per CTA: about three CTAs per SM where the batch is small, at most 8 tiles
        const int nbt = (rest + NB - 1) / NB, np = (nbt + 1) / 2;
        long long tiles = 0;
        for (int p = 0; p < np; p++) tiles += std::min(2 * p + 2, nbt);
        const int chunk = (int)std::max(1LL, std::min(8LL, tiles * ntask / (3LL * sms)));
        int items = 0;
        for (int p = 0; p < np; p++) items += (std::min(2 * p + 2, nbt) + chunk - 1) / chunk;
        k_fix_syrk<<<dim3(items, ntask), SY_THREADS, SY_SMEM, st>>>(ntask, n, t0, chunk, S, lda, mstride, status, wk);
        COUNT_LAUNCH(1);
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
