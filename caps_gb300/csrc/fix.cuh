// fix.cuh -- 64-bit fixed-point matrices as FP16 digit images, shared by the Cholesky factorisation
// (cholesky.cu, which explains the format) and the square of M (square.cu)
#pragma once
#include "common.cuh"
#include <cuda_fp16.h>

namespace capsgpu {

constexpr int NB = 64;
constexpr int FQ = 60;                       // fixed point: value = integer 2^-60
constexpr int ND = 6, NG = 7;                // digits of a factor, accumulators (i + j = 0..6)
constexpr int SY_G0 = 4;                     // accumulators of a first part, see k_fix_syrk
constexpr int IMG_BLK = NB * NB * 2;         // bytes of one digit of one 64 x 64 block
constexpr int FIX_WAIT_ITERS = 1 << 22;      // polls of a bounded mbarrier wait

// per-task workspace: W image, two X images (panels alternate; one digit after the other, a spare row block so
// that a pair of row blocks can always be read), exponents
__host__ __device__ inline int fix_nbk(int n) { return (n + NB - 1) / NB; }
__host__ __device__ inline size_t fix_ximg_bytes(int n) { return (size_t)(fix_nbk(n) + 1) * ND * IMG_BLK; }
__host__ __device__ inline size_t fix_task_bytes(int n) { return (size_t)ND * IMG_BLK + 2 * fix_ximg_bytes(n); }
struct FixInfo { int sexp, wexp; };          // A 2^-sexp is factored; W 2^-wexp is in the image
// first[task * (nbk + 1) + block] (one table per image): the first digit of the panel's X that is not zero in the whole 64-row
// block (block counted below the diagonal block; NG: none)
// rn[task * n + row]: squares of a row's part of the factor so far
struct FixWork {
    unsigned char *img;
    FixInfo *info;
    int *first;
    float *rn;
    int par; // the image in use
    __host__ __device__ unsigned char *wimg(int task, int n) const { return img + (size_t)task * fix_task_bytes(n); }
    __host__ __device__ unsigned char *ximg(int task, int n) const { return wimg(task, n) + (size_t)ND * IMG_BLK + par * fix_ximg_bytes(n); }
};

// byte offset of element (row, k) inside one digit of a 64-row block: the operand layout of
// umma.cuh (8 x 16-byte core matrices), k innermost, 1024 bytes per 8 rows
CAPS_DEV int img_off(int row, int kcore) { return (row >> 3) * 1024 + kcore * 128 + (row & 7) * 16; }

// ---- digits ----
// the magnitude of x (units of 2^-60) as digits see it, in units of 2^-53: its bit length bounds the digits
// that are not zero (k digits hold +-255 (512^k - 1) / 511)
CAPS_DEV unsigned long long digit_mag(long long x)
{
    const long long y = (x + 64) >> 7;
    return (unsigned long long)(y < 0 ? -y : y);
}
// first digit that may be nonzero, from the bitwise or of magnitudes; NG: none is
CAPS_DEV int first_digit(unsigned long long any)
{
    const int bits = 64 - __clzll((long long)any);
    return bits == 0 ? NG : bits <= 8 ? 5 : bits <= 16 ? 4 : bits <= 25 ? 3 : bits <= 34 ? 2 : bits <= 43 ? 1 : 0;
}

// Conversions.  Per warp, F2I holds its scheduler for 13 clocks and a conversion of 64-bit integers the FP64 pipe of
// the SM for 25; adding 1.5 2^23 leaves an integer below 2^22 in the low bits of an FP32 number.
constexpr float FX_MAGIC = 12582912.0f;
constexpr unsigned FX_MBITS = 0x4B400000u;
// to the nearest integer, |x| < 2^31
CAPS_DEV int fx_f2i(float x)
{
    const float h = fmaf(x, 0x1p-12f, FX_MAGIC), l = fmaf(h - FX_MAGIC, -0x1p12f, x) + FX_MAGIC;
    return ((__float_as_int(h) - (int)FX_MBITS) << 12) + (__float_as_int(l) - (int)FX_MBITS);
}
// x 2^-60 to 2^-23 relative
CAPS_DEV float fx_value(long long x)
{
    return fmaf((float)(int)((x + 0x80000000LL) >> 32), 0x1p-28f, (float)(int)x * 0x1p-60f);
}

// v in units of 2^-q, rounded, saturated at +-2^62 (integer work only).  err: status bits; a matrix whose diagonal is
// below 2 and that has an entry of 2 or more is not positive definite
CAPS_DEV long long to_fix(double v, int q, int &err)
{
    const long long b = __double_as_longlong(v);
    const int ex = (int)((b >> 52) & 0x7ff);
    const int sh = ex - 1075 + q;
    if (sh >= 9) err |= ex == 0x7ff ? ST_ERR_NONFINITE : ST_ERR_PIVOT; // |v| >= 2^61 units
    long long mnt = (b & 0xfffffffffffffLL) | (1LL << 52);
    if (sh >= 10) mnt = 1LL << 62;
    else if (sh >= 0) mnt <<= sh;
    else mnt = sh < -54 ? 0 : (mnt + (1LL << (-sh - 1))) >> -sh;
    return b < 0 ? -mnt : mnt;
}

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
            f[u][0] = (unsigned)min(max((int)(t >> 45), -1023), 1023);
        }
        {
            // 1024 + |top| is 0x6400 | |top| (the conversion instruction takes 12 clocks of a scheduler per warp)
            const unsigned raw = (unsigned)abs((int)f[0][0]) | (unsigned)abs((int)f[1][0]) << 16 | 0x64006400u;
            const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&raw), __half2half2(__ushort_as_half(0x6400)));
            w[0][p] = *reinterpret_cast<const unsigned *>(&h) | (f[0][0] >> 16 & 0x8000u) | (f[1][0] & 0x80000000u);
        }
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

// cholesky.cu: the parts of a workspace of cholesky_work_bytes; FP64 -> fixed point in place, with the exponents;
// S -= X X^T over the rows and columns from t0 on, X the 64 columns in the image, first digits in wk.first; column
// blocks j0 .. j1 - 1 of it
FixWork fix_work(int ntask, int n, void *work);
void fix_convert(int ntask, int n, double *A, size_t lda, size_t mstride, int *status, const double *mdiag, const FixWork &wk,
                 cudaStream_t st);
void fix_syrk(int ntask, int n, int t0, long long *S, size_t lda, size_t mstride, int *status, const FixWork &wk, cudaStream_t st,
              int j0 = 0, int j1 = 1 << 30);

} // namespace capsgpu
