// square.cu -- the sphere-sphere round trip (the reference's cass.c:23-64).
//
// For two equal spheres at separation d the round-trip operator is M^2, with M the
// plane-sphere round trip at L = d/2, and the reference takes log det(1 - M^2) from the
// dense matrix M^2 = M M (matrix_mult + matrix_logdet_dense, cass.c:42-60).  Here the
// batch already holds A = 1 - M (lower triangle) and M_ii.  M is symmetric, so 1 - M^2 = 1 - M M^T is
// what the trailing update of the fixed-point Cholesky computes, with the columns of M in the place of a
// panel: per 64 columns k_sq_image writes their digits and the update subtracts their products
// from B = 1.  48 matrices of dimension 280: 240 us for all of it, against 1270 us of
// FP64 products (two per clock and SM).  Digits end at 2^-54, the units that 1 - (M^2)_ii has in FP64.
// tr M^2 = |M|^2 and |M^2|^2, which the dense shortcut rules read to their own precision, are
// summed in FP64.
#include "fix.cuh"
#include "internal.h"
#include <type_traits>

namespace capsgpu {

// fixed point: integers of 2^-60.  Row norms are bounded by k_sq_image, so that no sum leaves the integers' range
CAPS_DEV bool sq_live(int st) { return st == ST_OK || st == ST_FACTOR; }

// B = 1, undecided tasks to ST_FACTOR.  Grid (ceil(n / 8), ntask), 256 threads, 8 columns per block
__global__ void __launch_bounds__(256) k_sq_begin(int ntask, int n, long long *B, size_t lda, size_t mstride, FixInfo *info, float *rn, int *status)
{
    const int task = blockIdx.y;
    if (task >= ntask || !sq_live(status[task])) return; // either value of the two: uniform
    for (int c = blockIdx.x * 8; c < min(n, (int)blockIdx.x * 8 + 8); c++) {
        long long *col = B + (size_t)task * mstride + (size_t)c * lda;
        for (int r = c + threadIdx.x; r < n; r += 256) col[r] = r == c ? 1LL << FQ : 0;
        if (threadIdx.x == 0) rn[(size_t)task * n + c] = 0.0f;
    }
    // the next launch reads the status and the exponent, blocks of this one only that it is live
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(status + task, ST_OK, ST_FACTOR);
}

// columns k0 .. k0 + 63 of M as digit images of all row blocks.  Grid (row blocks, ntask), 256 threads: row
// tid mod 64, 8 columns at a time.  A matrix with M_ii <= -1 (its exponent is not 0) or a row of norm above
// sqrt 2 has a 1 - (M^2)_ii < 0: its status becomes that of a pivot which is not positive.
__global__ void __launch_bounds__(256) k_sq_image(int ntask, int n, int k0, const long long *A, size_t lda, size_t mstride, float *rn, int *status,
                                                  FixWork wk)
{
    const int task = blockIdx.y;
    if (task >= ntask || (status[task] & 0xF) != ST_FACTOR) return; // error bits may be set by this launch: not read
    __shared__ unsigned any_lo, any_hi;
    __shared__ float part[4][NB];
    const int r = threadIdx.x & 63, q = threadIdx.x >> 6, R = blockIdx.x * NB + r;
    const long long *Am = A + (size_t)task * mstride;
    if (threadIdx.x == 0) any_lo = any_hi = 0;
    __syncthreads();
    const size_t dst = (size_t)(fix_nbk(n) + 1) * IMG_BLK; // digit to digit
    unsigned char *img = wk.ximg(task, n) + (size_t)blockIdx.x * IMG_BLK;
    unsigned long long any = 0;
    float sum = 0.0f;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int kc = q + 4 * h;
        long long x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int k = k0 + kc * 8 + u;
            x[u] = R >= n || k >= n ? 0
                 : R > k ? -Am[(size_t)k * lda + R] : R < k ? -Am[(size_t)R * lda + k] : (1LL << FQ) - Am[(size_t)k * lda + R];
            any |= digit_mag(x[u]);
            const float f = (float)(int)(x[u] >> 32) * 0x1p-28f;
            sum = fmaf(f, f, sum);
        }
        uint4 d[ND];
        split8(x, d);
#pragma unroll
        for (int i = 0; i < ND; i++) *reinterpret_cast<uint4 *>(img + i * dst + img_off(r, kc)) = d[i];
    }
    const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)any), hi = __reduce_or_sync(0xffffffffu, (unsigned)(any >> 32));
    if ((threadIdx.x & 31) == 0 && (lo | hi)) {
        atomicOr(&any_lo, lo);
        atomicOr(&any_hi, hi);
    }
    part[q][r] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        wk.first[(size_t)task * (fix_nbk(n) + 1) + blockIdx.x] = first_digit((unsigned long long)any_hi << 32 | any_lo);
        if (wk.info[task].sexp) atomicOr(status + task, ST_ERR_PIVOT);
    }
    if (threadIdx.x < NB && R < n) {
        float *t = rn + (size_t)task * n + R;
        const float s = *t + ((part[0][r] + part[1][r]) + (part[2][r] + part[3][r]));
        *t = s;
        if (!(s <= 2.0f)) atomicOr(status + task, ST_ERR_PIVOT);
    }
}

// sums of squares of a symmetric matrix from its lower triangle X, off the diagonal as it is and the diagonal
// 1 - X_ii (fixed point) or mdiag: out[task * gridDim.x + block], warp per column
template <typename T>
__global__ void __launch_bounds__(256) k_sq_norm(int ntask, int n, const T *X, size_t lda, size_t mstride, const double *mdiag, const int *status,
                                                 double *out)
{
    const int task = blockIdx.y;
    if (task >= ntask || !sq_live(status[task])) return;
    __shared__ double red[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x * 8 + warp;
    double s = 0.0;
    if (c < n) {
        const T *col = X + (size_t)task * mstride + (size_t)c * lda;
        const double unit = std::is_integral_v<T> ? 0x1p-60 : 1.0;
#pragma unroll 4
        for (int r = c + 1 + lane; r < n; r += 32) {
            const double v = (double)col[r] * unit;
            s = fma(v, v, s);
        }
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const double d = mdiag ? mdiag[(size_t)task * n + c] : (double)((T)(1LL << FQ) - col[c]) * unit;
        s = fma(d, d, 2.0 * s);
    }
    if (lane == 0) red[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        s = red[0];
        for (int w = 1; w < 8; w++) s += red[w];
        out[(size_t)task * gridDim.x + blockIdx.x] = s;
    }
}

int square_nsum(int n) { return (n + 7) / 8; }

void launch_square_norm(int ntask, int n, const double *A, size_t lda, size_t mstride, const double *mdiag, const int *status, double *out,
                        cudaStream_t st)
{
    k_sq_norm<double><<<dim3(square_nsum(n), ntask), 256, 0, st>>>(ntask, n, A, lda, mstride, mdiag, status, out);
    COUNT_LAUNCH(1);
    CK(cudaGetLastError());
}

void launch_square(int ntask, int n, double *A, size_t lda, size_t mstride, const double *mdiag, double *B, int *status, float *rn, double *fro,
                   void *work, bool fixed, cudaStream_t st)
{
    const FixWork wk = fix_work(ntask, n, work);
    long long *Bf = (long long *)B;
    const dim3 g8(square_nsum(n), ntask);
    k_sq_begin<<<g8, 256, 0, st>>>(ntask, n, Bf, lda, mstride, wk.info, rn, status);
    if (!fixed) fix_convert(ntask, n, A, lda, mstride, status, mdiag, wk, st);
    for (int k0 = 0; k0 < n; k0 += NB) {
        k_sq_image<<<dim3(fix_nbk(n), ntask), 256, 0, st>>>(ntask, n, k0, (const long long *)A, lda, mstride, rn, status, wk);
        fix_syrk(ntask, n, 0, Bf, lda, mstride, status, wk, st);
        COUNT_LAUNCH(1);
    }
    k_sq_norm<long long><<<g8, 256, 0, st>>>(ntask, n, Bf, lda, mstride, nullptr, status, fro);
    COUNT_LAUNCH(2);
    CK(cudaGetLastError());
}

} // namespace capsgpu
