// C entry to the FP64 form's factorisation for matrices of a test's own: ntask symmetric n x n matrices A (lower
// triangle, column-major), log det and status out
#include "internal.h"

using namespace capsgpu;

extern "C" int fixed_logdet(const double *A, int n, int ntask, double *logdet, int *status)
{
    const size_t nn = (size_t)n * n;
    double *d_A, *d_md, *d_ld, *d_res;
    int *d_st;
    void *work;
    CK(cudaMalloc(&d_A, ntask * nn * sizeof(double)));
    CK(cudaMalloc(&d_md, (size_t)ntask * n * sizeof(double)));
    CK(cudaMalloc(&d_ld, (size_t)ntask * n * sizeof(double)));
    CK(cudaMalloc(&d_res, (size_t)2 * ntask * sizeof(double)));
    CK(cudaMalloc(&d_st, ntask * sizeof(int)));
    CK(cudaMalloc(&work, cholesky_work_bytes(ntask, n)));
    CK(cudaMemset(work, 0xa5, cholesky_work_bytes(ntask, n))); // nothing is read that was not written
    CK(cudaMemset(d_res, 0, (size_t)2 * ntask * sizeof(double)));
    CK(cudaMemcpy(d_A, A, ntask * nn * sizeof(double), cudaMemcpyHostToDevice));
    for (int t = 0; t < ntask; t++) {
        const int st = ST_FACTOR;
        CK(cudaMemcpy(d_st + t, &st, sizeof st, cudaMemcpyHostToDevice));
        for (int i = 0; i < n; i++) {
            const double m = 1.0 - A[t * nn + (size_t)i * n + i];
            CK(cudaMemcpy(d_md + (size_t)t * n + i, &m, sizeof m, cudaMemcpyHostToDevice));
        }
    }
    launch_cholesky(ntask, n, d_A, n, nn, d_st, d_md, d_ld, work, 0);
    launch_final(ntask, n, d_ld, work, d_res + ntask, d_st, d_res, 0, 0);
    CK(cudaMemcpy(logdet, d_res, ntask * sizeof(double), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(status, d_st, ntask * sizeof(int), cudaMemcpyDeviceToHost));
    for (void *p : {(void *)d_A, (void *)d_md, (void *)d_ld, (void *)d_res, (void *)d_st, work}) CK(cudaFree(p));
    return 0;
}
