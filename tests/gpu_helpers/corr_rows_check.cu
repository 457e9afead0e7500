// Test helper (built by tests/test_gpu_corr_rows.py): one CTA of k_lr_correct
// whose rows start at `base` of the row lists (which are allocated up to there
// and filled from there on only).  m = 2, S = Id, u = (u0, u1).
#include "../../multigridmc_gb300/csrc/kernels.cuh"

extern "C" int corr_rows_check(long long base, int n, const unsigned *rows, const int *cols, const float *vals, float u0, float u1,
                               float *x, int nx) {
    using namespace mgmc;
    constexpr int M = 2;
    unsigned *r1;
    int *c1, *jcols;
    float *v1, *dx;
    float2 *S, *w, *part;
    CorrJob *dj;
    if (cudaMalloc(&r1, (base + n) * 4) || cudaMalloc(&c1, (base + n) * 4) || cudaMalloc(&v1, (base + n) * 4) ||
        cudaMalloc(&dx, nx * 4) || cudaMalloc(&S, M * M * 8) || cudaMalloc(&w, M * 8) || cudaMalloc(&part, M * 8) ||
        cudaMalloc(&dj, sizeof(CorrJob)) || cudaMalloc(&jcols, M * 4))
        return 1;
    const float2 Sh[M * M] = {{1.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {1.f, 0.f}}, wh[M] = {{u0, 0.f}, {u1, 0.f}};
    const int jc[M] = {0, 1};
    CorrJob job{};
    job.r0 = base;
    job.n = n;
    job.nc = M;
    cudaMemcpy(r1 + base, rows, n * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(c1 + base, cols, n * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(v1 + base, vals, n * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(dx, x, nx * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(S, Sh, sizeof(Sh), cudaMemcpyHostToDevice);
    cudaMemcpy(w, wh, sizeof(wh), cudaMemcpyHostToDevice);
    cudaMemset(part, 0, M * 8);
    cudaMemcpy(dj, &job, sizeof(job), cudaMemcpyHostToDevice);
    cudaMemcpy(jcols, jc, sizeof(jc), cudaMemcpyHostToDevice);
    LowRankArg lr{};
    lr.m = M;
    lr.SinvT_ff = S;
    lr.w = w;
    lr.part = reinterpret_cast<double *>(part);
    CorrRows C;
    C.n1 = base + n;
    C.r1 = r1;
    C.c1 = c1;
    C.v1 = v1;
    const size_t sm = sizeof(double) * (2 * M + 64 * 8 + LRC_MAX_M);
    k_lr_correct<float, 1, 1><<<1, 256, sm>>>(dx, lr, 1, C, dj, jcols);
    cudaMemcpy(x, dx, nx * 4, cudaMemcpyDeviceToHost);
    const int err = cudaGetLastError() != cudaSuccess;
    cudaFree(r1); cudaFree(c1); cudaFree(v1); cudaFree(dx); cudaFree(S); cudaFree(w); cudaFree(part); cudaFree(dj); cudaFree(jcols);
    return err;
}
