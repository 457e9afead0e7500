// Test helper (built by tests/test_gpu_lowrank_cholesky_memory.py): the m x m
// product and the product with Q of the low-rank Cholesky sampler, for m
// columns and `rows` rows of Q, in the form that the sampler would take.
#include "../../multigridmc_gb300/csrc/kernels.cuh"

// v = (W^T - Id) sum of the parts, then xi += g + Q v; wide < 0: the form by m
extern "C" int chol_wide_check(const double *part, int nparts, int m, const double *W, const double *Q, int rows,
                               const double *g, double *xi, double *v, int wide) {
    using namespace mgmc;
    double *dp, *dW, *dQ, *dg, *dx, *dv;
    const size_t sz = sizeof(double), mm = (size_t)m * m;
    if (cudaMalloc(&dp, nparts * m * sz) || cudaMalloc(&dW, mm * sz) || cudaMalloc(&dQ, (size_t)rows * m * sz) ||
        cudaMalloc(&dg, rows * sz) || cudaMalloc(&dx, rows * sz) || cudaMalloc(&dv, 2 * m * sz))
        return 1;
    cudaMemcpy(dp, part, nparts * m * sz, cudaMemcpyHostToDevice);
    W ? cudaMemcpy(dW, W, mm * sz, cudaMemcpyHostToDevice) : cudaMemset(dW, 0, mm * sz);
    cudaMemcpy(dQ, Q, (size_t)rows * m * sz, cudaMemcpyHostToDevice);
    cudaMemcpy(dg, g, rows * sz, cudaMemcpyHostToDevice);
    cudaMemcpy(dx, xi, rows * sz, cudaMemcpyHostToDevice);
    const size_t sm = m * sz;
    const unsigned blocks = (rows + 127) / 128;
    if (m <= CHOL_V_COLS) {
        k_chol_v<true><<<1, 8 * CHOL_V_COLS>>>(dp, nparts, m, dW, dv);
    } else {
        k_chol_t<<<(m + 31) / 32, 256>>>(dp, nparts, m, dv + m);
        k_chol_w<true><<<(m + 31) / 32, 256>>>(dW, m, dv + m, dv);
    }
    if (wide < 0 ? m > CHOL_STAGE_M : wide) {
        k_chol_add<true, true><<<blocks, 128>>>(dx, dg, dQ, rows, m, dv);
    } else {
        cudaFuncSetAttribute(k_chol_add<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        k_chol_add<true, false><<<blocks, 128, sm>>>(dx, dg, dQ, rows, m, dv);
    }
    cudaMemcpy(xi, dx, rows * sz, cudaMemcpyDeviceToHost);
    cudaMemcpy(v, dv, m * sz, cudaMemcpyDeviceToHost);
    const int err = cudaGetLastError() != cudaSuccess;
    cudaFree(dp); cudaFree(dW); cudaFree(dQ); cudaFree(dg); cudaFree(dx); cudaFree(dv);
    return err;
}
