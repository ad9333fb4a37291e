// Device harness of the branch-free correctly rounded quotients
// (piernik_b200/csrc/pk_quotient.cuh): quo, quoz, quoc and mean of n operand pairs,
// whether the operands were in their range, and CUDA's division, for the GPU test.
#include <cuda_runtime.h>

#include "../../piernik_b200/csrc/pk_quotient.cuh"

__global__ void k_quotients(const double* n, const double* d, int cnt, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cnt) return;
    const double x = n[i], y = d[i];
    double* o = out + 9 * (long long)i;
    pk::Exact a, b, c, m;
    o[0] = a.quo(x, y, a.inv(y));
    o[1] = b.quoz(x, y, b.inv(y));
    o[2] = c.quoc(x, y, 1.0 / y);
    o[3] = a.ok();
    o[4] = b.ok();
    o[5] = c.ok();
    o[6] = x / y;
    o[7] = m.mean(x, y);
    o[8] = m.ok();
}

// n, d, out: host arrays (cnt, cnt, 9 cnt doubles); returns a cudaError_t
extern "C" int quotient_eval(const double* n, const double* d, int cnt, double* out)
{
    double *dn = nullptr, *dd = nullptr, *dout = nullptr;
    cudaError_t e = cudaMalloc(&dn, sizeof(double) * cnt);
    if (e == cudaSuccess) e = cudaMalloc(&dd, sizeof(double) * cnt);
    if (e == cudaSuccess) e = cudaMalloc(&dout, sizeof(double) * 9 * (size_t)cnt);
    if (e == cudaSuccess) e = cudaMemcpy(dn, n, sizeof(double) * cnt, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dd, d, sizeof(double) * cnt, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_quotients<<<(cnt + 255) / 256, 256>>>(dn, dd, cnt, dout);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, sizeof(double) * 9 * (size_t)cnt, cudaMemcpyDeviceToHost);
    cudaFree(dn);
    cudaFree(dd);
    cudaFree(dout);
    return (int)e;
}
