// Device harness of the branch-free correctly rounded quotients
// (piernik_b200/csrc/pk_quotient.cuh): quo, quoz, quoc and mean of n operand pairs (mean
// of n / 2 and d),
// whether the operands were in their range, and CUDA's division; and of van
// Leer's half slopes of groups of five, next to half of slope_interior, and of
// the sums and comparisons of quoa and quob, for the GPU test.
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
    o[7] = m.mean(0.5 * x, y);
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

constexpr int G = 5;

__global__ void k_vanleer(int on, const double* dl, const double* dr, int cnt, double* got, double* want)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cnt) return;
    double a[G], b[G], h[G];
    for (int k = 0; k < G; ++k) {
        a[k] = dl[(long long)i * G + k];
        b[k] = dr[(long long)i * G + k];
    }
    pk::vanleer_half(on != 0, a, b, h, [&](int k, double& x, double& y) {
        x = on ? a[k] : 0.0;
        y = b[k];
    });
    for (int k = 0; k < G; ++k) {
        got[(long long)i * G + k] = h[k];
        want[(long long)i * G + k] = on ? 0.5 * pk::slope_interior(pk::L_VANLEER, a[k], b[k]) : 0.0;
    }
}

// dl, dr, got, want: host arrays of 5 cnt doubles; on = 0: a pencil end; returns a cudaError_t
extern "C" int vanleer_eval(int on, const double* dl, const double* dr, int cnt, double* got, double* want)
{
    const size_t bytes = sizeof(double) * G * (size_t)cnt;
    double* d[4] = {nullptr, nullptr, nullptr, nullptr};
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 4 && e == cudaSuccess; ++k) e = cudaMalloc(&d[k], bytes);
    if (e == cudaSuccess) e = cudaMemcpy(d[0], dl, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d[1], dr, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_vanleer<<<(cnt + 255) / 256, 256>>>(on, d[0], d[1], cnt, d[2], d[3]);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(got, d[2], bytes, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(want, d[3], bytes, cudaMemcpyDeviceToHost);
    for (double* p : d) cudaFree(p);
    return (int)e;
}

__global__ void k_absorbed(const double* n, const double* d, const double* big, int cnt, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cnt) return;
    double* o = out + 8 * (long long)i;
    pk::Exact a, b;
    const double x = a.quoa(n[i], d[i], a.inv(d[i]), big[i]), y = b.quob(n[i], d[i], 1.0 / d[i], big[i], 1.0), q = n[i] / d[i];
    o[0] = big[i] - x;
    o[1] = big[i] + x;
    o[2] = a.ok();
    o[3] = big[i] - q;
    o[4] = big[i] + q;
    o[5] = y <= big[i];
    o[6] = b.ok();
    o[7] = q <= big[i];
}

// n, d, big, out: host arrays (cnt each, out 8 cnt doubles); returns a cudaError_t
extern "C" int absorbed_eval(const double* n, const double* d, const double* big, int cnt, double* out)
{
    const size_t bytes = sizeof(double) * (size_t)cnt;
    const double* src[3] = {n, d, big};
    double* p[4] = {nullptr, nullptr, nullptr, nullptr};
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 4 && e == cudaSuccess; ++k) e = cudaMalloc(&p[k], (k == 3 ? 8 : 1) * bytes);
    for (int k = 0; k < 3 && e == cudaSuccess; ++k) e = cudaMemcpy(p[k], src[k], bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_absorbed<<<(cnt + 255) / 256, 256>>>(p[0], p[1], p[2], cnt, p[3]);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, p[3], 8 * bytes, cudaMemcpyDeviceToHost);
    for (double* q : p) cudaFree(q);
    return (int)e;
}
