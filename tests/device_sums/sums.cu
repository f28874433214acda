// One warp: the double-float sums and quotients of the one-launch solves
// (isl_device.cuh) on given inputs.
#include "../../insilico_gb300/csrc/isl_device.cuh"

using namespace isl;

// x [n][32], y [n][32]: sums over the lanes; num, den [n] (hi, lo): quotients
__global__ void k_run(int n, const float* x, const float* y, const df* num, const df* den, df* sx, df* sy, float* q) {
    for (int i = 0; i < n; ++i) {
        df a = {x[32 * i + threadIdx.x], 0.f}, b = {y[32 * i + threadIdx.x], 0.f};
        warp_sum_df2<true, true, 16>(a, b);
        if (threadIdx.x) continue;
        sx[i] = a;
        sy[i] = b;
        q[i] = df_quotient(num[i], den[i]);
    }
}

extern "C" int run(int n, const float* x, const float* y, const float* num, const float* den, float* sx, float* sy, float* q) {
    const size_t v = (size_t)n * 32 * 4, d = (size_t)n * 8;
    char* p = nullptr;
    if (cudaMalloc((void**)&p, 2 * v + 5 * d) != cudaSuccess) return 1;
    float *dx = (float*)p, *dy = (float*)(p + v), *dq = (float*)(p + 2 * v + 4 * d);
    df *dn = (df*)(p + 2 * v), *dd = dn + n, *ox = dd + n, *oy = ox + n;
    cudaMemcpy(dx, x, v, cudaMemcpyHostToDevice);
    cudaMemcpy(dy, y, v, cudaMemcpyHostToDevice);
    cudaMemcpy(dn, num, d, cudaMemcpyHostToDevice);
    cudaMemcpy(dd, den, d, cudaMemcpyHostToDevice);
    k_run<<<1, 32>>>(n, dx, dy, dn, dd, ox, oy, dq);
    cudaMemcpy(sx, ox, d, cudaMemcpyDeviceToHost);
    cudaMemcpy(sy, oy, d, cudaMemcpyDeviceToHost);
    cudaMemcpy(q, dq, (size_t)n * 4, cudaMemcpyDeviceToHost);
    const int e = (int)cudaGetLastError();
    cudaFree(p);
    return e;
}
