// Runs the helpers of pair2.cuh on arrays of operands (tests/test_gpu_rounding.py): one
// thread takes two of them, as the passes do.
#include <cuda_runtime.h>

#include "../armando_gb300/csrc/pair2.cuh"

using namespace ag;

// out[0 .. n): the helper's result, out[n .. 2n): CUDA's correctly rounded one, or the
// low part of a float-float result.
__global__ void k_helpers(int what, const float* a, const float* b, int n, float* out) {
    const int i = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (i + 1 >= n) return;
    const f2 x = make_float2(a[i], a[i + 1]), y = make_float2(b[i], b[i + 1]);
    f2 r = bc2(0.f), w = r;
    if (what == 0) {
        r = div2(x, y);
        w = make_float2(__fdiv_rn(x.x, y.x), __fdiv_rn(x.y, y.y));
    } else if (what == 1) {
        r = rcp2_rn(y, rcp2(y));
        w = make_float2(__frcp_rn(y.x), __frcp_rn(y.y));
    } else if (what == 2) {
        r = sqrt2(x, rsqrt2(x));
        w = make_float2(__fsqrt_rn(x.x), __fsqrt_rn(x.y));
    } else if (what == 3) {
        const ff2 q = recip_ff2(x);
        r = q.hi;
        w = q.lo;
    } else if (what == 4) {
        const ff2 q = sqrt_ff2(ff2{x, y});
        r = q.hi;
        w = q.lo;
    } else if (what == 5) {
        r = rcp2(x);
        w = make_float2(__frcp_rn(x.x), __frcp_rn(x.y));
    } else if (what == 6) {
        r = rsqrt2(x);
    }
    out[i] = r.x;
    out[i + 1] = r.y;
    out[n + i] = w.x;
    out[n + i + 1] = w.y;
}

extern "C" int run_helpers(int what, const float* a, const float* b, int n, float* out) {
    float *da = nullptr, *db = nullptr, *dout = nullptr;
    cudaError_t e = cudaMalloc(&da, n * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&db, n * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&dout, 2 * n * sizeof(float));
    if (e == cudaSuccess) e = cudaMemcpy(da, a, n * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(db, b, n * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_helpers<<<(n / 2 + 255) / 256, 256>>>(what, da, db, n, dout);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, 2 * n * sizeof(float), cudaMemcpyDeviceToHost);
    cudaFree(da);
    cudaFree(db);
    cudaFree(dout);
    return (int)e;
}
