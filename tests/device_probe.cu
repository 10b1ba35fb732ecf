// device_probe.cu -- the scalar helpers of pb_device.cuh over host arrays, one element per thread, for
// tests/test_gpu_arithmetic.py.  Returns the CUDA status.
#include <cuda_runtime.h>

#include "../plabundle_gb300/csrc/pb_device.cuh"

namespace {

__global__ void k_to_pair(int n, const double* in, float2* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const pb::ff v = pb::ff_make_bits(in[i]);
    out[i] = make_float2(v.hi, v.lo);
}

__global__ void k_to_double(int n, const float* in, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = pb::f64_of(in[i]);
}

// out[5 i ..] of the pair (x, y): rcp64(x), sqrt64(x) where x > 0, and where x is a plain pivot (else -1)
// plain_quotient(y, x) and the reciprocal root and root of plain_roots.
__global__ void k_arith(int n, const double2* in, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = in[i].x, y = in[i].y;
    double* o = out + 5 * static_cast<size_t>(i);
    o[0] = pb::rcp64(x);
    o[1] = x > 0.0 ? pb::sqrt64(x) : 0.0;
    const bool plain = pb::plain_pivot(x);
    o[2] = plain ? pb::plain_quotient(y, x) : -1.0;
    o[3] = o[4] = -1.0;
    if (plain) pb::plain_roots(x, o[4], o[3]);
}

struct Five {
    double v[5];
};

template <typename In, typename Out, typename Launch>
int over(int n, const In* in, Out* out, Launch launch) {
    In* a = nullptr;
    Out* b = nullptr;
    cudaError_t e = cudaMalloc(&a, n * sizeof(In));
    if (e == cudaSuccess) e = cudaMalloc(&b, n * sizeof(Out));
    if (e == cudaSuccess) e = cudaMemcpy(a, in, n * sizeof(In), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        launch((n + 255) / 256, a, b);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, b, n * sizeof(Out), cudaMemcpyDeviceToHost);
    cudaFree(a);
    cudaFree(b);
    return static_cast<int>(e);
}

}  // namespace

extern "C" int probe_to_pair(int n, const double* in, float* out) {
    return over(n, in, reinterpret_cast<float2*>(out),
                [n](int grid, const double* a, float2* b) { k_to_pair<<<grid, 256>>>(n, a, b); });
}

extern "C" int probe_arith(int n, const double* in, double* out) {
    return over(n, reinterpret_cast<const double2*>(in), reinterpret_cast<Five*>(out),
                [n](int grid, const double2* a, Five* b) { k_arith<<<grid, 256>>>(n, a, reinterpret_cast<double*>(b)); });
}

extern "C" int probe_to_double(int n, const float* in, double* out) {
    return over(n, in, out, [n](int grid, const float* a, double* b) { k_to_double<<<grid, 256>>>(n, a, b); });
}
