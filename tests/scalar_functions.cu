// Calls the device functions of hc_scalar.cuh, one value a thread, for the test that
// compares them with extended precision.
#include "hc_scalar.cuh"

template <typename T>
__global__ void run(int what, int n, const T *x, const T *y, const T *z, T *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = what == 0 ? hc::inv(x[i]) : (what == 1 ? hc::inv_sqrt(x[i]) : hc::tangent(x[i], y[i], z[i]));
}

template <typename T>
static int call(int what, int n, const T *x, const T *y, const T *z, T *out) {
    T *d = nullptr;
    cudaError_t e = cudaMalloc(&d, (size_t)4 * n * sizeof(T));
    if (e != cudaSuccess) return (int)e;
    const T *in[3] = {x, y, z};
    for (int q = 0; q < 3 && e == cudaSuccess; ++q)
        e = cudaMemcpy(d + (size_t)q * n, in[q], n * sizeof(T), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        run<T><<<(n + 255) / 256, 256>>>(what, n, d, d + n, d + 2 * (size_t)n, d + 3 * (size_t)n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + 3 * (size_t)n, n * sizeof(T), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}

extern "C" int scalar_f64(int what, int n, const double *x, const double *y, const double *z, double *out) {
    return call(what, n, x, y, z, out);
}
extern "C" int scalar_f32(int what, int n, const float *x, const float *y, const float *z, float *out) {
    return call(what, n, x, y, z, out);
}
