// Test helper (not product): runs the point-wise routines of dgsem_line.cuh over
// host arrays.  Built by tests/test_gpu_line_math.py with nvcc into a temporary folder.
#include "../../prandtl_b200/csrc/dgsem_impl.cuh"

namespace line_math {

using namespace prandtl;

// which: 0 sqrt_pos(x), 1 log_ratio(x, y), 2 atanh(f)/f of f = (y-x)/(y+x) on the branch line_flux takes
__global__ void scalar_kernel(int which, const double *x, const double *y, double *out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (which == 0) out[i] = sqrt_pos(x[i]);
    else if (which == 1) out[i] = log_ratio(x[i], y[i]);
    else {
        const double f = (y[i] - x[i]) * rcp(y[i] + x[i]), u = f * f;
        out[i] = u < 1e-4 ? 1.0 + log_q_near(u) : log_q_far(x[i], y[i], f, u);
    }
}
// two-point fluxes of (rho, v, beta) states a, b along m, [n][5] and [n][3]
template <bool NEAR>
__global__ void flux_kernel(const double *a, const double *b, const double *m, double gm1i, double *F, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) line_flux<3, NEAR>(a + 5 * i, b + 5 * i, m + 3 * i, gm1i, F + 5 * i);
}
struct Buffer {
    double *p = nullptr;
    Buffer(const double *src, size_t n) {
        if (cudaMalloc(&p, n * sizeof(double)) != cudaSuccess) p = nullptr;
        else if (src && cudaMemcpy(p, src, n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess) drop();
    }
    ~Buffer() { drop(); }
    void drop() {
        cudaFree(p);
        p = nullptr;
    }
};
int fetch(double *dst, const Buffer &b, size_t n) {
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) return 4;
    return cudaMemcpy(dst, b.p, n * sizeof(double), cudaMemcpyDeviceToHost) == cudaSuccess ? 0 : 5;
}

}   // namespace line_math

using namespace line_math;
extern "C" {
int lm_scalar(int which, const double *x, const double *y, double *out, int n) {
    Buffer dx(x, n), dy(y, n), d(nullptr, n);
    if (n <= 0 || !dx.p || !dy.p || !d.p) return 1;
    scalar_kernel<<<(n + 255) / 256, 256>>>(which, dx.p, dy.p, d.p, n);
    return fetch(out, d, n);
}
int lm_flux(int near, const double *a, const double *b, const double *m, double gm1i, double *F, int n) {
    Buffer da(a, 5 * (size_t)n), db(b, 5 * (size_t)n), dm(m, 3 * (size_t)n), d(nullptr, 5 * (size_t)n);
    if (n <= 0 || !da.p || !db.p || !dm.p || !d.p) return 1;
    if (near) flux_kernel<true><<<(n + 255) / 256, 256>>>(da.p, db.p, dm.p, gm1i, d.p, n);
    else flux_kernel<false><<<(n + 255) / 256, 256>>>(da.p, db.p, dm.p, gm1i, d.p, n);
    return fetch(F, d, 5 * (size_t)n);
}
}
