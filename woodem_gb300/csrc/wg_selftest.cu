// Entries for the tests that run compiled device functions on arrays of their own: the quotients of wg_div.cuh, and
// the FP32 decision on a periodic overlap (wg_geom.cuh).
#include <vector>

#include "wg_div.cuh"
#include "wg_geom.cuh"

namespace wg {
int selftest_overlap32(int64_t n, const double4_32a* mn, const double4_32a* mx, const double* size, int32_t* quick, int32_t* exact);

constexpr int kQuotients = 13;
__global__ void k_quotients(int64_t n, const double* __restrict__ a, const double* __restrict__ b, const double* __restrict__ z,
                            double* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const D3 u{a[3 * i], a[3 * i + 1], a[3 * i + 2]}, v{b[3 * i], b[3 * i + 1], b[3 * i + 2]};
    const D3 by = divBy(u, v.x), by3 = divBy3(u, v, D3{z[3 * i], z[3 * i + 1], z[3 * i + 2]}), unit = normalizedQ(u);
    const DQ q = qnormalizedQ(DQ{v.x, u.x, u.y, u.z});
    const double o[kQuotients] = {by.x, by.y, by.z, by3.x, by3.y, by3.z, unit.x, unit.y, unit.z, q.w, q.x, q.y, q.z};
    for (int k = 0; k < kQuotients; k++) out[kQuotients * i + k] = o[k];
}
}  // namespace wg

using namespace wg;

extern "C" {

int wg_selftest_quotients(int64_t n, const double* a3, const double* b3, const double* rb3, double* out13) {
    if (n < 0 || (n > 0 && (!a3 || !b3 || !rb3 || !out13))) return WG_ERR_ARG;
    if (n == 0) return WG_OK;
    double* d = nullptr;
    if (cudaMalloc(&d, sizeof(double) * n * (9 + kQuotients)) != cudaSuccess) {
        cudaGetLastError();
        return WG_ERR_CUDA;
    }
    const size_t in = sizeof(double) * 3 * n;
    cudaError_t r = cudaMemcpy(d, a3, in, cudaMemcpyHostToDevice);
    if (r == cudaSuccess) r = cudaMemcpy(d + 3 * n, b3, in, cudaMemcpyHostToDevice);
    if (r == cudaSuccess) r = cudaMemcpy(d + 6 * n, rb3, in, cudaMemcpyHostToDevice);
    if (r == cudaSuccess) {
        k_quotients<<<(unsigned)((n + 255) / 256), 256>>>(n, d, d + 3 * n, d + 6 * n, d + 9 * n);
        r = cudaGetLastError();
    }
    if (r == cudaSuccess) r = cudaMemcpy(out13, d + 9 * n, sizeof(double) * kQuotients * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return r == cudaSuccess ? WG_OK : WG_ERR_CUDA;
}

int wg_selftest_overlap(int64_t n, const double* min6, const double* max6, const double* size3, int32_t* quick, int32_t* exact) {
    if (n < 0 || !size3 || (n > 0 && (!min6 || !max6 || !quick))) return WG_ERR_ARG;
    std::vector<double4_32a> mn, mx;
    try {
        mn.resize(2 * n);
        mx.resize(2 * n);
    } catch (...) {
        return WG_ERR_ARG;
    }
    for (int64_t k = 0; k < 2 * n; k++) {
        mn[k] = make_double4_32a(min6[3 * k], min6[3 * k + 1], min6[3 * k + 2], 0.);
        mx[k] = make_double4_32a(max6[3 * k], max6[3 * k + 1], max6[3 * k + 2], 0.);
    }
    if (exact) return selftest_overlap32(n, mn.data(), mx.data(), size3, quick, exact) ? WG_ERR_CUDA : WG_OK;
    for (int64_t i = 0; i < n; i++) quick[i] = overlapPeriQuick(mn[2 * i], mx[2 * i], mn[2 * i + 1], mx[2 * i + 1], size3);
    return WG_OK;
}

}  // extern "C"
