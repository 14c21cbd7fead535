// Shared by the FP64 eigensolver's translation units.
#pragma once

#include "tbgpu_internal.cuh"

namespace tbg {

// 1 / x and 1 / sqrt(x) from the hardware's approximations (about 20 bits) and
// one third-order step of the Newton family on the residual e = 1 - x y
// (e = 1 - x y^2): y (1 + e + e^2), y (1 + e / 2 + 3 e^2 / 8).  For arguments
// well inside the normal range.
__device__ __forceinline__ double fast_rcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double fast_rsqrt(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y, e * fma(0.375, e, 0.5), y);
}
// sign flips and magnitude tests on the high word (integer pipe)
__device__ __forceinline__ double flip_if(double x, bool f) {
    return __hiloint2double(__double2hiint(x) ^ (f ? 0x80000000 : 0), __double2loint(x));
}
__device__ __forceinline__ int hi_abs(double x) { return __double2hiint(x) & 0x7fffffff; }

// Reflector H = I - tau v v^H, v = (1, scal x_1, ...), of a column with first
// entry alpha and xn = sum of |x_i|^2 over the others: H^H x = beta e_0, beta real.
__device__ __forceinline__ void reflector_scalars64(zc alpha, double xn, zc& tau, zc& scal, double& beta) {
    if (xn == 0.0 && alpha.im == 0.0) {
        tau = mk(0.0, 0.0);
        scal = mk(0.0, 0.0);
        beta = alpha.re;
        return;
    }
    const double n2 = fma(alpha.re, alpha.re, fma(alpha.im, alpha.im, xn));
    if (n2 > 1e-280 && n2 < 1e280) {
        const double y = fast_rsqrt(n2);
        double nrm = n2 * y;
        nrm = fma(fma(-nrm, nrm, n2), 0.5 * y, nrm);
        const bool neg = __double2hiint(alpha.re) >= 0;  // beta opposite in sign to Re(alpha)
        beta = flip_if(nrm, neg);
        const double ib = flip_if(y, neg);
        const double dr = alpha.re - beta;
        tau = mk(-dr * ib, -alpha.im * ib);
        const double r = fast_rcp(fma(dr, dr, alpha.im * alpha.im));
        scal = mk(dr * r, -alpha.im * r);
    } else {
        const double nrm = sqrt(n2);
        beta = (alpha.re >= 0.0) ? -nrm : nrm;
        tau = mk((beta - alpha.re) / beta, -alpha.im / beta);
        const double dr = alpha.re - beta, dd = dr * dr + alpha.im * alpha.im;
        scal = mk(dr / dd, -alpha.im / dd);
    }
}

// Reduction by a cluster of CTAs per matrix (eig64_big.cu); a column stays in
// shared memory (models have at most 4096 bands).
int hetrd64_big(cudaStream_t st, int N, int64_t batch, zc* A, int* status_d);
// Back-transformation with blocked reflectors on the tensor cores (eig64_big.cu).
int bt64_wy(cudaStream_t st, int N, int64_t batch, const zc* A, zc* U, int* status_d, int first, int ncol);

}  // namespace tbg
