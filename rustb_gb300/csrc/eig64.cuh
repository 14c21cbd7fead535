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

// Reflector H = I - tau v v^H, v = (1, scal up x_1, ...), of a column with first
// entry alpha and xn = sum of |x_i|^2 over the others: H^H x = beta e_0, beta real.
// A column whose squares leave the range is taken times up = 2^900 or 2^-600
// (rescaled(up): the sum of |up x_i|^2, by the same threads), else H would not be
// unitary: the columns of a rank-deficient matrix fall by 10^16 a step, and vectors were
// off by up to 10^-2 where one fell to 10^-160.
struct Reflector64 {
    zc tau, scal;
    double beta, up;
    bool far;  // up != 1
};
template <typename F>
__device__ __forceinline__ Reflector64 reflector64_of(zc alpha, double xn, F rescaled) {
    Reflector64 r;
    r.up = 1.0;
    double n2 = fma(alpha.re, alpha.re, fma(alpha.im, alpha.im, xn));
    r.far = (unsigned)(__double2hiint(n2) - 0x05d00000) >= 0x74400000u;  // outside [2^-930, 2^930)
    if (r.far) {
        r.up = n2 < 1.0 ? 0x1p900 : 0x1p-600;
        alpha = r.up * alpha;
        xn = rescaled(r.up);
        n2 = fma(alpha.re, alpha.re, fma(alpha.im, alpha.im, xn));
    }
    if (xn == 0.0 && alpha.im == 0.0) {
        r.tau = r.scal = mk(0.0, 0.0);
        r.beta = alpha.re;
    } else {
        const double y = fast_rsqrt(n2);
        double nrm = n2 * y;
        nrm = fma(fma(-nrm, nrm, n2), 0.5 * y, nrm);
        const bool neg = __double2hiint(alpha.re) >= 0;  // beta opposite in sign to Re(alpha)
        r.beta = flip_if(nrm, neg);
        const double ib = flip_if(y, neg);
        const double dr = alpha.re - r.beta;
        r.tau = mk(-dr * ib, -alpha.im * ib);
        const double q = fast_rcp(fma(dr, dr, alpha.im * alpha.im));
        r.scal = mk(dr * q, -alpha.im * q);
    }
    if (r.far) r.beta *= r.up > 1.0 ? 0x1p-900 : 0x1p600;
    return r;
}

// Dynamic shared memory of a CTA of that reduction, C of them per matrix.
inline size_t panel64_smem_bytes(int N, int C) { return sizeof(zc) * ((size_t)N + 2 * (((size_t)N + C - 1) / C)); }
// Reduction by a cluster of CTAs per matrix (eig64_big.cu); a column stays in
// shared memory (models have at most 4096 bands).
int hetrd64_big(cudaStream_t st, int N, int64_t batch, zc* A, int* status_d);
// Back-transformation with blocked reflectors on the tensor cores (eig64_big.cu).
int bt64_wy(cudaStream_t st, int N, int64_t batch, const zc* A, zc* U, int* status_d, int first, int ncol);

}  // namespace tbg
