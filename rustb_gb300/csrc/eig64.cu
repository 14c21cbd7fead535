// FP64 batched Hermitian eigensolver (plain path), replacing LAPACK zheev as
// reached from Rustb (src/response/traits.rs:168 via ndarray-linalg Eigh;
// src/ndarray_lapack.rs:412-448).
//
// The part's FP64 pipe does about 1.7 FMA per clock and SM (1/64 of FP32), so
// every stage is laid out to spend few FP64 instructions, each with all its
// lanes in use; integer, FP32 and shared-memory work beside them is free by
// comparison.
//
//   1. hetrd64: Householder reduction T = Q^H A Q (unblocked, 8/3 N^3 FMA),
//      the packed upper triangle in shared memory.  One warp per matrix up to
//      32 bands (no block barriers), one CTA above.  The rank-2 update
//      A22 -= v u^H + u v^H runs over the packed triangle folded into a
//      rectangle (row p with row m - 1 - p), the product A22 v over
//      (row, part of the row) pairs, so lanes stay filled as the trailing
//      block shrinks.  u = tau A v - (|tau|^2 / 2)(v^H A v) v.
//   2. tri64: eigenvalues and eigenvectors of T, one thread per eigenvalue.
//      FP32 bisection (Sturm counts) brings each to about 2e-7 ||T||; then
//      Rayleigh-quotient iteration on the twisted factorisation of T - x I
//      (Fernando 1997; Parlett and Dhillon 1997) in FP64, which converges
//      cubically: x <- x + gamma_r / ||z||^2 with z the twisted vector, two
//      or three passes of N - 1 reciprocals against the 53 FP64 Sturm counts
//      of a bisection.  A pass needs no storage for the value, only the ratios
//      for the vector.  Eigenvalues nearer than 2e-5 ||T|| to a neighbour are
//      bisected in FP64 from the FP32 bracket; the vectors of clusters (gaps
//      up to 1e-3 ||T||) are left to tri64_cluster (inverse iteration with
//      Gram-Schmidt).
//   3. bt64: U = H_0 ... H_{N-2} Z, columns in registers, one or several
//      lanes per column (4 N^3 FMA).
//
// Between the stages everything is kept in A: row j holds v_j right of the
// diagonal, A(j, j) = (d_j, e_j), A(j + 1, j) = tau_j, and the cluster marks
// sit in A(N - 1, 0 ..).  Nothing is allocated.
//
// Eigenpairs of 1024 matrices of 128 bands 82.9 -> 21.6 ms (reduction 13.7,
// tridiagonal 2.7, back-transformation 17.3 by single reflectors and 5.2 in
// blocks on the tensor cores; the first two at 0.8 to 1.0 of the 1.06 TFLOP/s
// that the FP64 pipe does), 4032 of 64 bands 77 -> 15.7,
// 2304 of 26 bands 7.5 -> 1.14, against one kernel with FP64 bisection, the
// matrix in L2 and reflectors applied by eight lanes per column.

#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>

#include "eig64.cuh"
#include "tbgpu_internal.cuh"

namespace tbg {
namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

__host__ __device__ __forceinline__ int pk_off(int N, int i) { return i * N - (i * (i - 1)) / 2; }

// Reflector of step j by one warp: x = conj(row) (row = A(j, j + 1 ..), length
// m, packed in shared memory), H^H x = beta e_0 with beta real.  v (v_0 = 1)
// goes to sv and to global row j; returns tau, beta in all lanes.
__device__ __forceinline__ void reflector64(const zc* row, int m, int lane, zc* sv, zc* gv, zc& tau, double& beta) {
    double part = 0.0;
    for (int i = lane; i < m; i += 32)
        if (i > 0) part += abs2(row[i]);
    const Reflector64 r = reflector64_of(conj(row[0]), wsum(part), [&](double up) {
        double p = 0.0;
        for (int i = lane; i < m; i += 32)
            if (i > 0) p += abs2(up * row[i]);
        return wsum(p);
    });
    tau = r.tau;
    beta = r.beta;
    if (r.far) {
        for (int i = lane; i < m; i += 32) {
            const zc vi = (i == 0) ? mk(1.0, 0.0) : (r.up * conj(row[i])) * r.scal;
            sv[i] = vi;
            gv[i] = vi;
        }
        return;
    }
    for (int i = lane; i < m; i += 32) {
        const zc vi = (i == 0) ? mk(1.0, 0.0) : conj(row[i]) * r.scal;
        sv[i] = vi;
        gv[i] = vi;
    }
}

// Element t of the triangle of order m folded into rows of m + 1: row p and
// row m - 1 - p side by side.
__device__ __forceinline__ void fold_index(int m, int t, int& i, int& l) {
    const int p = t / (m + 1), c = t - p * (m + 1);
    if (c < m - p) {
        i = p;
        l = p + c;
    } else {
        i = m - 1 - p;
        l = i + c - (m - p);
    }
}

// A22(i, l) -= v_i conj(u_l) + u_i conj(v_l), real on the diagonal
__device__ __forceinline__ void rank2_elem(zc* x, const zc* sv, const zc* su, int i, int l) {
    zc a = *x;
    fms_mulc(a, sv[i], su[l]);
    fms_mulc(a, su[i], sv[l]);
    if (i == l) a.im = 0.0;
    *x = a;
}

// Part of row i of A22 v: columns l = q, q + Q, ...  (A22(i, l) from the upper
// triangle; conj(A22(l, i)) left of the diagonal).  T22 points at the packed
// trailing triangle of order m.
__device__ __forceinline__ zc row_times(const zc* T22, int m, int i, int q, int Q, const zc* sv) {
    zc a0 = mk(0.0, 0.0), a1 = mk(0.0, 0.0);
    const int oi = pk_off(m, i) - i;
    auto elem = [&](int l) {
        const bool up = l >= i;
        zc a = T22[up ? oi + l : pk_off(m, l) + i - l];
        a.im = flip_if(a.im, !up);
        return a;
    };
    int l = q;
    for (; l + Q < m; l += 2 * Q) {
        fma_cx(a0, elem(l), sv[l]);
        fma_cx(a1, elem(l + Q), sv[l + Q]);
    }
    if (l < m) fma_cx(a0, elem(l), sv[l]);
    return a0 + a1;
}

constexpr int kWarpMax = 32;  // bands up to which one warp holds a matrix
constexpr int kWarpsPerCta = 4;  // at most

__host__ __device__ inline size_t warp_smem_elems(int N) { return (size_t)N * (N + 1) / 2 + 2 * (size_t)N; }

__global__ void __launch_bounds__(32 * kWarpsPerCta) hetrd64_warp_kernel(int N, int64_t batch, zc* __restrict__ Ain) {
    extern __shared__ __align__(16) unsigned char smem64[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    zc* P = reinterpret_cast<zc*>(smem64) + warp * warp_smem_elems(N);
    zc* sv = P + N * (N + 1) / 2;
    zc* su = sv + N;
    const int wpc = blockDim.x >> 5;
    for (int64_t b = (int64_t)blockIdx.x * wpc + warp; b < batch; b += (int64_t)gridDim.x * wpc) {
        zc* A = Ain + b * N * N;
        for (int e = lane; e < N * N; e += 32) {
            const int r = e / N, c = e - r * N;
            if (c < r) continue;
            zc a = A[e];
            if (c == r) a.im = 0.0;
            P[pk_off(N, r) + c - r] = a;
        }
        __syncwarp();
        for (int j = 0; j < N - 1; ++j) {
            const int m = N - 1 - j;
            zc* row = P + pk_off(N, j);
            zc tau;
            double beta;
            reflector64(row + 1, m, lane, sv, A + (size_t)j * N + j + 1, tau, beta);
            if (lane == 0) {
                A[(size_t)j * N + j] = mk(row[0].re, beta);
                A[(size_t)(j + 1) * N + j] = tau;
            }
            __syncwarp();
            zc* T22 = row + m + 1;  // rows j + 1 .. packed: order m
            // w = tau A22 v: 1, 2 or 4 lanes per row
            const int sh = m > 16 ? 5 : (m > 8 ? 4 : 3);
            const int i = lane & ((1 << sh) - 1), q = lane >> sh, Q = 32 >> sh;
            zc acc = mk(0.0, 0.0);
            if (i < m) acc = row_times(T22, m, i, q, Q, sv);
            for (int o = 1 << sh; o < 32; o <<= 1) {
                acc.re += __shfl_xor_sync(kFull, acc.re, o);
                acc.im += __shfl_xor_sync(kFull, acc.im, o);
            }
            const bool own = q == 0 && i < m;
            const zc vi = own ? sv[i] : mk(0.0, 0.0);
            const double s = wsum(fma(vi.re, acc.re, vi.im * acc.im));  // v^H A v (real)
            const double a2 = -0.5 * fma(tau.re, tau.re, tau.im * tau.im) * s;
            if (own) {
                const zc w = tau * acc;
                su[i] = mk(fma(a2, vi.re, w.re), fma(a2, vi.im, w.im));
            }
            __syncwarp();
            const int tot = m * (m + 1) / 2;
            for (int t = lane; t < tot; t += 32) {
                int r, l;
                fold_index(m, t, r, l);
                rank2_elem(T22 + pk_off(m, r) + l - r, sv, su, r, l);
            }
            __syncwarp();
        }
        if (lane == 0) A[(size_t)N * N - 1] = mk(P[pk_off(N, N - 1)].re, 0.0);
        __syncwarp();
    }
}

// One CTA per matrix.  The reflectors are made by one warp (its number taken
// from the block's, so that the serial FP64 work of the blocks on an SM falls
// on different sub-partitions) while the others update the rest of A22.
__host__ __device__ inline size_t cta_smem_bytes(int N, int nthr) {
    return sizeof(zc) * ((size_t)N * (N + 1) / 2 + 3 * (size_t)N + nthr) + (4 + nthr / 32) * sizeof(double);
}

// Threads from which u is summed by all warps: equal times at 256 (70 - 112 bands),
// 4 % slower at 128 (33 bands 0.69 -> 0.72 ms), where several CTAs share the SM.
constexpr int kWideU = 512;
template <int NT>
__global__ void __launch_bounds__(NT) hetrd64_cta_kernel(int N, int64_t batch, zc* __restrict__ Ain) {
    extern __shared__ __align__(16) unsigned char smem64[];
    zc* P = reinterpret_cast<zc*>(smem64);
    zc* svb = P + (size_t)N * (N + 1) / 2;  // two reflectors
    zc* su = svb + 2 * N;
    zc* part = su + N;
    double* sc = reinterpret_cast<double*>(part + NT);  // tau of even and odd steps
    double* s_vav = sc + 4;                              // partial v^H A v per warp
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = NT / 32;
    for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
        const int lead = (int)((b / gridDim.x + blockIdx.x) % NW);
        zc* A = Ain + b * N * N;
        for (int e = tid; e < N * N; e += NT) {
            const int r = e / N, c = e - r * N;
            if (c < r) continue;
            zc a = A[e];
            if (c == r) a.im = 0.0;
            P[pk_off(N, r) + c - r] = a;
        }
        __syncthreads();
        auto make = [&](int j) {
            zc tau;
            double beta;
            zc* row = P + pk_off(N, j);
            reflector64(row + 1, N - 1 - j, lane, svb + (j & 1) * N, A + (size_t)j * N + j + 1, tau, beta);
            if (lane == 0) {
                A[(size_t)j * N + j] = mk(row[0].re, beta);
                A[(size_t)(j + 1) * N + j] = tau;
                sc[2 * (j & 1)] = tau.re;
                sc[2 * (j & 1) + 1] = tau.im;
            }
        };
        if (warp == lead) make(0);
        __syncthreads();
        for (int j = 0; j < N - 1; ++j) {
            const int m = N - 1 - j;
            const zc* sv = svb + (j & 1) * N;
            zc* T22 = P + pk_off(N, j + 1);
            const int Q = max(1, NT / m);
            for (int t = tid; t < m * Q; t += NT) {
                const int q = t / m, i = t - q * m;
                part[t] = row_times(T22, m, i, q, Q, sv);
            }
            __syncthreads();
            if constexpr (NT >= kWideU) {
                // one CTA on the SM: u with one row per thread, as a lone warp would have a
                // quarter of the FP64 rate (1024 x 128 bands 14.5 -> 13.7 ms)
                const zc tau = mk(sc[2 * (j & 1)], sc[2 * (j & 1) + 1]);
                zc u = mk(0.0, 0.0), v = mk(0.0, 0.0);
                if (warp * 32 < m) {
                    double s = 0.0;
                    if (tid < m) {
                        zc acc = part[tid];
                        for (int q = 1; q < Q; ++q) acc = acc + part[q * m + tid];
                        v = sv[tid];
                        s = fma(v.re, acc.re, v.im * acc.im);
                        u = tau * acc;
                    }
                    s = wsum(s);
                    if (lane == 0) s_vav[warp] = s;
                }
                __syncthreads();
                if (tid < m) {
                    double s = s_vav[0];  // v^H A v (real)
                    for (int w = 1; w < (m + 31) / 32; ++w) s += s_vav[w];
                    const double a2 = -0.5 * fma(tau.re, tau.re, tau.im * tau.im) * s;
                    su[tid] = mk(fma(a2, v.re, u.re), fma(a2, v.im, u.im));
                }
                __syncthreads();
            } else {
                // the other CTAs of the SM fill the gap: one warp, one barrier less
                if (warp == lead) {
                    const zc tau = mk(sc[2 * (j & 1)], sc[2 * (j & 1) + 1]);
                    double s = 0.0;
                    for (int i = lane; i < m; i += 32) {
                        zc acc = part[i];
                        for (int q = 1; q < Q; ++q) acc = acc + part[q * m + i];
                        s = fma(sv[i].re, acc.re, fma(sv[i].im, acc.im, s));
                        su[i] = tau * acc;
                    }
                    s = wsum(s);
                    const double a2 = -0.5 * fma(tau.re, tau.re, tau.im * tau.im) * s;
                    for (int i = lane; i < m; i += 32) {
                        const zc w = su[i];
                        su[i] = mk(fma(a2, sv[i].re, w.re), fma(a2, sv[i].im, w.im));
                    }
                }
                __syncthreads();
            }
            if (warp == lead) {
                for (int l = lane; l < m; l += 32) rank2_elem(T22 + l, sv, su, 0, l);
                __syncwarp();
                if (m > 1) make(j + 1);
            } else {
                const int ot = tid - (warp > lead ? 32 : 0), m1 = m - 1, tot = m1 * m / 2;
                zc* T1 = T22 + m;  // rows 1 .. of A22: order m - 1
                for (int t = ot; t < tot; t += NT - 32) {
                    int r, l;
                    fold_index(m1, t, r, l);
                    rank2_elem(T1 + pk_off(m1, r) + l - r, sv + 1, su + 1, r, l);
                }
            }
            __syncthreads();
        }
        if (tid == 0) A[(size_t)N * N - 1] = mk(P[pk_off(N, N - 1)].re, 0.0);
        __syncthreads();
    }
}

// ------------------------------------------------------ tridiagonal stage --
// Cluster marks of a matrix: bit i of the first ceil(N / 32) words = eigenvalue
// i is within 1e-3 ||T|| of eigenvalue i - 1, then as many words marking the
// eigenvalues whose vector tri64 has not formed, then a count of those.
__device__ __forceinline__ unsigned* marks_of(zc* A, int N) {
    return reinterpret_cast<unsigned*>(A + (size_t)(N - 1) * N);
}

struct TriShared {
    double *d, *e, *lam;
    float *fd, *fe2, *x0;
    unsigned* marks;  // 2 W + 1 words
    double *lo, *hi;  // Gershgorin bounds, one each
    int* sc;          // exponent of the scaling, bad flag
};
__host__ __device__ inline size_t tri_smem_bytes(int N) {
    return 8 * (3 * (size_t)N + 2) + 4 * (3 * (size_t)N) + 4 * (2 * (size_t)((N + 31) / 32) + 1) + 4 * 2 + 16;
}
__device__ __forceinline__ TriShared tri_carve(unsigned char* base, int N) {
    TriShared s;
    s.d = reinterpret_cast<double*>(base);
    s.e = s.d + N;
    s.lam = s.e + N;
    s.lo = s.lam + N;
    s.hi = s.lo + 1;
    s.fd = reinterpret_cast<float*>(s.hi + 1);
    s.fe2 = s.fd + N;
    s.x0 = s.fe2 + N;
    s.marks = reinterpret_cast<unsigned*>(s.x0 + N);
    s.sc = reinterpret_cast<int*>(s.marks + 2 * ((N + 31) / 32) + 1);
    return s;
}

// pivots nearer to zero than this (T scaled to norm 1 .. 2) are replaced by it, negative
constexpr double kPert = DBL_EPSILON;
__device__ __forceinline__ double guard(double q) {
    // hi word of 2^-52: compare magnitudes as integers (NaN passes through)
    return (hi_abs(q) < 0x3cb00000) ? -kPert : q;
}

__device__ __forceinline__ int sturm64(int N, const double* d, const double* e, double x) {
    double q = guard(d[0] - x);
    int cnt = __double2hiint(q) < 0;
    for (int k = 1; k < N; ++k) {
        const double ek = e[k - 1];
        q = guard(fma(-ek, ek * fast_rcp(q), d[k] - x));
        cnt += __double2hiint(q) < 0;
    }
    return cnt;
}

constexpr float kSame = 2e-5f;     // FP32 eigenvalues nearer than this are bisected in FP64
constexpr double kReach = 5e-6;    // bound on the FP32 stage's error (about 1e-6 at worst, ||T|| < 2)
constexpr float kCluster = 1e-3f;  // gap below which vectors are orthogonalised (of ||T||)

// z_i = -p_i z_(i -+ 1) from the twist outwards, over the ratios p_i in u(i).re
// (four loads ahead of the multiplications)
__device__ __forceinline__ void vector_side(zc* u, int r, int dir, int n, int N, double z) {
    const int64_t step = (int64_t)dir * N;
    zc* p = u + (int64_t)r * N + step;
    for (; n >= 4; n -= 4, p += 4 * step) {
        const double p0 = p[0].re, p1 = p[step].re, p2 = p[2 * step].re, p3 = p[3 * step].re;
        z *= -p0;
        p[0] = mk(z, 0.0);
        z *= -p1;
        p[step] = mk(z, 0.0);
        z *= -p2;
        p[2 * step] = mk(z, 0.0);
        z *= -p3;
        p[3 * step] = mk(z, 0.0);
    }
    for (; n > 0; --n, p += step) {
        z *= -p->re;
        *p = mk(z, 0.0);
    }
}

// Values only: the FP32 pivots of row k (N floats) go to A beside the diagonal.
__device__ __forceinline__ float* pivot_row(zc* A, int N, int k) {
    return reinterpret_cast<float*>(A + (size_t)k * N + (k < N / 2 ? N / 2 : 0));
}

// MPC matrices per CTA (1 when N > 64), one thread per eigenvalue; with few
// matrices each is shared by `parts` CTAs of `len` eigenvalues (MPC = 1; E is then
// put in order by tri64_order_kernel, the marks are cleared by the caller).
// Scratch: VEC: the ratios of the twisted factorisation go to U(k, i).re, where
// the vector then goes; values only: pivot_row.
template <bool VEC>
__global__ void __launch_bounds__(512) tri64_kernel(int N, int64_t batch, int MPC, int parts, int len,
                                                    zc* __restrict__ Ain,
                                                    double* __restrict__ Eout, zc* __restrict__ Uout,
                                                    int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smem64[];
    const size_t stride = (tri_smem_bytes(N) + 15) & ~size_t(15);
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nthr >> 5;
    const int W = (N + 31) / 32;
    for (int64_t unit = blockIdx.x; unit < (batch + MPC - 1) / MPC * parts; unit += gridDim.x) {
        const int64_t b0 = unit / parts * MPC;
        const int nm = (int)min((int64_t)MPC, batch - b0);
        // this CTA's eigenvalues [i0, i0 + ni) of each matrix, [h0, h0 + nh) with their neighbours
        const int i0 = (int)(unit % parts) * len, ni = min(len, N - i0);
        const int h0 = max(i0 - 1, 0), nh = min(i0 + ni + 1, N) - h0;
        for (int t = tid; t < nm * N; t += nthr) {
            const int mt = t / N, k = t - mt * N;
            const TriShared s = tri_carve(smem64 + mt * stride, N);
            const zc de = Ain[((b0 + mt) * N + k) * N + k];
            s.d[k] = de.re;
            s.e[k] = (k < N - 1) ? de.im : 0.0;
            if (k < 2 * W + 1) s.marks[k] = 0;
            for (int w = N + k; w < 2 * W + 1; w += N) s.marks[w] = 0;
        }
        __syncthreads();
        // per matrix: deflation (off-diagonals below eps (|d_i| + |d_i+1|) are set to
        // zero, as QR-type solvers do, so decoupled 1x1 blocks give d_i exactly),
        // Gershgorin bounds, power-of-two scaling to ||T|| in [1, 2), FP32 copies
        for (int mt = warp; mt < nm; mt += nw) {
            const TriShared s = tri_carve(smem64 + mt * stride, N);
            bool bad = false;
            for (int k = lane; k < N; k += 32) {
                double ek = s.e[k];
                bad = bad || !isfinite(s.d[k]) || !isfinite(ek);
                if (k < N - 1 && fabs(ek) <= DBL_EPSILON * (fabs(s.d[k]) + fabs(s.d[k + 1]))) ek = 0.0;
                s.e[k] = ek;
            }
            __syncwarp();
            double lo = INFINITY, hi = -INFINITY;
            for (int k = lane; k < N; k += 32) {
                const double r = (k > 0 ? fabs(s.e[k - 1]) : 0.0) + fabs(s.e[k]);
                lo = fmin(lo, s.d[k] - r);
                hi = fmax(hi, s.d[k] + r);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                lo = fmin(lo, __shfl_xor_sync(kFull, lo, o));
                hi = fmax(hi, __shfl_xor_sync(kFull, hi, o));
            }
            bad = __any_sync(kFull, bad);
            double tn = fmax(fabs(lo), fabs(hi));
            if (bad || !(tn < INFINITY)) {
                bad = true;
                tn = 1.0;
                lo = -1.0;
                hi = 1.0;
            }
            const int ex = (tn > 0.0) ? ilogb(tn) : 0;
            if (lane == 0) {
                s.sc[0] = ex;
                s.sc[1] = bad;
                *s.lo = scalbn(lo, -ex);
                *s.hi = scalbn(hi, -ex);
                if (bad && status) atomicOr(status, 1);
            }
            __syncwarp();
            for (int k = lane; k < N; k += 32) {
                const double dk = scalbn(s.d[k], -ex), ek = scalbn(s.e[k], -ex);
                s.d[k] = dk;
                s.e[k] = ek;
                s.fd[k] = (float)dk;
                s.fe2[k] = (float)ek * (float)ek;
            }
        }
        __syncthreads();
        // FP32 bisection on the FP32 copy of T
        for (int t = tid; t < nm * nh; t += nthr) {
            const int mt = t / nh, i = h0 + t - mt * nh;
            const TriShared s = tri_carve(smem64 + mt * stride, N);
            float a = (float)*s.lo - 1e-6f, c = (float)*s.hi + 1e-6f;
            for (int it = 0; it < 26 && c - a > 1.5e-7f; ++it) {
                const float x = 0.5f * (a + c);
                float q = s.fd[0] - x;
                if (fabsf(q) < 1e-30f) q = -1e-30f;
                int cnt = q < 0.f;
                for (int k = 1; k < N; ++k) {
                    q = (s.fd[k] - x) - __fdividef(s.fe2[k - 1], q);
                    if (fabsf(q) < 1e-30f) q = -1e-30f;
                    cnt += q < 0.f;
                }
                if (cnt > i)
                    c = x;
                else
                    a = x;
            }
            s.x0[i] = 0.5f * (a + c);
        }
        __syncthreads();
        for (int t = tid; t < nm * ni; t += nthr) {
            const int mt = t / ni, i = i0 + t - mt * ni;
            const int64_t b = b0 + mt;
            const TriShared s = tri_carve(smem64 + mt * stride, N);
            const float x0 = s.x0[i];
            const float gl = (i > 0) ? x0 - s.x0[i - 1] : INFINITY, gr = (i < N - 1) ? s.x0[i + 1] - x0 : INFINITY;
            const double tn = fmax(fabs(*s.lo), fabs(*s.hi));
            const float ctol = kCluster * (float)tn;
            const bool iso = gl > ctol && gr > ctol;
            if (VEC && gl <= ctol) atomicOr(&s.marks[i >> 5], 1u << (i & 31));
            bool done = false;
            double lam = 0.0;
            if (gl > kSame && gr > kSame) {
                // twist index from the FP32 factorisation
                float* uf = VEC ? reinterpret_cast<float*>(Uout + b * N * N + i) : nullptr;
                zc* Ab = Ain + b * N * N;
                auto fs = [&](int k) -> float& { return VEC ? uf[4 * (size_t)N * k] : pivot_row(Ab, N, k)[i]; };
                float q = s.fd[0] - x0;
                if (fabsf(q) < 1e-7f) q = -1e-7f;
                fs(0) = q;
                for (int k = 1; k < N; ++k) {
                    q = (s.fd[k] - x0) - __fdividef(s.fe2[k - 1], q);
                    if (fabsf(q) < 1e-7f) q = -1e-7f;
                    fs(k) = q;
                }
                int r = N - 1;
                float best = fabsf(q);
                q = s.fd[N - 1] - x0;
                if (fabsf(q) < 1e-7f) q = -1e-7f;
                for (int k = N - 2; k >= 0; --k) {
                    const float dk = s.fd[k] - x0;
                    q = dk - __fdividef(s.fe2[k], q);
                    if (fabsf(q) < 1e-7f) q = -1e-7f;
                    const float g = fabsf(fs(k) + q - dk);
                    if (g < best) {
                        best = g;
                        r = k;
                    }
                }
                double* ps = VEC ? &(Uout + b * N * N + i)->re : nullptr;
                double x = (double)x0;
                for (int it = 0; it < 8; ++it) {
                    // D+ from the top to r, then D- from the bottom to r: N - 1 steps in all
                    int pos = 0, dir = 1;
                    double raw = s.d[0] - x, sum = 0.0, qt = 0.0, st = 0.0;
                    if (r == 0) {
                        qt = raw;
                        pos = N - 1;
                        dir = -1;
                        raw = s.d[N - 1] - x;
                    }
                    double qq = guard(raw);
                    for (int k = 1; k < N; ++k) {
                        const double ek = s.e[dir > 0 ? pos : pos - 1];
                        const double p = ek * fast_rcp(qq);
                        if (VEC) ps[2 * (size_t)pos * N] = p;
                        const double p2 = p * p;
                        sum = fma(p2, sum, p2);
                        pos += dir;
                        raw = fma(-ek, p, s.d[pos] - x);
                        if (dir > 0 && pos == r) {  // the twist: on to the bottom part
                            qt = raw;
                            st = sum;
                            sum = 0.0;
                            pos = N - 1;
                            dir = -1;
                            raw = s.d[N - 1] - x;
                        }
                        qq = guard(raw);
                    }
                    const double g = qt + raw - (s.d[r] - x);
                    const double n2 = 1.0 + st + sum;
                    // ratios that outgrow the range would pass for convergence (g / n2 = 0)
                    if (hi_abs(n2) >= 0x7ff00000) break;
                    const double cor = g / n2;
                    x += cor;
                    if (!(fabs(x - (double)x0) <= kReach)) break;
                    // the vector is that of x before the correction: with 4 eps here vectors of
                    // neighbours were 2.5 times as far from orthogonal (64 bands 1.1e-13, 2.6e-14 with
                    // 1), for no pass less
                    if (fabs(cor) <= DBL_EPSILON * tn) {
                        lam = x;
                        done = true;
                        if (VEC && iso) {
                            const double inv = 1.0 / sqrt(n2);
                            zc* u = Uout + b * N * N + i;
                            u[(size_t)r * N] = mk(inv, 0.0);
                            vector_side(u, r, -1, r, N, inv);
                            vector_side(u, r, 1, N - 1 - r, N, inv);
                        }
                        break;
                    }
                }
            }
            if (VEC && !(done && iso)) {
                atomicOr(&s.marks[W + (i >> 5)], 1u << (i & 31));
                atomicAdd(&s.marks[2 * W], 1u);
            }
            if (!done) {
                // FP64 bisection from the FP32 bracket (from the Gershgorin bounds if that does not hold it)
                double a = (double)x0 - kReach, c = (double)x0 + kReach;
                if (sturm64(N, s.d, s.e, a) > i || sturm64(N, s.d, s.e, c) <= i) {
                    a = *s.lo - 8.0 * DBL_EPSILON * fmax(tn, 1.0);
                    c = *s.hi + 8.0 * DBL_EPSILON * fmax(tn, 1.0);
                }
                for (int it = 0; it < 64 && c - a > 2.0 * DBL_EPSILON * (tn + fmax(fabs(a), fabs(c))); ++it) {
                    const double x = 0.5 * (a + c);
                    if (sturm64(N, s.d, s.e, x) > i)
                        c = x;
                    else
                        a = x;
                }
                lam = 0.5 * (a + c);
                // an isolated diagonal entry inside the final bracket is the exact eigenvalue
                for (int k = 0; k < N; ++k) {
                    const bool one = (k == 0 || s.e[k - 1] == 0.0) && s.e[k] == 0.0;
                    if (one && s.d[k] >= a && s.d[k] <= c) {
                        lam = s.d[k];
                        break;
                    }
                }
            }
            s.lam[i] = lam;
        }
        __syncthreads();
        // eigenvalues bisected from their own brackets may differ in the last bits in
        // either order: each run of neighbours nearer than kSame is put in order
        if (parts == 1) for (int t = tid; t < nm * N; t += nthr) {
            const int mt = t / N, i = t - mt * N;
            const TriShared s = tri_carve(smem64 + mt * stride, N);
            if ((i > 0 && s.x0[i] - s.x0[i - 1] <= kSame) || i == N - 1 || s.x0[i + 1] - s.x0[i] > kSame) continue;
            for (int k = i + 1; k < N && s.x0[k] - s.x0[k - 1] <= kSame; ++k) {
                const double v = s.lam[k];
                int p = k - 1;
                for (; p >= i && s.lam[p] > v; --p) s.lam[p + 1] = s.lam[p];
                s.lam[p + 1] = v;
            }
        }
        __syncthreads();
        for (int t = tid; t < nm * ni; t += nthr) {
            const int mt = t / ni, i = i0 + t - mt * ni;
            const TriShared s = tri_carve(smem64 + mt * stride, N);
            Eout[(b0 + mt) * N + i] = scalbn(s.lam[i], s.sc[0]);
        }
        if (VEC)
            for (int t = tid; t < nm * (2 * W + 1); t += nthr) {
                const int mt = t / (2 * W + 1), w = t - mt * (2 * W + 1);
                const unsigned v = tri_carve(smem64 + mt * stride, N).marks[w];
                unsigned* g = marks_of(Ain + (b0 + mt) * N * N, N) + w;
                if (parts == 1)
                    *g = v;
                else if (w < 2 * W)
                    atomicOr(g, v);
                else
                    atomicAdd(g, v);
            }
        __syncthreads();
    }
}

// Eigenvalues of a matrix whose parts were found by different CTAs: neighbours
// bisected from their own brackets may differ in the last bits in either order.
__global__ void __launch_bounds__(256) tri64_order_kernel(int N, int64_t batch, double* __restrict__ E) {
    for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
        double* e = E + b * N;
        bool out = false;
        for (int i = threadIdx.x; i < N - 1; i += blockDim.x) out = out || e[i] > e[i + 1];
        if (__syncthreads_or(out) && threadIdx.x == 0)
            for (int i = 1; i < N; ++i) {
                const double v = e[i];
                int p = i - 1;
                for (; p >= 0 && e[p] > v; --p) e[p + 1] = e[p];
                e[p + 1] = v;
            }
        __syncthreads();
    }
}

// One inverse-iteration solve (T - lam I) y = x in place (stride G), by
// elimination with partial pivoting; u0 (reciprocals), u1, u2 hold the rows of U.
__device__ void tri_solve64(int N, const double* d, const double* e, double lam, double pert, double* x, double* u0,
                            double* u1, double* u2, int G) {
    double cd = d[0] - lam, cs = (N > 1) ? e[0] : 0.0, cr = x[0];
    for (int i = 0; i < N - 1; ++i) {
        const double b = e[i], a1 = d[i + 1] - lam, b1 = (i + 2 < N) ? e[i + 1] : 0.0, xn = x[(i + 1) * G];
        if (fabs(cd) >= fabs(b)) {
            double piv = cd;
            if (fabs(piv) < pert) piv = (piv < 0.0) ? -pert : pert;
            const double inv = fast_rcp(piv), mlt = b * inv;
            u0[i * G] = inv;
            u1[i * G] = cs;
            u2[i * G] = 0.0;
            x[i * G] = cr;
            cd = a1 - mlt * cs;
            cs = b1;
            cr = xn - mlt * cr;
        } else {
            const double inv = fast_rcp(b), mlt = cd * inv;
            u0[i * G] = inv;
            u1[i * G] = a1;
            u2[i * G] = b1;
            x[i * G] = xn;
            cd = cs - mlt * a1;
            cs = -mlt * b1;
            cr = cr - mlt * xn;
        }
    }
    if (fabs(cd) < pert) cd = (cd < 0.0) ? -pert : pert;
    double y2 = 0.0, y1 = cr * fast_rcp(cd);
    x[(N - 1) * G] = y1;
    for (int i = N - 2; i >= 0; --i) {
        double r = fma(-u1[i * G], y1, x[i * G]);
        if (i + 2 < N) r = fma(-u2[i * G], y2, r);
        const double yi = r * u0[i * G];
        x[i * G] = yi;
        y2 = y1;
        y1 = yi;
    }
}

// Clusters that a warp takes at once, with 4 N doubles of scratch each.
int cluster_lanes(int N) { return (int)std::max<size_t>(1, std::min<size_t>(32, (64 * 1024) / (32 * (size_t)N))); }
size_t cluster_smem_bytes(int N) { return sizeof(double) * (size_t)N * (3 + 4 * cluster_lanes(N)); }

// Vectors that tri64 left: clusters (runs of marked neighbours) and single
// vectors that did not converge, one lane per cluster, inverse iteration with
// modified Gram-Schmidt against the earlier members.  One warp per matrix, or per
// `len` eigenvalues of it (clusters that start there) when there are few matrices;
// one without marks costs one read.
__global__ void __launch_bounds__(32) tri64_cluster_kernel(int N, int64_t batch, int G, int parts, int len,
                                                           const zc* __restrict__ Ain,
                                                           const double* __restrict__ Ein, zc* __restrict__ Uout) {
    extern __shared__ __align__(16) unsigned char smem64[];
    double* d = reinterpret_cast<double*>(smem64);
    double* e = d + N;
    double* lam = e + N;
    double* scr = lam + N;  // 4 N G
    const int lane = threadIdx.x, W = (N + 31) / 32;
    for (int64_t unit = blockIdx.x; unit < batch * parts; unit += gridDim.x) {
        const int64_t b = unit / parts;
        const int i0 = (int)(unit % parts) * len, i1 = min(i0 + len, N);
        const zc* A = Ain + b * N * N;
        const unsigned* mk_ = marks_of(const_cast<zc*>(A), N);
        if (mk_[2 * W] == 0) continue;
        zc* U = Uout + b * N * N;
        double tn = 0.0;
        for (int k = lane; k < N; k += 32) {
            const zc de = A[(size_t)k * N + k];
            d[k] = de.re;
            e[k] = (k < N - 1) ? de.im : 0.0;
            lam[k] = Ein[b * N + k];
        }
        __syncwarp();
        for (int k = lane; k < N - 1; k += 32)
            if (fabs(e[k]) <= DBL_EPSILON * (fabs(d[k]) + fabs(d[k + 1]))) e[k] = 0.0;
        __syncwarp();
        for (int k = lane; k < N; k += 32)
            tn = fmax(tn, fabs(d[k]) + fabs(e[k]) + (k > 0 ? fabs(e[k - 1]) : 0.0));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tn = fmax(tn, __shfl_xor_sync(kFull, tn, o));
        const int ex = (tn > 0.0 && tn < INFINITY) ? ilogb(tn) : 0;
        __syncwarp();
        for (int k = lane; k < N; k += 32) {
            const double ek = scalbn(e[k], -ex);
            d[k] = scalbn(d[k], -ex);
            e[k] = hi_abs(ek) < 0x04000000 ? 0.0 : ek;  // 2^-959: a pivot of tri_solve64 has its reciprocal
            lam[k] = scalbn(lam[k], -ex);
        }
        tn = scalbn(tn, -ex);
        const double pert = fmax(DBL_EPSILON * tn, DBL_MIN);
        __syncwarp();
        auto joined = [&](int i) { return (mk_[i >> 5] >> (i & 31)) & 1u; };
        auto redo = [&](int i) { return (mk_[W + (i >> 5)] >> (i & 31)) & 1u; };
        for (int g0 = i0; g0 < i1; g0 += G) {
            const int i = g0 + lane;
            if (lane < G && i < i1 && !(i > 0 && joined(i)) && redo(i)) {
                int c1 = i;
                while (c1 + 1 < N && joined(c1 + 1)) ++c1;
                double* x = scr + lane;
                double* u0 = x + (size_t)N * G;
                double* u1 = u0 + (size_t)N * G;
                double* u2 = u1 + (size_t)N * G;
                double prev = -INFINITY;
                for (int jj = i; jj <= c1; ++jj) {
                    double shift = lam[jj];
                    // separate coincident shifts inside a cluster
                    const double tol = 10.0 * DBL_EPSILON * fmax(fabs(shift), tn * 1e-3);
                    if (jj > i && shift - prev < tol) shift = prev + tol;
                    prev = shift;
                    for (int r = 0; r < N; ++r) {
                        const unsigned h = hash32((unsigned)(r * 7919 + jj * 104729 + 12345));
                        x[r * G] = 1.0 + 0.5 * ((double)(h & 0xffff) / 65535.0 - 0.5);
                    }
                    for (int iter = 0; iter < 3; ++iter) {
                        tri_solve64(N, d, e, shift, pert, x, u0, u1, u2, G);
                        double amax = 0.0;
                        for (int r = 0; r < N; ++r) amax = fmax(amax, fabs(x[r * G]));
                        if (!(amax > 0.0) || isinf(amax)) {
                            for (int r = 0; r < N; ++r) x[r * G] = (r == (jj % N)) ? 1.0 : 0.0;
                            amax = 1.0;
                        }
                        const double sc = 1.0 / amax;
                        for (int r = 0; r < N; ++r) x[r * G] *= sc;
                        auto norm2 = [&]() {
                            double s = 0.0;
                            for (int r = 0; r < N; ++r) s += x[r * G] * x[r * G];
                            return s;
                        };
                        // once more where little is left (eigenvalues that the shifts do not tell
                        // apart give the earlier members again): what is left is then orthogonal
                        double nrm = norm2();
                        for (int pass = 0; pass < 2; ++pass) {
                            const double before = nrm;
                            for (int pp = i; pp < jj; ++pp) {
                                double dot = 0.0;
                                for (int r = 0; r < N; ++r) dot += U[(size_t)r * N + pp].re * x[r * G];
                                for (int r = 0; r < N; ++r) x[r * G] -= dot * U[(size_t)r * N + pp].re;
                            }
                            nrm = norm2();
                            if (!(nrm < 0.01 * before)) break;
                        }
                        const double inv = (nrm > 0.0) ? 1.0 / sqrt(nrm) : 0.0;
                        for (int r = 0; r < N; ++r) x[r * G] *= inv;
                    }
                    for (int r = 0; r < N; ++r) U[(size_t)r * N + jj] = mk(x[r * G], 0.0);
                }
            }
            __syncwarp();
        }
    }
}

// ---------------------------------------------------- back-transformation --
// U <- H_0 ... H_{N-2} U, in place, RS lanes per column (rows q, q + RS, ...,
// at most T each, in registers; the reflector is read twice, the second time
// from L1).  Columns first .. first + ncol - 1 of consecutive matrices follow each
// other, so warps are full for any N.
template <int T, int RS>
__global__ void __launch_bounds__(128, T <= 16 ? 5 : 3) bt64_kernel(int N, int64_t batch, const zc* __restrict__ Ain,
                                                      zc* __restrict__ Uout, int first, int ncol) {
    const int lane = threadIdx.x & 31, q = lane & (RS - 1);
    const int64_t cols = batch * ncol;
    const int64_t col0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / RS;
    const bool on = col0 < cols;
    const int64_t col = on ? col0 : cols - 1;
    const int64_t b = col / ncol;
    const int c = first + (int)(col - b * ncol);
    const zc* A = Ain + b * (int64_t)N * N + q;
    zc* U = Uout + b * (int64_t)N * N + c;
    zc u[T];
#pragma unroll
    for (int t = 0; t < T; ++t) {
        const int i = q + RS * t;
        u[t] = (i < N) ? U[(size_t)i * N] : mk(0.0, 0.0);
    }
    for (int j = N - 2; j >= 0; --j) {
        const zc* vrow = A + (size_t)j * N;
        const zc tau = A[(size_t)(j + 1) * N + j - q];
        const int t0 = (j + 1) / RS;
        auto velem = [&](int t) {
            const int i = q + RS * t;
            return (i > j && i < N) ? vrow[RS * t] : mk(0.0, 0.0);
        };
        zc a0 = mk(0.0, 0.0), a1 = mk(0.0, 0.0);
#pragma unroll
        for (int t = 0; t < T; ++t) {
            if (t >= t0 && RS * t < N) {
                if (t & 1)
                    fma_cjx(a1, velem(t), u[t]);
                else
                    fma_cjx(a0, velem(t), u[t]);
            }
        }
        zc acc = a0 + a1;
#pragma unroll
        for (int o = 1; o < RS; o <<= 1) {
            acc.re += __shfl_xor_sync(kFull, acc.re, o);
            acc.im += __shfl_xor_sync(kFull, acc.im, o);
        }
        zc s = tau * acc;
        s = mk(flip_if(s.re, true), flip_if(s.im, true));
#pragma unroll
        for (int t = 0; t < T; ++t)
            if (t >= t0 && RS * t < N) fma_cx(u[t], velem(t), s);
    }
    if (on) {
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int i = q + RS * t;
            if (i < N) U[(size_t)i * N] = u[t];
        }
    }
}

int sm_count() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 1;
    return n;
}

constexpr size_t kSmemCta = 226 * 1024;

int cta_threads(int N) { return N <= 64 ? 128 : (N <= 112 ? 256 : 512); }

template <int NT>
int launch_cta(cudaStream_t st, int N, int64_t batch, zc* A, int nsm) {
    const size_t smem = cta_smem_bytes(N, NT);
    if (int rc = allow_smem(hetrd64_cta_kernel<NT>, smem)) return rc;
    const int64_t per = std::max<int64_t>(1, std::min<int64_t>(2048 / NT, (int64_t)(kSmemCta / smem)));
    hetrd64_cta_kernel<NT><<<(unsigned)std::min<int64_t>(batch, nsm * per), NT, smem, st>>>(N, batch, A);
    TBG_LAUNCHED("hetrd64_cta_kernel");
    return TBG_OK;
}

template <int T, int RS>
int launch_bt(cudaStream_t st, int N, int64_t batch, const zc* A, zc* U, int first, int ncol) {
    const int64_t cols = 128 / RS;
    bt64_kernel<T, RS><<<(unsigned)((batch * ncol + cols - 1) / cols), 128, 0, st>>>(N, batch, A, U, first, ncol);
    TBG_LAUNCHED("bt64_kernel");
    return TBG_OK;
}

}  // namespace

// Whether the back-transformation takes the blocked form.  Its FP64 work (T) is a
// small part of the 4 N^3 FMA of bt64, which does not go beyond 256 bands; below
// kWYWork a block of reflectors the launches cost more than that saves, and below kWYMinN
// bands too little of a 128-row tile is used.  Blocks / single reflectors: 1000 x 56 bands
// 1.58 / 1.31 ms, 100 x 64 0.38 / 0.40, 1000 x 64 1.83 / 2.41, 50 x 97 0.62 / 0.53, 100 x 97
// 0.72 / 0.97, 16 and 24 x 128 0.66 / 0.70 and 0.67 / 0.81, 1024 x 128 5.2 / 17.3, 12 and
// 100 x 160 0.86 / 0.73 and 1.4 / 4.7, 10 x 200 1.16 / 1.14, 8 x 250 1.36 / 1.65.
constexpr int kWYMinN = 64;
constexpr double kWYWork = 1.0e8;
static bool use_wy(int N, int64_t batch, int ncol) {
    // (T's part is the same for fewer columns: 32 of 64 bands, 4032 matrices, 5.2 ms before the
    // leading ones were added apart, against 4.5)
    return N > 256 || (N >= kWYMinN && (2 * ncol > N || N >= 96) &&
                       4.0 * N * N * (double)ncol * batch >= kWYWork * ((N + 62) / 64));
}

// Largest matrix whose packed triangle and vectors fit one CTA's shared memory.
bool eig64_fits(int N) { return N <= kWarpMax || cta_smem_bytes(N, cta_threads(N)) <= kSmemCta; }

// Eigenvalues E (ascending) and, when U is given, eigenvectors (columns) of
// batch N x N matrices A (upper triangles read, destroyed), N >= 1 (>= 4 with
// vectors).  With timed = false nothing is allocated, which
// requires eig64_fits(N) (and N <= 256 with vectors).  Only the vectors first ..
// first + ncol - 1 (all for ncol < 0) are finished; the other columns hold scratch.
int eig64(cudaStream_t st, int N, int64_t batch, zc* A, double* E, zc* U, int* status_d, bool timed, int first,
          int ncol) {
    if (batch <= 0) return TBG_OK;
    if (ncol < 0) ncol = N - first;
    const int nsm = sm_count();
    const double n3 = (double)N * N * N * batch;
    int rc = TBG_OK;
    auto reduce = [&]() -> int {
        if (!eig64_fits(N)) return hetrd64_big(st, N, batch, A, status_d);
        if (N <= kWarpMax) {
            // one warp per CTA while that spreads a small batch over more SMs
            const int wpc = batch > (int64_t)nsm * 8 ? kWarpsPerCta : 1;
            const size_t smem = sizeof(zc) * warp_smem_elems(N) * wpc;
            if (int r = allow_smem(hetrd64_warp_kernel, smem)) return r;
            const int64_t ctas = (batch + wpc - 1) / wpc;
            hetrd64_warp_kernel<<<(unsigned)std::min<int64_t>(ctas, nsm * 16), 32 * wpc, smem, st>>>(N, batch, A);
            TBG_LAUNCHED("hetrd64_warp_kernel");
            return TBG_OK;
        }
        switch (cta_threads(N)) {
            case 128: return launch_cta<128>(st, N, batch, A, nsm);
            case 256: return launch_cta<256>(st, N, batch, A, nsm);
            default: return launch_cta<512>(st, N, batch, A, nsm);
        }
    };
    auto tri = [&]() -> int {
        const int mpc = N <= 64 ? std::max(1, 128 / N) : 1;
        // few large matrices: the eigenvalues of each over several CTAs (12 matrices of
        // 512: 1.3 ms over 16 CTAs each; with vectors, most of them in clusters, 12.0
        // against 51.6 ms when one warp per matrix does the clusters)
        int parts = 1, len = N;
        if (N > 64 && batch < 2 * nsm) {
            parts = (int)std::min<int64_t>((N + 31) / 32, (2 * nsm + batch - 1) / batch);
            len = ((N + parts - 1) / parts + 31) & ~31;
            parts = (N + len - 1) / len;
        }
        const int thr = std::min(512, (mpc * len + 31) & ~31);
        const size_t smem = mpc * ((tri_smem_bytes(N) + 15) & ~size_t(15));
        const int64_t ctas = std::min<int64_t>((batch + mpc - 1) / mpc * parts, (int64_t)nsm * 64);
        auto order = [&]() -> int {
            if (parts == 1) return TBG_OK;
            tri64_order_kernel<<<(unsigned)std::min<int64_t>(batch, nsm * 8), 256, 0, st>>>(N, batch, E);
            TBG_LAUNCHED("tri64_order_kernel");
            return TBG_OK;
        };
        if (U) {
            if (int r = allow_smem(tri64_kernel<true>, smem)) return r;
            if (parts > 1)
                TBG_CUDA(cudaMemset2DAsync(A + (size_t)(N - 1) * N, sizeof(zc) * (size_t)N * N, 0,
                                           4 * (2 * (size_t)((N + 31) / 32) + 1), batch, st));
            tri64_kernel<true><<<(unsigned)ctas, thr, smem, st>>>(N, batch, mpc, parts, len, A, E, U, status_d);
            TBG_LAUNCHED("tri64_kernel");
            if (int r = order()) return r;
            const int G = cluster_lanes(N);
            const size_t csm = cluster_smem_bytes(N);
            if (int r = allow_smem(tri64_cluster_kernel, csm)) return r;
            tri64_cluster_kernel<<<(unsigned)std::min<int64_t>(batch * parts, (int64_t)nsm * 32), 32, csm, st>>>(
                N, batch, G, parts, len, A, E, U);
            TBG_LAUNCHED("tri64_cluster_kernel");
        } else {
            if (int r = allow_smem(tri64_kernel<false>, smem)) return r;
            tri64_kernel<false><<<(unsigned)ctas, thr, smem, st>>>(N, batch, mpc, parts, len, A, E, nullptr, status_d);
            TBG_LAUNCHED("tri64_kernel");
            if (int r = order()) return r;
        }
        return TBG_OK;
    };
    auto back = [&]() -> int {
        if (timed && use_wy(N, batch, ncol)) return bt64_wy(st, N, batch, A, U, status_d, first, ncol);
        // 32 rows a lane (fewer shuffles per column) when that still gives every
        // sub-partition a warp, else 16: 128 bands 17.5 against 31.6 ms per 1024
        // matrices, 64 bands 8.5 against 14.4 per 4032; up to 32 bands 16 rows, whose
        // shorter warps leave a shorter last wave (26 bands 0.65 against 0.92 ms per 2304)
        const int64_t warps32 = batch * ncol * ((N + 31) / 32) / 32;
        const bool wide = warps32 >= 4 * (int64_t)nsm;
        if (N <= 16) return launch_bt<16, 1>(st, N, batch, A, U, first, ncol);
        if (N <= 32) return launch_bt<16, 2>(st, N, batch, A, U, first, ncol);
        if (N <= 64)
            return wide ? launch_bt<32, 2>(st, N, batch, A, U, first, ncol)
                        : launch_bt<16, 4>(st, N, batch, A, U, first, ncol);
        if (N <= 128)
            return wide ? launch_bt<32, 4>(st, N, batch, A, U, first, ncol)
                        : launch_bt<16, 8>(st, N, batch, A, U, first, ncol);
        return wide ? launch_bt<32, 8>(st, N, batch, A, U, first, ncol)
                    : launch_bt<16, 16>(st, N, batch, A, U, first, ncol);
    };
    if (!timed) {
        if ((rc = reduce()) || (rc = tri())) return rc;
        return U ? back() : TBG_OK;
    }
    {
        KTimer kt(st, "hetrd64_kernel", 16.0 / 3.0 * n3);
        if ((rc = reduce())) return rc;
    }
    {
        KTimer kt(st, "tri64_kernel");
        if ((rc = tri())) return rc;
    }
    if (!U) return TBG_OK;
    KTimer kt(st, "bt64_kernel", 8.0 * n3 * ncol / N);
    return back();
}

}  // namespace tbg

// Internal test hooks (not part of the public header).
// Dynamic shared memory of the solver's largest CTA for n bands (the panel kernel's with one
// CTA per matrix), bytes.
extern "C" int64_t tbg_internal_eig64_smem(int n) {
    using namespace tbg;
    size_t most = std::max(cluster_smem_bytes(n), (n <= 64 ? std::max(1, 128 / n) : 1) * ((tri_smem_bytes(n) + 15) & ~size_t(15)));
    if (n <= kWarpMax)
        most = std::max(most, sizeof(zc) * warp_smem_elems(n) * kWarpsPerCta);
    else
        most = std::max(most, eig64_fits(n) ? cta_smem_bytes(n, cta_threads(n)) : panel64_smem_bytes(n, 1));
    return (int64_t)most;
}
namespace {
__global__ void fast_math_kernel(int n, const double* x, double* rcp, double* rsq) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    rcp[i] = tbg::fast_rcp(x[i]);
    rsq[i] = tbg::fast_rsqrt(fabs(x[i]));
}
}  // namespace
// fast_rcp(x) and fast_rsqrt(|x|), host arrays.
extern "C" int tbg_internal_fast_math(int n, const double* x, double* rcp, double* rsq) {
    using namespace tbg;
    if (n <= 0) return TBG_OK;
    double* d = nullptr;
    TBG_CUDA(cudaMalloc(&d, sizeof(double) * 3 * (size_t)n));
    cudaError_t e = cudaMemcpy(d, x, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        fast_math_kernel<<<(n + 255) / 256, 256>>>(n, d, d + n, d + 2 * (size_t)n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(rcp, d + n, sizeof(double) * n, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(rsq, d + 2 * (size_t)n, sizeof(double) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? TBG_OK : cuda_error(e, "fast_math test");
}
