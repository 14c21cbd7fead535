// FP64 Hermitian reduction to tridiagonal form for matrices beyond one SM's
// shared memory: a cluster of CTAs per matrix, the matrix in L2.
//
// Blocked Householder reduction (the panel form of LAPACK's xLATRD): within a
// panel of kNB columns the trailing matrix A is left as it was at the panel's
// start and A_true = A - V W^H - W V^H; each step needs one product A v over the
// trailing block (4 FP64 FMA per element, two thirds less than updating it as it
// goes) and short products with the panel.  After the panel A -= [V W][W V]^H runs
// on the tensor cores (oz64.cu).  The FP64 pipe bounds the product A v, so a
// matrix is spread over as many SMs as the batch leaves free (clusters of up to
// 16 CTAs, rows dealt cyclically so that the shares stay equal as the block
// shrinks); two cluster barriers a step.
//
// 12 matrices of 512 bands (eigenvalues) 176 -> 15.5 ms, against one CTA per matrix; a
// step is 12.5 us of A v (10 at the pipe's rate, ten CTAs) and about as much of
// exchange, reductions and the panel's products.

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "eig64.cuh"
#include "tbgpu_internal.cuh"

namespace tbg {
namespace {

namespace cg = cooperative_groups;

constexpr int kNB = 16;          // columns of a panel: a row of [V | W] is one warp of complex values
constexpr int kPW = 2 * kNB;
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxCluster = 16;
constexpr int kRows = 4;         // rows of A v that a warp takes together

// Published by the CTAs of a matrix to each other, per matrix.
struct Exchange {
    zc* a;         // (N) current column below the diagonal
    zc* p;         // (N) A v
    zc* gh;        // (C, kPW) partial [V W]^H v
    double* norm;  // (C, kWarps) partial |a|^2 without the first entry
    double* s;     // (C, kWarps) partial v^H A v
};
__host__ __device__ inline size_t exchange_bytes(int N, int C) {
    return sizeof(zc) * (2 * (size_t)N + (size_t)C * kPW) + sizeof(double) * 2 * (size_t)C * kWarps;
}
__device__ __forceinline__ Exchange exchange_of(unsigned char* base, int N, int C) {
    Exchange x;
    x.a = reinterpret_cast<zc*>(base);
    x.p = x.a + N;
    x.gh = x.p + N;
    x.norm = reinterpret_cast<double*>(x.gh + C * kPW);
    x.s = x.norm + C * kWarps;
    return x;
}
__device__ __forceinline__ zc ldcg(const zc* p) {
    const double2 t = __ldcg(reinterpret_cast<const double2*>(p));
    return mk(t.x, t.y);
}

// Sums over the warp of R complex values per lane: lane l ends with the sum of
// value l mod R, in R - 1 + (5 - log2 R) additions per component
// instead of 5 R.
template <int R>
__device__ __forceinline__ zc warp_sums(zc (&v)[R], int lane) {
    constexpr unsigned all = 0xffffffffu;
#pragma unroll
    for (int h = R / 2; h > 0; h >>= 1) {
        const bool up = (lane & h) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const zc mine = up ? v[i + h] : v[i], give = up ? v[i] : v[i + h];
            v[i] = mk(mine.re + __shfl_xor_sync(all, give.re, h), mine.im + __shfl_xor_sync(all, give.im, h));
        }
    }
    zc r = v[0];
#pragma unroll
    for (int o = R; o < 32; o <<= 1) {
        r.re += __shfl_xor_sync(all, r.re, o);
        r.im += __shfl_xor_sync(all, r.im, o);
    }
    return r;
}

// Sum of n values in pairs (FP64 latency is long here: log2 n steps, not n).
template <int n>
__device__ __forceinline__ zc pair_sum(zc (&v)[n]) {
#pragma unroll
    for (int h = n / 2; h > 0; h >>= 1)
#pragma unroll
        for (int i = 0; i < h; ++i) v[i] = v[i] + v[i + h];
    return v[0];
}
// Sum over the C CTAs' warps of a published partial, by one warp; all requested at once.
__device__ __forceinline__ double sum_published(const double* x, int C, int lane) {
    constexpr int n = kMaxCluster * kWarps / 32;
    double v[n];
#pragma unroll
    for (int w = 0; w < n; ++w) v[w] = lane + 32 * w < C * kWarps ? __ldcg(x + lane + 32 * w) : 0.0;
#pragma unroll
    for (int h = n / 2; h > 0; h >>= 1)
#pragma unroll
        for (int i = 0; i < h; ++i) v[i] += v[i + h];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

// Matrices whose largest entry lies beyond 2^-300 or 2^300 are reduced times a power
// of two that brings it to 1 (products of their entries would leave the range); n: the
// exponent field of the largest entry, 0x7ff for NaN and Inf.
__device__ __forceinline__ int reduced_exp(int n) { return n == 0x7ff || (n >= 723 && n <= 1323) ? n : 1023; }

// One panel: columns j0 .. j0 + steps - 1 of every matrix.  Writes the reflectors,
// (d, e) and tau into A as hetrd64 does, and P = [V | W], Q = [W | V] (N x kPW),
// with V times and W over a power of two near the root of A's largest entry
// (nexp: its exponent field): the digit products share an exponent along a row.
// Cluster of C CTAs per matrix; CTA `rank` has the rows r = rank mod C.
__global__ void __launch_bounds__(kThreads) panel64_kernel(int N, int j0, int steps, zc* __restrict__ Ain,
                                                           zc* __restrict__ Pin, zc* __restrict__ Qin,
                                                           const int* __restrict__ nexp,
                                                           unsigned char* __restrict__ xin, int64_t xbytes) {
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int64_t b = blockIdx.x / C;
    zc* A = Ain + b * (int64_t)N * N;
    zc* P = Pin + b * (int64_t)N * kPW;
    zc* Q = Qin + b * (int64_t)N * kPW;
    const int half = (reduced_exp(nexp[b]) - 1022) / 2;
    const double vscale = scalbn(1.0, half), wscale = scalbn(1.0, -half);
    const Exchange X = exchange_of(xin + b * xbytes, N, C);
    extern __shared__ __align__(16) unsigned char smem_p[];
    zc* sa = reinterpret_cast<zc*>(smem_p);  // (N) column below the diagonal
    zc* sq = sa + N;                         // (own rows) A a, then p
    zc* sx = sq + (N + C - 1) / C;           // (own rows) part of the next column
    __shared__ zc s_part[kWarps][kPW];       // partial [V W]^H a per warp
    __shared__ zc s_mul[kPW], s_row[kPW];    // coefficients of V, W; the next row of [W V]
    __shared__ zc s_scal, s_tau, s_u1;
    __shared__ double s_beta, s_ca, s_d, s_up;
    __shared__ int s_next;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto first_own = [&](int r) { return r + ((rank - r) % C + C) % C; };  // own row at or after r

    // the first column as it stands
    {
        double nrm = 0.0;
        for (int r = first_own(j0) + C * tid; r < N; r += C * kThreads) {
            const zc x = A[(size_t)r * N + j0];
            if (r == j0) {
                s_d = x.re;
            } else {
                X.a[r] = x;
                if (r > j0 + 1) nrm += abs2(x);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
        if (lane == 0) X.norm[rank * kWarps + warp] = nrm;
    }
    for (int i = 0; i < steps; ++i) {
        const int j = j0 + i, f = j + 1;  // f: first row of the column
        const int r0 = first_own(f), nrows = r0 < N ? (N - 1 - r0) / C + 1 : 0;
        cl.sync();
        for (int t = tid; t < N - f; t += kThreads) sa[t] = ldcg(X.a + f + t);
        if (tid == 0) s_next = 0;
        __syncthreads();
        if (warp == 0) {
            // reflector of the column: H^H x = beta e_0 with beta real
            const double xn = sum_published(X.norm, C, lane);
            const Reflector64 r = reflector64_of(sa[0], xn, [&](double up) {
                double p = 0.0;
                for (int t = 1 + lane; t < N - f; t += 32) p += abs2(up * sa[t]);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
                return p;
            });
            if (lane == 0) {
                s_tau = r.tau;
                s_scal = r.scal;
                s_beta = r.beta;
                s_up = r.up;
            }
        }
        // q = A a without the first column, kRows own rows at a time by whichever warp is
        // free: a row's sum does not depend on who takes it
        const bool on = (lane & (kNB - 1)) < i;
        for (;;) {
            int g = 0;
            if (lane == 0) g = atomicAdd(&s_next, kRows);
            g = __shfl_sync(0xffffffffu, g, 0);
            if (g >= nrows) break;
            zc acc[kRows] = {};
            const zc* row[kRows];
#pragma unroll
            for (int k = 0; k < kRows; ++k) row[k] = A + (size_t)(r0 + C * min(g + k, nrows - 1)) * N + f;
#pragma unroll 2
            for (int c = lane; c < N - f; c += 32) {
                const zc x = c > 0 ? sa[c] : mk(0.0, 0.0);
#pragma unroll
                for (int k = 0; k < kRows; ++k) fma_cx(acc[k], row[k][c], x);
            }
            const zc q = warp_sums<kRows>(acc, lane);
            if (lane < kRows && g + lane < nrows) sq[g + lane] = q;
        }
        // partial [V W]^H a without the first row: a sum over rows, which are dealt out
        // in a fixed order so that a call's results are the same every time
        zc gh = mk(0.0, 0.0);
        if (on)
            for (int t = warp; t < nrows; t += kWarps) {
                const int r = r0 + C * t;
                if (r > f) fma_cjx(gh, P[(size_t)r * kPW + lane], sa[r - f]);
            }
        s_part[warp][lane] = gh;
        __syncthreads();
        // p = A v, v = (1, scal up a); publish p, [V W]^H v and v^H p of the own rows
        double s = 0.0;
        const zc scal = s_scal;
        const double up = s_up;
        for (int t = tid; t < nrows; t += kThreads) {
            const int r = r0 + C * t;
            zc p = A[(size_t)r * N + f];
            if (r == f) p.im = 0.0;
            fma_cx(p, scal, up * sq[t]);
            const zc v = r == f ? mk(1.0, 0.0) : scal * (up * sa[r - f]);
            sq[t] = p;
            X.p[r] = p;
            s += fma(v.re, p.re, v.im * p.im);
        }
        if (warp * 32 < nrows)  // the others have no row
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) X.s[rank * kWarps + warp] = s;
        if (warp == kWarps - 1) {
            zc part[kWarps];
#pragma unroll
            for (int w = 0; w < kWarps; ++w) part[w] = s_part[w][lane];
            zc t = scal * (up * pair_sum(part));
            if (r0 == f && on) t = t + conj(P[(size_t)f * kPW + lane]);
            X.gh[rank * kPW + lane] = t;
        }
        cl.sync();
        if (warp < 2) {
            // h = V^H v (lanes 0 ..), g = W^H v (lanes kNB ..), both by two warps
            zc part[kMaxCluster];  // all requested at once
#pragma unroll
            for (int c = 0; c < kMaxCluster; ++c) part[c] = c < C ? ldcg(X.gh + c * kPW + lane) : mk(0.0, 0.0);
            const zc pf = ldcg(X.p + f), pr = on ? P[(size_t)f * kPW + lane] : mk(0.0, 0.0);
            zc t = pair_sum(part);
            if (!on) t = mk(0.0, 0.0);
            const zc o = mk(__shfl_xor_sync(0xffffffffu, t.re, kNB), __shfl_xor_sync(0xffffffffu, t.im, kNB));
            const zc tau = s_tau;
            if (warp == 0) {
                // A_true v = p - V g - W h; its row f and row f of [W | V], columns before i
                zc dot = pr * o;
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) {
                    dot.re += __shfl_xor_sync(0xffffffffu, dot.re, d);
                    dot.im += __shfl_xor_sync(0xffffffffu, dot.im, d);
                }
                s_mul[lane] = o;
                s_row[lane] = mk(__shfl_xor_sync(0xffffffffu, pr.re, kNB), __shfl_xor_sync(0xffffffffu, pr.im, kNB));
                if (lane == 0) {
                    s_u1 = tau * (pf - dot);
                    if (rank == j % C) A[(size_t)j * N + j] = mk(s_d, s_beta);
                    if (rank == 0) A[(size_t)f * N + j] = tau;
                }
            } else {
                // v^H A_true v = v^H p - 2 Re sum conj(h) g; each pair is seen by two lanes
                double cr = fma(t.re, o.re, t.im * o.im);
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) cr += __shfl_xor_sync(0xffffffffu, cr, d);
                const double st = sum_published(X.s, C, lane) - cr;
                if (lane == 0) s_ca = -0.5 * fma(tau.re, tau.re, tau.im * tau.im) * st;
            }
        }
        __syncthreads();
        // own rows: u = tau A_true v + ca v, and the next column.  Four lanes a row
        // for the two products with its [V W], then one lane a row.
        const bool more = i + 1 < steps || f == N - 1;
        for (int t0 = tid >> 2; (t0 & ~7) < nrows; t0 += kThreads / 4) {  // whole warps
            const int r = r0 + C * min(t0, nrows - 1);
            const zc* Pr = P + (size_t)r * kPW;
            zc q1 = mk(0.0, 0.0), q2 = mk(0.0, 0.0);
            zc v[kNB / 4], w[kNB / 4], z1 = mk(0.0, 0.0), z2 = mk(0.0, 0.0);
#pragma unroll
            for (int kk = 0; kk < kNB / 4; ++kk) {  // all requested at once
                const int k = (tid & 3) + 4 * kk;
                v[kk] = k < i ? Pr[k] : mk(0.0, 0.0);
                w[kk] = k < i ? Pr[kNB + k] : mk(0.0, 0.0);
            }
#pragma unroll
            for (int kk = 0; kk < kNB / 4; ++kk) {
                const int k = (tid & 3) + 4 * kk;
                if (4 * kk >= i) break;
                fma_cx(q1, v[kk], s_mul[k]);
                fma_cx(z1, w[kk], s_mul[kNB + k]);
                fma_cx(q2, v[kk], conj(s_row[k]));
                fma_cx(z2, w[kk], conj(s_row[kNB + k]));
            }
            q1 = q1 + z1;
            q2 = q2 + z2;
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                q1.re += __shfl_xor_sync(0xffffffffu, q1.re, o);
                q1.im += __shfl_xor_sync(0xffffffffu, q1.im, o);
                q2.re += __shfl_xor_sync(0xffffffffu, q2.re, o);
                q2.im += __shfl_xor_sync(0xffffffffu, q2.im, o);
            }
            if ((tid & 3) == 0 && t0 < nrows) {
                sq[t0] = sq[t0] - q1;
                sx[t0] = q2;
            }
        }
        __syncthreads();
        const zc tau = s_tau, u1 = mk(s_u1.re + s_ca, s_u1.im);
        const double ca = s_ca;
        double nrm = 0.0;
        for (int t = tid; t < nrows; t += kThreads) {
            const int r = r0 + C * t;
            const zc v = r == f ? mk(1.0, 0.0) : scal * (up * sa[r - f]);
            zc u = tau * sq[t];
            u = mk(fma(ca, v.re, u.re), fma(ca, v.im, u.im));
            const zc vs = vscale * v, us = wscale * u;
            P[(size_t)r * kPW + i] = vs;
            P[(size_t)r * kPW + kNB + i] = us;
            Q[(size_t)r * kPW + i] = us;
            Q[(size_t)r * kPW + kNB + i] = vs;
            A[(size_t)j * N + r] = v;
            if (more) {
                // column f of A_true: a - [V W] conj(row f of [W V]) - v conj(u_f) - u
                const zc x = A[(size_t)r * N + f] - sx[t] - u - mulc(v, u1);
                if (r == f) {
                    s_d = x.re;
                    if (f == N - 1) A[(size_t)f * N + f] = mk(x.re, 0.0);
                } else {
                    X.a[r] = x;
                    if (r > f + 1) nrm += abs2(x);
                }
            }
        }
        if (warp * 32 < nrows)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
        if (lane == 0) X.norm[rank * kWarps + warp] = nrm;
        __syncthreads();
    }
    cl.sync();  // no CTA leaves while its cluster still reads what it published
}

// Lower triangle from the upper one, real diagonal; nexp (zeroed) gets each
// matrix's largest exponent field.
__global__ void __launch_bounds__(256) mirror64_kernel(int N, int64_t batch, zc* __restrict__ A, int* __restrict__ nexp) {
    __shared__ zc t[16][17];
    const int nt = (N + 15) / 16, x = threadIdx.x & 15, y = threadIdx.x >> 4;
    const int64_t per = (int64_t)nt * nt;
    for (int64_t w = blockIdx.x; w < batch * per; w += gridDim.x) {
        const int ti = (int)(w % per) / nt, tj = (int)(w % per) % nt;  // source tile (ti, tj), ti <= tj
        if (ti > tj) continue;
        zc* M = A + (w / per) * (int64_t)N * N;
        const int r = ti * 16 + y, c = tj * 16 + x;
        int ex = 0;
        if (r < N && c < N) {
            const zc v = M[(size_t)r * N + c];
            t[y][x] = v;
            ex = max((__double2hiint(v.re) >> 20) & 0x7ff, (__double2hiint(v.im) >> 20) & 0x7ff);
        }
        ex = __reduce_max_sync(0xffffffffu, ex);
        if ((threadIdx.x & 31) == 0) atomicMax(nexp + w / per, ex);
        __syncthreads();
        const int r2 = tj * 16 + y, c2 = ti * 16 + x;  // element (r2, c2) = conj of (c2, r2)
        if (r2 < N && c2 < N) {
            const zc v = conj(t[x][y]);
            if (r2 > c2)
                M[(size_t)r2 * N + c2] = v;
            else if (r2 == c2)
                M[(size_t)r2 * N + c2] = mk(v.re, 0.0);
        }
        __syncthreads();
    }
}

// Matrices out of range: all entries before the reduction, the diagonal (d, e) after it.
__global__ void __launch_bounds__(256) rescale64_kernel(int N, int64_t batch, zc* __restrict__ A,
                                                        const int* __restrict__ nexp, bool back) {
    for (int64_t b = blockIdx.y; b < batch; b += gridDim.y) {
        const int sh = reduced_exp(nexp[b]) - nexp[b];
        if (sh == 0) continue;
        zc* M = A + b * (int64_t)N * N;
        const int64_t n = back ? N : (int64_t)N * N, step = back ? N + 1 : 1;
        for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
            const zc x = M[i * step];
            M[i * step] = mk(scalbn(x.re, back ? -sh : sh), scalbn(x.im, back ? -sh : sh));
        }
    }
}

// ---------------------------------------------------- back-transformation --
constexpr int kWY = 64;  // reflectors of a block

// Reflectors j0 .. j0 + w - 1 of every matrix as rows of length m = N - 1 - j0 without
// their leading ones (reflector jj has its at jj; zeros up to there), w = kWY rows held.
//
// The ones, and T's diagonal, are added apart in FP64 (wy_preset_kernel, wy_scale_kernel,
// wy_ones_kernel): a digit product's error is relative to the largest entry of a line, and
// beside them the rest is some ten times smaller (H U - U E of 128 bands 1.8e-13 in the
// Frobenius norm with them in the products, 1.8e-14 by single reflectors).
__global__ void __launch_bounds__(256) wy_rows_kernel(int N, int64_t batch, int j0, int w, const zc* __restrict__ A,
                                                      zc* __restrict__ Y) {
    const int m = N - 1 - j0;
    const int64_t total = batch * w;
    for (int64_t row = blockIdx.x; row < total; row += gridDim.x) {
        const int64_t b = row / w;
        const int jj = (int)(row % w);
        const zc* src = A + (b * N + j0 + jj) * (int64_t)N + j0 + 1;
        zc* dst = Y + (b * kWY + jj) * (int64_t)m;
        for (int r = threadIdx.x; r < m; r += blockDim.x) dst[r] = r > jj ? src[r] : mk(0.0, 0.0);
    }
}

// What the leading ones add to G = Y^H Y above the diagonal (conj(Y(i, j))) and to Y^H U
// (rows of U); ldu, sU: of U's rows and matrices.
__global__ void __launch_bounds__(256) wy_preset_kernel(int64_t batch, int w, int m, int ncol,
                                                        const zc* __restrict__ Y, const zc* __restrict__ U,
                                                        int64_t ldu, int64_t sU, zc* __restrict__ G,
                                                        zc* __restrict__ X) {
    const int64_t total = batch * w;
    for (int64_t row = blockIdx.x; row < total; row += gridDim.x) {
        const int64_t b = row / w;
        const int i = (int)(row % w);
        const zc* y = Y + (b * kWY + i) * (int64_t)m;
        zc* g = G + (b * kWY + i) * (int64_t)kWY;
        for (int j = threadIdx.x; j < w; j += blockDim.x) g[j] = j > i ? conj(y[j]) : mk(0.0, 0.0);
        const zc* u = U + b * sU + i * ldu;
        zc* x = X + (b * kWY + i) * (int64_t)ncol;
        for (int c = threadIdx.x; c < ncol; c += blockDim.x) x[c] = u[c];
    }
}
// X2 = diag(tau) X1, and U's rows of the leading ones -= X2 (ones).
__global__ void __launch_bounds__(256) wy_scale_kernel(int N, int64_t batch, int j0, int w, int ncol,
                                                       const zc* __restrict__ A, const zc* __restrict__ X1,
                                                       zc* __restrict__ X2) {
    const int64_t total = batch * w;
    for (int64_t row = blockIdx.x; row < total; row += gridDim.x) {
        const int64_t b = row / w;
        const int i = (int)(row % w);
        const zc tau = A[(b * N + j0 + i + 1) * (int64_t)N + j0 + i];
        const int64_t at = (b * kWY + i) * (int64_t)ncol;
        for (int c = threadIdx.x; c < ncol; c += blockDim.x) X2[at + c] = tau * X1[at + c];
    }
}
__global__ void __launch_bounds__(256) wy_ones_kernel(int64_t batch, int w, int ncol, const zc* __restrict__ X2,
                                                      zc* __restrict__ U, int64_t ldu, int64_t sU) {
    const int64_t total = batch * w;
    for (int64_t row = blockIdx.x; row < total; row += gridDim.x) {
        const int64_t b = row / w;
        const int i = (int)(row % w);
        zc* u = U + b * sU + i * ldu;
        const zc* x = X2 + (b * kWY + i) * (int64_t)ncol;
        for (int c = threadIdx.x; c < ncol; c += blockDim.x) u[c] = u[c] - x[c];
    }
}

// T of H_0 ... H_{w-1} = I - Y T Y^H from G = Y^H Y and tau (columns left to right:
// T(0:j, j) = -tau_j T(0:j, 0:j) G(0:j, j)); T without its diagonal tau over G in place,
// one CTA per matrix, four lanes per row.
__global__ void __launch_bounds__(4 * kWY) wy_t_kernel(int N, int64_t batch, int j0, int w, const zc* __restrict__ A,
                                                       zc* __restrict__ G) {
    __shared__ zc T[kWY * (kWY + 1) / 2], g[kWY], s_tau[kWY];  // T by packed columns
    const int i = threadIdx.x >> 2, q = threadIdx.x & 3;
    for (int64_t b = blockIdx.x; b < batch; b += gridDim.x) {
        zc* Gb = G + b * kWY * kWY;
        if (threadIdx.x < w) {
            const int j = j0 + threadIdx.x;
            s_tau[threadIdx.x] = A[(b * N + j + 1) * (int64_t)N + j];
        }
        __syncthreads();
        for (int j = 0; j < w; ++j) {
            if (threadIdx.x < j) g[threadIdx.x] = Gb[threadIdx.x * kWY + j];
            __syncthreads();
            zc acc = mk(0.0, 0.0);
            if (i < j)
                for (int l = i + q; l < j; l += 4) fma_cx(acc, T[l * (l + 1) / 2 + i], g[l]);
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                acc.re += __shfl_xor_sync(0xffffffffu, acc.re, o);
                acc.im += __shfl_xor_sync(0xffffffffu, acc.im, o);
            }
            const zc tau = s_tau[j];
            if (q == 0 && i < j) T[j * (j + 1) / 2 + i] = mk(-tau.re, -tau.im) * acc;
            if (threadIdx.x == 0) T[j * (j + 1) / 2 + j] = tau;
            __syncthreads();
        }
        for (int e = threadIdx.x; e < w * kWY; e += blockDim.x) {
            const int r = e / kWY, c = e - r * kWY;
            Gb[e] = (c < w && r < c) ? T[c * (c + 1) / 2 + r] : mk(0.0, 0.0);
        }
        __syncthreads();
    }
}

}  // namespace

// U <- H_0 ... H_{N-2} U (columns first .. first + ncol - 1) in blocks of kWY reflectors, last block first:
// U -= Y (T (Y^H U)), all products on the tensor cores.
int bt64_wy(cudaStream_t st, int N, int64_t batch, const zc* A, zc* U, int* status_d, int first, int ncol) {
    int nsm = 0, dev = 0;
    TBG_CUDA(cudaGetDevice(&dev));
    TBG_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) & ~size_t(255);
        return o;
    };
    const size_t nb = (size_t)batch;
    const size_t oY = take(sizeof(zc) * nb * kWY * (N - 1)), oG = take(sizeof(zc) * nb * kWY * kWY);
    const size_t o1 = take(sizeof(zc) * nb * kWY * ncol), o2 = take(sizeof(zc) * nb * kWY * ncol);
    const size_t oE = take(sizeof(int) * nb * (3 * kWY + 4 * N));
    unsigned char* buf = nullptr;
    TBG_CUDA(cudaMallocAsync(&buf, off, st));
    zc *Y = reinterpret_cast<zc*>(buf + oY), *G = reinterpret_cast<zc*>(buf + oG);
    zc *X1 = reinterpret_cast<zc*>(buf + o1), *X2 = reinterpret_cast<zc*>(buf + o2);
    int *ey = reinterpret_cast<int*>(buf + oE), *et = ey + nb * kWY, *ec = et + nb * kWY;
    int *eu = ec + nb * N, *e1 = eu + nb * N, *e2 = e1 + nb * N;
    int rc = TBG_OK;
    const int last = (N - 2) / kWY * kWY;
    for (int j0 = last; j0 >= 0 && !rc; j0 -= kWY) {
        const int w = std::min(kWY, N - 1 - j0), m = N - 1 - j0;
        const int64_t sY = (int64_t)kWY * m, sG = kWY * kWY, sX = (int64_t)kWY * ncol, sU = (int64_t)N * N;
        zc* Ut = U + (int64_t)(j0 + 1) * N + first;
        wy_rows_kernel<<<(unsigned)std::min<int64_t>(batch * w, nsm * 64), 256, 0, st>>>(N, batch, j0, w, A, Y);
        TBG_LAUNCHED("wy_rows_kernel");
        const unsigned rows = (unsigned)std::min<int64_t>(batch * w, nsm * 64);
        wy_preset_kernel<<<rows, 256, 0, st>>>(batch, w, m, ncol, Y, Ut, N, sU, G, X1);
        TBG_LAUNCHED("wy_preset_kernel");
        if ((rc = oz64_row_exps(st, batch, w, m, Y, m, sY, ey))) break;
        const Oz64Operand yh{Y, m, 1, sY, 1, ey};
        if ((rc = oz64_gemm(st, batch, w, w, m, yh, {Y, m, 1, sY, 0, ey}, G, kWY, sG, 1, status_d))) break;
        wy_t_kernel<<<(unsigned)std::min<int64_t>(batch, nsm * 64), 4 * kWY, 0, st>>>(N, batch, j0, w, A, G);
        TBG_LAUNCHED("wy_t_kernel");
        if ((rc = oz64_row_exps(st, batch, w, w, G, kWY, sG, et)) || (rc = oz64_col_exps(st, batch, m, ncol, Ut, N, sU, eu)) ||
            (rc = oz64_col_exps(st, batch, w, m, Y, m, sY, ec)))
            break;
        if ((rc = oz64_gemm(st, batch, w, ncol, m, yh, {Ut, 1, N, sU, 0, eu}, X1, ncol, sX, 1, status_d))) break;
        wy_scale_kernel<<<rows, 256, 0, st>>>(N, batch, j0, w, ncol, A, X1, X2);
        TBG_LAUNCHED("wy_scale_kernel");
        if ((rc = oz64_col_exps(st, batch, w, ncol, X1, ncol, sX, e1))) break;
        if ((rc = oz64_gemm(st, batch, w, ncol, w, {G, kWY, 1, sG, 0, et}, {X1, 1, ncol, sX, 0, e1}, X2, ncol, sX, 1,
                            status_d)))
            break;
        wy_ones_kernel<<<rows, 256, 0, st>>>(batch, w, ncol, X2, Ut, N, sU);
        TBG_LAUNCHED("wy_ones_kernel");
        if ((rc = oz64_col_exps(st, batch, w, ncol, X2, ncol, sX, e2))) break;
        rc = oz64_gemm(st, batch, m, ncol, w, {Y, 1, m, sY, 0, ec}, {X2, 1, ncol, sX, 0, e2}, Ut, N, sU, -1, status_d);
    }
    cudaFreeAsync(buf, st);
    return rc;
}

// Reduction of batch N x N matrices (upper triangles read); A then holds what
// tri64 and the back-transformation take.
int hetrd64_big(cudaStream_t st, int N, int64_t batch, zc* A, int* status_d) {
    int dev = 0, nsm = 0;
    TBG_CUDA(cudaGetDevice(&dev));
    TBG_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    TBG_CUDA(cudaFuncSetAttribute(panel64_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    // the largest cluster with which the whole batch runs at once; one CTA per
    // matrix when it cannot
    int C = (int)std::min<int64_t>(std::min(kMaxCluster, std::max(1, N / 32)), std::max<int64_t>(1, nsm / batch));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cfg.blockDim = dim3(kThreads);
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    for (;; --C) {
        const size_t smem = panel64_smem_bytes(N, C);
        if (int r = allow_smem(panel64_kernel, smem)) return r;
        cfg.dynamicSmemBytes = smem;
        cfg.gridDim = dim3((unsigned)(batch * C));
        at[0].val.clusterDim.x = C;
        int fit = 0;
        if (C == 1) break;
        if (cudaOccupancyMaxActiveClusters(&fit, panel64_kernel, &cfg) != cudaSuccess) cudaGetLastError();
        if (fit >= batch) break;
    }
    const int64_t xb = (int64_t)((exchange_bytes(N, C) + 255) & ~size_t(255));
    const size_t pb = sizeof(zc) * (size_t)batch * N * kPW;
    unsigned char* buf = nullptr;
    TBG_CUDA(cudaMallocAsync(&buf, 2 * pb + xb * batch + sizeof(int) * batch * (N + 1), st));
    zc* P = reinterpret_cast<zc*>(buf);
    zc* Q = P + (size_t)batch * N * kPW;
    unsigned char* X = buf + 2 * pb;
    int* ex = reinterpret_cast<int*>(X + xb * batch);
    int* nexp = ex + batch * N;
    int rc = TBG_OK;
    TBG_CUDA(cudaMemsetAsync(nexp, 0, sizeof(int) * batch, st));
    mirror64_kernel<<<(unsigned)std::min<int64_t>(batch * ((N + 15) / 16) * ((N + 15) / 16), nsm * 64), 256, 0, st>>>(
        N, batch, A, nexp);
    count_launch();
    const dim3 rs(std::min(64, (N * N + 255) / 256), (unsigned)std::min<int64_t>(batch, 65535));
    rescale64_kernel<<<rs, 256, 0, st>>>(N, batch, A, nexp, false);
    count_launch();
    cudaError_t e = cudaGetLastError();
    for (int j0 = 0; j0 < N - 1 && e == cudaSuccess && !rc; j0 += kNB) {
        const int steps = std::min(kNB, N - 1 - j0);
        e = cudaLaunchKernelEx(&cfg, panel64_kernel, N, j0, steps, A, P, Q, nexp, X, xb);
        count_launch();
        const int t = j0 + steps, m = N - t;
        if (e != cudaSuccess || t >= N - 1) break;
        // trailing block -= [V W][W V]^H
        const zc *Pt = P + (size_t)t * kPW, *Qt = Q + (size_t)t * kPW;
        const int64_t sP = (int64_t)N * kPW;
        rc = oz64_row_exps(st, batch, m, kPW, Pt, kPW, sP, ex);
        if (!rc)
            rc = oz64_gemm(st, batch, m, m, kPW, {Pt, kPW, 1, sP, 0, ex}, {Qt, kPW, 1, sP, 1, ex},
                           A + (size_t)t * N + t, N, (int64_t)N * N, -1, status_d);
    }
    if (e == cudaSuccess && !rc) {
        rescale64_kernel<<<dim3(1, rs.y), 256, 0, st>>>(N, batch, A, nexp, true);
        count_launch();
        e = cudaGetLastError();
    }
    if (e != cudaSuccess && !rc) rc = cuda_error(e, "panel64_kernel");
    cudaFreeAsync(buf, st);
    return rc;
}

}  // namespace tbg
