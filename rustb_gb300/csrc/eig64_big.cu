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
// 12 matrices of 512 bands (eigenvalues) 176 -> 17.7 ms, against one CTA per matrix.

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

// Published by the CTAs of a matrix to each other, per matrix.
struct Exchange {
    zc* a;         // (N) current column below the diagonal
    zc* p;         // (N) A v
    zc* gh;        // (C, kPW) partial [V W]^H v
    double* norm;  // (C, kWarps) partial |a|^2 without the first entry
    double* s;     // (C) partial v^H A v
};
__host__ __device__ inline size_t exchange_bytes(int N, int C) {
    return sizeof(zc) * (2 * (size_t)N + (size_t)C * kPW) + sizeof(double) * ((size_t)C * kWarps + C + (C & 1));
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

// Sums over the warp of R complex values per lane (R = 4 or 8): lane l ends with
// the sum of value l mod R, in R - 1 + (5 - log2 R) additions per component
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
    const int half = (nexp[b] - 1022) / 2;
    const double up = scalbn(1.0, half), down = scalbn(1.0, -half);
    const Exchange X = exchange_of(xin + b * xbytes, N, C);
    extern __shared__ __align__(16) unsigned char smem_p[];
    zc* sa = reinterpret_cast<zc*>(smem_p);  // (N) column below the diagonal
    zc* sq = sa + N;                         // (own rows) A a, then p
    __shared__ zc s_part[kWarps][kPW];       // partial [V W]^H a per warp
    __shared__ zc s_mul[kPW], s_row[kPW];    // coefficients of V, W; the next row of [W V]
    __shared__ zc s_scal, s_tau, s_u1;
    __shared__ double s_beta, s_ca, s_d, s_sw[kWarps];
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
            double xn = 0.0;
            for (int t = lane; t < C * kWarps; t += 32) xn += __ldcg(X.norm + t);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) xn += __shfl_xor_sync(0xffffffffu, xn, o);
            if (lane == 0) {
                const zc alpha = sa[0];
                zc tau, scal;
                double beta;
                reflector_scalars64(alpha, xn, tau, scal, beta);
                s_tau = tau;
                s_scal = scal;
                s_beta = beta;
            }
        }
        // q = A a without the first column, partial [V W]^H a without the first row;
        // four own rows at a time
        zc gh = mk(0.0, 0.0);
        const bool on = (lane & (kNB - 1)) < i;
        for (;;) {
            int g = 0;
            if (lane == 0) g = atomicAdd(&s_next, 4);
            g = __shfl_sync(0xffffffffu, g, 0);
            if (g >= nrows) break;
            zc acc[4] = {};
            const zc* row[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) row[k] = A + (size_t)(r0 + C * min(g + k, nrows - 1)) * N + f;
#pragma unroll 2
            for (int c = lane; c < N - f; c += 32) {
                const zc x = c > 0 ? sa[c] : mk(0.0, 0.0);
#pragma unroll
                for (int k = 0; k < 4; ++k) fma_cx(acc[k], row[k][c], x);
            }
            if (on) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int r = r0 + C * (g + k);
                    if (g + k < nrows && r > f) fma_cjx(gh, P[(size_t)r * kPW + lane], sa[r - f]);
                }
            }
            const zc q = warp_sums<4>(acc, lane);
            if (lane < 4 && g + lane < nrows) sq[g + lane] = q;
        }
        s_part[warp][lane] = gh;
        __syncthreads();
        // p = A v, v = (1, scal a); publish p, [V W]^H v and v^H p of the own rows
        double s = 0.0;
        const zc scal = s_scal;
        for (int t = tid; t < nrows; t += kThreads) {
            const int r = r0 + C * t;
            zc p = A[(size_t)r * N + f];
            if (r == f) p.im = 0.0;
            fma_cx(p, scal, sq[t]);
            const zc v = r == f ? mk(1.0, 0.0) : scal * sa[r - f];
            sq[t] = p;
            X.p[r] = p;
            s += fma(v.re, p.re, v.im * p.im);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) s_sw[warp] = s;
        if (warp == kWarps - 1) {
            zc t = mk(0.0, 0.0);
#pragma unroll
            for (int w = 0; w < kWarps; ++w) t = t + s_part[w][lane];
            t = scal * t;
            if (r0 == f && on) t = t + conj(P[(size_t)f * kPW + lane]);
            X.gh[rank * kPW + lane] = t;
        }
        __syncthreads();
        if (tid == 0) {
            double t = 0.0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) t += s_sw[w];
            X.s[rank] = t;
        }
        cl.sync();
        if (warp == 0) {
            // h = V^H v (lanes 0 ..), g = W^H v (lanes kNB ..)
            zc t = mk(0.0, 0.0);
            double st = 0.0;
            for (int c = 0; c < C; ++c) {
                t = t + ldcg(X.gh + c * kPW + lane);
                st += __ldcg(X.s + c);
            }
            if (!on) t = mk(0.0, 0.0);
            const zc o = mk(__shfl_xor_sync(0xffffffffu, t.re, kNB), __shfl_xor_sync(0xffffffffu, t.im, kNB));
            // v^H A_true v = v^H p - 2 Re sum conj(h) g; each pair is seen by two lanes
            double cr = fma(t.re, o.re, t.im * o.im);
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) cr += __shfl_xor_sync(0xffffffffu, cr, d);
            st -= cr;
            const zc tau = s_tau;
            const double ca = -0.5 * fma(tau.re, tau.re, tau.im * tau.im) * st;
            // A_true v = p - V g - W h
            const zc pr = on ? P[(size_t)f * kPW + lane] : mk(0.0, 0.0);
            zc d1[4] = {pr * o, mk(0.0, 0.0), mk(0.0, 0.0), mk(0.0, 0.0)};
            const zc dot0 = warp_sums<4>(d1, lane);
            const zc dot = mk(__shfl_sync(0xffffffffu, dot0.re, 0), __shfl_sync(0xffffffffu, dot0.im, 0));
            zc u1 = tau * (ldcg(X.p + f) - dot);
            u1.re += ca;
            s_mul[lane] = o;
            const zc sw = mk(__shfl_xor_sync(0xffffffffu, pr.re, kNB), __shfl_xor_sync(0xffffffffu, pr.im, kNB));
            s_row[lane] = sw;  // row f of [W | V], columns before i
            if (lane == 0) {
                s_ca = ca;
                s_u1 = u1;
                if (rank == j % C) A[(size_t)j * N + j] = mk(s_d, s_beta);
                if (rank == 0) A[(size_t)f * N + j] = tau;
            }
        }
        __syncthreads();
        // own rows: u = tau A_true v + ca v, and the next column
        const zc tau = s_tau, mul = s_mul[lane], nrow = conj(s_row[lane]), u1 = s_u1;
        const double ca = s_ca;
        const bool more = i + 1 < steps || f == N - 1;
        double nrm = 0.0;
        for (int g = 4 * warp; g < nrows; g += 4 * kWarps) {
            zc acc[8];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int r = r0 + C * min(g + k, nrows - 1);
                const zc x = on ? P[(size_t)r * kPW + lane] : mk(0.0, 0.0);
                acc[k] = x * mul;
                acc[4 + k] = x * nrow;
            }
            const zc q = warp_sums<8>(acc, lane);
            const zc q2 = mk(__shfl_down_sync(0xffffffffu, q.re, 4), __shfl_down_sync(0xffffffffu, q.im, 4));
            if (lane < 4 && g + lane < nrows) {
                const int r = r0 + C * (g + lane);
                const zc v = r == f ? mk(1.0, 0.0) : scal * sa[r - f];
                zc u = tau * (sq[g + lane] - q);
                u = mk(fma(ca, v.re, u.re), fma(ca, v.im, u.im));
                const zc vs = up * v, us = down * u;
                P[(size_t)r * kPW + i] = vs;
                P[(size_t)r * kPW + kNB + i] = us;
                Q[(size_t)r * kPW + i] = us;
                Q[(size_t)r * kPW + kNB + i] = vs;
                A[(size_t)j * N + r] = v;
                if (more) {
                    // column f of A_true: a - [V W] conj(row f of [W V]) - v conj(u_f) - u
                    zc x = A[(size_t)r * N + f] - q2 - u;
                    x = x - mulc(v, u1);
                    if (r == f) {
                        s_d = x.re;
                        if (f == N - 1) A[(size_t)f * N + f] = mk(x.re, 0.0);
                    } else {
                        X.a[r] = x;
                        if (r > f + 1) nrm += abs2(x);
                    }
                }
            }
        }
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

// ---------------------------------------------------- back-transformation --
constexpr int kWY = 64;  // reflectors of a block

// Reflectors j0 .. j0 + w - 1 of every matrix as rows of length m = N - 1 - j0
// (zeros before the leading one), w = kWY rows held.
__global__ void __launch_bounds__(256) wy_rows_kernel(int N, int64_t batch, int j0, int w, const zc* __restrict__ A,
                                                      zc* __restrict__ Y) {
    const int m = N - 1 - j0;
    const int64_t total = batch * w;
    for (int64_t row = blockIdx.x; row < total; row += gridDim.x) {
        const int64_t b = row / w;
        const int jj = (int)(row % w);
        const zc* src = A + (b * N + j0 + jj) * (int64_t)N + j0 + 1;
        zc* dst = Y + (b * kWY + jj) * (int64_t)m;
        for (int r = threadIdx.x; r < m; r += blockDim.x) dst[r] = r >= jj ? src[r] : mk(0.0, 0.0);
    }
}

// T of H_0 ... H_{w-1} = I - Y T Y^H from G = Y^H Y and tau (columns left to right:
// T(0:j, j) = -tau_j T(0:j, 0:j) G(0:j, j)); T over G in place, one CTA per matrix,
// four lanes per row.
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
            Gb[e] = (c < w && r <= c) ? T[c * (c + 1) / 2 + r] : mk(0.0, 0.0);
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
        if ((rc = oz64_row_exps(st, batch, w, m, Y, m, sY, ey))) break;
        const Oz64Operand yh{Y, m, 1, sY, 1, ey};
        if ((rc = oz64_gemm(st, batch, w, w, m, yh, {Y, m, 1, sY, 0, ey}, G, kWY, sG, 0, status_d))) break;
        wy_t_kernel<<<(unsigned)std::min<int64_t>(batch, nsm * 64), 4 * kWY, 0, st>>>(N, batch, j0, w, A, G);
        TBG_LAUNCHED("wy_t_kernel");
        if ((rc = oz64_row_exps(st, batch, w, w, G, kWY, sG, et)) || (rc = oz64_col_exps(st, batch, m, ncol, Ut, N, sU, eu)) ||
            (rc = oz64_col_exps(st, batch, w, m, Y, m, sY, ec)))
            break;
        if ((rc = oz64_gemm(st, batch, w, ncol, m, yh, {Ut, 1, N, sU, 0, eu}, X1, ncol, sX, 0, status_d))) break;
        if ((rc = oz64_col_exps(st, batch, w, ncol, X1, ncol, sX, e1))) break;
        if ((rc = oz64_gemm(st, batch, w, ncol, w, {G, kWY, 1, sG, 0, et}, {X1, 1, ncol, sX, 0, e1}, X2, ncol, sX, 0,
                            status_d)))
            break;
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
    auto smem_of = [&](int c) { return sizeof(zc) * ((size_t)N + (N + c - 1) / c + 1); };
    for (;; --C) {
        const size_t smem = smem_of(C);
        TBG_CUDA(cudaFuncSetAttribute(panel64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
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
    if (e != cudaSuccess && !rc) rc = cuda_error(e, "panel64_kernel");
    cudaFreeAsync(buf, st);
    return rc;
}

}  // namespace tbg
