// Bloch Fourier sum H(k) and direction-projected velocities, direct form.
//
// Replaces the zaxpy loops of Model::gen_ham (src/model_physics.rs:92-96) and
// Model::gen_v_projected (src/velocity.rs:538-541, 581-613):
//
//   H_lat(k)[e] = sum_R u(k,R) ham[R][e],                u = e^{2 pi i k.R}
//   V_p(k)[e]   = i sum_R (w_p . R_cart) u(k,R) ham[R][e]
//   Atom gauge:   H[m,n] = conj(phi_m) H_lat[m,n] phi_n,       phi = e^{2 pi i k.tau}
//                 V_p[m,n] = (V_p[m,n] + i (w_p.tau_n - w_p.tau_m) H_lat[m,n]) conj(phi_m) phi_n
//
// As a contraction this is phase[nk x nR] . hop[nR x N^2] for H and the same
// with the phase column scaled by w_p.R_cart for each V_p.  The kernel stages
// tiles of the hop table and of the phases in shared memory and keeps one
// complex accumulator per output in registers; the gauge / tau epilogue is
// fused.  FP64 throughout (plain path).

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cmath>
#include <mutex>
#include <vector>

#include "tbgpu_internal.cuh"

namespace tbg {
namespace {

constexpr double kTwoPi = 6.283185307179586476925286766559;

// u(k,R) = exp(2 pi i k.R) for R rows [0, nR); phi(k,s) = exp(2 pi i k.tau_s).
__global__ void phases_kernel(int64_t nk, int dim, const double* __restrict__ k, int nR,
                              const int* __restrict__ hamR, int nsta, const double* __restrict__ tau,
                              zc* __restrict__ ph, zc* __restrict__ orbph) {
    const int64_t total = nk * (int64_t)(nR + nsta);
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t kk = idx / (nR + nsta);
        const int j = (int)(idx % (nR + nsta));
        const double* kv = k + kk * dim;
        double s = 0.0;
        if (j < nR) {
            const int* r = hamR + 3 * j;
            // same operation order as the reference: r0*k0 + r1*k1 + r2*k2
            s = (double)r[0] * kv[0];
            if (dim > 1) s += (double)r[1] * kv[1];
            if (dim > 2) s += (double)r[2] * kv[2];
            double sn, cs;
            sincos(kTwoPi * s, &sn, &cs);
            ph[kk * nR + j] = mk(cs, sn);
        } else {
            const double* t = tau + 3 * (j - nR);
            s = t[0] * kv[0];
            if (dim > 1) s += t[1] * kv[1];
            if (dim > 2) s += t[2] * kv[2];
            double sn, cs;
            sincos(kTwoPi * s, &sn, &cs);
            orbph[kk * nsta + (j - nR)] = mk(cs, sn);
        }
    }
}

constexpr int TK = 32;   // k-points per tile
constexpr int TE = 64;   // matrix elements per tile
constexpr int RC = 8;    // R rows per shared-memory stage

// A (nk, N^2) = sum_R ph(k, R) hop(R): the position-matrix sums of few k-points.
__global__ void __launch_bounds__(256) fourier_gemm_kernel(int64_t nk, int nR, int ldph, int N,
                                                           const zc* __restrict__ ph, const zc* __restrict__ hop,
                                                           zc* __restrict__ H) {
    __shared__ zc s_hop[RC][TE];
    __shared__ zc s_ph[RC][TK];
    const int tid = threadIdx.x;
    const int te = tid & 15;  // element lane: e = te + 16 j
    const int tk = tid >> 4;  // k lane: k = tk + 16 i
    const int64_t NN = (int64_t)N * N;
    const int64_t e0 = (int64_t)blockIdx.x * TE;
    const int64_t k0 = (int64_t)blockIdx.y * TK;

    zc acc[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = mk(0.0, 0.0);

    for (int r0 = 0; r0 < nR; r0 += RC) {
        for (int idx = tid; idx < RC * TE; idx += 256) {
            const int r = idx / TE, e = idx % TE;
            zc h = mk(0.0, 0.0);
            if (r0 + r < nR && e0 + e < NN) h = hop[(int64_t)(r0 + r) * NN + e0 + e];
            s_hop[r][e] = h;
        }
        {
            const int r = tid / TK, kk = tid % TK;  // 256 == RC*TK
            zc u = mk(0.0, 0.0);
            if (r0 + r < nR && k0 + kk < nk) u = ph[(k0 + kk) * ldph + r0 + r];
            s_ph[r][kk] = u;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < RC; ++r) {
            zc h[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) h[j] = s_hop[r][te + 16 * j];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const zc u = s_ph[r][tk + 16 * i];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const zc t = u * h[j];
                    acc[i][j].re += t.re;
                    acc[i][j].im += t.im;
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int64_t kk = k0 + tk + 16 * i;
        if (kk >= nk) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t e = e0 + te + 16 * j;
            if (e < NN) H[kk * NN + e] = acc[i][j];
        }
    }
}

// coef[p][r] = w_p . R_cart[r];  taup[p][s] = w_p . tau_cart[s]
__global__ void proj_coef_kernel(int nproj, int dim, const double* __restrict__ dirs, int nR,
                                 const double* __restrict__ Rcart, int nsta, const double* __restrict__ taucart,
                                 double* __restrict__ coef, double* __restrict__ taup) {
    const int total = nproj * (nR + nsta);
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
        const int p = idx / (nR + nsta), j = idx % (nR + nsta);
        const double* w = dirs + p * dim;
        if (j < nR) {
            const double* r = Rcart + 3 * j;
            double s = w[0] * r[0];
            if (dim > 1) s += w[1] * r[1];
            if (dim > 2) s += w[2] * r[2];
            coef[p * nR + j] = s;
        } else {
            const double* t = taucart + 3 * (j - nR);
            double s = w[0] * t[0];
            if (dim > 1) s += w[1] * t[1];
            if (dim > 2) s += w[2] * t[2];
            taup[p * nsta + (j - nR)] = s;
        }
    }
}

int launch_gemm(cudaStream_t st, int64_t nk, int nR, int ldph, int N, const zc* ph, const zc* hop, zc* H) {
    const int64_t NN = (int64_t)N * N;
    KTimer kt(st, "fourier_gemm_kernel", 8.0 * nR * (double)NN * nk);
    for (int64_t kb = 0; kb < nk; kb += (int64_t)TK * 65535) {
        const int64_t nkb = std::min<int64_t>(nk - kb, (int64_t)TK * 65535);
        dim3 grid((unsigned)((NN + TE - 1) / TE), (unsigned)((nkb + TK - 1) / TK));
        fourier_gemm_kernel<<<grid, 256, 0, st>>>(nkb, nR, ldph, N, ph + kb * ldph, hop, H + kb * NN);
        TBG_LAUNCHED("fourier_gemm_kernel");
    }
    return TBG_OK;
}

// Fourier sums from the +-R paired table (FP64; rows 2q, 2q + 1 of T are A_q,
// B_q, pair 0 is R = 0 with A_0 = t(0), B_0 = 0): with (c, s) = (cos, sin) of
// 2 pi k . R_q,
//   H += c A_q + s B_q,   V_p += c_p(R_q) (c B_q - s A_q)   (c_p(R_0) = 0),
// 8 + 2 NP FMAs per pair and element for two R (10 + 2 NP per R unpaired).
//
// The form for little work (large sums go to the tensor cores), where latency and
// launches count: one launch, no scratch.  A block has 32 consecutive (k, element)
// outputs, one per lane, and deals the pairs to G warps; phases and projection
// coefficients of kPairChunk pairs at a time are made in shared memory.  One k-point
// of 18 bands, 125 R and three projections 490 -> 22 us, 10201 k-points of two
// bands 186 -> 32 us, against 32 k x 64 element tiles (mostly padding there)
// behind three launches for the phases.
constexpr int kPairChunk = 64;
template <int NP>
__global__ void __launch_bounds__(256) fourier_few_kernel(
    int64_t nk, int dim, const double* __restrict__ k, int np, const int* __restrict__ pair,
    const int* __restrict__ hamR, const double* __restrict__ Rcart, const zc* __restrict__ T, int N,
    const double* __restrict__ tau, const double* __restrict__ taucart, const double* __restrict__ dirs, int gauge,
    zc* __restrict__ H, int64_t ldH, zc* __restrict__ V, int64_t ldV) {
    constexpr int NV = NP > 0 ? NP : 1;
    extern __shared__ __align__(16) unsigned char few_smem[];
    __shared__ double s_coef[NV][kPairChunk];
    const int lane = threadIdx.x, g = threadIdx.y, G = blockDim.y, tid = g * 32 + lane;
    const int64_t NN = (int64_t)N * N, total = nk * NN, first = blockIdx.x * (int64_t)32;
    const int64_t kf = first / NN, idx = min(first + lane, total - 1), kk = idx / NN;
    const int nks = (int)(min(first + 31, total - 1) / NN - kf) + 1;
    const int64_t e = idx - kk * NN;
    zc* s_cs = reinterpret_cast<zc*>(few_smem);       // (nks, kPairChunk)
    zc* s_red = s_cs;                                 // then (G, 1 + NP, 32)
    const int Kc = np + 1;
    zc accH = mk(0.0, 0.0), accV[NV];
#pragma unroll
    for (int p = 0; p < NV; ++p) accV[p] = mk(0.0, 0.0);
    for (int q0 = 0; q0 < Kc; q0 += kPairChunk) {
        const int nq = min(kPairChunk, Kc - q0);
        __syncthreads();
        for (int t = tid; t < nks * nq; t += 32 * G) {
            const int kl = t / nq, q = t - kl * nq;
            zc u = mk(1.0, 0.0);
            if (q0 + q > 0) {
                const int* r = hamR + 3 * pair[q0 + q - 1];
                const double* kv = k + (kf + kl) * dim;
                double s = (double)r[0] * kv[0];
                if (dim > 1) s += (double)r[1] * kv[1];
                if (dim > 2) s += (double)r[2] * kv[2];
                sincospi(2.0 * s, &u.im, &u.re);
            }
            s_cs[kl * kPairChunk + q] = u;
        }
        if (NP > 0)
            for (int t = tid; t < NP * nq; t += 32 * G) {
                const int p = t / nq, q = t - p * nq;
                double c = 0.0;
                if (q0 + q > 0) {
                    const double *r = Rcart + 3 * pair[q0 + q - 1], *w = dirs + p * dim;
                    c = w[0] * r[0];
                    if (dim > 1) c += w[1] * r[1];
                    if (dim > 2) c += w[2] * r[2];
                }
                s_coef[p][q] = c;
            }
        __syncthreads();
        const zc* cs = s_cs + (kk - kf) * kPairChunk;
        const zc* t0 = T + (int64_t)(2 * q0) * NN + e;
#pragma unroll 4
        for (int q = g; q < nq; q += G) {
            const zc a = t0[(2 * q) * NN], b = t0[(2 * q + 1) * NN], u = cs[q];  // (cos, sin)
            accH.re = fma(u.re, a.re, accH.re);
            accH.re = fma(u.im, b.re, accH.re);
            accH.im = fma(u.re, a.im, accH.im);
            accH.im = fma(u.im, b.im, accH.im);
            if (NP > 0) {
                const double wr = fma(u.re, b.re, -u.im * a.re), wi = fma(u.re, b.im, -u.im * a.im);
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    accV[p].re = fma(s_coef[p][q], wr, accV[p].re);
                    accV[p].im = fma(s_coef[p][q], wi, accV[p].im);
                }
            }
        }
    }
    __syncthreads();
    // sums over the G warps: warp p takes output p
    s_red[(g * (1 + NP)) * 32 + lane] = accH;
#pragma unroll
    for (int p = 0; p < NP; ++p) s_red[(g * (1 + NP) + 1 + p) * 32 + lane] = accV[p];
    __syncthreads();
    const bool on = first + lane < total;
    const int m = (int)(e / N), n = (int)(e - (int64_t)m * N);
    for (int o = g; o <= NP; o += G) {
        auto sum = [&](int i) {
            zc t = s_red[i * 32 + lane];
            for (int w = 1; w < G; ++w) t = t + s_red[(w * (1 + NP) + i) * 32 + lane];
            return t;
        };
        const zc hl = sum(0);
        zc ph = mk(1.0, 0.0), v = o > 0 ? sum(o) : hl;
        if (gauge == TBG_GAUGE_ATOM) {
            // conj(phi_m) phi_n
            const double *kv = k + kk * dim, *tm = tau + 3 * m, *tn = tau + 3 * n;
            double sm = tm[0] * kv[0], sn = tn[0] * kv[0];
            if (dim > 1) sm += tm[1] * kv[1], sn += tn[1] * kv[1];
            if (dim > 2) sm += tm[2] * kv[2], sn += tn[2] * kv[2];
            zc fm, fn;
            sincospi(2.0 * sm, &fm.im, &fm.re);
            sincospi(2.0 * sn, &fn.im, &fn.re);
            ph = cmul(fm, fn);
            if (o > 0) {
                const double* w = dirs + (o - 1) * dim;
                const double *cm = taucart + 3 * m, *cn = taucart + 3 * n;
                double pm = w[0] * cm[0], pn = w[0] * cn[0];
                if (dim > 1) pm += w[1] * cm[1], pn += w[1] * cn[1];
                if (dim > 2) pm += w[2] * cm[2], pn += w[2] * cn[2];
                const double diff = pn - pm;
                v.re -= diff * hl.im;
                v.im += diff * hl.re;
            }
            v = v * ph;
        }
        if (!on) continue;
        if (o > 0)
            V[kk * ldV + (o - 1) * NN + e] = v;
        else if (H)
            H[kk * ldH + e] = v;
    }
}

template <int NP>
int launch_few(cudaStream_t st, const ModelDev& m, int64_t nk, const double* k_d, const double* dirs, int gauge, zc* H,
               int64_t ldH, zc* V, int64_t ldV) {
    const int N = (int)m.nsta, Kc = m.hop_K;
    const int64_t NN = (int64_t)N * N;
    // algorithmic work as for the unpaired sum (8 nR N^2 per output matrix)
    KTimer kt(st, "fourier_gemm_kernel", 8.0 * m.nR * (double)NN * nk * ((H ? 1 : 0) + NP));
    int G = 1;
    while (G < 8 && 4 * G < Kc) G *= 2;
    const int64_t nks = std::min<int64_t>(nk, 31 / NN + 2);
    const size_t smem = sizeof(zc) * std::max<size_t>((size_t)nks * kPairChunk, (size_t)G * (1 + NP) * 32);
    const int64_t step = std::max<int64_t>(1, (int64_t(1) << 35) / NN);  // blocks within a grid's limit
    for (int64_t kb = 0; kb < nk; kb += step) {
        const int64_t n = std::min(step, nk - kb);
        fourier_few_kernel<NP><<<(unsigned)((n * NN + 31) / 32), dim3(32, G), smem, st>>>(
            n, m.dim, k_d + kb * m.dim, m.hop_np, m.hop_pair_d, m.hamR_d, m.Rcart_d, m.pair_T, N, m.tau_d, m.taucart_d,
            dirs, gauge, H ? H + kb * ldH : nullptr, ldH, V ? V + kb * ldV : nullptr, ldV);
        TBG_LAUNCHED("fourier_few_kernel");
    }
    return TBG_OK;
}

// i A of the rmatrix Fourier sum, with the gauge transform and the zeroed
// diagonal of the Atom gauge (velocity.rs:646-656), in place.
__global__ void rmat_gauge_kernel(int64_t nk, int N, int gauge, const zc* __restrict__ orbph, zc* __restrict__ A) {
    const int64_t NN = (int64_t)N * N;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < nk * NN;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t kk = idx / NN;
        const int e = (int)(idx % NN), m = e / N, n = e % N;
        zc a = A[idx];
        if (gauge == TBG_GAUGE_ATOM)
            a = (m == n) ? mk(0.0, 0.0) : a * cmul(orbph[kk * N + m], orbph[kk * N + n]);
        A[idx] = mk(-a.im, a.re);
    }
}

// V[k] += i (H A - A H) for up to kCommSmemMaxN bands, one CTA per k-point with
// H and A in shared memory and one element of the result per thread at a time
// (FP64-pipe bound, as rotate_smem_kernel); the Atom-gauge phases and the zeroed
// diagonal of A (velocity.rs:646-656) are applied while it is loaded.  Above, the
// two products run on the tensor cores (oz64.cu): 33 bands, 1681 k-points, two
// projections 1.5 ms against 1.9 here.
constexpr int kCommSmemMaxN = 25;
__global__ void __launch_bounds__(256) commutator_smem_kernel(int N, int64_t nk, const zc* __restrict__ H,
                                                              const zc* __restrict__ Alat,
                                                              const zc* __restrict__ orbph, int gauge,
                                                              zc* __restrict__ V, int64_t ldV) {
    extern __shared__ __align__(16) unsigned char comm_smem[];
    const int NN = N * N;
    zc* sH = reinterpret_cast<zc*>(comm_smem);
    zc* sA = sH + NN;
    for (int64_t kk = blockIdx.x; kk < nk; kk += gridDim.x) {
        const zc* ph = orbph + kk * N;
        for (int e = threadIdx.x; e < NN; e += blockDim.x) {
            sH[e] = H[kk * NN + e];
            zc a = Alat[kk * NN + e];
            if (gauge == TBG_GAUGE_ATOM) {
                const int m = e / N, n = e - m * N;
                a = (m == n) ? mk(0.0, 0.0) : a * cmul(ph[m], ph[n]);
            }
            sA[e] = a;
        }
        __syncthreads();
        zc* Vk = V + kk * ldV;
        for (int e = threadIdx.x; e < NN; e += blockDim.x) {
            const int i = e / N, j = e - i * N;
            zc ha = mk(0.0, 0.0), ah = mk(0.0, 0.0);
            for (int l = 0; l < N; ++l) {
                fma_cx(ha, sH[i * N + l], sA[l * N + j]);
                fma_cx(ah, sA[i * N + l], sH[l * N + j]);
            }
            zc v = Vk[e];
            v.re -= ha.im - ah.im;  // + i (HA - AH)
            v.im += ha.re - ah.re;
            Vk[e] = v;
        }
        __syncthreads();
    }
}

// combined rmatrix table for projection p: rm_p[r][e] = sum_d w_pd rmatrix[r][d][e];
// step 2 leaves room for i rm_p in the odd rows and fills it (the real-coefficient
// form (cos + i sin) t = cos t + sin (i t))
__global__ void rmat_combine_kernel(int64_t n_rmat, int dim, int N, const double* __restrict__ w,
                                    const zc* __restrict__ rm, int step, zc* __restrict__ out) {
    const int64_t NN = (int64_t)N * N;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < n_rmat * NN;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = idx / NN, e = idx % NN;
        zc s = mk(0.0, 0.0);
        for (int d = 0; d < dim; ++d) {
            const zc a = rm[(r * dim + d) * NN + e];
            s.re += w[d] * a.re;
            s.im += w[d] * a.im;
        }
        out[r * step * NN + e] = s;
        if (step == 2) out[(r * 2 + 1) * NN + e] = mk(-s.im, s.re);
    }
}

// ph3 rows: [0, nk) = u(k,R); [nk, 2nk) = i c_0(R) u; [2nk, 3nk) = i c_1(R) u.
__global__ void phases3_kernel(int64_t nk, int dim, const double* __restrict__ k, int nR,
                               const int* __restrict__ hamR, const double* __restrict__ coef,
                               zc* __restrict__ ph3) {
    const int64_t total = nk * (int64_t)nR;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t kk = idx / nR;
        const int j = (int)(idx % nR);
        const double* kv = k + kk * dim;
        const int* r = hamR + 3 * j;
        double s = (double)r[0] * kv[0];
        if (dim > 1) s += (double)r[1] * kv[1];
        if (dim > 2) s += (double)r[2] * kv[2];
        double sn, cs;
        sincos(kTwoPi * s, &sn, &cs);
        ph3[idx] = mk(cs, sn);
        const double c0 = coef[j], c1 = coef[nR + j];
        ph3[total + idx] = mk(-c0 * sn, c0 * cs);      // i c0 u
        ph3[2 * total + idx] = mk(-c1 * sn, c1 * cs);  // i c1 u
    }
}

// Atom gauge and tau term from the lattice-gauge float-pair sums:
//   H = conj(phi_m) H_l phi_n,  V_p = (V_l,p + i (tau_p,n - tau_p,m) H_l) conj(phi_m) phi_n
// Contraction output C, component c (0: H, 1, 2: V_p) of k-point kk, element
// (m, n): full N x N columns, or only the upper triangle (packed row by row);
// then the lower triangle is the conjugate of its mirror (H and V_p are Hermitian).
__host__ __device__ __forceinline__ int64_t upper_index(int N, int m, int n) {
    return (int64_t)m * N - (int64_t)m * (m - 1) / 2 + (n - m);
}
__device__ __forceinline__ float4 c_elem(const float4* __restrict__ C, bool packed, int64_t nk, int N, int c,
                                         int64_t kk, int m, int n) {
    if (!packed) return C[(c * nk + kk) * (int64_t)N * N + (int64_t)m * N + n];
    const int64_t np = (int64_t)N * (N + 1) / 2;
    if (m <= n) return C[(c * nk + kk) * np + upper_index(N, m, n)];
    const float4 v = C[(c * nk + kk) * np + upper_index(N, n, m)];
    return make_float4(v.x, v.y, -v.z, -v.w);
}

__global__ void gauge_pairs_kernel(int64_t nk, int N, const float4* __restrict__ C, bool packed,
                                   const zc* __restrict__ orbph, const double* __restrict__ taup, zc* __restrict__ H,
                                   zc* __restrict__ V) {
    const int64_t NN = (int64_t)N * N;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < nk * NN;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t kk = idx / NN;
        const int e = (int)(idx % NN), mrow = e / N, ncol = e % N;
        const float4 h4 = c_elem(C, packed, nk, N, 0, kk, mrow, ncol);
        const zc hl = mk((double)h4.x + (double)h4.y, (double)h4.z + (double)h4.w);
        const zc g = cmul(orbph[kk * N + mrow], orbph[kk * N + ncol]);
        H[idx] = hl * g;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const float4 v4 = c_elem(C, packed, nk, N, 1 + p, kk, mrow, ncol);
            zc v = mk((double)v4.x + (double)v4.y, (double)v4.z + (double)v4.w);
            const double diff = taup[p * N + ncol] - taup[p * N + mrow];
            v.re -= diff * hl.im;
            v.im += diff * hl.re;
            V[kk * 2 * NN + p * NN + e] = v * g;
        }
    }
}

// taup (FP64) -> float pairs
__global__ void tau_split_kernel(int n, const double* __restrict__ taup, float2* __restrict__ tau2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) tau2[i] = df_of(taup[i]);
}

// Lattice gauge, float-pair arithmetic, in place on the contraction output:
//   V_p += i (tau_p,n - tau_p,m) H_l   (velocity.rs:602-610 before the phase).
// The Atom-gauge phase conj(phi_m) phi_n is a diagonal unitary similarity
// (H_atom = P^H H_l P, V_atom = P^H V_l P), so energies and band-basis
// velocities, hence Omega, do not depend on it; the mixed path skips it.
__global__ void tau_pairs_kernel(int64_t nk, int N, float4* __restrict__ C, const float2* __restrict__ tau2) {
    const int64_t NN = (int64_t)N * N;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= NN) return;
    const int mrow = e / N, ncol = e - mrow * N;
    float2 d[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) d[p] = df_add(tau2[p * N + ncol], df_neg(tau2[p * N + mrow]));
    for (int64_t kk = blockIdx.y; kk < nk; kk += gridDim.y) {
        const int64_t idx = kk * NN + e;
        const float4 h = C[idx];
        const float2 hr = make_float2(h.x, h.y), hi = make_float2(h.z, h.w);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            float4* vp = C + (1 + p) * nk * NN + idx;
            const float4 v = *vp;
            const float2 vr = df_add(make_float2(v.x, v.y), df_neg(df_mul(d[p], hi)));
            const float2 vi = df_add(make_float2(v.z, v.w), df_mul(d[p], hr));
            *vp = make_float4(vr.x, vr.y, vi.x, vi.y);
        }
    }
}

// Packed upper-triangle contraction output -> full float-pair H, V_0, V_1
// (P: three blocks of nk N^2 elements, blk elements apart) with the
// orbital-position term V_p += i (tau_p,n - tau_p,m) H, in float-pair arithmetic.
// A block writes 32 rows of one k-point's three matrices, 32 columns at a time, so
// with rexp (three blocks of nk N ints) it has the rows' exponents as well.  Tiles
// right of the diagonal are read as they lie; those below it are read as rows of
// the upper triangle and turned over in shared memory, since element by element
// a warp touched 32 lines per load (8192 k-points of 128 bands 2.36 -> 1.89 ms, 6.4 GB
// written; 304 of 251 bands 0.38 -> 0.34).
constexpr int kUnpackThreads = 256, kUnpackTile = 32;

__global__ void __launch_bounds__(kUnpackThreads) unpack_tau_kernel(int64_t nk, int N, const float4* __restrict__ Cp,
                                                                   const float2* __restrict__ tau2,
                                                                   float4* __restrict__ P, int64_t blk,
                                                                   int* __restrict__ rexp) {
    constexpr int TL = kUnpackTile, NW = kUnpackThreads / 32, NR = TL / NW;  // NR rows per warp
    // units of a row permuted by its low bits: no bank conflicts by rows or columns
    __shared__ float4 tile[3][TL * TL];
    const int64_t NN = (int64_t)N * N, np = (int64_t)N * (N + 1) / 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int R = blockIdx.x, T = (N + TL - 1) / TL;
    for (int64_t kk = blockIdx.y; kk < nk; kk += gridDim.y) {
        float mag[3][NR] = {};
        for (int J = 0; J < T; ++J) {
            const int n = J * TL + lane;
            if (J <= R) {
                __syncthreads();
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    const int r = warp + NW * i, gm = J * TL + r, gn = R * TL + lane;
                    if (gm <= gn && gn < N)
#pragma unroll
                        for (int c = 0; c < 3; ++c)
                            tile[c][r * TL + (lane ^ (r & 7))] = Cp[(c * nk + kk) * np + upper_index(N, gm, gn)];
                }
                __syncthreads();
            }
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const int r = warp + NW * i, m = R * TL + r;
                if (m >= N || n >= N) continue;
                auto elem = [&](int c) {
                    if (J > R) return Cp[(c * nk + kk) * np + upper_index(N, m, n)];
                    if (m <= n) return tile[c][r * TL + (lane ^ (r & 7))];
                    const float4 v = tile[c][lane * TL + (r ^ (lane & 7))];
                    return make_float4(v.x, v.y, -v.z, -v.w);
                };
                const float4 h = elem(0);
                float4* out = P + kk * NN + (int64_t)m * N + n;
                out[0] = h;
                // a NaN counts as 0, as fmaxf over a row would skip it
                mag[0][i] = fmaxf(mag[0][i], pair_mag(h));
                const float2 hr = make_float2(h.x, h.y), hi = make_float2(h.z, h.w);
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const float4 v = elem(1 + p);
                    const float2 d = df_add(tau2[p * N + n], df_neg(tau2[p * N + m]));
                    const float2 vr = df_add(make_float2(v.x, v.y), df_neg(df_mul(d, hi)));
                    const float2 vi = df_add(make_float2(v.z, v.w), df_mul(d, hr));
                    const float4 o = make_float4(vr.x, vr.y, vi.x, vi.y);
                    out[(1 + p) * blk] = o;
                    mag[1 + p][i] = fmaxf(mag[1 + p][i], pair_mag(o));
                }
            }
        }
        if (rexp) {
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int i = 0; i < NR; ++i) {
                    // magnitudes are >= 0: their bit patterns order as integers
                    const int v = __reduce_max_sync(0xffffffffu, __float_as_int(mag[c][i])), m = R * TL + warp + NW * i;
                    if (lane == 0 && m < N) rexp[(c * nk + kk) * N + m] = line_exp_of(__int_as_float(v));
                }
        }
    }
}

std::mutex g_hop_mu;

}  // namespace

int ozaki_fourier_max_k();
size_t ozaki_hop_slices_bytes(int K, int64_t Nc);
int ozaki_build_hop_slices_real(cudaStream_t st, int Kc, int64_t Nc, const zc* T, int* EB, void* Bs,
                                const int* colmap, int64_t ncols);
int ozaki_build_hop_slices(cudaStream_t st, int K, int64_t Nc, const zc* ham, int* EB, void* Bs, const int* colmap,
                           int64_t ncols);
int ozaki_fourier(cudaStream_t st, int64_t M, int64_t Nc, int K, const zc* A, int* EA, const int* EB,
                  const void* Bs, float4* C, int* err, int64_t high_rows, void* aimg);
size_t ozaki_fourier_img_bytes(int64_t M, int K);

// Class of the velocity rows of the exact-slice Fourier sum: MID (five digits,
// about 2^-35 of the row scale; the velocities only enter the rotation, which
// is a MID product itself) unless TBG_FOURIER_V_HIGH=1.  The Hamiltonian rows
// stay HIGH.
static bool fourier_v_mid() {
    static const bool mid = [] {
        const char* e = std::getenv("TBG_FOURIER_V_HIGH");
        return !(e && e[0] == '1');
    }();
    return mid;
}

bool fourier_mixed_ok(const ModelDev& m) { return m.nR <= ozaki_fourier_max_k(); }

size_t fourier_mixed_scratch_bytes(const ModelDev& m, int64_t nk) {
    const size_t N = (size_t)m.nsta, nR = (size_t)m.nR;
    // phases, orbital phases, exponents; the packed (upper-triangle) contraction
    // output; the phases' stage images
    return (size_t)nk * (3 * (nR + 1) * sizeof(zc) + N * sizeof(zc) + 3 * sizeof(int) +
                         3 * (N * (N + 1) / 2) * sizeof(float4)) +
           ozaki_fourier_img_bytes(3 * nk, (int)nR + 1) + 2 * nR * sizeof(double) + 2 * N * sizeof(double) +
           2 * N * sizeof(float2) + 11 * 256;
}

namespace {

// Phases and the tensor-core contraction: C (3 nk N^2 float pairs) = lattice-
// gauge H, V_0, V_1 without the orbital-position term.  orbph (nk, N) and
// taup (2, N) are left in the scratch for the gauge step.
// With the tcgen05 kernels the contraction covers only the upper-triangle
// elements (m <= n) of H and V_p, which are Hermitian: N(N+1)/2 columns, written
// packed to *Cg in the scratch; otherwise all N^2 columns are written to C.
__global__ void gather_exps_kernel(int64_t n, const int* __restrict__ idx, const int* __restrict__ src,
                                   int* __restrict__ dst) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = src[idx[i]];
}

// The table paired over +-R for real coefficients: with theta = 2 pi k . R,
//   t(R) e^{i theta} + t(-R) e^{-i theta} = A cos(theta) + B sin(theta),
//   A = t(R) + t(-R),  B = i (t(R) - t(-R))
// (an R without its -R partner takes t(-R) = 0).  Rows: 0 = t(0), 1 = 0,
// 2 + 2p = A_p, 3 + 2p = B_p.  pi[p] is the pair's R, pj[p] its -R or -1.
// A non-finite entry sets bit 0 of *flags (the exact-slice digits of the
// tensor-core form cannot carry NaN or Inf, so the mixed path refuses such a
// table up front), one of 2^960 or more bit 1 (no room for the pairs' weights).
__global__ void pair_table_kernel(int np, const int* __restrict__ pi, const int* __restrict__ pj, int z, int64_t NN,
                                  const zc* __restrict__ ham, zc* __restrict__ T, int* __restrict__ flags) {
    const int64_t total = (int64_t)(np + 1) * NN;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = idx / NN - 1, e = idx % NN;
        zc a, b;
        if (p < 0) {
            a = (z >= 0) ? ham[(int64_t)z * NN + e] : mk(0.0, 0.0);
            b = mk(0.0, 0.0);
            T[e] = a;
            T[NN + e] = b;
        } else {
            a = ham[(int64_t)pi[p] * NN + e];
            b = (pj[p] >= 0) ? ham[(int64_t)pj[p] * NN + e] : mk(0.0, 0.0);
            T[(2 + 2 * p) * NN + e] = mk(a.re + b.re, a.im + b.im);
            T[(3 + 2 * p) * NN + e] = mk(-(a.im - b.im), a.re - b.re);
        }
        const double big = fmax(fmax(fabs(a.re), fabs(a.im)), fmax(fabs(b.re), fabs(b.im)));
        if (!(isfinite(a.re) && isfinite(a.im) && isfinite(b.re) && isfinite(b.im)))
            atomicOr(flags, 1);
        else if (big >= 0x1p960)
            atomicOr(flags, 2);
    }
}

// Real coefficients of the paired table, as complex numbers whose real and
// imaginary parts are consecutive rows (Phi (1 + nproj, nk, Kc), Kc = 1 + np): H
// row (1, 0 | cos, sin ...), V_p rows (0, 0 | -c_p(R) sin, c_p(R) cos ...), from
//   i c_p(R) (t(R) e^{i theta} - t(-R) e^{-i theta}) = c_p(R) (B cos - A sin).
// skip 1 leaves the R = 0 column out (Kc = np); wexp: columns over their pair's weight.
__global__ void phases_real_kernel(int64_t nk, int dim, const double* __restrict__ k, int np,
                                   const int* __restrict__ pair, const int* __restrict__ hamR, int nR, int nproj,
                                   const double* __restrict__ coef, int skip, const int* __restrict__ wexp,
                                   zc* __restrict__ Phi) {
    const int Kc = np + 1 - skip;
    const int64_t total = nk * (int64_t)Kc;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t kk = idx / Kc;
        const int c = (int)(idx % Kc);
        if (c + skip == 0) {
            Phi[idx] = mk(1.0, 0.0);
            for (int p = 0; p < nproj; ++p) Phi[(1 + p) * total + idx] = mk(0.0, 0.0);
            continue;
        }
        const int j = pair[c + skip - 1];
        const int* r = hamR + 3 * j;
        const double* kv = k + kk * dim;
        // same operation order as the reference: r0*k0 + r1*k1 + r2*k2
        double s = (double)r[0] * kv[0];
        if (dim > 1) s += (double)r[1] * kv[1];
        if (dim > 2) s += (double)r[2] * kv[2];
        double sn, cs;
        sincos(kTwoPi * s, &sn, &cs);
        if (wexp) {
            const double w = __hiloint2double((1023 - wexp[c + skip - 1]) << 20, 0);  // 2^-wexp
            cs *= w;
            sn *= w;
        }
        Phi[idx] = mk(cs, sn);
        for (int p = 0; p < nproj; ++p) {
            const double cp = coef[(int64_t)p * nR + j];
            Phi[(1 + p) * total + idx] = mk(-cp * sn, cp * cs);
        }
    }
}

// The +-R paired table (pair_table_kernel) and the index of each pair's R,
// built once per model for both Fourier forms; the caller holds g_hop_mu.
int ensure_pair_table(ModelDev& m, cudaStream_t st) {
    if (m.pair_T) return TBG_OK;
    const int nR = (int)m.nR;
    const int64_t NN = (int64_t)m.nsta * m.nsta;
    int z = -1;
    std::vector<int> pi, pj;
    std::vector<char> used((size_t)nR, 0);
    auto rvec = [&](int i, int d) { return d < m.dim ? m.hamR[(size_t)i * m.dim + d] : (int64_t)0; };
    for (int i = 0; i < nR; ++i) {
        if (used[i]) continue;
        used[i] = 1;
        if (rvec(i, 0) == 0 && rvec(i, 1) == 0 && rvec(i, 2) == 0 && z < 0) {
            z = i;  // a repeated R = 0 entry is paired below as a singleton (theta = 0)
            continue;
        }
        int partner = -1;
        for (int j = i + 1; j < nR && partner < 0; ++j)
            if (!used[j] && rvec(j, 0) == -rvec(i, 0) && rvec(j, 1) == -rvec(i, 1) && rvec(j, 2) == -rvec(i, 2))
                partner = j;
        if (partner >= 0) used[partner] = 1;
        pi.push_back(i);
        pj.push_back(partner);
    }
    const int np = (int)pi.size(), Kc = np + 1;
    // Weights of the pairs in the FP64-accurate products, whose error is relative to the
    // largest coefficient and the largest table entry of a column: the velocities' c_p(R)
    // grow with |R| while t(R) falls, so |R| (over the shortest, as a power of two) goes
    // from the coefficients to the table.
    std::vector<int> wexp((size_t)std::max(np, 1), 0);
    std::vector<double> len((size_t)np, 0.0);
    double shortest = 0.0;
    for (int p = 0; p < np; ++p) {
        double l2 = 0.0;
        for (int c = 0; c < m.dim; ++c) {
            double x = 0.0;
            for (int d = 0; d < m.dim; ++d) x += (double)rvec(pi[p], d) * m.lat[(size_t)d * m.dim + c];
            l2 += x * x;
        }
        len[p] = std::sqrt(l2);
        if (len[p] > 0.0 && (shortest == 0.0 || len[p] < shortest)) shortest = len[p];
    }
    for (int p = 0; p < np; ++p)
        if (len[p] > 0.0 && std::isfinite(len[p]))
            wexp[p] = std::min(48, std::max(0, (int)std::lround(std::log2(len[p] / shortest))));
    // one block for what the device needs beside the table: the pairs' R, their weights, their
    // -R and the flags
    const int n1 = std::max(np, 1);
    std::vector<int> idx((size_t)3 * n1 + 1, 0);
    std::copy(pi.begin(), pi.end(), idx.begin());
    std::copy(wexp.begin(), wexp.end(), idx.begin() + n1);
    std::copy(pj.begin(), pj.end(), idx.begin() + 2 * n1);
    int* idx_d = nullptr;
    zc* T = nullptr;
    int rc = TBG_OK;
    if (cudaMalloc(&T, sizeof(zc) * 2 * (size_t)Kc * NN) != cudaSuccess ||
        cudaMalloc(&idx_d, sizeof(int) * idx.size()) != cudaSuccess)
        rc = set_error(TBG_E_OOM, "paired hop table");
    if (!rc && cudaMemcpyAsync(idx_d, idx.data(), sizeof(int) * idx.size(), cudaMemcpyHostToDevice, st) != cudaSuccess)
        rc = set_error(TBG_E_CUDA, "paired hop table indices");
    if (!rc) {
        int* flags_d = idx_d + 3 * n1;
        pair_table_kernel<<<(unsigned)std::min<int64_t>(((int64_t)Kc * NN + 255) / 256, 152 * 64), 256, 0, st>>>(
            np, idx_d, idx_d + 2 * n1, z, NN, m.ham, T, flags_d);
        count_launch();
        int flags = 0;
        cudaError_t e = cudaMemcpyAsync(&flags, flags_d, sizeof(int), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);  // other streams use the table next
        if (e == cudaSuccess && (flags & 2)) {
            e = cudaMemsetAsync(idx_d + n1, 0, sizeof(int) * n1, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        }
        if (e != cudaSuccess) rc = cuda_error(e, "paired hop table");
        m.nonfinite = (flags & 1) != 0;
    }
    if (rc) {
        cudaFree(T);
        cudaFree(idx_d);
        return rc;
    }
    m.hop_pair_d = idx_d;
    m.hop_wexp_d = idx_d + n1;
    m.pair_T = T;
    m.hop_np = np;
    m.hop_K = Kc;
    return TBG_OK;
}

int build_hop_table(ModelDev& m, cudaStream_t st) {
    const int N = (int)m.nsta, nR = (int)m.nR;
    const int64_t NN = (int64_t)N * N, NP = (int64_t)N * (N + 1) / 2;
    const bool packed = ozaki_use_tc();
    const int64_t ncols = packed ? NP : NN;
    if (packed) {
        int rc = ensure_pair_table(m, st);
        if (rc) return rc;
    }
    const int Kc = packed ? m.hop_K : nR;
    const zc* T = m.pair_T;
    void* bs = nullptr;
    int *eb_full = nullptr, *eb = nullptr, *colmap = nullptr;
    int rc = TBG_OK;
    if (cudaMalloc(&bs, ozaki_hop_slices_bytes(Kc, ncols)) != cudaSuccess) return set_error(TBG_E_OOM, "hop table digit planes");
    if (cudaMalloc(&eb_full, sizeof(int) * NN) != cudaSuccess ||
        (packed && (cudaMalloc(&eb, sizeof(int) * NP) != cudaSuccess ||
                    cudaMalloc(&colmap, sizeof(int) * NP) != cudaSuccess)))
        rc = set_error(TBG_E_OOM, "hop table digit planes");
    if (!rc && packed) {
        std::vector<int> cm((size_t)NP);
        for (int a = 0; a < N; ++a)
            for (int b = a; b < N; ++b) cm[(size_t)upper_index(N, a, b)] = a * N + b;
        if (cudaMemcpyAsync(colmap, cm.data(), sizeof(int) * NP, cudaMemcpyHostToDevice, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)  // cm goes
            rc = set_error(TBG_E_CUDA, "hop table column map");
    }
    if (!rc)
        rc = packed ? ozaki_build_hop_slices_real(st, Kc, NN, T, eb_full, bs, colmap, ncols)
                    : ozaki_build_hop_slices(st, nR, NN, m.ham, eb_full, bs, nullptr, ncols);
    if (!rc && packed) {
        gather_exps_kernel<<<(unsigned)std::min<int64_t>((NP + 255) / 256, 1024), 256, 0, st>>>(NP, colmap, eb_full,
                                                                                                  eb);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = cuda_error(e, "hop table exponents");
    }
    if (!rc) {
        cudaError_t e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) rc = cuda_error(e, "hop table digit planes");
    }
    cudaFree(colmap);
    if (rc) {
        cudaFree(bs);
        cudaFree(eb_full);
        cudaFree(eb);
        return rc;
    }
    if (packed) cudaFree(eb_full);
    m.hop_slices = bs;
    m.hop_EB = packed ? eb : eb_full;
    m.hop_packed = packed;
    return TBG_OK;
}

int fourier_mixed_gemm(ModelDev& m, cudaStream_t st, int64_t nk, const double* k_d, const double* dirs_d, float4* C,
                       void* scratch, zc** orbph_out, double** taup_out, float2** tau2_out, float4** Cg_out) {
    const int N = (int)m.nsta, nR = (int)m.nR;
    const int64_t NN = (int64_t)N * N, NP = (int64_t)N * (N + 1) / 2;
    {
        std::lock_guard<std::mutex> lk(g_hop_mu);
        if (!m.hop_slices) {
            int rc = build_hop_table(m, st);
            if (rc) return rc;
        }
    }
    if (m.nonfinite) return set_error(TBG_E_NOCONV, "the hopping table contains NaN or Inf");
    unsigned char* p = static_cast<unsigned char*>(scratch);
    auto take = [&](size_t bytes) {
        void* q = p;
        p += (bytes + 255) & ~size_t(255);
        return q;
    };
    zc* ph3 = static_cast<zc*>(take(sizeof(zc) * 3 * nk * (nR + 1)));  // Phi (3 nk x hop_K <= nR + 1) when packed
    zc* orbph = static_cast<zc*>(take(sizeof(zc) * nk * N));
    double* coef = static_cast<double*>(take(sizeof(double) * 2 * nR));
    double* taup = static_cast<double*>(take(sizeof(double) * 2 * N));
    float2* tau2 = static_cast<float2*>(take(sizeof(float2) * 2 * N));
    int* EA = static_cast<int*>(take(sizeof(int) * 3 * nk));
    int* err = static_cast<int*>(take(sizeof(int)));
    float4* Cpk = static_cast<float4*>(take(sizeof(float4) * 3 * nk * NP));
    void* aimg = take(ozaki_fourier_img_bytes(3 * nk, m.hop_packed ? m.hop_K : nR));
    float4* Cg = m.hop_packed ? Cpk : C;
    {
        KTimer kt(st, "phases_kernel");
        const int total = 2 * (nR + N);
        proj_coef_kernel<<<(total + 255) / 256, 256, 0, st>>>(2, m.dim, dirs_d, nR, m.Rcart_d, N, m.taucart_d, coef,
                                                              taup);
        if (m.hop_packed) {
            // orbital phases only, then the real coefficients of the paired table
            const int64_t t1 = nk * (int64_t)N;
            phases_kernel<<<(unsigned)std::min<int64_t>((t1 + 255) / 256, 65535 * 8), 256, 0, st>>>(
                nk, m.dim, k_d, 0, m.hamR_d, N, m.tau_d, ph3, orbph);
            const int64_t t2 = nk * (int64_t)m.hop_K;
            phases_real_kernel<<<(unsigned)std::min<int64_t>((t2 + 255) / 256, 65535 * 8), 256, 0, st>>>(
                nk, m.dim, k_d, m.hop_np, m.hop_pair_d, m.hamR_d, nR, 2, coef, 0, nullptr, ph3);
        } else {
            const int64_t t1 = nk * (int64_t)(nR + N);
            phases_kernel<<<(unsigned)std::min<int64_t>((t1 + 255) / 256, 65535 * 8), 256, 0, st>>>(
                nk, m.dim, k_d, nR, m.hamR_d, N, m.tau_d, ph3, orbph);  // ph3[0 .. nk*nR) reused below
            const int64_t t2 = nk * (int64_t)nR;
            phases3_kernel<<<(unsigned)std::min<int64_t>((t2 + 255) / 256, 65535 * 8), 256, 0, st>>>(
                nk, m.dim, k_d, nR, m.hamR_d, coef, ph3);
        }
        tau_split_kernel<<<(2 * N + 255) / 256, 256, 0, st>>>(2 * N, taup, tau2);
        count_launch(4);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_error(e, "phases");
    }
    int rc = cudaMemsetAsync(err, 0, sizeof(int), st) == cudaSuccess ? TBG_OK : set_error(TBG_E_CUDA, "memset");
    if (rc) return rc;
    // rows [H | Vx | Vy] (nk each): H in the HIGH class, the velocities in MID
    rc = ozaki_fourier(st, 3 * nk, m.hop_packed ? NP : NN, m.hop_packed ? m.hop_K : nR, ph3, EA, m.hop_EB,
                       m.hop_slices, Cg, err, fourier_v_mid() ? nk : -1, aimg);
    if (rc) return rc;
    *Cg_out = Cg;
    *orbph_out = orbph;
    *taup_out = taup;
    *tau2_out = tau2;
    return TBG_OK;
}

}  // namespace

int fourier_mixed(ModelDev& m, cudaStream_t st, int64_t nk, const double* k_d, const double* dirs_d, zc* H, zc* V,
                  float4* C, void* scratch, size_t scratch_bytes, int* status_d) {
    if (nk <= 0) return TBG_OK;
    const int N = (int)m.nsta;
    const int64_t NN = (int64_t)N * N;
    if (!fourier_mixed_ok(m) || !C || scratch_bytes < fourier_mixed_scratch_bytes(m, nk))
        return fourier_direct(m, st, nk, k_d, TBG_GAUGE_ATOM, 2, dirs_d, H, V, NN, 2 * NN, status_d);
    zc* orbph;
    double* taup;
    float2* tau2;
    float4* Cg;
    int rc = fourier_mixed_gemm(m, st, nk, k_d, dirs_d, C, scratch, &orbph, &taup, &tau2, &Cg);
    if (rc) return rc;
    KTimer kt(st, "gauge_pairs_kernel");
    gauge_pairs_kernel<<<(unsigned)std::min<int64_t>((nk * NN + 255) / 256, 152 * 64), 256, 0, st>>>(
        nk, N, Cg, m.hop_packed, orbph, taup, H, V);
    TBG_LAUNCHED("gauge_pairs_kernel");
    return TBG_OK;
}

int fourier_mixed_packed(ModelDev& m, cudaStream_t st, bool* packed) {
    std::lock_guard<std::mutex> lk(g_hop_mu);
    if (!m.hop_slices) {
        int rc = build_hop_table(m, st);
        if (rc) return rc;
    }
    *packed = m.hop_packed;
    return TBG_OK;
}

int fourier_mixed_pairs(ModelDev& m, cudaStream_t st, int64_t nk, const double* k_d, const double* dirs_d,
                        float4* C, void* scratch, size_t scratch_bytes, float4* out, int64_t blk, int* rexp,
                        bool* rexp_filled) {
    if (rexp_filled) *rexp_filled = false;
    if (nk <= 0) return TBG_OK;
    if (!fourier_mixed_ok(m) || scratch_bytes < fourier_mixed_scratch_bytes(m, nk))
        return set_error(TBG_E_UNSUPPORTED, "fourier_mixed_pairs: nR beyond the exact contraction length");
    const int N = (int)m.nsta;
    const int64_t NN = (int64_t)N * N;
    if (!out) {
        out = C;
        blk = nk * NN;
    }
    zc* orbph;
    double* taup;
    float2* tau2;
    float4* Cg;
    int rc = fourier_mixed_gemm(m, st, nk, k_d, dirs_d, C, scratch, &orbph, &taup, &tau2, &Cg);
    if (rc) return rc;
    KTimer kt(st, "tau_pairs_kernel");
    dim3 grid((unsigned)((NN + 255) / 256), (unsigned)std::min<int64_t>(nk, 65535));
    if (m.hop_packed) {
        if (rexp && rexp_filled) *rexp_filled = true;
        const dim3 tiles((unsigned)((N + kUnpackTile - 1) / kUnpackTile), grid.y);
        unpack_tau_kernel<<<tiles, kUnpackThreads, 0, st>>>(nk, N, Cg, tau2, out, blk, rexp);
        TBG_LAUNCHED("unpack_tau_kernel");
    } else {
        tau_pairs_kernel<<<grid, 256, 0, st>>>(nk, N, C, tau2);
        TBG_LAUNCHED("tau_pairs_kernel");
        if (out != C)
            for (int p = 0; p < 3; ++p)
                TBG_CUDA(cudaMemcpyAsync(out + p * blk, C + p * nk * NN, sizeof(float4) * nk * NN,
                                         cudaMemcpyDeviceToDevice, st));
    }
    return TBG_OK;
}

namespace {

// Lattice-gauge sums G (1 + nproj blocks of nk N^2: H without its R = 0 term t0, V_p) -> H, V
// with the orbital-position term and the gauge phases, as the epilogue of fourier_few_kernel.
__global__ void __launch_bounds__(256) gauge64_kernel(int64_t nk, int N, int nproj, const zc* __restrict__ G,
                                                      const zc* __restrict__ t0,
                                                      const zc* __restrict__ orbph, const double* __restrict__ taup,
                                                      int gauge, zc* __restrict__ H, int64_t ldH, zc* __restrict__ V,
                                                      int64_t ldV) {
    const int64_t NN = (int64_t)N * N;
    for (int64_t kk = blockIdx.y; kk < nk; kk += gridDim.y) {
        for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < (int)NN; e += gridDim.x * blockDim.x) {
            const int mrow = e / N, ncol = e - mrow * N;
            const zc hl = G[kk * NN + e] + t0[e];
            zc g = mk(1.0, 0.0);
            if (gauge == TBG_GAUGE_ATOM) g = cmul(orbph[kk * N + mrow], orbph[kk * N + ncol]);
            if (H) H[kk * ldH + e] = gauge == TBG_GAUGE_ATOM ? hl * g : hl;
            for (int p = 0; p < nproj; ++p) {
                zc v = G[((1 + p) * nk + kk) * NN + e];
                if (gauge == TBG_GAUGE_ATOM) {
                    const double diff = taup[p * N + ncol] - taup[p * N + mrow];
                    v.re -= diff * hl.im;
                    v.im += diff * hl.re;
                    v = v * g;
                }
                V[kk * ldV + p * NN + e] = v;
            }
        }
    }
}

// The digit image of the paired table for the tensor-core form, built once per
// model; the caller holds g_hop_mu.  R = 0 is left to gauge64_kernel: on-site energies are often
// a thousand times the hoppings, and the velocities, which have no such term, would
// carry errors relative to them.  The image is 1.8 times the hopping table and stays while
// the model does, so it is made only while it takes at most an eighth of the free memory
// (sets of many models); without it m.oz_img stays null and the sums take the direct form.
int ensure_table_image(ModelDev& m, cudaStream_t st) {
    if (m.oz_img || m.nonfinite || m.hop_np == 0) return TBG_OK;
    const int64_t NN = (int64_t)m.nsta * m.nsta;
    const size_t bytes = oz64_table_image_bytes(m.hop_np, NN);
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
        cudaGetLastError();
        return TBG_OK;
    }
    if (bytes > std::min(free_b / 8, scratch_cap())) return TBG_OK;
    void* img = nullptr;
    int* eb = nullptr;
    if (cudaMalloc(&img, bytes) != cudaSuccess ||
        cudaMalloc(&eb, sizeof(int) * NN) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(img);
        return TBG_OK;
    }
    int rc = oz64_table_image(st, m.hop_np, NN, m.pair_T + 2 * NN, m.hop_wexp_d, eb, img);
    if (!rc) {
        cudaError_t e = cudaStreamSynchronize(st);  // other streams use the image next
        if (e != cudaSuccess) rc = cuda_error(e, "table image");
    }
    if (rc) {
        cudaFree(img);
        cudaFree(eb);
        return rc;
    }
    m.oz_img = img;
    m.oz_EB = eb;
    return TBG_OK;
}

// Whether M x NN sums over Kc pairs (work: FP64 instructions of the direct form, per
// output lane) take the tensor-core form.  Both sides in us: the launches and, per
// round of tiles over the SMs, 8 and 1 a stage, against the direct form at 0.6 of
// the FP64 pipe's rate (60 instructions an element for its gauge phases).  301 k-points
// of 14 bands, 125 R: 34 against 64 us; 12 of 512 bands, 9 R: 0.41 against 0.73 ms.
bool oz64_sum_pays(int64_t M, int64_t NN, int Kc, double work) {
    const int64_t rounds = ((M + 127) / 128 * ((NN + 31) / 32) + 151) / 152;
    return 25.0 + (double)rounds * (8.0 + (Kc + 15) / 16) < work / 3.2e5;
}
// Sums held at a time: about this much, but a row tile's 128 k-points at least, so that the
// table's image is read once for full tiles; less where that does not fit.
constexpr int64_t kOzFourierBytes = 512LL << 20;

// H and nproj projections on the tensor cores at FP64 accuracy (oz64.cu): the
// real coefficients of every output (rows: H, V_0, V_1, ... per k-point) times
// the paired table.  TBG_E_OOM, with nothing done, when not even one k-point's scratch fits.
int fourier_oz64(const ModelDev& m, cudaStream_t st, int64_t nk, const double* k_d, int gauge, int nproj,
                 const double* dirs_d, zc* H, zc* V, int64_t ldH, int64_t ldV, int* status_d) {
    const int N = (int)m.nsta, nR = (int)m.nR, Kc = m.hop_np;  // R = 0 apart
    const int64_t NN = (int64_t)N * N;
    int64_t sub = std::max<int64_t>(1, kOzFourierBytes / (int64_t)(sizeof(zc) * NN * (1 + nproj)));
    sub = sub >= 128 ? sub / 128 * 128 : std::min<int64_t>(128, nk);
    sub = std::min(sub, nk);
    const int npc = std::max(nproj, 1);
    size_t off, o_phi, o_orb, o_coef, o_tau, o_ea, o_img, o_g;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) & ~size_t(255);
        return o;
    };
    void* mem = nullptr;
    for (;; sub = (sub + 1) / 2) {
        const int64_t M = sub * (1 + nproj);
        off = 0;
        o_phi = take(sizeof(zc) * M * Kc), o_orb = take(sizeof(zc) * sub * N);
        o_coef = take(sizeof(double) * npc * nR), o_tau = take(sizeof(double) * npc * N);
        o_ea = take(sizeof(int) * M), o_img = take(oz64_row_image_bytes(M, Kc));
        o_g = take(sizeof(zc) * M * NN);
        const cudaError_t e = scratch_alloc(&mem, off, st);
        if (e == cudaSuccess) break;
        if (sub == 1) return cuda_error(e, "fourier_oz64 scratch");
    }
    unsigned char* buf = static_cast<unsigned char*>(mem);
    zc* phi = reinterpret_cast<zc*>(buf + o_phi);
    zc* orbph = reinterpret_cast<zc*>(buf + o_orb);
    double* coef = reinterpret_cast<double*>(buf + o_coef);
    double* taup = reinterpret_cast<double*>(buf + o_tau);
    int* EA = reinterpret_cast<int*>(buf + o_ea);
    zc* G = reinterpret_cast<zc*>(buf + o_g);
    int rc = TBG_OK;
    auto launched = [&](const char* what) {
        count_launch();
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess && !rc) rc = cuda_error(e, what);
    };
    if (nproj > 0) {
        const int total = nproj * (nR + N);
        proj_coef_kernel<<<(total + 255) / 256, 256, 0, st>>>(nproj, m.dim, dirs_d, nR, m.Rcart_d, N, m.taucart_d, coef,
                                                              taup);
        launched("proj_coef_kernel");
    }
    for (int64_t k0 = 0; k0 < nk && !rc; k0 += sub) {
        const int64_t nks = std::min(sub, nk - k0);
        {
            KTimer kt(st, "phases_kernel");
            const int64_t t1 = nks * (int64_t)N, t2 = nks * (int64_t)Kc;
            if (gauge == TBG_GAUGE_ATOM) {
                phases_kernel<<<(unsigned)std::min<int64_t>((t1 + 255) / 256, 65535 * 8), 256, 0, st>>>(
                    nks, m.dim, k_d + k0 * m.dim, 0, m.hamR_d, N, m.tau_d, phi, orbph);
                launched("phases_kernel");
            }
            phases_real_kernel<<<(unsigned)std::min<int64_t>((t2 + 255) / 256, 65535 * 8), 256, 0, st>>>(
                nks, m.dim, k_d + k0 * m.dim, m.hop_np, m.hop_pair_d, m.hamR_d, nR, nproj, coef, 1, m.hop_wexp_d, phi);
            launched("phases_real_kernel");
        }
        if (!rc)
            rc = oz64_table_product(st, nks * (1 + nproj), NN, Kc, phi, Kc, m.oz_EB, m.oz_img, G, EA, buf + o_img,
                                    status_d);
        if (rc) break;
        KTimer kt(st, "gauge64_kernel");
        const dim3 grid((unsigned)std::min<int64_t>((NN + 255) / 256, 1024), (unsigned)std::min<int64_t>(nks, 65535));
        gauge64_kernel<<<grid, 256, 0, st>>>(nks, N, nproj, G, m.pair_T, orbph, taup, gauge, H ? H + k0 * ldH : nullptr, ldH,
                                             V ? V + k0 * ldV : nullptr, ldV);
        launched("gauge64_kernel");
    }
    cudaFreeAsync(buf, st);
    return rc;
}

}  // namespace

int fourier_direct(const ModelDev& m, cudaStream_t st, int64_t nk, const double* k_d, int gauge, int nproj,
                   const double* dirs_d, zc* H, zc* V, int64_t ldH, int64_t ldV, int* status_d) {
    if (nk <= 0) return TBG_OK;
    const int N = (int)m.nsta;
    bool oz = false;
    {
        // the +-R paired table, built once per model (a cache: logically const)
        std::lock_guard<std::mutex> lk(g_hop_mu);
        int rc = ensure_pair_table(const_cast<ModelDev&>(m), st);
        if (rc) return rc;
        oz = oz64_sum_pays(nk * (1 + nproj), (int64_t)N * N, m.hop_K,
                                       (double)nk * N * N * (m.hop_K * (nproj > 0 ? 8 + 2 * nproj : 4) + 60));
        if (oz && (rc = ensure_table_image(const_cast<ModelDev&>(m), st))) return rc;
        oz = oz && m.oz_img;
    }
    int rc = TBG_OK;
    if (oz) {
        rc = fourier_oz64(m, st, nk, k_d, gauge, nproj, dirs_d, H, V, ldH, ldV, status_d);
        if (rc != TBG_E_OOM) return rc;
        rc = TBG_OK;  // the direct form needs no scratch
    }
    // H together with up to 3 projections per pass
    for (int p0 = 0; rc == TBG_OK && (p0 < nproj || p0 == 0); p0 += 3) {
        const double* w = dirs_d + (int64_t)p0 * m.dim;
        zc* Ho = p0 == 0 ? H : nullptr;
        zc* Vo = V ? V + (int64_t)p0 * N * N : nullptr;
        switch (std::min(3, nproj - p0)) {
            case 0: rc = launch_few<0>(st, m, nk, k_d, w, gauge, Ho, ldH, Vo, ldV); break;
            case 1: rc = launch_few<1>(st, m, nk, k_d, w, gauge, Ho, ldH, Vo, ldV); break;
            case 2: rc = launch_few<2>(st, m, nk, k_d, w, gauge, Ho, ldH, Vo, ldV); break;
            default: rc = launch_few<3>(st, m, nk, k_d, w, gauge, Ho, ldH, Vo, ldV);
        }
    }
    return rc;
}

int rmatrix_term(const ModelDev& m, cudaStream_t st, int64_t nk, const double* k_d, int gauge, int nproj,
                 const double* dirs_d, const zc* H, zc* V, int* status_d) {
    if (m.n_rmat <= 0 || nk <= 0 || nproj <= 0) return TBG_OK;
    KTimer kt(st, "rmatrix_term");
    const int N = (int)m.nsta, nR = (int)m.nR, nr = (int)m.n_rmat;
    const int64_t NN = (int64_t)N * N;
    // the same forms as fourier_direct's for the sums, as the rotation's for the products
    const bool oz = oz64_sum_pays(nk, NN, nr, (double)nk * NN * nr * 4.0), tc = N > kCommSmemMaxN;
    const int step = oz ? 2 : 1;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) & ~size_t(255);
        return o;
    };
    const size_t o_ph = take(sizeof(zc) * nk * nR), o_orb = take(sizeof(zc) * nk * N);
    const size_t o_tab = take(sizeof(zc) * step * nr * NN), o_A = take(sizeof(zc) * nk * NN);
    const size_t o_eb = take(oz ? sizeof(int) * NN : 0), o_ea = take(oz ? sizeof(int) * nk : 0);
    const size_t o_tim = take(oz ? oz64_table_image_bytes(nr, NN) : 0), o_aim = take(oz ? oz64_row_image_bytes(nk, nr) : 0);
    const size_t o_ex = take(tc ? sizeof(int) * 4 * nk * N : 0);
    unsigned char* buf = nullptr;
    TBG_CUDA(cudaMallocAsync(&buf, off, st));
    zc* ph = reinterpret_cast<zc*>(buf + o_ph);
    zc* orbph = reinterpret_cast<zc*>(buf + o_orb);
    zc* tab = reinterpret_cast<zc*>(buf + o_tab);
    zc* A = reinterpret_cast<zc*>(buf + o_A);
    int *EB = reinterpret_cast<int*>(buf + o_eb), *EA = reinterpret_cast<int*>(buf + o_ea);
    int *hr = reinterpret_cast<int*>(buf + o_ex), *hc = hr + nk * N, *ar = hc + nk * N, *ac = ar + nk * N;
    int rc = TBG_OK;
    auto launched = [&](const char* what) {
        count_launch();
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess && !rc) rc = cuda_error(e, what);
        return rc;
    };
    const unsigned wide = 65535 * 8;
    phases_kernel<<<(unsigned)std::min<int64_t>((nk * (int64_t)(nR + N) + 255) / 256, wide), 256, 0, st>>>(
        nk, m.dim, k_d, nR, m.hamR_d, N, m.tau_d, ph, orbph);
    launched("phases_kernel");
    if (tc && !rc) {
        rc = oz64_row_exps(st, nk, N, N, H, N, NN, hr);
        if (!rc) rc = oz64_col_exps(st, nk, N, N, H, N, NN, hc);
    }
    for (int p = 0; rc == TBG_OK && p < nproj; ++p) {
        rmat_combine_kernel<<<(unsigned)std::min<int64_t>((nr * NN + 255) / 256, wide), 256, 0, st>>>(
            nr, m.dim, N, dirs_d + (int64_t)p * m.dim, m.rmatrix, step, tab);
        if (launched("rmat_combine_kernel")) break;
        // A = sum_{r < n_rmat} u(k,r) rm_p[r]   (lattice gauge)
        if (oz) {
            rc = oz64_table_image(st, nr, NN, tab, nullptr, EB, buf + o_tim);
            if (!rc) rc = oz64_table_product(st, nk, NN, nr, ph, nR, EB, buf + o_tim, A, EA, buf + o_aim, status_d);
        } else {
            rc = launch_gemm(st, nk, nr, nR, N, ph, tab, A);
        }
        if (rc) break;
        zc* Vp = V + (int64_t)p * NN;
        const int64_t ldV = (int64_t)nproj * NN;
        if (!tc) {
            const size_t smem = 2 * sizeof(zc) * NN;
            commutator_smem_kernel<<<(unsigned)std::min<int64_t>(nk, 152LL * 64), fit_threads((int)NN), smem, st>>>(
                N, nk, H, A, orbph, gauge, Vp, ldV);
            launched("commutator_smem_kernel");
            continue;
        }
        rmat_gauge_kernel<<<(unsigned)std::min<int64_t>((nk * NN + 255) / 256, wide), 256, 0, st>>>(nk, N, gauge, orbph,
                                                                                                   A);
        if (launched("rmat_gauge_kernel")) break;
        // V += H (iA) - (iA) H
        if ((rc = oz64_row_exps(st, nk, N, N, A, N, NN, ar)) || (rc = oz64_col_exps(st, nk, N, N, A, N, NN, ac))) break;
        rc = oz64_gemm(st, nk, N, N, N, {H, N, 1, NN, 0, hr}, {A, 1, N, NN, 0, ac}, Vp, N, ldV, 1, status_d);
        if (!rc) rc = oz64_gemm(st, nk, N, N, N, {A, N, 1, NN, 0, ar}, {H, 1, N, NN, 0, hc}, Vp, N, ldV, -1, status_d);
    }
    cudaFreeAsync(buf, st);
    return rc;
}

}  // namespace tbg
