// Fused path for small models (nsta <= 8): one thread per k-point runs the
// whole of berry_curvature_at_impl (src/response/traits.rs:160-200) in
// registers / local memory, FP64:
//   H, V_0, V_1 by the Fourier sum over R with the tau term (lattice gauge)
//   (src/velocity.rs:538-622), optional spin dressing (traits.rs:170-175),
//   eigenpairs by cyclic complex Jacobi, U^H V U, Omega_n (and optionally
//   the quantum metric, src/quantum_geometry.rs:160-187), and the
//   occupation sums per chemical potential (linear/mod.rs:204-223).
// For nsta <= 8 the per-k work is a few thousand flops, so one launch covers
// tens of thousands of k-points and the batched per-matrix kernels would be
// dominated by launch and synchronisation overhead.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "tbgpu_internal.cuh"

namespace tbg {
namespace {

__device__ __forceinline__ double fermi_s(double e, double mu, double width) {
    if (width == 0.0) return (e < mu) ? 1.0 : ((e > mu) ? 0.0 : 0.5);
    const double x = (e - mu) / width;
    if (x > 50.0) return 0.0;
    if (x < -50.0) return 1.0;
    return 1.0 / (1.0 + exp(x));
}

// The rotation that annihilates a_pq: tan 2 theta = 2 |a_pq| / (a_pp - a_qq), theta
// in [0, pi / 2], and a_pq / |a_pq|.  Half-angle formulas over reciprocal square
// roots, the larger of cosine and sine first (no cancellation): a fraction of the
// FP64 instructions of sqrt, division, atan2 and sincos.
__device__ __forceinline__ void jacobi_rotation(zc apq, double m2, double d, zc& ph, double& cs, double& sn) {
    const double rm = rsqrt(m2), mag = m2 * rm;
    ph = mk(apq.re * rm, apq.im * rm);
    const double rh = rsqrt(fma(d, d, 4.0 * m2)), q = fma(0.5 * fabs(d), rh, 0.5);
    const double rb = rsqrt(q), big = q * rb, little = mag * rh * rb;
    cs = d >= 0.0 ? big : little;
    sn = d >= 0.0 ? little : big;
}

// Cyclic complex Jacobi on the Hermitian NM x NM (active N) matrix A; W gets
// the eigenvectors in columns.  Rotation: G = diag(1, e^{-i phi}) [[c,-s],[s,c]]
// with e^{i phi} = a_pq / |a_pq|.
template <int NM, bool WANT_W>
__device__ __forceinline__ void jacobi(int N, zc (&A)[NM][NM], zc (&W)[NM][NM]) {
    if (WANT_W)
#pragma unroll
        for (int i = 0; i < NM; ++i)
#pragma unroll
            for (int j = 0; j < NM; ++j) W[i][j] = mk(i == j ? 1.0 : 0.0, 0.0);
#pragma unroll 1
    for (int sweep = 0; sweep < 40; ++sweep) {
        double off = 0.0, dia = 0.0;
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
            for (int j = 0; j < N; ++j) {
                if (i != j)
                    off += abs2(A[i][j]);
                else
                    dia += abs2(A[i][j]);
            }
        if (off <= 1e-32 * dia || off == 0.0) break;
#pragma unroll
        for (int p = 0; p < N - 1; ++p)
#pragma unroll
            for (int q = p + 1; q < N; ++q) {
                const zc apq = A[p][q];
                const double m2 = abs2(apq);
                if (m2 == 0.0) continue;
                zc ph;
                double sn, cs;
                jacobi_rotation(apq, m2, A[p][p].re - A[q][q].re, ph, cs, sn);
                const zc emi = conj(ph);
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const zc akp = A[k][p], akq = emi * A[k][q];
                    A[k][p] = cs * akp + sn * akq;
                    A[k][q] = cs * akq - sn * akp;
                }
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const zc apk = A[p][k], aqk = ph * A[q][k];
                    A[p][k] = cs * apk + sn * aqk;
                    A[q][k] = cs * aqk - sn * apk;
                }
                A[p][q] = mk(0.0, 0.0);
                A[q][p] = mk(0.0, 0.0);
                A[p][p].im = 0.0;
                A[q][q].im = 0.0;
                if (WANT_W)
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        const zc wkp = W[k][p], wkq = emi * W[k][q];
                        W[k][p] = cs * wkp + sn * wkq;
                        W[k][q] = cs * wkq - sn * wkp;
                    }
            }
    }
}

// Ascending order of E, f(i) exchanging what goes with entries i and i + 1 (bubble
// network: constant indices keep the arrays in registers; ties stay as they are).
template <int NM, typename F>
__device__ __forceinline__ void sort_bands(int N, double (&E)[NM], F f) {
#pragma unroll
    for (int a = N - 1; a > 0; --a)
#pragma unroll
        for (int i = 0; i < a; ++i)
            if (E[i] > E[i + 1]) {
                const double t = E[i];
                E[i] = E[i + 1];
                E[i + 1] = t;
                f(i);
            }
}
__device__ __forceinline__ void swap_d(double& a, double& b) {
    const double t = a;
    a = b;
    b = t;
}

// z^r for |z| = 1 (r uniform over the warp: no divergence)
__device__ __forceinline__ void times_power(zc& u, bool& one, zc z, int r) {
    if (r == 0) return;
    if (r < 0) z.im = -z.im;
    for (unsigned n = (unsigned)(r < 0 ? -r : r);;) {
        if (n & 1) {
            u = one ? z : u * z;
            one = false;
        }
        n >>= 1;
        if (!n) break;
        z = z * z;
    }
}

// e^{2 pi i i_d / n_d} along each axis of a mesh, axes one after the other.
__global__ void mesh_phase_kernel(int64_t n0, int64_t n1, int64_t n2, zc* __restrict__ z) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n0 + n1 + n2;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t n = t < n0 ? n0 : (t < n0 + n1 ? n1 : n2), i = t < n0 ? t : (t < n0 + n1 ? t - n0 : t - n0 - n1);
        double sn, cs;
        sincospi(2.0 * ((double)i / (double)n), &sn, &cs);
        z[t] = mk(cs, sn);
    }
}

// VALS: band energies only (E_out); no velocities, eigenvectors or curvature.
// EXACT: N == NM, known to the compiler, so the matrices stay in registers (they
// are indexed, in local memory, otherwise).  The FP64 pipe is the bound, so the
// phase of R comes from the e^{2 pi i k_d} by R_d-fold products, one sincospi per
// axis and k-point (none with ztab, the mesh's table) instead of one sincos per R,
// and energies of two bands from the quadratic formula: 10^6 k-points of the
// honeycomb model 0.92 -> 0.185 ms, 961 of the Haldane model's curvature 62 -> 35 us.
template <int NM, bool VALS, bool EXACT>
__global__ void __launch_bounds__(64) small_fused_kernel(
    int Nrt, int norb, int dim, int nR, int64_t nk, const double* __restrict__ klist, int64_t k0, int64_t n0,
    int64_t n1, int64_t n2, const zc* __restrict__ ztab, const zc* __restrict__ ham, const int* __restrict__ hamR,
    const double* __restrict__ Rcart, const double* __restrict__ taucart, const double* __restrict__ dirs, int spin,
    double eta, int nmu, const double* __restrict__ mu, double width, double* __restrict__ Om_out,
    double* __restrict__ E_out, double* __restrict__ S_out, double* __restrict__ Met_out, double* __restrict__ SM_out) {
    const int N = EXACT ? NM : Nrt;
    // the model in shared memory, all of it requested at once
    extern __shared__ __align__(16) unsigned char small_smem[];
    zc* s_ham = reinterpret_cast<zc*>(small_smem);                      // (nR, N, N)
    double* s_c = reinterpret_cast<double*>(s_ham + (int64_t)nR * N * N);  // (nR, 2) w . R
    double* s_tau = s_c + 2 * nR;                                       // (N, 2) w . tau
    int* s_R = reinterpret_cast<int*>(s_tau + 2 * N);                   // (nR, 3)
    for (int i = threadIdx.x; i < nR * N * N; i += blockDim.x) s_ham[i] = ham[i];
    for (int i = threadIdx.x; i < 3 * nR; i += blockDim.x) s_R[i] = hamR[i];
    if (!VALS) {
        auto along = [&](int d, const double* v) {  // w_d . v
            const double* w = dirs + d * dim;
            double c = w[0] * v[0];
            if (dim > 1) c += w[1] * v[1];
            if (dim > 2) c += w[2] * v[2];
            return c;
        };
        for (int i = threadIdx.x; i < 2 * nR; i += blockDim.x) s_c[i] = along(i & 1, Rcart + 3 * (i >> 1));
        for (int i = threadIdx.x; i < 2 * N; i += blockDim.x) s_tau[i] = along(i & 1, taucart + 3 * (i >> 1));
    }
    __syncthreads();
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nk) return;
    double kv[3] = {0.0, 0.0, 0.0}, nan = 0.0;  // nan: NaN unless k is finite, also where no R reaches along an axis
    zc z[3];
    if (klist) {
        for (int d = 0; d < dim; ++d) {
            kv[d] = klist[t * dim + d];
            nan = fma(0.0, kv[d], nan);
        }
    } else {
        const int64_t idx = k0 + t;  // gen_kmesh order (src/kpoints.rs:49-87), n1 = n2 = 1 beyond dim
        int64_t i0, i1, i2;
        if (n0 * n1 * n2 <= 0xffffffffll) {  // 32-bit divisions
            const unsigned u = (unsigned)idx, q = u / (unsigned)n2;
            i2 = u - q * (unsigned)n2;
            i0 = q / (unsigned)n1;
            i1 = q - (unsigned)i0 * (unsigned)n1;
        } else {
            i2 = idx % n2;
            i1 = (idx / n2) % n1;
            i0 = idx / (n1 * n2);
        }
        if (!VALS || !ztab) {
            kv[0] = (double)i0 / (double)n0;
            if (dim > 1) kv[1] = (double)i1 / (double)n1;
            if (dim > 2) kv[2] = (double)i2 / (double)n2;
        }
        if (ztab) {
            z[0] = ztab[i0];
            z[1] = ztab[n0 + i1];
            z[2] = ztab[n0 + n1 + i2];
        }
    }
    if (!ztab) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            z[d] = mk(1.0, 0.0);
            if (d < dim) sincospi(2.0 * kv[d], &z[d].im, &z[d].re);
            z[d].re += nan;
        }
    }
    zc H[NM][NM], V0[NM][NM], V1[NM][NM];
#pragma unroll
    for (int i = 0; i < NM; ++i)
#pragma unroll
        for (int j = 0; j < NM; ++j) H[i][j] = V0[i][j] = V1[i][j] = mk(0.0, 0.0);
    for (int r = 0; r < nR; ++r) {
        const int* R = s_R + 3 * r;
        zc u = mk(1.0 + nan, 0.0);
        bool one = true;
        times_power(u, one, z[0], R[0]);
        if (dim > 1) times_power(u, one, z[1], R[1]);
        if (dim > 2) times_power(u, one, z[2], R[2]);
        const zc* hr = s_ham + r * N * N;
        if (VALS) {
#pragma unroll
            for (int i = 0; i < N; ++i)
#pragma unroll
                for (int j = i; j < N; ++j) {  // upper triangle
                    const zc h = hr[i * N + j];
                    H[i][j].re = fma(u.re, h.re, fma(-u.im, h.im, H[i][j].re));
                    if (j > i) H[i][j].im = fma(u.re, h.im, fma(u.im, h.re, H[i][j].im));
                }
            continue;
        }
        const double c0 = s_c[2 * r], c1 = s_c[2 * r + 1];
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const zc tt = u * hr[i * N + j];
                H[i][j] = H[i][j] + tt;
                // i c t
                V0[i][j] = mk(fma(-c0, tt.im, V0[i][j].re), fma(c0, tt.re, V0[i][j].im));
                V1[i][j] = mk(fma(-c1, tt.im, V1[i][j].re), fma(c1, tt.re, V1[i][j].im));
            }
    }
    if (VALS) {
        double E[NM];
        if constexpr (EXACT && NM == 2) {
            const double a = H[0][0].re, b = H[1][1].re, off = 2.0 * abs2(H[0][1]);
            E[0] = a > b ? b : a;
            E[1] = a > b ? a : b;
            // coupled above the rounding of the diagonal, by the test of jacobi() (its squares
            // out of range leave the diagonal as well)
            if (!(off <= 1e-32 * fma(a, a, b * b) || off == 0.0)) {
                const double m = 0.5 * (a + b), d = 0.5 * (a - b), h = sqrt(fma(d, d, 0.5 * off));
                E[0] = m - h;
                E[1] = m + h;
            }
        } else {
#pragma unroll
            for (int i = 1; i < N; ++i)
#pragma unroll
                for (int j = 0; j < i; ++j) H[i][j] = conj(H[j][i]);
            jacobi<NM, false>(N, H, V0);
#pragma unroll
            for (int i = 0; i < N; ++i) E[i] = H[i][i].re;
            sort_bands<NM>(N, E, [](int) {});
        }
#pragma unroll
        for (int i = 0; i < N; ++i) E_out[t * N + i] = E[i];
        return;
    }
    // tau term.  The Atom gauge's phases conj(phi_m) phi_n are a diagonal unitary
    // similarity of H and the velocities (one phase per orbital, both spins): E, Omega
    // and the metric are the same without them.
#pragma unroll
    for (int m = 0; m < N; ++m)
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const zc hl = H[m][n];
            const double d0 = s_tau[2 * n] - s_tau[2 * m], d1 = s_tau[2 * n + 1] - s_tau[2 * m + 1];
            V0[m][n] = V0[m][n] + mk(-d0 * hl.im, d0 * hl.re);
            V1[m][n] = V1[m][n] + mk(-d1 * hl.im, d1 * hl.re);
        }
    if (spin >= 0) {  // J = 1/2 (S V0 + V0 S), S = sigma (x) I / 2
        zc J[NM][NM];
        for (int i = 0; i < N; ++i)
            for (int j = 0; j < N; ++j) {
                auto ent = [&](int x, int& px, zc& sx) {
                    const bool up = x < norb;
                    if (spin == TBG_SPIN_X) {
                        px = up ? x + norb : x - norb;
                        sx = mk(0.5, 0.0);
                    } else if (spin == TBG_SPIN_Y) {
                        px = up ? x + norb : x - norb;
                        sx = up ? mk(0.0, -0.5) : mk(0.0, 0.5);
                    } else {
                        px = x;
                        sx = up ? mk(0.5, 0.0) : mk(-0.5, 0.0);
                    }
                };
                int pi, pj, ppj;
                zc si, sj;
                ent(i, pi, si);
                ent(j, pj, sj);
                ent(pj, ppj, sj);  // (V S)[i][j] = V[i][pi(j)] S[pi(j)][j]
                zc vi = V0[0][0], vj = V0[0][0];  // V0[pi][j], V0[i][pj] by constant indices
#pragma unroll
                for (int x = 0; x < N; ++x) {
                    if (x == pi) vi = V0[x][j];
                    if (x == pj) vj = V0[i][x];
                }
                const zc a = si * vi;
                const zc c = vj * sj;
                J[i][j] = mk(0.5 * (a.re + c.re), 0.5 * (a.im + c.im));
            }
#pragma unroll
        for (int i = 0; i < N; ++i)
#pragma unroll
            for (int j = 0; j < N; ++j) V0[i][j] = J[i][j];
    }
    zc W[NM][NM];
    jacobi<NM, true>(N, H, W);
    double E[NM];
#pragma unroll
    for (int i = 0; i < N; ++i) E[i] = H[i][i].re;
    // band-basis velocities B = W^H V W
    zc Bx[NM][NM], By[NM][NM];
#pragma unroll
    for (int b = 0; b < N; ++b) {
        zc tx[NM], ty[NM];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            tx[i] = ty[i] = mk(0.0, 0.0);
#pragma unroll
            for (int j = 0; j < N; ++j) {
                fma_cx(tx[i], V0[i][j], W[j][b]);
                fma_cx(ty[i], V1[i][j], W[j][b]);
            }
        }
#pragma unroll
        for (int a = 0; a < N; ++a) {
            zc sx = mk(0.0, 0.0), sy = mk(0.0, 0.0);
#pragma unroll
            for (int i = 0; i < N; ++i) {
                fma_cjx(sx, W[i][a], tx[i]);
                fma_cjx(sy, W[i][a], ty[i]);
            }
            Bx[a][b] = sx;
            By[a][b] = sy;
        }
    }
    const double eta2 = eta * eta;
    const bool met = Met_out || SM_out;
    double Om[NM], G[NM];
#pragma unroll
    for (int a = 0; a < N; ++a) {
        double v = 0.0, g = 0.0;
#pragma unroll
        for (int b = 0; b < N; ++b) {
            if (a == b) continue;
            const double im = Bx[a][b].re * By[b][a].im + Bx[a][b].im * By[b][a].re;
            const double de = E[a] - E[b];
            const double den = de * de + eta2;
            v += -2.0 * im / den;
            if (met) g += (Bx[a][b].re * By[b][a].re - Bx[a][b].im * By[b][a].im) / den;
        }
        Om[a] = v;
        G[a] = g;
    }
    sort_bands<NM>(N, E, [&](int i) {
        swap_d(Om[i], Om[i + 1]);
        swap_d(G[i], G[i + 1]);
    });
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (Om_out) Om_out[t * N + i] = Om[i];
        if (E_out) E_out[t * N + i] = E[i];
        if (Met_out) Met_out[t * N + i] = G[i];
    }
    if (S_out) {
        for (int j = 0; j < nmu; ++j) {
            double s = 0.0, sg = 0.0;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const double f = fermi_s(E[i], mu[j], width);
                s += Om[i] * f;
                sg += G[i] * f;
            }
            S_out[t * nmu + j] = s;
            if (SM_out) SM_out[t * nmu + j] = sg;
        }
    }
}

// Eigenpairs of batched N x N (N <= 8) Hermitian matrices, one thread per
// matrix: cyclic Jacobi in registers, E ascending, U with the eigenvectors in
// columns (row-major, the layout of the batched solver); U may be null.
// Non-finite input sets bit 0 of *status, as the batched solver does.
template <int NM, bool EXACT>
__global__ void __launch_bounds__(64) small_eig_kernel(int Nrt, int64_t batch, const zc* __restrict__ H,
                                                      double* __restrict__ E_out, zc* __restrict__ U_out,
                                                      int* __restrict__ status) {
    const int N = EXACT ? NM : Nrt;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= batch) return;
    const int64_t NN = (int64_t)N * N;
    zc A[NM][NM], W[NM][NM];
#pragma unroll
    for (int i = 0; i < NM; ++i)
#pragma unroll
        for (int j = 0; j < NM; ++j) A[i][j] = (i < N && j < N) ? H[t * NN + i * N + j] : mk(0.0, 0.0);
    jacobi<NM, true>(N, A, W);
    double E[NM];
    bool bad = false;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        E[i] = A[i][i].re;
        bad = bad || !isfinite(E[i]);
    }
    if (bad && status) atomicOr(status, 1);
    sort_bands<NM>(N, E, [&](int i) {
#pragma unroll
        for (int r = 0; r < N; ++r) {
            const zc w = W[r][i];
            W[r][i] = W[r][i + 1];
            W[r][i + 1] = w;
        }
    });
#pragma unroll
    for (int i = 0; i < N; ++i) E_out[t * N + i] = E[i];
    if (U_out)
#pragma unroll
        for (int r = 0; r < N; ++r)
#pragma unroll
            for (int c = 0; c < N; ++c) U_out[t * NN + r * N + c] = W[r][c];
}

}  // namespace

int small_fused(const ModelDev& m, cudaStream_t st, int64_t nk, const double* klist_d, int64_t k0,
                const int64_t* kmesh, const double* dirs_d, int spin, double eta, int nmu, const double* mu_d,
                double width, double* Om, double* E, double* S, double* Met, double* SM) {
    if (nk <= 0) return TBG_OK;
    const int N = (int)m.nsta;
    const int64_t n0 = kmesh ? kmesh[0] : 1, n1 = (kmesh && m.dim > 1) ? kmesh[1] : 1,
                  n2 = (kmesh && m.dim > 2) ? kmesh[2] : 1;
    KTimer kt(st, "small_fused_kernel");
    // energies only when nothing else is asked for
    const bool vals = !Om && !S && !Met && !SM;
    if (vals && !E) return TBG_OK;
    // a table of the mesh's phases once it saves more than its launch takes
    zc* ztab = nullptr;
    if (kmesh && !klist_d && nk >= 65536) {
        const int64_t n = n0 + n1 + n2;
        TBG_CUDA(cudaMallocAsync(&ztab, sizeof(zc) * n, st));
        mesh_phase_kernel<<<(unsigned)std::min<int64_t>((n + 127) / 128, 152LL * 8), 128, 0, st>>>(n0, n1, n2, ztab);
        TBG_LAUNCHED("mesh_phase_kernel");
    }
    // one warp per block while that spreads a small mesh over more SMs
    const int thr = nk <= 152 * 64 ? 32 : 64;
    const unsigned blocks = (unsigned)((nk + thr - 1) / thr);
    const size_t smem = sizeof(zc) * m.nR * N * N + sizeof(double) * (2 * m.nR + 2 * N) + sizeof(int) * 3 * m.nR;
#define SMALL_LAUNCH(NM, EX)                                                                                         \
    do {                                                                                                             \
        if (vals)                                                                                                    \
            small_fused_kernel<NM, true, EX><<<blocks, thr, smem, st>>>(                                             \
                N, (int)m.norb, m.dim, (int)m.nR, nk, klist_d, k0, n0, n1, n2, ztab, m.ham, m.hamR_d, m.Rcart_d,    \
                m.taucart_d, dirs_d, spin, eta, nmu, mu_d, width, Om, E, S, Met, SM);                      \
        else                                                                                                         \
            small_fused_kernel<NM, false, EX><<<blocks, thr, smem, st>>>(                                            \
                N, (int)m.norb, m.dim, (int)m.nR, nk, klist_d, k0, n0, n1, n2, ztab, m.ham, m.hamR_d, m.Rcart_d,    \
                m.taucart_d, dirs_d, spin, eta, nmu, mu_d, width, Om, E, S, Met, SM);                      \
    } while (0)
    if (N == 2)
        SMALL_LAUNCH(2, true);
    else if (N <= 2)
        SMALL_LAUNCH(2, false);
    else if (N == 3)
        SMALL_LAUNCH(3, true);
    else if (N == 4)
        SMALL_LAUNCH(4, true);
    else if (N <= 8)
        SMALL_LAUNCH(8, false);
    else
        return set_error(TBG_E_UNSUPPORTED, "small_fused: nsta > 8");
#undef SMALL_LAUNCH
    if (ztab) cudaFreeAsync(ztab, st);
    TBG_LAUNCHED("small_fused_kernel");
    return TBG_OK;
}

}  // namespace tbg

namespace tbg {
int eig_small(cudaStream_t st, int N, int64_t batch, const zc* H, double* E, zc* U, int* status) {
    if (batch <= 0) return TBG_OK;
    const int thr = batch <= 152 * 64 ? 32 : 64;
    const unsigned blocks = (unsigned)((batch + thr - 1) / thr);
    if (N == 2)
        small_eig_kernel<2, true><<<blocks, thr, 0, st>>>(N, batch, H, E, U, status);
    else if (N == 3)
        small_eig_kernel<3, true><<<blocks, thr, 0, st>>>(N, batch, H, E, U, status);
    else if (N == 4)
        small_eig_kernel<4, true><<<blocks, thr, 0, st>>>(N, batch, H, E, U, status);
    else
        small_eig_kernel<8, false><<<blocks, thr, 0, st>>>(N, batch, H, E, U, status);
    TBG_LAUNCHED("small_eig_kernel");
    return TBG_OK;
}
}  // namespace tbg

namespace tbg {
namespace {

// Warp-per-matrix cyclic complex Jacobi (FP64) for kSmallMaxN < N <= 32.  The
// matrix (upper triangle read, as by the Householder solver) and the
// eigenvector accumulator sit in shared memory; the N(N-1)/2 rotations of a
// sweep run as N-1 rounds of N/2 disjoint pairs (circle-method round robin:
// the last index fixed, the others turning), and in each round every 2x2 block
// (rows of pair I, columns of pair J) becomes G_I^H B G_J, one block per lane,
// with the rotation of the one-thread solver above:
//   G = [[c, -s], [s e^{-i phi}, c e^{-i phi}]],  e^{i phi} = a_pq / |a_pq|,
//   tan 2 theta = 2 |a_pq| / (a_pp - a_qq), |theta| <= pi/4
// (the small angle: with every pair of a round rotated at once, the near-swaps
// that the angle up to pi/2 allows make the rounds cycle without converging).
// Sweeps stop when the off-diagonal norm is 1e-15 of the diagonal's: blocks
// off the diagonal only reach rounding level, never exact zeros (at most 40).
template <int NP>
struct JacobiWarp {
    zc A[NP * NP];
    zc V[NP * NP];
    zc em[NP / 2];
    double c[NP / 2], s[NP / 2];
    int p[NP / 2], q[NP / 2], rank[NP];
};

template <int NP>
__global__ void __launch_bounds__(64) jacobi_warp_kernel(int N, int64_t batch, const zc* __restrict__ H,
                                                         double* __restrict__ E_out, zc* __restrict__ U_out,
                                                         int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char jacobi_smem[];
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    JacobiWarp<NP>& w = reinterpret_cast<JacobiWarp<NP>*>(jacobi_smem)[threadIdx.x >> 5];
    const int n2 = (N + 1) & ~1, nh = n2 / 2, NN = N * N;
    for (int64_t m = blockIdx.x * (int64_t)nw + (threadIdx.x >> 5); m < batch; m += (int64_t)gridDim.x * nw) {
        const zc* h = H + m * NN;
        for (int e = lane; e < n2 * n2; e += 32) {
            const int i = e / n2, j = e - i * n2;
            zc a = mk(0.0, 0.0);
            if (i < N && j < N) a = j >= i ? h[i * N + j] : conj(h[j * N + i]);
            if (i == j) a.im = 0.0;
            w.A[i * NP + j] = a;
            w.V[i * NP + j] = mk(i == j ? 1.0 : 0.0, 0.0);
        }
        __syncwarp();
        for (int sweep = 0; sweep < 40; ++sweep) {
            double off = 0.0, dia = 0.0;
            for (int e = lane; e < n2 * n2; e += 32) {
                const int i = e / n2, j = e - i * n2;
                const double v = abs2(w.A[i * NP + j]);
                if (i == j)
                    dia += v;
                else
                    off += v;
            }
            for (int o = 16; o; o >>= 1) {
                off += __shfl_xor_sync(0xffffffffu, off, o);
                dia += __shfl_xor_sync(0xffffffffu, dia, o);
            }
            if (off <= 1e-30 * dia || off == 0.0) break;  // warp-uniform
            for (int r = 0; r < n2 - 1; ++r) {
                if (lane < nh) {
                    const int p = lane == 0 ? r : (r + lane) % (n2 - 1);
                    const int q = lane == 0 ? n2 - 1 : (r - lane + n2 - 1) % (n2 - 1);
                    const zc apq = w.A[p * NP + q];
                    const double mag = sqrt(abs2(apq));
                    double sn = 0.0, cs = 1.0;
                    zc em = mk(1.0, 0.0);
                    if (mag > 0.0) {
                        em = mk(apq.re / mag, -apq.im / mag);
                        const double dl = w.A[p * NP + p].re - w.A[q * NP + q].re;
                        sincos(0.5 * atan2(copysign(2.0 * mag, dl), fabs(dl)), &sn, &cs);
                    }
                    w.p[lane] = p;
                    w.q[lane] = q;
                    w.c[lane] = cs;
                    w.s[lane] = sn;
                    w.em[lane] = em;
                }
                __syncwarp();
                for (int b = lane; b < nh * nh; b += 32) {
                    const int I = b / nh, J = b - I * nh;
                    const int pi = w.p[I], qi = w.q[I], pj = w.p[J], qj = w.q[J];
                    const double ci = w.c[I], si = w.s[I], cj = w.c[J], sj = w.s[J];
                    const zc ei = conj(w.em[I]), ej = w.em[J];
                    const zc b00 = w.A[pi * NP + pj], b01 = w.A[pi * NP + qj];
                    const zc b10 = w.A[qi * NP + pj], b11 = w.A[qi * NP + qj];
                    // columns: B G_J
                    const zc t01 = ej * b01, t11 = ej * b11;
                    const zc r00 = cj * b00 + sj * t01, r01 = cj * t01 - sj * b00;
                    const zc r10 = cj * b10 + sj * t11, r11 = cj * t11 - sj * b10;
                    // rows: G_I^H (B G_J)
                    const zc u10 = ei * r10, u11 = ei * r11;
                    zc a00 = ci * r00 + si * u10, a01 = ci * r01 + si * u11;
                    zc a10 = ci * u10 - si * r00, a11 = ci * u11 - si * r01;
                    if (I == J) {
                        a00.im = 0.0;
                        a11.im = 0.0;
                        a01 = mk(0.0, 0.0);
                        a10 = mk(0.0, 0.0);
                    }
                    w.A[pi * NP + pj] = a00;
                    w.A[pi * NP + qj] = a01;
                    w.A[qi * NP + pj] = a10;
                    w.A[qi * NP + qj] = a11;
                }
                for (int e = lane; e < n2 * nh; e += 32) {
                    const int row = e / nh, J = e - row * nh;
                    const int pj = w.p[J], qj = w.q[J];
                    const double cj = w.c[J], sj = w.s[J];
                    const zc v0 = w.V[row * NP + pj], v1 = w.em[J] * w.V[row * NP + qj];
                    w.V[row * NP + pj] = cj * v0 + sj * v1;
                    w.V[row * NP + qj] = cj * v1 - sj * v0;
                }
                __syncwarp();
            }
        }
        // ascending order: rank of each diagonal entry, ties by index
        for (int i = lane; i < N; i += 32) {
            const double di = w.A[i * NP + i].re;
            int rk = 0;
            for (int j = 0; j < N; ++j) {
                const double dj = w.A[j * NP + j].re;
                rk += (dj < di) || (dj == di && j < i);
            }
            w.rank[i] = rk;
            E_out[m * N + rk] = di;
            if (!isfinite(di) && status) atomicOr(status, 1);
        }
        __syncwarp();
        if (U_out)
            for (int e = lane; e < NN; e += 32) {
                const int r = e / N, c = e - r * N;
                U_out[m * NN + r * N + w.rank[c]] = w.V[r * NP + c];
            }
        __syncwarp();
    }
}

template <int NP>
int launch_jacobi(cudaStream_t st, int N, int64_t batch, const zc* H, double* E, zc* U, int* status) {
    constexpr int kWarps = 2;
    const size_t smem = kWarps * sizeof(JacobiWarp<NP>);
    auto kern = jacobi_warp_kernel<NP>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_error(e, "jacobi_warp_kernel smem");
    int dev = 0, nsm = 0, perSM = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, kern, 32 * kWarps, smem);
    if (e != cudaSuccess || perSM < 1) perSM = 1;
    const int64_t grid = std::min<int64_t>((int64_t)nsm * perSM, (batch + kWarps - 1) / kWarps);
    KTimer kt(st, "jacobi_warp_kernel");
    kern<<<(unsigned)grid, 32 * kWarps, smem, st>>>(N, batch, H, E, U, status);
    TBG_LAUNCHED("jacobi_warp_kernel");
    return TBG_OK;
}

}  // namespace

int eig_jacobi(cudaStream_t st, int N, int64_t batch, const zc* H, double* E, zc* U, int* status) {
    if (batch <= 0) return TBG_OK;
    if (N < 2 || N > kJacobiMaxN) return set_error(TBG_E_UNSUPPORTED, "eig_jacobi: N outside [2, 32]");
    return N <= 16 ? launch_jacobi<16>(st, N, batch, H, E, U, status)
                   : launch_jacobi<32>(st, N, batch, H, E, U, status);
}

}  // namespace tbg
