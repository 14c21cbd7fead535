// FP64-accurate complex matrix products on the 5th-generation tensor cores.
//
// The part's FP64 pipe does about 1/64 of its FP32 rate, its BF16 tensor cores
// some 2000 times as much, so a product is run as exact digit products (error-free
// splitting after Ozaki, Ogita, Oishi and Rump 2012): a row of A (column of B)
// with |x| < 2^E is written on the grid 2^(E - 55) and cut into seven signed
// digits of eight bits, which BF16 holds exactly.  Digit pairs of level
// s + t <= 6 are kept (28 of 49), each level in an FP32 accumulator of its own: a
// sum of up to 512 products of two digits is below 2^23, and what the last levels
// may lose is below 2^-60 of the product's scale 2^(EA + EB).  The sums are put
// together as 64-bit integers (an FP64 addition costs as much as dozens of integer
// instructions here) and rounded once to FP64.  The tensor core truncates, so
// levels with different last places must not share an accumulator early: with
// levels 4 to 6 in one the error of a 128-term product was 300 x 2^-54 of the
// scale, against 10 x for an FP64 sum and 6.8 x now.
//
// CTA = 14 (13) warps, one output tile of 128 rows x 40 (32) complex columns:
//   warps 0..7    digits of A, thread = (row, 8 consecutive k); afterwards the
//                 epilogue, one TMEM lane = one row
//   next 5 (4)    digits of B, thread = (column, 8 consecutive k, component); for
//                 operands cut beforehand one thread copies the stage images of
//                 both with cp.async.bulk
//   last          allocates TMEM and issues the MMAs (M = 128, N = 80 or 64, K = 16)
// 40 columns fill 480 of the 512 TMEM columns with six accumulators (levels 5 and 6
// share the last), 32 columns 448 with seven.  Complex products keep the blocks
// -Im B, Re B, Im B, so [Re B; Im B] and [-Im B; Re B] are the same memory at two
// offsets.  Stage hand-off by mbarriers; every wait is bounded, as in the
// float-pair products (ozaki_tc.cu).
//
// 1024 products of 128 bands: one of the four of the rotation 13.8 -> 0.93 ms
// against 64 x 64 tiles on the FP64 pipe.

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "tbgpu_internal.cuh"
#include "tc_ptx.cuh"

namespace tbg {
namespace {

using namespace tc;

constexpr int S = 7;        // digits per value
constexpr int TM = 128;     // rows of a tile
constexpr int TK = 16;      // complex k per stage
constexpr int APLANE = TM * 2 * TK * 2;  // bytes of one digit plane of A in a stage
constexpr int A_THREADS = 256;
constexpr int kMaxK = 256;  // complex k that one launch keeps exact
enum { CPLX = 0, REALC = 1 };  // blocks of a B plane: complex product, or real coefficients (pre-cut)

template <int TNC>
struct Shape {
    static constexpr int NR = 2 * TNC;               // real columns of a tile
    static constexpr int NLEV = TNC > 32 ? 6 : 7;    // accumulators (level 6 with level 5 in the first case)
    static_assert(NLEV * NR <= 512, "TMEM columns");
    static constexpr int BLK = TNC * TK * 2;         // one block: TNC rows x 16 k
    static constexpr int B_THREADS = TNC * 4;        // (column, half of the 16 k, component)
    static constexpr int THREADS = A_THREADS + B_THREADS + 32;
    static constexpr uint32_t IDESC =
        (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NR >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
    static constexpr int bplane(int mode) { return (mode == REALC ? 4 : 3) * BLK; }
    static constexpr int stage(int mode) { return S * (APLANE + bplane(mode)); }
    static constexpr int EPI = 8 * 32 * 5 * 16;      // 4 columns of 32 rows per warp, rows padded to 5
    static constexpr int smem(int mode) { return 2 * stage(mode) + EPI + 1024; }
};

// byte offset of (row, half of the 16 k) in a block of core matrices (8 rows x 16 bytes)
__host__ __device__ __forceinline__ int blk_off(int row, int half) {
    return (((row >> 3) * 2 + half) << 7) + ((row & 7) << 4);
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(su32(bar))
                 : "memory");
}

// One MMA; COL: use of the collector buffer for A (0 none, 1 fill, 2 use, 3 last use).
template <int COL>
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
#define TBG_MMA(Q)                                                                                          \
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16" Q    \
                 " [%0], %1, %2, %3, p;\n\t}" ::"r"(d),                                                      \
                 "l"(a), "l"(b), "r"(idesc), "r"(acc)                                                        \
                 : "memory")
    if constexpr (COL == 1)
        TBG_MMA(".collector::a::fill");
    else if constexpr (COL == 2)
        TBG_MMA(".collector::a::use");
    else if constexpr (COL == 3)
        TBG_MMA(".collector::a::lastuse");
    else
        TBG_MMA("");
#undef TBG_MMA
}

// Biased exponent of |x| (0x7ff: NaN or Inf); a line's largest one, at least 1,
// is its exponent e: |x| < 2^(e - 1022).
__device__ __forceinline__ int exp_field(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
__device__ __forceinline__ int elem_exp(zc z) { return max(exp_field(z.re), exp_field(z.im)); }
constexpr int kNonFinite = 0x7ff;

// round(x 2^(55 - E)) + 128 sum_i 2^(8 i) (i < 6) for |x| < 2^E, e = E + 1022:
// bytes 0..5 are then the digits 6..1 plus 128, the rest digit 0.
__device__ __forceinline__ long long fixed55(double x, int e) {
    const int hi = __double2hiint(x);
    const int ex = (hi >> 20) & 0x7ff;
    const unsigned long long frac = ((unsigned long long)(unsigned)(hi & 0xfffff) << 32) | (unsigned)__double2loint(x);
    const unsigned long long M = frac | ((unsigned long long)(ex > 0) << 52);
    const int rs = min(max(e - max(ex, 1), 0), 57);
    const long long F = (long long)(((M << 2) + ((1ull << rs) >> 1)) >> rs);
    return (hi < 0 ? -F : F) + 0x0000808080808080ll;
}
// digit planes of 8 consecutive-k values: out[s] = 8 BF16, digit s times 2^(-8 s)
__device__ __forceinline__ uint32_t bf16x2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ void digits(long long F, float (&P)[S]) {
    const unsigned lo = (unsigned)F;
    const int hi = (int)(F >> 32);
    // 0x4B0000bb is 2^23 + bb
    constexpr float C = 8388736.f;  // 2^23 + 128
    P[0] = __fsub_rn(__int_as_float(0x4B000000 + ((hi >> 16) + 128)), C);
    P[1] = fmaf(__uint_as_float(__byte_perm(hi, 0x4B000000, 0x7441)), 0x1p-8f, -C * 0x1p-8f);
    P[2] = fmaf(__uint_as_float(__byte_perm(hi, 0x4B000000, 0x7440)), 0x1p-16f, -C * 0x1p-16f);
    P[3] = fmaf(__uint_as_float(__byte_perm(lo, 0x4B000000, 0x7443)), 0x1p-24f, -C * 0x1p-24f);
    P[4] = fmaf(__uint_as_float(__byte_perm(lo, 0x4B000000, 0x7442)), 0x1p-32f, -C * 0x1p-32f);
    P[5] = fmaf(__uint_as_float(__byte_perm(lo, 0x4B000000, 0x7441)), 0x1p-40f, -C * 0x1p-40f);
    P[6] = fmaf(__uint_as_float(__byte_perm(lo, 0x4B000000, 0x7440)), 0x1p-48f, -C * 0x1p-48f);
}
template <int PART>
__device__ __forceinline__ void planes(const zc (&v)[8], int e, bool neg, uint4 (&out)[S]) {
    uint32_t pk[S][4];
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        float P0[S], P1[S];
        digits(fixed55(PART ? v[i].im : v[i].re, e), P0);
        digits(fixed55(PART ? v[i + 1].im : v[i + 1].re, e), P1);
#pragma unroll
        for (int s = 0; s < S; ++s) pk[s][i >> 1] = bf16x2(P0[s], P1[s]);
    }
    const uint32_t m = neg ? 0x80008000u : 0u;
#pragma unroll
    for (int s = 0; s < S; ++s) out[s] = make_uint4(pk[s][0] ^ m, pk[s][1] ^ m, pk[s][2] ^ m, pk[s][3] ^ m);
}
__device__ __forceinline__ uint4 neg8(uint4 v) {
    const uint32_t m = 0x80008000u;
    return make_uint4(v.x ^ m, v.y ^ m, v.z ^ m, v.w ^ m);
}

__device__ __forceinline__ void ld8(const zc* p, int64_t stride, int nvalid, zc (&r)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        double2 t = make_double2(0.0, 0.0);
        if (i < nvalid) t = __ldg(reinterpret_cast<const double2*>(p + i * stride));
        r[i] = mk(t.x, t.y);
    }
}

// The level sums -> their FP64 value times 2^(ea + eb - 2058) (e - 1022 - 7 per operand).
template <int NLEV>
__device__ __forceinline__ double combine(const uint32_t (&a)[NLEV], int ea, int eb) {
    if (ea == kNonFinite || eb == kNonFinite) return __longlong_as_double(0x7ff8000000000000ll);
    float tail = __uint_as_float(a[5]);  // levels 5 and 6, below 2^-14
    if (NLEV == 7) tail += __uint_as_float(a[NLEV - 1]);
    const long long I = ((long long)__float2int_rn(__uint_as_float(a[0])) << 39) +
                        ((long long)__float2int_rn(__uint_as_float(a[1]) * 0x1p8f) << 31) +
                        ((long long)__float2int_rn(__uint_as_float(a[2]) * 0x1p16f) << 23) +
                        ((long long)__float2int_rn(__uint_as_float(a[3]) * 0x1p24f) << 15) +
                        ((long long)__float2int_rn(__uint_as_float(a[4]) * 0x1p32f) << 7) +
                        __float2int_rn(tail * 0x1p39f);
    if (I == 0) return 0.0;
    const unsigned long long sg = (unsigned long long)I & 0x8000000000000000ull;
    unsigned long long m = (unsigned long long)(I < 0 ? -I : I);
    const int lz = __clzll((long long)m);
    m <<= lz;
    unsigned long long q = m >> 11;
    q += (m >> 10) & 1ull & (((m & 0x3ffull) != 0) | (q & 1ull));  // to nearest, ties to even
    // I 2^-39 = q 2^(11 - lz - 39); biased exponent of the result's leading bit
    const int be = ea + eb - lz - 2058 + 1023 + 52 - 28;
    if (be > 0 && be < 0x7fe) return __longlong_as_double((long long)(sg | (((unsigned long long)(be - 1) << 52) + q)));
    const double r = scalbn((double)q, be - 1023 - 52);
    return sg ? -r : r;
}

// C (M x Nc per matrix) = / += / -= op(A) op(B).  Element (i, k) of op(A) is at
// A + b sA + i ai + k ak (conjugated when conjA), (k, j) of op(B) at
// B + b sB + k bk + j bj.  EA, EB: line exponents per (matrix, row) and (matrix,
// column).  PRE: A and B are stage images (row tile, nst_img stages) and (column
// tile, nst_img stages), from stage it0 on.
struct OzArgs {
    int M, Nc, K;
    const void* A;
    int64_t ai, ak, sA;
    const void* B;
    int64_t bk, bj, sB;
    int conjA, conjB;
    const int *EA, *EB;
    zc* C;
    int64_t ldc, sC;
    int mode;  // 0: store, 1: add, -1: subtract
    int* err;
    int wait_limit;
    int gx, gy, rows_fast;
    int64_t ntiles;
    int it0, nst_img;
};

struct Tile {
    int rt, ct;
    int64_t b;
};
__device__ __forceinline__ Tile tile_at(const OzArgs& p, int64_t L) {
    const int x = (int)(L % p.gx);
    const int64_t r = L / p.gx;
    const int y = (int)(r % p.gy);
    Tile t;
    t.b = r / p.gy;
    t.rt = p.rows_fast ? x : y;
    t.ct = p.rows_fast ? y : x;
    return t;
}
__device__ __forceinline__ int kleft(int K, int k) { return max(0, min(8, K - k)); }
// OR over the eight epilogue warps
__device__ __forceinline__ bool any256(bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.or.pred p, 1, 256, q;\n\tselp.u32 %0, 1, 0, "
        "p;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)v)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}

template <int TNC, bool PRE>
__global__ void __launch_bounds__(Shape<TNC>::THREADS, 1) oz64_kernel(OzArgs p) {
    using Sh = Shape<TNC>;
    constexpr int MODE = PRE ? REALC : CPLX;
    constexpr int BPLANE = Sh::bplane(MODE), ABYTES = S * APLANE, STAGE = Sh::stage(MODE), NR = Sh::NR, BLK = Sh::BLK;
    constexpr int NLEV = Sh::NLEV;
    extern __shared__ __align__(1024) unsigned char oz_smem[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)oz_smem + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bar_full[2], bar_empty[2], bar_done, bar_tmem;
    __shared__ uint32_t tmem_sh;
    __shared__ volatile int abort_sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int MMA_WARP = (A_THREADS + Sh::B_THREADS) / 32;
    const int nst = (p.K + TK - 1) / TK;
    const uint32_t sbase = su32(base);
    if (tid == 0) {
        const uint32_t nfull = PRE ? 1 : A_THREADS + Sh::B_THREADS;
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_full[i], nfull);
            mbar_init(&bar_empty[i], 1);
        }
        mbar_init(&bar_done, 1);
        mbar_init(&bar_tmem, 8);
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(su32(&tmem_sh))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_sh;
    int ndone = 0;  // tiles committed to bar_done

    if (warp == MMA_WARP) {
        if (lane == 0) {
            int tn = 0;
            for (int64_t L = blockIdx.x; L < p.ntiles; L += gridDim.x, ++tn) {
                if (tn > 0 && !mbar_wait(&bar_tmem, (tn - 1) & 1, &abort_sh, p.wait_limit)) {
                    abort_sh = 1;
                    break;
                }
                tc_fence_after();
                bool stop = false;
                for (int it = 0; it < nst; ++it) {
                    const int64_t gs = (int64_t)tn * nst + it;
                    const int bi = (int)(gs & 1);
                    if (!mbar_wait(&bar_full[bi], (uint32_t)((gs >> 1) & 1), &abort_sh, p.wait_limit)) {
                        abort_sh = 1;
                        stop = true;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = sbase + bi * STAGE, sb = sa + ABYTES;
#pragma unroll
                    for (int ks = 0; ks < 2; ++ks) {
                        // [Re B; Im B] then [-Im B; Re B] (blocks -Im, Re, Im), or the
                        // even then the odd rows of a real-coefficient table
                        const int boff = MODE == CPLX ? (ks == 0 ? BLK : 0) : ks * 2 * BLK;
#pragma unroll
                        for (int s = 0; s < S; ++s) {
#pragma unroll
                            for (int t = 0; t < S - s; ++t) {
                                const int lv = s + t < NLEV - 1 ? s + t : NLEV - 1;
                                const uint64_t ad = smem_desc(sa + s * APLANE + ks * (APLANE / 2), 128, 256);
                                const uint64_t bd = smem_desc(sb + t * BPLANE + boff, 128, 256);
                                const uint32_t acc = (it == 0 && ks == 0 && s == 0 && t < NLEV) ? 0u : 1u;
                                const uint32_t dst = tmem + (uint32_t)(lv * NR);
                                if (s == S - 1)
                                    mma<0>(dst, ad, bd, Sh::IDESC, acc);
                                else if (t == 0)
                                    mma<1>(dst, ad, bd, Sh::IDESC, acc);
                                else if (t == S - 1 - s)
                                    mma<3>(dst, ad, bd, Sh::IDESC, acc);
                                else
                                    mma<2>(dst, ad, bd, Sh::IDESC, acc);
                            }
                        }
                    }
                    umma_commit(&bar_empty[bi]);
                }
                umma_commit(&bar_done);
                ++ndone;
                if (stop) break;
            }
        }
        __syncwarp();
    } else if (tid < A_THREADS) {
        // rows of consecutive threads when op(A) is stored by columns, else pairs of threads per row
        const bool bycol = p.ak != 1;
        const int r = bycol ? (tid & 127) : (tid >> 1);
        const int g = bycol ? (tid >> 7) : (tid & 1);
        const int q = warp & 3, h = warp >> 2;
        const uint32_t lane_addr = tmem + ((uint32_t)(32 * q) << 16);
        double2* epi = reinterpret_cast<double2*>(base + 2 * STAGE) + warp * (32 * 5);
        zc nxt[8];
        auto load = [&](int64_t L, int it) {
            const Tile t = tile_at(p, L);
            const int gi = t.rt * TM + r, k = it * TK + 8 * g;
            ld8(static_cast<const zc*>(p.A) + t.b * p.sA + gi * p.ai + k * p.ak, p.ak, gi < p.M ? kleft(p.K, k) : 0, nxt);
        };
        if constexpr (!PRE)
            if (blockIdx.x < p.ntiles) load(blockIdx.x, 0);
        int tn = 0;
        for (int64_t L = blockIdx.x; L < p.ntiles; L += gridDim.x, ++tn) {
            const Tile t = tile_at(p, L);
            if constexpr (!PRE) {
                const int gi = t.rt * TM + r;
                const int e = gi < p.M ? p.EA[t.b * p.M + gi] : 1;
                for (int it = 0; it < nst; ++it) {
                    const int64_t gs = (int64_t)tn * nst + it;
                    const int bi = (int)(gs & 1);
                    zc cur[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) cur[i] = nxt[i];
                    if (it + 1 < nst)
                        load(L, it + 1);
                    else if (L + gridDim.x < p.ntiles)
                        load(L + gridDim.x, 0);
                    uint4 d[S];
                    const bool live = gi < p.M;
#pragma unroll
                    for (int s = 0; s < S; ++s) d[s] = make_uint4(0, 0, 0, 0);
                    if (live) planes<0>(cur, e, false, d);
                    if (gs >= 2 && !mbar_wait(&bar_empty[bi], (uint32_t)(((gs >> 1) - 1) & 1), &abort_sh, p.wait_limit)) {
                        abort_sh = 1;
                        break;
                    }
                    if (abort_sh) break;
                    const uint32_t sa = sbase + bi * STAGE + blk_off(r, g);
#pragma unroll
                    for (int s = 0; s < S; ++s) st_shared_v4(sa + s * APLANE, d[s]);
                    if (live) planes<1>(cur, e, p.conjA != 0, d);
#pragma unroll
                    for (int s = 0; s < S; ++s) st_shared_v4(sa + s * APLANE + APLANE / 2, d[s]);
                    fence_async_smem();
                    mbar_arrive(&bar_full[bi]);
                }
            }
            // epilogue: a tile is written whole or not at all
            bool bad = abort_sh != 0;
            if (!bad && !mbar_wait(&bar_done, tn & 1, &abort_sh, p.wait_limit)) {
                abort_sh = 1;
                bad = true;
            }
            if (any256(bad)) break;
            tc_fence_after();
            const int row = t.rt * TM + 32 * q + lane;
            const int ea = row < p.M ? p.EA[t.b * p.M + row] : 1;
            const int col0 = t.ct * TNC + h * (TNC / 2);
            zc* Cb = p.C + t.b * p.sC;
            if (t.rt * TM + 32 * q >= p.M || col0 >= p.Nc) {  // nothing of the tile in this warp
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_tmem);
                continue;
            }
#pragma unroll 1
            for (int c0 = 0; c0 < TNC / 2; c0 += 4) {
                uint32_t re[NLEV][4], im[NLEV][4];
#pragma unroll
                for (int lv = 0; lv < NLEV; ++lv) {
                    tmem_ld4(lane_addr + (uint32_t)(lv * NR + h * (TNC / 2) + c0), re[lv]);
                    tmem_ld4(lane_addr + (uint32_t)(lv * NR + TNC + h * (TNC / 2) + c0), im[lv]);
                }
                tmem_wait_ld();
                if (c0 + 4 >= TNC / 2) {  // the accumulators are in registers: the next tile may have them
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bar_tmem);
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int j = col0 + c0 + c;
                    const int eb = j < p.Nc ? p.EB[t.b * p.Nc + j] : 1;
                    uint32_t x[NLEV], y[NLEV];
#pragma unroll
                    for (int lv = 0; lv < NLEV; ++lv) {
                        x[lv] = re[lv][c];
                        y[lv] = im[lv][c];
                    }
                    epi[lane * 5 + c] = make_double2(combine<NLEV>(x, ea, eb), combine<NLEV>(y, ea, eb));
                }
                __syncwarp();
                // 8 rows of 4 columns (64 bytes) at a time
#pragma unroll
                for (int rr = 0; rr < 32; rr += 8) {
                    const int rl = rr + (lane >> 2), c = lane & 3;
                    const int gi = t.rt * TM + 32 * q + rl, j = col0 + c0 + c;
                    if (gi < p.M && j < p.Nc) {
                        double2 v = epi[rl * 5 + c];
                        double2* dst = reinterpret_cast<double2*>(Cb + gi * p.ldc + j);
                        if (p.mode) {
                            const double2 o = *dst;
                            v = p.mode > 0 ? make_double2(o.x + v.x, o.y + v.y) : make_double2(o.x - v.x, o.y - v.y);
                        }
                        *dst = v;
                    }
                }
                __syncwarp();
            }
        }
    } else {
        const int tb = tid - A_THREADS;
        if constexpr (PRE) {
            if (tb == 0) {
                int64_t last[2] = {-1, -1};
                int tn = 0;
                bool stop = false;
                for (int64_t L = blockIdx.x; L < p.ntiles && !stop; L += gridDim.x, ++tn) {
                    const Tile t = tile_at(p, L);
                    const unsigned char* ia =
                        static_cast<const unsigned char*>(p.A) + ((int64_t)t.rt * p.nst_img + p.it0) * ABYTES;
                    const unsigned char* ib =
                        static_cast<const unsigned char*>(p.B) + ((int64_t)t.ct * p.nst_img + p.it0) * (S * BPLANE);
                    for (int it = 0; it < nst; ++it) {
                        const int64_t gs = (int64_t)tn * nst + it;
                        const int bi = (int)(gs & 1);
                        if (abort_sh || (gs >= 2 && !mbar_wait(&bar_empty[bi], (uint32_t)(((gs >> 1) - 1) & 1), &abort_sh,
                                                               p.wait_limit))) {
                            abort_sh = 1;
                            stop = true;
                            break;
                        }
                        mbar_arrive_tx(&bar_full[bi], STAGE);
                        bulk_copy(sbase + bi * STAGE, ia + (int64_t)it * ABYTES, ABYTES, &bar_full[bi]);
                        bulk_copy(sbase + bi * STAGE + ABYTES, ib + (int64_t)it * (S * BPLANE), S * BPLANE, &bar_full[bi]);
                        last[bi] = gs;
                    }
                }
                // every copy has landed before the CTA can leave
                for (int bi = 0; bi < 2; ++bi)
                    if (last[bi] >= 0) mbar_wait_plain(&bar_full[bi], (uint32_t)((last[bi] >> 1) & 1));
            }
        } else {
            const int j = tb % TNC, g = (tb / TNC) & 1, part = tb / (2 * TNC);
            zc nxt[8];
            auto load = [&](int64_t L, int it) {
                const Tile t = tile_at(p, L);
                const int gj = t.ct * TNC + j, k = it * TK + 8 * g;
                ld8(static_cast<const zc*>(p.B) + t.b * p.sB + k * p.bk + gj * p.bj, p.bk, gj < p.Nc ? kleft(p.K, k) : 0,
                    nxt);
            };
            if (blockIdx.x < p.ntiles) load(blockIdx.x, 0);
            int tn = 0;
            bool stop = false;
            for (int64_t L = blockIdx.x; L < p.ntiles && !stop; L += gridDim.x, ++tn) {
                const Tile t = tile_at(p, L);
                const int gj = t.ct * TNC + j;
                const int e = gj < p.Nc ? p.EB[t.b * p.Nc + gj] : 1;
                for (int it = 0; it < nst; ++it) {
                    const int64_t gs = (int64_t)tn * nst + it;
                    const int bi = (int)(gs & 1);
                    uint4 d[S];
                    if (part == 0)
                        planes<0>(nxt, e, false, d);
                    else
                        planes<1>(nxt, e, p.conjB != 0, d);
                    if (it + 1 < nst)
                        load(L, it + 1);
                    else if (L + gridDim.x < p.ntiles)
                        load(L + gridDim.x, 0);
                    if (abort_sh || (gs >= 2 && !mbar_wait(&bar_empty[bi], (uint32_t)(((gs >> 1) - 1) & 1), &abort_sh,
                                                           p.wait_limit))) {
                        abort_sh = 1;
                        stop = true;
                        break;
                    }
                    const uint32_t sb = sbase + bi * STAGE + ABYTES + blk_off(j, g);
                    if (part == 0) {
#pragma unroll
                        for (int s = 0; s < S; ++s) st_shared_v4(sb + s * BPLANE + BLK, d[s]);
                    } else {
#pragma unroll
                        for (int s = 0; s < S; ++s) {
                            st_shared_v4(sb + s * BPLANE + 2 * BLK, d[s]);
                            st_shared_v4(sb + s * BPLANE, neg8(d[s]));
                        }
                    }
                    fence_async_smem();
                    mbar_arrive(&bar_full[bi]);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (abort_sh && tid == 0) atomicOr(p.err, 2);  // bit 1: a bounded wait ran out
    if (warp == MMA_WARP) {
        if (lane == 0 && ndone > 0) mbar_wait_plain(&bar_done, (uint32_t)((ndone - 1) & 1));
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

// Row exponents (one warp per row) of batch matrices of M rows and K columns, row-major.
__global__ void row_exp64_kernel(int64_t rows, int M, int K, const zc* __restrict__ A, int64_t ld, int64_t sA,
                                 int* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < rows; w += nw) {
        const zc* a = A + (w / M) * sA + (w % M) * ld;
        int e = 1;
        for (int k = lane; k < K; k += 32) e = max(e, elem_exp(a[k]));
        e = __reduce_max_sync(0xffffffffu, e);
        if (lane == 0) out[w] = e;
    }
}
// Column exponents: a warp takes 32 columns (lanes) of one matrix; the rows are
// dealt to the block's warps.
__global__ void __launch_bounds__(256) col_exp64_kernel(int64_t batch, int K, int64_t Nc, const zc* __restrict__ B,
                                                        int64_t ld, int64_t sB, int* __restrict__ out) {
    __shared__ int part[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t nct = (Nc + 31) / 32;
    for (int64_t w = blockIdx.x; w < batch * nct; w += gridDim.x) {
        const int64_t b = w / nct, c = (w % nct) * 32 + lane;
        int e = 1;
        if (c < Nc)
            for (int k = warp; k < K; k += 8) e = max(e, elem_exp(B[b * sB + (int64_t)k * ld + c]));
        part[warp][lane] = e;
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int i = 1; i < 8; ++i) e = max(e, part[i][lane]);
            if (c < Nc) out[b * Nc + c] = e;
        }
        __syncthreads();
    }
}

// Stage images of A (M x K row-major, row exponents EA): thread = (row, 8 k).
__global__ void __launch_bounds__(256) a_image_kernel(int64_t M, int K, const zc* __restrict__ A, int64_t ld,
                                                      const int* __restrict__ EA, unsigned char* __restrict__ img) {
    const int nst = (K + TK - 1) / TK;
    const int64_t total = ((M + TM - 1) / TM) * nst * 256;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int q = (int)(idx & 255), r = q >> 1, g = q & 1;
        const int64_t blk = idx >> 8, gi = blk / nst * TM + r;
        const int k = (int)(blk % nst) * TK + 8 * g;
        const int e = gi < M ? EA[gi] : 1;
        zc v[8];
        ld8(A + gi * ld + k, 1, gi < M ? kleft(K, k) : 0, v);
        unsigned char* dst = img + blk * (int64_t)(S * APLANE) + blk_off(r, g);
        uint4 d[S];
        planes<0>(v, e, false, d);
#pragma unroll
        for (int s = 0; s < S; ++s) *reinterpret_cast<uint4*>(dst + s * APLANE) = d[s];
        planes<1>(v, e, false, d);
#pragma unroll
        for (int s = 0; s < S; ++s) *reinterpret_cast<uint4*>(dst + s * APLANE + APLANE / 2) = d[s];
    }
}
// Stage images of a real-coefficient table (2 Kc rows of Nc complex entries):
// blocks Re even, Im even, Re odd, Im odd rows; thread = (column, 8 kappa, even / odd).
template <int TNC>
__global__ void __launch_bounds__(TNC * 4) table_image_kernel(int Kc, int64_t Nc, const zc* __restrict__ T,
                                                              const int* __restrict__ EB,
                                                              unsigned char* __restrict__ img) {
    using Sh = Shape<TNC>;
    constexpr int BPLANE = Sh::bplane(REALC);
    const int nst = (Kc + TK - 1) / TK;
    const int64_t nblk = ((Nc + TNC - 1) / TNC) * nst;
    const int j = threadIdx.x % TNC, g = (threadIdx.x / TNC) & 1, odd = threadIdx.x / (2 * TNC);
    for (int64_t blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
        const int64_t gj = blk / nst * TNC + j;
        const int k = (int)(blk % nst) * TK + 8 * g;
        const int e = gj < Nc ? EB[gj] : 1;
        zc v[8];
        ld8(T + (int64_t)(2 * k + odd) * Nc + gj, 2 * Nc, gj < Nc ? kleft(Kc, k) : 0, v);
        unsigned char* dst = img + blk * (int64_t)(S * BPLANE) + odd * 2 * Sh::BLK + blk_off(j, g);
        uint4 d[S];
        planes<0>(v, e, false, d);
#pragma unroll
        for (int s = 0; s < S; ++s) *reinterpret_cast<uint4*>(dst + s * BPLANE) = d[s];
        planes<1>(v, e, false, d);
#pragma unroll
        for (int s = 0; s < S; ++s) *reinterpret_cast<uint4*>(dst + s * BPLANE + Sh::BLK) = d[s];
    }
}

int sms() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) {
        cudaGetLastError();
        n = 1;
    }
    return n;
}
inline unsigned blocks(int64_t n) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>(n, 152LL * 64)); }

template <int TNC, bool PRE>
int launch(cudaStream_t st, OzArgs p, int64_t batch, int rows_fast) {
    const int smem = Shape<TNC>::smem(PRE ? REALC : CPLX);
    auto kern = oz64_kernel<TNC, PRE>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(oz64)");
    const int nr = (p.M + TM - 1) / TM, nc = (p.Nc + TNC - 1) / TNC;
    p.rows_fast = rows_fast;
    p.gx = rows_fast ? nr : nc;
    p.gy = rows_fast ? nc : nr;
    p.ntiles = (int64_t)nr * nc * batch;
    p.wait_limit = tc_wait_limit();
    kern<<<(unsigned)std::min<int64_t>(p.ntiles, sms()), Shape<TNC>::THREADS, smem, st>>>(p);
    TBG_LAUNCHED("oz64_kernel");
    return TBG_OK;
}

}  // namespace

// Line exponents of batch matrices stored row-major (K rows or columns as named).
int oz64_row_exps(cudaStream_t st, int64_t batch, int M, int K, const zc* A, int64_t ld, int64_t sA, int* out) {
    row_exp64_kernel<<<blocks((batch * M + 7) / 8), 256, 0, st>>>(batch * M, M, K, A, ld, sA, out);
    TBG_LAUNCHED("row_exp64_kernel");
    return TBG_OK;
}
int oz64_col_exps(cudaStream_t st, int64_t batch, int K, int64_t Nc, const zc* B, int64_t ld, int64_t sB, int* out) {
    col_exp64_kernel<<<blocks(batch * ((Nc + 31) / 32)), 256, 0, st>>>(batch, K, Nc, B, ld, sB, out);
    TBG_LAUNCHED("col_exp64_kernel");
    return TBG_OK;
}

int oz64_gemm(cudaStream_t st, int64_t batch, int M, int Nc, int K, const Oz64Operand& A, const Oz64Operand& B, zc* C,
              int64_t ldc, int64_t sC, int mode, int* err) {
    if (batch <= 0 || M <= 0 || Nc <= 0) return TBG_OK;
    if (K <= 0) return set_error(TBG_E_INVALID_ARGUMENT, "oz64_gemm: empty contraction");
    KTimer kt(st, "oz64_kernel", 8.0 * M * Nc * (double)K * batch);
    OzArgs p = {};
    p.M = M;
    p.Nc = Nc;
    p.ai = A.line;
    p.ak = A.k;
    p.sA = A.batch;
    p.conjA = A.conj;
    p.EA = A.exps;
    p.bj = B.line;
    p.bk = B.k;
    p.sB = B.batch;
    p.conjB = B.conj;
    p.EB = B.exps;
    p.C = C;
    p.ldc = ldc;
    p.sC = sC;
    p.err = err;
    for (int k0 = 0; k0 < K; k0 += kMaxK) {
        p.K = std::min(kMaxK, K - k0);
        p.A = A.p + k0 * A.k;
        p.B = B.p + k0 * B.k;
        p.mode = k0 ? (mode < 0 ? -1 : 1) : mode;
        // 40 columns a tile unless 32 leave fewer idle ones
        const int w40 = (Nc + 39) / 40 * 40, w32 = (Nc + 31) / 32 * 32;
        const int rc = w32 <= w40 ? launch<32, false>(st, p, batch, 0) : launch<40, false>(st, p, batch, 0);
        if (rc) return rc;
    }
    return TBG_OK;
}

constexpr int kTab = 40;  // columns of a table image's tiles
size_t oz64_table_image_bytes(int Kc, int64_t Nc) {
    return (size_t)((Nc + kTab - 1) / kTab) * ((Kc + TK - 1) / TK) * S * Shape<kTab>::bplane(REALC);
}
size_t oz64_row_image_bytes(int64_t M, int Kc) {
    return (size_t)((M + TM - 1) / TM) * ((Kc + TK - 1) / TK) * S * APLANE;
}
// Image of a table of 2 Kc rows x Nc entries and its column exponents EB (Nc).
int oz64_table_image(cudaStream_t st, int Kc, int64_t Nc, const zc* T, int* EB, void* img) {
    if (int rc = oz64_col_exps(st, 1, 2 * Kc, Nc, T, Nc, 0, EB)) return rc;
    const int64_t nblk = ((Nc + kTab - 1) / kTab) * ((Kc + TK - 1) / TK);
    table_image_kernel<kTab><<<blocks(nblk), kTab * 4, 0, st>>>(Kc, Nc, T, EB, static_cast<unsigned char*>(img));
    TBG_LAUNCHED("table_image_kernel");
    return TBG_OK;
}
// C (M x Nc) = coefficients (M x Kc pairs of reals, rows ld apart) times the table behind (img, EB);
// EA (M ints) and aimg (oz64_row_image_bytes) are scratch.
int oz64_table_product(cudaStream_t st, int64_t M, int64_t Nc, int Kc, const zc* coef, int64_t ld, const int* EB,
                       const void* img, zc* C, int* EA, void* aimg, int* err) {
    if (M <= 0) return TBG_OK;
    if (M > 0x7fffffff || Nc > 0x7fffffff) return set_error(TBG_E_UNSUPPORTED, "oz64_table_product: too large");
    const int nst = (Kc + TK - 1) / TK;
    {
        KTimer kt(st, "oz64_image_kernel");
        if (int rc = oz64_row_exps(st, 1, (int)M, Kc, coef, ld, 0, EA)) return rc;
        a_image_kernel<<<blocks((M + TM - 1) / TM * nst), 256, 0, st>>>(M, Kc, coef, ld, EA,
                                                                        static_cast<unsigned char*>(aimg));
        TBG_LAUNCHED("a_image_kernel");
    }
    KTimer kt(st, "oz64_fourier_kernel", 8.0 * (double)M * Nc * Kc);
    OzArgs p = {};
    p.M = (int)M;
    p.Nc = (int)Nc;
    p.A = aimg;
    p.ak = 1;
    p.B = img;
    p.EA = EA;
    p.EB = EB;
    p.C = C;
    p.ldc = Nc;
    p.err = err;
    p.nst_img = nst;
    for (int k0 = 0; k0 < Kc; k0 += kMaxK) {
        p.K = std::min(kMaxK, Kc - k0);
        p.it0 = k0 / TK;
        p.mode = k0 ? 1 : 0;
        // row tiles fastest: CTAs running together share a column tile's image in L2
        if (int rc = launch<kTab, true>(st, p, 1, 1)) return rc;
    }
    return TBG_OK;
}

}  // namespace tbg

// Internal test hook (not part of the public header): host arrays, row-major
// operands; a conjugate-transposed one is given as stored (K x M, Nc x K).
extern "C" int tbg_internal_oz64_gemm(int conj_a, int conj_b, int64_t batch, int M, int Nc, int K, int mode,
                                      const double* A, const double* B, double* C) {
    using namespace tbg;
    const size_t na = (size_t)M * K * batch, nb = (size_t)K * Nc * batch, nc = (size_t)M * Nc * batch;
    zc *dA = nullptr, *dB = nullptr, *dC = nullptr;
    int *e = nullptr, h = 0;
    int rc = TBG_OK;
    if (cudaMalloc(&dA, sizeof(zc) * na) || cudaMalloc(&dB, sizeof(zc) * nb) || cudaMalloc(&dC, sizeof(zc) * nc) ||
        cudaMalloc(&e, sizeof(int) * ((size_t)batch * (M + Nc) + 1)))
        rc = set_error(TBG_E_OOM, "oz64 test alloc");
    if (!rc) {
        int *ea = e, *eb = e + batch * M, *err = eb + batch * Nc;
        cudaMemcpy(dA, A, sizeof(zc) * na, cudaMemcpyHostToDevice);
        cudaMemcpy(dB, B, sizeof(zc) * nb, cudaMemcpyHostToDevice);
        cudaMemcpy(dC, C, sizeof(zc) * nc, cudaMemcpyHostToDevice);
        cudaMemset(err, 0, sizeof(int));
        const int64_t sA = (int64_t)M * K, sB = (int64_t)K * Nc;
        rc = conj_a ? oz64_col_exps(nullptr, batch, K, M, dA, M, sA, ea) : oz64_row_exps(nullptr, batch, M, K, dA, K, sA, ea);
        if (!rc)
            rc = conj_b ? oz64_row_exps(nullptr, batch, Nc, K, dB, K, sB, eb)
                        : oz64_col_exps(nullptr, batch, K, Nc, dB, Nc, sB, eb);
        const Oz64Operand a = conj_a ? Oz64Operand{dA, 1, M, sA, 1, ea} : Oz64Operand{dA, K, 1, sA, 0, ea};
        const Oz64Operand b = conj_b ? Oz64Operand{dB, K, 1, sB, 1, eb} : Oz64Operand{dB, 1, Nc, sB, 0, eb};
        if (!rc) rc = oz64_gemm(nullptr, batch, M, Nc, K, a, b, dC, Nc, (int64_t)M * Nc, mode, err);
        if (!rc) {
            cudaError_t er = cudaMemcpy(C, dC, sizeof(zc) * nc, cudaMemcpyDeviceToHost);
            if (er == cudaSuccess) er = cudaMemcpy(&h, err, sizeof(int), cudaMemcpyDeviceToHost);
            if (er != cudaSuccess)
                rc = cuda_error(er, "oz64 test");
            else if (h)
                rc = set_error(TBG_E_TIMEOUT, "oz64 test: a bounded wait ran out");
        }
    }
    cudaFree(dA);
    cudaFree(dB);
    cudaFree(dC);
    cudaFree(e);
    return rc;
}
