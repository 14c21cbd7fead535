// FP64-accurate complex matrix products on the 5th-generation tensor cores.
//
// The part's FP64 pipe does about 1/64 of its FP32 rate, its BF16 tensor cores
// some 2000 times as much, so a product is run as exact digit products (error-free
// splitting after Ozaki, Ogita, Oishi and Rump 2012): a row of A (column of B)
// with |x| < 2^E is written on the grid 2^(E - 55) and cut into seven signed
// digits of eight bits, which BF16 holds exactly.  Digit pairs of level
// s + t <= 6 are kept (28 of 49), each level in an FP32 accumulator of its own.
// Digits are at most 128, so L + 1 pairs of level L sum to at most (L + 1) 2^15 a
// complex term: FP32's 2^24 holds levels 0 to 4 exactly over 96 terms, level 0 over
// 256.  So after every 96 terms at most the levels 4 .. 1 pass what exceeds a digit
// on to the level before them, in tensor memory and exactly (carry), and after 256
// the sums are drained and added in FP64.  (All 256 in one go lost the last bits of
// levels 2 to 4 when the digits were large and their products did not cancel: 10^-8 of
// the scale.)  Levels 5 and 6 may lose their last place, 2^-54 of the product's scale
// 2^(EA + EB), but only where the sum itself is some 100 times the scale.  The level sums are put
// together as 64-bit integers (an FP64 addition costs as much as dozens of integer
// instructions here) and rounded once to FP64.  The tensor core truncates, so
// levels with different last places must not share an accumulator early: with
// levels 4 to 6 in one the error of a 128-term product was 300 x 2^-54 of the
// scale, against 10 x for an FP64 sum and 6.8 x now.
//
// The error is relative to (largest of the line of A) x (largest of the line of B):
// elements below an eighth of their line's largest keep fewer than 53 bits, where an
// FP64 sum's error follows the sum of |a| |b|.
//
// Shared memory feeds the tensor cores 128 bytes a clock, so an MMA of 128 rows pays
// 32 clocks for A and 16 per 64 columns of B, against 16 of arithmetic: digit pairs
// (s, t), (s, t + 1), ... are one MMA, the digits of B side by side as its columns and
// the accumulators of the levels side by side as its output (10 MMAs for the 28
// pairs; one each took 55 clocks a pair).
//
// A's digits are cut into stage images first (a_image_kernel: one pass, not one per
// column tile, and with every SM's issue slots).  A CTA then walks output tiles of
// 128 rows x 32 complex columns (seven accumulators of 64 of the 512 TMEM columns):
//   warps 0..15    epilogue, one TMEM lane = one row
//   warps 16..23   digits of B, thread = (column, 8 consecutive k, component), two
//                  groups that fill the two stage buffers in turn; idle when B too
//                  comes as images
//   warp 24        copies the images with cp.async.bulk
//   warp 25        allocates TMEM and issues the MMAs (M = 128, N <= 256, K = 16)
// so a tile's epilogue runs beside the next tile's copies and cutting.  A k step of
// complex operands is [Re A] with [Re B; Im B], then [Im A] with [-Im B; Re B].
// Stage hand-off by mbarriers; every wait is bounded, as in the float-pair products
// (ozaki_tc.cu).
//
// 1024 products of 128 bands: one of the four of the rotation 13.8 ms on the FP64
// pipe in 64 x 64 tiles, 0.53 here (0.93 with one MMA per pair and A cut by the
// tiles' own warps).

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
constexpr int TNC = 32;     // complex columns of a tile
constexpr int NR = 2 * TNC; // real columns: of a digit of B, and of a level's accumulator
constexpr int BBLK = NR * TK * 2;            // bytes of one digit of B for one k step: NR rows x 16 k
constexpr int BKS = S * BBLK;                // the digits side by side
constexpr int ABYTES = S * APLANE, BBYTES = 2 * BKS, STAGE = ABYTES + BBYTES;
constexpr int E_THREADS = 512;               // epilogue
constexpr int B_THREADS = TNC * 4;           // (column, half of the 16 k, component), per group
constexpr int THREADS = E_THREADS + 2 * B_THREADS + 64;
constexpr int EPI = E_THREADS / 32 * 32 * 5 * 16;  // 4 columns of 32 rows per warp, rows padded to 5
constexpr int SMEM = 2 * STAGE + EPI + 1024;
// How a contraction of nst stages is held exact: up to PLAIN_STAGES as it is; up to
// SPLIT_STAGES with pair (4, 0) in an eighth accumulator (level 4 then has four pairs
// in its own: 2^24 over 128 terms); beyond, in groups of at most GROUP stages, each in
// parts of at most PLAIN_STAGES with a carry between them, cut evenly.  What it costs,
// against the same kernel without: the 12 products of 128 bands, 1024 k-points (K = 64
// and 128) 4.94 ms, 4.77; the Fourier sums of 172 pairs there 1.63, 1.35 (2.07 when drained
// at 96 terms instead of carried).
enum Form { PLAIN, SPLIT, CARRY };
constexpr int PLAIN_STAGES = 6, SPLIT_STAGES = 8, GROUP = 16;  // 96, 128 and 256 complex k
struct Cuts {
    int group, part;  // stages
};
__host__ __device__ __forceinline__ Cuts cuts_of(int nst) {
    const int groups = (nst + GROUP - 1) / GROUP, group = (nst + groups - 1) / groups;
    const int parts = (group + PLAIN_STAGES - 1) / PLAIN_STAGES;
    return {group, (group + parts - 1) / parts};
}
// kind::f16: D = F32, A = B = BF16, K-major, M = 128, N = n NR
__host__ __device__ constexpr uint32_t idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n * NR >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
}

// byte offset of (row, half of the 16 k) in a block of core matrices (8 rows x 16 bytes)
__host__ __device__ __forceinline__ int blk_off(int row, int half) {
    return (((row >> 3) * 2 + half) << 7) + ((row & 7) << 4);
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(su32(bar))
                 : "memory");
}

__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, "
        "p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
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
__device__ __forceinline__ void planes(const double (&v)[8], int e, bool neg, uint4 (&out)[S]) {
    uint32_t pk[S][4];
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        float P0[S], P1[S];
        digits(fixed55(v[i], e), P0);
        digits(fixed55(v[i + 1], e), P1);
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

// 8 consecutive-k elements (stride in elements), and the same of one component.
__device__ __forceinline__ void ld8(const zc* p, int64_t stride, int nvalid, double (&re)[8], double (&im)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        double2 t = make_double2(0.0, 0.0);
        if (i < nvalid) t = __ldg(reinterpret_cast<const double2*>(p + i * stride));
        re[i] = t.x;
        im[i] = t.y;
    }
}
__device__ __forceinline__ void ld8(const zc* p, int part, int64_t stride, int nvalid, double (&v)[8]) {
    const double* d = reinterpret_cast<const double*>(p) + part;
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = i < nvalid ? __ldg(d + 2 * i * stride) : 0.0;
}

// The level sums -> their FP64 value times 2^(ea + eb - 2058) (e - 1022 - 7 per operand).
template <int N>
__device__ __forceinline__ double combine(const uint32_t (&a)[N], int ea, int eb) {
    if (ea == kNonFinite || eb == kNonFinite) return __longlong_as_double(0x7ff8000000000000ll);
    const float tail = __uint_as_float(a[5]) + __uint_as_float(a[6]);  // below 2^-14
    int l4 = __float2int_rn(__uint_as_float(a[4]) * 0x1p32f);
    if (N > S) l4 += __float2int_rn(__uint_as_float(a[N - 1]) * 0x1p32f);  // pair (4, 0)
    const long long I = ((long long)__float2int_rn(__uint_as_float(a[0])) << 39) +
                        ((long long)__float2int_rn(__uint_as_float(a[1]) * 0x1p8f) << 31) +
                        ((long long)__float2int_rn(__uint_as_float(a[2]) * 0x1p16f) << 23) +
                        ((long long)__float2int_rn(__uint_as_float(a[3]) * 0x1p24f) << 15) +
                        ((long long)l4 << 7) +
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

// C (M x Nc per matrix) = / += / -= A op(B).  A: stage images per (matrix, row
// tile).  Element (k, j) of op(B) is at
// B + b sB + k bk + j bj (conjugated when conjB); PRE: B is images too, per column
// tile.  EA, EB: line exponents per (matrix, row) and (matrix, column).
struct OzArgs {
    int M, Nc, K;
    const unsigned char* A;
    const void* B;
    int64_t bk, bj, sB;
    int conjB;
    const int *EA, *EB;
    zc* C;
    int64_t ldc, sC;
    int mode;  // 0: store, 1: add, -1: subtract
    int* err;
    int wait_limit;
    int gx, gy, rows_fast;
    int64_t ntiles;
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
// OR over the epilogue warps
__device__ __forceinline__ bool any_epilogue(bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.or.pred p, 1, %2, q;\n\tselp.u32 %0, 1, 0, "
        "p;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)v), "n"(E_THREADS)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ void tmem_ld2(uint32_t taddr, uint32_t& a, uint32_t& b) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(a), "=r"(b) : "r"(taddr));
}

// Levels 4 .. 1 of 8 columns: what exceeds half a place of the level before goes
// there, that of level 1 first, so that no level holds more than a digit when it
// receives (level L counts in 2^(-8 L); |level| < 2^24 of that).
__device__ __forceinline__ void carry_levels(uint32_t taddr) {
    uint32_t v[5][8];
#pragma unroll
    for (int lv = 0; lv < 5; ++lv) tmem_ld8(taddr + (uint32_t)(lv * NR), v[lv]);
    tmem_wait_ld();
#pragma unroll
    for (int lv = 1; lv < 5; ++lv) {
        const float C = lv == 1 ? 0x1.8p23f : lv == 2 ? 0x1.8p15f : lv == 3 ? 0x1.8p7f : 0x1.8p-1f;  // 1.5 2^(31 - 8 lv)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float x = __uint_as_float(v[lv][i]), c = __fsub_rn(__fadd_rn(x, C), C);
            v[lv - 1][i] = __float_as_uint(__fadd_rn(__uint_as_float(v[lv - 1][i]), c));
            v[lv][i] = __float_as_uint(__fsub_rn(x, c));
        }
    }
#pragma unroll
    for (int lv = 0; lv < 5; ++lv) tmem_st8(taddr + (uint32_t)(lv * NR), v[lv]);
}

template <bool PRE, int FORM>
__global__ void __launch_bounds__(THREADS, 1) oz64_kernel(OzArgs p) {
    extern __shared__ __align__(1024) unsigned char oz_smem[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)oz_smem + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bar_full[2], bar_empty[2], bar_done, bar_tmem;
    __shared__ uint32_t tmem_sh;
    __shared__ volatile int abort_sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int MMA_WARP = THREADS / 32 - 1, COPY_WARP = MMA_WARP - 1;
    const int nst = (p.K + TK - 1) / TK;
    const Cuts cut = FORM == CARRY ? cuts_of(nst) : Cuts{nst, nst};
    const uint32_t sbase = su32(base);
    if (tid == 0) {
        const uint32_t nfull = PRE ? 1 : 1 + B_THREADS;
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_full[i], nfull);
            mbar_init(&bar_empty[i], 1);
        }
        mbar_init(&bar_done, 1);
        mbar_init(&bar_tmem, E_THREADS / 32);
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
    int ndone = 0;  // parts committed to bar_done

    if (warp == MMA_WARP) {
        if (lane == 0) {
            int tn = 0;
            bool stop = false, open = false;  // open: MMAs issued behind the last commit to bar_done
            for (int64_t L = blockIdx.x; L < p.ntiles && !stop; L += gridDim.x, ++tn) {
                for (int it = 0, ig = 0, ip = 0; it < nst; ++it) {  // ig, ip: stage of the group, of the part
                    // the accumulators have been read out, or have carried
                    if (ip == 0 && ndone > 0) {
                        if (!mbar_wait(&bar_tmem, (uint32_t)((ndone - 1) & 1), &abort_sh, p.wait_limit)) {
                            abort_sh = 1;
                            stop = true;
                            break;
                        }
                        tc_fence_after();
                    }
                    const int64_t gs = (int64_t)tn * nst + it;
                    const int bi = (int)(gs & 1);
                    if (!mbar_wait(&bar_full[bi], (uint32_t)((gs >> 1) & 1), &abort_sh, p.wait_limit)) {
                        abort_sh = 1;
                        stop = true;
                        break;
                    }
                    tc_fence_after();
                    open = true;
                    const uint32_t sa = sbase + bi * STAGE, sb = sa + ABYTES;
#pragma unroll
                    for (int ks = 0; ks < 2; ++ks) {
#pragma unroll
                        for (int s = 0; s < S; ++s) {
                            const uint64_t ad = smem_desc(sa + s * APLANE + ks * (APLANE / 2), 128, 256);
                            // pairs (s, t) .. (s, t + n - 1) into the accumulators from `to` on
                            auto pairs = [&](int t, int n, int to) {
                                const uint64_t bd = smem_desc(sb + ks * BKS + t * BBLK, 128, 256);
                                // digit 0 of A meets every level first
                                const uint32_t acc = (ig == 0 && ks == 0 && (s == 0 || to == S)) ? 0u : 1u;
                                mma(tmem + (uint32_t)(to * NR), ad, bd, idesc(n), acc);
                            };
                            const bool apart = FORM == SPLIT && s == 4;
                            if (apart) pairs(0, 1, S);
#pragma unroll
                            for (int t = apart ? 1 : 0; t < S - s; t += 4) pairs(t, S - s - t < 4 ? S - s - t : 4, s + t);
                        }
                    }
                    umma_commit(&bar_empty[bi]);
                    ++ig;
                    if (++ip == cut.part || ig == cut.group || it + 1 == nst) {
                        umma_commit(&bar_done);
                        ++ndone;
                        open = false;
                        ip = 0;
                        if (ig == cut.group) ig = 0;
                    }
                }
            }
            if (open) {  // an abort: the part before has been read, so the wait below meets this commit
                umma_commit(&bar_done);
                ++ndone;
            }
        }
        __syncwarp();
    } else if (warp == COPY_WARP) {
        if (lane == 0) {
            const int nrt = p.rows_fast ? p.gx : p.gy;
            int64_t last[2] = {-1, -1};
            int tn = 0;
            bool stop = false;
            for (int64_t L = blockIdx.x; L < p.ntiles && !stop; L += gridDim.x, ++tn) {
                const Tile t = tile_at(p, L);
                const unsigned char* ia = p.A + (t.b * nrt + t.rt) * nst * ABYTES;
                const unsigned char* ib = static_cast<const unsigned char*>(p.B) + (int64_t)t.ct * nst * BBYTES;
                for (int it = 0; it < nst; ++it) {
                    const int64_t gs = (int64_t)tn * nst + it;
                    const int bi = (int)(gs & 1);
                    if (abort_sh || (gs >= 2 && !mbar_wait(&bar_empty[bi], (uint32_t)(((gs >> 1) - 1) & 1), &abort_sh,
                                                           p.wait_limit))) {
                        abort_sh = 1;
                        stop = true;
                        break;
                    }
                    mbar_arrive_tx(&bar_full[bi], PRE ? STAGE : ABYTES);
                    bulk_copy(sbase + bi * STAGE, ia + (int64_t)it * ABYTES, ABYTES, &bar_full[bi]);
                    if (PRE) bulk_copy(sbase + bi * STAGE + ABYTES, ib + (int64_t)it * BBYTES, BBYTES, &bar_full[bi]);
                    last[bi] = gs;
                }
            }
            // every copy has landed before the CTA can leave (after an abort the other
            // producers may not arrive: the bounded wait then outlasts the copies)
            for (int bi = 0; bi < 2; ++bi)
                if (last[bi] >= 0) mbar_wait_plain(&bar_full[bi], (uint32_t)((last[bi] >> 1) & 1));
        }
        __syncwarp();
    } else if (tid < E_THREADS) {
        // warp: TMEM lanes 32 q .. and complex columns 8 h ..
        const int q = warp & 3, h = warp >> 2;
        constexpr int CW = TNC / (E_THREADS / 128);
        const uint32_t taddr = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(CW * h);
        double2* epi = reinterpret_cast<double2*>(base + 2 * STAGE) + warp * (32 * 5);
        int u = 0;  // parts so far
        auto part_done = [&]() {  // whether the MMAs of part u are done; a group is written whole or not at all
            bool bad = abort_sh != 0;
            if (!bad && !mbar_wait(&bar_done, u & 1, &abort_sh, p.wait_limit)) {
                abort_sh = 1;
                bad = true;
            }
            ++u;
            if (any_epilogue(bad)) return false;
            tc_fence_after();
            return true;
        };
        auto release = [&]() {  // the accumulators may be written again
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_tmem);
        };
        int g0 = 0;  // first stage of the group (CARRY; the others have one)
        for (int64_t L = blockIdx.x; L < p.ntiles; L += FORM == CARRY && g0 ? 0 : gridDim.x) {
            const int glen = min(cut.group, nst - g0);
            const int mode = FORM == CARRY && g0 ? (p.mode < 0 ? -1 : 1) : p.mode;
            if constexpr (FORM == CARRY) g0 = g0 + glen < nst ? g0 + glen : 0;
            const Tile t = tile_at(p, L);
            const int row = t.rt * TM + 32 * q + lane;
            const int ea = row < p.M ? p.EA[t.b * p.M + row] : 1;
            const int col0 = t.ct * TNC + CW * h;
            const int* EBt = p.EB + t.b * p.Nc;
            if constexpr (FORM == CARRY) {
                bool go = true;
                for (int i = cut.part; i < glen && (go = part_done()); i += cut.part) {
                    carry_levels(taddr);
                    carry_levels(taddr + TNC);
                    tmem_wait_st();
                    release();
                }
                if (!go) break;
            }
            if (!part_done()) break;
            zc* Cb = p.C + t.b * p.sC;
            if (t.rt * TM + 32 * q >= p.M || col0 >= p.Nc) {  // nothing of the tile in this warp
                release();
                continue;
            }
#pragma unroll 1
            for (int c0 = 0; c0 < CW; c0 += 4) {
#pragma unroll
                for (int c2 = 0; c2 < 4; c2 += 2) {
                    constexpr int NA = FORM == SPLIT ? S + 1 : S;
                    uint32_t x0[NA], x1[NA], y0[NA], y1[NA];
#pragma unroll
                    for (int lv = 0; lv < NA; ++lv) {
                        tmem_ld2(taddr + (uint32_t)(lv * NR + c0 + c2), x0[lv], x1[lv]);
                        tmem_ld2(taddr + (uint32_t)(lv * NR + TNC + c0 + c2), y0[lv], y1[lv]);
                    }
                    const int j = col0 + c0 + c2;
                    const int e0 = j < p.Nc ? EBt[j] : 1, e1 = j + 1 < p.Nc ? EBt[j + 1] : 1;
                    tmem_wait_ld();
                    if (c0 + 4 >= CW && c2 == 2) release();  // all of them are in registers
                    epi[lane * 5 + c2] = make_double2(combine(x0, ea, e0), combine(y0, ea, e0));
                    epi[lane * 5 + c2 + 1] = make_double2(combine(x1, ea, e1), combine(y1, ea, e1));
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
                        if (mode) {
                            const double2 o = *dst;
                            v = mode > 0 ? make_double2(o.x + v.x, o.y + v.y) : make_double2(o.x - v.x, o.y - v.y);
                        }
                        *dst = v;
                    }
                }
                __syncwarp();
            }
        }
    } else if constexpr (!PRE) {
        // group grp fills buffer grp: stages grp, grp + 2, ... of the CTA's sequence
        const int grp = (tid - E_THREADS) / B_THREADS, tb = (tid - E_THREADS) % B_THREADS;
        const int j = tb % TNC, g = (tb / TNC) & 1, part = tb / (2 * TNC);
        double nxt[8];
        int en = 1;
        auto load = [&](int gs) -> bool {
            const int tn = gs / nst, it = gs - tn * nst;
            const int64_t L = blockIdx.x + (int64_t)tn * gridDim.x;
            if (L >= p.ntiles) return false;
            const Tile t = tile_at(p, L);
            const int gj = t.ct * TNC + j, k = it * TK + 8 * g;
            en = gj < p.Nc ? p.EB[t.b * p.Nc + gj] : 1;
            ld8(static_cast<const zc*>(p.B) + t.b * p.sB + k * p.bk + gj * p.bj, part, p.bk,
                gj < p.Nc ? kleft(p.K, k) : 0, nxt);
            return true;
        };
        bool more = load(grp);
        for (int gs = grp; more; gs += 2) {
            uint4 d[S];
            planes(nxt, en, part && p.conjB, d);
            more = load(gs + 2);
            if (abort_sh ||
                (gs >= 2 && !mbar_wait(&bar_empty[grp], (uint32_t)(((gs >> 1) - 1) & 1), &abort_sh, p.wait_limit))) {
                abort_sh = 1;
                break;
            }
            // Re to [Re; .] and [.; Re], Im to [.; Im] and [-Im; .]
            const uint32_t sb = sbase + grp * STAGE + ABYTES;
            const uint32_t d0 = sb + blk_off(part ? TNC + j : j, g), d1 = sb + BKS + blk_off(part ? j : TNC + j, g);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                st_shared_v4(d0 + s * BBLK, d[s]);
                st_shared_v4(d1 + s * BBLK, part ? neg8(d[s]) : d[s]);
            }
            fence_async_smem();
            mbar_arrive(&bar_full[grp]);
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
// dealt to the block's warps.  Rows 2 q, 2 q + 1 count times 2^wexp[q] when given.
__global__ void __launch_bounds__(256) col_exp64_kernel(int64_t batch, int K, int64_t Nc, const zc* __restrict__ B,
                                                        int64_t ld, int64_t sB, const int* __restrict__ wexp,
                                                        int* __restrict__ out) {
    __shared__ int part[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t nct = (Nc + 31) / 32;
    for (int64_t w = blockIdx.x; w < batch * nct; w += gridDim.x) {
        const int64_t b = w / nct, c = (w % nct) * 32 + lane;
        int e = 1;
        if (c < Nc)
            for (int k = warp; k < K; k += 8) {
                zc x = B[b * sB + (int64_t)k * ld + c];
                if (wexp) x = scalbn(1.0, wexp[k >> 1]) * x;
                e = max(e, elem_exp(x));
            }
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

// Stage images of op(A) (batch matrices of M x K, element (i, k) at
// A + b sA + i ai + k ak, row exponents EA): thread = (row, 8 k), rows of consecutive
// threads when op(A) is stored by columns, else pairs of threads per row.
__global__ void __launch_bounds__(256) a_image_kernel(int64_t batch, int M, int K, const zc* __restrict__ A, int64_t ai,
                                                      int64_t ak, int64_t sA, int conj_a, const int* __restrict__ EA,
                                                      unsigned char* __restrict__ img) {
    const int nst = (K + TK - 1) / TK, nrt = (M + TM - 1) / TM;
    const int q = threadIdx.x, r = ak != 1 ? (q & 127) : (q >> 1), g = ak != 1 ? (q >> 7) : (q & 1);
    for (int64_t blk = blockIdx.x; blk < batch * nrt * nst; blk += gridDim.x) {
        const int it = (int)(blk % nst);
        const int64_t br = blk / nst, b = br / nrt;
        const int gi = (int)(br % nrt) * TM + r, k = it * TK + 8 * g;
        unsigned char* dst = img + blk * (int64_t)(S * APLANE) + blk_off(r, g);
        if (gi >= M) continue;  // rows beyond the matrix only meet rows of the tile that are not stored
        const int e = EA[b * M + gi];
        double re[8], im[8];
        ld8(A + b * sA + gi * ai + k * ak, ak, kleft(K, k), re, im);
        uint4 d[S];
        planes(re, e, false, d);
#pragma unroll
        for (int s = 0; s < S; ++s) *reinterpret_cast<uint4*>(dst + s * APLANE) = d[s];
        planes(im, e, conj_a != 0, d);
#pragma unroll
        for (int s = 0; s < S; ++s) *reinterpret_cast<uint4*>(dst + s * APLANE + APLANE / 2) = d[s];
    }
}
// Stage images of a real-coefficient table (2 Kc rows of Nc complex entries): k step 0
// the even rows, k step 1 the odd ones, [Re; Im]; thread = (column, 8 kappa, even / odd).
// Row pair q times 2^wexp[q] when given.
__global__ void __launch_bounds__(B_THREADS) table_image_kernel(int Kc, int64_t Nc, const zc* __restrict__ T,
                                                                const int* __restrict__ wexp,
                                                                const int* __restrict__ EB,
                                                                unsigned char* __restrict__ img) {
    const int nst = (Kc + TK - 1) / TK;
    const int64_t nblk = ((Nc + TNC - 1) / TNC) * nst;
    const int j = threadIdx.x % TNC, g = (threadIdx.x / TNC) & 1, odd = threadIdx.x / (2 * TNC);
    for (int64_t blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
        const int64_t gj = blk / nst * TNC + j;
        const int k = (int)(blk % nst) * TK + 8 * g;
        const int e = gj < Nc ? EB[gj] : 1;
        double re[8], im[8];
        ld8(T + (int64_t)(2 * k + odd) * Nc + gj, 2 * Nc, gj < Nc ? kleft(Kc, k) : 0, re, im);
        if (wexp)
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (k + i < Kc) {
                    const double w = scalbn(1.0, wexp[k + i]);
                    re[i] *= w;
                    im[i] *= w;
                }
        unsigned char* dst = img + blk * (int64_t)BBYTES + odd * BKS;
        uint4 d[S];
        planes(re, e, false, d);
#pragma unroll
        for (int s = 0; s < S; ++s) *reinterpret_cast<uint4*>(dst + s * BBLK + blk_off(j, g)) = d[s];
        planes(im, e, false, d);
#pragma unroll
        for (int s = 0; s < S; ++s) *reinterpret_cast<uint4*>(dst + s * BBLK + blk_off(TNC + j, g)) = d[s];
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

template <bool PRE>
int launch(cudaStream_t st, OzArgs p, int64_t batch, int rows_fast) {
    const int nst = (p.K + TK - 1) / TK;
    auto kern = nst <= PLAIN_STAGES   ? oz64_kernel<PRE, PLAIN>
                : nst <= SPLIT_STAGES ? oz64_kernel<PRE, SPLIT>
                                      : oz64_kernel<PRE, CARRY>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute(oz64)");
    const int nr = (p.M + TM - 1) / TM, nc = (p.Nc + TNC - 1) / TNC;
    p.rows_fast = rows_fast;
    p.gx = rows_fast ? nr : nc;
    p.gy = rows_fast ? nc : nr;
    p.ntiles = (int64_t)nr * nc * batch;
    p.wait_limit = tc_wait_limit();
    kern<<<(unsigned)std::min<int64_t>(p.ntiles, sms()), THREADS, SMEM, st>>>(p);
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
    col_exp64_kernel<<<blocks(batch * ((Nc + 31) / 32)), 256, 0, st>>>(batch, K, Nc, B, ld, sB, nullptr, out);
    TBG_LAUNCHED("col_exp64_kernel");
    return TBG_OK;
}

size_t oz64_row_image_bytes(int64_t M, int K) {
    return (size_t)((M + TM - 1) / TM) * ((K + TK - 1) / TK) * S * APLANE;
}
constexpr int64_t kImageBytes = 512LL << 20;  // images of A held at a time

int oz64_gemm(cudaStream_t st, int64_t batch, int M, int Nc, int K, const Oz64Operand& A, const Oz64Operand& B, zc* C,
              int64_t ldc, int64_t sC, int mode, int* err) {
    if (batch <= 0 || M <= 0 || Nc <= 0) return TBG_OK;
    if (K <= 0) return set_error(TBG_E_INVALID_ARGUMENT, "oz64_gemm: empty contraction");
    KTimer kt(st, "oz64_kernel", 8.0 * M * Nc * (double)K * batch);
    const int64_t per = (int64_t)oz64_row_image_bytes(M, K);
    int64_t sub = std::min(batch, std::max<int64_t>(1, kImageBytes / per));
    void* mem = nullptr;
    for (;; sub = (sub + 1) / 2) {  // fewer at a time where they do not fit
        const cudaError_t e = scratch_alloc(&mem, (size_t)(per * sub), st);
        if (e == cudaSuccess) break;
        if (sub == 1) return cuda_error(e, "oz64_gemm images");
    }
    unsigned char* img = static_cast<unsigned char*>(mem);
    int rc = TBG_OK;
    for (int64_t b0 = 0; b0 < batch && !rc; b0 += sub) {
        const int64_t nb = std::min(sub, batch - b0);
        a_image_kernel<<<blocks(nb * ((M + TM - 1) / TM) * ((K + TK - 1) / TK)), 256, 0, st>>>(
            nb, M, K, A.p + b0 * A.batch, A.line, A.k, A.batch, A.conj, A.exps + b0 * M, img);
        count_launch();
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) rc = cuda_error(e, "a_image_kernel");
        OzArgs p = {};
        p.M = M;
        p.Nc = Nc;
        p.A = img;
        p.EA = A.exps + b0 * M;
        p.bj = B.line;
        p.bk = B.k;
        p.sB = B.batch;
        p.conjB = B.conj;
        p.EB = B.exps + b0 * Nc;
        p.C = C + b0 * sC;
        p.ldc = ldc;
        p.sC = sC;
        p.err = err;
        p.K = K;
        p.B = B.p + b0 * B.batch;
        p.mode = mode;
        if (!rc) rc = launch<false>(st, p, nb, 0);
    }
    cudaFreeAsync(img, st);
    return rc;
}

size_t oz64_table_image_bytes(int Kc, int64_t Nc) {
    return (size_t)((Nc + TNC - 1) / TNC) * ((Kc + TK - 1) / TK) * BBYTES;
}
// Image of a table of 2 Kc rows x Nc entries, rows 2 q and 2 q + 1 times 2^wexp[q] (when
// given), and its column exponents EB (Nc).
int oz64_table_image(cudaStream_t st, int Kc, int64_t Nc, const zc* T, const int* wexp, int* EB, void* img) {
    col_exp64_kernel<<<blocks((Nc + 31) / 32), 256, 0, st>>>(1, 2 * Kc, Nc, T, Nc, 0, wexp, EB);
    TBG_LAUNCHED("col_exp64_kernel");
    const int64_t nblk = ((Nc + TNC - 1) / TNC) * ((Kc + TK - 1) / TK);
    table_image_kernel<<<blocks(nblk), B_THREADS, 0, st>>>(Kc, Nc, T, wexp, EB, static_cast<unsigned char*>(img));
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
        a_image_kernel<<<blocks((M + TM - 1) / TM * nst), 256, 0, st>>>(1, (int)M, Kc, coef, ld, 1, 0, 0, EA,
                                                                        static_cast<unsigned char*>(aimg));
        TBG_LAUNCHED("a_image_kernel");
    }
    KTimer kt(st, "oz64_fourier_kernel", 8.0 * (double)M * Nc * Kc);
    OzArgs p = {};
    p.M = (int)M;
    p.Nc = (int)Nc;
    p.A = static_cast<const unsigned char*>(aimg);
    p.B = img;
    p.EA = EA;
    p.EB = EB;
    p.C = C;
    p.ldc = Nc;
    p.err = err;
    p.K = Kc;
    // row tiles fastest: CTAs running together share a column tile's image in L2
    return launch<true>(st, p, 1, 1);
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
