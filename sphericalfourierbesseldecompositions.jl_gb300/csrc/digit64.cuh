// FP64 products on the tensor cores by 8-bit digits: the pieces that
// the Legendre (leg64_tc.cu) and ring (ring64_tc.cu) contractions share.
//
// A value is a 55-bit integer on a common scale, written as seven signed 8-bit
// digits that BF16 holds exactly; the digit products of level v = a + b (v =
// 0..6) are summed in one FP32 TMEM accumulator per level, exactly for v <= 5
// over at most SBK chunks of K, and the levels are joined as a 62-bit integer.
#pragma once

#include <cuda_bf16.h>

#include "sfb_internal.h"
#include "tc_common.cuh"

namespace sfb {
namespace t64 {

using namespace tc;

constexpr int ND = 7;                                  // digits, and levels kept
constexpr int KC = 16;                                 // K per chunk (one MMA K step)
constexpr int MTILE = 128;                             // data columns per CTA
constexpr int NT = LEG64_TILE;                         // table rows per CTA
constexpr int SBK = 10;                                // chunks per exact K block (160 values)
// A digit product is at most 2^14 and level v joins v + 1 of them: levels 0..5 of a block stay within the 2^24 up to
// which FP32 holds every integer.  A unit of level v is 2^(-14 - 8 v) of the scales, so level 4 and 5 have to be exact
// (2^-46, 2^-54); the roundings of level 6 (2^-61 each) stay below 2^-54 together.
static_assert(6 * SBK * KC <= 1 << 10, "levels 0..5 of a block must be exact");
static_assert(SBK % 2 == 0, "a block begins with the first of the two buffers");
// eight warps: a ninth for the MMAs would leave 96 registers a thread at two CTAs per SM instead of 128
constexpr int NTH = 256;
constexpr int MMA_WARP = NTH / 32 - 1;
constexpr uint32_t PLANE_A = MTILE * KC * 2;
constexpr int NSTAGE = 3;
constexpr uint32_t STAGE_BYTES = ND * (PLANE_A + NT * KC * 2);
constexpr uint32_t TMEM_COLS = 256;                    // 7 x 32 levels
constexpr size_t SMEM = NSTAGE * (size_t)STAGE_BYTES + 256;

__host__ __device__ __forceinline__ int ls_of(int n, int tile) {      // padded table rows of a tile
    const int left = n - tile * NT;
    return left >= NT ? NT : (left + 15) & ~15;
}
__device__ __forceinline__ uint32_t core_off(int row, int k) {
    return (uint32_t)((((row >> 3) * (KC / 8) + (k >> 3)) << 7) + ((row & 7) << 4) + ((k & 7) << 1));
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float (&v)[4]) {
    uint32_t r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}

// x on the unit 2^(emax - 1077): a 55-bit integer plus sign, rounded to nearest
// (emax: exponent field of the column's largest magnitude, |x| < 2^(emax - 1022))
__device__ __forceinline__ int64_t fixed55(double x, int emax) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    int e = (int)(hi >> 20) & 0x7ff;
    uint64_t mant = ((uint64_t)((hi & 0xfffffu) | (e ? 0x100000u : 0u)) << 32) | lo;
    e = max(e, 1);
    const uint32_t s = min((uint32_t)(emax - e), 63u);       // (a zero may come with e above emax)
    const int64_t q = (int64_t)((((mant << 3) >> s) + 1) >> 1);
    return (int32_t)hi < 0 ? -q : q;
}

// The digits of two integers as bf16x2 words, most significant first.  With 128 added to the six lower
// digits the bytes of the sum are the digits plus 128; a byte becomes a float through the mantissa of 2^23.
__device__ __forceinline__ void digits2(int64_t q0, int64_t q1, uint32_t (&w)[ND]) {
    constexpr int64_t BIAS = 0x0000808080808080LL;
    q0 += BIAS;
    q1 += BIAS;
    auto top = [](int64_t q) { return __int_as_float(0x4B400000 + (int)(q >> 48)) - 12582912.0f; };
    auto dig = [](int64_t q, int s) {
        const uint32_t half = s >= 4 ? (uint32_t)((uint64_t)q >> 32) : (uint32_t)q;
        return __uint_as_float(__byte_perm(half, 0x4B000000u, 0x7650u | (uint32_t)(s & 3))) - 8388736.0f;
    };
    w[0] = bf16x2(top(q0), top(q1));
#pragma unroll
    for (int s = 5; s >= 0; --s) w[6 - s] = bf16x2(dig(q0, s), dig(q1, s));
}

// sum_v L_v 2^(40 - 8 v)
__device__ __forceinline__ int64_t join_int(const float (&L)[ND]) {
    auto i = [](float v) { return __float2int_rn(v); };
    auto wide = [](int a, int b, int64_t c) { return (int64_t)a * b + c; };
    const int64_t H = wide(i(L[0]), 1 << 24, wide(i(L[1]), 1 << 16, wide(i(L[2]), 1 << 8, (int64_t)i(L[3]))));
    const int64_t W = wide(i(L[4]), 1 << 16, wide(i(L[5]), 1 << 8, (int64_t)(i(L[6]) + 128)));
    return (H << 16) + (W >> 8);
}

// T 2^S rounded to FP64 (integer operations: the FP64 pipe would take 16 cycles a warp for each one)
__device__ __forceinline__ double round_int(int64_t T, int S) {
    const uint32_t sign = (uint32_t)((uint64_t)T >> 32) & 0x80000000u;
    const uint64_t a = T < 0 ? (uint64_t)(-T) : (uint64_t)T;
    const int lz = __clzll((long long)a);
    const uint64_t frac = (((a << lz) >> 1) + 512u) >> 10;            // 2^52 <= frac <= 2^53
    const int ef = 11 - lz + S + 52 + 1023;                            // exponent field of frac 2^(11 - lz + S)
    if (a == 0) return 0.0;
    if (ef < 1 || ef > 2045) {                     // subnormal or overflowing: two scalings of the rounded value
        auto pow2 = [](int e) { return __hiloint2double((1023 + max(-1022, min(e, 1023))) << 20, 0); };
        const int e = 11 - lz + S, e1 = e / 2;
        const double v = (double)(int64_t)frac * pow2(e1) * pow2(e - e1);
        return sign ? -v : v;
    }
    const uint32_t hi = (uint32_t)(frac >> 32) + ((uint32_t)(ef - 1) << 20);
    return __hiloint2double((int)(hi | sign), (int)(uint32_t)frac);
}

struct Smem {
    unsigned char *base;
    uint64_t *full_a, *full_b, *empty, *done;
    uint32_t *slot;
    int *bad;
    __device__ __forceinline__ unsigned char *stage(int s) const { return base + s * STAGE_BYTES; }
};

__device__ __forceinline__ uint32_t setup(Smem &c, unsigned char *base) {
    c.base = base;
    c.full_a = reinterpret_cast<uint64_t *>(base + NSTAGE * STAGE_BYTES);
    c.full_b = c.full_a + NSTAGE;
    c.empty = c.full_b + NSTAGE;
    c.done = c.empty + NSTAGE;
    c.slot = reinterpret_cast<uint32_t *>(c.done + 1);
    c.bad = reinterpret_cast<int *>(c.slot + 1);
    if ((threadIdx.x >> 5) == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(c.slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < NSTAGE; ++i) {
            mbar_init(&c.full_a[i], NTH / 32);
            mbar_init(&c.full_b[i], 1);
            mbar_init(&c.empty[i], 1);
        }
        mbar_init(c.done, 1);
        *c.bad = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    return *c.slot;
}

// the products of one chunk: data digit a with the table digits 0..6-a, level a + b
__device__ __forceinline__ void issue(uint32_t tmem, uint32_t sa, uint32_t sb, int LS, bool first) {
    const uint32_t sbo = (KC / 8) * 128;
    const uint32_t planeB = (uint32_t)LS * KC * 2;
    const int per = 256 / LS;                             // table digits one MMA can take
    for (int a = 0; a < ND; ++a) {
        const uint64_t ad = smem_desc(sa + a * PLANE_A, 128, sbo);
        for (int b = 0; b < ND - a; b += per) {
            const int nb = min(per, ND - a - b);
            mma_bf16(tmem + (uint32_t)(LS * (a + b)), ad, smem_desc(sb + b * planeB, 128, sbo),
                     idesc_bf16(MTILE, LS * nb), (first && a == 0) ? 0u : 1u);
        }
    }
}

// One exact K block, chunks [k0, k1) of nch, up to its last MMA's issue: every warp turns its values
// into digits (load(kc, buf, i): this thread's eight values of chunk kc, row tid % 128, k = 8 (tid / 128)..; fix(v, i,
// j): value j of them as the integer; i is the buffer, pre[i]), the table digits of chunk kc come from tab + kc ND LS
// KC, and the last warp issues a chunk's MMAs once all have written theirs.  pre holds the values of chunks k0 and k0 + 1 on entry (in this
// order: an odd block swaps them at its end).  end_block waits for the MMAs.
template <typename T, typename Load, typename Fix>
__device__ __forceinline__ void run_block(const Smem &cs, uint32_t tmem, int k0, int k1, int nch, int LS,
                                          const uint16_t *tab, T (&pre)[2][8], const Load &load, const Fix &fix) {
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t bytesB = (uint32_t)ND * LS * KC * 2;
    const uint32_t off = core_off(tid & (MTILE - 1), 8 * (tid >> 7));
    auto chunk = [&](int kc, T (&cur)[8], int i) -> bool {
        const int s = kc % NSTAGE;
        if (kc >= NSTAGE) {
            if (*(volatile int *)cs.bad) return false;
            if (!mbar_wait(&cs.empty[s], (uint32_t)((kc / NSTAGE - 1) & 1))) {
                atomicExch(cs.bad, 1);
                return false;
            }
        }
        unsigned char *sa = cs.stage(s);
        if (tid == 0) {
            mbar_expect_tx(&cs.full_b[s], bytesB);
            bulk_g2s(sa + ND * PLANE_A, tab + (int64_t)kc * ND * LS * KC, bytesB, &cs.full_b[s]);
        }
        uint32_t w[ND][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t v[ND];
            digits2(fix(cur[2 * j], i, 2 * j), fix(cur[2 * j + 1], i, 2 * j + 1), v);
#pragma unroll
            for (int q = 0; q < ND; ++q) w[q][j] = v[q];
        }
#pragma unroll
        for (int q = 0; q < ND; ++q)
            *reinterpret_cast<uint4 *>(sa + q * PLANE_A + off) = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
        if (kc + 2 < nch) load(kc + 2, cur, i);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(&cs.full_a[s]);
            if (tid == 32 * MMA_WARP) {
                const uint32_t ph = (uint32_t)((kc / NSTAGE) & 1);
                if (!mbar_wait(&cs.full_a[s], ph) || !mbar_wait(&cs.full_b[s], ph)) {
                    atomicExch(cs.bad, 1);
                } else {
                    fence_after();
                    const uint32_t a = smem_u32(sa);
                    issue(tmem, a, a + ND * PLANE_A, LS, kc == k0);
                    mma_commit(&cs.empty[s]);
                }
            }
        }
        __syncwarp();
        return true;
    };
    for (int kc = k0; kc < k1; kc += 2) {
        if (!chunk(kc, pre[0], 0)) break;
        if (kc + 1 < k1 && !chunk(kc + 1, pre[1], 1)) break;
    }
    if (tid == 32 * MMA_WARP) mma_commit(cs.done);          // arrives once every MMA issued above has completed
    __syncwarp();
    if (k1 < nch && ((k1 - k0) & 1)) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const T v = pre[0][j];
            pre[0][j] = pre[1][j];
            pre[1][j] = v;
        }
    }
}

// Every MMA of block sb is complete; false when a wait gave up.
__device__ __forceinline__ bool end_block(const Smem &cs, int sb) {
    const bool ok = mbar_wait(cs.done, (uint32_t)(sb & 1));
    fence_after();
    return __syncthreads_and(ok) && !*(volatile int *)cs.bad;
}

__device__ __forceinline__ void release(uint32_t tmem) {
    fence_before();
    __syncthreads();
    if ((threadIdx.x >> 5) == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
}

// four TMEM columns of every level from column i0 on
__device__ __forceinline__ void load_levels(uint32_t taddr, int LS, float (&v)[ND][4]) {
#pragma unroll
    for (int q = 0; q < ND; ++q) tmem_ld4(taddr + (uint32_t)(q * LS), v[q]);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace t64
}  // namespace sfb
