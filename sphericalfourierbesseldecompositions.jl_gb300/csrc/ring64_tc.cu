// FP64 ring Fourier transforms of many maps on the tensor cores, in both
// directions, as digit products (digit64.cuh).
//
// The FFT kernels (ringfft.cu) are bound by the FP64 pipe: about 45 FP64
// operations a pixel at 2 per clock and SM, and 40 percent of them for
// frequencies above lmax that nobody reads.  Here a ring's DFT for m <= lmax is
// four real contractions a quarter as long as the ring.  With pixel j at
// phi_j = (j + 1/2) 2 pi / n (rings shifted by half a pixel) or j 2 pi / n, the
// pixels at phi, -phi, pi - phi and pi + phi share their cosines and sines up to
// signs, so with x0..x3 the values there
//   even m: sum cos = CE . (x0 + x1 + x2 + x3),  sum sin = SE . (x0 - x1 - x2 + x3)
//   odd  m: sum cos = CO . (x0 + x1 - x2 - x3),  sum sin = SO . (x0 - x1 + x2 - x3)
// over the n/4 values of j (n/4 + 1 without the shift, where j = 0 and n/4 are
// their own partners).  The half-pixel phase e^{-i m phi0} is inside the angles,
// so C and -S are the real and imaginary parts of F as they stand.  Frequencies
// above n/2 alias onto k <= n/2 with a sign and are written from there.
//
// Analysis: k_fold64 rounds the pixels of a ring pair to integers on a scale
// common to the pair and map, forms N + S and N - S and the four folded sums
// exactly (64-bit integer additions), k_rdft64 contracts them with digit tables
// of w cos and w sin.  Synthesis: k_rsyn64 contracts the coefficients with cos
// and sin tables into integers, k_unfold64 adds the eight parts of a pixel
// quadruple as integers and rounds each pixel once.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "digit64.cuh"

namespace sfb {
namespace r64 {

using namespace t64;

// chunks per exact block (144 values): the folded sums' leading digit reaches 256, so level v sums v + 2 times 2^14
constexpr int SBR = 9;
static_assert(7 * SBR * KC <= 1 << 10, "levels 0..5 of a block must be exact");
constexpr int KBMAX = 6;       // synthesis: coefficient chunks held at a time (exact as SBK)
static_assert(KBMAX <= SBK, "a block of the synthesis must be exact");

struct Ring {
    int n, shifted, kc, kp, cls;
};
__device__ __forceinline__ Ring ring_of(const RingGeom &g, int r, int ns) {
    Ring o;
    o.n = g.nph;
    o.shifted = g.phi0_den != 0;
    o.kc = o.n / 4 + (o.shifted ? 0 : 1);
    o.kp = (o.kc + KC - 1) & ~(KC - 1);
    o.cls = r < ns - 1 ? r : o.shifted ? ns - 1 : ns;
    return o;
}
// distinct frequencies e + 2 i <= min(lmax, n/2)
__host__ __device__ __forceinline__ int nfreq(int n, int lmax, int e) {
    const int top = lmax < n / 2 ? lmax : n / 2;
    return top >= e ? (top - e) / 2 + 1 : 0;
}
// ring of launch index z: the equatorial rings first (the longest), then the polar ones from the longest
__device__ __forceinline__ int ring_at(int z, int ns) { return z <= ns ? ns - 1 + z : 2 * ns - 1 - z; }

// x on the unit 2^(emax - 1075): 53 bits, so that sums of eight stay within 56
__device__ __forceinline__ int64_t fixed53(double x, int emax) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    int e = (int)(hi >> 20) & 0x7ff;
    const uint64_t mant = ((uint64_t)((hi & 0xfffffu) | (e ? 0x100000u : 0u)) << 32) | lo;
    e = max(e, 1);
    const int64_t q = (int64_t)((((mant << 1) >> min(emax - e, 63)) + 1) >> 1);
    return (int32_t)hi < 0 ? -q : q;
}

// Folded sums of a ring pair: one warp per map.  Q[ring][combination][parity nm + map][kp], ex[ring][map] the
// exponent field of the pair's largest magnitude (0: the pair is zero and its Q not written; 2047: not finite).
// Two passes over the pair's pixels, the second from L1.  Bound: 8 bytes read and about 9 written a pixel.
__global__ void __launch_bounds__(256) k_fold64(const RingGeom *rings, int ns, int64_t npix,
                                                const double *maps, int64_t nm,
                                                const int64_t *qoff, int64_t *Q,
                                                int *ex, int *nzr, int z0) {
    pdl_entry();
    const int r = ring_at(z0 + blockIdx.y, ns), lane = threadIdx.x & 31;
    const int64_t b = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (b >= nm) return;
    const RingGeom g = rings[r];
    const Ring R = ring_of(g, r, ns);
    const bool paired = g.start_s != g.start_n;
    const double *N = maps + b * npix + g.start_n, *S = maps + b * npix + g.start_s;
    uint32_t mx = 0;
    auto mag = [](double v) { return ((uint32_t)__double2hiint(v) & 0x7fffffffu) | (__double2loint(v) != 0 ? 1u : 0u); };
#pragma unroll 4
    for (int j = lane; j < R.n; j += 32) {
        mx = max(mx, mag(N[j]));
        if (paired) mx = max(mx, mag(S[j]));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    const int em = mx == 0 ? 0 : max(1, (int)(mx >> 20));
    if (lane == 0) {
        ex[(int64_t)r * nm + b] = em;
        if (nzr && em) {                 // span of the ring pairs with data
            if (r < *(volatile int *)nzr) atomicMin(nzr, r);
            if (r > *(volatile int *)(nzr + 1)) atomicMax(nzr + 1, r);
        }
    }
    if (em == 0 || em == 2047) return;
    int64_t *q0 = Q + qoff[r] * 2 * nm + b * R.kp;
    const int64_t ldc = 2 * nm * R.kp, ldp = nm * R.kp;
    const int n = R.n;
    for (int j = lane; j < R.kp; j += 32) {
        int64_t p[4] = {0, 0, 0, 0}, d[4] = {0, 0, 0, 0};
        if (j < R.kc) {
            const int sh = R.shifted;
            int i[4] = {j, n - sh - j, n / 2 - sh - j, n / 2 + j};
            if (!sh && j == 0) { i[1] = -1; i[3] = -1; i[2] = n / 2; }
            if (!sh && j == n / 4) { i[2] = -1; i[3] = -1; }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int64_t a = i[t] >= 0 ? fixed53(N[i[t]], em) : 0;
                const int64_t c = i[t] >= 0 && paired ? fixed53(S[i[t]], em) : 0;
                p[t] = a + c;
                d[t] = a - c;
            }
        }
        auto put = [&](int64_t *q, const int64_t (&x)[4]) {
            const int64_t s0 = x[0] + x[1], s1 = x[2] + x[3], d0 = x[0] - x[1], d1 = x[2] - x[3];
            q[j] = s0 + s1;
            q[ldc + j] = s0 - s1;
            q[2 * ldc + j] = d0 - d1;
            q[3 * ldc + j] = d0 + d1;
        };
        put(q0, p);
        put(q0 + ldp, d);
    }
}

// F of 128 rows (parity nm + map) x one tile of 32 frequencies of one combination and ring.
// Bound: MMA issue (about 450 cycles a chunk and tile) beside forming the digits (about 350).
__global__ void __launch_bounds__(NTH, 2) k_rdft64(const RingGeom *rings, int ns, int lmax, int64_t nm,
                                                   const int64_t *qoff, const int64_t *Q,
                                                   const int *ex, const uint16_t *dig,
                                                   const int64_t *off, int Ew, double *F,
                                                   int z0, int *err) {
    pdl_entry();
    extern __shared__ __align__(1024) unsigned char smem[];
    const int r = ring_at(z0 + blockIdx.z, ns), cb = blockIdx.y & 3, tile = blockIdx.y >> 2;
    const int e = cb & 1, isS = cb >> 1;
    const RingGeom g = rings[r];
    const Ring R = ring_of(g, r, ns);
    const int n = R.n, nf = nfreq(n, lmax, e);
    if (tile * NT >= nf) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kh = (tid >> 7) & 1;
    const int64_t nrow = 2 * nm, R0 = (int64_t)blockIdx.x * MTILE, row = R0 + (tid & (MTILE - 1));
    const bool rok = row < nrow;
    const int em0 = rok ? ex[(int64_t)r * nm + (row >= nm ? row - nm : row)] : 0;
    const int LS = ls_of(nf, tile);
    // this thread's output row: warps 0-7, TMEM lanes 32 (w % 4).., every other group of four
    // frequencies of the tile
    const int lq = warp & 3, hg = warp >> 2;
    const int64_t orow = R0 + lq * 32 + lane;
    const bool ook = orow < nrow;
    const int par = orow >= nm ? 1 : 0;
    const int64_t ob = orow - par * nm;
    const int64_t L1 = lmax + 1, ld = 2 * nm;
    double *Fo = F + (par * L1 * 2 * ns + r) * ld + 2 * ob + isS;
    // value v at frequency f: every m <= lmax that aliases onto it
    auto emit = [&](int f, double v, bool add) {
        auto put = [&](int m, double x) {
            double *d = Fo + (int64_t)m * 2 * ns * ld;
            *d = add ? *d + x : x;
        };
        int t = 0;
        for (int m = f; m <= lmax; m += n, ++t) put(m, R.shifted && (t & 1) ? -v : v);
        if (f == 0 || 2 * f == n) return;
        t = 1;
        for (int m = n - f; m <= lmax; m += n, ++t) put(m, (R.shifted && (t & 1)) != (isS != 0) ? -v : v);
    };
    if (!__syncthreads_or(em0 != 0)) {           // no data on this ring pair in any of the maps
        if (ook)
            for (int i = hg; i < NT; i += 2) {
                const int k = tile * NT + i;
                if (k < nf) emit(e + 2 * k, 0.0, false);
            }
        return;
    }
    const bool use = rok && em0 != 0 && em0 != 2047;
    const int64_t *q = Q + qoff[r] * nrow + (int64_t)cb * nrow * R.kp + row * R.kp + 8 * kh;
    const int nch = R.kp / KC;
    const uint16_t *tab = dig + off[4 * R.cls + cb] + (int64_t)tile * nch * ND * NT * KC;
    int64_t pre[2][8];
    auto load = [&](int kc, int64_t (&buf)[8], int) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const longlong2 v = use ? *reinterpret_cast<const longlong2 *>(q + kc * KC + 2 * j) : make_longlong2(0, 0);
            buf[2 * j] = v.x;
            buf[2 * j + 1] = v.y;
        }
    };
    load(0, pre[0], 0);
    if (nch > 1) load(1, pre[1], 1);
    Smem cs;
    const uint32_t tmem = setup(cs, smem);
    const int oem = ook ? ex[(int64_t)r * nm + ob] : 0;
    const int nsb = (nch + SBR - 1) / SBR;
    for (int sb = 0; sb < nsb; ++sb) {
        run_block(cs, tmem, sb * SBR, min(nch, (sb + 1) * SBR), nch, LS, tab, pre, load,
                  [](int64_t v, int, int) { return v; });
        if (!end_block(cs, sb)) {
            if (tid == 0) atomicOr(err, ERR_TC_TIMEOUT);
            break;
        }
        {
#pragma unroll 1
            for (int i0 = 4 * hg; i0 < LS && tile * NT + i0 < nf; i0 += 8) {      // warp-uniform
                float v[ND][4];
                load_levels(tmem + ((uint32_t)(lq * 32) << 16) + (uint32_t)i0, LS, v);
                if (!ook) continue;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int k = tile * NT + i0 + i;
                    if (k >= nf) break;
                    const float L[ND] = {v[0][i], v[1][i], v[2][i], v[3][i], v[4][i], v[5][i], v[6][i]};
                    double x = round_int(join_int(L), oem + Ew - 1074);
                    if (oem == 2047) x = __longlong_as_double(0x7ff8000000000000ll);
                    emit(e + 2 * k, isS ? -x : x, sb > 0);
                }
            }
        }
        fence_before();
        __syncthreads();
        fence_after();
    }
    release(tmem);
}

// Synthesis: 128 coefficient rows (parity nm + map) of one combination and ring, every j.  Their digits are
// formed once (KBMAX chunks of m at a time) and meet the table tiles of 32 j one after another.
// Y[ring][combination][row][kp] += the integers of sum_m c_m G_m cos / sin, shifted right by sh, on the unit of
// gex[ring][combination][row] (the exponent field of the row's largest coefficient).
// Bound: forming the integers (about 45 operations an output) beside the MMAs.
__global__ void __launch_bounds__(NTH, 2) k_rsyn64(const RingGeom *rings, int ns, int lmax, int64_t nm,
                                                   const double *G, const uint16_t *dig,
                                                   const int64_t *off, const int64_t *qoff,
                                                   int64_t *Y, int *gex, int kbmax, int sh,
                                                   int z0, int *err) {
    pdl_entry();
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint32_t red[2][MTILE];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ uint32_t slot;
    const int r = ring_at(z0 + blockIdx.z, ns), cb = blockIdx.y, e = cb & 1, isS = cb >> 1;
    const RingGeom g = rings[r];
    const Ring R = ring_of(g, r, ns);
    const int K = lmax >= e ? (lmax - e) / 2 + 1 : 0;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rl = tid & (MTILE - 1), kh = (tid >> 7) & 1;
    const int64_t nrow = 2 * nm, R0 = (int64_t)blockIdx.x * MTILE, row = R0 + rl;
    const bool rok = row < nrow;
    const int64_t L1 = lmax + 1, ld = 2 * nm;
    const int par = row >= nm ? 1 : 0;
    const double *Gr = G + (par * L1 * 2 * ns + r) * ld + 2 * (row - par * nm) + isS;
    auto at = [&](int k) { return Gr[(int64_t)(e + 2 * k) * 2 * ns * ld]; };
    uint32_t mx = 0;
    if (rok) {
#pragma unroll 8
        for (int k = kh; k < K; k += 2) {
            if (isS && k == 0 && e == 0) continue;            // the imaginary part of m = 0 is not used
            const double v = at(k);
            mx = max(mx, ((uint32_t)__double2hiint(v) & 0x7fffffffu) | (__double2loint(v) != 0 ? 1u : 0u));
        }
    }
    red[kh][rl] = mx;
    uint64_t *full_b = &bars[0], *done = &bars[1];
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        mbar_init(full_b, 1);
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = slot;
    const uint32_t cmx = max(red[0][rl], red[1][rl]);
    const int em = max(1, (int)(cmx >> 20));
    if (tid < MTILE && rok) gex[((int64_t)r * 4 + cb) * nrow + row] = em;
    const bool use = rok && cmx != 0 && em != 2047;
    unsigned char *sA = smem, *sB = smem + (size_t)kbmax * ND * PLANE_A;
    const int nK = (K + KC - 1) / KC, ntile = (R.kc + NT - 1) / NT;
    const uint16_t *tab0 = dig + off[4 * R.cls + cb];
    // table block of tile t, chunks [k0, k0 + nk)
    auto fetch = [&](int t, int k0, int nk) {
        const int LS = ls_of(R.kc, t);
        const uint32_t bytes = (uint32_t)nk * ND * LS * KC * 2;
        mbar_expect_tx(full_b, bytes);
        bulk_g2s(sB, tab0 + (int64_t)t * nK * ND * NT * KC + (int64_t)k0 * ND * LS * KC, bytes, full_b);
    };
    const int lq = warp & 3, hg = warp >> 2;
    const int64_t orow = R0 + lq * 32 + lane;
    int64_t *Yo = Y + qoff[r] * nrow + (int64_t)cb * nrow * R.kp + orow * R.kp;
    const bool ook = orow < nrow;
    int step = 0;
    bool ok = true;
    for (int k0 = 0; k0 < max(nK, 1) && ok; k0 += kbmax) {
        const int nk = min(kbmax, nK - k0);
        if (tid == 0 && nk > 0) fetch(0, k0, nk);
        {
            for (int kc = 0; kc < nk; ++kc) {
                double buf[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int k = (k0 + kc) * KC + 8 * kh + j;
                    buf[j] = use && k < K ? at(k) : 0.0;
                }
                // the table's sine of m = 0 is zero; a non-finite imaginary part there must not enter
                if (isS && e == 0 && k0 + kc == 0 && kh == 0) buf[0] = 0.0;
                uint32_t w[ND][4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint32_t v[ND];
                    digits2(fixed55(buf[2 * j], em), fixed55(buf[2 * j + 1], em), v);
#pragma unroll
                    for (int q = 0; q < ND; ++q) w[q][j] = v[q];
                }
                const uint32_t o = core_off(rl, 8 * kh);
#pragma unroll
                for (int q = 0; q < ND; ++q)
                    *reinterpret_cast<uint4 *>(sA + (kc * ND + q) * PLANE_A + o) =
                        make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
            }
            fence_proxy_async();
        }
        __syncthreads();
        for (int t = 0; t < ntile; ++t, ++step) {
            const int LS = ls_of(R.kc, t);
            if (nk > 0) {
                if (warp == MMA_WARP) {
                    if (lane == 0) {
                        ok = mbar_wait(full_b, (uint32_t)(step & 1));
                        fence_after();
                        if (ok)
                            for (int kc = 0; kc < nk; ++kc)
                                issue(tmem, smem_u32(sA) + kc * ND * PLANE_A, smem_u32(sB) + kc * ND * LS * KC * 2, LS,
                                      kc == 0);
                        mma_commit(done);
                    }
                    __syncwarp();
                }
                const bool fin = mbar_wait(done, (uint32_t)(step & 1));
                fence_after();
                ok = __syncthreads_and(ok && fin);
                if (!ok) {
                    if (tid == 0) atomicOr(err, ERR_TC_TIMEOUT);
                    break;
                }
                if (tid == 0 && t + 1 < ntile) fetch(t + 1, k0, nk);      // the MMAs have read this tile's block
            }
            {
#pragma unroll 1
                for (int i0 = 4 * hg; i0 < LS && t * NT + i0 < R.kc; i0 += 8) {       // warp-uniform
                    const int j0 = t * NT + i0;
                    float v[ND][4];
                    load_levels(tmem + ((uint32_t)(lq * 32) << 16) + (uint32_t)i0, LS, v);
                    if (!ook) continue;
                    int64_t y[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float L[ND] = {v[0][i], v[1][i], v[2][i], v[3][i], v[4][i], v[5][i], v[6][i]};
                        y[i] = nk > 0 ? (join_int(L) + ((1ll << sh) >> 1)) >> sh : 0;
                    }
                    longlong2 *d = reinterpret_cast<longlong2 *>(Yo + j0);
                    if (k0 > 0) {
                        const longlong2 a = d[0], b = d[1];
                        y[0] += a.x; y[1] += a.y; y[2] += b.x; y[3] += b.y;
                    }
                    d[0] = make_longlong2(y[0], y[1]);
                    d[1] = make_longlong2(y[2], y[3]);
                }
            }
            fence_before();
            __syncthreads();
            fence_after();
        }
    }
    release(tmem);
}

// The pixels of ring pair r: one thread per map and four j.  PIXMAJOR: out[pix ld + map] (lanes over maps),
// else out[map ld + pix] (lanes over j).
template <typename T, bool PIXMAJOR>
__global__ void __launch_bounds__(256) k_unfold64(const RingGeom *rings, int ns, int64_t nm,
                                                  const int64_t *qoff, const int64_t *Y,
                                                  const int *gex, int sh, T *out,
                                                  int64_t ld, int z0) {
    pdl_entry();
    const int r = ring_at(z0 + blockIdx.z, ns);
    const RingGeom g = rings[r];
    const Ring R = ring_of(g, r, ns);
    int64_t b;
    int j0;
    if (PIXMAJOR) {
        b = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
        j0 = 4 * (blockIdx.y * 8 + (threadIdx.x >> 5));
    } else {
        b = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
        j0 = 4 * (blockIdx.y * 32 + (threadIdx.x & 31));
    }
    if (b >= nm || j0 >= R.kc) return;
    const int64_t nrow = 2 * nm;
    const int64_t *y0 = Y + qoff[r] * nrow + b * R.kp + j0;
    int em[8], emx = 1;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        em[i] = gex[((int64_t)r * 4 + (i >> 1)) * nrow + (i & 1) * nm + b];
        emx = max(emx, em[i]);
    }
    int64_t v[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const longlong2 *p = reinterpret_cast<const longlong2 *>(y0 + ((int64_t)(i >> 1) * nrow + (i & 1) * nm) * R.kp);
        const longlong2 a = p[0], c = p[1];
        const int s = min(emx - em[i], 63);
        v[i][0] = a.x >> s;
        v[i][1] = a.y >> s;
        v[i][2] = c.x >> s;
        v[i][3] = c.y >> s;
    }
    const int n = R.n, d = R.shifted;
    const bool paired = g.start_s != g.start_n;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int j = j0 + i;
        if (j >= R.kc) break;
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            if (side && !paired) break;
            int64_t c[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) c[q] = side ? v[2 * q][i] - v[2 * q + 1][i] : v[2 * q][i] + v[2 * q + 1][i];
            const int64_t a0 = c[0] + c[1], a1 = c[0] - c[1], s0 = c[2] + c[3], s1 = c[2] - c[3];
            const int64_t start = side ? g.start_s : g.start_n;
            auto put = [&](int pix, int64_t t) {
                const double x = emx == 2047 ? __longlong_as_double(0x7ff8000000000000ll)
                                             : round_int(t, emx - 1075 + sh);
                out[PIXMAJOR ? (start + pix) * ld + b : b * ld + start + pix] = (T)x;
            };
            put(j, a0 - s0);
            if (d || j > 0) put(n - d - j, a0 + s0);
            put(n / 2 - d - j, a1 + s1);
            if (d || j > 0) put(n / 2 + j, a1 - s1);
        }
    }
}

// cos(pi t / n), sin(pi t / n): the angle is reduced to an octant in integers
__device__ __forceinline__ double trig(int64_t t, int n, bool sine) {
    int64_t a = t % (2 * n);                       // [0, 2n)
    double sg = 1.0;
    if (sine) {
        if (a >= n) { a -= n; sg = -1.0; }          // sin(x + pi) = -sin x
        if (2 * a > n) a = n - a;                   // sin(pi - x)
    } else {
        if (a > n) a = 2 * n - a;                   // cos(-x)
        if (2 * a > n) { a = n - a; sg = -1.0; }    // cos(pi - x) = -cos x
    }
    // 0 <= a <= n/2
    const bool swap = 4 * a > n;
    const double x = swap ? (double)(n - 2 * a) / (double)(2 * n) : (double)a / (double)n;
    return sg * (sine != swap ? sinpi(x) : cospi(x));
}

// Table of class cls and combination cb: SYN: rows n = j, columns k = coefficient m = e + 2 k (half weight for
// m = 0); else rows n = frequency e + 2 n, columns k = j, times wm (the quadrature weight's significand).
template <bool SYN>
__global__ void __launch_bounds__(256) k_ring_tab(const RingGeom *rings, int ns, int lmax, double wm,
                                                  const int64_t *off, uint16_t *dig) {
    pdl_entry();
    const int cls = blockIdx.z, cb = blockIdx.y, e = cb & 1;
    const bool sine = cb >> 1;
    int r = cls;
    if (cls >= ns - 1) {                            // the first equatorial ring with that phase
        r = ns - 1;
        if ((rings[r].phi0_den != 0) != (cls == ns - 1)) ++r;
    }
    const Ring R = ring_of(rings[r], r, ns);
    const int n = R.n;
    const int N = SYN ? R.kc : nfreq(n, lmax, e), K = SYN ? (lmax >= e ? (lmax - e) / 2 + 1 : 0) : R.kc;
    const int nK = SYN ? (K + KC - 1) / KC : R.kp / KC;
    const int ntile = (N + NT - 1) / NT;
    for (int blk = blockIdx.x; blk < ntile * nK; blk += gridDim.x) {
        const int tile = blk / nK, kc = blk % nK;
        const int LS = ls_of(N, tile);
        uint16_t *base = dig + off[4 * cls + cb] + (int64_t)tile * nK * ND * NT * KC + (int64_t)kc * ND * LS * KC;
        for (int el = threadIdx.x; el < LS * KC; el += 256) {
            const int nn = el / KC, k = el % KC;
            const int in = tile * NT + nn, ik = kc * KC + k;
            int64_t q = 0;
            if (in < N && ik < K) {
                const int m = e + 2 * (SYN ? ik : in), j = SYN ? in : ik;
                const double c = trig((int64_t)m * (2 * j + R.shifted), n, sine) * (SYN ? (m == 0 ? 0.5 : 1.0) : wm);
                q = llrint(ldexp(c, 55));
            }
            uint32_t w[ND];
            digits2(q, 0, w);
#pragma unroll
            for (int d = 0; d < ND; ++d) base[(int64_t)d * LS * KC + (core_off(nn, k) >> 1)] = (uint16_t)(w[d] & 0xffffu);
        }
    }
}

}  // namespace r64

// Digit tables of the ring transforms (dir 0: analysis, 1: synthesis), made at the first use that finds the memory;
// false: the FFT kernels do this call (tables above a sixteenth of the free device memory) or every one (an nside
// below 2, or SFBGPU_RING64=0).
static bool ensure_ring64(Plan &p, int dir, cudaStream_t st) {
    if (p.ring64_state[dir]) return p.ring64_state[dir] > 0;
    const int ns = (int)p.nside;
    const char *e = std::getenv("SFBGPU_RING64");
    if (ns < 2 || (e && e[0] == '0')) {
        p.ring64_state[dir] = -1;
        return false;
    }
    std::vector<int64_t> off;
    int64_t o = 0;
    for (int cls = 0; cls <= ns; ++cls) {
        const int n = cls < ns - 1 ? 4 * (cls + 1) : 4 * ns;
        const int kc = n / 4 + (cls == ns ? 1 : 0);
        for (int cb = 0; cb < 4; ++cb) {
            const int e = cb & 1;
            const int N = dir ? kc : r64::nfreq(n, p.lmax, e), K = dir ? (p.lmax >= e ? (p.lmax - e) / 2 + 1 : 0) : kc;
            const int64_t nK = (K + t64::KC - 1) / t64::KC;
            off.push_back(o);
            for (int t = 0; t * t64::NT < N; ++t) o += nK * t64::ND * t64::ls_of(N, t) * t64::KC;
        }
    }
    std::vector<int64_t> qoff(p.nrn + 1, 0);
    for (int64_t r = 0; r < p.nrn; ++r) {
        const int kc = p.h_rings[r].nph / 4 + (p.h_rings[r].phi0_den ? 0 : 1);
        qoff[r + 1] = qoff[r] + 4 * ((kc + t64::KC - 1) / t64::KC) * t64::KC;
    }
    p.ring64_row = qoff[p.nrn];
    const size_t bt = ((size_t)o * 2 + 511) & ~(size_t)255, bo = (off.size() + qoff.size()) * sizeof(int64_t);
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) != cudaSuccess || bt > fr / 16) {
        cudaGetLastError();
        return false;
    }
    unsigned char *d = nullptr;
    if (cudaMalloc(&d, bt + bo) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    auto give_back = [&] {
        cudaGetLastError();
        cudaFree(d);
        return false;
    };
    int64_t *doff = reinterpret_cast<int64_t *>(d + bt), *dq = doff + off.size();
    if (cudaMemcpyAsync(doff, off.data(), off.size() * sizeof(int64_t), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(dq, qoff.data(), qoff.size() * sizeof(int64_t), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return give_back();
    p.ring64_dig[dir] = reinterpret_cast<uint16_t *>(d);
    p.ring64_off[dir] = doff;
    p.ring64_qoff[dir] = dq;
    int Ew = 0;
    const double wm = std::frexp(4.0 * M_PI / (double)p.npix, &Ew);
    p.ring64_ew = Ew;
    const dim3 grid(64, 4, (unsigned)(ns + 1));
    if (dir) launch_pdl(r64::k_ring_tab<true>, dim3(grid), dim3(256), 0, st, p.d_rings, ns, p.lmax, 1.0, doff,
        p.ring64_dig[1]);
    else launch_pdl(r64::k_ring_tab<false>, dim3(grid), dim3(256), 0, st, p.d_rings, ns, p.lmax, wm, doff,
        p.ring64_dig[0]);
    note_launch();
    if (cudaGetLastError() != cudaSuccess) return give_back();
    p.ring64_mem[dir] = d;
    p.device_bytes += (int64_t)(bt + bo);
    p.ring64_state[dir] = 1;
    return true;
}

// room for the integers of nm maps and their exponents; false without memory
static bool ring64_room(Plan &p, int64_t nm, int *&ex) {
    const size_t q = (size_t)(2 * nm * p.ring64_row), e = (size_t)(p.nrn * 8 * nm + 1) / 2 + 1;
    if (grow(p, p.ring64, q + e) != SFB_OK) return false;
    ex = reinterpret_cast<int *>(p.ring64.ptr + q);
    return true;
}

bool launch_ring_analysis64(Plan &p, const double *maps, int64_t nm, double *F, cudaStream_t st, int *nzr, int z0,
                            int nz) {
    int *ex = nullptr;
    if (nz < 0) nz = (int)p.nrn;
    if (!ensure_ring64(p, 0, st) || !ring64_room(p, nm, ex)) return false;
    const int ns = (int)p.nside;
    int64_t *Q = reinterpret_cast<int64_t *>(p.ring64.ptr);
    launch_pdl(r64::k_fold64, dim3((unsigned)((nm + 7) / 8), (unsigned)nz), dim3(256), 0, st, p.d_rings, ns, p.npix,
        maps, nm, p.ring64_qoff[0], Q, ex, nzr, z0);
    const int ntile = (r64::nfreq(4 * ns, p.lmax, 0) + t64::NT - 1) / t64::NT;
    set_smem(r64::k_rdft64, t64::SMEM);
    launch_pdl(r64::k_rdft64,
        dim3((unsigned)((2 * nm + t64::MTILE - 1) / t64::MTILE), (unsigned)(4 * ntile), (unsigned)nz), dim3(t64::NTH),
        t64::SMEM, st, p.d_rings, ns, p.lmax, nm, p.ring64_qoff[0], Q, ex, p.ring64_dig[0], p.ring64_off[0],
        p.ring64_ew, F, z0, p.d_err);
    note_launch();
    note_launch();
    return true;
}

// Ring synthesis into maps out[map ld + pixel] or, pixel-major, out[pixel ld + map] of double or float.
bool launch_ring_synthesis64(Plan &p, const double *G, int64_t nm, void *out, int64_t ld, bool pixmajor, bool f32,
                             cudaStream_t st, int z0, int nz) {
    int *ex = nullptr;
    if (nz < 0) nz = (int)p.nrn;
    if (!ensure_ring64(p, 1, st) || !ring64_room(p, nm, ex)) return false;
    const int ns = (int)p.nside;
    int64_t *Y = reinterpret_cast<int64_t *>(p.ring64.ptr);
    const int K = p.lmax / 2 + 1, nK = (K + t64::KC - 1) / t64::KC;
    const int kb = nK <= 3 ? nK : std::min(nK, r64::KBMAX);       // up to three chunks: two CTAs per SM
    // the sum of eight integers below 2^(54 - sh) K stays within 63 bits
    int sh = 0;
    while (K >= (64 << sh)) ++sh;
    const size_t smem = (size_t)kb * t64::ND * (t64::PLANE_A + t64::NT * t64::KC * 2);
    set_smem(r64::k_rsyn64, smem);
    launch_pdl(r64::k_rsyn64, dim3((unsigned)((2 * nm + t64::MTILE - 1) / t64::MTILE), 4, (unsigned)nz),
        dim3(t64::NTH), smem, st, p.d_rings, ns, p.lmax, nm, G, p.ring64_dig[1], p.ring64_off[1], p.ring64_qoff[1], Y,
        ex, kb, sh, z0, p.d_err);
    const int kcmax = ns + 1;
    if (pixmajor) {
        const dim3 grid((unsigned)((nm + 31) / 32), (unsigned)((kcmax + 31) / 32), (unsigned)nz);
        if (f32)
            launch_pdl(r64::k_unfold64<float, true>, dim3(grid), dim3(256), 0, st, p.d_rings, ns, nm,
                p.ring64_qoff[1], Y, ex, sh, (float *)out, ld, z0);
        else
            launch_pdl(r64::k_unfold64<double, true>, dim3(grid), dim3(256), 0, st, p.d_rings, ns, nm,
                p.ring64_qoff[1], Y, ex, sh, (double *)out, ld, z0);
    } else {
        const dim3 grid((unsigned)((nm + 7) / 8), (unsigned)((kcmax + 127) / 128), (unsigned)nz);
        launch_pdl(r64::k_unfold64<double, false>, dim3(grid), dim3(256), 0, st, p.d_rings, ns, nm, p.ring64_qoff[1],
            Y, ex, sh, (double *)out, ld, z0);
    }
    note_launch();
    note_launch();
    return true;
}

}  // namespace sfb
