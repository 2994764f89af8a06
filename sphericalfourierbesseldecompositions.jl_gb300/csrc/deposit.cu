// Galaxy deposit without floating-point atomics.
//
// The deposit D_b[p] = sum_{i in p} w_i phi_b(r_i) is organised as a counting
// sort of the galaxies by key = slot * npix + pixel, where slot is the radial
// piece (0..pieces-1) or one of the two out-of-range slots (r < rmin,
// r > rmax):
//   1. keys:    per galaxy, pixel (bit-exact HEALPix), slot and local
//               coordinate x in [-1, 1]; an int atomic on the key's counter
//               gives the galaxy its rank inside the bin;
//   2. scan:    exclusive prefix sum of the (pieces + 2) * npix counters;
//   3. scatter: (x, w) to its sorted position;
//   4. moments: one thread per (slot, pixel) sums w P_k(x) over its galaxies
//               (mixed precision: in its own shared-memory column) and every
//               basis map element is written exactly once (coalesced over
//               consecutive pixels; empty bins write zeros, so the maps need
//               no clearing).
// Summation order inside a bin follows the int-atomic ranks, so repeated
// calls agree to rounding, not bit for bit.
//
// Mixed precision runs no FP64 instruction per galaxy (integer range tests and
// double-float splits; the records are double-float pairs) and stores the
// maps as double-float pairs (hi, lo), which the ring DFT slices exactly.
// With a reference angular map C, each map is written as the fluctuation
// D_b - mu_b C, with mu_b = <D_b, C> / <C, C> estimated in double-float (sums
// in FP64) on every STATS_STRIDE-th group of 32 bins; the caller adds
// mu_b C_lm back in FP64 after the transform.  Rings holding no galaxy are
// then left unwritten (ring_live), their readers treating them as zero.
// C is the weighted galaxy count map of all radial slots, so it carries the
// mean density and the survey boundary exactly as the galaxies sample them
// (a pixelised mask misses the partly covered boundary pixels).  The reduced
// precision of the transform then scales with the fluctuation, not with the
// mean density that the window term later cancels.
#include <algorithm>
#include <cstring>

#include "sfb_internal.h"

namespace sfb {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;                    // per thread
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

// Bin offsets as the scan leaves them: a prefix within the bin's tile and the tile's own.  The readers add the two
// (the tiles' few values stay in L1), which spares a pass over the counters (48 us for 11.8 million).
struct Offsets {
    const int32_t *in_tile, *tile;
    int64_t first;
    __device__ __forceinline__ int32_t operator[](int64_t i) const {
        const uint64_t k = (uint64_t)(first + i);
        return in_tile[k] + tile[k / SCAN_TILE];
    }
};

// Double-float arithmetic (value = hi + lo, |lo| <= ulp(hi)/2): ~48
// significant bits from FP32 operations, whose throughput on this GPU is
// many times that of FP64.  TwoSum / TwoProd with FMA (Dekker, Knuth).
struct dfl {
    float hi, lo;
};

__device__ __forceinline__ dfl df_of(double x) {
    const float h = (float)x;
    return {h, (float)(x - (double)h)};
}

__device__ __forceinline__ dfl df_add(dfl a, dfl b) {
    const float s = a.hi + b.hi;
    const float z = s - a.hi;
    const float e = ((a.hi - (s - z)) + (b.hi - z)) + (a.lo + b.lo);
    const float h = s + e;
    return {h, e - (h - s)};
}

__device__ __forceinline__ dfl df_mul(dfl a, dfl b) {
    const float p = a.hi * b.hi;
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, e));
    const float h = p + e;
    return {h, e - (h - p)};
}

__device__ __forceinline__ dfl df_neg(dfl a) { return {-a.hi, -a.lo}; }

// The same without the final renormalisation (|lo| may reach a few ulp of
// hi): for chains that renormalise where it matters.
__device__ __forceinline__ dfl dfs_mul(dfl a, dfl b) {
    const float p = a.hi * b.hi;
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, e));
    return {p, e};
}

__device__ __forceinline__ dfl dfs_add(dfl a, dfl b) {
    const float s = a.hi + b.hi;
    const float z = s - a.hi;
    return {s, ((a.hi - (s - z)) + (b.hi - z)) + (a.lo + b.lo)};
}

__device__ __forceinline__ dfl df_renorm(dfl a) {
    const float h = a.hi + a.lo;
    return {h, a.lo - (h - a.hi)};
}

__device__ __forceinline__ dfl df_of_bits(double d) {
    const float2 v = df_split_bits(d);
    return {v.x, v.y};
}

// IEEE order of finite doubles as signed 64-bit integers (-0 and +0 both 0),
// for range tests without FP64 compares.
__host__ __device__ __forceinline__ long long ord_of(double d) {
    long long b;
    memcpy(&b, &d, 8);
    return b >= 0 ? b : -(b & 0x7fffffffffffffffll);
}

__device__ __forceinline__ bool finite_bits(double d) {
    return (((unsigned long long)__double_as_longlong(d) >> 52) & 0x7ffu) != 0x7ffu;
}

// Slot and local coordinate of radius r: u = (r - rmin) / width in units of
// the pieces (inv_width = pieces / (rmax - rmin), formed once on the host),
// x in [-1, 1] on the piece; slots pieces / pieces + 1 below / above.
__device__ __forceinline__ int slot_of(double r, double rmin, double rmax, double inv_width, int pieces, double &x) {
    x = 0.0;
    if (r < rmin) return pieces;
    if (r > rmax) return pieces + 1;
    const double u = (r - rmin) * inv_width;
    int slot = (int)u;
    if (slot >= pieces) slot = pieces - 1;
    x = 2.0 * (u - (double)slot) - 1.0;
    x = fmin(1.0, fmax(-1.0, x));
    return slot;
}

// Mock of galaxy i (global index): the last j with off[j] <= i.
__device__ __forceinline__ int mock_of(const Mocks &mk, int64_t i) {
    int lo = 0, hi = mk.n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (mk.off[mid] <= i) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Keys of galaxies [0, ngal) of this chunk (global index gbase + i); mock j's slots are j (pieces + 2) + ....  A galaxy
// whose pixel the FP32 evaluation cannot settle goes to fb_list with key
// -2 - slot, and gets its key and rank from k_deposit_keys_fallback (FP64
// pixel), so no warp runs the FP64 pixel path for one lane.
__global__ void k_deposit_keys(const double *rtp, const double *wgt, int64_t ngal,
                               int64_t gbase, int64_t nside, int64_t npix, double rmin, double rmax,
                               double inv_width, int pieces, const __grid_constant__ Mocks mk, int32_t *counts,
                               int32_t *key, int32_t *rank, double *xloc,
                               int32_t *fb_list, int32_t *fb_count, int *err) {
    pdl_entry();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ngal) return;
    const double r = rtp[3 * i], th = rtp[3 * i + 1], ph = rtp[3 * i + 2];
    const double w = wgt ? wgt[i] : 1.0;
    int32_t k = -1;
    double x = 0.0;
    if (!(isfinite(r) && isfinite(th) && isfinite(ph) && isfinite(w))) {
        atomicOr(err, ERR_NONFINITE_INPUT);
    } else if (th < 0.0 || th > M_PI) {
        atomicOr(err, ERR_THETA_RANGE);
    } else {
        const int64_t pix = ang2pix_ring_try(nside, th, ph);
        const int slot = slot_of(r, rmin, rmax, inv_width, pieces, x) + mock_of(mk, gbase + i) * (pieces + 2);
        if (pix >= 0) {
            k = (int32_t)(slot * npix + pix);
            rank[i] = atomicAdd(counts + k, 1);
        } else {
            k = -2 - slot;
            fb_list[atomicAdd(fb_count, 1)] = (int32_t)(gbase + i);
        }
    }
    key[i] = k;
    xloc[i] = x;
}

// Mixed precision keys, with no FP64 instruction: the range tests compare the
// IEEE order of the doubles as integers, theta and phi are rounded to FP32 by
// integer operations for the FP32 pixel evaluation, and the local coordinate
// comes from the double-float split of r (x to ~1e-13, as a float2 pair).
// Slot boundaries follow u = (r - rmin) inv_width in double-float, so a
// galaxy within ~1e-13 of a piece boundary may take the neighbouring piece
// (at x = +-1, where both pieces represent the radial functions).
struct RadialKeyParams {
    long long ord_rmin, ord_rmax;      // ord_of(rmin), ord_of(rmax)
    float rmin_hi, rmin_lo, invw_hi, invw_lo;
};

__global__ void k_deposit_keys_mixed(const double *rtp, const double *wgt, int64_t ngal,
                                     int64_t gbase, int64_t nside, int64_t npix, RadialKeyParams rk, int pieces,
                                     const __grid_constant__ Mocks mk, int32_t *counts, int32_t *key,
                                     int32_t *rank, float2 *xdf,
                                     int32_t *fb_list, int32_t *fb_count, int *err) {
    pdl_entry();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ngal) return;
    const double r = rtp[3 * i], th = rtp[3 * i + 1], ph = rtp[3 * i + 2];
    const bool wfin = wgt ? finite_bits(wgt[i]) : true;
    constexpr long long ORD_PI = 0x400921fb54442d18ll;          // bits of M_PI
    constexpr long long ORD_4PI = 0x402921fb54442d18ll;         // bits of 4 M_PI
    int32_t k = -1;
    float2 x = make_float2(0.f, 0.f);
    if (!(finite_bits(r) && finite_bits(th) && finite_bits(ph) && wfin)) {
        atomicOr(err, ERR_NONFINITE_INPUT);
    } else {
        const long long oth = ord_of(th);
        if (oth < 0 || oth > ORD_PI) {
            atomicOr(err, ERR_THETA_RANGE);
        } else {
            const long long orr = ord_of(r);
            int slot;
            if (orr < rk.ord_rmin) {
                slot = pieces;
            } else if (orr > rk.ord_rmax) {
                slot = pieces + 1;
            } else {
                const dfl u = df_mul(df_add(df_of_bits(r), {-rk.rmin_hi, -rk.rmin_lo}), {rk.invw_hi, rk.invw_lo});
                float fl = floorf(u.hi);
                if (fl == u.hi && u.lo < 0.f) fl -= 1.f;
                slot = min(max((int)fl, 0), pieces - 1);
                const dfl d = df_add(u, {-(float)slot, 0.f});              // in [0, 1] up to rounding
                dfl xx = df_add({2.f * d.hi, 2.f * d.lo}, {-1.f, 0.f});
                if (xx.hi > 1.f || (xx.hi == 1.f && xx.lo > 0.f)) xx = {1.f, 0.f};
                if (xx.hi < -1.f || (xx.hi == -1.f && xx.lo < 0.f)) xx = {-1.f, 0.f};
                x = make_float2(xx.hi, xx.lo);
            }
            slot += mock_of(mk, gbase + i) * (pieces + 2);
            const long long phabs = __double_as_longlong(ph) & 0x7fffffffffffffffll;
            const int64_t pix = (nside <= (int64_t(1) << 16) && phabs <= ORD_4PI)
                                    ? ang2pix_ring_try32(nside, df_of_bits(th).hi, df_of_bits(ph).hi)
                                    : -1;
            if (pix >= 0) {
                k = (int32_t)(slot * npix + pix);
                rank[i] = atomicAdd(counts + k, 1);
            } else {
                k = -2 - slot;
                fb_list[atomicAdd(fb_count, 1)] = (int32_t)(gbase + i);
            }
        }
    }
    key[i] = k;
    xdf[i] = x;
}

// The galaxies the FP32 pixel evaluation left: exact FP64 pixel, then key and
// rank as above with the slot the keys pass found (rtp, key, rank indexed
// globally).
__global__ void k_deposit_keys_fallback(const double *rtp, int64_t nside, int64_t npix,
                                        int32_t *counts, int32_t *key,
                                        int32_t *rank, const int32_t *fb_list,
                                        const int32_t *fb_count) {
    pdl_entry();
    const int n = *fb_count;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int64_t i = fb_list[t];
        const double th = rtp[3 * i + 1], ph = rtp[3 * i + 2];
        const int64_t pix = ang2pix_ring_z(nside, cos(th), ph);
        const int slot = -2 - key[i];
        const int32_t k = (int32_t)(slot * npix + pix);
        rank[i] = atomicAdd(counts + k, 1);
        key[i] = k;
    }
}

// Exclusive scan, tile pass: each block scans SCAN_TILE counters in place and
// writes its total; the block that finishes last (counted in *done, zero on
// entry) scans the totals, so that step costs no launch of its own.
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_tiles(int32_t *data, int64_t n,
                                                             int32_t *tile_sums, int *done) {
    pdl_entry();
    __shared__ int32_t warp_tot[SCAN_THREADS / 32];
    __shared__ int32_t carry;
    __shared__ bool last;
    const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_ITEMS;
    alignas(16) int32_t v[SCAN_ITEMS];
    int32_t s = 0;
    const bool whole = base + SCAN_ITEMS <= n;             // (data is on a 16-byte boundary: launch_exclusive_scan)
    if (whole) {
#pragma unroll
        for (int j = 0; j < SCAN_ITEMS; j += 4)
            *reinterpret_cast<int4 *>(v + j) = *reinterpret_cast<const int4 *>(data + base + j);
    } else {
#pragma unroll
        for (int j = 0; j < SCAN_ITEMS; ++j) v[j] = base + j < n ? data[base + j] : 0;
    }
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) s += v[j];
    // exclusive scan of thread sums across the block
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int32_t inc = s;
    for (int off = 1; off < 32; off <<= 1) {
        const int32_t t = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += t;
    }
    if (lane == 31) warp_tot[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int32_t wv = lane < SCAN_THREADS / 32 ? warp_tot[lane] : 0;
        for (int off = 1; off < 32; off <<= 1) {
            const int32_t t = __shfl_up_sync(0xffffffffu, wv, off);
            if (lane >= off) wv += t;
        }
        if (lane < SCAN_THREADS / 32) warp_tot[lane] = wv;   // inclusive warp prefix
    }
    __syncthreads();
    int32_t run = inc - s + (wid > 0 ? warp_tot[wid - 1] : 0);
    alignas(16) int32_t o[SCAN_ITEMS];
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) {
        o[j] = run;
        run += v[j];
    }
    if (whole) {
#pragma unroll
        for (int j = 0; j < SCAN_ITEMS; j += 4)
            *reinterpret_cast<int4 *>(data + base + j) = *reinterpret_cast<const int4 *>(o + j);
    } else {
#pragma unroll
        for (int j = 0; j < SCAN_ITEMS; ++j)
            if (base + j < n) data[base + j] = o[j];
    }
    if (threadIdx.x == SCAN_THREADS - 1) {
        tile_sums[blockIdx.x] = run;
        __threadfence();
        last = atomicAdd(done, 1) == (int)gridDim.x - 1;
        carry = 0;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int64_t c0 = 0; c0 < gridDim.x; c0 += SCAN_TILE) {
        const int64_t b0 = c0 + (int64_t)threadIdx.x * SCAN_ITEMS;
        s = 0;
#pragma unroll
        for (int j = 0; j < SCAN_ITEMS; ++j) {
            v[j] = b0 + j < gridDim.x ? __ldcg(tile_sums + b0 + j) : 0;
            s += v[j];
        }
        inc = s;
        for (int off = 1; off < 32; off <<= 1) {
            const int32_t t = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += t;
        }
        __syncthreads();
        if (lane == 31) warp_tot[wid] = inc;
        __syncthreads();
        run = carry + inc - s;
        for (int w = 0; w < wid; ++w) run += warp_tot[w];
#pragma unroll
        for (int j = 0; j < SCAN_ITEMS; ++j) {
            if (b0 + j < gridDim.x) tile_sums[b0 + j] = run;
            run += v[j];
        }
        __syncthreads();
        if (threadIdx.x == SCAN_THREADS - 1) carry = run;
        __syncthreads();
    }
}

__global__ void k_scan_add(int32_t *data, int64_t n, const int32_t *tile_sums) {
    pdl_entry();
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < n) data[idx] += tile_sums[idx / SCAN_TILE];
}

__global__ void k_deposit_scatter(const double *wgt, int64_t ngal, const int32_t *key,
                                  const int32_t *rank, const double *xloc,
                                  Offsets offset, double2 *sorted) {
    pdl_entry();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ngal) return;
    const int32_t k = key[i];
    if (k < 0) return;
    const int64_t pos = (int64_t)offset[k] + rank[i];
    sorted[pos] = make_double2(xloc[i], wgt ? wgt[i] : 1.0);
}

// Mixed precision: (x, w) as double-float pairs {x.hi, x.lo, w.hi, w.lo}, w
// split from the double by integer operations.
__global__ void k_deposit_scatter_mixed(const double *wgt, int64_t ngal,
                                        const int32_t *key, const int32_t *rank,
                                        const float2 *xdf, Offsets offset,
                                        float4 *sorted) {
    pdl_entry();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ngal) return;
    const int32_t k = key[i];
    if (k < 0) return;
    const int64_t pos = (int64_t)offset[k] + rank[i];
    const float2 x = xdf[i];
    const dfl w = wgt ? df_of_bits(wgt[i]) : dfl{1.f, 0.f};
    sorted[pos] = make_float4(x.x, x.y, w.hi, w.lo);
}

// Legendre moments sum_i w_i P_k(x_i), k <= deg, of the galaxies g0..g1-1 of one bin, in FP64.  The
// recurrence runs on the monic polynomials r_{k+1} = x r_k - k^2/(4k^2 - 1) r_{k-1}, weighted from the start
// (three FP64 operations a degree and galaxy instead of four; the FP64 pipe bounds this), and each sum is
// scaled by P_k's leading coefficient once.
constexpr double monic_lead(int k) {
    double c = 1.0;
    for (int j = 1; j <= k; ++j) c *= (2.0 * j - 1.0) / j;
    return c;
}

template <int MAXDEG>
__device__ __forceinline__ void bin_moments(const double2 *sorted, int64_t g0, int64_t g1, int deg,
                                            double (&acc)[MAXDEG + 1]) {
#pragma unroll
    for (int k = 0; k <= MAXDEG; ++k) acc[k] = 0.0;
    double2 nxt = g0 < g1 ? sorted[g0] : make_double2(0.0, 0.0);
    for (int64_t g = g0; g < g1; ++g) {
        const double2 xw = nxt;
        if (g + 1 < g1) nxt = sorted[g + 1];
        const double x = xw.x;
        double p0 = xw.y, p1 = xw.y * x;
        acc[0] += p0;
        if (MAXDEG >= 1) acc[1] += p1;
#pragma unroll
        for (int k = 1; k < MAXDEG; ++k) {
            if (k >= deg) break;
            const double p2 = fma(x, p1, -((double)(k * k) / (4.0 * k * k - 1.0)) * p0);
            acc[k + 1] += p2;
            p0 = p1;
            p1 = p2;
        }
    }
#pragma unroll
    for (int k = 2; k <= MAXDEG; ++k) acc[k] *= monic_lead(k);
}

__device__ __forceinline__ int64_t basis_of(int slot, int k, int pieces, int deg, int64_t nbasis) {
    return slot < pieces ? (int64_t)slot * (deg + 1) + k : nbasis - 2 + (slot - pieces);
}

// Order the block's 128 bins by decreasing galaxy count (a counting sort in shared memory), so the threads of
// a warp walk bins of nearly equal length: the position of this thread's bin in that order.
__device__ __forceinline__ int rank_bins(int cnt, int *hist) {
    const int t = threadIdx.x;
    if (t < 64) hist[t] = 0;
    __syncthreads();
    const int key = 63 - min(cnt, 63);                 // longest bins first
    atomicAdd(&hist[key], 1);
    __syncthreads();
    if (t < 32) {
        const int h0 = hist[2 * t], h1 = hist[2 * t + 1];
        int sc = h0 + h1;
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sc, off);
            if (t >= off) sc += v;
        }
        const int base = sc - (h0 + h1);
        hist[2 * t] = base;
        hist[2 * t + 1] = base + h0;
    }
    __syncthreads();
    return atomicAdd(&hist[key], 1);
}

// FP64: one thread per (slot, pixel) bin, the bins handed out by decreasing count, the results written with
// consecutive threads on consecutive pixels.  Bound: the FP64 pipe, 72 operations a galaxy at degree 24 (with
// four operations a degree and unsorted bins 274 us for 6e5 galaxies at nside 128; 151 so).
template <int MAXDEG>
__global__ void __launch_bounds__(128) k_deposit_moments(Offsets offset,
                                                         const double2 *sorted, int64_t npix, int pieces,
                                                         int deg, int64_t nbasis, double *maps) {
    pdl_entry();
    extern __shared__ double out_s[];                  // [deg + 1][128]
    __shared__ int hist[64];
    __shared__ int perm[128];
    // grid.y: mocks
    offset.first += (int64_t)blockIdx.y * (pieces + 2) * npix;
    maps += (int64_t)blockIdx.y * nbasis * npix;
    const int t = threadIdx.x;
    const int64_t nkeys = (int64_t)(pieces + 2) * npix;
    const int64_t bt = (int64_t)blockIdx.x * 128 + t;
    const int cnt = bt < nkeys ? offset[bt + 1] - offset[bt] : 0;        // offset[nkeys] = number of keyed galaxies
    const int slot = bt < nkeys ? (int)(bt / npix) : 0;
    const int64_t pix = bt - (int64_t)slot * npix;
    const int64_t b0 = slot < pieces ? (int64_t)slot * (deg + 1) : nbasis - 2 + (slot - pieces);
    const int nk = slot < pieces ? deg + 1 : 1;        // one constant map for r < rmin, one for r > rmax
    double *base = maps + b0 * npix + pix;
    if (!__syncthreads_or(cnt != 0)) {
        if (bt < nkeys)
            for (int k = 0; k < nk; ++k) base[(int64_t)k * npix] = 0.0;
        return;
    }
    perm[rank_bins(cnt, hist)] = t;
    __syncthreads();
    {
        const int q = perm[t];
        const int64_t b = (int64_t)blockIdx.x * 128 + q;
        if (b < nkeys) {
            const int64_t g0 = offset[b], g1 = offset[b + 1];
            if (b / npix >= pieces) {
                double s = 0.0;
                for (int64_t g = g0; g < g1; ++g) s += sorted[g].y;
                out_s[q] = s;
            } else {
                double acc[MAXDEG + 1];
                bin_moments<MAXDEG>(sorted, g0, g1, deg, acc);
#pragma unroll
                for (int k = 0; k <= MAXDEG; ++k)
                    if (k <= deg) out_s[k * 128 + q] = acc[k];
            }
        }
    }
    __syncthreads();
    if (bt < nkeys)
        for (int k = 0; k < nk; ++k) base[(int64_t)k * npix] = out_s[k * 128 + t];
}

// One step of the basis recurrence on q_k = w P_k(x):
// (k+1) q_{k+1} = (2k+1) x q_k - k q_{k-1}, the ratios as double-float
// constants, every operation unnormalised: where the sum cancels, lo keeps
// its absolute accuracy (~2^-46 of the terms), which is all the moments need
// before their FP32 store.
template <int K>
__device__ __forceinline__ dfl leg_step(dfl x, dfl q1, dfl q0) {
    constexpr double C1 = (double)(2 * K + 1) / (K + 1), C2 = -(double)K / (K + 1);
    constexpr float C1H = (float)C1, C2H = (float)C2;
    constexpr float C1L = (float)(C1 - (double)C1H), C2L = (float)(C2 - (double)C2H);
    return dfs_add(dfs_mul({C1H, C1L}, dfs_mul(x, q1)), dfs_mul({C2H, C2L}, q0));
}

// acc[k+1] += q_{k+1} for K <= k < min(deg, MAXDEG), q0 = q_{K-1}, q1 = q_K
template <int K, int MAXDEG>
__device__ __forceinline__ void leg_chain(dfl x, dfl q0, dfl q1, dfl (&acc)[MAXDEG + 1], int deg) {
    if constexpr (K < MAXDEG) {
        if (K >= deg) return;
        const dfl q2 = leg_step<K>(x, q1, q0);
        acc[K + 1] = dfs_add(acc[K + 1], q2);
        leg_chain<K + 1, MAXDEG>(x, q1, q2, acc, deg);
    }
}

// Moments sum_g w_g P_k(x_g), k <= deg, of one bin in double-float, from the
// pairs of k_deposit_scatter_mixed; the next galaxy's load overlaps this
// one's basis.
template <int MAXDEG>
__device__ __forceinline__ void bin_moments_df(const float4 *sorted, int64_t g0, int64_t g1, int deg,
                                               dfl (&acc)[MAXDEG + 1]) {
#pragma unroll
    for (int k = 0; k <= MAXDEG; ++k) acc[k] = {0.f, 0.f};
    float4 nxt = g0 < g1 ? sorted[g0] : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int64_t g = g0; g < g1; ++g) {
        const float4 v = nxt;
        if (g + 1 < g1) nxt = sorted[g + 1];
        const dfl x = {v.x, v.y};
        dfl q0 = {v.z, v.w}, q1 = dfs_mul(q0, x);
        acc[0] = dfs_add(acc[0], q0);
        if (MAXDEG >= 1) acc[1] = dfs_add(acc[1], q1);
        leg_chain<1, MAXDEG>(x, q0, q1, acc, deg);
    }
#pragma unroll
    for (int k = 0; k <= MAXDEG; ++k) acc[k] = df_renorm(acc[k]);
}

// Mixed precision, one thread per (slot, pixel): the moments and the
// fluctuation acc - mu_b ref all in double-float (mudf = mu and cdf = ref as
// hi + lo pairs), stored as normalised double-float pairs.
template <int MAXDEG>
__global__ void k_deposit_moments_df(Offsets offset, const float4 *sorted,
                                     int64_t npix, int pieces, int deg, int64_t nbasis, const float2 *cdf,
                                     const float2 *mudf, float2 *maps) {
    pdl_entry();
    // grid.y: mocks
    offset.first += (int64_t)blockIdx.y * (pieces + 2) * npix;
    maps += (int64_t)blockIdx.y * nbasis * npix;
    if (cdf) {
        cdf += blockIdx.y * npix;
        mudf += blockIdx.y * nbasis;
    }
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t nkeys = (int64_t)(pieces + 2) * npix;
    if (idx >= nkeys) return;
    const int slot = (int)(idx / npix);
    const int64_t pix = idx - (int64_t)slot * npix;
    const int64_t g0 = offset[idx];
    const int64_t g1 = offset[idx + 1];
    const float2 c = cdf ? cdf[pix] : make_float2(0.f, 0.f);
    const dfl rv = {c.x, c.y};
    auto fluct = [&](dfl a, int64_t b) -> float2 {
        if (cdf) {
            const float2 m = mudf[b];
            a = dfs_add(a, df_neg(dfs_mul({m.x, m.y}, rv)));
        }
        a = df_renorm(a);
        return make_float2(a.hi, a.lo);
    };
    if (slot >= pieces) {
        dfl sw = {0.f, 0.f};
        for (int64_t g = g0; g < g1; ++g) {
            const float4 v = sorted[g];
            sw = df_add(sw, {v.z, v.w});
        }
        const int64_t b = nbasis - 2 + (slot - pieces);
        maps[b * npix + pix] = fluct(sw, b);
        return;
    }
    dfl acc[MAXDEG + 1];
    bin_moments_df<MAXDEG>(sorted, g0, g1, deg, acc);
    const int64_t b0 = (int64_t)slot * (deg + 1);
    float2 *base = maps + b0 * npix + pix;
#pragma unroll
    for (int k = 0; k <= MAXDEG; ++k)
        if (k <= deg) base[(int64_t)k * npix] = fluct(acc[k], b0 + k);
}

// The same moments with the block's bins handed to its threads in order of
// decreasing galaxy count (a counting sort of the 128 counts in shared
// memory), so the threads of a warp walk bins of nearly equal length instead
// of waiting on the longest bin of 32 neighbours.  The basis values are
// carried as q_k = w P_k(x) (leg_step).  Results pass through shared memory
// and are written with consecutive threads on consecutive pixels.  Needs
// npix >= 128 (a block spans at most two slots).
template <int MAXDEG>
__global__ void __launch_bounds__(128) k_deposit_moments_bal(Offsets offset,
                                                             const float4 *sorted, int64_t npix,
                                                             int pieces, int deg, int64_t nbasis,
                                                             const float2 *cdf,
                                                             const float2 *mudf,
                                                             float2 *maps, int64_t nside,
                                                             const int *ring_live) {
    pdl_entry();
    __shared__ int hist[64];
    __shared__ int perm[128];
    __shared__ float2 out[(MAXDEG + 1) * 128];
    // grid.y: mocks
    offset.first += (int64_t)blockIdx.y * (pieces + 2) * npix;
    maps += (int64_t)blockIdx.y * nbasis * npix;
    if (cdf) {
        cdf += blockIdx.y * npix;
        mudf += blockIdx.y * nbasis;
    }
    if (ring_live) ring_live += blockIdx.y * (4 * nside - 1);
    const int t = threadIdx.x;
    const int64_t nkeys = (int64_t)(pieces + 2) * npix;
    const int64_t B0 = (int64_t)blockIdx.x * 128;
    const int slot0 = (int)(B0 / npix);
    const int64_t bnd = (int64_t)(slot0 + 1) * npix;
    const int64_t bt = B0 + t;
    const int cnt = bt < nkeys ? offset[bt + 1] - offset[bt] : 0;
    // blocks of empty bins on pixels where the reference map is zero (outside the survey) write zeros
    bool busy = cnt != 0;
    if (cdf && bt < nkeys) {
        const int sl = bt < bnd ? slot0 : slot0 + 1;
        busy = busy || cdf[bt - (int64_t)sl * npix].x != 0.f;
    }
    if (!__syncthreads_or(busy)) {
        if (bt >= nkeys) return;
        const int sl = bt < bnd ? slot0 : slot0 + 1;
        const int64_t px = bt - (int64_t)sl * npix;
        // rings without galaxies are not written at all (their readers treat them as zero)
        if (ring_live && !ring_live[ring_of_pixel(nside, px)]) return;
        if (sl >= pieces) {
            maps[(nbasis - 2 + (sl - pieces)) * npix + px] = make_float2(0.f, 0.f);
            return;
        }
        float2 *z = maps + (int64_t)sl * (deg + 1) * npix + px;
        for (int k = 0; k <= deg; ++k) z[(int64_t)k * npix] = make_float2(0.f, 0.f);
        return;
    }
    perm[rank_bins(cnt, hist)] = t;
    __syncthreads();
    const int q = perm[t];
    const int64_t b = B0 + q;
    if (b < nkeys) {
        const int slot = b < bnd ? slot0 : slot0 + 1;
        const int64_t pix = b - (int64_t)slot * npix;
        const int64_t g0 = offset[b], g1 = offset[b + 1];
        const float2 c = cdf ? cdf[pix] : make_float2(0.f, 0.f);
        const dfl rv = {c.x, c.y};
        auto fluct = [&](dfl a, int64_t bi) -> float2 {
            if (cdf) {
                const float2 m = mudf[bi];
                a = dfs_add(a, df_neg(dfs_mul({m.x, m.y}, rv)));
            }
            a = df_renorm(a);
            return make_float2(a.hi, a.lo);
        };
        if (slot >= pieces) {
            dfl sw = {0.f, 0.f};
            for (int64_t g = g0; g < g1; ++g) {
                const float4 v = sorted[g];
                sw = df_add(sw, {v.z, v.w});
            }
            out[q] = fluct(sw, nbasis - 2 + (slot - pieces));
        } else {
            dfl acc[MAXDEG + 1];
            bin_moments_df<MAXDEG>(sorted, g0, g1, deg, acc);
            const int64_t bb = (int64_t)slot * (deg + 1);
#pragma unroll
            for (int k = 0; k <= MAXDEG; ++k)
                if (k <= deg) out[k * 128 + q] = fluct(acc[k], bb + k);
        }
    }
    __syncthreads();
    if (bt >= nkeys) return;
    const int slot = bt < bnd ? slot0 : slot0 + 1;
    const int64_t pix = bt - (int64_t)slot * npix;
    if (slot >= pieces) {
        maps[(nbasis - 2 + (slot - pieces)) * npix + pix] = out[t];
        return;
    }
    float2 *base = maps + (int64_t)slot * (deg + 1) * npix + pix;
    for (int k = 0; k <= deg; ++k) base[(int64_t)k * npix] = out[k * 128 + t];
}

// Shared-memory accumulators for the balanced moments (the default): thread t
// keeps the double-float sums of the bin it walks in column t of acc_s (one
// float2 per degree) instead of 25 register pairs, so a thread needs 48
// registers instead of 117 and twice the warps are resident to cover the
// dependent loads (offsets -> records) and the recurrence's latency.  The
// accesses are explicit shared-memory instructions (volatile asm), so the
// compiler cannot move the sums back into registers.  The arithmetic is that
// of k_deposit_moments_bal operation for operation: for the same order of the
// galaxies within each bin both kernels write the same bits.
__device__ __forceinline__ float2 lds2(uint32_t a) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
    return v;
}

__device__ __forceinline__ void sts2(uint32_t a, float2 v) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y));
}

// column stride of acc_s between degrees: 128 float2
constexpr uint32_t ACC_DEG_BYTES = 128 * 8;

template <int K, int MAXDEG>
__device__ __forceinline__ void leg_chain_sm(dfl x, dfl q0, dfl q1, uint32_t col, int deg) {
    if constexpr (K < MAXDEG) {
        if (K >= deg) return;
        const uint32_t a = col + (K + 1) * ACC_DEG_BYTES;
        const float2 s = lds2(a);
        const dfl q2 = leg_step<K>(x, q1, q0);
        const dfl r = dfs_add({s.x, s.y}, q2);
        sts2(a, make_float2(r.hi, r.lo));
        leg_chain_sm<K + 1, MAXDEG>(x, q1, q2, col, deg);
    }
}

template <int MAXDEG>
__device__ __forceinline__ void bin_moments_sm(const float4 *sorted, int64_t g0, int64_t g1, int deg,
                                               uint32_t col) {
#pragma unroll
    for (int k = 0; k <= MAXDEG; ++k)
        if (k <= deg) sts2(col + k * ACC_DEG_BYTES, make_float2(0.f, 0.f));
    float4 nxt = g0 < g1 ? sorted[g0] : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int64_t g = g0; g < g1; ++g) {
        const float4 v = nxt;
        if (g + 1 < g1) nxt = sorted[g + 1];
        const dfl x = {v.x, v.y};
        const dfl q0 = {v.z, v.w}, q1 = dfs_mul(q0, x);
        float2 s = lds2(col);
        dfl r = dfs_add({s.x, s.y}, q0);
        sts2(col, make_float2(r.hi, r.lo));
        if (MAXDEG >= 1 && deg >= 1) {
            s = lds2(col + ACC_DEG_BYTES);
            r = dfs_add({s.x, s.y}, q1);
            sts2(col + ACC_DEG_BYTES, make_float2(r.hi, r.lo));
        }
        leg_chain_sm<1, MAXDEG>(x, q0, q1, col, deg);
    }
}

template <int MAXDEG>
__global__ void __launch_bounds__(128, 8) k_deposit_moments_sm(Offsets offset,
                                                               const float4 *sorted, int64_t npix,
                                                               int pieces, int deg, int64_t nbasis,
                                                               const float2 *cdf,
                                                               const float2 *mudf,
                                                               float2 *maps, int64_t nside,
                                                               const int *ring_live) {
    pdl_entry();
    __shared__ int hist[64];
    __shared__ int perm[128];
    __shared__ __align__(16) float2 acc_s[(MAXDEG + 1) * 128];
    // grid.y: mocks
    offset.first += (int64_t)blockIdx.y * (pieces + 2) * npix;
    maps += (int64_t)blockIdx.y * nbasis * npix;
    if (cdf) {
        cdf += blockIdx.y * npix;
        mudf += blockIdx.y * nbasis;
    }
    if (ring_live) ring_live += blockIdx.y * (4 * nside - 1);
    const int t = threadIdx.x;
    const int64_t nkeys = (int64_t)(pieces + 2) * npix;
    const int64_t B0 = (int64_t)blockIdx.x * 128;
    const int slot0 = (int)(B0 / npix);
    const int64_t bnd = (int64_t)(slot0 + 1) * npix;
    const int64_t bt = B0 + t;
    const int cnt = bt < nkeys ? offset[bt + 1] - offset[bt] : 0;
    bool busy = cnt != 0;
    if (cdf && bt < nkeys) {
        const int sl = bt < bnd ? slot0 : slot0 + 1;
        busy = busy || cdf[bt - (int64_t)sl * npix].x != 0.f;
    }
    if (!__syncthreads_or(busy)) {
        if (bt >= nkeys) return;
        const int sl = bt < bnd ? slot0 : slot0 + 1;
        const int64_t px = bt - (int64_t)sl * npix;
        if (ring_live && !ring_live[ring_of_pixel(nside, px)]) return;
        if (sl >= pieces) {
            maps[(nbasis - 2 + (sl - pieces)) * npix + px] = make_float2(0.f, 0.f);
            return;
        }
        float2 *z = maps + (int64_t)sl * (deg + 1) * npix + px;
        for (int k = 0; k <= deg; ++k) z[(int64_t)k * npix] = make_float2(0.f, 0.f);
        return;
    }
    const int walker = rank_bins(cnt, hist);           // the thread that walks this thread's bin
    perm[walker] = t;
    __syncthreads();
    const uint32_t acc0 = (uint32_t)__cvta_generic_to_shared(acc_s);
    {
        const int64_t b = B0 + perm[t];
        if (b < nkeys) {
            const int slot = b < bnd ? slot0 : slot0 + 1;
            const int64_t g0 = offset[b], g1 = offset[b + 1];
            const uint32_t col = acc0 + t * 8;
            if (slot >= pieces) {
                dfl sw = {0.f, 0.f};
                for (int64_t g = g0; g < g1; ++g) {
                    const float4 v = sorted[g];
                    sw = df_add(sw, {v.z, v.w});
                }
                sts2(col, make_float2(sw.hi, sw.lo));
            } else {
                bin_moments_sm<MAXDEG>(sorted, g0, g1, deg, col);
            }
        }
    }
    __syncthreads();
    if (bt >= nkeys) return;
    // thread t writes its own bin (consecutive threads on consecutive pixels) from the walker's column
    const int slot = bt < bnd ? slot0 : slot0 + 1;
    const int64_t pix = bt - (int64_t)slot * npix;
    const uint32_t src = acc0 + walker * 8;
    const float2 c = cdf ? cdf[pix] : make_float2(0.f, 0.f);
    const dfl rv = {c.x, c.y};
    auto fluct = [&](dfl a, int64_t bi) -> float2 {
        if (cdf) {
            const float2 m = mudf[bi];
            a = dfs_add(a, df_neg(dfs_mul({m.x, m.y}, rv)));
        }
        a = df_renorm(a);
        return make_float2(a.hi, a.lo);
    };
    if (slot >= pieces) {
        const float2 s = lds2(src);
        const int64_t b = nbasis - 2 + (slot - pieces);
        maps[b * npix + pix] = fluct({s.x, s.y}, b);
        return;
    }
    const int64_t bb = (int64_t)slot * (deg + 1);
    float2 *base = maps + bb * npix + pix;
    for (int k = 0; k <= deg; ++k) {
        const float2 s = lds2(src + k * ACC_DEG_BYTES);
        base[(int64_t)k * npix] = fluct(df_renorm({s.x, s.y}), bb + k);
    }
}

constexpr int STATS_STRIDE = 32;

// Sampled projections onto ref over the bins of every STATS_STRIDE-th group of
// 32 bins (one warp per block): S[b] += <D_b, ref>, Q[slot] += <ref, ref>,
// with ref as the double-float pairs cdf.  A slot-uniform warp reduces
// through shared memory in double-float (lane k sums column k) and adds the
// column sums in FP64; a warp that straddles two slots adds per thread.  The
// block that finishes last (*done zero on entry) forms mu[b] = S[b] / Q[slot(b)]
// (0 where the sampled reference map is zero) and the same as a double-float pair.
template <int MAXDEG>
__global__ void __launch_bounds__(32) k_deposit_stats(Offsets offset,
                                                      const float4 *sorted, int64_t npix, int pieces,
                                                      int deg, int64_t nbasis, const float2 *cdf,
                                                      double *S, double *Q, double *mu,
                                                      float2 *mudf, int *done) {
    pdl_entry();
    __shared__ float2 red[32][MAXDEG + 3];
    // grid.y: mocks
    offset.first += (int64_t)blockIdx.y * (pieces + 2) * npix;
    cdf += blockIdx.y * npix;
    double *const S0 = S, *const Q0 = Q;
    S += blockIdx.y * nbasis;
    Q += blockIdx.y * (pieces + 2);
    const int lane = threadIdx.x;
    const int64_t idx = (int64_t)blockIdx.x * STATS_STRIDE * 32 + lane;
    const int64_t nkeys = (int64_t)(pieces + 2) * npix;
    const bool valid = idx < nkeys;
    const int slot = valid ? (int)(idx / npix) : -1;
    const int64_t pix = valid ? idx - (int64_t)slot * npix : 0;
    const float2 c = valid ? cdf[pix] : make_float2(0.f, 0.f);
    const dfl rv = {c.x, c.y};
    const unsigned full = 0xffffffffu;
    const bool any = __any_sync(full, c.x != 0.f);  // (a group whose reference is zero adds nothing)
    dfl acc[MAXDEG + 1];
    if (any && valid) {
        bin_moments_df<MAXDEG>(sorted, offset[idx], offset[idx + 1], slot < pieces ? deg : 0, acc);
    } else {
#pragma unroll
        for (int k = 0; k <= MAXDEG; ++k) acc[k] = {0.f, 0.f};
    }
    const int nk = slot < 0 ? 0 : (slot < pieces ? deg + 1 : 1);
    const int slot0 = __shfl_sync(full, slot, 0);
    auto to_d = [](dfl a) { return (double)a.hi + (double)a.lo; };
    if (!any) {
    } else if (__all_sync(full, slot == slot0)) {   // (a group is never without a valid bin)
#pragma unroll
        for (int k = 0; k <= MAXDEG; ++k)
            if (k < nk) {
                const dfl v = df_mul(acc[k], rv);
                red[lane][k] = make_float2(v.hi, v.lo);
            }
        const dfl rr = df_mul(rv, rv);
        red[lane][nk] = make_float2(rr.hi, rr.lo);
        __syncwarp();
        for (int k = lane; k <= nk; k += 32) {
            dfl v = {0.f, 0.f};
            for (int j = 0; j < 32; ++j) v = df_add(v, {red[j][k].x, red[j][k].y});
            if (k < nk) atomicAdd(S + basis_of(slot0, k, pieces, deg, nbasis), to_d(v));
            else atomicAdd(Q + slot0, to_d(v));
        }
    } else if (valid) {
#pragma unroll
        for (int k = 0; k <= MAXDEG; ++k)
            if (k < nk) atomicAdd(S + basis_of(slot, k, pieces, deg, nbasis), to_d(df_mul(acc[k], rv)));
        atomicAdd(Q + slot, to_d(df_mul(rv, rv)));
    }
    __threadfence();
    __syncwarp();
    int last = 0;
    if (lane == 0) last = atomicAdd(done, 1) == (int)(gridDim.x * gridDim.y) - 1;
    if (!__shfl_sync(full, last, 0)) return;
    __threadfence();
    const int64_t npoly = (int64_t)pieces * (deg + 1);
    const int64_t nmu = nbasis * gridDim.y;
    for (int64_t i0 = lane; i0 < nmu; i0 += 8 * 32) {
        double sv[8], qv[8];                             // eight loads on their way at a time
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const int64_t i = min(i0 + 32 * t, nmu - 1), mock = i / nbasis, b = i - mock * nbasis;
            const int sl = b < npoly ? (int)b / (deg + 1) : pieces + (int)(b - npoly);
            sv[t] = __ldcg(S0 + i);
            qv[t] = __ldcg(Q0 + mock * (pieces + 2) + sl);
        }
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const int64_t i = i0 + 32 * t;
            if (i >= nmu) break;
            const double v = qv[t] > 0.0 ? sv[t] / qv[t] : 0.0;
            mu[i] = v;
            const float h = (float)v;
            mudf[i] = make_float2(h, (float)(v - (double)h));
        }
    }
}

// Weighted galaxy count per pixel over all radial slots (the reference map of
// the mixed deposit), in double-float from the sorted pairs, stored as the
// FP64 value hi + lo (exact) and as the pair itself.
// ring_live[ring] is set to 1 for every ring holding a galaxy (preset to 0).
// The window's reference map W01 goes behind the count maps.
__global__ void k_weight_map_mixed(Offsets offset, const float4 *sorted,
                                   int64_t nside, int64_t npix, int nslots, double *C,
                                   float2 *cdf, int *ring_live,
                                   const double *W01) {
    pdl_entry();
    const int64_t pix = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= npix) return;
    // grid.y: mocks
    if (W01 && blockIdx.y == 0) C[gridDim.y * npix + pix] = W01[pix];
    offset.first += (int64_t)blockIdx.y * nslots * npix;
    C += blockIdx.y * npix;
    cdf += blockIdx.y * npix;
    ring_live += blockIdx.y * (4 * nside - 1);
    dfl s = {0.f, 0.f};
    bool any = false;
    for (int sl = 0; sl < nslots; ++sl) {
        const int64_t k = (int64_t)sl * npix + pix;
        const int64_t g0 = offset[k], g1 = offset[k + 1];
        any = any || g1 > g0;
        for (int64_t g = g0; g < g1; ++g) {
            const float4 v = sorted[g];
            s = df_add(s, {v.z, v.w});
        }
    }
    C[pix] = (double)s.hi + (double)s.lo;
    cdf[pix] = make_float2(s.hi, s.lo);
    if (any) ring_live[ring_of_pixel(nside, pix)] = 1;
}

// FP64 path: double (x, w); mixed: double-float pairs and the count map as cdf
template <int MAXDEG>
static void launch_moments(const Plan &p, int nmock, Offsets offset, const void *sorted, const float2 *cdf,
                           const float2 *mudf, double *maps, cudaStream_t st, const int *ring_live) {
    const int64_t nkeys = (int64_t)(p.pieces + 2) * p.npix;
    const dim3 blocks((unsigned)((nkeys + 127) / 128), (unsigned)nmock);
    const float4 *s4 = static_cast<const float4 *>(sorted);
    float2 *mf = reinterpret_cast<float2 *>(maps);
    bool done = false;
    if constexpr (MAXDEG <= 31) {
        if (p.precision == SFB_MIXED && p.npix >= 128) {
            if (p.moments_smem)
                launch_pdl(k_deposit_moments_sm<MAXDEG>, dim3(blocks), dim3(128), 0, st, offset, s4, p.npix, p.pieces,
                    p.degree, p.nbasis, cdf, mudf, mf, p.nside, ring_live);
            else
                launch_pdl(k_deposit_moments_bal<MAXDEG>, dim3(blocks), dim3(128), 0, st, offset, s4, p.npix,
                    p.pieces, p.degree, p.nbasis, cdf, mudf, mf, p.nside, ring_live);
            done = true;
        }
    }
    if (done) {
    } else if (p.precision == SFB_MIXED)
        launch_pdl(k_deposit_moments_df<MAXDEG>, dim3(blocks), dim3(128), 0, st, offset, s4, p.npix, p.pieces,
            p.degree, p.nbasis, cdf, mudf, mf);
    else {
        const size_t smem = (size_t)(p.degree + 1) * 128 * sizeof(double);
        set_smem(k_deposit_moments<MAXDEG>, smem);
        launch_pdl(k_deposit_moments<MAXDEG>, dim3(blocks), dim3(128), smem, st, offset,
            static_cast<const double2 *>(sorted), p.npix, p.pieces, p.degree, p.nbasis, maps);
    }
    note_launch();
}

template <int MAXDEG>
static void launch_stats(const Plan &p, int nmock, Offsets offset, const float4 *sorted, const float2 *cdf, double *S,
                         double *Q, double *mu, float2 *mudf, int *done, cudaStream_t st) {
    const int64_t nkeys = (int64_t)(p.pieces + 2) * p.npix;
    const int64_t blocks = (nkeys + 32 * STATS_STRIDE - 1) / (32 * STATS_STRIDE);
    launch_pdl(k_deposit_stats<MAXDEG>, dim3((unsigned)blocks, (unsigned)nmock), dim3(32), 0, st, offset, sorted,
        p.npix, p.pieces, p.degree, p.nbasis, cdf, S, Q, mu, mudf, done);
    note_launch();
}

// the moment kernels' degree instances: 15, 24 (the default radial basis), 31, 63
template <typename F>
static void by_degree(int deg, F &&f) {
    if (deg <= 15) f(std::integral_constant<int, 15>());
    else if (deg <= 24) f(std::integral_constant<int, 24>());
    else if (deg <= 31) f(std::integral_constant<int, 31>());
    else f(std::integral_constant<int, 63>());
}

int64_t scan_tile_count(int64_t n) { return (n + SCAN_TILE - 1) / SCAN_TILE; }

void launch_exclusive_scan(int32_t *data, int64_t n, int32_t *tile_sums, int *done, cudaStream_t st) {
    const int64_t ntiles = scan_tile_count(n);
    launch_pdl(k_scan_tiles, dim3((unsigned)ntiles), dim3(SCAN_THREADS), 0, st, data, n, tile_sums, done);
    note_launch();
    launch_pdl(k_scan_add, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, data, n, tile_sums);
    note_launch();
}

int deposit_sorted(Plan &p, const DepositArgs &a, cudaStream_t st, const int **ring_live) {
    const bool mixed = p.precision == SFB_MIXED;
    const double *rtp = a.rtp, *w = a.w;
    const int64_t ngal = a.ngal, nmock = a.mocks.n;
    double *ref = a.ref, *mu = a.mu;
    *ring_live = nullptr;
    const int64_t nkeys = nmock * (p.pieces + 2) * p.npix;
    if (nkeys > 0x7fffffff || ngal > 0x7fffffff) return fail(SFB_EINVAL, "catalogue or key range above 2^31 - 1");
    const int64_t nscan = nkeys + 1;            // one extra counter: its exclusive prefix is the total
    const int64_t ntiles = (nscan + SCAN_TILE - 1) / SCAN_TILE;
    // workspace: first what one clear presets to zero: counters/offsets [nscan] int32, three block counters and
    // the length of the FP64-pixel list, ring_live [nmock][nrings] int32, S [nmock][nbasis], Q [nmock][pieces + 2];
    // then mudf [nmock][nbasis] float2, cdf [nmock][npix] float2, local coordinate [ngal] double (mixed: float2), sorted (x, w) [ngal] double2
    // (mixed: float4), tile sums [ntiles], key, rank and the FP64-pixel list [ngal] int32
    const int64_t nrings = 4 * p.nside - 1;
    const int64_t off_S = (nscan + 4 + nmock * nrings + 1) / 2;
    const int64_t off_mudf = off_S + nmock * (p.nbasis + p.pieces + 2), off_cdf = off_mudf + nmock * p.nbasis;
    const int64_t off_x = off_cdf + nmock * p.npix;
    int64_t off_sorted = off_x + ngal;
    off_sorted += off_sorted & 1;
    const int64_t off_int = off_sorted + 2 * ngal;
    SFB_TRY(grow(p, p.dep, (size_t)(off_int + (ntiles + 3 * ngal + 1) / 2)));
    int32_t *counts = reinterpret_cast<int32_t *>(p.dep.ptr);
    int *scan_done = counts + nscan, *stats_done = scan_done + 1;
    int32_t *fb_count = scan_done + 2;
    int *live = scan_done + 4;
    double *S = p.dep.ptr + off_S, *Q = S + nmock * p.nbasis;
    float2 *mudf = reinterpret_cast<float2 *>(p.dep.ptr + off_mudf);
    float2 *cdf = reinterpret_cast<float2 *>(p.dep.ptr + off_cdf);
    double *xloc = p.dep.ptr + off_x;
    float2 *xdf = reinterpret_cast<float2 *>(xloc);
    void *sorted = p.dep.ptr + off_sorted;
    float4 *sorted4 = static_cast<float4 *>(sorted);
    int32_t *tsum = reinterpret_cast<int32_t *>(p.dep.ptr + off_int);
    int32_t *key = tsum + ntiles;
    int32_t *rank = key + ngal;
    int32_t *fb_list = rank + ngal;
    SFB_CUDA_TRY(cudaMemsetAsync(p.dep.ptr, 0, (size_t)off_mudf * sizeof(double), st));
    const double inv_width = (double)p.pieces / (p.rmax - p.rmin);
    RadialKeyParams rk;
    rk.ord_rmin = ord_of(p.rmin);
    rk.ord_rmax = ord_of(p.rmax);
    rk.rmin_hi = (float)p.rmin;
    rk.rmin_lo = (float)(p.rmin - (double)rk.rmin_hi);
    rk.invw_hi = (float)inv_width;
    rk.invw_lo = (float)(inv_width - (double)rk.invw_hi);
    // keys: in nchunks galaxy ranges, each after its event (the host entry's copy pipeline), or at once
    const int nck = (a.chunk_ready && a.nchunks > 0) ? a.nchunks : 1;
    const int64_t per = (ngal + nck - 1) / nck;
    for (int c = 0; c < nck; ++c) {
        const int64_t g0 = c * per, n = std::min<int64_t>(per, ngal - g0);
        if (a.chunk_ready && a.nchunks > 0) SFB_CUDA_TRY(cudaStreamWaitEvent(st, a.chunk_ready[c], 0));
        if (n <= 0) continue;
        const unsigned nb = (unsigned)((n + 255) / 256);
        if (mixed)
            launch_pdl(k_deposit_keys_mixed, dim3(nb), dim3(256), 0, st, rtp + 3 * g0, w ? w + g0 : nullptr, n, g0,
                p.nside, p.npix, rk, p.pieces, a.mocks, counts, key + g0, rank + g0, xdf + g0, fb_list, fb_count,
                p.d_err);
        else
            launch_pdl(k_deposit_keys, dim3(nb), dim3(256), 0, st, rtp + 3 * g0, w ? w + g0 : nullptr, n, g0, p.nside,
                p.npix, p.rmin, p.rmax, inv_width, p.pieces, a.mocks, counts, key + g0, rank + g0, xloc + g0, fb_list,
                fb_count, p.d_err);
        note_launch();
    }
    if (ngal > 0) {
        launch_pdl(k_deposit_keys_fallback, dim3(304), dim3(256), 0, st, rtp, p.nside, p.npix, counts, key, rank,
            fb_list, fb_count);
        note_launch();
    }
    launch_pdl(k_scan_tiles, dim3((unsigned)ntiles), dim3(SCAN_THREADS), 0, st, counts, nscan, tsum, scan_done);
    note_launch();
    const Offsets offset{counts, tsum, 0};
    if (ngal > 0) {
        if (mixed)
            launch_pdl(k_deposit_scatter_mixed, dim3((unsigned)((ngal + 255) / 256)), dim3(256), 0, st, w, ngal, key,
                rank, xdf, offset, sorted4);
        else
            launch_pdl(k_deposit_scatter, dim3((unsigned)((ngal + 255) / 256)), dim3(256), 0, st, w, ngal, key, rank,
                xloc, offset, static_cast<double2 *>(sorted));
        note_launch();
    }
    if (p.degree > 63) return fail(SFB_ENOTSUP, "radial degree above 63 is not supported by the sorted deposit");
    const bool split = ref != nullptr && mixed;
    if (split) {
        launch_pdl(k_weight_map_mixed, dim3((unsigned)((p.npix + 255) / 256), (unsigned)nmock), dim3(256), 0, st,
            offset, sorted4, p.nside, p.npix, p.pieces + 2, ref, cdf, live, a.w01);
        note_launch();
        if (a.ref_ready) SFB_CUDA_TRY(cudaEventRecord(a.ref_ready, st));
        by_degree(p.degree, [&](auto D) {
            launch_stats<decltype(D)::value>(p, (int)nmock, offset, sorted4, cdf, S, Q, mu, mudf, stats_done, st);
        });
        if (a.mu_ready) SFB_CUDA_TRY(cudaEventRecord(a.mu_ready, st));
    }
    // moments in FP64 (FP64 path) or double-float (mixed); stored in the transform's precision
    const bool skip_empty = split && p.npix >= 128 && p.degree <= 31;                 // the balanced kernel
    by_degree(p.degree, [&](auto D) {
        launch_moments<decltype(D)::value>(p, (int)nmock, offset, sorted, split ? cdf : nullptr, mudf, a.maps, st,
                                           skip_empty ? live : nullptr);
    });
    if (skip_empty) *ring_live = live;
    SFB_CUDA_TRY(cudaGetLastError());
    return SFB_OK;
}

}  // namespace sfb
