// Galaxy deposit, radial basis and radial projection kernels.
//
// cat2amln (reference src/cat2anlm.jl:257-310) forms, for every (n,l),
//   map_nl[p] = sum_{i in p} w_i g_nl(r_i) / (nbar dOmega) - W[p,l,n]
// and keeps row l of map2alm(map_nl).  map2alm is linear, so with
//   g_nl(r) ~= sum_b C[nl][b] phi_b(r)      (piecewise Legendre basis phi_b)
// the galaxy term becomes sum_b C[nl][b] map2alm(D_b) / (nbar dOmega) with
// D_b[p] = sum_{i in p} w_i phi_b(r_i): one transform per basis function
// instead of one per (n,l).  Galaxies below rmin / above rmax use the
// spline's boundary extrapolation (src/Splines.jl:72-77) through two
// constant basis maps.
#include <vector>

#include <algorithm>

#include "sfb_internal.h"

namespace sfb {

__device__ __forceinline__ bool galaxy_ok(double r, double th, double ph, double w, int *err) {
    if (!(isfinite(r) && isfinite(th) && isfinite(ph) && isfinite(w))) {
        atomicOr(err, ERR_NONFINITE_INPUT);
        return false;
    }
    if (th < 0.0 || th > M_PI) {
        atomicOr(err, ERR_THETA_RANGE);
        return false;
    }
    return true;
}

// Spline mode: maps[q][pix] += w * g_{pair0+q}(r) / (nbar dOmega) for a chunk of pairs.
__global__ void k_deposit_spline(const double *rtp, const double *wgt, int64_t ngal,
                                 int64_t nside, int64_t npix, const int64_t *spl_off, const double *sx,
                                 const double *sy, const double *sypp, int64_t pair0, int64_t npair_chunk,
                                 double scale, double *maps, int *err) {
    pdl_entry();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ngal) return;
    const double r = rtp[3 * i], th = rtp[3 * i + 1], ph = rtp[3 * i + 2];
    const double w = wgt ? wgt[i] : 1.0;
    if (!galaxy_ok(r, th, ph, w, err)) return;
    const int64_t pix = ang2pix_ring_fast(nside, th, ph);
    for (int64_t q = blockIdx.y; q < npair_chunk; q += gridDim.y) {
        const int64_t pr = pair0 + q;
        const int64_t o = spl_off[pr], N = spl_off[pr + 1] - o;
        const double g = spline_eval_dev(sx + o, sy + o, sypp + o, N, r);
        atomicAdd(maps + q * npix + pix, w * g * scale);
    }
}

void launch_deposit_spline_chunk(const Plan &p, const double *rtp, const double *w, int64_t ngal,
                                 int64_t pair0, int64_t npc, double scale, double *maps, cudaStream_t st) {
    if (ngal <= 0 || npc <= 0) return;
    unsigned gy = (unsigned)(npc < 64 ? npc : 64);
    dim3 grid((unsigned)((ngal + 255) / 256), gy);
    launch_pdl(k_deposit_spline, dim3(grid), dim3(256), 0, st, rtp, w, ngal, p.nside, p.npix, p.d_spl_off, p.d_spl_x,
        p.d_spl_y, p.d_spl_ypp, pair0, npc, scale, maps, p.d_err);
    note_launch();
}

// maps[q][p] -= dense[p + npix*(l + (lmax+1)*(n-1))] for the chunk's pairs.
__global__ void k_subtract_dense(double *maps, const double *dense, int64_t npix, int lmax, const int32_t *pair_n,
                                 const int32_t *pair_l, int64_t pair0, int64_t npc) {
    pdl_entry();
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t q = blockIdx.y;
    if (p >= npix || q >= npc) return;
    const int64_t pr = pair0 + q;
    const int64_t off = npix * ((int64_t)pair_l[pr] + (int64_t)(lmax + 1) * (pair_n[pr] - 1));
    maps[q * npix + p] -= dense[off + p];
}

void launch_subtract_dense_chunk(const Plan &p, double *maps, const double *dense, int64_t pair0, int64_t npc,
                                 cudaStream_t st) {
    if (npc <= 0) return;
    dim3 grid((unsigned)((p.npix + 255) / 256), (unsigned)npc);
    launch_pdl(k_subtract_dense, dim3(grid), dim3(256), 0, st, maps, dense, p.npix, p.lmax, p.d_pair_n, p.d_pair_l,
        pair0, npc);
    note_launch();
}

// maps[q][p] -= mask[p] * W_ln[l + (lmax+1)(n-1)] for the chunk's pairs (separable window).
__global__ void k_subtract_sep(double *maps, const double *mask, const double *w_ln, int64_t npix, int lmax,
                               const int32_t *pair_n, const int32_t *pair_l, int64_t pair0, int64_t npc) {
    pdl_entry();
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t q = blockIdx.y;
    if (p >= npix || q >= npc) return;
    const int64_t pr = pair0 + q;
    const double wl = w_ln[pair_l[pr] + (int64_t)(lmax + 1) * (pair_n[pr] - 1)];
    maps[q * npix + p] -= mask[p] * wl;
}

void launch_subtract_sep_chunk(const Plan &p, double *maps, const double *mask, const double *w_ln, int64_t pair0,
                               int64_t npc, cudaStream_t st) {
    if (npc <= 0) return;
    dim3 grid((unsigned)((p.npix + 255) / 256), (unsigned)npc);
    launch_pdl(k_subtract_sep, dim3(grid), dim3(256), 0, st, maps, mask, w_ln, p.npix, p.lmax, p.d_pair_n, p.d_pair_l,
        pair0, npc);
    note_launch();
}

__global__ void k_axpy(double *y, const double *x, int64_t n) {
    pdl_entry();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] += x[i];
}

void launch_axpy(double *y, const double *x, int64_t n, cudaStream_t st) {
    if (n <= 0) return;
    int64_t blocks = (n + 255) / 256;
    if (blocks > 8192) blocks = 8192;
    launch_pdl(k_axpy, dim3((unsigned)blocks), dim3(256), 0, st, y, x, n);
    note_launch();
}

// Gather dense window maps of a chunk of pairs: maps[q] = W[:, l, n].
__global__ void k_gather_dense(double *maps, const double *dense, int64_t npix, int lmax, const int32_t *pair_n,
                               const int32_t *pair_l, int64_t pair0, int64_t npc) {
    pdl_entry();
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t q = blockIdx.y;
    if (p >= npix || q >= npc) return;
    const int64_t pr = pair0 + q;
    const int64_t off = npix * ((int64_t)pair_l[pr] + (int64_t)(lmax + 1) * (pair_n[pr] - 1));
    maps[q * npix + p] = dense[off + p];
}

void launch_gather_dense_chunk(const Plan &p, double *maps, const double *dense, int64_t pair0, int64_t npc,
                               cudaStream_t st) {
    if (npc <= 0) return;
    dim3 grid((unsigned)((p.npix + 255) / 256), (unsigned)npc);
    launch_pdl(k_gather_dense, dim3(grid), dim3(256), 0, st, maps, dense, p.npix, p.lmax, p.d_pair_n, p.d_pair_l,
        pair0, npc);
    note_launch();
}

// Radial coefficients: C[pair][j*(deg+1)+k] = sum_q PQ[q][k] * g(r_q), with
// r_q the Gauss-Legendre nodes of piece j and PQ[q][k] = w_q (2k+1)/2 P_k(x_q)
// (L2 projection of the spline onto Legendre polynomials on each piece);
// C[pair][nbasis-2] / [nbasis-1] = first / last knot value (extrapolation).
__global__ void k_radial_coeffs(const int64_t *spl_off, const double *sx, const double *sy, const double *sypp,
                                double rmin, double rmax, int pieces, int deg, int64_t nbasis, const double *glx,
                                const double *pq, int Q, double *coef) {
    pdl_entry();
    extern __shared__ double gq[];
    const int64_t pr = blockIdx.x;
    const int j = blockIdx.y;
    const int64_t o = spl_off[pr], N = spl_off[pr + 1] - o;
    const double width = (rmax - rmin) / pieces;
    const double a = rmin + j * width;
    for (int q = threadIdx.x; q < Q; q += blockDim.x) {
        const double r = a + (glx[q] + 1.0) * 0.5 * width;
        gq[q] = spline_eval_dev(sx + o, sy + o, sypp + o, N, r);
    }
    __syncthreads();
    for (int k = threadIdx.x; k <= deg; k += blockDim.x) {
        double acc = 0.0;
        for (int q = 0; q < Q; ++q) acc = fma(pq[(int64_t)q * (deg + 1) + k], gq[q], acc);
        coef[pr * nbasis + (int64_t)j * (deg + 1) + k] = acc;
    }
    if (j == 0 && threadIdx.x == 0) {
        coef[pr * nbasis + nbasis - 2] = sy[o];
        coef[pr * nbasis + nbasis - 1] = sy[o + N - 1];
    }
}

void launch_radial_coeffs(const Plan &p, const double *gl_x, const double *pq, int Q, double *coef,
                          cudaStream_t st) {
    dim3 grid((unsigned)p.npairs, (unsigned)p.pieces);
    launch_pdl(k_radial_coeffs, dim3(grid), dim3(128), Q * sizeof(double), st, p.d_spl_off, p.d_spl_x, p.d_spl_y,
        p.d_spl_ypp, p.rmin, p.rmax, p.pieces, p.degree, p.nbasis, gl_x, pq, Q, coef);
    note_launch();
}

// max over knots of |expansion - y| / max|y| per pair; atomicMax on the bit
// pattern (non-negative doubles order like their bits).
__global__ void k_radial_error(const int64_t *spl_off, const double *sx, const double *sy, const double *ymax,
                               double rmin, double rmax, int pieces, int deg, int64_t nbasis, const double *coef,
                               unsigned long long *err_bits) {
    pdl_entry();
    const int64_t pr = blockIdx.x;
    const int64_t o = spl_off[pr], N = spl_off[pr + 1] - o;
    const double width = (rmax - rmin) / pieces;
    const double *C = coef + pr * nbasis;
    double worst = 0.0;
    // interior knots only: within a few knots of rmin/rmax the reference
    // spline carries its parabolic end-slope error, which no smooth expansion
    // (and no radial resolution below the knot spacing) can follow
    for (int64_t i = 8 + threadIdx.x; i < N - 8; i += blockDim.x) {
        const double r = sx[o + i];
        if (r < rmin || r > rmax) continue;
        int j = (int)((r - rmin) / width);
        if (j >= pieces) j = pieces - 1;
        double x = 2.0 * (r - (rmin + j * width)) / width - 1.0;
        x = fmin(1.0, fmax(-1.0, x));
        const double *Cj = C + (int64_t)j * (deg + 1);
        double p0 = 1.0, p1 = x, v = Cj[0] + (deg >= 1 ? Cj[1] * x : 0.0);
        for (int k = 1; k < deg; ++k) {
            const double p2 = ((2 * k + 1) * x * p1 - k * p0) / (k + 1);
            v = fma(Cj[k + 1], p2, v);
            p0 = p1;
            p1 = p2;
        }
        worst = fmax(worst, fabs(v - sy[o + i]));
    }
    worst /= ymax[pr] > 0 ? ymax[pr] : 1.0;
    atomicMax(err_bits, (unsigned long long)__double_as_longlong(worst));
}

void launch_radial_error_impl(const Plan &p, const double *coef, const double *ymax, unsigned long long *err_bits,
                              cudaStream_t st) {
    launch_pdl(k_radial_error, dim3((unsigned)p.npairs), dim3(128), 0, st, p.d_spl_off, p.d_spl_x, p.d_spl_y, ymax,
        p.rmin, p.rmax, p.pieces, p.degree, p.nbasis, coef, err_bits);
    note_launch();
}

// The FP64 radial projection of the FP64 catalogue transform and of fields,
//   out[n,l,m] (+)= scale (sum_s T[pair(n,l)][s] A[lm][s] - w_ln[l,n] A[lm][mask])   (src/cat2anlm.jl:347-353)
// with A in FP64 or as double-float pairs.  The outputs are few (25,295 at lmax 82) and the FP64 pipe bounds the sums
// (205 shells: 10.4 million FMAs, about 20 us), if rows come in coalesced and the quarters of the SMs get equal work:
// a block takes 16 orders of one degree and 2 PS_J radial indices, and its four warps each a quarter of the terms, 16
// at a time through its own part of the shared memory, the next ones' loads in flight meanwhile.  FP64 rows: PS_J = 1,
// small blocks, as most degrees have few radial indices (77 functions: 35 us as one thread an output, its rows
// uncoalesced; 22 now).  Double-float rows: PS_J = 4, so that a value is widened once for eight indices (205 shells:
// 73 us and 11 for a pass that widened all; 70 now).
constexpr int PS_M = 16, PS_S = 16, PS_W = 4;

struct Scales {
    double v[MOCKS_MAX];
};

__device__ __forceinline__ double2 ps_value(double2 a) { return a; }
// a float as a double in integer operations: the conversion instructions share the FP64 pipe with the sums
__device__ __forceinline__ double widen(float f) {
    const unsigned u = __float_as_uint(f), e = u << 1;
    if (e - 0x01000000u >= 0xfe000000u) return e ? (double)f : 0.0;          // zero; subnormal, infinite, NaN
    return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(u << 29));
}
__device__ __forceinline__ double2 ps_value(float4 a) {
    return make_double2(widen(a.x) + widen(a.y), widen(a.z) + widen(a.w));
}

// grid: (degree and 16 orders, 2 PS_J radial indices, mocks); mock j's columns start at j * mcols, the mask's is the last
template <typename TA, int PS_J>
__global__ void __launch_bounds__(32 * PS_W) k_project64(const int32_t *pair_index, int nmax, int lmax,
                                                         const int64_t *noff, const double *T, int64_t ldT, int K,
                                                         const TA *A, int64_t ldA,
                                                         const __grid_constant__ Scales scales, int64_t mcols,
                                                         const double *w_ln, int add, int64_t nlmsize, double *out,
                                                         int *err) {
    pdl_entry();
    constexpr int PS_N = 2 * PS_J;
    __shared__ double2 As[PS_W][PS_M][PS_S + 1];
    __shared__ double Ts[PS_W][PS_N][PS_S];
    __shared__ double2 part[PS_W - 1][PS_J][32];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, mock = blockIdx.z;
    const int i = lane % PS_M, w = lane / PS_M;
    // degrees 16 q .. 16 q + 15 have q + 1 blocks of orders each, 8 q (q + 1) blocks before them
    const int x = blockIdx.x;
    int q = (int)sqrtf((float)x * 0.125f);
    while (8 * q * (q + 1) > x) --q;
    while (8 * (q + 1) * (q + 2) <= x) ++q;
    const int rem = x - 8 * q * (q + 1), l = PS_M * q + rem / (q + 1), m0 = PS_M * (rem % (q + 1));
    const int n0 = blockIdx.y * PS_N + w, m = m0 + i;
    int pr[PS_J];                                                         // lane (i, w): radial indices n0 + 2 j
    bool any = false;
#pragma unroll
    for (int j = 0; j < PS_J; ++j) {
        pr[j] = n0 + 2 * j < nmax ? pair_index[(int64_t)(n0 + 2 * j) * (lmax + 1) + l] : -1;
        any |= pr[j] >= 0;
    }
    if (!__any_sync(0xffffffffu, any)) return;                            // (the same in every warp)
    bool live[PS_J];
#pragma unroll
    for (int j = 0; j < PS_J; ++j) live[j] = __any_sync(0xffffffffu, pr[j] >= 0);
    const int64_t lm0 = (int64_t)l * (l + 1) / 2;
    A += mock * mcols;
    // lane (i, w) loads column i of the rows w, w + 2, .. and of its own radial indices' rows of T
    constexpr int NA = PS_M * PS_S / 32;
    TA av[NA];
    double tv[PS_J];
    const TA *Ab = A + (lm0 + m0 + w) * ldA + i;
    const int k0 = (int)((int64_t)K * wp / PS_W), k1 = (int)((int64_t)K * (wp + 1) / PS_W);
    const int rows = l + 1 - m0 - w;                                      // row w + 2 j is there if 2 j < rows
    auto load = [&](int s0) {
        const bool in = s0 + i < k1;
#pragma unroll
        for (int j = 0; j < NA; ++j) {
            av[j] = TA{};
            if (in && 2 * j < rows) av[j] = Ab[2 * j * ldA + s0];
        }
#pragma unroll
        for (int j = 0; j < PS_J; ++j) tv[j] = in && pr[j] >= 0 ? T[pr[j] * ldT + s0 + i] : 0.0;
    };
    double re[PS_J], im[PS_J];
#pragma unroll
    for (int j = 0; j < PS_J; ++j) re[j] = im[j] = 0.0;
    if (k0 < k1) load(k0);
    for (int s0 = k0; s0 < k1; s0 += PS_S) {
        __syncwarp();
#pragma unroll
        for (int j = 0; j < NA; ++j) As[wp][2 * j + w][i] = ps_value(av[j]);
#pragma unroll
        for (int j = 0; j < PS_J; ++j) Ts[wp][w + 2 * j][i] = tv[j];
        __syncwarp();
        if (s0 + PS_S < k1) load(s0 + PS_S);
        const int ns = min(PS_S, k1 - s0);
#pragma unroll 4
        for (int s = 0; s < ns; ++s) {
            const double2 a = As[wp][i][s];
#pragma unroll
            for (int j = 0; j < PS_J; ++j)
                if (live[j]) {
                    const double t = Ts[wp][w + 2 * j][s];
                    re[j] = fma(t, a.x, re[j]);
                    im[j] = fma(t, a.y, im[j]);
                }
        }
    }
    if (wp > 0)
#pragma unroll
        for (int j = 0; j < PS_J; ++j) part[wp - 1][j][lane] = make_double2(re[j], im[j]);
    __syncthreads();
    if (wp > 0 || m > l) return;
#pragma unroll
    for (int j = 0; j < PS_J; ++j) {
        if (pr[j] < 0) continue;
        const int n1 = n0 + 2 * j;
        double vr = (re[j] + part[0][j][lane].x) + (part[1][j][lane].x + part[2][j][lane].x);
        double vi = (im[j] + part[0][j][lane].y) + (part[1][j][lane].y + part[2][j][lane].y);
        vr *= scales.v[mock];
        vi *= scales.v[mock];
        if (w_ln) {
            const double wl = w_ln[l + (int64_t)(lmax + 1) * n1];
            const double2 a = ps_value(A[(lm0 + m) * ldA + mcols * (gridDim.z - mock)]);
            vr -= wl * a.x;
            vi -= wl * a.y;
        }
        double *o = out + 2 * (mock * nlmsize + noff[n1] + lm0 + m);      // (a caller's pointer: eight-byte aligned)
        if (add) {
            vr += o[0];
            vi += o[1];
        }
        o[0] = vr;
        o[1] = vi;
        if (err && !(isfinite(vr) && isfinite(vi))) atomicOr(err, ERR_NONFINITE_OUTPUT);
    }
}

template <int PS_J, typename TA>
static void project64(const Plan &p, const int32_t *pair_index, const int64_t *noff, const double *T, int64_t ldT,
                      int64_t K, const TA *A, int64_t ldA, int nmock, const double *scale, int64_t mcols,
                      const double *w_ln, bool add, double *out, int *err, cudaStream_t st) {
    if (p.nlmsize <= 0) return;
    Scales sc;
    std::copy(scale, scale + nmock, sc.v);
    const unsigned full = (unsigned)((p.lmax + 1) / PS_M), rest = (unsigned)((p.lmax + 1) % PS_M);
    dim3 grid(8 * full * (full + 1) + rest * (full + 1), (unsigned)((p.nmax + 2 * PS_J - 1) / (2 * PS_J)), (unsigned)nmock);
    launch_pdl(k_project64<TA, PS_J>, grid, dim3(32 * PS_W), 0, st, pair_index, (int)p.nmax, (int)p.lmax, noff, T, ldT,
               (int)K, A, ldA, sc, mcols, w_ln, (int)add, p.nlmsize, out, err);
    note_launch();
}

void launch_project_poly(const Plan &p, const int32_t *pair_index, const int64_t *noff, const double *A, int64_t ncplx,
                         int nmock, const double *scale, const double *w_ln, double *out, int *err, cudaStream_t st) {
    project64<1>(p, pair_index, noff, p.d_coef, p.nbasis, p.nbasis, reinterpret_cast<const double2 *>(A), ncplx, nmock,
              scale, p.nbasis, w_ln, false, out, err, st);
}

void launch_project_shells_g(const Plan &p, const int32_t *pair_index, const int64_t *noff, const double *gtab,
                             int64_t ldg, int64_t nr, const double *A, const float2 *Adf, bool add, double *out,
                             int *err, cudaStream_t st) {
    const double one = 1.0;
    if (Adf)
        project64<4>(p, pair_index, noff, gtab, ldg, nr, reinterpret_cast<const float4 *>(Adf), nr, 1, &one, 0, nullptr,
                  add, out, err, st);
    else
        project64<1>(p, pair_index, noff, gtab, ldg, nr, reinterpret_cast<const double2 *>(A), nr, 1, &one, 0, nullptr,
                  add, out, err, st);
}

// out[o] -= Awin[lm][pair - pair0] for outputs whose pair lies in the chunk.
__global__ void k_sub_window_chunk(const int32_t *out_pair, const int32_t *out_lm, int64_t nlmsize,
                                   const double *Awin, int64_t ldW, int64_t pair0, int64_t npc, double *out) {
    pdl_entry();
    const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= nlmsize) return;
    const int64_t q = (int64_t)out_pair[o] - pair0;
    if (q < 0 || q >= npc) return;
    const double *a = Awin + (int64_t)out_lm[o] * ldW + 2 * q;
    out[2 * o] -= a[0];
    out[2 * o + 1] -= a[1];
}

void launch_sub_window_chunk(const Plan &p, const double *Awin, int64_t ldW, int64_t pair0, int64_t npc, double *out,
                             cudaStream_t st) {
    if (p.nlmsize <= 0) return;
    launch_pdl(k_sub_window_chunk, dim3((unsigned)((p.nlmsize + 127) / 128)), dim3(128), 0, st, p.d_out_pair,
        p.d_out_lm, p.nlmsize, Awin, ldW, pair0, npc, out);
    note_launch();
}

// Spline mode: out[o] = A[lm][pair - pair0] (map already scaled and window-subtracted).
__global__ void k_extract_spline(const int32_t *out_pair, const int32_t *out_lm, int64_t nlmsize, const double *A,
                                 int64_t ldA, int64_t pair0, int64_t npc, double *out) {
    pdl_entry();
    const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= nlmsize) return;
    const int64_t q = (int64_t)out_pair[o] - pair0;
    if (q < 0 || q >= npc) return;
    const double *a = A + (int64_t)out_lm[o] * ldA + 2 * q;
    out[2 * o] = a[0];
    out[2 * o + 1] = a[1];
}

void launch_extract_spline_chunk(const Plan &p, const double *A, int64_t ldA, int64_t pair0, int64_t npc, double *out,
                                 cudaStream_t st) {
    if (p.nlmsize <= 0) return;
    launch_pdl(k_extract_spline, dim3((unsigned)((p.nlmsize + 127) / 128)), dim3(128), 0, st, p.d_out_pair,
        p.d_out_lm, p.nlmsize, A, ldA, pair0, npc, out);
    note_launch();
}

// gtab[pair][s] = g_pair(r_s) * (with_r2dr ? r_s^2 dr : 1), r_s = rmin + (s+1/2) dr.
__global__ void k_gtab(const int64_t *spl_off, const double *sx, const double *sy, const double *sypp,
                       int64_t npairs, int64_t nr, double rmin, double dr, int with_r2dr, double *gtab) {
    pdl_entry();
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nr) return;
    const double r = rmin + dr / 2 + s * dr;
    for (int64_t pr = blockIdx.y; pr < npairs; pr += gridDim.y) {      // grid y is capped at 65535
        const int64_t o = spl_off[pr], N = spl_off[pr + 1] - o;
        double g = spline_eval_dev(sx + o, sy + o, sypp + o, N, r);
        if (with_r2dr) g *= r * r * dr;
        gtab[pr * nr + s] = g;
    }
}

void launch_gtab(const Plan &p, int64_t nr, double rmin, double dr, int with_r2dr, double *gtab, cudaStream_t st) {
    dim3 grid((unsigned)((nr + 127) / 128), (unsigned)std::min<int64_t>(p.npairs, 65535));
    launch_pdl(k_gtab, dim3(grid), dim3(128), 0, st, p.d_spl_off, p.d_spl_x, p.d_spl_y, p.d_spl_ypp, p.npairs, nr,
        rmin, dr, with_r2dr, gtab);
                                 note_launch();
}

// anlm2field radial sum: A[lm][s] = sum_n gtab[pair(n,l)][s] a[idx(n,l,m)] (src/cat2anlm.jl:403-414).  A block takes
// 128 shells of four orders of one degree: a shell's radial functions are read once for the four orders, whose
// coefficients wait in shared memory (each sum in the order of n, one thread).
// 128 shells at lmax 82: 46 us as one thread a coefficient, which found its degree by an FP64 root; 24 now.
constexpr int SA_M = 4, SA_N = 64;
__global__ void __launch_bounds__(128) k_shell_alm(const int32_t *pair_index, const int64_t *noff, int nmax, int lmax,
                                                   const double *gtab, int64_t ldg, int64_t nr, const double *anlm,
                                                   double *A, int64_t ldA) {
    pdl_entry();
    __shared__ double2 an[SA_N][SA_M];
    __shared__ int prs[SA_N];
    // degrees 4 q .. 4 q + 3 have q + 1 blocks of orders each, 2 q (q + 1) blocks before them
    const int x = blockIdx.x;
    int q = (int)sqrtf((float)x * 0.5f);
    while (2 * q * (q + 1) > x) --q;
    while (2 * (q + 1) * (q + 2) <= x) ++q;
    const int rem = x - 2 * q * (q + 1), l = SA_M * q + rem / (q + 1), m0 = SA_M * (rem % (q + 1));
    const int64_t lm0 = (int64_t)l * (l + 1) / 2;
    const int nm = min(SA_M, l + 1 - m0);
    for (int64_t s0 = (int64_t)blockIdx.y * 128; s0 < nr; s0 += (int64_t)gridDim.y * 128) {
        const int64_t s = s0 + threadIdx.x;
        double re[SA_M], im[SA_M];
#pragma unroll
        for (int j = 0; j < SA_M; ++j) re[j] = im[j] = 0.0;
        for (int n0 = 0; n0 < nmax; n0 += SA_N) {
            const int nn = min(SA_N, nmax - n0);
            __syncthreads();
            for (int i = threadIdx.x; i < nn; i += 128) prs[i] = pair_index[(int64_t)(n0 + i) * (lmax + 1) + l];
            __syncthreads();
            for (int i = threadIdx.x; i < nn * SA_M; i += 128) {
                const int n = i / SA_M, j = i % SA_M;
                if (prs[n] < 0 || j >= nm) continue;
                const double *a = anlm + 2 * (noff[n0 + n] + lm0 + m0 + j);
                an[n][j] = make_double2(a[0], a[1]);
            }
            __syncthreads();
            if (s >= nr) continue;
#pragma unroll 4
            for (int n = 0; n < nn; ++n) {
                const int pr = prs[n];
                if (pr < 0) continue;
                const double g = gtab[(int64_t)pr * ldg + s];
#pragma unroll
                for (int j = 0; j < SA_M; ++j)
                    if (j < nm) {
                        re[j] = fma(g, an[n][j].x, re[j]);
                        im[j] = fma(g, an[n][j].y, im[j]);
                    }
            }
        }
        if (s >= nr) continue;
#pragma unroll
        for (int j = 0; j < SA_M; ++j)
            if (j < nm)
                *reinterpret_cast<double2 *>(A + (lm0 + m0 + j) * ldA + 2 * s) =
                    make_double2(re[j], m0 + j == 0 ? 0.0 : im[j]);
    }
}

void launch_shell_alm_g(const Plan &p, const int32_t *pair_index, const int64_t *noff, const double *gtab, int64_t ldg,
                        int64_t nr, const double *anlm, double *A, int64_t ldA, cudaStream_t st) {
    const unsigned full = (unsigned)((p.lmax + 1) / SA_M), rest = (unsigned)((p.lmax + 1) % SA_M);
    dim3 grid(2 * full * (full + 1) + rest * (full + 1), (unsigned)std::min<int64_t>((nr + 127) / 128, 65535));
    launch_pdl(k_shell_alm, grid, dim3(128), 0, st, pair_index, noff, (int)p.nmax, (int)p.lmax, gtab, ldg, nr, anlm, A,
               ldA);
    note_launch();
}

// W_ln[l + (lmax+1)(n-1)] = sum_s gtab[pair][s] phi[s]  (gtab includes r^2 dr); NaN off-mode.
__global__ void k_win_sep(const int32_t *pair_n, const int32_t *pair_l, int64_t npairs, const double *gtab, int64_t nr,
                          const double *phi, int lmax, double *out) {
    pdl_entry();
    const int64_t pr = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (pr >= npairs) return;
    double acc = 0.0;
    for (int64_t s = 0; s < nr; ++s) acc += gtab[pr * nr + s] * phi[s];
    out[pair_l[pr] + (int64_t)(lmax + 1) * (pair_n[pr] - 1)] = acc;
}

void launch_win_sep_g(const Plan &p, const double *gtab, int64_t nr, const double *phi, double *out, cudaStream_t st) {
    launch_pdl(k_win_sep, dim3((unsigned)((p.npairs + 127) / 128)), dim3(128), 0, st, p.d_pair_n, p.d_pair_l,
        p.npairs, gtab, nr, phi, p.lmax, out);
    note_launch();
}

// Dense: W[p + npix(l + (lmax+1)(n-1))] = sum_s win[s + nr p] gtab[pair][s]
__global__ void k_win_dense(const int32_t *pair_n, const int32_t *pair_l, int64_t npairs, const double *gtab, int64_t nr,
                            const double *win, int64_t npix, int lmax, double *out) {
    pdl_entry();
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    const double *wc = win + p * nr;
    for (int64_t pr = blockIdx.y; pr < npairs; pr += gridDim.y) {      // grid y is capped at 65535
        const double *g = gtab + pr * nr;
        double acc = 0.0;
        for (int64_t s = 0; s < nr; ++s) acc += wc[s] * g[s];
        out[p + npix * ((int64_t)pair_l[pr] + (int64_t)(lmax + 1) * (pair_n[pr] - 1))] = acc;
    }
}

void launch_win_dense_g(const Plan &p, const double *gtab, int64_t nr, const double *win, double *out, cudaStream_t st) {
    dim3 grid((unsigned)((p.npix + 127) / 128), (unsigned)std::min<int64_t>(p.npairs, 65535));
    launch_pdl(k_win_dense, dim3(grid), dim3(128), 0, st, p.d_pair_n, p.d_pair_l, p.npairs, gtab, nr, win, p.npix,
        p.lmax, out);
    note_launch();
}

// amln2clnn (src/SphericalFourierBesselDecompositions.jl:114-150): one warp per
// (l, n1, n2) column of lnn (3 x nlnn, 1-based n), over nbatch coefficient vectors:
// C = [Re(a1_0 a2_0) + 2 sum_{m>=1} Re(a1_m conj(a2_m))] / (2l + 1).
__global__ void k_amln2clnn(const double *a1, const double *a2, int64_t nlmsize,
                            const int64_t *lnn, int64_t nlnn, int64_t nbatch, const int64_t *noff,
                            double *out) {
    pdl_entry();
    const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= nlnn * nbatch) return;
    const int64_t b = wid / nlnn, i = wid - b * nlnn;
    const int64_t l = lnn[3 * i], n1 = lnn[3 * i + 1], n2 = lnn[3 * i + 2];
    const double *x = a1 + 2 * (b * nlmsize + noff[n1 - 1] + l * (l + 1) / 2);
    const double *y = a2 + 2 * (b * nlmsize + noff[n2 - 1] + l * (l + 1) / 2);
    double c = 0.0;
    for (int64_t m = lane; m <= l; m += 32) {
        const double xr = x[2 * m], xi = x[2 * m + 1], yr = y[2 * m], yi = y[2 * m + 1];
        c += (m == 0) ? (xr * yr - xi * yi) : 2.0 * (xr * yr + xi * yi);
    }
    for (int off = 16; off > 0; off >>= 1) c += __shfl_xor_sync(0xffffffffu, c, off);
    if (lane == 0) out[b * nlnn + i] = c / (double)(2 * l + 1);
}

void launch_amln2clnn(const double *a1, const double *a2, int64_t nlmsize, const int64_t *lnn, int64_t nlnn,
                      int64_t nbatch, const int64_t *noff, double *out, cudaStream_t st) {
    const int64_t threads = nlnn * nbatch * 32;
    if (threads <= 0) return;
    launch_pdl(k_amln2clnn, dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, st, a1, a2, nlmsize, lnn, nlnn,
        nbatch, noff, out);
    note_launch();
}

// winweights2galweights (src/cat2anlm.jl:218-238): w_i = weights[bin(r_i), pix(theta_i, phi_i)]
// with bin = nr if r == rmax, else searchsortedlast(rbounds, r) (1-based), over
// the caller's rbounds[0..nr].  Out-of-range bins set ERR_RANGE_R and give NaN.
__global__ void k_winweights(const double *weights, int64_t nr, int64_t npix, int64_t nside,
                             const double *rbounds, double rmax, const double *rtp,
                             int64_t ngal, double *w, int *err) {
    pdl_entry();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ngal) return;
    const double r = rtp[3 * i], th = rtp[3 * i + 1], ph = rtp[3 * i + 2];
    if (!(isfinite(r) && isfinite(th) && isfinite(ph))) {
        atomicOr(err, ERR_NONFINITE_INPUT);
        w[i] = NAN;
        return;
    }
    const int64_t pix = ang2pix_ring_fast(nside, th, ph);
    int64_t bin;
    if (r == rmax) {
        bin = nr;
    } else {
        // largest 1-based j with rbounds[j] <= r (0 if none)
        int64_t lo = 0, hi = nr + 1;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (rbounds[mid] <= r) lo = mid + 1; else hi = mid;
        }
        bin = lo;
    }
    if (bin < 1 || bin > nr) {
        atomicOr(err, ERR_RANGE_R);
        w[i] = NAN;
        return;
    }
    w[i] = weights[(bin - 1) + nr * pix];
}

void launch_winweights(const double *weights, int64_t nr, int64_t nside, const double *rbounds, double rmax,
                       const double *rtp, int64_t ngal, double *w, int *err, cudaStream_t st) {
    if (ngal <= 0) return;
    launch_pdl(k_winweights, dim3((unsigned)((ngal + 255) / 256)), dim3(256), 0, st, weights, nr, 12 * nside * nside,
        nside, rbounds, rmax, rtp, ngal, w, err);
    note_launch();
}

// ---- mixed-precision radial projection ---------------------------------------
// Double-float helpers (FP32 pairs, ~48 significant bits).
struct df2 {
    float hi, lo;
};
__device__ __forceinline__ df2 dfa(df2 a, df2 b) {
    const float s = a.hi + b.hi;
    const float z = s - a.hi;
    const float e = ((a.hi - (s - z)) + (b.hi - z)) + (a.lo + b.lo);
    const float h = s + e;
    return {h, e - (h - s)};
}
__device__ __forceinline__ df2 dfm(df2 a, df2 b) {
    const float p = a.hi * b.hi;
    float e = fmaf(a.hi, b.hi, -p);
    e = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, e));
    const float h = p + e;
    return {h, e - (h - p)};
}

// CT[(l * nbasis + b) * nmax + n - 1] = coef[pair(n, l)][b] as hi + lo (0 where (n, l) is not a mode).
__global__ void k_coef_df(const double *coef, const int32_t *pair_index, int lmax, int nmax,
                          int64_t nbasis, float2 *CT) {
    pdl_entry();
    const int64_t total = (int64_t)(lmax + 1) * nbasis * nmax;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int n1 = (int)(i % nmax);
        const int64_t t = i / nmax;
        const int64_t b = t % nbasis;
        const int l = (int)(t / nbasis);
        const int pr = pair_index[(int64_t)n1 * (lmax + 1) + l];
        const double v = pr >= 0 ? coef[(int64_t)pr * nbasis + b] : 0.0;
        const float h = (float)v;
        CT[i] = make_float2(h, (float)(v - (double)h));
    }
}

void launch_coef_df(const Plan &p, const int32_t *pair_index, float2 *CT, cudaStream_t st) {
    launch_pdl(k_coef_df, dim3(1024), dim3(256), 0, st, p.d_coef, pair_index, p.lmax, (int)p.nmax, p.nbasis, CT);
    note_launch();
}

// s[pair] = sum_b coef[pair][b] mu_b (FP64): the mean part of every pair, one
// warp per pair (lanes over b, coalesced rows).
// (grid.y: mocks, their mu and s one after another)
__global__ void k_mean_proj(const double *coef, int64_t npairs, int64_t nbasis,
                            const double *mu, double *s) {
    pdl_entry();
    mu += blockIdx.y * nbasis;
    s += blockIdx.y * npairs;
    const int64_t pr = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (pr >= npairs) return;
    double a = 0.0;
    for (int64_t b = lane; b < nbasis; b += 32) a = fma(coef[pr * nbasis + b], mu[b], a);
    for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
    if (lane == 0) s[pr] = a;
}

// Tiles of the projection: block (l, m0, n0, npt) of the plan's tile list
// covers m = m0 .. m0 + 31 (lane = m) and n = n0 + 1 .. n0 + npt (npt <= 8
// accumulators per thread); its PJ_KS warps split the basis range and add
// their partial sums at the end:
//   a_nlm = scale * sum_b coef[n,l][b] dA_b[lm]              (double-float)
//         + scale * s[pair] * C_lm - w_ln(l, n) * M_lm        (FP64)
// with dA the fluctuation a_lm (double-float copy, row lm of width ldA, the
// pairs re, im of basis b side by side), C_lm / M_lm the FP64 a_lm of the
// count map / the mask (ralm [lm][4]); the mean and window terms are skipped
// when ralm is null / window_kind is not separable.  The coefficient rows CT
// (per (l, b) contiguous in n) are read through L1, each load a broadcast to
// the warp.  The products are formed exactly (TwoProd) and summed with
// TwoSum into the high word; the low word gathers the rounding errors and the
// cross terms, unnormalised until the end.
constexpr int PJ_NPT = 8, PJ_KS = 4;

struct pacc {
    float hi, lo;
};

__device__ __forceinline__ void pj_mac(pacc &a, float2 c, float xh, float xl) {
    const float p = c.x * xh;
    const float e = fmaf(c.x, xh, -p);
    const float s = a.hi + p;
    const float z = s - a.hi;
    const float err = (a.hi - (s - z)) + (p - z);
    a.hi = s;
    a.lo = fmaf(c.y, xh, fmaf(c.x, xl, (a.lo + err) + e));
}

// grid.y: mocks (launch_project_mixed says where each one's data lie)
template <int KS>
__global__ void __launch_bounds__(32 * KS) k_project_mixed(const float2 *Adf, int64_t ldA,
                                                              int64_t nbasis, const float2 *CT, int nmax,
                                                              int lmax, const int3 *tiles,
                                                              const int64_t *noff,
                                                              const int32_t *pair_index,
                                                              const __grid_constant__ Scales scales,
                                                              const double *smean, int64_t npairs,
                                                              const double *ralm, int64_t ldR,
                                                              int64_t nlmsize, int window_kind,
                                                              const double *w_ln,
                                                              double *out, int *err) {
    pdl_entry();
    __shared__ float4 part[KS - 1][PJ_NPT][32];
    const int mock = blockIdx.y;
    const double scale = scales.v[mock];
    Adf += (int64_t)mock * 2 * nbasis;
    smean += mock * npairs;
    out += (int64_t)mock * 2 * nlmsize;
    const int3 t = tiles[blockIdx.x];
    const int l = t.x, m0 = t.y, n0 = t.z & 0xffff, npt = t.z >> 16;
    const int lane = threadIdx.x & 31, ks = threadIdx.x >> 5;
    const int m = m0 + lane;
    const bool live = m <= l;
    const int64_t lm = (int64_t)l * (l + 1) / 2 + (live ? m : l);      // lanes past l read a valid row
    const int64_t kper = (nbasis + KS - 1) / KS;
    const int64_t kb0 = ks * kper, kb1 = kb0 + kper < nbasis ? kb0 + kper : nbasis;
    const float4 *arow = reinterpret_cast<const float4 *>(Adf + lm * ldA);
    const float2 *Cl = CT + (int64_t)l * nbasis * nmax + n0;
    pacc re[PJ_NPT], im[PJ_NPT];
#pragma unroll
    for (int j = 0; j < PJ_NPT; ++j) re[j] = im[j] = pacc{0.f, 0.f};
#pragma unroll 2
    for (int64_t b = kb0; b < kb1; ++b) {
        const float4 a = arow[b];                 // re.hi, re.lo, im.hi, im.lo
        const float2 *cb = Cl + b * nmax;
#pragma unroll
        for (int j = 0; j < PJ_NPT; ++j) {
            if (j < npt) {
                const float2 c = __ldg(cb + j);   // (a table of the plan)
                pj_mac(re[j], c, a.x, a.y);
                pj_mac(im[j], c, a.z, a.w);
            }
        }
    }
    if (ks > 0) {
#pragma unroll
        for (int j = 0; j < PJ_NPT; ++j) part[ks - 1][j][lane] = make_float4(re[j].hi, re[j].lo, im[j].hi, im[j].lo);
    }
    __syncthreads();
    if (ks > 0 || !live) return;
#pragma unroll
    for (int j = 0; j < PJ_NPT; ++j) {
        const int n1 = n0 + j;
        if (j >= npt) break;
        const int pr = pair_index[(int64_t)n1 * (lmax + 1) + l];
        if (pr < 0) continue;
        // the parts added in double-float (FP32 units), one conversion to FP64
        df2 sr = df2{re[j].hi, re[j].lo}, si = df2{im[j].hi, im[j].lo};
#pragma unroll
        for (int q = 0; q < KS - 1; ++q) {
            const float4 v = part[q][j][lane];
            sr = dfa(sr, df2{v.x, v.y});
            si = dfa(si, df2{v.z, v.w});
        }
        double vr = scale * ((double)sr.hi + (double)sr.lo);
        double vi = scale * ((double)si.hi + (double)si.lo);
        if (ralm) {
            const double mu = scale * smean[pr];
            const double *cm = ralm + ldR * lm + 2 * mock, *wm = ralm + ldR * lm + 2 * gridDim.y;
            vr = fma(mu, cm[0], vr);
            vi = fma(mu, cm[1], vi);
            if (window_kind == SFB_WINDOW_SEPARABLE) {
                const double wl = w_ln[l + (int64_t)(lmax + 1) * n1];
                vr = fma(-wl, wm[0], vr);
                vi = fma(-wl, wm[1], vi);
            }
        }
        const int64_t o = noff[n1] + lm;
        out[2 * o] = vr;
        out[2 * o + 1] = vi;
        if (err && !(isfinite(vr) && isfinite(vi))) atomicOr(err, ERR_NONFINITE_OUTPUT);
    }
}

// Tile list of the projection: (l, m0, n0 | npt << 16) for m0 = 0, 32, .. <= l
// and n0 = 0, 8, .. below the number of radial modes of l (the valid n form a
// prefix), npt = the modes left from n0 (at most 8).
std::vector<int3> project_tiles(const std::vector<int32_t> &pair_index, int lmax, int nmax) {
    std::vector<int3> t;
    for (int l = 0; l <= lmax; ++l) {
        int nl = 0;
        while (nl < nmax && pair_index[(size_t)nl * (lmax + 1) + l] >= 0) ++nl;
        for (int m0 = 0; m0 <= l; m0 += 32)
            for (int n0 = 0; n0 < nl; n0 += PJ_NPT)
                t.push_back(make_int3(l, m0, n0 | (std::min(PJ_NPT, nl - n0) << 16)));
    }
    return t;
}

void launch_mean_proj(const Plan &p, const double *mu, int nmock, double *smean, cudaStream_t st) {
    launch_pdl(k_mean_proj, dim3((unsigned)((p.npairs + 3) / 4), (unsigned)nmock), dim3(128), 0, st, p.d_coef,
        p.npairs, p.nbasis, mu, smean);
    note_launch();
}

void launch_project_mixed(const Plan &p, const float2 *Adf, int64_t ldA, const float2 *CT, const int64_t *noff,
                          const int32_t *pair_index, int nmock, const double *scale, const double *smean,
                          const double *ralm, int64_t ldR, int window_kind, const double *w_ln, double *out, int *err,
                          cudaStream_t st) {
    if (p.n_proj_tiles <= 0) return;
    Scales sc;
    std::copy(scale, scale + nmock, sc.v);
    launch_pdl(k_project_mixed<PJ_KS>, dim3((unsigned)p.n_proj_tiles, (unsigned)nmock), dim3(32 * PJ_KS), 0, st,
        Adf, ldA, p.nbasis, CT, (int)p.nmax, p.lmax, p.d_proj_tiles, noff, pair_index, sc, smean, p.npairs, ralm, ldR,
        p.nlmsize, window_kind, w_ln, out, err);
    note_launch();
}

// <ref, ref> of one map, by one block
__global__ void __launch_bounds__(1024) k_ref_square(const double *ref, int64_t npix, double *refsq) {
    pdl_entry();
    __shared__ double red[32];
    double q = 0.0;
#pragma unroll 4
    for (int64_t p = threadIdx.x; p < npix; p += 1024) q = fma(ref[p], ref[p], q);
    for (int off = 16; off > 0; off >>= 1) q += __shfl_xor_sync(0xffffffffu, q, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = q;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 32; ++w) q += red[w];
        *refsq = q;
    }
}

void launch_ref_square(const double *ref, int64_t npix, double *refsq, cudaStream_t st) {
    launch_pdl(k_ref_square, dim3(1), dim3(1024), 0, st, ref, npix, refsq);
    note_launch();
}

// One block per pair: nu = <W, ref> / <ref, ref>, then the fluctuation W - nu ref as double-float pairs (the
// split by integer operations).  The window map is read where the caller's array has it, the second time from L2,
// and written once.  Bound: the FP64 pipe (two operations a pixel) beside HBM (16 bytes); as a gather, an in-place
// split with three FP64 operations and a conversion pass it took 446 us for 507 maps of nside 64.
__global__ void __launch_bounds__(512) k_dense_maps_df(const double *dense, int64_t npix, int lmax,
                                                       const int32_t *pair_n,
                                                       const int32_t *pair_l, int64_t pair0,
                                                       const double *ref,
                                                       const double *refsq, double *nu,
                                                       float2 *maps) {
    pdl_entry();
    __shared__ double red[16];
    const int64_t pr = pair0 + blockIdx.x;
    const double *W = dense + npix * ((int64_t)pair_l[pr] + (int64_t)(lmax + 1) * (pair_n[pr] - 1));
    float2 *m = maps + (int64_t)blockIdx.x * npix;
    double d = 0.0;
#pragma unroll 8
    for (int64_t p = threadIdx.x; p < npix; p += 512) d = fma(W[p], ref[p], d);
    for (int off = 16; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = d;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 16; ++w) d += red[w];
        const double q = *refsq;
        red[0] = q > 0.0 ? d / q : 0.0;
        nu[blockIdx.x] = red[0];
    }
    __syncthreads();
    const double v = red[0];
#pragma unroll 8
    for (int64_t p = threadIdx.x; p < npix; p += 512) {
        const double x = fma(-v, ref[p], W[p]);
        // a non-finite value keeps its kind (the split by bits takes finite ones)
        m[p] = isfinite(x) ? df_split_bits(x) : make_float2((float)x, 0.f);
    }
}

void launch_dense_maps_df(const Plan &p, const double *dense, const double *ref, const double *refsq, int64_t pair0,
                          int64_t npc, double *nu, float2 *maps, cudaStream_t st) {
    if (npc <= 0) return;
    launch_pdl(k_dense_maps_df, dim3((unsigned)npc), dim3(512), 0, st, dense, p.npix, p.lmax, p.d_pair_n, p.d_pair_l,
        pair0, ref, refsq, nu, maps);
    note_launch();
}

// The window's part of every coefficient of the chunk's pairs, from the double-float a_lm (the rows l of pair (n,
// l) only) and the reference map's FP64 ones.
__global__ void k_sub_window_df(const int32_t *out_pair, const int32_t *out_lm,
                                int64_t nlmsize, const float2 *Adf, int64_t ldA, int64_t pair0, int64_t npc,
                                const double *nu, const double *rref, int64_t ldR,
                                double *out, int *err) {
    pdl_entry();
    const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= nlmsize) return;
    const int64_t q = (int64_t)out_pair[o] - pair0;
    if (q < 0 || q >= npc) return;
    const int64_t lm = out_lm[o];
    const float4 a = *reinterpret_cast<const float4 *>(Adf + lm * ldA + 2 * q);
    const double v = nu[q];
    const double re = out[2 * o] - fma(v, rref[lm * ldR], (double)a.x + (double)a.y);
    const double im = out[2 * o + 1] - fma(v, rref[lm * ldR + 1], (double)a.z + (double)a.w);
    out[2 * o] = re;
    out[2 * o + 1] = im;
    if (!(isfinite(re) && isfinite(im))) atomicOr(err, ERR_NONFINITE_OUTPUT);
}

void launch_sub_window_df(const Plan &p, const float2 *Adf, int64_t ldA, int64_t pair0, int64_t npc, const double *nu,
                          const double *rref, int64_t ldR, double *out, int *err, cudaStream_t st) {
    launch_pdl(k_sub_window_df, dim3((unsigned)((p.nlmsize + 127) / 128)), dim3(128), 0, st, p.d_out_pair, p.d_out_lm,
        p.nlmsize, Adf, ldA, pair0, npc, nu, rref, ldR, out, err);
    note_launch();
}

__global__ void k_fill(double *x, int64_t n, double v) {
    pdl_entry();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        x[i] = v;
}

void launch_fill(double *x, int64_t n, double v, cudaStream_t st) {
    if (n <= 0) return;
    int64_t blocks = (n + 255) / 256;
    if (blocks > 8192) blocks = 8192;
    launch_pdl(k_fill, dim3((unsigned)blocks), dim3(256), 0, st, x, n, v);
    note_launch();
}

}  // namespace sfb

namespace sfb {

// w00[s] = Re a_00 of map s of an FP64 a_lm set (row lm = 0, columns 2 s / 2 s + 1)
__global__ void k_extract_a00(const double *alm, int64_t nm, double *w00) {
    pdl_entry();
    const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s < nm) w00[s] = alm[2 * s];
}

void launch_extract_a00(const double *alm, int64_t ldA, int64_t nm, double *w00, cudaStream_t st) {
    (void)ldA;
    launch_pdl(k_extract_a00, dim3((unsigned)((nm + 127) / 128)), dim3(128), 0, st, alm, nm, w00);
    note_launch();
}

// win_lnn radial integrals (reference calc_intr_gg_fn, src/windows.jl:394-422, trapezoidal
// nodes = shell midpoints, weights = dr, f = W00 / sqrt(4 pi)): one warp per column i of lnn,
//   out[i] = sum_s (g_nl(r_s) r_s sqrt(dr) sqrt(f_s)) (g_n'l(r_s) r_s sqrt(dr) sqrt(f_s)).
__global__ void k_win_lnn(const int32_t *pair_index, int lmax, const double *gtab,
                          int64_t nr, double rmin, double dr, const double *w00,
                          const int64_t *lnn, int64_t nlnn, double *out) {
    pdl_entry();
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= nlnn) return;
    const int64_t l = lnn[3 * i], n1 = lnn[3 * i + 1], n2 = lnn[3 * i + 2];
    const double *g1 = gtab + (int64_t)pair_index[(n1 - 1) * (lmax + 1) + l] * nr;
    const double *g2 = gtab + (int64_t)pair_index[(n2 - 1) * (lmax + 1) + l] * nr;
    const double sdr = sqrt(dr), inv4pi = 1.0 / sqrt(4.0 * M_PI);
    double acc = 0.0;
    for (int64_t s = lane; s < nr; s += 32) {
        const double r = rmin + dr / 2 + s * dr;                 // the shell midpoints of k_gtab
        const double w = r * sdr * sqrt(w00[s] * inv4pi);
        acc = fma(g1[s] * w, g2[s] * w, acc);
    }
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0) out[i] = acc;
}

void launch_win_lnn(const Plan &p, const int32_t *pair_index, const double *gtab, int64_t nr, double rmin, double dr,
                    const double *w00, const int64_t *lnn, int64_t nlnn, double *out, cudaStream_t st) {
    launch_pdl(k_win_lnn, dim3((unsigned)((nlnn * 32 + 127) / 128)), dim3(128), 0, st, pair_index, p.lmax, gtab, nr,
        rmin, dr, w00, lnn, nlnn, out);
    note_launch();
}

}  // namespace sfb
