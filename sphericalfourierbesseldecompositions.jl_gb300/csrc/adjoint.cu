// Adjoint (vector-Jacobian products) of the transforms, FP64: the transpose
// of map2alm with niter refinement, of the radial projection and of the
// deposit, for gradients of a loss through cat2amln (dL/dw_i) and
// field2anlm (dL/dfield).
//
// With A = analysis (weighted ring DFT, then Legendre analysis) and S =
// synthesis (Legendre synthesis, then inverse ring DFT), map2alm with niter
// refinements is  a = sum_{j=0}^{niter} (I - A S)^j A f.  As real-linear maps
// (re and im parts of a_lm as separate coordinates) A^T = w S E and
// S^T = (1/w) E^-1 A, w = 4 pi / npix, E = 1 for m = 0 and 1/2 for m >= 1
// (the synthesis counts the m >= 1 terms twice), so
//   f_bar = S sum_{j=0}^{niter} (I - A S)^j (w E a_bar),
// evaluated as x <- b + x - A S x (niter times, from x = b = w E a_bar).  That
// is the forward refinement a <- a0 + a - A S a with b for its first pass a0,
// so it runs through the same Gram form (or, without Gram tables, the same
// synthesis, aliasing fold and analysis over every ring).  Reference: the transforms are those of src/cat2anlm.jl:257-357
// (cat2amln, field2anlm_v2) around src/healpix_helpers.jl:50-56 (map2alm).
#include <algorithm>
#include <cmath>

#include "sfb_internal.h"

namespace sfb {

// alm[lm][c] *= s (m = 0) or s / 2 (m >= 1) (w E above); lm = l (l+1)/2 + m
__global__ void k_halve_m(double *alm, int64_t lmsize, int64_t ncol, double s) {
    pdl_entry();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= lmsize * ncol) return;
    const int64_t lm = i / ncol;
    int l = (int)((sqrtf(8.0f * (float)lm + 1.0f) - 1.0f) * 0.5f);
    while ((int64_t)(l + 1) * (l + 2) / 2 <= lm) ++l;               // (the FP32 root's rounding)
    while ((int64_t)l * (l + 1) / 2 > lm) --l;
    alm[i] *= lm - (int64_t)l * (l + 1) / 2 >= 1 ? 0.5 * s : s;
}

// Transpose of the radial projection a_nlm = s sum_b c[pair(n,l)][b] A_b[lm]:
//   Abar[lm][2b + t] = s sum_n c[pair(n,l)][b] abar[noff(n) + lm][t]   (t = re, im)
// for the basis functions b in [b0, b0 + nbc).
// The deposit's transpose sums in the monic form of the Legendre polynomials, P_k = c_k p_k with
// c_k = (1 3 .. (2k - 1)) / k!, so every function of degree k carries c_k from here on.
constexpr int MONIC_MAX = 64;
struct MonicScale {
    double c[MONIC_MAX];
};
__device__ __forceinline__ double monic_scale(const MonicScale &t, int k) {
    double c = t.c[min(k, MONIC_MAX - 1)];
    for (int j = MONIC_MAX; j <= k; ++j) c *= (2.0 * j - 1.0) / j;
    return c;
}

__global__ void k_proj_adjoint(const double *abar, const double *coef, int64_t nbasis,
                               const int32_t *pair_index, const int64_t *noff, int lmax,
                               int nmax, int64_t lmsize, int64_t b0, int64_t nbc, double s, int deg,
                               const __grid_constant__ MonicScale monic, double *Abar) {
    pdl_entry();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= lmsize * nbc) return;
    const int64_t lm = i / nbc, b = b0 + (i - lm * nbc);
    int l = (int)((sqrtf(8.0f * (float)lm + 1.0f) - 1.0f) * 0.5f);
    while ((int64_t)(l + 1) * (l + 2) / 2 <= lm) ++l;
    while ((int64_t)l * (l + 1) / 2 > lm) --l;
    double re = 0.0, im = 0.0;
    for (int n1 = 0; n1 < nmax; ++n1) {
        const int pr = pair_index[(int64_t)n1 * (lmax + 1) + l];
        if (pr < 0) continue;
        const double c = coef[(int64_t)pr * nbasis + b];
        const int64_t o = noff[n1] + lm;
        re = fma(c, abar[2 * o], re);
        im = fma(c, abar[2 * o + 1], im);
    }
    if (b < nbasis - 2) s *= monic_scale(monic, (int)(b % (deg + 1)));      // (the last two are the constants outside)
    Abar[lm * (2 * nbc) + 2 * (b - b0)] = s * re;
    Abar[lm * (2 * nbc) + 2 * (b - b0) + 1] = s * im;
}

// Transpose of the deposit for the basis functions [b0, b0 + nbc):
//   dw[i] += sum_{b in range} phi_b(r_i) Dbar_b[pix(i)]
// with phi_b the piecewise Legendre basis of the deposit in its monic form
// (p_k on the galaxy's piece, the constants outside [rmin, rmax]; Dbar carries
// the scales); galaxies are keyed exactly as
// the deposit keys them.
__global__ void k_deposit_adjoint(const double *rtp, int64_t ngal, int64_t nside, int64_t npix,
                                  double rmin, double rmax, double inv_width, int pieces, int deg, int64_t nbasis,
                                  const double *Dbar, int64_t sb, int64_t sp, int64_t b0, int64_t nbc,
                                  double *dw, int *err) {
    pdl_entry();
    __shared__ double gam[64];                        // -(k+1)^2 / (4 (k+1)^2 - 1) for k < 64
    for (int k = threadIdx.x; k <= min(deg, 63); k += blockDim.x)
        gam[k] = -((k + 1.0) * (k + 1.0)) / (4.0 * (k + 1.0) * (k + 1.0) - 1.0);
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ngal) return;
    const double r = rtp[3 * i], th = rtp[3 * i + 1], ph = rtp[3 * i + 2];
    if (!(isfinite(r) && isfinite(th) && isfinite(ph))) {
        atomicOr(err, ERR_NONFINITE_INPUT);
        return;
    }
    if (th < 0.0 || th > M_PI) {
        atomicOr(err, ERR_THETA_RANGE);
        return;
    }
    const int64_t pix = ang2pix_ring_fast(nside, th, ph);
    double acc = 0.0;
    if (r < rmin || r > rmax) {
        const int64_t b = nbasis - 2 + (r < rmin ? 0 : 1);
        if (b >= b0 && b < b0 + nbc) acc = Dbar[(b - b0) * sb + pix * sp];
    } else {
        const double u = (r - rmin) * inv_width;
        int slot = (int)u;
        if (slot >= pieces) slot = pieces - 1;
        double x = 2.0 * (u - (double)slot) - 1.0;
        x = fmin(1.0, fmax(-1.0, x));
        // sum_k p_k(x) D_k by Clenshaw's recurrence b_k = D_k + x b_{k+1} - g_{k+1} b_{k+2}, g_k = k^2 / (4 k^2 - 1):
        // two FP64 operations a degree, one fewer than for P_k (the FP64 pipe bounds this kernel: 5e5
        // galaxies and 77 functions take 97 us with P_k, 74 so)
        const int64_t bs = (int64_t)slot * (deg + 1);
        const double *D = Dbar + (bs - b0) * sb + pix * sp;
        double c1 = 0.0, c2 = 0.0;
        for (int k = deg; k >= 0; --k) {
            const int64_t b = bs + k;
            const double d = b >= b0 && b < b0 + nbc ? D[k * sb] : 0.0;
            const double ng = k < 64 ? gam[k] : -((k + 1.0) * (k + 1.0)) / (4.0 * (k + 1.0) * (k + 1.0) - 1.0);
            const double c0 = fma(x, c1, fma(ng, c2, d));
            c2 = c1;
            c1 = c0;
        }
        acc = c1;
    }
    dw[i] += acc;
}

void launch_halve_m(double *alm, int64_t lmsize, int64_t ncol, double s, cudaStream_t st) {
    const int64_t n = lmsize * ncol;
    if (n <= 0) return;
    launch_pdl(k_halve_m, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, alm, lmsize, ncol, s);
    note_launch();
}

void launch_proj_adjoint(const Plan &p, const double *abar, const int32_t *pair_index, const int64_t *noff, int64_t b0,
                         int64_t nbc, double s, double *Abar, cudaStream_t st) {
    const int64_t n = p.lmsize * nbc;
    if (n <= 0) return;
    MonicScale monic;
    monic.c[0] = 1.0;
    for (int k = 1; k < MONIC_MAX; ++k) monic.c[k] = monic.c[k - 1] * (2.0 * k - 1.0) / k;
    launch_pdl(k_proj_adjoint, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, abar, p.d_coef, p.nbasis,
        pair_index, noff, p.lmax, (int)p.nmax, p.lmsize, b0, nbc, s, p.degree, monic, Abar);
    note_launch();
}

void launch_deposit_adjoint(const Plan &p, const double *rtp, int64_t ngal, const double *Dbar, int64_t sb, int64_t sp,
                            int64_t b0, int64_t nbc, double *dw, cudaStream_t st) {
    if (ngal <= 0) return;
    launch_pdl(k_deposit_adjoint, dim3((unsigned)((ngal + 255) / 256)), dim3(256), 0, st,
        rtp, ngal, p.nside, p.npix, p.rmin, p.rmax, (double)p.pieces / (p.rmax - p.rmin), p.pieces, p.degree,
        p.nbasis, Dbar, sb, sp, b0, nbc, dw, p.d_err);
    note_launch();
}

}  // namespace sfb
