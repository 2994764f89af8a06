// FP64 Legendre and Gram contractions on the tensor cores (tcgen05), many
// columns: the analysis, the synthesis and the Gram update of the FP64
// transform, as products of 8-bit digits.
//
// GB300 does about 2 FP64 FMA per clock and SM, so a tiled FP64 GEMM of these
// contractions is bound by the FP64 pipe at 0.6 TFMA/s.  The BF16 tensor cores
// do 4096 MAC per clock and SM; 28 of them per FP64 product leave 146.  Each
// operand value is rounded to a 55-bit integer on a scale common to its whole
// K range (per data column, per table row) and written as seven signed 8-bit
// digits, which BF16 holds exactly (Ozaki, Ogita, Oishi, Rump, Numer.
// Algorithms 59, 2012).  The digit products of level v = a + b (v = 0..6, 28
// of the 49 products; each of the others is below 2^-56 of the scales) are
// summed in one FP32 TMEM accumulator per level.  Their sums over a block of SBK
// chunks are exact in all levels that matter, whatever the tensor cores'
// accumulation order or rounding (SBK says why); after each block the levels are
// joined as a 62-bit integer, rounded once to FP64 and added to the output.  The
// result is as close to the exact sum as an FP64 accumulation in the norm of the
// scales (the whole FP64 field2anlm against 64-bit references: 3.6e-15 on the
// FP64 units, 2.4e-15 so); a value far below its column's largest one keeps
// fewer bits than in FP64, which the ring scales (KXR) make up for in the analysis.
//
// MMA shape: M = 128 data columns, N = table rows (<= 32 a tile), K = 16 a
// step.  Data digit a multiplies the table digits 0..6-a in as few MMAs as N <=
// 256 allows (their planes are stored back to back, and level v is TMEM
// columns [v LS, (v + 1) LS)).  Eight warps read FP64 columns, form the digits
// with integer operations and store them as K-major core matrices; the table
// digits arrive by bulk copy; the last warp issues the MMAs.  7 x 32 TMEM columns and
// three 35 KB stages: two CTAs per SM, one working while the other starts or
// ends (one CTA of 64 rows a SM was slower at every size: field_f64's four
// analyses 150 us against 117, an lmax 189 call 22.4 ms against 21.5).
//
// Measured at 200 columns, nside 64, lmax 58: first analysis 39 us (36 with one scale
// for all rings), a Gram update with the aliased synthesis 22, an aliased analysis 15
// (the transform of these 100 shells took 2332 us a call with tiled FP64 kernels and 1043
// with this file's alone).
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "digit64.cuh"

namespace sfb {
namespace t64 {

__device__ __forceinline__ int rows_of(int m, int par, int lmax) {
    return (m + par <= lmax) ? (lmax - m - par) / 2 + 1 : 0;
}

// Exponents in which the rings of the analysis differ: a ring's values are held on the scale of its largest lambda in
// the block (2^(kx - KXR), kx = KXR for the ring with the largest of all), down to 2^-KXR, and its table column on the
// inverse.  The scale of a data column is then that of its largest contribution, not of its largest value: a
// bright pixel on the short polar rings, whose spectra reach every m, costs the m bits only that it contributes to,
// for contrasts up to 2^KXR between the rings (1e8 near a pole on unit noise, nside 64, lmax 120, each m on its own
// scale: 2e-10 with one scale for all rings, 3e-16 so; an FP64 sum 2e-15).  The sums over l (synthesis, Gram) keep the
// scale of the largest coefficient of an m and parity.
constexpr int KXR = 40;
// Largest value of a column: the key orders the magnitudes on the rings' scales by exponent (its bits 20..); `all`
// also the values that do not enter a product.  A column with a value that is not finite gets the key BAD.
constexpr uint32_t BAD = 0xffffffffu;
struct ColMax {
    uint32_t key = 0, all = 0;
    __device__ __forceinline__ void add(double v, int kx, bool live) {
        const uint32_t hi = (uint32_t)__double2hiint(v) & 0x7fffffffu;
        all = max(all, hi);
        if (live && (hi | (uint32_t)__double2loint(v))) key = max(key, max(hi, 0x100000u) + ((uint32_t)kx << 20));
    }
    __device__ __forceinline__ uint32_t get() const { return all >= 0x7ff00000u ? BAD : key; }
};
// value j of eight packed bytes
__device__ __forceinline__ int byte_of(uint2 w, int j) { return (int)(((j < 4 ? w.x : w.y) >> (8 * (j & 3))) & 0xffu); }

// One CTA: data columns [128 blockIdx.x, +128) x table rows of one tile of block z = (m, parity).
// LMROWS: the data rows are coefficients l = m + parity + 2 k (synthesis, Gram); else rings k (analysis).
// Tiles blockIdx.y < ny0 use task 0, the others task 1 (the Gram update and the aliased rings' synthesis of
// one refinement pass share a launch: both read the current coefficients).
template <bool LMROWS>
__global__ void __launch_bounds__(NTH, 2) k_leg64(const double *data, int64_t ncol, int lmax, int nrn,
                                                  int klim, const int *nzr, Task64 t0, Task64 t1, int ny0,
                                                  int *err) {
    pdl_entry();
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint32_t red[2][MTILE];
    __shared__ int ex_s[NT];
    const int z = blockIdx.z, m = z >> 1, par = z & 1;
    const bool first_task = (int)blockIdx.y < ny0;
    const Task64 &t = first_task ? t0 : t1;
    const int tile = (first_task ? blockIdx.y : blockIdx.y - ny0) + (first_task ? t0.tile0 : t1.tile0);
    const int nrows = rows_of(m, par, lmax);
    const int N = t.n_is_rows ? nrows : t.nout;                  // table rows of the block
    const int nwrite = t.n_is_rows ? nrows : t.nlim;             // rows written
    if (tile * NT >= nwrite || (nrows == 0 && t.n_is_rows)) return;
    const int K = LMROWS ? nrows : min(klim, nrn);               // data rows
    const int64_t col0 = (int64_t)blockIdx.x * MTILE;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c = tid & (MTILE - 1), kh = (tid >> 7) & 1;
    const bool cok = col0 + c < ncol;
    const double *D = LMROWS ? data + col0 + c
                             : data + ((int64_t)(par * (lmax + 1) + m) * nrn) * ncol + col0 + c;
    auto row_at = [&](int k) -> int64_t {
        if constexpr (LMROWS) {
            const int l = m + par + 2 * k;
            return (int64_t)((uint64_t)(uint32_t)(l * (l + 1) / 2 + m) * (uint32_t)ncol);
        }
        return (int64_t)((uint64_t)(uint32_t)k * (uint32_t)ncol);
    };
    int kbeg = 0, kend = K;
    if (!LMROWS && nzr) {                     // zero spectra outside the ring pairs [nzr[0], nzr[1]]
        kbeg = nzr[0];
        kend = min(K, nzr[1] + 1);
        if (kbeg >= kend) kbeg = kend = 0;
    }
    // chunks with a non-zero table digit (the products with the others are exactly zero)
    int lo = kbeg / KC, hi = (kend + KC - 1) / KC - 1;
    if (t.live) {
        const int2 lv = t.live[(int64_t)z * t.ntile + tile];
        lo = max(lo, lv.x);
        hi = min(hi, lv.y);
    }
    if (hi < lo && t.mode == 1) return;       // nothing to add
    const int nch = hi < lo ? 0 : hi - lo + 1;
    const int LS = ls_of(N, tile);
    const int nKtab = ((LMROWS ? nrows : nrn) + KC - 1) / KC;    // chunks of the table's block
    const uint16_t *tab = t.dig + t.off[z] + (int64_t)tile * nKtab * ND * NT * KC + (int64_t)lo * ND * LS * KC;

    // The column's values: largest magnitude over every chunk (the high word orders the magnitudes by exponent);
    // those of the first two chunks to be worked stay in registers.
    double pre[2][8];
    uint2 kxs[2];                             // their rings' scales
    bool use = cok;
    auto load_at = [&](int c16, double (&buf)[8]) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int k = c16 * KC + 8 * kh + j;
            buf[j] = (use && k >= kbeg && k < kend) ? D[row_at(k)] : 0.0;
        }
    };
    auto kx_at = [&](int c16) -> uint2 {
        if constexpr (LMROWS) return make_uint2(0u, 0u);
        return *reinterpret_cast<const uint2 *>(t.kx + (int64_t)z * t.nkx + c16 * KC + 8 * kh);
    };
    auto load = [&](int kc, double (&buf)[8], int i) {
        load_at(lo + kc, buf);
        kxs[i] = kx_at(lo + kc);
    };
    ColMax mx;
    auto top = [&](const double (&buf)[8], uint2 kx, bool in) {
#pragma unroll
        for (int j = 0; j < 8; ++j) mx.add(buf[j], LMROWS ? 0 : byte_of(kx, j), in);
    };
    if (tid < NT && tile * NT + tid < nwrite) ex_s[tid] = t.ex[(int64_t)z * t.exs + tile * NT + tid];
    {
        if (nch > 0) load(0, pre[0], 0);
        if (nch > 1) load(1, pre[1], 1);
        const int skip0 = nch > 0 ? lo : -1, skip1 = nch > 1 ? lo + 1 : -1;
        for (int c16 = kbeg / KC; c16 * KC < kend; ++c16) {
            if (c16 == skip0 || c16 == skip1) continue;
            double buf[8];
            load_at(c16, buf);
            top(buf, kx_at(c16), c16 >= lo && c16 <= hi);
        }
        if (nch > 0) top(pre[0], kxs[0], true);
        if (nch > 1) top(pre[1], kxs[1], true);
        red[kh][c] = mx.get();
    }
    Smem cs;
    const uint32_t tmem = setup(cs, smem);    // includes a __syncthreads
    const uint32_t cmx = max(red[0][c], red[1][c]);
    const int emax = max(1, (int)(cmx >> 20));
    if (cmx == 0 || cmx == BAD) {             // no digits: zero or non-finite columns
        use = false;
#pragma unroll
        for (int j = 0; j < 8; ++j) pre[0][j] = pre[1][j] = 0.0;
    }
    auto fix = [&](double v, int i, int j) { return fixed55(v, LMROWS ? emax : emax - byte_of(kxs[i], j)); };

    // warp w of the epilogue: TMEM lanes 32 (w % 4).. (columns), every other group of four table rows of the tile
    const int lq = warp & 3, hg = warp >> 2;
    const uint32_t lane_base = (uint32_t)(lq * 32) << 16;
    const int cl = lq * 32 + lane;
    const int64_t cc = col0 + cl;
    const bool ook = cc < ncol;
    const uint32_t lmx = max(red[0][cl], red[1][cl]);
    const int lemax = max(1, (int)(lmx >> 20)) - (LMROWS ? 0 : KXR);
    auto at = [&](int i) -> int64_t {                       // output row i of the tile, this lane's column; rows < 2^31
        const int n = tile * NT + i, l = m + par + 2 * n;
        const uint32_t row = t.n_is_rows ? (uint32_t)(l * (l + 1) / 2 + m) : (uint32_t)((par * (lmax + 1) + m) * t.nout + n);
        return (int64_t)((uint64_t)row * (uint32_t)ncol) + cc;
    };
    const int nsb = max(1, (nch + SBK - 1) / SBK);
    for (int sb = 0; sb < nsb; ++sb) {
        const int k0 = sb * SBK, k1 = min(nch, k0 + SBK);
        run_block(cs, tmem, k0, k1, nch, LS, tab, pre, load, fix);
        // what the sums are added to, a group of rows ahead (the first on its way while the MMAs run)
        const double *base = sb > 0 || t.mode == 1 ? t.out : t.mode == 2 ? t.a0 : nullptr;
        double old[4], nold[4];
        auto load_old = [&](int i0, double (&o)[4]) {
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i] = (base && ook && i0 + i < LS && tile * NT + i0 + i < nwrite) ? base[at(i0 + i)] : 0.0;
        };
        load_old(4 * hg, old);
        if (!end_block(cs, sb)) {
            if (tid == 0) atomicOr(err, ERR_TC_TIMEOUT);
            break;                                        // uniform: every thread saw the same value
        }
#pragma unroll 1
        for (int i0 = 4 * hg; i0 < LS && tile * NT + i0 < nwrite; i0 += 8) {           // warp-uniform
            load_old(i0 + 8, nold);
            float v[ND][4];
            load_levels(tmem + lane_base + (uint32_t)i0, LS, v);
            if (ook) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int n = tile * NT + i0 + i;
                    if (n >= nwrite) break;
                    double val = 0.0;
                    if (lmx == BAD) {                     // non-finite data: the plain FP64 sum
                        if (sb == 0)
                            for (int k = kbeg; k < kend; ++k)
                                val = fma(t.tab64[t.tab64_off[z] + n * t.sn + k * t.sk],
                                          data[(D - data) - (col0 + c) + cc + row_at(k)], val);
                    } else if (nch > 0) {
                        const float L[ND] = {v[0][i], v[1][i], v[2][i], v[3][i], v[4][i], v[5][i], v[6][i]};
                        val = round_int(join_int(L), lemax + ex_s[i0 + i] - 1076);
                    }
                    t.out[at(i0 + i)] = t.mode == 2 ? old[i] - val : base ? old[i] + val : val;
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) old[i] = nold[i];
        }
        fence_before();
        __syncthreads();                                      // TMEM is read before the next block's MMAs
        fence_after();
    }
    release(tmem);
}

// The same for short sums (K <= 16 RES, the refinement passes: rows, or the aliased rings).  The column digits are
// formed once and stay in shared memory; the table tiles of both tasks (every gridDim.y-th) come past them one
// after another, the next one's digits copied in during a tile's epilogue.  Of a tile-a-CTA launch half the
// instructions formed the same digits again for each tile (102 maps, lmax 82: 68 us a refinement's Gram update and
// aliased synthesis, 40 so).  Bound: the epilogue's integer operations (about 80 an output), a third of the issue
// slots at four warps a scheduler.
constexpr int RES = 3;
static_assert(RES <= SBK, "a short sum is one exact block");
constexpr size_t SMEM_RES = (size_t)RES * ND * (PLANE_A + NT * KC * 2);

struct TileJob {
    int task, tile, lo, nch, LS, nwrite;
    const uint16_t *tab;
};

template <bool LMROWS>
__global__ void __launch_bounds__(NTH, 2) k_leg64_short(const double *data, int64_t ncol, int lmax,
                                                        int nrn, int klim, Task64 t0, Task64 t1, int ny0, int ny1,
                                                        int *err) {
    pdl_entry();
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint32_t red[2][MTILE];
    __shared__ int ex_s[2][NT];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ uint32_t slot;
    const int z = blockIdx.z, m = z >> 1, par = z & 1;
    const int nrows = rows_of(m, par, lmax);
    const int K = LMROWS ? nrows : min(klim, nrn);
    const int nK = (K + KC - 1) / KC, nKtab = LMROWS ? nK : (nrn + KC - 1) / KC;
    const int64_t col0 = (int64_t)blockIdx.x * MTILE;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c = tid & (MTILE - 1), kh = tid >> 7;
    const bool cok = col0 + c < ncol;
    const double *D = LMROWS ? data : data + ((int64_t)(par * (lmax + 1) + m) * nrn) * ncol;
    auto row_at = [&](int k) -> int64_t {
        const int l = m + par + 2 * k;
        const uint32_t row = LMROWS ? (uint32_t)(l * (l + 1) / 2 + m) : (uint32_t)k;
        return (int64_t)((uint64_t)row * (uint32_t)ncol);
    };
    // job i of this block: tiles of task 0, then of task 1; false: nothing to do there
    auto job_at = [&](int i, TileJob &j) -> bool {
        j.task = i < ny0 ? 0 : 1;
        const Task64 &t = j.task ? t1 : t0;
        j.tile = (j.task ? i - ny0 : i) + t.tile0;
        const int N = t.n_is_rows ? nrows : t.nout;
        j.nwrite = t.n_is_rows ? nrows : t.nlim;
        if (j.tile * NT >= j.nwrite || (t.n_is_rows && nrows == 0)) return false;
        int lo = 0, hi = nK - 1;
        if (t.live) {
            const int2 lv = t.live[(int64_t)z * t.ntile + j.tile];
            lo = max(lo, lv.x);
            hi = min(hi, lv.y);
        }
        j.nch = hi < lo ? 0 : hi - lo + 1;
        j.lo = j.nch ? lo : 0;
        if (t.mode == 1 && j.nch == 0) return false;
        j.LS = ls_of(N, j.tile);
        j.tab = t.dig + t.off[z] + (int64_t)j.tile * nKtab * ND * NT * KC + (int64_t)j.lo * ND * j.LS * KC;
        return true;
    };
    auto next_job = [&](int i, TileJob &j) -> int {          // the first job at or after i, or -1
        for (; i < ny0 + ny1; i += gridDim.y)
            if (job_at(i, j)) return i;
        return -1;
    };
    TileJob job;
    int cur = next_job(blockIdx.y, job);
    if (cur < 0) return;

    double v[RES][8];
    uint2 kxs[RES];                                           // the rings' scales
    ColMax mx;
#pragma unroll
    for (int q = 0; q < RES; ++q) {
        if constexpr (!LMROWS)
            if (q < nK) kxs[q] = *reinterpret_cast<const uint2 *>(t0.kx + (int64_t)z * t0.nkx + q * KC + 8 * kh);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int k = q * KC + 8 * kh + j;
            v[q][j] = (cok && k < K) ? D[row_at(k) + col0 + c] : 0.0;
        }
    }
#pragma unroll
    for (int q = 0; q < RES; ++q)
#pragma unroll
        for (int j = 0; j < 8; ++j) mx.add(v[q][j], LMROWS || q >= nK ? 0 : byte_of(kxs[q], j), true);
    red[kh][c] = mx.get();
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
    unsigned char *sA = smem, *sB = smem + (size_t)RES * ND * PLANE_A;
    auto fetch = [&](const TileJob &j) {
        const uint32_t bytes = (uint32_t)j.nch * ND * j.LS * KC * 2;
        mbar_expect_tx(full_b, bytes);
        bulk_g2s(sB, j.tab, bytes, full_b);
    };
    if (tid == 0 && job.nch > 0) fetch(job);
    {
        const uint32_t cmx = max(red[0][c], red[1][c]);
        const int emax = max(1, (int)(cmx >> 20));
        const bool dead = cmx == 0 || cmx == BAD;                // no digits: zero or non-finite columns
        const uint32_t off = core_off(c, 8 * kh);
#pragma unroll
        for (int q = 0; q < RES; ++q) {
            if (q >= nK) break;
            uint32_t w[ND][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t u[ND];
                const int e0 = LMROWS ? emax : emax - byte_of(kxs[q], 2 * j);
                const int e1 = LMROWS ? emax : emax - byte_of(kxs[q], 2 * j + 1);
                digits2(dead ? 0 : fixed55(v[q][2 * j], e0), dead ? 0 : fixed55(v[q][2 * j + 1], e1), u);
#pragma unroll
                for (int d = 0; d < ND; ++d) w[d][j] = u[d];
            }
#pragma unroll
            for (int d = 0; d < ND; ++d)
                *reinterpret_cast<uint4 *>(sA + (q * ND + d) * PLANE_A + off) = make_uint4(w[d][0], w[d][1], w[d][2], w[d][3]);
        }
        fence_proxy_async();
    }
    // warp w of the epilogue: TMEM lanes 32 (w % 4).. (columns), every other group of four table rows of the tile
    const int lq = warp & 3, hg = warp >> 2;
    const uint32_t lane_base = (uint32_t)(lq * 32) << 16;
    const int cl = lq * 32 + lane;
    const int64_t cc = col0 + cl;
    const bool ook = cc < ncol;
    const uint32_t lmx = max(red[0][cl], red[1][cl]);
    const int lemax = max(1, (int)(lmx >> 20)) - (LMROWS ? 0 : KXR);
    int uses = 0;                                             // tiles whose digits were fetched: barrier phases
    for (int step = 0; cur >= 0; ++step) {
        const Task64 &t = job.task ? t1 : t0;
        int *exs = ex_s[step & 1];
        if (tid < NT && job.tile * NT + tid < job.nwrite) exs[tid] = t.ex[(int64_t)z * t.exs + job.tile * NT + tid];
        auto at = [&](int i) -> int64_t {                   // output row i of the tile, this lane's column; rows < 2^31
            const int n = job.tile * NT + i, l = m + par + 2 * n;
            const uint32_t row = t.n_is_rows ? (uint32_t)(l * (l + 1) / 2 + m)
                                             : (uint32_t)((par * (lmax + 1) + m) * t.nout + n);
            return (int64_t)((uint64_t)row * (uint32_t)ncol) + cc;
        };
        if (step == 0) __syncthreads();                       // every digit is written
        const uint32_t ph = (uint32_t)(uses & 1);
        if (job.nch > 0 && tid == 32 * MMA_WARP) {
            if (mbar_wait(full_b, ph)) {
                fence_after();
                for (int q = 0; q < job.nch; ++q)
                    issue(tmem, smem_u32(sA) + (job.lo + q) * ND * PLANE_A, smem_u32(sB) + q * ND * job.LS * KC * 2, job.LS,
                          q == 0);
                mma_commit(done);
            }                                                 // (else done stays pending and the wait below gives up)
        }
        __syncwarp();
        const double *base = t.mode == 1 ? t.out : t.mode == 2 ? t.a0 : nullptr;
        double old[4], nold[4];                               // what the sums are added to, a group of rows ahead
        auto load_old = [&](int i0, double (&o)[4]) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                o[i] = (base && ook && i0 + i < job.LS && job.tile * NT + i0 + i < job.nwrite) ? base[at(i0 + i)] : 0.0;
        };
        load_old(4 * hg, old);
        const bool fin = job.nch == 0 || mbar_wait(done, ph);
        fence_after();
        if (!__syncthreads_and(fin)) {
            if (tid == 0) atomicOr(err, ERR_TC_TIMEOUT);
            break;
        }
        if (job.nch > 0) ++uses;
        TileJob nxt;
        const int ni = next_job(cur + gridDim.y, nxt);
        if (tid == 0 && ni >= 0 && nxt.nch > 0) fetch(nxt);      // the MMAs have read this tile's digits
#pragma unroll 1
        for (int i0 = 4 * hg; i0 < job.LS && job.tile * NT + i0 < job.nwrite; i0 += 8) {         // warp-uniform
            load_old(i0 + 8, nold);
            float L4[ND][4];
            load_levels(tmem + lane_base + (uint32_t)i0, job.LS, L4);
            if (ook) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int n = job.tile * NT + i0 + i;
                    if (n >= job.nwrite) break;
                    double val = 0.0;
                    if (lmx == BAD) {                         // non-finite data: the plain FP64 sum
                        for (int k = 0; k < K; ++k)
                            val = fma(t.tab64[t.tab64_off[z] + n * t.sn + k * t.sk], D[row_at(k) + cc], val);
                    } else if (job.nch > 0) {
                        const float L[ND] = {L4[0][i], L4[1][i], L4[2][i], L4[3][i], L4[4][i], L4[5][i], L4[6][i]};
                        val = round_int(join_int(L), lemax + exs[i0 + i] - 1076);
                    }
                    t.out[at(i0 + i)] = t.mode == 2 ? old[i] - val : base ? old[i] + val : val;
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) old[i] = nold[i];
        }
        fence_before();
        __syncthreads();                                      // TMEM is read before the next tile's MMAs
        fence_after();
        cur = ni;
        job = nxt;
    }
    release(tmem);
}

// ---- tables ---------------------------------------------------------------------------------------------------
// kind 0: analysis (N = rows li, K = rings), 1: synthesis (N = rings, K = rows), 2: Gram (N = K = rows);
// element (n, k) of block z at off64[z] + n sn + k sk.
__device__ __forceinline__ void dims(int kind, int z, int lmax, int nrn, int &N, int &K) {
    const int nrows = rows_of(z >> 1, z & 1, lmax);
    N = kind == 1 ? nrn : nrows;
    K = kind == 0 ? nrn : nrows;
}

// the analysis table's ring scales kx (KXR above), one block per (m, parity)
__global__ void __launch_bounds__(256) k64_ringexp(const double *tab, const int64_t *off64, int lmax, int nrn, int nkx,
                                                   uint8_t *kx) {
    pdl_entry();
    __shared__ int most;
    const int z = blockIdx.x, nrows = rows_of(z >> 1, z & 1, lmax);
    if (threadIdx.x == 0) most = -(1 << 20);
    __syncthreads();
    auto exponent = [&](int r) {
        double mx = 0.0;
        for (int n = 0; n < nrows; ++n) mx = fmax(mx, fabs(tab[off64[z] + (int64_t)n * nrn + r]));
        return mx > 0.0 && isfinite(mx) ? ilogb(mx) : -(1 << 20);
    };
    for (int r = threadIdx.x; r < nrn; r += 256) atomicMax(&most, exponent(r));
    __syncthreads();
    for (int r = threadIdx.x; r < nkx; r += 256)
        kx[(int64_t)z * nkx + r] = (uint8_t)(r < nrn ? max(0, KXR + exponent(r) - most) : 0);
}
// element (n, k) of a table on its column's scale
__device__ __forceinline__ double element(const double *tab, int64_t at, const uint8_t *kx, int64_t k) {
    return kx ? ldexp(tab[at], KXR - (int)kx[k]) : tab[at];
}

// exponent E of every table row, |v| < 2^E (one warp per row)
__global__ void k64_rowexp(int kind, const double *tab, const int64_t *off64, int64_t sn,
                           int64_t sk, int lmax, int nrn, int exs, int16_t *ex, const uint8_t *kx, int nkx) {
    pdl_entry();
    const int z = blockIdx.y, lane = threadIdx.x & 31;
    int N, K;
    dims(kind, z, lmax, nrn, N, K);
    for (int n = blockIdx.x * 8 + (threadIdx.x >> 5); n < N; n += gridDim.x * 8) {
        double mx = 0.0;
        for (int k = lane; k < K; k += 32)
            mx = fmax(mx, fabs(element(tab, off64[z] + n * sn + k * sk, kx, (int64_t)z * nkx + k)));
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) ex[(int64_t)z * exs + n] = (int16_t)(mx > 0.0 && isfinite(mx) ? ilogb(mx) + 1 : 0);
    }
}

// one block per (tile and chunk, z): the digit planes and the live chunk range of the tile
__global__ void __launch_bounds__(256) k64_build(int kind, const double *tab,
                                                 const int64_t *off64, int64_t sn, int64_t sk, int lmax,
                                                 int nrn, int exs, const int16_t *ex, int ntile,
                                                 int nkmax, const int64_t *off,
                                                 uint16_t *dig, int2 *live, const uint8_t *kx, int nkx) {
    pdl_entry();
    const int z = blockIdx.y, tile = blockIdx.x / nkmax, kc = blockIdx.x % nkmax;
    int N, K;
    dims(kind, z, lmax, nrn, N, K);
    const int nK = (K + KC - 1) / KC;
    if (tile * NT >= N || kc >= nK) return;
    const int LS = ls_of(N, tile);
    uint16_t *base = dig + off[z] + (int64_t)tile * nK * ND * NT * KC + (int64_t)kc * ND * LS * KC;
    int any = 0;
    for (int e = threadIdx.x; e < LS * KC; e += blockDim.x) {
        const int nn = sn == 1 ? e % LS : e / KC, k = sn == 1 ? e / LS : e % KC;
        const int n = tile * NT + nn, kk = kc * KC + k;
        int64_t q = 0;
        if (n < N && kk < K)
            q = llrint(ldexp(element(tab, off64[z] + n * sn + kk * sk, kx, (int64_t)z * nkx + kk),
                             55 - (int)ex[(int64_t)z * exs + n]));
        any |= q != 0;
        uint32_t w[ND];
        digits2(q, 0, w);
#pragma unroll
        for (int d = 0; d < ND; ++d) base[(int64_t)d * LS * KC + (core_off(nn, k) >> 1)] = (uint16_t)(w[d] & 0xffffu);
    }
    if (__syncthreads_or(any) && threadIdx.x == 0) {
        atomicMin(&live[(int64_t)z * ntile + tile].x, kc);
        atomicMax(&live[(int64_t)z * ntile + tile].y, kc);
    }
}

__global__ void k64_fill(int2 *r, int64_t n) {
    pdl_entry();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        r[i] = make_int2(0x7fffffff, -1);
}

}  // namespace t64

// Digit tables of the plan, built at the first FP64 transform of many columns that finds the memory for them: 14 bytes
// a table element against 8 in FP64, at most a sixteenth of the free device memory.  Without it the call runs on the
// FP64 units and the next one asks again; SFBGPU_TC64=0 keeps the plan on them (state -1).
bool ensure_tc64(Plan &p, cudaStream_t st) {
    if (p.tc64_state) return p.tc64_state > 0;
    if (const char *e = std::getenv("SFBGPU_TC64"))
        if (e[0] == '0') {
            p.tc64_state = -1;
            return false;
        }
    const int nz = 2 * (p.lmax + 1);
    const int nrows0 = p.lmax / 2 + 1;
    constexpr int NT = t64::NT;
    std::vector<int64_t> off[3];
    size_t bytes[3] = {};
    int exs[3], ntile[3], nkmax[3];
    const int nkind = p.d_gram64 ? 3 : 2;
    size_t total = 0;
    for (int kind = 0; kind < nkind; ++kind) {
        const int Nmax = kind == 1 ? (int)p.nrn : nrows0, Kmax = kind == 0 ? (int)p.nrn : nrows0;
        exs[kind] = Nmax;
        ntile[kind] = (Nmax + NT - 1) / NT;
        nkmax[kind] = (Kmax + t64::KC - 1) / t64::KC;
        int64_t o = 0;
        for (int z = 0; z < nz; ++z) {
            const int m = z >> 1, par = z & 1;
            const int nr = (m + par <= p.lmax) ? (p.lmax - m - par) / 2 + 1 : 0;
            const int N = kind == 1 ? (int)p.nrn : nr, K = kind == 0 ? (int)p.nrn : nr;
            off[kind].push_back(o);
            const int64_t nK = (K + t64::KC - 1) / t64::KC;
            if (nr == 0) continue;
            for (int t = 0; t * NT < N; ++t) o += nK * t64::ND * t64::ls_of(N, t) * t64::KC;
        }
        bytes[kind] = (size_t)o * 2;
        total += bytes[kind];
    }
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) != cudaSuccess || total > fr / 16) {
        cudaGetLastError();
        return false;
    }
    auto give_back = [&] {
        cudaGetLastError();
        for (int kind = 0; kind < nkind; ++kind) {
            if (p.t64_mem[kind]) cudaFree(p.t64_mem[kind]);
            p.t64_mem[kind] = nullptr;
            p.device_bytes -= p.t64_bytes[kind];
            p.t64_bytes[kind] = 0;
        }
        return false;
    };
    for (int kind = 0; kind < nkind; ++kind) {
        // one allocation: [digits][offsets][live ranges][exponents][ring scales], each part 256-byte aligned
        auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
        const size_t b0 = up(bytes[kind] + 16), b1 = up(nz * sizeof(int64_t)),
                     b2 = up((size_t)nz * ntile[kind] * sizeof(int2)), b3 = up((size_t)nz * exs[kind] * sizeof(int16_t));
        const int nkx = kind == 0 ? nkmax[0] * t64::KC : 0;
        const size_t b4 = up((size_t)nz * nkx);
        unsigned char *d = nullptr;
        if (cudaMalloc(&d, b0 + b1 + b2 + b3 + b4) != cudaSuccess) return give_back();
        Task64 &t = p.t64[kind];
        p.t64_mem[kind] = d;
        p.t64_bytes[kind] = (int64_t)(b0 + b1 + b2 + b3 + b4);
        p.device_bytes += p.t64_bytes[kind];
        t.dig = reinterpret_cast<uint16_t *>(d);
        t.off = reinterpret_cast<int64_t *>(d + b0);
        t.live = reinterpret_cast<int2 *>(d + b0 + b1);
        t.ex = reinterpret_cast<int16_t *>(d + b0 + b1 + b2);
        t.kx = kind == 0 ? d + b0 + b1 + b2 + b3 : nullptr;
        t.nkx = nkx;
        t.exs = exs[kind];
        t.ntile = ntile[kind];
        t.n_is_rows = kind != 1;
        t.nout = (int)p.nrn;
        t.tab64 = kind == 2 ? p.d_gram64 : p.d_lam;
        t.tab64_off = kind == 2 ? p.d_gram_off : p.d_lam_off;
        t.sn = kind == 0 ? p.nrn : 1;
        t.sk = kind == 0 ? 1 : kind == 1 ? p.nrn : p.gram_rows;
        if (cudaMemcpyAsync(d + b0, off[kind].data(), nz * sizeof(int64_t), cudaMemcpyHostToDevice, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return give_back();
        const int64_t nl = (int64_t)nz * ntile[kind];
        launch_pdl(t64::k64_fill, dim3((unsigned)((nl + 255) / 256)), dim3(256), 0, st, const_cast<int2 *>(t.live),
            nl);
        if (kind == 0) {
            launch_pdl(t64::k64_ringexp, dim3((unsigned)nz), dim3(256), 0, st, t.tab64, t.tab64_off, p.lmax,
                (int)p.nrn, nkx, const_cast<uint8_t *>(t.kx));
            note_launch();
        }
        launch_pdl(t64::k64_rowexp, dim3(16, (unsigned)nz), dim3(256), 0, st, kind, t.tab64, t.tab64_off, t.sn, t.sk,
            p.lmax, (int)p.nrn, t.exs, const_cast<int16_t *>(t.ex), t.kx, nkx);
        launch_pdl(t64::k64_build, dim3((unsigned)(ntile[kind] * nkmax[kind]), (unsigned)nz), dim3(256), 0, st,
            kind, t.tab64, t.tab64_off, t.sn, t.sk, p.lmax, (int)p.nrn, t.exs, t.ex, t.ntile, nkmax[kind], t.off,
            const_cast<uint16_t *>(t.dig), const_cast<int2 *>(t.live), t.kx, nkx);
        note_launch();
        note_launch();
        note_launch();
    }
    if (cudaGetLastError() != cudaSuccess) return give_back();
    p.tc64_state = 1;
    return true;
}

static dim3 grid64(const Plan &p, int64_t ncol, int ny) {
    return dim3((unsigned)((ncol + t64::MTILE - 1) / t64::MTILE), (unsigned)ny, (unsigned)(2 * (p.lmax + 1)));
}

// blocks a column tile and (m, parity) are split into, so that two CTAs per SM have work
static unsigned short_split(const Plan &p, int64_t ncol, int ntile) {
    const int64_t ctas = ((ncol + t64::MTILE - 1) / t64::MTILE) * 2 * (p.lmax + 1);
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ntile, 304 / ctas));
}

void launch_leg_analysis64(const Plan &p, const double *F, int64_t ncol, double *A, bool accumulate, cudaStream_t st,
                           int rlim, const int *nzr) {
    Task64 t = p.t64[0];
    t.out = A;
    t.mode = accumulate ? 1 : 0;
    if (!nzr && rlim <= t64::RES * t64::KC) {
        set_smem(t64::k_leg64_short<false>, t64::SMEM_RES);
        launch_pdl(t64::k_leg64_short<false>, dim3(grid64(p, ncol, (int)short_split(p, ncol, t.ntile))),
            dim3(t64::NTH), t64::SMEM_RES, st, F, ncol, p.lmax, (int)p.nrn, rlim, t, t, t.ntile, 0, p.d_err);
        note_launch();
        return;
    }
    set_smem(t64::k_leg64<false>, t64::SMEM);
    launch_pdl(t64::k_leg64<false>, dim3(grid64(p, ncol, t.ntile)), dim3(t64::NTH), t64::SMEM, st, F, ncol, p.lmax,
        (int)p.nrn, rlim, nzr, t, t, t.ntile, p.d_err);
    note_launch();
}

static void leg_synthesis64(const Plan &p, const double *A, int64_t ncol, const Task64 &g, const Task64 &s, int ny0,
                            int ny1, cudaStream_t st) {
    if (ny0 + ny1 == 0) return;
    if (p.lmax / 2 + 1 <= t64::RES * t64::KC) {
        set_smem(t64::k_leg64_short<true>, t64::SMEM_RES);
        launch_pdl(t64::k_leg64_short<true>, dim3(grid64(p, ncol, (int)short_split(p, ncol, ny0 + ny1))),
            dim3(t64::NTH), t64::SMEM_RES, st, A, ncol, p.lmax, (int)p.nrn, 0, g, s, ny0, ny1, p.d_err);
    } else {
        set_smem(t64::k_leg64<true>, t64::SMEM);
        launch_pdl(t64::k_leg64<true>, dim3(grid64(p, ncol, ny0 + ny1)), dim3(t64::NTH), t64::SMEM, st, A, ncol,
            p.lmax, (int)p.nrn, 0, nullptr, g, s, ny0, p.d_err);
    }
    note_launch();
}

// G of the rings r < rlim (G may be null) and, with Anew, the Gram update Anew = A0 - D A.
void launch_leg_synthesis64(const Plan &p, const double *A, int64_t ncol, double *G, cudaStream_t st, int rlim,
                            const double *A0, double *Anew) {
    Task64 g = p.t64[2], s = p.t64[1];
    g.out = Anew;
    g.a0 = A0;
    g.mode = 2;
    s.out = G;
    s.mode = 0;
    s.nlim = rlim;
    leg_synthesis64(p, A, ncol, g, s, Anew ? g.ntile : 0, G && rlim > 0 ? (rlim + t64::NT - 1) / t64::NT : 0, st);
}

// G of the tiles of LEG64_TILE rings that hold the rings [r0, r1).
void launch_leg_synthesis64_rings(const Plan &p, const double *A, int64_t ncol, double *G, int r0, int r1,
                                  cudaStream_t st) {
    Task64 s = p.t64[1];
    s.out = G;
    s.mode = 0;
    s.tile0 = r0 / t64::NT;
    const int t1 = (r1 + t64::NT - 1) / t64::NT;
    s.nlim = std::min((int)p.nrn, t1 * t64::NT);
    if (r1 > r0) leg_synthesis64(p, A, ncol, s, s, 0, t1 - s.tile0, st);
}

}  // namespace sfb
