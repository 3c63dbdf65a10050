// fpho_flux.cu -- the linear flux solve of fixed-shape sources on the device.
//
// forcepho's optimize_fluxes (forcepho/fitting.py:573-627) takes the design
// matrix X (n_sources x n_pix per band: each source's model at unit flux,
// forcepho/patches/device_patch.py:185-238) and the data y, and solves the
// weighted normal equations per band:
//     ATA = (X w)(X w)^T,  ATb = (X w)(y w),  fluxes = ATA^-1 ATb,
// returning ATA as the flux precision matrix.  Here the normal equations are
// formed without writing X anywhere:
//   normal_tiles   one CTA per pixel tile builds the unit-flux model of every
//                  source at the tile's pixels into shared memory (the design
//                  kernel's scan, staging and exponential), then forms the
//                  tile's FP64 partial sums of ATA (upper triangle) and ATb;
//                  normal_tiles_mma, for up to 63 sources over 256-pixel
//                  tiles, forms them on the FP64 tensor cores;
//   normal_reduce  sums the partials of each band's tiles in a fixed order
//                  (FP64) into ATA (both triangles) and ATb;
//   normal_solve   one CTA per band: FP64 Cholesky factorisation and the two
//                  triangular solves; a band whose ATA is not positive definite
//                  gets NaN fluxes and a status of 1.
// The data y are the patch's device data (after fpho_patch_swap_data_residual
// of subtract_fixed, the data with the fixed sources subtracted).
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "fpho_handle.h"
#include "fpho_impl.cuh"
#include "fpho_internal.h"
#include "fpho_kernels.cuh"
#include "fpho_tile.cuh"

namespace fpho {
namespace {

// Shared memory of normal_tiles: [records live_cap x 128 B][kept idx_cap x 4 B]
// [unit-flux rows ns x (tile + 1) floats][w, y: 2 x tile floats].  Rows are
// padded by one float so that threads reading different rows at the same
// pixel hit different banks.
__host__ __device__ inline size_t normal_smem_bytes(int tile, int live_cap, int idx_cap, int ns) {
    return (size_t)live_cap * GSTAGE * 4 + (size_t)idx_cap * 4 + (size_t)ns * (tile + 1) * 4 +
           (size_t)2 * tile * 4;
}

// the (s, t) pair, s <= t, of upper-triangle index p of an ns x ns matrix
__device__ __forceinline__ void upper_pair(int p, int ns, int &s, int &t) {
    s = 0;
    while (p >= ns - s) {
        p -= ns - s;
        ++s;
    }
    t = s + p;
}

// A tile's partial normal equations from its unit-flux rows (ns rows of
// TP + 1 floats), weights ws and data ys: the upper triangle of
// sum w^2 X_s X_t, then sum w^2 X_s y, each term summed in FP64 over the
// tile's pixels in order.  Every thread of the CTA takes terms.
template <int NT, int TP>
__device__ __forceinline__ void tile_normal_partials(const float *rows, const float *ws,
                                                     const float *ys, int ns, int count,
                                                     int n_terms, double *out) {
    const int n_pairs = ns * (ns + 1) / 2;
    for (int p = threadIdx.x; p < n_terms; p += NT) {
        int s, t;
        const float *other;
        if (p < n_pairs) {
            upper_pair(p, ns, s, t);
            other = rows + (size_t)t * (TP + 1);
        } else {
            s = p - n_pairs;
            other = ys;
        }
        const float *xs_ = rows + (size_t)s * (TP + 1);
        double acc = 0.0;
        for (int li = 0; li < count; ++li) {
            const double w = (double)ws[li];
            acc = fma(w * w * (double)xs_[li], (double)other[li], acc);
        }
        out[p] = acc;
    }
}

template <int NT, int K>
__global__ void __launch_bounds__(NT) normal_tiles(TileArgs A, double *pnorm, int n_terms) {
    static_assert(K % 2 == 0, "pixels per thread must be even (packed pairs)");
    constexpr int KP = K / 2;
    constexpr int TP = NT * K;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t mbar;
    const int tid = threadIdx.x;
    if (tid == 0) {
        mbar_init(&mbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    let_next_kernel_start();
    uint32_t phase = 0;
    const int tile = blockIdx.x;
    const int cap = A.live_cap;
    const int ns = A.pv.n_sources;
    float *recs = reinterpret_cast<float *>(smem);
    int *kept = reinterpret_cast<int *>(smem + (size_t)cap * GSTAGE * 4);
    float *rows = reinterpret_cast<float *>(kept + A.idx_cap);  // [ns][TP + 1]
    float *ws = rows + (size_t)ns * (TP + 1);
    float *ys = ws + TP;

    const TileDesc td = A.tiles[tile];
    const float4 bb = A.tbox_all[tile];
    const int g0 = A.pv.gauss_start[td.exposure];
    const int g1 = A.pv.gauss_start[td.exposure + 1];
    const int npsf = A.pv.exp_npsf[td.exposure];
    for (int j = tid; j < ns * (TP + 1); j += NT) rows[j] = 0.0f;
    wait_for_earlier_kernel();  // before the pixel arrays, which a kernel may have filled
    for (int li = tid; li < TP; li += NT) {
        const bool ok = li < td.count;
        ws[li] = ok ? A.pv.ierr[td.pix_begin + li] : 0.0f;
        ys[li] = ok ? A.pv.data[td.pix_begin + li] : 0.0f;
    }
    __syncthreads();  // barrier initialised, rows cleared

    const float xmid = 0.5f * (bb.x + bb.y), ymid = 0.5f * (bb.z + bb.w);
    v2 Xp[KP], Yp[KP], M[KP];
#pragma unroll
    for (int j = 0; j < KP; ++j) {
        float xs[2], yv[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int li = tid + (2 * j + h) * NT;
            const bool ok = li < td.count;
            const int pix = td.pix_begin + (ok ? li : 0);
            xs[h] = ok ? A.pv.xpix[pix] : xmid;
            yv[h] = ok ? A.pv.ypix[pix] : ymid;
        }
        Xp[j] = pk(xs[0], xs[1]);
        Yp[j] = pk(yv[0], yv[1]);
        M[j] = 0ull;
    }
    const int n_live = scan_tile<NT, true>(A, bb, g0, g1, npsf, kept,
                                            reinterpret_cast<unsigned *>(recs), cap * GSTAGE);
    const v2 KEXP2 = pk1(KEXP), KEXPLO2 = pk1(KEXP_LO), CM24 = pk1(-1.0f / 24.0f);
    for (int c0 = 0; c0 < n_live; c0 += cap) {
        const int n = min(cap, n_live - c0);
        if (c0 > 0) __syncthreads();
        stage_records<NT, GSTAGE>(recs, A.gtab + (size_t)g0 * GREC, kept, c0, n, 0, &mbar, phase, A.err);
        for (int i = 0; i < n; ++i) {
            const float *r = recs + (size_t)i * GSTAGE;
            int flag = kept[c0 + i];
            if (!(flag & FLAG_LAST_SRC) && i + 1 < n) {
                // two Gaussians of the same source: their exponentials interleave
                design_pairs2<KP>(Xp, Yp, M, r, r + GSTAGE, CM24, KEXP2, KEXPLO2);
                ++i;
                r += GSTAGE;
                flag = kept[c0 + i];
            } else {
                design_one<KP>(Xp, Yp, M, r, CM24, KEXP2, KEXPLO2);
            }
            if ((flag & FLAG_LAST_SRC) || i == n - 1) {
                // a source's Gaussians are contiguous in the kept list; one
                // that spans two chunks is flushed twice and added
                const int src = min((unsigned)__float_as_int(r[R_SRC]), (unsigned)(ns - 1));
                float *row = rows + (size_t)src * (TP + 1);
#pragma unroll
                for (int j = 0; j < KP; ++j) {
                    float m0, m1;
                    unpk(M[j], m0, m1);  // accumulated -model
                    row[tid + 2 * j * NT] -= m0;
                    row[tid + (2 * j + 1) * NT] -= m1;
                    M[j] = 0ull;
                }
            }
        }
    }
    __syncthreads();
    tile_normal_partials<NT, TP>(rows, ws, ys, ns, td.count, n_terms,
                                 pnorm + (size_t)tile * n_terms);
}

// index of the pair (s, t), s <= t, in the upper triangle of an ns x ns matrix
__device__ __forceinline__ int upper_index(int s, int t, int ns) {
    return s * ns - s * (s - 1) / 2 + (t - s);
}

__device__ __forceinline__ void mma_f64(double &c0, double &c1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}

// The same partials with the products on the FP64 tensor cores, for tiles of
// 256 pixels and ns <= NORMAL_MMA_SOURCES.  Each of two warps takes 128 pixels,
// four consecutive ones per lane, through all kept Gaussians (four warps of two
// per lane took 304 us: the shared coordinate and the record loads then serve
// one pair each); a source's model stays in registers (flushed where the other kernel's stages of
// DESIGN_LIVE_CAP records end, so the unit-flux rows are the same floats) and
// goes to shared memory; row ns is y.  Then each warp multiplies its own
// pixels' rows, times w in double (exact, as a product of two floats), with
// one another, eight by eight rows and four pixels an instruction: a lane's
// element of the left operand is its element of the right one, so a block of
// rows is loaded once.  (One thread per term, three conversions and three
// FP64 operations a pixel and term, took more than half of 383 us on the
// 20-source patch.)  Rows are MMA_ROW floats apart: the lanes of a load (eight
// rows, four pixels) then hit different banks.
constexpr int NORMAL_MMA_SOURCES = 63;
constexpr int MMA_WARPS = 2, MMA_TILE = 256, MMA_ROW = MMA_TILE + 4, MMA_STAGE = 64;
constexpr int MMA_PX = MMA_TILE / MMA_WARPS, MMA_K = MMA_PX / 32;  // pixels per warp, per lane
static_assert(MMA_STAGE == DESIGN_LIVE_CAP, "a stage is a flush interval");
__host__ __device__ inline int mma_rows(int ns) { return (ns + 1 + 7) / 8 * 8; }
__host__ __device__ inline size_t mma_smem_bytes(int idx_cap, int ns) {
    return (size_t)MMA_STAGE * GSTAGE * 4 + (size_t)(mma_rows(ns) * MMA_ROW + MMA_TILE) * 4 +
           (size_t)idx_cap * 4;
}

__global__ void __launch_bounds__(32 * MMA_WARPS) normal_tiles_mma(TileArgs A, double *pnorm,
                                                                   int n_terms) {
    constexpr int NT = 32 * MMA_WARPS;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t mbar;
    __shared__ __align__(16) float s_zero[GSTAGE];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < GSTAGE) s_zero[tid] = 0.0f;
    if (tid == 0) {
        mbar_init(&mbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    let_next_kernel_start();
    uint32_t phase = 0;
    const int tile = blockIdx.x;
    const int ns = A.pv.n_sources, nr = mma_rows(ns);
    float *recs = reinterpret_cast<float *>(smem);
    float *rows = recs + MMA_STAGE * GSTAGE;  // [nr][MMA_ROW]
    float *ws = rows + (size_t)nr * MMA_ROW;  // [MMA_TILE]
    int *kept = reinterpret_cast<int *>(ws + MMA_TILE);

    const TileDesc td = A.tiles[tile];
    const float4 bb = A.tbox_all[tile];
    const int g0 = A.pv.gauss_start[td.exposure];
    const int g1 = A.pv.gauss_start[td.exposure + 1];
    const int npsf = A.pv.exp_npsf[td.exposure];
    for (int j = tid; j < nr * MMA_ROW; j += NT) rows[j] = 0.0f;
    wait_for_earlier_kernel();  // before the pixel arrays, which a kernel may have filled
    const float xmid = 0.5f * (bb.x + bb.y), ymid = 0.5f * (bb.z + bb.w);
    constexpr int KP = MMA_K / 2;
    float w[MMA_K], y[MMA_K];
    bool counts[MMA_K];
    v2 Xp[KP], Yp[KP], M[KP], X[KP];  // X: the source's unit-flux model so far
#pragma unroll
    for (int j = 0; j < KP; ++j) {
        float xs[2], ys[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = 2 * j + h, li = MMA_PX * warp + MMA_K * lane + k;
            const bool ok = li < td.count;
            const int pix = td.pix_begin + (ok ? li : 0);
            xs[h] = ok ? A.pv.xpix[pix] : xmid;
            ys[h] = ok ? A.pv.ypix[pix] : ymid;
            w[k] = ok ? A.pv.ierr[pix] : 0.0f;
            y[k] = ok ? A.pv.data[pix] : 0.0f;
            counts[k] = w[k] != 0.0f;  // others have no part in the sums
        }
        Xp[j] = pk(xs[0], xs[1]);
        Yp[j] = pk(ys[0], ys[1]);
        M[j] = X[j] = 0ull;
    }
    const int share = share_of<8>(A.tile_misfit[tile], false);
    const int n_live = scan_tile<NT, true>(A, bb, g0, g1, npsf, kept,
                                           reinterpret_cast<unsigned *>(recs),
                                           MMA_STAGE * GSTAGE);
    const v2 KEXP2 = pk1(KEXP), KEXPLO2 = pk1(KEXP_LO), CM24 = pk1(-1.0f / 24.0f);
    const v2 MINUS1 = pk1(-1.0f);
    float *mine = rows + MMA_PX * warp + lane;  // the lane's pixels, 32 apart
    auto models = [&](auto tag) {
        constexpr int SH = decltype(tag)::value;
        for (int c0 = 0; c0 < n_live; c0 += MMA_STAGE) {
            const int n = min(MMA_STAGE, n_live - c0);
            if (c0 > 0) __syncthreads();
            stage_records<NT, GSTAGE>(recs, A.gtab + (size_t)g0 * GREC, kept, c0, n, 0, &mbar,
                                      phase, A.err);
#pragma unroll 1
            for (int i = 0; i < n; ++i) {
                const float *r = recs + (size_t)i * GSTAGE;
                int flag = kept[c0 + i];
                // two Gaussians of the same source at once: their exponentials
                // interleave (an odd last one with a record of zeros)
                const bool two = !(flag & FLAG_LAST_SRC) && i + 1 < n;
                design_pairs2<KP, SH>(Xp, Yp, M, r, two ? r + GSTAGE : s_zero, CM24, KEXP2,
                                      KEXPLO2);
                if (two) flag = kept[c0 + ++i];
                const bool last = flag & FLAG_LAST_SRC;
                if (!last && i != n - 1) continue;
                // the source ends, or the stage does (flushed twice and added then)
#pragma unroll
                for (int j = 0; j < KP; ++j) {
                    X[j] = fma2(M[j], MINUS1, X[j]);  // M accumulates -model
                    M[j] = 0ull;
                }
                if (!last) continue;
                float *row = mine + (size_t)(kept[c0 + i] >> 1) / npsf * MMA_ROW;
#pragma unroll
                for (int j = 0; j < KP; ++j) {
                    row[64 * j] = lo(X[j]);
                    row[64 * j + 32] = hi(X[j]);
                    X[j] = 0ull;
                }
            }
        }
    };
    if (share == SHARE_Y) {
        share_coordinate<KP>(Yp, counts);
        models(ShareTag<SHARE_Y>());
    } else if (share == SHARE_X) {
        share_coordinate<KP>(Xp, counts);
        models(ShareTag<SHARE_X>());
    } else {
        models(ShareTag<SHARE_NONE>());
    }
#pragma unroll
    for (int k = 0; k < MMA_K; ++k) {
        mine[(size_t)ns * MMA_ROW + 32 * k] = y[k];
        ws[MMA_PX * warp + 32 * k + lane] = w[k];
    }
    __syncwarp();
    // products of the warp's pixels, four by four blocks of eight rows at a
    // time; the warps' sums are added in warp order through the record stage,
    // eight blocks at a time
    const int nb = nr / 8;
    const int n_pairs = ns * (ns + 1) / 2;
    const float *frag = rows + (size_t)(lane >> 2) * MMA_ROW + MMA_PX * warp + (lane & 3);
    const float *wfrag = ws + MMA_PX * warp + (lane & 3);
    double *sums = reinterpret_cast<double *>(recs);  // [warp][8 blocks][64]
    static_assert(MMA_WARPS * 8 * 64 * 8 <= MMA_STAGE * GSTAGE * 4, "the stage holds the sums");
    for (int I = 0; I < nb; I += 4)
        for (int J = I; J < nb; J += 4) {
            double c[4][4][2] = {};
#pragma unroll 2
            for (int k = 0; k < MMA_PX; k += 4) {
                double a[4], b[4];
                const double wk = (double)wfrag[k];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    a[i] = I + i < nb ? wk * (double)frag[8 * (I + i) * MMA_ROW + k] : 0.0;
                    b[i] = J == I       ? a[i]
                           : J + i < nb ? wk * (double)frag[8 * (J + i) * MMA_ROW + k]
                                        : 0.0;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (I + i < nb && J + j < nb && (J > I || j >= i))
                            mma_f64(c[i][j][0], c[i][j][1], a[i], b[j]);
            }
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                __syncthreads();  // the stage (or the sums before) is read
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    double *d = sums + (warp * 8 + q) * 64 + 2 * lane;
                    d[0] = c[2 * half + q / 4][q % 4][0];
                    d[1] = c[2 * half + q / 4][q % 4][1];
                }
                __syncthreads();
                for (int e = tid; e < 512; e += NT) {
                    const int i = 2 * half + (e >> 8), j = (e >> 6) & 3, l = (e >> 1) & 31;
                    const int s = 8 * (I + i) + (l >> 2), t = 8 * (J + j) + 2 * (l & 3) + (e & 1);
                    if (s >= ns || t > ns || s > t) continue;
                    double v = 0.0;
#pragma unroll
                    for (int w2 = 0; w2 < MMA_WARPS; ++w2) v += sums[w2 * 512 + e];
                    pnorm[(size_t)tile * n_terms +
                          (t < ns ? upper_index(s, t, ns) : n_pairs + s)] = v;
                }
            }
        }
}

// grid (n_bands, ceil(n_terms / 32)): ATA[b] (both triangles) and ATb[b] from
// the tiles' partial sums.  A warp reads 32 terms of a partial together and
// takes every eighth partial; fixed order.  (One thread
// per term over all of a band's tiles: 47 us on the 20-source patch.)
__global__ void __launch_bounds__(256) normal_reduce(const int *tile_band_start,
                                                     const double *pnorm, int n_terms, int ns,
                                                     double *ata, double *atb) {
    __shared__ double part[8][32];
    const int b = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int p = blockIdx.y * 32 + lane;
    let_next_kernel_start();
    wait_for_earlier_kernel();
    const int t0 = tile_band_start[b], t1 = tile_band_start[b + 1];
    double acc = 0.0;
    if (p < n_terms) {
#pragma unroll 8
        for (int t = t0 + w; t < t1; t += 8) acc += pnorm[(size_t)t * n_terms + p];
    }
    part[w][lane] = acc;
    __syncthreads();
    if (w > 0 || p >= n_terms) return;
    acc = 0.0;
#pragma unroll
    for (int v = 0; v < 8; ++v) acc += part[v][lane];
    const int n_pairs = ns * (ns + 1) / 2;
    if (p < n_pairs) {
        int s, t;
        upper_pair(p, ns, s, t);
        ata[((size_t)b * ns + s) * ns + t] = acc;
        ata[((size_t)b * ns + t) * ns + s] = acc;
    } else if (atb) {
        atb[(size_t)b * ns + (p - n_pairs)] = acc;
    }
}

// Cholesky ATA = L L^T (FP64) and the two triangular solves of one band by one
// warp, for ns <= 32: lane i holds row i in registers, a column's elements go
// round by shuffles.  A chain of latencies throughout (the diagonal's
// reciprocal root, then products); in shared memory, whose loads wait for the
// stores before them, it took 20 us for 20 sources, this form 11 us.
__global__ void __launch_bounds__(32) normal_solve_warp(const double *ata, const double *atb,
                                                        int ns, double *flux, int *status) {
    const int b = blockIdx.x, lane = threadIdx.x;
    wait_for_earlier_kernel();
    const double *row = ata + (size_t)b * ns * ns + (size_t)min(lane, ns - 1) * ns;
    double a[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) a[j] = j < ns ? row[j] : 0.0;
    double z = lane < ns ? atb[(size_t)b * ns + lane] : 0.0;
    double inv = 0.0;  // 1 / L[lane][lane]
    int bad = 0;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
        if (k >= ns) break;
        const double d = __shfl_sync(0xffffffffu, a[k], k);
        bad |= !(d > 0.0);
        const double r = d > 0.0 ? rsqrt(d) : 1.0;
        a[k] *= r;  // column k (rows below k use it)
        if (lane == k) inv = r;
        // L z = ATb alongside
        const double zk = __shfl_sync(0xffffffffu, z, k) * r;
        z = lane == k ? zk : z - (lane > k ? a[k] * zk : 0.0);
#pragma unroll
        for (int j = k + 1; j < 32; ++j) {
            if (j >= ns) break;
            a[j] -= a[k] * __shfl_sync(0xffffffffu, a[k], j);
        }
    }
#pragma unroll
    for (int i = 31; i >= 0; --i) {  // L^T x = z
        if (i >= ns) continue;
        double s = lane > i && lane < ns ? a[i] * z : 0.0;  // z of lanes above i is x
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == i) z = (z - s) * inv;
    }
    if (status && lane == 0) status[b] = bad;
    if (lane < ns)
        flux[(size_t)b * ns + lane] = bad ? __longlong_as_double(0x7ff8000000000000ll) : z;
}

// The same for up to 64 sources in shared memory, 256 threads: the trailing
// update spread over all of them, the triangular solves column by column in
// one warp.
constexpr int SOLVE_THREADS = 256;
__global__ void __launch_bounds__(SOLVE_THREADS) normal_solve(const double *ata,
                                                              const double *atb, int ns,
                                                              double *flux, int *status) {
    __shared__ double L[64 * 65];
    __shared__ double z[64], inv[64];
    __shared__ int bad;
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const int ld = ns | 1;  // odd: a column's elements lie in different banks
    wait_for_earlier_kernel();
    const double *Ab = ata + (size_t)b * ns * ns;
    for (int i = tid; i < ns * ns; i += SOLVE_THREADS) L[i / ns * ld + i % ns] = Ab[i];
    if (tid < ns) z[tid] = atb[(size_t)b * ns + tid];
    if (tid == 0) bad = 0;
    __syncthreads();
    for (int k = 0; k < ns; ++k) {
        const double d = L[k * ld + k];
        const double r = d > 0.0 ? rsqrt(d) : 1.0;
        if (tid == 0) {
            if (!(d > 0.0)) bad = 1;
            inv[k] = r;
        }
        for (int i = k + 1 + tid; i < ns; i += SOLVE_THREADS) L[i * ld + k] *= r;
        __syncthreads();
        // trailing rows, four threads each
        for (int i = k + 1 + (tid & 63); i < ns; i += 64) {
            const double lik = L[i * ld + k];
            for (int j = k + 1 + (tid >> 6); j <= i; j += 4) L[i * ld + j] -= lik * L[j * ld + k];
        }
        __syncthreads();
    }
    if (tid < 32) {
        for (int j = 0; j < ns; ++j) {  // L z = ATb
            const double zj = z[j] * inv[j];
            __syncwarp();
            if (lane == 0) z[j] = zj;
            for (int i = j + 1 + lane; i < ns; i += 32) z[i] -= L[i * ld + j] * zj;
            __syncwarp();
        }
        for (int j = ns - 1; j >= 0; --j) {  // L^T x = z
            const double xj = z[j] * inv[j];
            __syncwarp();
            if (lane == 0) z[j] = xj;
            for (int i = lane; i < j; i += 32) z[i] -= L[j * ld + i] * xj;
            __syncwarp();
        }
        if (status && lane == 0) status[b] = bad;
    }
    __syncthreads();
    for (int i = tid; i < ns; i += SOLVE_THREADS)
        flux[(size_t)b * ns + i] = bad ? __longlong_as_double(0x7ff8000000000000ll) : z[i];
}

// the normal-equation kernel for a plan's tile size: four pixels per thread
// (two pixel pairs, two Gaussians interleaved: four independent exponential
// chains); whole warps, so the 192-pixel tile takes six pixels per thread.
// (A form with 4 warps of 8 pixels per thread sharing each 256-pixel tile's
// Gaussians, as the split tile kernels do, measured no faster: 0.430 against
// 0.427 ms for the 20-source patch.)
struct NormalShape {
    int tile, nt;
    const void *fn;
};
const NormalShape kNormalShapes[] = {
    {128, 32, (const void *)normal_tiles<32, 4>},
    {192, 32, (const void *)normal_tiles<32, 6>},
    {256, 64, (const void *)normal_tiles<64, 4>},
    {512, 128, (const void *)normal_tiles<128, 4>},
    {1024, 256, (const void *)normal_tiles<256, 4>},
};


std::mutex g_norm_mu;
size_t g_norm_attr[64][8];  // the last entry: normal_tiles_mma

}  // namespace
}  // namespace fpho

using namespace fpho;

#define CUDA_TRY(call)                                                                  \
    do {                                                                                \
        cudaError_t e_ = (call);                                                        \
        if (e_ != cudaSuccess)                                                          \
            return set_error(FPHO_ERR_CUDA, "%s failed: %s (%s:%d)", #call,             \
                             cudaGetErrorString(e_), __FILE__, __LINE__);               \
    } while (0)

// Enqueue normal_tiles + normal_reduce; ATA into d_ata, ATb into d_atb.
static int enqueue_normal(fpho_patch *p, const fpho_source *d_prop, double *d_ata, double *d_atb,
                          cudaStream_t s) {
    const int ns = p->n_sources;
    const int n_terms = ns * (ns + 1) / 2 + ns;
    const int tile = variant_tile_pixels(p->variant);
    constexpr int n_shapes = sizeof(kNormalShapes) / sizeof(kNormalShapes[0]);
    int shape = -1;
    for (int i = 0; i < n_shapes; ++i)
        if (kNormalShapes[i].tile == tile) shape = i;
    if (shape < 0)
        return set_error(FPHO_ERR_STATE, "no normal-equation kernel for %d-pixel tiles", tile);
    const NormalShape &S = kNormalShapes[shape];
    const int idx_cap = std::max(p->max_g, 1);
    const int live_cap = std::min(p->live_cap, DESIGN_LIVE_CAP);
    // on the tensor cores where the rows fit in shared memory (with what that
    // kernel has there statically)
    constexpr size_t MMA_STATIC = 256;
    const size_t mma_smem = mma_smem_bytes(idx_cap, ns);
    const bool mma = tile == MMA_TILE && live_cap == DESIGN_LIVE_CAP &&
                     ns <= NORMAL_MMA_SOURCES && mma_smem + MMA_STATIC <= 227 * 1024;
    const void *fn = mma ? (const void *)normal_tiles_mma : S.fn;
    const size_t smem = mma ? mma_smem : normal_smem_bytes(tile, live_cap, idx_cap, ns);
    if (smem > 227 * 1024)
        return set_error(FPHO_ERR_LIMIT, "the normal equations of %d sources over %d-pixel tiles "
                         "need %zu bytes of shared memory (max 227 KB)", ns, tile, smem);
    const size_t need = (size_t)std::max(p->n_tiles, 1) * n_terms;
    if (p->d_pnorm_cap < need) {
        pool_free(p->d_pnorm);
        p->d_pnorm = nullptr;
        p->d_pnorm_cap = 0;
        CUDA_TRY(pool_malloc((void **)&p->d_pnorm, need * sizeof(double)));
        p->d_pnorm_cap = need;
    }
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 64) return set_error(FPHO_ERR_LIMIT, "device ordinal %d >= 64", dev);
    {
        std::lock_guard<std::mutex> lk(g_norm_mu);
        size_t &allowed = g_norm_attr[dev][mma ? 7 : shape];
        if (allowed < smem) {
            CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
            allowed = smem;
        }
    }
    const PatchView pv = make_view(p);
    if (p->max_g > 0) {
        dim3 grid((p->max_g + 127) / 128, p->n_exp);
        build_image_gaussians<<<grid, 128, 0, s>>>(pv, d_prop, p->d_gtab, p->d_gbox,
                                                p->d_err);
        CUDA_TRY(cudaGetLastError());
    } else {
        CUDA_TRY(cudaMemsetAsync(p->d_err, 0, sizeof(int), s));
    }
    TileArgs A;
    A.pv = pv;
    A.tiles = p->d_tiles;
    A.tbox_all = p->d_tbox_all;
    A.tbox_w = p->d_tbox_w;
    A.gtab = p->d_gtab;
    A.gbox = p->d_gbox;
    A.pchi2 = p->d_pchi2;
    A.pgrad = p->d_pgrad;
    A.pgrad_stride = 7 * ns;
    A.want_residual = 1;
    A.live_cap = live_cap;
    A.idx_cap = idx_cap;
    A.err = p->d_err;
    A.pairs = nullptr;
    A.tile_misfit = p->d_tile_misfit;
    if (p->n_tiles > 0) {
        double *pn = p->d_pnorm;
        int nt = n_terms;
        void *args[] = {(void *)&A, (void *)&pn, (void *)&nt};
        CUDA_TRY(launch_dependent(fn, dim3(p->n_tiles), dim3(mma ? 32 * MMA_WARPS : S.nt), args,
                                  smem, s));
    }
    void *rargs[] = {&p->d_tile_band_start, &p->d_pnorm, (void *)&n_terms, (void *)&ns,
                     &d_ata, &d_atb};
    CUDA_TRY(launch_dependent((const void *)normal_reduce,
                              dim3(p->n_bands, (n_terms + 31) / 32), dim3(256), rargs, 0, s));
    return FPHO_OK;
}

extern "C" int fpho_patch_flux_normal_equations(fpho_patch *p, const void *dev_proposal,
                                                int n_sources, double *dev_ata, double *dev_atb,
                                                void *stream) {
    clear_error();
    if (!p || !dev_proposal || !dev_ata || !dev_atb)
        return set_error(FPHO_ERR_INVALID, "NULL argument");
    if (n_sources != p->n_sources)
        return set_error(FPHO_ERR_INVALID, "n_sources=%d but the patch has %d", n_sources,
                         p->n_sources);
    return enqueue_normal(p, (const fpho_source *)dev_proposal, dev_ata, dev_atb,
                          (cudaStream_t)stream);
}

extern "C" int fpho_patch_optimize_fluxes(fpho_patch *p, const void *dev_proposal, int n_sources,
                                          double *dev_flux, double *dev_precision,
                                          int *dev_status, void *stream) {
    clear_error();
    if (!p || !dev_proposal || !dev_flux || !dev_precision)
        return set_error(FPHO_ERR_INVALID, "NULL argument");
    if (n_sources != p->n_sources)
        return set_error(FPHO_ERR_INVALID, "n_sources=%d but the patch has %d", n_sources,
                         p->n_sources);
    if (n_sources > 64)
        return set_error(FPHO_ERR_LIMIT, "the device flux solve takes at most 64 sources (%d)",
                         n_sources);
    cudaStream_t s = (cudaStream_t)stream;
    const size_t nb = (size_t)p->n_bands * n_sources;
    if (p->d_atb_cap < nb) {
        pool_free(p->d_atb);
        p->d_atb = nullptr;
        p->d_atb_cap = 0;
        CUDA_TRY(pool_malloc((void **)&p->d_atb, nb * sizeof(double)));
        p->d_atb_cap = nb;
    }
    int rc = enqueue_normal(p, (const fpho_source *)dev_proposal, dev_precision, p->d_atb, s);
    if (rc) return rc;
    void *args[] = {&dev_precision, &p->d_atb, &n_sources, &dev_flux, &dev_status};
    const bool small = n_sources <= 32;
    const void *fn = small ? (const void *)normal_solve_warp : (const void *)normal_solve;
    CUDA_TRY(launch_dependent(fn, dim3(p->n_bands), dim3(small ? 32 : SOLVE_THREADS),
                              args, 0, s));
    return FPHO_OK;
}
