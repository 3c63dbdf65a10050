// fpho_kernels.cuh -- small kernels around the tile kernel, included (with
// internal linkage) by every translation unit that launches them.
#pragma once

#include "fpho_impl.cuh"

namespace fpho {

// One thread per image Gaussian of exposure blockIdx.y: record + culling box.
// Clears the error word.
static __global__ void build_image_gaussians(PatchView pv, const fpho_source *src, float *gtab,
                                             float4 *gbox, int *err) {
    let_next_kernel_start();
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *err = 0;
    const int e = blockIdx.y;
    const int g0 = pv.gauss_start[e];
    const int n = pv.gauss_start[e + 1] - g0;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int npsf = pv.exp_npsf[e];
    const int s = i / npsf, p = i - s * npsf;
    build_one_gaussian(pv, src, e, s, p, gtab + (size_t)(g0 + i) * GREC, gbox + g0 + i);
}

// Bounding boxes of every tile: over all pixels and over pixels with
// ierr != 0.  If n_tiles_dev is given, blocks at or beyond *n_tiles_dev exit.
// With `misfit`, also the tile's misfit bits and its runs (`runs_per_tile` of
// them).
static __global__ void tile_bboxes(PatchView pv, const TileDesc *tiles, float4 *tbox_all,
                                   float4 *tbox_w, const int *n_tiles_dev,
                                   int *misfit = nullptr, float2 *runs = nullptr,
                                   int runs_per_tile = 0) {
    if (n_tiles_dev && (int)blockIdx.x >= *n_tiles_dev) return;
    const TileDesc td = tiles[blockIdx.x];
    float ax0 = INFINITY, ax1 = -INFINITY, ay0 = INFINITY, ay1 = -INFINITY;
    float wx0 = INFINITY, wx1 = -INFINITY, wy0 = INFINITY, wy1 = -INFINITY;
    for (int i = threadIdx.x; i < td.count; i += blockDim.x) {
        const int pix = td.pix_begin + i;
        const float x = pv.xpix[pix], y = pv.ypix[pix];
        ax0 = fminf(ax0, x); ax1 = fmaxf(ax1, x);
        ay0 = fminf(ay0, y); ay1 = fmaxf(ay1, y);
        if (pv.ierr[pix] != 0.0f) {
            wx0 = fminf(wx0, x); wx1 = fmaxf(wx1, x);
            wy0 = fminf(wy0, y); wy1 = fmaxf(wy1, y);
        }
    }
    __shared__ float red[8][32];
    float v[8] = {ax0, -ax1, ay0, -ay1, wx0, -wx1, wy0, -wy1};
#pragma unroll
    for (int k = 0; k < 8; ++k)
        for (int o = 16; o > 0; o >>= 1) v[k] = fminf(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
        for (int k = 0; k < 8; ++k) red[k][warp] = v[k];
    __syncthreads();
    if (threadIdx.x == 0) {
        const int nw = blockDim.x / 32;
        for (int k = 0; k < 8; ++k)
            for (int w = 1; w < nw; ++w) red[k][0] = fminf(red[k][0], red[k][w]);
        tbox_all[blockIdx.x] = make_float4(red[0][0], -red[1][0], red[2][0], -red[3][0]);
        tbox_w[blockIdx.x] = make_float4(red[4][0], -red[5][0], red[6][0], -red[7][0]);
    }
    if (!misfit) return;
    __shared__ int s_misfit;
    if (threadIdx.x == 0) s_misfit = 0;
    __syncthreads();
    int bits = 0, first;
    for (int i = threadIdx.x; i < 8 * runs_per_tile; i += blockDim.x) {  // whole warps
        const bool ok = i < td.count;
        const int pix = td.pix_begin + (ok ? i : 0);
        const float x = pv.xpix[pix], y = pv.ypix[pix];
        bits |= run_misfit(x, y, ok && pv.ierr[pix] != 0.0f, first);
        bits |= run_misfit(x, y, ok, first) << MISFIT_ALL;
    }
    if (bits) atomicOr(&s_misfit, bits);
    __syncthreads();
    const bool shared_x = runs_share_x(s_misfit);
    for (int i = threadIdx.x; i < 8 * runs_per_tile; i += blockDim.x) {
        const bool ok = i < td.count;
        const int pix = td.pix_begin + (ok ? i : 0);
        const float2 uv = run_start(pv.xpix[pix], pv.ypix[pix], ok && pv.ierr[pix] != 0.0f,
                                    shared_x);
        if ((i & 7) == 0) runs[(size_t)blockIdx.x * runs_per_tile + (i >> 3)] = uv;
    }
    if (threadIdx.x == 0) misfit[blockIdx.x] = s_misfit;
}

// Work order for the persistent tile kernel: tiles by decreasing cost in the
// previous evaluation (kept image Gaussians x pixels, written by the tile
// body), approximately -- a counting sort into 64 equal-width buckets of
// [0, max cost]; within a bucket the order is whatever the shared-memory
// atomics give.  The result does not depend on the order, since every tile
// writes its own partials and reduce_bands sums them in tile-index order.
// One CTA (at least 64 threads).  Also resets the work counter.
__device__ __forceinline__ void order_tiles_body(const int *cost, int n_tiles, int *order,
                                                 int *counter) {
    constexpr int NB = 64;
    __shared__ int hist[NB];
    __shared__ int smax;
    const int tid = threadIdx.x;
    if (tid < NB) hist[tid] = 0;
    if (tid == 0) {
        smax = 0;
        *counter = 0;
    }
    __syncthreads();
    int m = 0;
    for (int i = tid; i < n_tiles; i += blockDim.x) m = max(m, cost[i]);
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((tid & 31) == 0) atomicMax(&smax, m);
    __syncthreads();
    const long long span = (long long)smax + 1;
    for (int i = tid; i < n_tiles; i += blockDim.x)
        atomicAdd(&hist[NB - 1 - (int)((long long)cost[i] * NB / span)], 1);
    __syncthreads();
    if (tid == 0) {
        int acc = 0;
        for (int b = 0; b < NB; ++b) {
            const int h = hist[b];
            hist[b] = acc;
            acc += h;
        }
    }
    __syncthreads();
    for (int i = tid; i < n_tiles; i += blockDim.x)
        order[atomicAdd(&hist[NB - 1 - (int)((long long)cost[i] * NB / span)], 1)] = i;
}

// The launch before the tile kernel of an evaluation: blocks (x, e < n_exp)
// build exposure e's image Gaussians (as build_image_gaussians); with
// `order`, the block (0, n_exp) orders the tiles by the previous
// evaluation's costs (as order_tiles) at the same time; and block (0, 0)
// clears the error word.  One launch instead of a memset and two kernels.
// Launched with PREP_THREADS threads per block: the ordering block is then
// as wide as a standalone sort would be (its passes over the costs are
// latency-bound), and one block covers an exposure's image Gaussians.
constexpr int PREP_THREADS = 1024;
__device__ __forceinline__ void prepare_body(const PatchView &pv, const fpho_source *src,
                                             float *gtab, float4 *gbox, const int *cost,
                                             int n_tiles, int *order, int *counter, int *err,
                                             bool early) {
    if (early) let_next_kernel_start();
    wait_for_earlier_kernel();  // the proposal, and the last evaluation's readers
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *err = 0;
    const int e = blockIdx.y;
    if (e == pv.n_exp) {
        if (blockIdx.x == 0 && order) order_tiles_body(cost, n_tiles, order, counter);
        return;
    }
    const int g0 = pv.gauss_start[e];
    const int n = pv.gauss_start[e + 1] - g0;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int npsf = pv.exp_npsf[e];
    const int s = i / npsf, p = i - s * npsf;
    build_one_gaussian(pv, src, e, s, p, gtab + (size_t)(g0 + i) * GREC, gbox + g0 + i);
}
static __global__ void __launch_bounds__(PREP_THREADS) prepare_evaluation(
    PatchView pv, const fpho_source *src, float *gtab, float4 *gbox, const int *cost, int n_tiles,
    int *order, int *counter, int *err, bool early) {
    prepare_body(pv, src, gtab, gbox, cost, n_tiles, order, counter, err, early);
}
// The same with the proposal in the launch itself, for one that comes from
// host memory: no transfer, and the caller's array is read when the call
// returns.  N sources at most.
template <int N>
struct ProposalArg {
    fpho_source s[N];
};
template <int N>
static __global__ void __launch_bounds__(PREP_THREADS) prepare_evaluation_arg(
    const __grid_constant__ ProposalArg<N> prop, PatchView pv, float *gtab, float4 *gbox,
    const int *cost, int n_tiles, int *order, int *counter, int *err, bool early) {
    prepare_body(pv, prop.s, gtab, gbox, cost, n_tiles, order, counter, err, early);
}

// Sums of tile partials in double, for reduce_bands and batch_reduce alike (a
// patch's batched result equals its single one with the same tile shape bit for
// bit, unless that one deals its tiles to several CTAs, which adds their
// partials in another order): one block of
// REDUCE_THREADS per 32 gradient components of a band and one for its chi2.
// Component blocks: a warp reads a tile's 32 adjacent partials together and
// takes every REDUCE_WARPS-th tile of [t0, t1); the warps' sums are added in
// warp order, and the 32 results written together (to host memory when the
// caller's arrays are there, where single words would each be a transfer of
// their own).  Deterministic.
constexpr int REDUCE_THREADS = 256, REDUCE_WARPS = REDUCE_THREADS / 32;
// Blocks a band needs for `n` components and its chi2.
__host__ __device__ inline int reduce_blocks(int n) { return (n + 31) / 32 + 1; }
// Component block: sum of column c0 + lane (0 where it is >= n_cols), in warp 0.
__device__ __forceinline__ double column_sums(const float *pgrad, int stride, int n_cols, int c0,
                                              int t0, int t1) {
    __shared__ double part[REDUCE_WARPS][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int j = c0 + lane;
    double acc = 0.0;
    if (j < n_cols) {
        const float *col = pgrad + j;
#pragma unroll 8
        for (int t = t0 + w; t < t1; t += REDUCE_WARPS) acc += (double)col[(size_t)t * stride];
    }
    part[w][lane] = acc;
    __syncthreads();
    acc = 0.0;
#pragma unroll
    for (int v = 0; v < REDUCE_WARPS; ++v) acc += part[v][lane];
    return acc;
}
// chi2 block: the sum over the tiles, in every thread.
__device__ __forceinline__ double chi2_sum(const double *pchi2, int t0, int t1) {
    __shared__ double part[REDUCE_WARPS];
    double acc = 0.0;
#pragma unroll 4
    for (int t = t0 + (int)threadIdx.x; t < t1; t += REDUCE_THREADS) acc += pchi2[t];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    acc = 0.0;
#pragma unroll
    for (int v = 0; v < REDUCE_WARPS; ++v) acc += part[v];
    return acc;
}

// grid (n_bands, reduce_blocks(out_stride) or, without dchi2_out, 1).  A tile
// has `parts` partials.  With err_out, block (0, 0) also copies the
// evaluation's error word there.
static __global__ void __launch_bounds__(REDUCE_THREADS) reduce_bands(
    const int *tile_band_start, const double *pchi2, const float *pgrad, int stride,
    double *chi2_out, float *dchi2_out, int out_stride, int parts = 1, const int *err = nullptr,
    int *err_out = nullptr) {
    wait_for_earlier_kernel();
    const int b = blockIdx.x;
    const int t0 = parts * tile_band_start[b], t1 = parts * tile_band_start[b + 1];
    if (blockIdx.y == 0) {
        if (err_out && b == 0 && threadIdx.x == 0) *err_out = *err;
        const double c = chi2_sum(pchi2, t0, t1);
        if (threadIdx.x == 0) chi2_out[b] = c;
        return;
    }
    const int c0 = 32 * (blockIdx.y - 1);
    const double g = column_sums(pgrad, stride, stride, c0, t0, t1);
    const int j = c0 + (int)threadIdx.x;
    if (threadIdx.x < 32 && j < out_stride) dchi2_out[(size_t)b * out_stride + j] = (float)g;
}

}  // namespace fpho
