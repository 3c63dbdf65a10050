// fpho_tile.cuh -- the pixel-tile kernel body shared by the single-patch and
// the batched evaluation.
//
// One CTA evaluates one tile of up to NT*K pixels of one exposure:
//   1. cull: keep the exposure's image Gaussians whose exp-argument <= 36 box
//      overlaps the tile's pixel bounding box (provably equivalent to the
//      reference's per-pixel `exparg > 36` skip, which is still applied to
//      every Gaussian that can cross the threshold inside the tile);
//   2. stage the kept records into shared memory with asynchronous copies
//      issued by every thread of the CTA (completion on an mbarrier);
//   3. residual pass: r = data - sum_g amp G H over kept Gaussians, in the
//      reference's Gaussian order (ComputeResidualImage, common_kernel.cc:57-83);
//   4. chi2 per pixel in double, exactly as compute_gaussians_kernel.cc:286-293;
//   5. gradient pass, one kept Gaussian per lane (gradient_lanes): each lane
//      walks the tile's pixels, broadcast from shared memory, and forms the
//      twelve sums of its Gaussian's weight from which the derivatives of the
//      model w.r.t. the Gaussian's image-space parameters (A, x, y, fxx, fyy,
//      fxy) and, through its Jacobian, w.r.t. the source's follow
//      (ComputeGaussianDerivative, common_kernel.cc:95-143, with the per-pixel
//      Jacobian product moved out of the pixel loop);
//   6. per-source sums are reduced across the warp and the CTA in a fixed
//      order and written as this tile's partial; chi2 partials stay double.
// Pixel pairs are processed as packed .f32x2 operands (two pixels per
// instruction).
#pragma once

#include "fpho_impl.cuh"

namespace fpho {

struct TileArgs {
    PatchView pv;
    const TileDesc *tiles;
    const float4 *tbox_all;   // per tile bounding box of all pixels (x0, x1, y0, y1)
    const float4 *tbox_w;     // per tile bounding box of pixels with ierr != 0
    const float *gtab;        // image-Gaussian records
    const float4 *gbox;       // culling boxes
    double *pchi2;            // [n_tiles] chi2 partial per tile
    float *pgrad;             // [n_tiles][pgrad_stride] gradient partial per tile
    int pgrad_stride;         // 7 * n_sources
    int want_residual;
    int live_cap;             // records that fit in the shared-memory stage (>= 1)
    int idx_cap;              // most image Gaussians of any exposure (kept-list capacity)
    int *err;                 // error word (bit 0: a staging wait gave up)
    long long *pairs;         // optional: evaluated (pixel, Gaussian) pairs, or nullptr
    const int *tile_misfit = nullptr; // the plan's misfit bits and runs of every tile, or nullptr
    const float2 *runs = nullptr;     // (formed per tile then)
    int *tile_cost = nullptr; // optional: [n_tiles] kept Gaussians x pixels, written per tile
    int test_extra_tx = 0;    // test of the error path only: bytes the staging wait
                              // expects beyond those copied, so that it runs out
};

// ------------------------------------------------------------ mbarrier + asynchronous copies
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void copy16_async(void *dst_smem, const void *src_gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst_smem)),
                 "l"(src_gmem)
                 : "memory");
}
// The thread's copies so far, when they complete, arrive on the barrier; the
// arrival is added to the phase's pending count here.
__device__ __forceinline__ void mbar_arrive_on_copies(uint64_t *bar) {
    asm volatile("cp.async.mbarrier.arrive.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Bounded wait on an mbarrier phase.  Gives up after `limit` polls, records
// bit 0 in the error word and returns false; never spins forever.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, int *err) {
    const int limit = 1 << 22;
    for (int i = 0; i < limit; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    atomicOr(err, 1);
    return false;
}

// ------------------------------------------------------------ warp helpers
__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ------------------------------------------------------------ shared layout
// Dynamic shared memory of a tile CTA, in order:
//   stage   first the masks and queues of the scan; then `live_cap` staged records
//           of the residual pass (the first MODEL_STAGE floats of each: all it
//           reads); then the pixels of the gradient pass, PX_BYTES each
//           (px_block pixels at a time);
//   kept    the kept list, one int per Gaussian of the exposure (local index
//           << 1 | flags);
//   wacc    per-warp gradient sums, `stride` floats each;
//   part    split tiles only: the warps' partial models, one float per pixel.
// The design passes stage whole records (they need the unit-flux amplitude
// and the source index) and have neither gradient pixels nor partial models.
constexpr int MODEL_STAGE = 16;  // floats of a record staged for the residual pass
constexpr int GSTAGE = GREC;     // floats of a record staged for the design passes
constexpr int PX_BYTES = 5;      // -2 r ie^2 of a pixel, the coordinates of its run of 8

// Pixels of the tile that the gradient pass holds at a time: all of them,
// unless `live_cap` is so small that they would need more than the 128 bytes
// per staged record that a patch's limits are counted with.
__host__ __device__ inline int px_block(int tile_pixels, int live_cap) {
    int n = tile_pixels;
    while (n * PX_BYTES > live_cap * 128) n >>= 1;
    return n;
}
// The scan's queues (scan_tile), and the least it has with its masks.  128 bytes
// per record, less the 128 of static shared memory that a tile kernel has had
// since, is what a patch's limits are counted with; no stage takes more.
constexpr int QUEUE = 64;  // Gaussians a warp queues
constexpr size_t MIN_STAGE = 32 * 128 - 128;
__host__ __device__ inline size_t stage_bytes(int tile_pixels, int live_cap) {
    const size_t rec = (size_t)live_cap * MODEL_STAGE * 4;
    const size_t px = ((size_t)px_block(tile_pixels, live_cap) * PX_BYTES + 127) / 128 * 128;
    const size_t n = rec > px ? rec : px;
    return n > MIN_STAGE ? n : MIN_STAGE;
}
__host__ __device__ inline size_t tile_smem_layout_bytes(int nw, int tile_pixels, int live_cap,
                                                         int idx_cap, int stride) {
    return stage_bytes(tile_pixels, live_cap) + (size_t)idx_cap * 4 + (size_t)nw * stride * 4;
}
__host__ __device__ inline size_t design_smem_layout_bytes(int live_cap, int idx_cap) {
    return (size_t)live_cap * GSTAGE * 4 + (size_t)idx_cap * 4;
}

// Stage the first FLOATS floats of the records of kept entries [c0, c0 + n) of
// an exposure (first record `gexp`) into `recs`, in list order, and wait for
// them: 16-byte asynchronous copies, consecutive threads on consecutive
// sixteen bytes, whose completion arrives on the CTA's mbarrier (initialised
// with a count of one, which thread 0 takes once every thread's copies are
// issued).  One bulk copy per record, 64 bytes each, took longer: a stage of
// 27 records 2,300 cycles.  Callers have finished reading `recs`, and the kept
// list is complete, at a barrier before the call.
template <int NT, int FLOATS>
__device__ __forceinline__ void stage_records(float *recs, const float *gexp, const int *kept,
                                              int c0, int n, int extra_tx, uint64_t *mbar,
                                              uint32_t &phase, int *err) {
    constexpr int PER = FLOATS / 4;  // copies per record
    for (int i = threadIdx.x; i < n * PER; i += NT) {
        const int k = i / PER, part = i - k * PER;
        copy16_async(recs + (size_t)i * 4,
                     gexp + (size_t)(kept[c0 + k] >> 1) * GREC + 4 * part);
    }
    mbar_arrive_on_copies(mbar);
    __syncthreads();  // every thread's arrival is pending before thread 0's
    if (threadIdx.x == 0) mbar_arrive_expect_tx(mbar, (uint32_t)extra_tx);
    mbar_wait_bounded(mbar, phase, err);
    phase ^= 1u;
}

// ------------------------------------------------------------ culling
// Minimum over the rectangle [x0,x1] x [y0,y1] of the exp-argument
// q(p) = (p-c)^T F (p-c): 0 if the centre is inside, else the smallest of the
// four edge minima (q is convex, so its minimum over the rectangle lies on the
// boundary; on an edge it is a clamped 1-D quadratic minimum).
__device__ __forceinline__ float rect_min_q(float4 bb, float xc, float yc, float fxx, float fxy,
                                            float fyy) {
    if (xc >= bb.x && xc <= bb.y && yc >= bb.z && yc <= bb.w) return 0.0f;
    float best = INFINITY;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const float dx = (e ? bb.y : bb.x) - xc;
        const float dy = fminf(fmaxf(-fxy * dx / fyy, bb.z - yc), bb.w - yc);
        best = fminf(best, dx * (fxx * dx + fxy * dy) + dy * (fyy * dy + fxy * dx));
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const float dy = (e ? bb.w : bb.z) - yc;
        const float dx = fminf(fmaxf(-fxy * dy / fxx, bb.x - xc), bb.y - xc);
        best = fminf(best, dx * (fxx * dx + fxy * dy) + dy * (fyy * dy + fxy * dx));
    }
    return best;
}

// Is an image Gaussian possibly within exp-argument 36 of some point of the
// tile box?  Conservative: cull only when the exact minimum, less a 2e-3
// relative + 2e-3 margin for float rounding, exceeds 36.  `a` and `b` are the
// record's first two float4 (-xc -xc -yc -yc, fxx fxx fxy fxy).
__device__ __forceinline__ bool keeps_tile(float4 a, float4 b, float fyy, float4 bb) {
    const float fxx = b.x, fxy = b.z;
    if (!(fxx > 0.0f && fyy > 0.0f)) return true;
    const float q = rect_min_q(bb, -a.x, -a.z, fxx, fxy, fyy);
    return !(q * (1.0f - 2.0e-3f) - 2.0e-3f > FPHO_MAX_EXP_ARG);
}

// Does the Gaussian certainly pass keeps_tile: is its exp-argument at the point
// of the tile box nearest its centre, which is no less than the minimum over the
// box, below the bound by more than rounding (1e-5)?  (Also where keeps_tile
// asks nothing: a diagonal of F that is not positive.)
__device__ __forceinline__ bool near_tile(float4 a, float4 b, float fyy, float4 bb) {
    const float fxx = b.x, fxy = b.z;
    const float dx = fminf(fmaxf(-a.x, bb.x), bb.y) + a.x;
    const float dy = fminf(fmaxf(-a.z, bb.z), bb.w) + a.z;
    const float q = dx * (fxx * dx + fxy * dy) + dy * (fyy * dy + fxy * dx);
    return !(fxx > 0.0f && fyy > 0.0f) ||
           q * (1.0f - 2.0e-3f) - 2.0e-3f < FPHO_MAX_EXP_ARG * (1.0f - 1.0e-5f);
}

// ------------------------------------------------------------ per-Gaussian helpers
// Two packed operands from one 16-byte shared-memory load.
__device__ __forceinline__ void ld2(const float *p, v2 &a, v2 &b) {
    const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(p);
    a = t.x;
    b = t.y;
}

// What a thread's pixels share in the residual pass (see run_misfit): nothing,
// y, or x.  The shared offset and its product with F are then formed once per
// Gaussian instead of once per pixel pair -- 83 packed instructions for 8
// pixels instead of 89, each result rounded exactly as without sharing.
enum Share : int { SHARE_NONE = 0, SHARE_Y = 1, SHARE_X = 2 };
template <int V>
struct ShareTag {
    static constexpr int value = V;
};

// Pass 1 for one Gaussian over the thread's KP pixel pairs: R -= amp G H.
template <int KP>
__device__ __forceinline__ void residual_pairs(const v2 (&X)[KP], const v2 (&Y)[KP], v2 (&R)[KP],
                                               v2 NXC, v2 NYC, v2 FXX, v2 FXY, v2 FYY, v2 HA,
                                               v2 HB, v2 KEXP2, v2 KEXPLO2) {
#pragma unroll
    for (int j = 0; j < KP; ++j) {
        const v2 DX = add2(X[j], NXC), DY = add2(Y[j], NYC);
        const v2 VX = fma2(FXY, DY, mul2(FXX, DX));
        const v2 VY = fma2(FXY, DX, mul2(FYY, DY));
        const v2 Q = fma2(DY, VY, mul2(DX, VX));
        // the residual needs an unbiased exponential (see exp_neg_half)
        v2 Gp = exp_neg_half(Q, KEXP2, KEXPLO2);
        float g0, g1, q0, q1;
        unpk(Gp, g0, g1);
        unpk(Q, q0, q1);
        Gp = pk(q0 > FPHO_MAX_EXP_ARG ? 0.0f : g0, q1 > FPHO_MAX_EXP_ARG ? 0.0f : g1);
        const v2 S = fma2(VY, VY, mul2(VX, VX));
        R[j] = fma2(fma2(S, HA, HB), Gp, R[j]);  // fma(S, -amp/24, -amp c0) = -amp H
    }
}

// Pass 1 for two consecutive kept Gaussians a, b at once: their exponentials
// are independent, and R is updated with a's term and then b's, exactly as two
// calls of residual_pairs in order would.
//
// Written operation by operation over all 2 KP chains: a packed FMA reads three
// register pairs and takes three cycles when all differ, two when it shares one
// with its neighbour (measured: 3.07 and 2.25), so the chains take turns with
// each constant.  The register file's reads are what bounds this loop.  With
// the chains one after the other it took 8 registers more, and a fifth CTA no
// longer fitted an SM (60-source patch 3% slower).
template <int KP, int SH = SHARE_NONE>
__device__ __forceinline__ void residual_pairs2(const v2 (&X)[KP], const v2 (&Y)[KP], v2 (&R)[KP],
                                                const float *ra, const float *rb, v2 CM24,
                                                v2 KEXP2, v2 KEXPLO2) {
    constexpr int N = 2 * KP;  // chain i: Gaussian i / KP, pixel pair i % KP
    v2 NX[2], NY[2], FXX[2], FXY[2], FYY[2], AMP[2], HA[2], HB[2], C0[2];
#pragma unroll
    for (int g = 0; g < 2; ++g) {
        const float *r = g ? rb : ra;
        ld2(r + R_NXC, NX[g], NY[g]);
        ld2(r + R_FXX, FXX[g], FXY[g]);
        ld2(r + R_FYY, FYY[g], AMP[g]);
        ld2(r + R_HB, HB[g], C0[g]);
        HA[g] = mul2(AMP[g], CM24);
    }
    v2 DX[N], DY[N], VX[N], VY[N], Q[N], S[N];
#pragma unroll
    for (int i = 0; i < N; ++i) DX[i] = add2(X[SH == SHARE_X ? 0 : i % KP], NX[i / KP]);
#pragma unroll
    for (int i = 0; i < N; ++i) DY[i] = add2(Y[SH == SHARE_Y ? 0 : i % KP], NY[i / KP]);
#pragma unroll
    for (int i = 0; i < N; ++i) VX[i] = mul2(FXX[i / KP], DX[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) VX[i] = fma2(FXY[i / KP], DY[i], VX[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) VY[i] = mul2(FYY[i / KP], DY[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) VY[i] = fma2(FXY[i / KP], DX[i], VY[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) Q[i] = mul2(DX[i], VX[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) Q[i] = fma2(DY[i], VY[i], Q[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) S[i] = mul2(VX[i], VX[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) S[i] = fma2(VY[i], VY[i], S[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) S[i] = fma2(S[i], HA[i / KP], HB[i / KP]);
    // the residual needs an unbiased exponential
    v2 G[N];
    exp_neg_half(Q, G, KEXP2, KEXPLO2);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float g0, g1, q0, q1;
        unpk(G[i], g0, g1);
        unpk(Q[i], q0, q1);
        G[i] = pk(q0 > FPHO_MAX_EXP_ARG ? 0.0f : g0, q1 > FPHO_MAX_EXP_ARG ? 0.0f : g1);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) R[i % KP] = fma2(S[i], G[i], R[i % KP]);
}

// Pass 1 for the staged records [i0, i1), two at a time; an odd last one is
// paired with a record of zeros, whose term adds nothing.
template <int KP, int SH>
__device__ __forceinline__ void residual_range(const v2 (&X)[KP], const v2 (&Y)[KP], v2 (&R)[KP],
                                               const float *recs, int i0, int i1,
                                               const float *zero, v2 KEXP2, v2 KEXPLO2) {
    const v2 CM24 = pk1(-1.0f / 24.0f);
#pragma unroll 1
    for (int i = i0; i < i1; i += 2) {
        const float *r = recs + (size_t)i * MODEL_STAGE;
        residual_pairs2<KP, SH>(X, Y, R, r, i + 1 < i1 ? r + MODEL_STAGE : zero, CM24, KEXP2,
                                KEXPLO2);
    }
}

// Pass 1 in the reference's float arithmetic, for the exact-residual mode:
// ComputeResidualImage (forcepho/src/common_kernel.cc:57-83) operation by
// operation, each rounded once (no multiply-add contraction), the
// exp-argument test before the exponential, H with its division by 24, and
// exp evaluated in double and rounded once to float -- the correctly rounded
// float exp wherever double exp's error does not straddle a float rounding
// boundary.  Pixels of the pair are taken one at a time.
template <int KP>
__device__ __forceinline__ void residual_exact(const v2 (&X)[KP], const v2 (&Y)[KP], v2 (&R)[KP],
                                               const float *rec) {
    const float nxc = rec[R_NXC], nyc = rec[R_NYC];
    const float fxx = rec[R_FXX], fxy = rec[R_FXY], fyy = rec[R_FYY], amp = rec[R_AMP];
#pragma unroll
    for (int j = 0; j < KP; ++j) {
        float xs[2], ys[2], rs[2];
        unpk(X[j], xs[0], xs[1]);
        unpk(Y[j], ys[0], ys[1]);
        unpk(R[j], rs[0], rs[1]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float dx = __fadd_rn(xs[h], nxc);  // xp - xcen (nxc = -xcen exactly)
            const float dy = __fadd_rn(ys[h], nyc);
            const float vx = __fadd_rn(__fmul_rn(fxx, dx), __fmul_rn(fxy, dy));
            const float vy = __fadd_rn(__fmul_rn(fyy, dy), __fmul_rn(fxy, dx));
            const float ea = __fadd_rn(__fmul_rn(dx, vx), __fmul_rn(dy, vy));
            if (ea > FPHO_MAX_EXP_ARG) continue;
            const float gp = (float)exp((double)__fmul_rn(-0.5f, ea));
            const float t = __fsub_rn(__fsub_rn(__fadd_rn(__fmul_rn(vx, vx), __fmul_rn(vy, vy)),
                                                fxx), fyy);
            const float H = __fadd_rn(1.0f, __fdiv_rn(t, 24.0f));
            rs[h] = __fsub_rn(rs[h], __fmul_rn(__fmul_rn(amp, gp), H));
        }
        R[j] = pk(rs[0], rs[1]);
    }
}

__device__ __forceinline__ float lanesum(v2 v) {
    float a, b;
    unpk(v, a, b);
    return a + b;
}

// ------------------------------------------------------------ gradient pass
// The pixels of the gradient pass in shared memory: the weights r2 = -2 r ie^2
// and, per run of eight pixels, where it starts: (u, v) = the coordinate along
// the run at its first pixel and the shared one.  A tile whose runs share
// nothing reads its coordinates from the patch's arrays instead.
struct PixelStage {
    float *r2;       // [pixels], in slot order (run_slot)
    float *ru, *rv;  // [pixels / 8]
};
// Misfit bits of the pixels [p0, p0 + 32 N) of a tile, in every lane of the
// calling warp: the plan's, or formed here where the caller has none.
template <int N>
__device__ __forceinline__ int tile_misfit(const TileArgs &A, const TileDesc &td, int tile,
                                           int p0) {
    if (A.tile_misfit) return A.tile_misfit[tile];
    const int lane = threadIdx.x & 31;
    int bits = 0, first;
#pragma unroll 1
    for (int i = 0; i < N; ++i) {
        const int li = p0 + 32 * i + lane;
        const bool ok = li < td.count;
        const int pix = td.pix_begin + (ok ? li : 0);
        const float x = A.pv.xpix[pix], y = A.pv.ypix[pix];
        bits |= run_misfit(x, y, ok && A.pv.ierr[pix] != 0.0f, first);
        bits |= run_misfit(x, y, ok, first) << MISFIT_ALL;
    }
    return __reduce_or_sync(0xffffffffu, bits);
}
// What the residual pass may share, for threads that hold whole runs
// (K = 8 consecutive pixels each), from a tile's misfit bits.
template <int K>
__device__ __forceinline__ int share_of(int misfit, bool all) {
    if (K != 8) return SHARE_NONE;
    if (all) misfit >>= MISFIT_ALL;
    return !(misfit & MISFIT_Y) ? SHARE_Y : !(misfit & MISFIT_X) ? SHARE_X : SHARE_NONE;
}
// The shared coordinate of a thread's counting pixels in every pair (where
// other pixels' values are neither weighted nor written).
template <int KP>
__device__ __forceinline__ void share_coordinate(v2 (&C)[KP], const bool (&counts)[2 * KP]) {
    float c = lo(C[0]);
#pragma unroll
    for (int k = 2 * KP - 1; k >= 0; --k)
        if (counts[k]) c = k & 1 ? hi(C[k / 2]) : lo(C[k / 2]);
#pragma unroll
    for (int j = 0; j < KP; ++j) C[j] = pk1(c);
}
// The runs of the pixels [b0, b0 + n) of a tile of TP (n a multiple of 32), by
// the whole CTA: the plan's, or found here.
template <int NT, int TP>
__device__ __forceinline__ void stage_runs(const TileArgs &A, const TileDesc &td, int tile, int b0,
                                           int n, bool shared_x, const PixelStage &px) {
    if (A.runs) {
        for (int r = threadIdx.x; r < n / 8; r += NT) {
            const float2 uv = A.runs[(size_t)tile * (TP / 8) + b0 / 8 + r];
            px.ru[r] = uv.x;
            px.rv[r] = uv.y;
        }
        return;
    }
    for (int p = threadIdx.x; p < n; p += NT) {  // whole warps
        const int li = b0 + p;
        const bool ok = li < td.count;
        const int pix = td.pix_begin + (ok ? li : 0);
        const float2 uv = run_start(A.pv.xpix[pix], A.pv.ypix[pix],
                                    ok && A.pv.ierr[pix] != 0.0f, shared_x);
        px.ru[p >> 3] = uv.x;
        px.rv[p >> 3] = uv.y;
    }
}

// The sums over pixels that the derivatives of one Gaussian need, with the
// weight W = r2 G, the offset (du, dv) from its centre, v = F (du, dv) and the
// pixel correction H: of W H (1, vu, vv, du^2, du dv, dv^2), and of W the same.
template <typename T>
struct GradSums {
    T h0 = 0, hu = 0, hv = 0, huu = 0, huv = 0, hvv = 0;
    T w0 = 0, wu = 0, wv = 0, wuu = 0, wuv = 0, wvv = 0;
    __device__ __forceinline__ void add(const GradSums<float> &o) {
        h0 += o.h0; hu += o.hu; hv += o.hv; huu += o.huu; huv += o.huv; hvv += o.hvv;
        w0 += o.w0; wu += o.wu; wv += o.wv; wuu += o.wuu; wuv += o.wuv; wvv += o.wvv;
    }
};

// One Gaussian in a lane.  Along a run (u) at offset dv the exp-argument is
//   fuu t^2 + 2 fx t dv + k dv^2,  t = du + rq dv,
// rq being fuv / fuu to the nearest half: fx = fuv - rq fuu is small, so that
// nothing cancels for a long thin Gaussian, and t has no more bits than the
// offsets, so that it is exact where they are.  (In du and dv the three terms
// cancel, and each coefficient's rounding is the same at every pixel: that
// error does not average out.)  vu = fuu t + fx dv and vv = fuv t + kv dv.
struct LaneForm {
    float nu, nv;            // -centre
    float fuu, rq, fx, k;
    float hA, h11, h02, c0;  // H = hA t^2 + h11 t dv + h02 dv^2 + c0
    __device__ __forceinline__ LaneForm(float nu_, float nv_, float fuu_, float fuv, float fvv,
                                        float c0_)
        : nu(nu_), nv(nv_), fuu(fuu_), c0(c0_) {
        rq = fuu > 0.0f ? 0.5f * rintf(2.0f * fuv / fuu) : 0.0f;
        const double x = (double)fuv - (double)rq * fuu, y = (double)fvv - (double)rq * fuv;
        const float kv = (float)y;
        fx = (float)x;
        k = (float)(y - rq * x);
        hA = (fuu * fuu + fuv * fuv) * (1.0f / 24.0f);
        h11 = (fuu * fx + fuv * kv) * (1.0f / 12.0f);
        h02 = (fx * fx + kv * kv) * (1.0f / 24.0f);
    }
    // the sums with vu and vv, from those with t and dv in their place
    __device__ __forceinline__ void finish(GradSums<double> &m, float fuv, float fvv) const {
        const double kv = (double)fvv - (double)rq * fuv;
        const double ht = m.hu, wt = m.wu;
        m.hu = fuu * ht + fx * m.hv;
        m.hv = fuv * ht + kv * m.hv;
        m.wu = fuu * wt + fx * m.wv;
        m.wv = fuv * wt + kv * m.wv;
    }
};
// F along the run above which the sums along a run are not taken about its
// middle (a Gaussian not much wider than a pixel).  The error of the sums of one
// Gaussian against double, in those of a kernel that forms every derivative at
// every pixel, over PSF components of 1 to 2 pixels: 0.9 with 1/4, 1.2 with 1/2,
// 1.3 with 1; the 20-source patch takes 333, 331 and 329 us.
constexpr float NARROW = 0.25f;

// A slot of the staged weights: the second half of a run is staged in reverse
// (pixels 0 1 2 3 7 6 5 4), so that the packed pairs 0 and 2, 1 and 3 of a run
// hold mirror pixels.
__device__ __forceinline__ int run_slot(int p) { return (p & 4) ? (p ^ 3) : p; }

// Sums over the runs [r0, r1).  The sums s_a = sum W t^a (a <= 4) of a run give
// all twelve of its sums, since H is a quadratic in t there.  They are added up
// eight runs at a time in float, then in double: a lane walks up to 256 pixels,
// and a float sum of that length loses what a sum over 32 lanes does not.
//
// CENTRED: s_a is taken about the run's middle, where the offsets are the
// constants -7/2 ... 7/2 and mirror pixels share their even and negate their odd
// powers, and then moved by the middle's offset.  Rounding is then relative to
// W (7/2)^a, not to W t^a, so this form is for Gaussians wide enough along the
// run that the two compare (NARROW above).
//
// Moments about the centre up to the fourth order, in du and dv and all in float,
// took 30 us less of the 20-source patch's 333 and 600 less of the 60-source
// patch's 6500, but their error against double was up to three times that of
// derivatives formed at every pixel for PSF components, ten for q = 0.2 (here:
// 0.4 to 1.1 times).
template <bool CENTRED>
__device__ __forceinline__ void run_sums(const PixelStage &px, int r0, int r1, const LaneForm &f,
                                         GradSums<double> &m) {
    const v2 FUU = pk1(f.fuu), KEXP2 = pk1(KEXP);
#pragma unroll 1
    for (int r = r0; r < r1;) {
        const int end = min(r1, (r | 7) + 1);
        GradSums<float> c;  // hu, hv, wu, wv: sums with t and dv in the place of vu and vv
#pragma unroll 1
        for (; r < end; ++r) {
            const float dv = px.rv[r] + f.nv, dv2 = dv * dv;
            const float d = (px.ru[r] + f.nu) + 3.5f;  // the run's middle: du, t
            const float t = fmaf(f.rq, dv, d);
            const v2 Q1 = pk1(2.0f * f.fx * dv), Q0 = pk1(f.k * dv2);
            v2 W[4], T[4];
            ld2(px.r2 + 8 * r, W[0], W[1]);
            ld2(px.r2 + 8 * r + 4, W[2], W[3]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float z = j < 2 ? 2.0f * j - 3.5f : 7.5f - 2.0f * j;
                T[j] = pk(t + z, t + (j < 2 ? z + 1.0f : z - 1.0f));
                const v2 Q = fma2(fma2(FUU, T[j], Q1), T[j], Q0);
                float q0, q1, e0, e1;
                unpk(Q, q0, q1);
                unpk(mul2(Q, KEXP2), e0, e1);
                W[j] = mul2(W[j], pk(q0 > FPHO_MAX_EXP_ARG ? 0.0f : ex2f(e0),
                                     q1 > FPHO_MAX_EXP_ARG ? 0.0f : ex2f(e1)));
            }
            const float hB = f.h11 * dv, hC = fmaf(f.h02, dv2, f.c0);
            float s0, st, suu, su, p0, pt, puu, pu;
            if (CENTRED) {
                // sums and differences of mirror pixels, 7/2 5/2 and 3/2 1/2 off
                // the middle; scalars, whose constants are immediates (as packed
                // operands they would take sixteen registers)
                const v2 NEG = pk1(-1.0f);
                float a0, a1, a2, a3, b0, b1, b2, b3;
                unpk(add2(W[2], W[0]), a0, a1);
                unpk(add2(W[3], W[1]), a2, a3);
                unpk(fma2(W[0], NEG, W[2]), b0, b1);
                unpk(fma2(W[1], NEG, W[3]), b2, b3);
                const float z0 = (a0 + a1) + (a2 + a3);
                const float z1 = fmaf(3.5f, b0, fmaf(2.5f, b1, fmaf(1.5f, b2, 0.5f * b3)));
                const float z2 = fmaf(12.25f, a0, fmaf(6.25f, a1, fmaf(2.25f, a2, 0.25f * a3)));
                const float z3 =
                    fmaf(42.875f, b0, fmaf(15.625f, b1, fmaf(3.375f, b2, 0.125f * b3)));
                const float z4 =
                    fmaf(150.0625f, a0, fmaf(39.0625f, a1, fmaf(5.0625f, a2, 0.0625f * a3)));
                // H about the middle: hA z^2 + h1 z + h0
                const float hm = fmaf(f.hA, t, hB);
                const float h1 = fmaf(f.hA, t, hm), h0 = fmaf(hm, t, hC);
                const float q0 = fmaf(f.hA, z2, fmaf(h1, z1, h0 * z0));
                const float q1 = fmaf(f.hA, z3, fmaf(h1, z2, h0 * z1));
                const float q2 = fmaf(f.hA, z4, fmaf(h1, z3, h0 * z2));
                s0 = z0;
                st = fmaf(t, z0, z1);
                su = fmaf(d, z0, z1);
                suu = fmaf(d, z1 + su, z2);
                p0 = q0;
                pt = fmaf(t, q0, q1);
                pu = fmaf(d, q0, q1);
                puu = fmaf(d, q1 + pu, q2);
            } else {
                v2 S0, S1, S2, S3, S4;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const v2 T1 = mul2(W[j], T[j]), T2 = mul2(T1, T[j]), T3 = mul2(T2, T[j]);
                    S0 = j ? add2(S0, W[j]) : W[j];
                    S1 = j ? add2(S1, T1) : T1;
                    S2 = j ? add2(S2, T2) : T2;
                    S3 = j ? add2(S3, T3) : T3;
                    S4 = j ? fma2(T3, T[j], S4) : mul2(T3, T[j]);
                }
                s0 = lanesum(S0);
                st = lanesum(S1);
                const float s2 = lanesum(S2), s3 = lanesum(S3), s4 = lanesum(S4);
                p0 = fmaf(f.hA, s2, fmaf(hB, st, hC * s0));
                pt = fmaf(f.hA, s3, fmaf(hB, s2, hC * st));
                const float p2 = fmaf(f.hA, s4, fmaf(hB, s3, hC * s2));
                const float x = d - t;  // du = t + x
                su = fmaf(x, s0, st);
                suu = fmaf(x, st + su, s2);
                pu = fmaf(x, p0, pt);
                puu = fmaf(x, pt + pu, p2);
            }
            c.h0 += p0;
            c.hu += pt;
            c.hv = fmaf(dv, p0, c.hv);
            c.huu += puu;
            c.huv = fmaf(dv, pu, c.huv);
            c.hvv = fmaf(dv2, p0, c.hvv);
            c.w0 += s0;
            c.wu += st;
            c.wv = fmaf(dv, s0, c.wv);
            c.wuu += suu;
            c.wuv = fmaf(dv, su, c.wuv);
            c.wvv = fmaf(dv2, s0, c.wvv);
        }
        m.add(c);
    }
}
// The same over the pixels [p0, p1) of a tile whose runs share nothing (u is x);
// `x` and `y` are the coordinates of the tile's first staged pixel.
__device__ __forceinline__ void pixel_sums(const PixelStage &px, const float *x, const float *y,
                                           int p0, int p1, const LaneForm &f, float fuv,
                                           float fvv, GradSums<double> &m) {
#pragma unroll 1
    for (int p = p0; p < p1;) {
        const int end = min(p1, (p | 15) + 1);
        GradSums<float> c;
#pragma unroll 1
        for (; p < end; ++p) {
            const float r2 = px.r2[run_slot(p)];
            if (r2 == 0.0f) continue;  // (the same in every lane)
            const float du = x[p] + f.nu, dv = y[p] + f.nv;
            const float vu = fmaf(fuv, dv, f.fuu * du), vv = fmaf(fuv, du, fvv * dv);
            const float q = fmaf(dv, vv, du * vu);
            const float w = r2 * (q > FPHO_MAX_EXP_ARG ? 0.0f : ex2f(q * KEXP));
            const float h = w * fmaf(fmaf(vv, vv, vu * vu), 1.0f / 24.0f, f.c0);
            const float duu = du * du, duv = du * dv, dvv = dv * dv;
            c.h0 += h;
            c.hu = fmaf(h, vu, c.hu);
            c.hv = fmaf(h, vv, c.hv);
            c.huu = fmaf(h, duu, c.huu);
            c.huv = fmaf(h, duv, c.huv);
            c.hvv = fmaf(h, dvv, c.hvv);
            c.w0 += w;
            c.wu = fmaf(w, vu, c.wu);
            c.wv = fmaf(w, vv, c.wv);
            c.wuu = fmaf(w, duu, c.wuu);
            c.wuv = fmaf(w, duv, c.wuv);
            c.wvv = fmaf(w, dvv, c.wvv);
        }
        m.add(c);
    }
}

// The gradient pass over `n_px` staged pixels, the first at index `pix` of the
// patch's arrays: every kept Gaussian of the tile in a lane of its own.
//
// A lane forms the twelve sums of GradSums; every derivative is a combination of
// them, taken once per Gaussian; then its Jacobian, and a sum over the lanes of
// each source.
//
// Against pixels in the lanes and Gaussians in the loop (each thread forming
// the sums of its own 8 pixels), the per-Gaussian work is done once for a
// whole tile instead of once per 8 pixels, and per-row work once per row.
// Work is dealt to the warps in units of (32 Gaussians, UNIT pixels), in order
// and evenly, so that a kept list that is no multiple of 32 NW still keeps
// every warp busy.
template <int NW, int UNIT = 64>
__device__ __forceinline__ void gradient_lanes(const TileArgs &A, const int *kept, int n_live,
                                               int g0, const PixelStage &px, int pix, int n_px,
                                               int misfit, float *wacc) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nq = (n_px + UNIT - 1) / UNIT;
    const int units = ((n_live + 31) >> 5) * nq;
    int left = units * (warp + 1) / NW - units * warp / NW;
    int g = units * warp / NW / nq, q = units * warp / NW - g * nq;
    float *row = wacc + warp * A.pgrad_stride;
    const bool shared_x = runs_share_x(misfit);
    for (; left > 0; ++g, q = 0) {
        const int nm = min(left, nq - q);
        left -= nm;
        const bool alive = g * 32 + lane < n_live;
        const int k = kept[min(g * 32 + lane, n_live - 1)] >> 1;
        const float4 *r4 = reinterpret_cast<const float4 *>(A.gtab + (size_t)(g0 + k) * GREC);
        const bool in_runs = shared_x || !(misfit & MISFIT_Y);
        GradSums<double> m;
        const float4 ra = r4[0];
        float fxx = r4[1].x, fxy = r4[1].z, fyy = r4[2].x;
        const LaneForm f(shared_x ? ra.z : ra.x, shared_x ? ra.x : ra.z, shared_x ? fyy : fxx, fxy,
                         shared_x ? fxx : fyy, r4[3].z);
        if (!in_runs)
            pixel_sums(px, A.pv.xpix + pix, A.pv.ypix + pix, UNIT * q, min(UNIT * (q + nm), n_px),
                       f, fxy, fyy, m);
        else if (__any_sync(0xffffffffu, !(f.fuu <= NARROW)))
            run_sums<false>(px, UNIT / 8 * q, UNIT / 8 * (q + nm), f, m);
        else
            run_sums<true>(px, UNIT / 8 * q, UNIT / 8 * (q + nm), f, m);
        // the record is read again here: kept through the loops, it would take
        // the registers of the fifth CTA on an SM
        asm volatile("" : "+l"(r4));
        fxx = r4[1].x, fxy = r4[1].z, fyy = r4[2].x;
        if (in_runs) f.finish(m, fxy, shared_x ? fxx : fyy);
        // derivatives w.r.t. (A, x, y, fxx, fyy, fxy) and, through the Jacobian
        // (amp factors are folded into its rows), the parameters; in double
        // until they are summed over a Gaussian's derivatives, which cancel
        const double hx = shared_x ? m.hv : m.hu, hy = shared_x ? m.hu : m.hv;
        const double wx = shared_x ? m.wv : m.wu, wy = shared_x ? m.wu : m.wv;
        const double hxx = shared_x ? m.hvv : m.huu, hyy = shared_x ? m.huu : m.hvv;
        const double wxx = shared_x ? m.wvv : m.wuu, wyy = shared_x ? m.wuu : m.wvv;
        const double fx = fxx, fz = fxy, fy = fyy, gA = m.h0;
        const double gx = hx - (fx * wx + fz * wy) * (1.0 / 12.0);
        const double gy = hy - (fz * wx + fy * wy) * (1.0 / 12.0);
        const double gfxx = (fx * wxx + fz * m.wuv) * (1.0 / 12.0) - 0.5 * hxx - m.w0 * (1.0 / 24.0);
        const double gfyy = (fy * wyy + fz * m.wuv) * (1.0 / 12.0) - 0.5 * hyy - m.w0 * (1.0 / 24.0);
        const double gfxy = (fz * (wxx + wyy) + (fx + fy) * m.wuv) * (1.0 / 12.0) - m.huv;
        const float4 j0 = r4[4], j1 = r4[5], j2 = r4[6], j3 = r4[7];
        float P[7];
        P[0] = (float)(j0.x * gA);
        P[1] = (float)(j1.y * gx + j1.z * gy);
        P[2] = (float)(j1.w * gx + j2.x * gy);
        P[3] = (float)(j0.y * gA + j2.y * gfxx + j2.z * gfxy + j2.w * gfyy);
        P[4] = (float)(j0.z * gA + j3.x * gfxx + j3.y * gfxy + j3.z * gfyy);
        P[5] = (float)(j0.w * gA);
        P[6] = (float)(j1.x * gA);
        // per-source sums: sources are contiguous in the kept list, so each
        // source's first lane collects the lanes after it
        const int src = alive ? (int)min((unsigned)__float_as_int(j3.w),
                                         (unsigned)(A.pv.n_sources - 1))
                              : -1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int so = __shfl_down_sync(0xffffffffu, src, o);
            const bool same = lane + o < 32 && so == src;
#pragma unroll
            for (int c = 0; c < 7; ++c) {
                const float v = __shfl_down_sync(0xffffffffu, P[c], o);
                P[c] += same ? v : 0.0f;
            }
        }
        const int before = __shfl_up_sync(0xffffffffu, src, 1);
        if (src >= 0 && (lane == 0 || before != src))
#pragma unroll
            for (int c = 0; c < 7; ++c) row[src * 7 + c] += P[c];
        __syncwarp();
    }
}

// kept-list flag: the low bit of each entry
constexpr int FLAG_LAST_SRC = 1;   // last kept Gaussian of its source

// ------------------------------------------------------------ tile scan
// The ordered list of the exposure's image Gaussians [g0, g1) that can reach
// the tile (box overlap, then the exact minimum of the exp-argument over the
// tile box `bb`), each entry its local index << 1 | flags; with LAST_SRC,
// FLAG_LAST_SRC marks the last kept Gaussian of each source.  Returns the
// number kept; the list is visible to the whole CTA after the next barrier
// (at once with LAST_SRC).
//
// First every warp tests its share, 32 Gaussians at a time, and leaves one
// mask word per 32 in shared memory (`work`, `n_work` words, the last QUEUE of
// every warp its queue); the loads of a
// Gaussian's box and record do not wait on each other, nor one group's on
// another's, and no barrier stands between groups.  A Gaussian whose
// exp-argument at the tile point nearest its centre is clearly below 36 is
// kept; the few whose box reaches the tile but that point does not (a tenth)
// queue up for the exact test, 32 at a time, so that its four edge minima are
// not evaluated for a few lanes of every group.  Then every warp ranks its
// words against the words before them and writes its entries.  (With a barrier
// pair and two dependent load latencies per NT Gaussians the scan took 19,700
// of the 155,700 cycles of a tile of the 20-source patch; with the exact test
// in every group 16,300 of 142,100.)
template <int NT, bool LAST_SRC = false>
__device__ __forceinline__ int scan_tile(const TileArgs &A, float4 bb, int g0, int g1, int npsf,
                                         int *kept, unsigned *work, int n_work) {
    constexpr int NW = NT / 32;
    const int n_mask = n_work - NW * QUEUE;
    unsigned *mask = work;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned below = (1u << lane) - 1u;
    int *queue = reinterpret_cast<int *>(work + n_mask + warp * QUEUE);
    int n_live = 0;
    for (int b0 = g0; b0 < g1; b0 += 32 * n_mask) {
        const int words = (min(g1 - b0, 32 * n_mask) + 31) >> 5;
        if (b0 > g0) __syncthreads();  // the masks of the block before are read
        int queued = 0;
        // the exact test of the first min(queued, 32) Gaussians in the queue
        auto drain = [&] {
            __syncwarp();
            if (lane < queued) {
                const int at = queue[lane];
                const float *r = A.gtab + (size_t)at * GREC;
                if (keeps_tile(*reinterpret_cast<const float4 *>(r),
                               *reinterpret_cast<const float4 *>(r + 4), r[R_FYY], bb))
                    atomicOr(&mask[(at - b0) >> 5], 1u << ((at - b0) & 31));
            }
            const bool more = lane + 32 < queued;
            const int next = more ? queue[lane + 32] : 0;
            __syncwarp();  // every slot is read before it is filled again,
            if (more) queue[lane] = next;
            __syncwarp();  // and this is in place before another lane queues
            queued = max(queued - 32, 0);
        };
#pragma unroll 2
        for (int w = warp; w < words; w += NW) {
            const int idx = b0 + 32 * w + lane;
            const int at = min(idx, g1 - 1);
            const float4 gb = A.gbox[at];
            const float *r = A.gtab + (size_t)at * GREC;
            const float4 ra = *reinterpret_cast<const float4 *>(r);
            const float4 rb = *reinterpret_cast<const float4 *>(r + 4);
            const float fyy = r[R_FYY];
            const bool reach =
                idx < g1 && !(gb.y < bb.x || gb.x > bb.y || gb.w < bb.z || gb.z > bb.w);
            const bool near_enough = reach && near_tile(ra, rb, fyy, bb);
            const unsigned keep = __ballot_sync(0xffffffffu, near_enough);
            const unsigned ask = __ballot_sync(0xffffffffu, reach && !near_enough);
            if (lane == 0) mask[w] = keep;
            if (ask >> lane & 1u) queue[queued + __popc(ask & below)] = at;
            queued += __popc(ask);
            if (queued >= 32) drain();
        }
        if (queued > 0) drain();
        __syncthreads();
        for (int w0 = 0; w0 < words; w0 += 32) {
            const unsigned mine = w0 + lane < words ? mask[w0 + lane] : 0u;
            int upto = __popc(mine);  // inclusive prefix sum over the 32 words
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            const int n = min(32, words - w0);
            for (int j = (warp - w0 % NW + NW) % NW; j < n; j += NW) {
                const unsigned m = __shfl_sync(0xffffffffu, mine, j);
                const int before = __shfl_sync(0xffffffffu, upto, j) - __popc(m);
                if (m >> lane & 1u)
                    kept[n_live + before + __popc(m & below)] =
                        (b0 - g0 + 32 * (w0 + j) + lane) << 1;
            }
            n_live += __shfl_sync(0xffffffffu, upto, 31);
        }
    }
    if (!LAST_SRC) return n_live;
    __syncthreads();
    // last kept Gaussian of each source (sources are contiguous in the list)
    for (int i = tid; i < n_live; i += NT) {
        const int src = (kept[i] >> 1) / npsf;
        const int nxt = (i + 1 < n_live) ? (kept[i + 1] >> 1) / npsf : -1;
        if (nxt != src) kept[i] |= FLAG_LAST_SRC;
    }
    __syncthreads();
    return n_live;
}

// ------------------------------------------------------------ the tile body
// GRAD = false runs the residual pass and chi2 only (no gradient pass, no
// gradient partials written).  EXACT = true runs the residual pass in the
// reference's float arithmetic (residual_exact) instead of the packed pass.
// WAIT = false: the caller has waited for the kernels before.
template <int NT, int K, bool GRAD = true, bool EXACT = false, bool WAIT = true>
__device__ __forceinline__ void tile_body(const TileArgs &A, int tile, unsigned char *smem,
                                          uint64_t *mbar, uint32_t &phase) {
    static_assert(K % 2 == 0, "pixels per thread must be even (packed pairs)");
    constexpr int NW = NT / 32;
    constexpr int KP = K / 2;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cap = A.live_cap;
    const int stride = A.pgrad_stride;

    constexpr int TP = NT * K;  // pixels per tile
    float *recs = reinterpret_cast<float *>(smem);
    // kept list: exposure-local Gaussian index << 1 | FLAG_* bits
    int *kept = reinterpret_cast<int *>(smem + stage_bytes(TP, cap));
    float *wacc = reinterpret_cast<float *>(kept + A.idx_cap);

    __shared__ double s_chi2[NW];
    __shared__ int s_any_weight, s_misfit;
    __shared__ __align__(16) float s_zero[MODEL_STAGE];
    if (tid < MODEL_STAGE) s_zero[tid] = 0.0f;

    const TileDesc td = A.tiles[tile];
    const float4 bb = A.want_residual ? A.tbox_all[tile] : A.tbox_w[tile];
    const int g0 = A.pv.gauss_start[td.exposure];
    const int g1 = A.pv.gauss_start[td.exposure + 1];
    const int npsf = A.pv.exp_npsf[td.exposure];

    for (int j = tid; j < NW * stride; j += NT) wacc[j] = 0.0f;

    // ---- this thread's pixels: K consecutive ones, pair j holds pixels 2j and 2j + 1
    // (the caller may reach the pixel arrays through the device struct, and fill
    // them in a kernel before this one)
    if (WAIT) wait_for_earlier_kernel();
    const float xmid = 0.5f * (bb.x + bb.y), ymid = 0.5f * (bb.z + bb.w);
    v2 X[KP], Y[KP], R[KP], R2[KP];
    float D[K], IE[K];
    bool counts[K];
    int any_w = 0;
#pragma unroll
    for (int j = 0; j < KP; ++j) {
        float xs[2], ys[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int li = tid * K + 2 * j + h;
            const bool ok = li < td.count;
            const int pix = td.pix_begin + (ok ? li : 0);
            xs[h] = ok ? A.pv.xpix[pix] : xmid;
            ys[h] = ok ? A.pv.ypix[pix] : ymid;
            D[2 * j + h] = ok ? A.pv.data[pix] : 0.0f;
            IE[2 * j + h] = ok ? A.pv.ierr[pix] : 0.0f;
            any_w |= (IE[2 * j + h] != 0.0f);
            counts[2 * j + h] = ok && (A.want_residual || IE[2 * j + h] != 0.0f);
        }
        X[j] = pk(xs[0], xs[1]);
        Y[j] = pk(ys[0], ys[1]);
        R[j] = pk(D[2 * j], D[2 * j + 1]);
    }
    const int my_misfit = tile_misfit<K>(A, td, tile, warp * 32 * K);
    if (tid == 0) s_any_weight = s_misfit = 0;

    // ---- the ordered list of kept image Gaussians
    const int n_live = scan_tile<NT>(A, bb, g0, g1, npsf, kept,
                                      reinterpret_cast<unsigned *>(recs),
                                      (int)(stage_bytes(TP, cap) / 4));
    if (any_w) s_any_weight = 1;
    if (my_misfit && lane == 0) atomicOr(&s_misfit, my_misfit);
    __syncthreads();
    const bool tile_has_weight = s_any_weight != 0;
    const int misfit = s_misfit;

    // ---- stage kept records [c0, c0 + n) into shared memory
    auto stage = [&](int c0, int n) {
        stage_records<NT, MODEL_STAGE>(recs, A.gtab + (size_t)g0 * GREC, kept, c0, n,
                                       A.test_extra_tx, mbar, phase, A.err);
    };

    const v2 KEXP2 = pk1(KEXP), KEXPLO2 = pk1(KEXP_LO);
    const int n_chunks = (n_live + cap - 1) / cap;

    // ------------------------------------------------------------ pass 1
    auto pass1 = [&](auto tag) {
        constexpr int SH = decltype(tag)::value;
        for (int c = 0; c < n_chunks; ++c) {
            const int c0 = c * cap, n = min(cap, n_live - c0);
            if (c > 0) __syncthreads();  // previous chunk fully consumed
            stage(c0, n);
            if constexpr (EXACT) {
                for (int i = 0; i < n; ++i)
                    residual_exact<KP>(X, Y, R, recs + (size_t)i * MODEL_STAGE);
            } else {
                residual_range<KP, SH>(X, Y, R, recs, 0, n, s_zero, KEXP2, KEXPLO2);
            }
        }
    };
    const int share = EXACT ? SHARE_NONE : share_of<K>(misfit, A.want_residual);
    if (K == 8 && share == SHARE_Y) {
        share_coordinate<KP>(Y, counts);
        pass1(ShareTag<K == 8 ? SHARE_Y : SHARE_NONE>());
    } else if (K == 8 && share == SHARE_X) {
        share_coordinate<KP>(X, counts);
        pass1(ShareTag<K == 8 ? SHARE_X : SHARE_NONE>());
    } else {
        pass1(ShareTag<SHARE_NONE>());
    }

    // ---- residual store, chi2 (double) and the per-pixel adjoint -2 r ie^2
    double chi2 = 0.0;
#pragma unroll
    for (int j = 0; j < KP; ++j) {
        float r[2];
        unpk(R[j], r[0], r[1]);
        float r2v[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = 2 * j + h;
            const int li = tid * K + k;
            if (A.want_residual && li < td.count) A.pv.residual[td.pix_begin + li] = r[h];
            const float ie = IE[k];
            const float rie = r[h] * ie;
            const float die = D[k] * ie;
            double c = ((double)rie - (double)die);
            c *= ((double)rie + (double)die);
            chi2 += (ie != 0.0f) ? c : 0.0;
            r2v[h] = (ie != 0.0f) ? -2.0f * (rie * ie) : 0.0f;
        }
        R2[j] = pk(r2v[0], r2v[1]);
    }
    chi2 = warp_sum_d(chi2);
    if (lane == 0) s_chi2[warp] = chi2;

    // ------------------------------------------------------------ pass 2
    // the pixels in shared memory (over the staged records), px_block of them
    // at a time; every kept Gaussian in a lane
    if (GRAD && tile_has_weight && n_live > 0) {
        const int pxb = px_block(TP, cap);
        const PixelStage px = {recs, recs + pxb, recs + pxb + pxb / 8};
        for (int b0 = 0; b0 < td.count; b0 += pxb) {
            __syncthreads();  // records (or the previous pixels) fully consumed
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int p = tid * K + k - b0;
                if (p >= 0 && p < pxb) px.r2[run_slot(p)] = k & 1 ? hi(R2[k / 2]) : lo(R2[k / 2]);
            }
            stage_runs<NT, TP>(A, td, tile, b0, pxb, runs_share_x(misfit), px);
            __syncthreads();
            gradient_lanes<NW>(A, kept, n_live, g0, px, td.pix_begin + b0,
                               min(pxb, td.count - b0), misfit, wacc);
        }
    }
    __syncthreads();

    // ---- tile partials (fixed-order sums)
    if (tid == 0) {
        double c = 0.0;
#pragma unroll
        for (int w = 0; w < NW; ++w) c += s_chi2[w];
        A.pchi2[tile] = c;
    }
    for (int j = tid; GRAD && j < stride; j += NT) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; ++w) v += wacc[w * stride + j];
        A.pgrad[(size_t)tile * stride + j] = v;
    }
    if (A.tile_cost && tid == 0) A.tile_cost[tile] = n_live * td.count;
    if (A.pairs && tid == 0) atomicAdd(reinterpret_cast<unsigned long long *>(A.pairs),
                                       (unsigned long long)((long long)n_live * td.count));
}

// ------------------------------------------------------------ split tile body
// A tile of 32*K pixels evaluated by NW warps that share the tile's kept
// Gaussians: every warp holds all of the tile's pixels (lane l holds pixels
// l, l+32, ..., K per thread, as K/2 packed pairs) and takes a contiguous
// 1/NW of each staged chunk of kept Gaussians.
//   pass 1: each warp sums -model over its Gaussians; the NW partial models
//           are added to the data in warp order through shared memory;
//   chi2:   each thread its share of the pixels, in double;
//   pass 2: gradient_lanes, as tile_body; each warp sums into its own
//           shared-memory row; the rows are added in warp order at the end.
// Against tile_body with NT = 32 NW threads and K' = K / NW pixels per thread
// on the same tile, each thread does the per-Gaussian work (record loads,
// exp-argument set-up, Jacobian epilogue) for NW times as many pixels, and a
// CTA slot takes NW times fewer pixels per Gaussian, so tiles stay small (good
// culling) while a launch has more tiles per resident CTA (a shorter tail).
// Results are deterministic; the residual is summed in a different order from
// tile_body's, so the two agree to rounding, not bit for bit.
//
// With PS > 1 a CTA takes one of PS parts of the tile's pixels (K / PS per
// lane) and writes partial PS tile + part; the list of kept Gaussians and its
// shares are the whole tile's, so every pixel's residual is the same bit for
// bit.  For patches whose tiles do not fill the GPU's SMs evenly.
__host__ __device__ inline size_t split_smem_layout_bytes(int nw, int k, int live_cap, int idx_cap,
                                                         int stride) {
    return tile_smem_layout_bytes(nw, 32 * k, live_cap, idx_cap, stride) + (size_t)nw * 32 * k * 4;
}

template <int NW, int K, bool GRAD = true, int PS = 1, bool WAIT = true>
__device__ __forceinline__ void tile_body_split(const TileArgs &A, int tile, int part,
                                                unsigned char *smem, uint64_t *mbar,
                                                uint32_t &phase) {
    static_assert(K % (2 * PS) == 0, "pixels per lane must be even (packed pairs)");
    constexpr int NT = 32 * NW;
    constexpr int KL = K / PS;  // pixels per lane
    constexpr int KP = KL / 2;
    constexpr int TP = 32 * K;   // pixels per tile
    constexpr int PP = TP / PS;  // pixels of a part
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cap = A.live_cap;
    const int stride = A.pgrad_stride;

    float *recs = reinterpret_cast<float *>(smem);
    int *kept = reinterpret_cast<int *>(smem + stage_bytes(TP, cap));
    float *wacc = reinterpret_cast<float *>(kept + A.idx_cap);
    float *pmodel = wacc + (size_t)NW * stride;  // [NW][PP] partial models

    __shared__ double s_chi2[NW];
    __shared__ __align__(16) float s_zero[MODEL_STAGE];
    if (tid < MODEL_STAGE) s_zero[tid] = 0.0f;

    TileDesc td = A.tiles[tile];
    const float4 bb = A.want_residual ? A.tbox_all[tile] : A.tbox_w[tile];
    const int g0 = A.pv.gauss_start[td.exposure];
    const int g1 = A.pv.gauss_start[td.exposure + 1];
    const int npsf = A.pv.exp_npsf[td.exposure];
    if (PS > 1) {  // this part's pixels
        td.pix_begin += part * PP;
        td.count = max(0, min(PP, td.count - part * PP));
        if (td.count == 0) td.pix_begin -= part * PP;  // (an index that exists)
    }

    for (int j = tid; j < NW * stride; j += NT) wacc[j] = 0.0f;

    // ---- the pixels, in every warp: KL consecutive ones per lane (after the
    // wait, as in tile_body)
    if (WAIT) wait_for_earlier_kernel();
    const float xmid = 0.5f * (bb.x + bb.y), ymid = 0.5f * (bb.z + bb.w);
    v2 X[KP], Y[KP], R[KP];
    bool counts[KL];
#pragma unroll
    for (int j = 0; j < KP; ++j) {
        float xs[2], ys[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int li = lane * KL + 2 * j + h;
            const bool ok = li < td.count;
            const int pix = td.pix_begin + (ok ? li : 0);
            xs[h] = ok ? A.pv.xpix[pix] : xmid;
            ys[h] = ok ? A.pv.ypix[pix] : ymid;
            counts[2 * j + h] = ok && (A.want_residual || A.pv.ierr[pix] != 0.0f);
        }
        X[j] = pk(xs[0], xs[1]);
        Y[j] = pk(ys[0], ys[1]);
        R[j] = 0ull;  // -model of this warp's Gaussians
    }
    const float4 wbox = A.tbox_w[tile];
    const bool tile_has_weight = wbox.x <= wbox.y;  // the box of no pixels is empty
    const int misfit = tile_misfit<KL>(A, td, tile, 0);

    const int n_live = scan_tile<NT>(A, bb, g0, g1, npsf, kept,
                                      reinterpret_cast<unsigned *>(recs),
                                      (int)(stage_bytes(TP, cap) / 4));
    __syncthreads();  // the list is complete, the masks are read

    auto stage = [&](int c0, int n) {
        stage_records<NT, MODEL_STAGE>(recs, A.gtab + (size_t)g0 * GREC, kept, c0, n,
                                       A.test_extra_tx, mbar, phase, A.err);
    };
    // this warp's share [i0, i1) of a chunk of n records: contiguous, even
    // lengths (two Gaussians per step)
    auto share = [&](int n, int &i0, int &i1) {
        const int per = 2 * ((n + 2 * NW - 1) / (2 * NW));
        i0 = min(n, warp * per);
        i1 = min(n, i0 + per);
    };

    const v2 KEXP2 = pk1(KEXP), KEXPLO2 = pk1(KEXP_LO);
    const int n_chunks = (n_live + cap - 1) / cap;

    // ------------------------------------------------------------ pass 1
    auto pass1 = [&](auto tag) {
        constexpr int SH = decltype(tag)::value;
        for (int c = 0; c < n_chunks; ++c) {
            const int c0 = c * cap, n = min(cap, n_live - c0);
            if (c > 0) __syncthreads();
            stage(c0, n);
            int i0, i1;
            share(n, i0, i1);
            residual_range<KP, SH>(X, Y, R, recs, i0, i1, s_zero, KEXP2, KEXPLO2);
        }
    };
    const int shared = share_of<K>(misfit, A.want_residual);
    if (K == 8 && shared == SHARE_Y) {
        share_coordinate<KP>(Y, counts);
        pass1(ShareTag<K == 8 ? SHARE_Y : SHARE_NONE>());
    } else if (K == 8 && shared == SHARE_X) {
        share_coordinate<KP>(X, counts);
        pass1(ShareTag<K == 8 ? SHARE_X : SHARE_NONE>());
    } else {
        pass1(ShareTag<SHARE_NONE>());
    }

    // ---- the residual: data plus the warps' partial (negative) models, in warp order
#pragma unroll
    for (int j = 0; j < KP; ++j) {
        float m0, m1;
        unpk(R[j], m0, m1);
        pmodel[warp * PP + lane * KL + 2 * j] = m0;
        pmodel[warp * PP + lane * KL + 2 * j + 1] = m1;
    }
    __syncthreads();
    // each thread finishes its share of the pixels: residual, chi2 (double) and
    // the gradient pass's pixels, over the staged records (no longer read)
    const PixelStage px = {recs, recs + PP, recs + PP + PP / 8};
    double chi2 = 0.0;
#pragma unroll
    for (int i = 0; i < (PP + NT - 1) / NT; ++i) {
        const int li = tid + i * NT;
        if (li >= PP) break;  // whole warps
        const bool ok = li < td.count;
        const int pix = td.pix_begin + (ok ? li : 0);
        const float d = ok ? A.pv.data[pix] : 0.0f;
        const float ie = ok ? A.pv.ierr[pix] : 0.0f;
        float r = d;
#pragma unroll
        for (int w = 0; w < NW; ++w) r += pmodel[w * PP + li];
        if (A.want_residual && ok) A.pv.residual[pix] = r;
        const float rie = r * ie, die = d * ie;
        double c = ((double)rie - (double)die);
        c *= ((double)rie + (double)die);
        chi2 += (ie != 0.0f) ? c : 0.0;
        if (GRAD) px.r2[run_slot(li)] = (ie != 0.0f) ? -2.0f * ((r * ie) * ie) : 0.0f;
    }
    if (GRAD)
        stage_runs<NT, PP>(A, td, tile * PS + part, 0, PP, runs_share_x(misfit), px);
    chi2 = warp_sum_d(chi2);
    if (lane == 0) s_chi2[warp] = chi2;

    // ------------------------------------------------------------ pass 2
    if (GRAD && tile_has_weight && n_live > 0) {
        __syncthreads();  // every pixel staged
        gradient_lanes<NW, 64 / PS>(A, kept, n_live, g0, px, td.pix_begin, td.count, misfit,
                                    wacc);
    }
    __syncthreads();

    // ---- tile partials (fixed-order sums)
    if (tid == 0) {
        double c = 0.0;
#pragma unroll
        for (int w = 0; w < NW; ++w) c += s_chi2[w];
        A.pchi2[tile * PS + part] = c;
    }
    for (int j = tid; GRAD && j < stride; j += NT) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; ++w) v += wacc[w * stride + j];
        A.pgrad[(size_t)(tile * PS + part) * stride + j] = v;
    }
    if (A.tile_cost && tid == 0) A.tile_cost[tile] = n_live * td.count;
    if (A.pairs && tid == 0) atomicAdd(reinterpret_cast<unsigned long long *>(A.pairs),
                                       (unsigned long long)((long long)n_live * td.count));
}

// ------------------------------------------------------------ design rows
// Records per shared-memory stage of the design passes (the design matrix and
// the flux solve's normal equations): each chunk is staged once, so a small
// stage costs little and lets more CTAs reside.  Both passes use it, so their
// unit-flux rows -- flushed at source boundaries and chunk ends -- are the
// same floats.
constexpr int DESIGN_LIVE_CAP = 64;
// The unit-flux model of one Gaussian (dA/dflux in place of the amplitude)
// accumulated, negated, into M, as residual_pairs does for the model.
template <int KP>
__device__ __forceinline__ void design_one(const v2 (&Xp)[KP], const v2 (&Yp)[KP], v2 (&M)[KP],
                                           const float *r, v2 CM24, v2 KEXP2, v2 KEXPLO2) {
    v2 NXC, NYC, FXX, FXY, FYY, AMP, HB, C0;
    ld2(r + R_NXC, NXC, NYC);
    ld2(r + R_FXX, FXX, FXY);
    ld2(r + R_FYY, FYY, AMP);
    ld2(r + R_HB, HB, C0);
    const v2 UA = pk1(r[R_JA_FLUX]);
    const v2 HA = mul2(UA, CM24);
    const v2 UB = mul2(pk1(-1.0f), mul2(UA, C0));
    residual_pairs<KP>(Xp, Yp, M, NXC, NYC, FXX, FXY, FYY, HA, UB, KEXP2, KEXPLO2);
}

// The same for two consecutive Gaussians a, b of one source at once (their
// exponentials interleave), M updated with a's term and then b's.
template <int KP, int SH = SHARE_NONE>
__device__ __forceinline__ void design_pairs2(const v2 (&Xp)[KP], const v2 (&Yp)[KP],
                                              v2 (&M)[KP], const float *ra, const float *rb,
                                              v2 CM24, v2 KEXP2, v2 KEXPLO2) {
    v2 NXa, NYa, FXXa, FXYa, FYYa, AMPa, HBa, C0a;
    v2 NXb, NYb, FXXb, FXYb, FYYb, AMPb, HBb, C0b;
    ld2(ra + R_NXC, NXa, NYa);
    ld2(ra + R_FXX, FXXa, FXYa);
    ld2(ra + R_FYY, FYYa, AMPa);
    ld2(ra + R_HB, HBa, C0a);
    ld2(rb + R_NXC, NXb, NYb);
    ld2(rb + R_FXX, FXXb, FXYb);
    ld2(rb + R_FYY, FYYb, AMPb);
    ld2(rb + R_HB, HBb, C0b);
    const v2 UAa = pk1(ra[R_JA_FLUX]), UAb = pk1(rb[R_JA_FLUX]);
    const v2 HAa = mul2(UAa, CM24), HAb = mul2(UAb, CM24);
    const v2 UBa = mul2(pk1(-1.0f), mul2(UAa, C0a)), UBb = mul2(pk1(-1.0f), mul2(UAb, C0b));
#pragma unroll
    for (int j = 0; j < KP; ++j) {
        const v2 DXa = add2(Xp[SH == SHARE_X ? 0 : j], NXa), DYa = add2(Yp[SH == SHARE_Y ? 0 : j], NYa);
        const v2 DXb = add2(Xp[SH == SHARE_X ? 0 : j], NXb), DYb = add2(Yp[SH == SHARE_Y ? 0 : j], NYb);
        const v2 VXa = fma2(FXYa, DYa, mul2(FXXa, DXa));
        const v2 VXb = fma2(FXYb, DYb, mul2(FXXb, DXb));
        const v2 VYa = fma2(FXYa, DXa, mul2(FYYa, DYa));
        const v2 VYb = fma2(FXYb, DXb, mul2(FYYb, DYb));
        const v2 Qa = fma2(DYa, VYa, mul2(DXa, VXa));
        const v2 Qb = fma2(DYb, VYb, mul2(DXb, VXb));
        v2 Ga = exp_neg_half(Qa, KEXP2, KEXPLO2);
        v2 Gb = exp_neg_half(Qb, KEXP2, KEXPLO2);
        {
            float g0, g1, q0, q1;
            unpk(Ga, g0, g1);
            unpk(Qa, q0, q1);
            Ga = pk(q0 > FPHO_MAX_EXP_ARG ? 0.0f : g0, q1 > FPHO_MAX_EXP_ARG ? 0.0f : g1);
            unpk(Gb, g0, g1);
            unpk(Qb, q0, q1);
            Gb = pk(q0 > FPHO_MAX_EXP_ARG ? 0.0f : g0, q1 > FPHO_MAX_EXP_ARG ? 0.0f : g1);
        }
        const v2 Sa = fma2(VYa, VYa, mul2(VXa, VXa));
        const v2 Sb = fma2(VYb, VYb, mul2(VXb, VXb));
        M[j] = fma2(fma2(Sa, HAa, UBa), Ga, M[j]);
        M[j] = fma2(fma2(Sb, HAb, UBb), Gb, M[j]);
    }
}
// The unit-flux model of every source at every pixel of the tile:
// X[src][pix] = sum over the source's image Gaussians of dA/dflux * G * H
// (dA/dflux = the record's R_JA_FLUX; with the source's flux this is its model
// divided by the flux, as the reference's design matrix,
// forcepho/patches/device_patch.py:198-238).  Same scan, staging and
// exponential as the residual pass; X must be zero on entry, and every
// (src, pixel) is written by one thread only.
template <int NT, int K>
__device__ __forceinline__ void design_body(const TileArgs &A, int tile, unsigned char *smem,
                                            uint64_t *mbar, uint32_t &phase, float *X,
                                            long long npix) {
    static_assert(K % 2 == 0, "pixels per thread must be even (packed pairs)");
    constexpr int KP = K / 2;
    const int tid = threadIdx.x;
    const int cap = A.live_cap;
    float *recs = reinterpret_cast<float *>(smem);
    int *kept = reinterpret_cast<int *>(smem + (size_t)cap * GSTAGE * 4);

    const TileDesc td = A.tiles[tile];
    const float4 bb = A.tbox_all[tile];
    const int g0 = A.pv.gauss_start[td.exposure];
    const int g1 = A.pv.gauss_start[td.exposure + 1];
    const int npsf = A.pv.exp_npsf[td.exposure];
    const float xmid = 0.5f * (bb.x + bb.y), ymid = 0.5f * (bb.z + bb.w);
    v2 Xp[KP], Yp[KP], M[KP];
#pragma unroll
    for (int j = 0; j < KP; ++j) {
        float xs[2], ys[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int li = tid + (2 * j + h) * NT;
            const bool ok = li < td.count;
            const int pix = td.pix_begin + (ok ? li : 0);
            xs[h] = ok ? A.pv.xpix[pix] : xmid;
            ys[h] = ok ? A.pv.ypix[pix] : ymid;
        }
        Xp[j] = pk(xs[0], xs[1]);
        Yp[j] = pk(ys[0], ys[1]);
        M[j] = 0ull;
    }
    const int n_live = scan_tile<NT, true>(A, bb, g0, g1, npsf, kept,
                                            reinterpret_cast<unsigned *>(recs), cap * GSTAGE);
    const v2 KEXP2 = pk1(KEXP), KEXPLO2 = pk1(KEXP_LO), CM24 = pk1(-1.0f / 24.0f);
    for (int c0 = 0; c0 < n_live; c0 += cap) {
        const int n = min(cap, n_live - c0);
        if (c0 > 0) __syncthreads();
        stage_records<NT, GSTAGE>(recs, A.gtab + (size_t)g0 * GREC, kept, c0, n, 0, mbar, phase, A.err);
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
                const int src = min((unsigned)__float_as_int(r[R_SRC]),
                                    (unsigned)(A.pv.n_sources - 1));
                float *row = X + (size_t)src * npix + td.pix_begin;
#pragma unroll
                for (int j = 0; j < KP; ++j) {
                    float m0, m1;
                    unpk(M[j], m0, m1);  // accumulated -model
                    const int l0 = tid + 2 * j * NT, l1 = l0 + NT;
                    if (l0 < td.count) row[l0] -= m0;
                    if (l1 < td.count) row[l1] -= m1;
                    M[j] = 0ull;
                }
            }
        }
    }
}

}  // namespace fpho
