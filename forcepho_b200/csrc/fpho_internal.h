// fpho_internal.h -- host-side helpers shared by the forcepho_b200 translation units.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "fpho.h"

struct fpho_patch;

namespace fpho {

struct PatchView;
struct TileArgs;

// Record a failure message for fpho_last_error() and return `code`.
int set_error(int code, const char *fmt, ...);
void clear_error();

// Tile-kernel variants (threads per CTA x pixels per thread).
int variant_count();
int variant_tile_pixels(int v);
int variant_threads(int v);
bool variant_has_exact(int v);  // exact-residual kernels compiled for variant v
int variant_split(int v);       // 0: tile_body; NW: tile_body_split with NW warps per tile
size_t tile_smem_bytes(int variant, int live_cap, int idx_cap, int stride);
int device_sms();  // SMs of the current device (cached)
// Parts a tile's pixels are dealt to (a CTA each, a partial result each) when
// the tiles are too few to fill the GPU evenly; at most MAX_TILE_PARTS.
constexpr int MAX_TILE_PARTS = 4;
int tile_parts(int variant, int n_tiles);
// One CTA per part of a tile; or, with `order` and `counter` (both device pointers), the
// persistent form taking tiles in that order (see order_tiles).
// `exact` selects the exact-residual kernel (variant_has_exact must hold).
int launch_tile_kernel(int variant, const TileArgs &A, int n_tiles, cudaStream_t stream,
                       bool grad, const int *order = nullptr, int *counter = nullptr,
                       bool exact = false, int parts = 1);

// Launch of a kernel that may start while the kernel before it on the stream
// runs; the kernel itself waits (wait_for_earlier_kernel) before it touches
// what that one writes, or what any launch between the two of them read.
cudaError_t launch_dependent(const void *fn, dim3 grid, dim3 block, void **args, size_t smem,
                             cudaStream_t s);

PatchView make_view(const fpho_patch *p);

// Device memory of handles (patches, batches, store scratch) comes from the
// device's default memory pool, told to keep freed memory: creating and
// freeing handles one after another then reuses pool memory instead of a
// driver allocation each time (on a busy machine those took milliseconds to
// seconds, erratically).  pool_malloc returns only once the allocation is
// usable from any stream; pool_free first waits for the device, as cudaFree
// does, so memory still read by a kernel is never reused.  The pool keeps
// the high-water mark of handle memory until the process exits.
cudaError_t pool_malloc(void **p, size_t bytes);
void pool_free(void *p);

// Pinned host memory that kernels address directly (at the same address).  A
// block given back, which no kernel may still use, is kept for the next
// pinned_get of the process (16 blocks of up to 1 MiB at most; others are
// freed): allocating and freeing one took from 0.1 to 13 ms beside other
// allocations.  `bytes`: in, the least needed; out, the block's size, which
// pinned_put is told.
constexpr size_t PINNED_KEEP_BYTES = 1 << 20;
cudaError_t pinned_get(void **p, size_t *bytes);
void pinned_put(void *p, size_t bytes);

}  // namespace fpho
