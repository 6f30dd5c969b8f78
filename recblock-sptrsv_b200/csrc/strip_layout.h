// strip_layout.h -- layout of the strip kernel (level_strip.cuh), shared by
// the host builder (strip_build.h) and the kernel.
//
// For matrices whose levels are made of chains, e.g. factors of grids: rows
// are dealt to chains so that a chain has at most one row per level and a
// row's dependencies lie in its own chain or chains opened earlier.  32
// consecutive chains are a strip: one warp walks it level by level, a lane
// per chain, and depends only on strips before it.
//
// Strip order: position = (strip's first chunk + chunk) * 256 + step * 32 +
// lane; a chunk is 8 steps (levels in which the strip has a row).  Positions
// without a row are padding: zero values, zero inverse diagonal.
//
// Rows that another strip reads (or their own strip, once they have left its
// window) are published: they have a number, ascending with the position, and
// their values go through an exchange vector indexed by it.
//
// Slots of a strip's shared memory (values): x of step s of the strip, lane
// l, at (s mod ST_WIN) * 32 + l; values read from the exchange in two buffers
// of 32, chunk k's in buffer k mod 2, from ST_WIN * 32; then a slot that is
// always zero.
//
// Record of a chunk: int remote[32] (numbers read from the exchange, -1:
// none), int first published number, int published rows, 2 unused, then
// 16-bit words: ST_PUB positions in the chunk of the published rows, per lane
// W slots for each of 8 steps ([32][8][W]); then values [8][W / 2][32][2] and
// inverse diagonals [8][32].  Beside the records, per chunk its original rows
// ascending (-1 last) and the position in the chunk of each, entry i of that
// order at (i mod 32) * 8 + i / 32.
#pragma once

#ifndef __CUDACC__
#ifndef __host__
#define __host__
#define __device__
#endif
#endif

namespace rbs {

constexpr int ST_STEPS = 8;              // steps per chunk
constexpr int ST_ROWS = 32 * ST_STEPS;   // positions per chunk
constexpr int ST_WIN = 32;               // steps in the window (a multiple of ST_STEPS)
constexpr int ST_REM = ST_WIN * 32;      // first remote slot
constexpr int ST_ZERO = ST_REM + 64;
constexpr int ST_VALS = ST_ZERO + 16;    // values of shared memory per column
constexpr int ST_PUB = 64;               // published rows per chunk at most
constexpr int ST_HEAD = 64 + 8 + ST_PUB; // 16-bit words before the slots
constexpr int ST_ASK = 3;                // step of a chunk at which the next one's remote values are asked for
// records in the ring: four CTAs of one or two columns fit an SM
__host__ __device__ constexpr int st_slots(int G) { return G == 1 ? 4 : 3; }

__host__ __device__ constexpr int st_words(int W) { return ST_HEAD + ST_ROWS * W; }  // 16-bit words before the values
__host__ __device__ constexpr int st_values(int W) { return ST_ROWS * (W + 1); }
__host__ __device__ constexpr int st_rec_bytes(int W, int es) { return 2 * st_words(W) + es * st_values(W); }
__host__ __device__ constexpr int st_v_val(int W, int step, int lane, int k) {
    return ((step * (W / 2) + k / 2) * 32 + lane) * 2 + k % 2;
}
__host__ __device__ constexpr int st_v_inv(int W, int step, int lane) { return ST_ROWS * W + step * 32 + lane; }
__host__ __device__ constexpr int st_w_slot(int W, int step, int lane, int k) { return ST_HEAD + (lane * ST_STEPS + step) * W + k; }

}  // namespace rbs
