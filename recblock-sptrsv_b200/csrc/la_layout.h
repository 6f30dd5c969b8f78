// la_layout.h -- layout of the look-ahead level kernel (level_la.cuh),
// shared by the host builder (la_build.h) and the kernel.
//
// The WHOLE matrix (every independent segment of it, for a batch) is cut
// into chunks: rows of one level, contiguous processing positions
// [lo, lo+nr).  A row's strictly-lower entries are split by where the
// dependency's x is found:
//   late  -- the dependency is a row of the chunk just before: read by the
//            row's own thread after that chunk's barrier;
//   early -- an earlier row: summed one chunk ahead by the helper threads,
//            from the shared-memory window of the last xw rows;
//   old   -- an early entry whose row has left the window: its x is copied
//            from global memory into a slot of the LA_AUX ring ahead of use
//            and the entry points at that slot.
// "Virtual row" = the row's index in its segment's chunk sequence.
//
// Slots (indices into one shared array of values): virtual row v at v mod
// xw; the ring of old values from xw; two buffers of helper sums, one per
// helper thread, from xw + LA_AUX (chunk j's in buffer j mod 2); then a slot
// that is always zero (padding).
//
// Every record has the same size and places: with NM = 32 * main warps and
// NH = 32 * helper warps,
//   int4 {lo, v0 mod xw, nr, 0}
//   main words   4 per thread t < NM: slots of the row's first LA_LATE terms
//                (the zero slot where it has fewer), then its extra terms:
//                first << 5 | count
//   helper slots Q per thread h < NH, per warp four words at a time:
//                [NH / 32][Q / 4][32][4]
//   extra slots  NX
//   values       main: [NM / 32][2][32][2] (first two terms; third term,
//                inverse diagonal); helper: [NH / 32][Q / 2][32][2]; extra: NX
// Helper thread h < nr sums up to Q early entries of row h; a row with more
// has them in further threads >= nr.  A row's terms are its late entries and
// the sums of those further threads (with the value 1).
#pragma once

#ifndef __CUDACC__
#ifndef __host__
#define __host__
#define __device__
#endif
#endif

namespace rbs {

constexpr int LA_RMAX = 256;     // rows per chunk at most
constexpr int LA_AUX = 512;      // ring of gathered old values
constexpr int LA_LATE = 3;       // terms of a row read ahead of the barrier
constexpr int LA_OLD = 64;       // old entries per chunk at most
constexpr int LA_XW_MIN = 2048, LA_XW_MAX = 8192;
constexpr int LA_SLOTS = 32;     // record ring slots at most
constexpr int LA_SLOTS_MIN = 5;  // and at least
constexpr int LA_AHEAD = 5;      // old values are gathered this many chunks ahead,
constexpr int LA_IDX = 9;        // their positions read this many chunks ahead
static_assert(LA_XW_MIN >= (LA_AHEAD + 1) * LA_RMAX, "old values are final when they are gathered");
static_assert(LA_AUX >= (LA_AHEAD + 2) * LA_OLD, "gathered values are used before their slots are");
constexpr int LA_SMEM = 232448 - 1024;
constexpr int LA_THREADS = 960;  // main and helper threads at most
// FP64 records at most: eight times the matrix's CSR (12 bytes an entry), or 16
// MB.  A record is as large for one row as for a full chunk, so levels of a few
// rows take many times the matrix: bands of 128 with 4 to 12 entries a row 3.8
// to 5.4 times, a batch of 256 bands of 256 2.4 times, a band of 24 with 10
// entries 14 times, a chain that reads its last 9 rows 31 times.
constexpr double la_most_bytes(int nnz, int n) {
    const double csr = 12.0 * nnz + 4.0 * (n + 1.0);
    return 8 * csr > 16e6 ? 8 * csr : 16e6;
}

struct LaChunk {
    int lo, nr;    // processing positions [lo, lo + nr)
    int ooff, on;  // old entries: positions old[ooff, ooff + on)
};
constexpr int LA_TAB_INTS = 4;
static_assert(sizeof(LaChunk) == LA_TAB_INTS * sizeof(int), "table rows are LA_TAB_INTS ints");

// Sizes of one plan's layout and byte offsets inside a record.
struct LaDim {
    int xw, nm, nh, q, nx;  // window, main threads, helper threads, lines, extra terms (a multiple of 8)
    static constexpr int o_main = 16;
    __host__ __device__ int o_help() const { return o_main + 8 * nm; }
    __host__ __device__ int o_extra() const { return o_help() + 2 * q * nh; }
    __host__ __device__ int o_val() const { return o_extra() + 2 * nx; }
    // word of helper thread h's line k (from o_help), value places (from o_val)
    __host__ __device__ int w_help(int h, int k) const { return ((h >> 5) * (q / 4) + k / 4) * 128 + (h & 31) * 4 + k % 4; }
    __host__ __device__ int v_help(int h, int k) const {
        return 4 * nm + ((h >> 5) * (q / 2) + k / 2) * 64 + (h & 31) * 2 + k % 2;
    }
    __host__ __device__ static constexpr int v_main(int t, int k) { return ((t >> 5) * 2 + k / 2) * 64 + (t & 31) * 2 + k % 2; }
    // offsets in values from o_val
    __host__ __device__ int v_extra() const { return 4 * nm + q * nh; }
    __host__ __device__ int v_count() const { return v_extra() + nx; }
    __host__ __device__ int rec_bytes(int es) const { return o_val() + es * v_count(); }
    __host__ __device__ int s_part() const { return xw + LA_AUX; }
    __host__ __device__ int s_zero() const { return s_part() + 2 * nh; }
    // right-hand sides behind the record: a 16-byte copy window of nm values
    __host__ __device__ int slot_bytes(int es) const { return (rec_bytes(es) + es * nm + 32 + 127) / 128 * 128; }
    // shared memory besides the record slots: values, mbarriers, ring of old positions
    __host__ __device__ int fixed_bytes(int es) const {
        return ((s_zero() + 16) * es + 2 * LA_SLOTS * 8 + 8 * LA_OLD * 4 + 127) / 128 * 128;
    }
    __host__ __device__ int slots(int es) const {
        const int s = (LA_SMEM - fixed_bytes(es)) / slot_bytes(es);
        return s < LA_SLOTS ? s : LA_SLOTS;
    }
};

}  // namespace rbs
