// level_strip.cuh -- strip kernel: the whole matrix in one launch, one warp
// per strip of 32 chains (strip_layout.h).
//
// A warp walks its strip level by level without any barrier: a step is one
// row per lane, its dependencies read from a shared-memory window that only
// this warp writes.  Values of other strips come through an exchange vector
// in global memory that starts as a sentinel arithmetic never produces, so a
// relaxed load both polls and fetches.  They are asked for one chunk (8
// steps) ahead; a strip that catches up with the one before it falls back
// until that succeeds at once, so the round trip to L2 is paid per strip and
// not per level.  A chunk's published rows are written when it ends, and the
// same numbers of the other exchange vector, which the next walk uses, are
// set back to the sentinel.  Strips are handed out by a ticket and depend on
// earlier ones only, so any residency makes progress.  The ticket counts to
// twice the strips and starts anew: its half is the walk's parity, which says
// which of the two exchange vectors is clean, so that state is the device's
// alone and a walk can be recorded in a graph and replayed.
//
// A second warp streams the records through a ring with bulk copies and, for
// a walk on the caller's vectors (IO), gathers the right-hand sides of a
// chunk with asynchronous copies in the order of the original rows (a grid's
// chunk: runs of 64 bytes); a third writes a chunk's solutions from the
// window to the caller's vector in that order.  So such a walk reads each
// right-hand side once and writes each solution once.  Walks of the FP32
// sweeps (not IO) read and write work vectors in strip order.
//
// What bounds it: the step's chain (window write, window read, two
// multiply-adds, subtraction, multiplication) and the instructions around it,
// about 80 ns a step for a strip alone (8,192 x 32 grid), and the steps every strip falls behind
// the one before it (122 ns a level over 32 strips).  Measured against the
// block walk of staged level triangles it replaces (one B200, whole solve):
// 1024 x 1024 grid forward 945 -> 260 us (265 with the ticket set to zero by a
// memset before each walk), 777 x 777 backward 587 -> 199 us, 32 columns
// 1,340 -> 512 us, 64 columns 1,830 -> 863 us.  Without the fused moves
// (gather and scatter kernels in strip order) 32 columns took 1,255 us; asking
// for remote values a whole chunk ahead, with chunks not shifted, 288 us for
// one column.  Past 16 columns the caller's vectors bound it: 64-byte pieces of
// rows 8 KB apart, read with 256-byte L2 prefetch (564 -> 505 us at 32).
//
// G columns per CTA (blockIdx.y selects them) share a record's reads.
#pragma once

#include "level_la.cuh"
#include "strip_layout.h"

namespace rbs {

template <typename VT>
struct StripArgs {
    const unsigned char *rec;
    const int *first;  // first chunk of every strip, and the end
    int nstrip;
    // IO: the caller's columns, b + c * ldb and x + c * ld (or the tables'), c < k
    const double *b64;
    double *x64;
    const double *const *bcols;
    double *const *xcols;
    int ldb, ld, k;
    const int *rows;             // per chunk its original rows ascending (-1 last)
    const unsigned char *rows_at;  // and the position in the chunk of each
    // otherwise: work vectors in strip order, column group y at + y * gstride
    const VT *b;
    VT *x;
    long long gstride;
    VT *ex0, *ex1;     // exchange vectors of even and odd walks, column group y at + y * published * G
    int published;
    unsigned *ticket;  // one per column group, kept from walk to walk
    int *status;
    long long limit;
};

// A lane's eight of a chunk's original rows and their positions: entry q *
// 32 + lane of the ascending order, so that one access of a warp covers 32
// neighbouring rows.
struct StripList {
    int4 r0, r1;
    uint2 a;
    __device__ __forceinline__ void load(const int *rows, const unsigned char *at, int chunk, int lane) {
        const long long o = (long long)chunk * ST_ROWS + 8 * lane;
        r0 = *reinterpret_cast<const int4 *>(rows + o);
        r1 = *reinterpret_cast<const int4 *>(rows + o + 4);
        a = *reinterpret_cast<const uint2 *>(at + o);
    }
    __device__ __forceinline__ int row(int q) const {
        return q == 0 ? r0.x : q == 1 ? r0.y : q == 2 ? r0.z : q == 3 ? r0.w : q == 4 ? r1.x : q == 5 ? r1.y : q == 6 ? r1.z : r1.w;
    }
    __device__ __forceinline__ unsigned at(int q) const { return ((q < 4 ? a.x : a.y) >> (8 * (q & 3))) & 255u; }
};

// bytes of a right-hand side in shared memory: the caller's doubles, or work-vector values
template <typename VT, bool IO> constexpr int st_b_bytes() { return IO ? 8 : (int)sizeof(VT); }
template <typename VT, int W, int G, bool IO>
constexpr int st_slot_bytes() { return (st_rec_bytes(W, sizeof(VT)) + 127) / 128 * 128 + ST_ROWS * G * st_b_bytes<VT, IO>(); }
template <typename VT, int W, int G, bool IO>
constexpr int st_smem() {
    return st_slots(G) * st_slot_bytes<VT, W, G, IO>() + (ST_VALS * G * (int)sizeof(VT) + 127) / 128 * 128 + 128;
}

// FP32 records from the FP64 ones: the words copied, the values rounded.
static __global__ void k_strip_rec32(int W, const unsigned char *__restrict__ r64, unsigned char *__restrict__ r32) {
    const unsigned char *s = r64 + (size_t)blockIdx.x * st_rec_bytes(W, 8);
    unsigned char *t = r32 + (size_t)blockIdx.x * st_rec_bytes(W, 4);
    const int wb = 2 * st_words(W);
    for (int i = threadIdx.x; i < wb / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(t)[i] = reinterpret_cast<const uint4 *>(s)[i];
    const double *sv = reinterpret_cast<const double *>(s + wb);
    float *dv = reinterpret_cast<float *>(t + wb);
    for (int i = threadIdx.x; i < st_values(W); i += blockDim.x) dv[i] = (float)sv[i];
}

// G consecutive values at a shared address
template <int G, typename T>
__device__ __forceinline__ void lds_g(T (&v)[G], unsigned p) {
    if constexpr (G == 1) {
        lds_v(v[0], p);
    } else {
#pragma unroll
        for (int g = 0; g < G; g += 2) {
            T t[2];
            lds_v2(t, p + (unsigned)sizeof(T) * g);
            v[g] = t[0];
            v[g + 1] = t[1];
        }
    }
}
__device__ __forceinline__ void sts_v2(unsigned p, double a, double b) {
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(p), "d"(a), "d"(b) : "memory");
}
__device__ __forceinline__ void sts_v2(unsigned p, float a, float b) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(p), "f"(a), "f"(b) : "memory");
}
template <int G, typename T>
__device__ __forceinline__ void sts_g(unsigned p, const T (&v)[G]) {
    if constexpr (G == 1) {
        sts_v(p, v[0]);
    } else {
#pragma unroll
        for (int g = 0; g < G; g += 2) sts_v2(p + (unsigned)sizeof(T) * g, v[g], v[g + 1]);
    }
}

template <typename VT, int W, int G, bool IO>
__global__ void __launch_bounds__(96, 4) k_tri_strip(const __grid_constant__ StripArgs<VT> a) {
    static_assert((W == 2 || W == 4) && (G == 1 || G == 2), "record and column forms");
    extern __shared__ __align__(128) unsigned char sm[];
    constexpr int SLOTS = st_slots(G), NW = ST_WIN / ST_STEPS;  // ring slots, chunks in the window
    using BT = std::conditional_t<IO, double, VT>;
    constexpr unsigned E = sizeof(VT), EG = E * G, BG = sizeof(BT) * G;
    constexpr unsigned rec_bytes = st_rec_bytes(W, E), b_off = (rec_bytes + 127) / 128 * 128;
    constexpr unsigned slot_bytes = st_slot_bytes<VT, W, G, IO>();
    __shared__ int s_strip, s_odd;
    __shared__ __align__(8) unsigned long long mbar[3 * SLOTS + 2 * NW];  // landed, free, b landed; solved, written
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned u_ring = smem_u32(sm), u_win = u_ring + SLOTS * slot_bytes;
    const unsigned u_full = smem_u32(mbar), u_empty = u_full + 8 * SLOTS, u_b = u_empty + 8 * SLOTS;
    const unsigned u_done = u_b + 8 * SLOTS, u_out = u_done + 8 * NW;
    if (threadIdx.x == 0) {
        const int t = (int)atomicInc(a.ticket + blockIdx.y, 2u * a.nstrip - 1);
        s_odd = t >= a.nstrip;
        s_strip = s_odd ? t - a.nstrip : t;
        for (int i = 0; i < 2 * SLOTS; ++i) mbar_init(mbar + i, 1);
        for (int i = 0; i < SLOTS; ++i) mbar_init(mbar + 2 * SLOTS + i, 32);
        for (int i = 0; i < 2 * NW; ++i) mbar_init(mbar + 3 * SLOTS + i, 1);
        fence_mbar_init();
        VT z[G] = {};
        sts_g<G>(u_win + EG * ST_ZERO, z);
    }
    __syncthreads();
    const int c0 = a.first[s_strip], nch = a.first[s_strip + 1] - c0;
    const int col0 = blockIdx.y * G;

    if (warp == 1) {
        // ---------------- producer ----------------
        const unsigned char *rec = a.rec + (size_t)c0 * rec_bytes;
        const double *bp[G];
        if constexpr (IO) {
#pragma unroll
            for (int g = 0; g < G; ++g)
                bp[g] = col0 + g >= a.k ? nullptr : a.bcols ? a.bcols[col0 + g] : a.b64 + (long long)(col0 + g) * a.ldb;
        }
        StripList L;
        auto ahead = [&](int j) {  // chunk j's lists into L2: their latency there is what a chunk has to hide
            if (IO && j < nch && lane < 10) {
                const char *p = lane < 8 ? reinterpret_cast<const char *>(a.rows + (long long)(c0 + j) * ST_ROWS) + 128 * lane
                                         : reinterpret_cast<const char *>(a.rows_at + (long long)(c0 + j) * ST_ROWS) + 128 * (lane - 8);
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
            }
        };
        for (int j = 0; j < 8; ++j) ahead(j);
        if constexpr (IO) L.load(a.rows, a.rows_at, c0, lane);
        unsigned sl = 0, par = 1;
        int issued = 0;
        for (; issued < nch; ++issued) {
            const bool ok = la_wait(u_empty + 8 * sl, par, a.limit);
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) atomicOr(a.status, RBS_STATUS_TIMEOUT);
                break;
            }
            if (lane == 0) {
                unsigned char *dst = sm + sl * slot_bytes;
                mbar_arrive_expect_tx(mbar + sl, rec_bytes + (IO ? 0u : ST_ROWS * EG));
                bulk_g2s(dst, rec + (size_t)issued * rec_bytes, rec_bytes, mbar + sl);
                if constexpr (!IO)
                    bulk_g2s(dst + b_off, a.b + blockIdx.y * a.gstride + (long long)(c0 + issued) * ST_ROWS * G, ST_ROWS * EG,
                             mbar + sl);
            }
            if constexpr (IO) {
                const unsigned ub = u_ring + sl * slot_bytes + b_off;
#pragma unroll
                for (int q = 0; q < 8; ++q)
#pragma unroll
                    for (int g = 0; g < G; ++g)
                        if (L.row(q) >= 0 && bp[g])
                            asm volatile("cp.async.ca.shared.global.L2::256B [%0], [%1], 8;" ::"r"(ub + BG * L.at(q) + 8 * g),
                                         "l"(bp[g] + L.row(q))
                                         : "memory");
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(u_b + 8 * sl) : "memory");
                if (issued + 1 < nch) L.load(a.rows, a.rows_at, c0 + issued + 1, lane);
                ahead(issued + 8);
            }
            if (++sl == SLOTS) {
                sl = 0;
                par ^= 1;
            }
        }
        // every copy lands before the CTA exits (bounded)
        asm volatile("cp.async.wait_all;" ::: "memory");
        for (int j = issued > SLOTS ? issued - SLOTS : 0; j < issued; ++j)
            if (!la_wait(u_full + 8 * (j % SLOTS), (unsigned)((j / SLOTS) & 1), a.limit) && lane == 0)
                atomicOr(a.status, RBS_STATUS_TIMEOUT);
        return;
    }
    if (warp == 2) {
        // ---------------- writer (IO): solutions of a chunk to the caller's columns ----------------
        if constexpr (IO) {
            double *xp[G];
#pragma unroll
            for (int g = 0; g < G; ++g)
                xp[g] = col0 + g >= a.k ? nullptr : a.xcols ? a.xcols[col0 + g] : a.x64 + (long long)(col0 + g) * a.ld;
            StripList L;
            L.load(a.rows, a.rows_at, c0, lane);
            for (int k = 0; k < nch; ++k) {
                const bool ok = la_wait(u_done + 8 * (k % NW), (unsigned)((k / NW) & 1), a.limit);
                if (!__all_sync(0xffffffffu, ok)) {
                    if (lane == 0) atomicOr(a.status, RBS_STATUS_TIMEOUT);
                    break;
                }
                const unsigned w = u_win + EG * ST_ROWS * (k % NW);
                VT v[8][G];
#pragma unroll
                for (int q = 0; q < 8; ++q) lds_g<G>(v[q], w + EG * L.at(q));
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(u_out + 8 * (k % NW)) : "memory");
#pragma unroll
                for (int q = 0; q < 8; ++q)
#pragma unroll
                    for (int g = 0; g < G; ++g)
                        if (L.row(q) >= 0 && xp[g]) xp[g][L.row(q)] = (double)v[q][g];
                if (k + 1 < nch) L.load(a.rows, a.rows_at, c0 + k + 1, lane);
            }
        }
        return;
    }

    // ---------------- the strip's warp ----------------
    VT *ex = (s_odd ? a.ex1 : a.ex0) + (long long)blockIdx.y * a.published * G;
    VT *exn = (s_odd ? a.ex0 : a.ex1) + (long long)blockIdx.y * a.published * G;
    unsigned sl = u_ring, mb = u_full, par = 0;  // the chunk after the one in hand
    bool bad = false;
    VT r[G];        // remote value of this lane for the next chunk
    int rnum = -1;  // its number
#pragma unroll
    for (int g = 0; g < G; ++g) r[g] = 0;
    // wait for a record, ask for its remote values: late in the chunk before,
    // about a round trip to L2 ahead (each step of it is a step that every
    // strip falls behind the one before)
    auto ask = [&]() {
        rnum = -1;
        if (!la_wait(mb, par, a.limit)) {
            bad = true;
            return;
        }
        rnum = lds_s32(sl + 4 * lane);
        if (rnum >= 0) {
#pragma unroll
            for (int g = 0; g < G; ++g) r[g] = ld_relaxed(ex + (long long)rnum * G + g);
        }
    };
    ask();
    unsigned wrow = u_win + EG * lane;  // window rows of the chunk
    VT *xw = IO ? nullptr : a.x + blockIdx.y * a.gstride + ((long long)c0 * ST_ROWS + lane) * G;
    for (int k = 0; k < nch; ++k) {
        const unsigned rec = sl;
        // this chunk's remote values into their buffer
        if (rnum >= 0) {
#pragma unroll
            for (int g = 0; g < G; ++g)
                if (Sent<VT>::is(r[g])) r[g] = bad ? Sent<VT>::nan() : wait_value(ex + (long long)rnum * G + g, a.status, a.limit);
            sts_g<G>(u_win + EG * (ST_REM + (k & 1) * 32 + lane), r);
        }
        if constexpr (IO) {
            // its right-hand sides are here, and the rows that left the window are written out
            if (!la_wait(mb + 16 * SLOTS, par, a.limit)) bad = true;
            if (k >= NW && !la_wait(u_out + 8 * (k % NW), (unsigned)((k / NW - 1) & 1), a.limit)) bad = true;
        }
        if (__any_sync(0xffffffffu, bad)) {
            if (lane == 0) atomicOr(a.status, RBS_STATUS_TIMEOUT);
            break;
        }
        const unsigned freed = mb + 8 * SLOTS;
        sl += slot_bytes;
        mb += 8;
        if (sl == u_win) {
            sl = u_ring;
            mb = u_full;
            par ^= 1;
        }
        // slots of the 8 steps
        uint4 w[W];
#pragma unroll
        for (int i = 0; i < W; ++i) w[i] = lds_4(rec + 2 * ST_HEAD + lane * (ST_STEPS * W * 2) + 16 * i);
        const unsigned uv = rec + 2 * st_words(W) + 2 * E * lane, ui = rec + 2 * st_words(W) + E * (ST_ROWS * W + lane);
        const unsigned ub = rec + b_off + BG * lane;
        VT v[W / 2][2], iv;
        BT bv[G];
        auto fetch = [&](int s) {
#pragma unroll
            for (int i = 0; i < W / 2; ++i) lds_v2(v[i], uv + E * 64 * (s * (W / 2) + i));
            lds_v(iv, ui + E * 32 * s);
            lds_g<G>(bv, ub + BG * 32 * s);
        };
        fetch(0);
#pragma unroll
        for (int s = 0; s < ST_STEPS; ++s) {
            unsigned sw[W / 2];  // two slots each
#pragma unroll
            for (int i = 0; i < W / 2; ++i) {
                const int at = s * (W / 2) + i;
                sw[i] = at % 4 == 0 ? w[at / 4].x : at % 4 == 1 ? w[at / 4].y : at % 4 == 2 ? w[at / 4].z : w[at / 4].w;
            }
            __syncwarp();  // the last step's window row
            VT xv[W][G], sum[G];
#pragma unroll
            for (int i = 0; i < W / 2; ++i) {
                lds_g<G>(xv[2 * i], u_win + EG * (sw[i] & 0xffffu));
                lds_g<G>(xv[2 * i + 1], u_win + EG * (sw[i] >> 16));
            }
            VT cv[W / 2][2], ci = iv;
            BT cb[G];
#pragma unroll
            for (int i = 0; i < W / 2; ++i) {
                cv[i][0] = v[i][0];
                cv[i][1] = v[i][1];
            }
#pragma unroll
            for (int g = 0; g < G; ++g) cb[g] = bv[g];
            if (s + 1 < ST_STEPS) fetch(s + 1);
            if (s == ST_ASK && k + 1 < nch) ask();
#pragma unroll
            for (int g = 0; g < G; ++g) {
                // the products first, as everywhere: b - v0 x0 - v1 x1 in two
                // multiply-adds is 5 % faster but rounds b twice (error 1.0 ->
                // 1.3e-16)
                sum[g] = cv[0][0] * xv[0][g];
                sum[g] = fma(cv[0][1], xv[1][g], sum[g]);
#pragma unroll
                for (int i = 1; i < W / 2; ++i) {
                    sum[g] = fma(cv[i][0], xv[2 * i][g], sum[g]);
                    sum[g] = fma(cv[i][1], xv[2 * i + 1][g], sum[g]);
                }
                sum[g] = ((VT)cb[g] - sum[g]) * ci;
            }
            sts_g<G>(wrow + EG * 32 * s, sum);
            if constexpr (!IO) {
#pragma unroll
                for (int g = 0; g < G; ++g) xw[32 * G * s + g] = sum[g];
            }
        }
        __syncwarp();
        // publish, and clear the next walk's numbers
        const uint2 pb = lds_2(rec + 128);
        for (unsigned i = lane; i < pb.y; i += 32) {
            VT pv[G];
            lds_g<G>(pv, wrow - EG * lane + EG * lds_u16(rec + 144 + 2 * i));
#pragma unroll
            for (int g = 0; g < G; ++g) {
                st_relaxed(ex + (long long)(pb.x + i) * G + g, finalize(pv[g]));
                exn[(long long)(pb.x + i) * G + g] = Sent<VT>::value();
            }
        }
        wrow += EG * ST_ROWS;
        if (wrow >= u_win + EG * ST_REM) wrow -= EG * ST_REM;
        if constexpr (!IO) xw += ST_ROWS * G;
        __syncwarp();
        if (lane == 0) {
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(freed) : "memory");
            if constexpr (IO)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(u_done + 8 * (k % NW)) : "memory");
        }
    }
}

}  // namespace rbs
