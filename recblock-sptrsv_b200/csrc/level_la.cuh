// level_la.cuh -- look-ahead level kernel: one CTA walks all levels of a
// matrix (or of every system of a batch, one CTA per system at a time) with
// most of each row's sum taken off the level-to-level chain.
//
// A chunk (rows of one level, la_layout.h) is solved between two barriers.
// Only the entries whose dependency is a row of the chunk just before
// ("late", about one to two per row) have to wait for that barrier;
// everything else of the row is summed one chunk ahead by the helper warps.
// In iteration c
//   main warps    solve chunk c: x = (b - (sum + late)) / d, one thread per
//                 row, x into the shared-memory window and to global; then
//                 they read what does not depend on x (slots, values, b, 1/d)
//                 of chunk c + 1 into registers;
//   helper warps  sum the early entries of chunk c + 1, up to Q per thread
//                 with no branch or reduction, and read the slots and values
//                 of chunk c + 2;
//   gather warp   (when rows are read after they left the window) copies the
//                 old values of chunk c + LA_AHEAD into their ring slots.
// The producer warp stays out of those barriers: it refills the ring of
// records with bulk copies as slots free up (one mbarrier per slot for
// landed, one for free), so a copy's issue time is off the chain.
//
// What bounds it: on narrow levels the instructions of one role between two
// barriers, 5-6 cycles each as every role is one short dependent chain (ncu,
// 16k-row band factor: 526 cycles and 495 warp instructions per chunk); hence
// records with every thread's data at fixed places (descriptors, variable
// line counts and lane reductions took 1,000-1,900 cycles per chunk).  Two
// sets of warps taking chunks in turn, so that one reads ahead while the
// other sums, was no faster (560 cycles: all warps meet at every barrier, and
// reading ahead is the longer half).  On wide levels the shared-memory pipe
// (10 bytes per entry staged and read back, 8 random window bytes).
//
// Measured against the level-chunk kernel and block walk it replaces (one
// B200, whole solve): 16k rows, band 512, 445 levels: 335 -> 134 us; 4M rows,
// band 4096, 23k levels: 27.2 -> 15.1 ms; 200k rows, band 1024, 5 columns
// (sync-free kernel before): 2.99 -> 1.03 ms; 256 systems of 1k-50k rows, band
// 256 (sync-free kernel before): 10.8 -> 0.83 ms.
//
// Several right-hand sides: column y = blockIdx.y has its own CTA, window and
// queue; the records of all columns come through L2.  b and x are column-
// contiguous (column y at + y * n).
#pragma once

#include "la_layout.h"
#include "tma.cuh"

namespace rbs {

template <typename VT>
struct LaArgs {
    const LaChunk *tab;
    const int2 *segs;  // first chunk, chunks
    int nseg;
    const unsigned char *rec;  // records of this precision
    const int *old;            // positions of old entries
    const VT *b;
    VT *x;
    long long n;  // elements from one column to the next
    int *queue;   // one counter per column, zero before the launch
    int *status;
    long long limit;
    LaDim d;
    int slots;
    int gather;  // 1 when the matrix has old entries
};

// Shared memory by 32-bit address (a pointer kept over the loop would be a
// generic one), in program order with the barriers.
__device__ __forceinline__ unsigned lds_u16(unsigned p) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(p));
    return v;
}
__device__ __forceinline__ int lds_s32(unsigned p) {
    int v;
    asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(p));
    return v;
}
__device__ __forceinline__ uint2 lds_2(unsigned p) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(p));
    return v;
}
__device__ __forceinline__ uint4 lds_4(unsigned p) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(p));
    return v;
}
__device__ __forceinline__ void lds_v(double &v, unsigned p) { asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(p)); }
__device__ __forceinline__ void lds_v(float &v, unsigned p) { asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(p)); }
__device__ __forceinline__ void lds_v2(double (&v)[2], unsigned p) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(p));
}
__device__ __forceinline__ void lds_v2(float (&v)[2], unsigned p) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "r"(p));
}
__device__ __forceinline__ void sts_v(unsigned p, double v) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(p), "d"(v) : "memory"); }
__device__ __forceinline__ void sts_v(unsigned p, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(p), "f"(v) : "memory"); }
// the first iteration at which a role ran out of records stands
__device__ __forceinline__ void la_give_up(unsigned p, int c) {
    asm volatile("red.shared.min.s32 [%0], %1;" ::"r"(p), "r"(c) : "memory");
}
__device__ __forceinline__ void la_bar(int threads) {
    __syncwarp();  // the barrier counts whole warps
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}
// bounded wait for a phase of the mbarrier at shared address p
__device__ __forceinline__ bool la_try(unsigned p, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(p), "r"(parity)
        : "memory");
    return ok != 0;
}
static __device__ __noinline__ bool la_wait_slow(unsigned p, unsigned parity, long long limit) {
    for (long long it = 0; it < limit; ++it)
        if (la_try(p, parity)) return true;
    return false;
}
__device__ __forceinline__ bool la_wait(unsigned p, unsigned parity, long long limit) {
    return la_try(p, parity) || la_wait_slow(p, parity, limit);
}

// FP32 records from the FP64 ones: the words copied, the values rounded.
// One CTA per chunk.
static __global__ void k_la_rec32(LaDim d, const unsigned char *__restrict__ r64, unsigned char *__restrict__ r32) {
    const unsigned char *s = r64 + (size_t)blockIdx.x * d.rec_bytes(8);
    unsigned char *t = r32 + (size_t)blockIdx.x * d.rec_bytes(4);
    for (int i = threadIdx.x; i < d.o_val() / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(t)[i] = reinterpret_cast<const uint4 *>(s)[i];
    const double *sv = reinterpret_cast<const double *>(s + d.o_val());
    float *dv = reinterpret_cast<float *>(t + d.o_val());
    for (int i = threadIdx.x; i < d.v_count(); i += blockDim.x) dv[i] = (float)sv[i];
}

template <typename VT, int Q>
__global__ void __launch_bounds__(1024, 1) k_tri_la(const __grid_constant__ LaArgs<VT> a) {
    extern __shared__ __align__(128) unsigned char sm[];
    constexpr unsigned E = sizeof(VT);
    const LaDim D = a.d;
    const unsigned mask = D.xw - 1;
    VT *xs = reinterpret_cast<VT *>(sm);
    unsigned long long *full = reinterpret_cast<unsigned long long *>(xs + D.s_zero() + 16);
    unsigned long long *empty = full + LA_SLOTS;
    int *oidx = reinterpret_cast<int *>(empty + LA_SLOTS);  // ring of 8 chunks' old positions
    unsigned char *ring = sm + D.fixed_bytes(E);
    __shared__ int s_seg, s_abort;
    const unsigned u_xs = smem_u32(xs), u_ring = smem_u32(ring), u_abort = smem_u32(&s_abort);
    const unsigned u_part = u_xs + E * D.s_part();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int M = D.nm >> 5, H = D.nh >> 5, S = a.slots;
    const int nbar = 32 * (M + H + a.gather);
    const unsigned slot_bytes = D.slot_bytes(E), rec_bytes = D.rec_bytes(E);
    const unsigned u_full = smem_u32(full), u_empty = smem_u32(empty), u_end = u_ring + S * slot_bytes;
    const VT *__restrict__ bcol = a.b + (long long)blockIdx.y * a.n;
    VT *__restrict__ xcol = a.x + (long long)blockIdx.y * a.n;
    if (tid == 0) xs[D.s_zero()] = VT(0);
    bool inited = false;
    for (;;) {
        __syncthreads();  // the previous segment is finished by every thread
        if (tid == 0) {
            s_seg = atomicAdd(a.queue + blockIdx.y, 1);
            s_abort = 0x7fffffff;  // chunk iteration at whose end the walk is given up
            if (s_seg < a.nseg) {
                for (int i = 0; i < S; ++i) {
                    if (inited) {
                        asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(full + i)) : "memory");
                        asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(empty + i)) : "memory");
                    }
                    mbar_init(full + i, 1);
                    mbar_init(empty + i, 1);
                }
                fence_mbar_init();
            }
        }
        __syncthreads();
        if (s_seg >= a.nseg) break;
        inited = true;
        const int2 sd = a.segs[s_seg];
        const int nch = sd.y;
        const LaChunk *tab = a.tab + sd.x;
        volatile int *abt = &s_abort;
        bool stop = false;
        int issued = 0;  // producer: records asked for

        if (warp == M + H + a.gather) {
            // ---------------- producer ----------------
            const LaChunk none{0, 0, 0, 0};
            const unsigned char *rec = a.rec + (size_t)sd.x * rec_bytes;
            // lane l holds table entry base + l, the next 32 are on their way
            int base = 0, slot = 0;
            unsigned par = 1;  // of the free barrier: the first pass finds every slot free
            LaChunk cur = lane < nch ? tab[lane] : none, nxw = 32 + lane < nch ? tab[32 + lane] : none;
            for (int j = 0; j < nch && !stop; ++j) {
                if (j - base >= 32) {
                    base += 32;
                    cur = nxw;
                    nxw = base + 32 + lane < nch ? tab[base + 32 + lane] : none;
                }
                long long it = 0;
                while (!mbar_try_wait(empty + slot, par))
                    if (*abt != 0x7fffffff || ++it > a.limit) {
                        stop = true;
                        break;
                    }
                stop = __any_sync(0xffffffffu, stop);
                if (stop) break;
                if (lane == j - base) {
                    unsigned char *sl = ring + (unsigned)slot * slot_bytes;
                    const void *bs;
                    int delta;
                    const unsigned bb = bulk_window(bcol + cur.lo, cur.nr, (int)sizeof(VT), bs, delta);
                    mbar_arrive_expect_tx(full + slot, rec_bytes + bb);
                    bulk_g2s(sl, rec + (size_t)j * rec_bytes, rec_bytes, full + slot);
                    bulk_g2s(sl + rec_bytes, bs, bb, full + slot);
                }
                ++issued;
                if (++slot == S) {
                    slot = 0;
                    par ^= 1;
                }
            }
            // a producer that gave up only stops: the roles that meet at the
            // barrier run out of records, and give up together
        } else if (warp < M) {
            // ---------------- main: one thread per row ----------------
            const int t = tid;
            unsigned sl = u_ring, mb = u_full, par = 0;  // the next chunk's slot, its mbarrier and phase
            uint4 d{};           // the chunk's header
            uint2 w{};           // this row's words
            unsigned xo = 0;     // its record's extra slots
            VT v01[2] = {}, v2i[2] = {}, bv = 0;  // term values, inverse diagonal, right-hand side
            const unsigned ow = D.o_main + 8 * t, ov = D.o_val() + E * LaDim::v_main(t, 0), ob = rec_bytes + E * t;
            const unsigned oe = D.o_extra(), oev = D.o_val() + E * D.v_extra() - D.o_extra();
            const unsigned b0 = (unsigned)(unsigned long long)bcol;
            unsigned ps = u_part + E * t, pd = E * D.nh;  // this row's sum, in two buffers in turn
            auto load = [&]() {
                if (!la_wait(mb, par, a.limit)) {
                    d.z = w.x = w.y = 0;
                    return false;
                }
                d = lds_4(sl);
                w = lds_2(sl + ow);
                lds_v2(v01, sl + ov);
                lds_v2(v2i, sl + ov + 64 * E);
                lds_v(bv, sl + ob + ((b0 + E * d.x) & 15u));
                xo = sl + oe;
                sl += slot_bytes;
                mb += 8;
                if (sl == u_end) {
                    sl = u_ring;
                    mb = u_full;
                    par ^= 1;
                }
                return true;
            };
            auto solve = [&]() {
                // slots become addresses here: before the barrier that would
                // wait for their words (4M-row band factor 16.2 -> 21.5 ms)
                VT sum, x0, x1, x2;
                lds_v(x0, u_xs + E * (w.x & 0xffffu));
                lds_v(x1, u_xs + E * (w.x >> 16));
                lds_v(x2, u_xs + E * (w.y & 0xffffu));
                lds_v(sum, ps);
                ps += pd;
                pd = 0u - pd;
                sum += v01[0] * x0;
                sum += v01[1] * x1;
                sum += v2i[0] * x2;
                if (w.y & 0x1f0000u) {
                    const unsigned k0 = w.y >> 21, k1 = k0 + ((w.y >> 16) & 31u);
                    for (unsigned k = k0; k < k1; ++k) {
                        VT v, xv;
                        lds_v(v, xo + oev + E * k);
                        lds_v(xv, u_xs + E * lds_u16(xo + 2 * k));
                        sum += v * xv;
                    }
                }
                const VT xv = (bv - sum) * v2i[1];
                if (t < (int)d.z) {
                    sts_v(u_xs + E * ((d.y + t) & mask), xv);
                    xcol[(int)d.x + t] = xv;
                }
            };
            if (!load()) la_give_up(u_abort, -1);
            la_bar(nbar);  // sums of chunk 0
            int ab = lds_s32(u_abort);
            stop = ab < 0;
            for (int c = 0; c < nch && !stop; ++c) {
                solve();
                if (c + 1 < nch && !load()) la_give_up(u_abort, c);
                stop = ab < c;  // read after the last barrier: the same for every thread
                la_bar(nbar);
                ab = lds_s32(u_abort);
            }
        } else if (warp < M + H) {
            // ---------------- helpers: early sums one chunk ahead ----------------
            const int h = tid - D.nm;
            unsigned sl = u_ring, mb = u_full, par = 0;
            uint2 e[Q / 4] = {};
            VT u[Q / 2][2] = {};
            const unsigned oh = D.o_help() + 2 * D.w_help(h, 0), ov = D.o_val() + E * D.v_help(h, 0);
            unsigned ps = u_part + E * h, pd = E * D.nh;
            auto load = [&]() {
                if (!la_wait(mb, par, a.limit)) {
#pragma unroll
                    for (int k = 0; k < Q / 4; ++k) e[k] = make_uint2(0, 0);
                    return false;
                }
#pragma unroll
                for (int k = 0; k < Q / 4; ++k) e[k] = lds_2(sl + oh + 256 * k);
#pragma unroll
                for (int k = 0; k < Q / 2; ++k) lds_v2(u[k], sl + ov + 64 * E * k);
                sl += slot_bytes;
                mb += 8;
                if (sl == u_end) {
                    sl = u_ring;
                    mb = u_full;
                    par ^= 1;
                }
                return true;
            };
            auto sums = [&]() {
                VT x[Q];
#pragma unroll
                for (int k = 0; k < Q / 4; ++k) {
                    lds_v(x[4 * k], u_xs + E * (e[k].x & 0xffffu));
                    lds_v(x[4 * k + 1], u_xs + E * (e[k].x >> 16));
                    lds_v(x[4 * k + 2], u_xs + E * (e[k].y & 0xffffu));
                    lds_v(x[4 * k + 3], u_xs + E * (e[k].y >> 16));
                }
                VT s0 = u[0][0] * x[0], s1 = u[0][1] * x[1];
#pragma unroll
                for (int k = 1; k < Q / 2; ++k) {
                    s0 += u[k][0] * x[2 * k];
                    s1 += u[k][1] * x[2 * k + 1];
                }
                sts_v(ps, s0 + s1);
                ps += pd;
                pd = 0u - pd;
            };
            bool ok = load();
            if (ok) {
                sums();
                if (1 < nch) ok = load();
            }
            if (!ok) la_give_up(u_abort, -1);
            la_bar(nbar);  // sums of chunk 0
            int ab = lds_s32(u_abort);
            stop = ab < 0;
            unsigned fb = u_empty;
            const bool frees = h == 0;
            for (int c = 0; c < nch && !stop; ++c) {
                if (c + 1 < nch) sums();
                if (c + 2 < nch && !load()) la_give_up(u_abort, c);
                stop = ab < c;
                la_bar(nbar);
                ab = lds_s32(u_abort);
                if (frees) {  // chunk c's slot is free
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(fb) : "memory");
                    fb += 8;
                    if (fb == u_empty + 8 * S) fb = u_empty;
                }
            }
        } else {
            // ---------------- gather: values of rows that left the window ----------------
            // lane l: counts of chunks base + l and base + 32 + l; fi, fv: entries
            // before the next chunk of either stage
            const int o0 = tab[0].ooff;
            int base = 0, fi = 0, fv = 0;
            auto entry = [&](int j) { return j < nch ? tab[j].on : 0; };
            int cur = entry(lane), nxw = entry(32 + lane);
            auto get = [&](int j) {  // j in [base, base + 64)
                return __shfl_sync(0xffffffffu, j - base < 32 ? cur : nxw, (j - base) & 31);
            };
            const unsigned u_idx = smem_u32(oidx);
            auto idx_stage = [&](int j) {
                const int cnt = get(j);
                for (int i = lane; i < cnt; i += 32)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(u_idx + 4 * ((j & 7) * LA_OLD + i)),
                                 "l"(a.old + o0 + fi + i)
                                 : "memory");
                fi += cnt;
            };
            auto val_stage = [&](int j) {
                const int cnt = get(j);
                for (int i = lane; i < cnt; i += 32) {
                    const VT *src = xcol + lds_s32(u_idx + 4 * ((j & 7) * LA_OLD + i));
                    const unsigned dst = u_xs + E * (D.xw + ((fv + i) & (LA_AUX - 1)));
                    if (sizeof(VT) == 8)
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
                    else
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
                }
                fv += cnt;
            };
            // chunks below LA_AHEAD + 1 have none (their segment is younger than the window)
            for (int j = 0; j < LA_IDX; ++j) idx_stage(j);
            for (int j = 0; j < LA_AHEAD; ++j) fv += get(j);  // none
            asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;" ::: "memory");
            la_bar(nbar);  // partials of chunk 0
            int ab = lds_s32(u_abort);
            stop = ab < 0;
            for (int c = 0; c < nch && !stop; ++c) {
                // base <= c + LA_AHEAD, c + LA_IDX < base + 64
                if (c + LA_AHEAD - base >= 32) {
                    base += 32;
                    cur = nxw;
                    nxw = entry(base + 32 + lane);
                }
                idx_stage(c + LA_IDX);
                val_stage(c + LA_AHEAD);
                // the copies of iteration c - 3 have landed: chunk c + 2's values
                asm volatile("cp.async.commit_group;\n cp.async.wait_group 3;" ::: "memory");
                __syncwarp();
                stop = ab < c;
                la_bar(nbar);
                ab = lds_s32(u_abort);
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        if (__syncthreads_or(stop)) {
            // given up: every copy in flight lands before the CTA exits (bounded)
            if (warp == M + H + a.gather && lane == 0) {
                atomicOr(a.status, RBS_STATUS_TIMEOUT);
                for (int j = issued > S ? issued - S : 0; j < issued; ++j)
                    la_wait(u_full + 8 * (j % S), (unsigned)((j / S) & 1), a.limit);
            }
            __syncthreads();
            return;
        }
    }
}

}  // namespace rbs
