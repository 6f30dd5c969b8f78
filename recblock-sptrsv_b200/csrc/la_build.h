// la_build.h -- host builder of the look-ahead level layout (la_layout.h),
// part of analysis.cpp.
#pragma once

#include <algorithm>
#include <atomic>
#include <climits>
#include <cstring>
#include <numeric>
#include <vector>

#include "la_layout.h"
#include "rbs_internal.h"

namespace rbs {

bool la_build(const Plan &P, LaHost &H) {
    H = LaHost{};
    const int n = P.n;
    if (n < 1 || (int)P.perm.size() != n || (int)P.full_rp.size() != n + 1 || P.bfs_ptr.size() < 2) return false;
    const int *rp = P.full_rp.data(), *col = P.full_col.data();
    const double *val = P.full_val.data();

    // segments: (segment, level) ranges in level order; a segment's rows of
    // one level are contiguous positions (the level search keeps the order
    // of its queue), checked here
    struct Range { int seg, lo, hi; };
    std::vector<Range> ranges;
    int nseg = 1;
    if (P.seg_rows.empty()) {
        for (size_t l = 0; l + 1 < P.bfs_ptr.size(); ++l) ranges.push_back({0, P.bfs_ptr[l], P.bfs_ptr[l + 1]});
    } else {
        nseg = (int)P.seg_rows.size();
        std::vector<int> seg((size_t)n);
        constexpr int kRows = 1 << 14;
        parallel_for(((size_t)n + kRows - 1) / kRows, [&](size_t ch) {
            for (int p = (int)ch * kRows; p < std::min(n, (int)ch * kRows + kRows); ++p)
                seg[(size_t)p] = (int)(std::upper_bound(P.seg_rows.begin(), P.seg_rows.end(), P.perm[(size_t)p]) -
                                       P.seg_rows.begin()) - 1;
        });
        std::vector<int> seen((size_t)nseg, -1);
        for (size_t l = 0; l + 1 < P.bfs_ptr.size(); ++l)
            for (int a = P.bfs_ptr[l]; a < P.bfs_ptr[l + 1];) {
                int b = a + 1;
                while (b < P.bfs_ptr[l + 1] && seg[(size_t)b] == seg[(size_t)a]) ++b;
                const int s = seg[(size_t)a];
                if (s < 0 || s >= nseg || seen[(size_t)s] == (int)l) return false;
                seen[(size_t)s] = (int)l;
                ranges.push_back({s, a, b});
                a = b;
            }
        std::stable_sort(ranges.begin(), ranges.end(), [](const Range &x, const Range &y) { return x.seg < y.seg; });
    }

    // lines per helper thread: the fewest that take most rows' early entries
    // (two entries of a row are late on average); threads for an ordinary
    // level's rows
    LaDim &D = H.dim;
    {
        std::vector<long long> hist(64, 0);
        for (int p = 0; p < n; ++p) hist[(size_t)std::min(63, rp[p + 1] - rp[p] - 1)]++;
        auto above = [&](int len) {
            long long s = 0;
            for (int i = len + 1; i < 64; ++i) s += hist[(size_t)i];
            return s;
        };
        D.q = 8 * above(5) <= n ? 4 : 2 * above(10) <= n ? 8 : 12;
        long long groups = 0;
        for (int i = 0; i < 64; ++i) groups += hist[(size_t)i] * std::max(1, (i - 2 + D.q - 1) / D.q);
        const double rows = (double)n / (double)ranges.size(), per = (double)groups / (double)n;
        D.xw = LA_XW_MAX;
        D.nx = 32;
        for (int m = std::max(1, std::min(LA_RMAX / 32, (int)((rows * 1.25 + 31) / 32)));; --m) {
            D.nm = 32 * m;
            D.nh = 32 * std::max(m, std::min(16, (int)((std::min(rows * 1.25, 32.0 * m) * per + 31) / 32)));
            // eight records in the ring: fewer and larger chunks were no faster
            // (4M-row band factor, levels of 173 rows: 128-row chunks 15.0 ms,
            // 192-row chunks with five records 16.3 ms)
            if (m == 1 || (D.slots(8) >= 8 && D.nm + D.nh <= LA_THREADS)) break;
        }
        D.xw = D.nx = 0;
    }
    const int Q = D.q, NM = D.nm, NH = D.nh;

    // chunks, segment after segment
    struct Ch { int lo, nr, v0, seg, prev_lo; };  // prev_lo: first position of the chunk before, -1 for a first one
    std::vector<Ch> ch;
    std::vector<int> seg_first((size_t)nseg + 1, 0);
    std::vector<int> vrow;  // position -> virtual row (identity for one segment)
    if (nseg > 1) vrow.resize((size_t)n);
    {
        std::vector<size_t> range0((size_t)nseg + 1, ranges.size());  // first range of every segment
        for (size_t i = ranges.size(); i-- > 0;) range0[(size_t)ranges[i].seg] = i;
        for (size_t q = (size_t)nseg; q-- > 0;) range0[q] = std::min(range0[q], range0[q + 1]);
        std::vector<std::vector<Ch>> parts((size_t)nseg);
        std::atomic<bool> ok{true};
        parallel_for((size_t)nseg, [&](size_t q) {  // segments on host threads
            int v0 = 0, prev = -1;
            for (size_t i = range0[q]; i < range0[q + 1] && ok; ++i) {
                const Range &g = ranges[i];
                for (int a = g.lo; a < g.hi;) {
                    int nr = 0, used = 0;
                    while (a + nr < g.hi && nr < NM) {
                        const int p = a + nr;
                        int e = rp[p + 1] - rp[p] - 1;  // early entries: columns ascend, the late ones are at the end
                        for (int k = rp[p + 1] - 1; prev >= 0 && k >= rp[p] && col[k] >= prev; --k) e -= col[k] != p;
                        const int need = std::max(1, (e + Q - 1) / Q);
                        if (need > NH || need > 24) {  // a long row: another kernel's work
                            ok = false;
                            return;
                        }
                        if (used + need > NH) break;
                        used += need;
                        ++nr;
                    }
                    parts[q].push_back({a, nr, v0, g.seg, prev});
                    if (nseg > 1)
                        for (int t = 0; t < nr; ++t) vrow[(size_t)(a + t)] = v0 + t;
                    prev = a;
                    v0 += nr;
                    a += nr;
                }
            }
        });
        if (!ok) return false;
        for (int q = 0; q < nseg; ++q) seg_first[(size_t)q + 1] = seg_first[(size_t)q] + (int)parts[(size_t)q].size();
        ch.reserve((size_t)seg_first[(size_t)nseg]);
        for (const auto &v : parts) ch.insert(ch.end(), v.begin(), v.end());
    }
    const size_t nch = ch.size();
    if (nch == 0 || (double)nch * D.rec_bytes(8) > la_most_bytes(rp[n], n)) return false;
    auto vr = [&](int q) { return nseg > 1 ? vrow[(size_t)q] : q; };

    // window size: the smallest that leaves few entries outside
    constexpr int kNw = 3;  // LA_XW_MIN << i
    std::vector<long long> outside(kNw, 0);
    {
        std::vector<std::vector<long long>> part((nch + 255) / 256, std::vector<long long>(kNw, 0));
        parallel_for(part.size(), [&](size_t g) {
            long long beyond[kNw] = {};  // (a row's own entry is within every window)
            for (size_t c = g * 256; c < std::min(nch, g * 256 + 256); ++c) {
                const Ch &C = ch[c];
                for (int k = rp[C.lo]; k < rp[C.lo + C.nr]; ++k) {
                    const int d = C.v0 + C.nr - vr(col[k]);
                    for (int w = 0; w < kNw; ++w) beyond[w] += d > (LA_XW_MIN << w);
                }
            }
            std::copy(beyond, beyond + kNw, part[g].begin());
        });
        for (const auto &v : part)
            for (int w = 0; w < kNw; ++w) outside[(size_t)w] += v[(size_t)w];
    }
    const long long off = (long long)rp[n] - n;
    int wsel = kNw - 1;
    for (int w = 0; w < kNw; ++w)
        if (outside[(size_t)w] * 200 <= off) {
            wsel = w;
            break;
        }
    if (outside[(size_t)wsel] * 20 > off) return false;  // scattered dependencies: another kernel's work
    const int xw = LA_XW_MIN << wsel;
    D.xw = xw;

    // per-chunk split of the entries: count pass, offsets, fill pass
    H.tab.resize(nch);
    auto kind = [&](const Ch &C, int q) {  // 0 late, 1 early, 2 old
        if (C.prev_lo >= 0 && q >= C.prev_lo) return 0;
        return vr(q) < C.v0 + C.nr - xw ? 2 : 1;
    };
    constexpr size_t kGroup = 64;
    const size_t ngrp = (nch + kGroup - 1) / kGroup;
    std::vector<int> extra(nch, 0);
    std::atomic<bool> ok{true};
    parallel_for(ngrp, [&](size_t g) {
        for (size_t c = g * kGroup; c < std::min(nch, (g + 1) * kGroup); ++c) {
            const Ch &C = ch[c];
            int nold = 0;
            for (int p = C.lo; p < C.lo + C.nr; ++p) {
                int late = 0, early = 0;
                for (int k = rp[p]; k < rp[p + 1]; ++k) {
                    if (col[k] == p) continue;
                    const int kd = kind(C, col[k]);
                    if (kd == 0) ++late;
                    else ++early;
                    nold += kd == 2;
                }
                const int x = std::max(0, late + std::max(0, (early + Q - 1) / Q - 1) - LA_LATE);
                if (x > 31) ok = false;
                extra[c] += x;
            }
            H.tab[c] = LaChunk{C.lo, C.nr, 0, nold};
            if (nold > LA_OLD || extra[c] > 2000) ok = false;
        }
    });
    if (!ok) return false;
    long long oo = 0;
    for (size_t c = 0; c < nch; ++c) {
        H.tab[c].ooff = (int)oo;
        oo += H.tab[c].on;
        D.nx = std::max(D.nx, (extra[c] + 7) / 8 * 8);
    }
    if (oo > INT_MAX - 65536 || D.slots(8) < LA_SLOTS_MIN) return false;
    if ((double)nch * D.rec_bytes(8) > la_most_bytes(rp[n], n)) return false;  // with the extra terms
    const size_t recw = (size_t)D.rec_bytes(8) / 4;
    H.rec.resize(nch * recw);
    H.old.resize((size_t)oo);

    parallel_for(ngrp, [&](size_t g) {
        for (size_t c = g * kGroup; c < std::min(nch, (g + 1) * kGroup); ++c) {
            const Ch &C = ch[c];
            const LaChunk &T = H.tab[c];
            unsigned char *rec = reinterpret_cast<unsigned char *>(H.rec.data() + c * recw);
            uint16_t *mw = reinterpret_cast<uint16_t *>(rec + D.o_main), *hs = reinterpret_cast<uint16_t *>(rec + D.o_help()),
                     *xsl = reinterpret_cast<uint16_t *>(rec + D.o_extra());
            double *v = reinterpret_cast<double *>(rec + D.o_val()), *xv = v + D.v_extra();
            const int hdr[4] = {C.lo, C.v0 & (xw - 1), C.nr, 0};
            std::memcpy(rec, hdr, 16);
            const uint16_t zero = (uint16_t)D.s_zero();
            for (int t = 0; t < NM; ++t) {
                mw[4 * t] = mw[4 * t + 1] = mw[4 * t + 2] = zero;
                mw[4 * t + 3] = 0;
            }
            std::fill(hs, hs + (size_t)Q * NH, zero);
            std::fill(xsl, xsl + D.nx, zero);
            std::fill(v, v + D.v_count(), 0.0);
            const int buf = (int)((c - (size_t)seg_first[(size_t)C.seg]) & 1);
            const int o0 = H.tab[(size_t)seg_first[(size_t)C.seg]].ooff;
            int nx = 0, no = 0, next = C.nr;  // next: the first helper thread without a row
            for (int t = 0; t < C.nr; ++t) {
                const int p = C.lo + t;
                int terms = 0, early = 0, h = t;
                const int x0 = nx;
                auto term = [&](int slot, double value) {
                    if (terms < LA_LATE) {
                        mw[4 * t + terms] = (uint16_t)slot;
                        v[LaDim::v_main(t, terms)] = value;
                    } else {
                        xsl[nx] = (uint16_t)slot;
                        xv[nx++] = value;
                    }
                    ++terms;
                };
                for (int k = rp[p]; k < rp[p + 1]; ++k) {
                    if (col[k] == p) continue;
                    const int kd = kind(C, col[k]);
                    if (kd == 0) {
                        term(vr(col[k]) & (xw - 1), val[k]);
                        continue;
                    }
                    const int q = early % Q;
                    if (early && q == 0) {
                        h = next++;
                        term(D.s_part() + buf * NH + h, 1.0);
                    }
                    int slot = vr(col[k]) & (xw - 1);
                    if (kd == 2) {
                        H.old[(size_t)(T.ooff + no)] = col[k];
                        slot = xw + ((T.ooff - o0 + no) & (LA_AUX - 1));
                        ++no;
                    }
                    hs[D.w_help(h, q)] = (uint16_t)slot;
                    v[D.v_help(h, q)] = val[k];
                    ++early;
                }
                mw[4 * t + 3] = (uint16_t)(x0 << 5 | (nx - x0));
                v[LaDim::v_main(t, 3)] = P.inv_diag[(size_t)p];
            }
        }
    });

    // segments in order of decreasing work (the kernel's queue)
    std::vector<int> order((size_t)nseg);
    std::iota(order.begin(), order.end(), 0);
    std::vector<long long> wk((size_t)nseg);
    for (int s = 0; s < nseg; ++s) wk[(size_t)s] = seg_first[(size_t)s + 1] - seg_first[(size_t)s];
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return wk[(size_t)a] > wk[(size_t)b]; });
    for (int s : order)
        if (seg_first[(size_t)s + 1] > seg_first[(size_t)s])
            H.segs.insert(H.segs.end(), {seg_first[(size_t)s], seg_first[(size_t)s + 1] - seg_first[(size_t)s]});
    H.ok = true;
    return true;
}

}  // namespace rbs
