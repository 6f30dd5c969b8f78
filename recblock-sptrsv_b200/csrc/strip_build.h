// strip_build.h -- host builder of the strip layout (strip_layout.h), part of
// analysis.cpp.
#pragma once

#include <algorithm>
#include <atomic>
#include <climits>
#include <cstring>
#include <vector>

#include "rbs_internal.h"
#include "strip_layout.h"

namespace rbs {

bool strip_build(const Plan &P, StripHost &H) {
    H = StripHost{};
    const int n = P.n;
    if (n < 1 || (int)P.perm.size() != n || (int)P.full_rp.size() != n + 1 || P.bfs_ptr.size() < 2) return false;
    const int *rp = P.full_rp.data(), *col = P.full_col.data();
    const double *val = P.full_val.data();

    // chains: a row continues the latest chain among its dependencies, or,
    // when that chain already has a row in this level (or there are no
    // dependencies), opens a new one; many more chains than an average level
    // has rows means that there are none to speak of
    const int nlev = (int)P.bfs_ptr.size() - 1;
    const long long most = std::min<long long>(32 * 4096, 64 + 16LL * n / std::max(1, nlev));
    // The rows of a level in either order: of two rows that could continue a
    // chain the first does, so on a grid one order makes chains of its rows
    // and the other of its columns; the one with fewer chains is kept.
    std::vector<int> chain, last;  // last: level of a chain's latest row
    int wmax = 0;
    for (int p = 0; p < n; ++p) wmax = std::max(wmax, rp[p + 1] - rp[p] - 1);
    if (wmax > 4) return false;
    {
        std::vector<int> ch[2], lt[2];
        parallel_for(2, [&](size_t back) {
            std::vector<int> &c = ch[back], &t = lt[back];
            c.resize((size_t)n);
            for (int l = 0; l < nlev; ++l) {
                const int lo = P.bfs_ptr[(size_t)l], hi = P.bfs_ptr[(size_t)l + 1];
                for (int i = lo; i < hi; ++i) {
                    const int p = back ? hi - 1 - (i - lo) : i;
                    int m = -1;
                    for (int k = rp[p]; k < rp[p + 1]; ++k)
                        if (col[k] != p) m = std::max(m, c[(size_t)col[k]]);
                    if (m < 0 || t[(size_t)m] == l) {
                        m = (int)t.size();
                        if (m >= most) {
                            c.clear();
                            return;
                        }
                        t.push_back(l);
                    }
                    c[(size_t)p] = m;
                    t[(size_t)m] = l;
                }
            }
        });
        // Of two orders with as many chains, the one that puts neighbouring
        // original rows into neighbouring lanes: a row of a grid across the
        // lanes keeps a strip's part of the caller's vectors in pieces of 256
        // bytes (1M-row grid, 32 columns: 505 us, the other way 727 us).
        long long across[2] = {0, 0};
        if (!ch[0].empty() && !ch[1].empty() && lt[0].size() == lt[1].size()) {
            std::vector<int> place((size_t)n);
            for (int p = 0; p < n; ++p) place[(size_t)P.perm[(size_t)p]] = p;
            for (int back = 0; back < 2; ++back)
                for (int o = 0; o + 1 < n; o += 61)  // a sample
                    across[back] += std::abs(ch[back][(size_t)place[(size_t)o]] - ch[back][(size_t)place[(size_t)o + 1]]) == 1;
        }
        const int keep = ch[0].empty() || (!ch[1].empty() && (lt[1].size() < lt[0].size() ||
                                                              (lt[1].size() == lt[0].size() && across[1] > across[0])));
        chain.swap(ch[keep]);
        last.swap(lt[keep]);
    }
    if (chain.empty()) return false;
    const int W = H.w = wmax <= 2 ? 2 : 4;
    const int nstrip = ((int)last.size() + 31) / 32;

    // steps: the levels in which a strip has a row
    std::vector<int> steps((size_t)nstrip, 0), lastl((size_t)nstrip, -1);
    std::vector<int> pos((size_t)n);  // step * 32 + lane, then the position
    for (int l = 0; l < nlev; ++l)
        for (int p = P.bfs_ptr[(size_t)l]; p < P.bfs_ptr[(size_t)l + 1]; ++p) {
            const size_t s = (size_t)chain[(size_t)p] >> 5;
            if (lastl[s] != l) {
                lastl[s] = l;
                ++steps[s];
            }
            pos[(size_t)p] = (steps[s] - 1) * 32 + (chain[(size_t)p] & 31);
        }
    // Idle steps at the start of a strip, 0 to 7, so that its chunks end where
    // the values they need become available: a chunk can start when the
    // chunks that publish its remote values have ended, so each strip takes
    // the shift with the earliest estimated end (in steps; kHop for the way
    // of a value from one strip to another).
    std::vector<int> shift((size_t)nstrip, 0);
    {
        constexpr int kHop = 10;
        std::vector<std::vector<int>> rowsof((size_t)nstrip);
        for (int p = 0; p < n; ++p) rowsof[(size_t)chain[(size_t)p] >> 5].push_back(p);
        std::vector<std::vector<int>> end((size_t)nstrip);  // estimated end of every chunk
        for (size_t s = 0; s < (size_t)nstrip; ++s) {
            // latest remote end per step
            std::vector<int> need((size_t)steps[s], 0);
            for (int p : rowsof[s])
                for (int e = rp[p]; e < rp[p + 1]; ++e) {
                    const size_t q = (size_t)col[e], t = (size_t)chain[q] >> 5;
                    if (t == s) continue;
                    int &d = need[(size_t)pos[(size_t)p] / 32];
                    d = std::max(d, end[t][(size_t)(shift[t] + pos[q] / 32) / ST_STEPS] + kHop);
                }
            int best = INT_MAX;
            for (int sh = 0; sh < ST_STEPS; ++sh) {
                const int nc = (sh + steps[s] + ST_STEPS - 1) / ST_STEPS;
                std::vector<int> f((size_t)nc);
                int t = 0;
                for (int c = 0; c < nc; ++c) {
                    for (int st = std::max(0, c * ST_STEPS - sh); st < std::min(steps[s], (c + 1) * ST_STEPS - sh); ++st)
                        t = std::max(t, need[(size_t)st]);
                    f[(size_t)c] = t += ST_STEPS;
                }
                if (t < best) {
                    best = t;
                    shift[s] = sh;
                    end[s].swap(f);
                }
            }
        }
        for (int p = 0; p < n; ++p) pos[(size_t)p] += 32 * shift[(size_t)chain[(size_t)p] >> 5];
        for (int s = 0; s < nstrip; ++s) steps[(size_t)s] += shift[(size_t)s];
    }
    H.first.assign((size_t)nstrip + 1, 0);
    for (int s = 0; s < nstrip; ++s) H.first[(size_t)s + 1] = H.first[(size_t)s] + (steps[(size_t)s] + ST_STEPS - 1) / ST_STEPS;
    const long long nch = H.first[(size_t)nstrip];
    // at least a quarter of the positions hold rows (the last strip of a
    // small grid may have few chains)
    if (nch * ST_ROWS > 4LL * n + 32 * ST_ROWS || nch * ST_ROWS > INT_MAX / 2) return false;
    H.rows = (int)(nch * ST_ROWS);
    for (int p = 0; p < n; ++p) pos[(size_t)p] += H.first[(size_t)chain[(size_t)p] >> 5] * ST_ROWS;
    H.perm.assign((size_t)H.rows, -1);  // position -> processing position
    for (int p = 0; p < n; ++p) H.perm[(size_t)pos[(size_t)p]] = p;

    // published rows: read by another strip, or by their own after ST_WIN steps
    auto strip_of = [&](int p) { return chain[(size_t)p] >> 5; };
    auto step_of = [&](int p) {
        const int q = pos[(size_t)p];
        return (q / ST_ROWS - H.first[(size_t)strip_of(p)]) * ST_STEPS + q % ST_ROWS / 32;
    };
    auto local = [&](int p, int d) {  // row p reads row d from its strip's window
        return strip_of(p) == strip_of(d) && step_of(p) - step_of(d) < ST_WIN;
    };
    std::vector<char> pub((size_t)n, 0);
    constexpr int kRows = 1 << 14;
    parallel_for(((size_t)n + kRows - 1) / kRows, [&](size_t g) {
        for (int p = (int)g * kRows; p < std::min(n, (int)g * kRows + kRows); ++p)
            for (int e = rp[p]; e < rp[p + 1]; ++e)
                if (col[e] != p && !local(p, col[e])) __atomic_store_n(&pub[(size_t)col[e]], (char)1, __ATOMIC_RELAXED);
    });
    std::vector<int> number((size_t)n, -1);
    std::vector<int> pub0((size_t)nch + 1, 0);  // first published number of every chunk
    for (long long c = 0; c < nch; ++c) {
        pub0[(size_t)c] = H.published;
        for (int i = 0; i < ST_ROWS; ++i) {
            const int p = H.perm[(size_t)c * ST_ROWS + i];
            if (p >= 0 && pub[(size_t)p]) number[(size_t)p] = H.published++;
        }
        if (H.published - pub0[(size_t)c] > ST_PUB) return false;
    }
    pub0[(size_t)nch] = H.published;

    const size_t recw = (size_t)st_rec_bytes(W, 8) / 4;
    H.rec.resize((size_t)nch * recw);
    H.rows_sorted.resize((size_t)H.rows);
    H.rows_at.resize((size_t)H.rows);
    std::atomic<bool> ok{true};
    parallel_for((size_t)nstrip, [&](size_t s) {
        std::vector<std::pair<int, int>> order((size_t)ST_ROWS);
        for (int c = H.first[s]; c < H.first[s + 1]; ++c) {
            unsigned char *rec = reinterpret_cast<unsigned char *>(H.rec.data() + (size_t)c * recw);
            int *rem = reinterpret_cast<int *>(rec);
            uint16_t *words = reinterpret_cast<uint16_t *>(rec);
            double *v = reinterpret_cast<double *>(rec + 2 * st_words(W));
            std::fill(rem, rem + 32, -1);
            rem[32] = pub0[(size_t)c];
            rem[33] = pub0[(size_t)c + 1] - pub0[(size_t)c];
            rem[34] = rem[35] = 0;
            std::fill(words + 72, words + ST_HEAD, (uint16_t)0);
            std::fill(words + ST_HEAD, words + st_words(W), (uint16_t)ST_ZERO);
            std::fill(v, v + st_values(W), 0.0);
            const int k0 = c - H.first[s];  // chunk of the strip
            int nrem = 0, npub = 0;
            for (int st = 0; st < ST_STEPS; ++st)
                for (int lane = 0; lane < 32; ++lane) {
                    const int at = st * 32 + lane, p = H.perm[(size_t)c * ST_ROWS + at];
                    order[(size_t)at] = {p < 0 ? INT_MAX : P.perm[(size_t)p], at};
                    if (p < 0) continue;
                    if (number[(size_t)p] >= 0) words[72 + npub++] = (uint16_t)at;
                    int k = 0;
                    for (int e = rp[p]; e < rp[p + 1]; ++e) {
                        const int d = col[e];
                        if (d == p) continue;
                        int slot;
                        if (local(p, d)) {
                            slot = (step_of(d) % ST_WIN) * 32 + pos[(size_t)d] % 32;
                        } else {
                            const int q = number[(size_t)d];
                            int i = 0;
                            while (i < nrem && rem[i] != q) ++i;
                            if (i == 32) {
                                ok = false;
                                return;
                            }
                            if (i == nrem) rem[nrem++] = q;
                            slot = ST_REM + (k0 & 1) * 32 + i;
                        }
                        words[st_w_slot(W, st, lane, k)] = (uint16_t)slot;
                        v[st_v_val(W, st, lane, k)] = val[e];
                        ++k;
                    }
                    v[st_v_inv(W, st, lane)] = P.inv_diag[(size_t)p];
                }
            std::sort(order.begin(), order.end());
            for (int i = 0; i < ST_ROWS; ++i) {
                const size_t o = (size_t)c * ST_ROWS + (size_t)(i % 32 * 8 + i / 32);  // a lane's eight side by side
                H.rows_sorted[o] = order[(size_t)i].first == INT_MAX ? -1 : order[(size_t)i].first;
                H.rows_at[o] = (unsigned char)order[(size_t)i].second;
            }
        }
    });
    H.ok = ok;
    return ok;
}

}  // namespace rbs
