// tile_plan.cpp — see tile_plan.h.
//
// A tile is a compact block of a model's rows, so that most of its rows read
// only its own rows.  A mesh numbered row by row (a grid cloth) is cut into
// rectangles of its logical grid; any other mesh by recursive bisection of its
// rest positions.
#include "tile_plan.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <exception>
#include <new>
#include <numeric>
#include <thread>
#include <unordered_map>

namespace pdipc {

namespace {

constexpr int kLanes = 32;

struct Model {
    int lo, hi;      // rows
    int stride = 0;  // row length of a mesh numbered as a grid, else 0
};

// The logical row length of a mesh numbered row by row: the most frequent
// column distance above one among its stencils, if nearly every stencil entry
// then lies within one step in both grid directions; else 0.
int grid_stride(const HostTables& H, int lo, int hi) {
    std::unordered_map<int, int> freq;
    int64_t total = 0;
    const int step = std::max(1, (hi - lo) / 4096);  // a sample of the rows
    for (int i = lo; i < hi; i += step)
        for (int e = H.lPtr[i] + 1; e < H.lPtr[i + 1]; ++e) {
            ++freq[std::abs(H.lNbr[e] - i)];
            ++total;
        }
    int s = 0, best = 0;
    for (auto& kv : freq)
        if (kv.first > 1 && (kv.second > best || (kv.second == best && kv.first < s))) {
            best = kv.second;
            s = kv.first;
        }
    if (s < 2) return 0;
    int64_t near = 0;
    for (auto& kv : freq)
        if (kv.first == 1 || std::abs(kv.first - s) <= 1) near += kv.second;
    return near * 20 >= total * 19 ? s : 0;
}

int even_up(int v) { return (v + 1) & ~1; }

// Slices a full w x h tile takes: two parities of the grid, each cut into runs
// of 32; `span`: a run stays within one grid row.
int rect_slices(int w, int h, bool span) {
    const int half = (w + 1) / 2;
    return span ? 2 * h * ((half + kLanes - 1) / kLanes) : 2 * ((half * h + kLanes - 1) / kLanes);
}

struct Cut {
    int bx = 1, by = 1;
    bool ok = false;
};
// The split of an s x rows grid into at most k rectangles that costs least per
// sweep: a slice's sums weigh about five times the exchange of 32 halo rows.
Cut best_cut(int s, int rows, int k, int max_slices) {
    Cut best;
    double cost = 0.0;
    for (int bx = 1; bx <= std::min(k, std::max(1, s / 2)); ++bx) {
        const int by = std::min(k / bx, rows);
        if (by < 1) break;
        const int w = std::min(s, even_up((s + bx - 1) / bx)), h = (rows + by - 1) / by;
        const int sl = std::min(rect_slices(w, h, true), (int)(1.15 * rect_slices(w, h, false)));
        if (rect_slices(w, h, false) > max_slices) continue;
        const double ew = w + (bx > 1 ? 2 : 0) + (bx > 2 ? 2 : 0), eh = h + (by > 1 ? 2 : 0) + (by > 2 ? 2 : 0);
        const double c = sl * 100.0 + (ew * eh - (double)w * h) / kLanes * 20.0;
        if (!best.ok || c < cost) {
            best.bx = bx;
            best.by = by;
            best.ok = true;
            cost = c;
        }
    }
    return best;
}

// Recursive bisection of rows [b, e) of `ids` by rest position into k parts.
void bisect(const HostTables& H, std::vector<int>& ids, int b, int e, int k, std::vector<std::vector<int>>& out) {
    if (k <= 1 || e - b <= 1) {
        out.emplace_back(ids.begin() + b, ids.begin() + e);
        std::sort(out.back().begin(), out.back().end());
        return;
    }
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int q = b; q < e; ++q)
        for (int c = 0; c < 3; ++c) {
            lo[c] = std::min(lo[c], H.X[3 * (size_t)ids[q] + c]);
            hi[c] = std::max(hi[c], H.X[3 * (size_t)ids[q] + c]);
        }
    int ax = 0;
    for (int c = 1; c < 3; ++c)
        if (hi[c] - lo[c] > hi[ax] - lo[ax]) ax = c;
    const int kl = k / 2, mid = b + (int)((int64_t)(e - b) * kl / k);
    std::nth_element(ids.begin() + b, ids.begin() + mid, ids.begin() + e, [&](int x, int y) {
        const double a = H.X[3 * (size_t)x + ax], c = H.X[3 * (size_t)y + ax];
        return a < c || (a == c && x < y);
    });
    bisect(H, ids, b, mid, kl, out);
    bisect(H, ids, mid, e, k - kl, out);
}

// Cuts model m into at most k tiles of at most max_slices slices each; false
// when that takes more than k.
bool cut_model(const HostTables& H, const Model& m, int k, int max_slices, std::vector<std::vector<int>>& out) {
    const int nv = m.hi - m.lo;
    if (nv <= 0) return true;
    if (m.stride > 0) {
        const int s = m.stride, rows = (nv + s - 1) / s;
        const Cut c = best_cut(s, rows, k, max_slices);
        if (!c.ok) return false;
        const size_t first = out.size();
        out.resize(first + (size_t)c.bx * c.by);
        // block edges on even columns, so that both parities fill their runs alike
        auto xb = [&](int i) { return i >= c.bx ? s : (int)((int64_t)(s / 2) * i / c.bx) * 2; };
        auto yb = [&](int i) { return (int)((int64_t)rows * i / c.by); };
        std::vector<int> colBlock(s);
        for (int i = 0; i < c.bx; ++i)
            for (int x = xb(i); x < xb(i + 1); ++x) colBlock[x] = i;
        for (int j = 0; j < c.by; ++j)
            for (int y = yb(j); y < yb(j + 1); ++y)
                for (int x = 0; x < s; ++x) {
                    const int v = y * s + x;
                    if (v < nv) out[first + (size_t)j * c.bx + colBlock[x]].push_back(m.lo + v);
                }
        for (size_t q = first; q < out.size(); ++q)
            if ((int)out[q].size() > max_slices * kLanes) return false;
        out.erase(std::remove_if(out.begin() + first, out.end(), [](const std::vector<int>& v) { return v.empty(); }),
                  out.end());
        return true;
    }
    if ((nv + k - 1) / k > max_slices * kLanes - kLanes) return false;
    std::vector<int> ids(nv);
    std::iota(ids.begin(), ids.end(), m.lo);
    bisect(H, ids, 0, nv, k, out);
    return true;
}

}  // namespace

size_t tile_smem_bytes(const TileInfo& t, int pat_stride, int value_bytes, int vectors, bool slot_rhs, bool pairs) {
    auto a16 = [](size_t b) { return (b + 15) / 16 * 16; };
    return (pairs ? 0 : a16((size_t)t.nent * value_bytes)) + a16((size_t)t.npat * pat_stride * sizeof(int16_t)) +
           vectors * a16(3 * (size_t)t.nloc * value_bytes) + (slot_rhs ? 96 * (size_t)t.nslice * value_bytes : 0);
}

namespace {

// pairs: slices are of pairs of rows; the tiles are cut for `spare` slices less than
// they may have, since rows without a partner take more.
void try_plan(const HostTables& H, const TileLimits& lim, int order_block, bool pairs, int spare, TilePlan& P) {
    const int ns = H.nsim;
    if (ns == 0 || ns >= 1 << 30) return;
    std::vector<Model> models;
    for (int i = 0; i < ns;) {
        int e = i + 1;
        while (e < ns && H.vertexModel[e] == H.vertexModel[i]) ++e;
        models.push_back(Model{i, e, grid_stride(H, i, e)});
        i = e;
    }
    const int max_slices = lim.max_warps * lim.max_rows_per_thread;
    const int cut_slices = max_slices - spare, max_rows = cut_slices * kLanes;

    // ---- rows per tile: one tile per SM where a tile then has at most one row
    // per thread, else two per SM (a count in between leaves SMs with half the
    // work of others); never fewer than min_rows (a smaller tile only adds
    // halo).  When one launch cannot hold every row, full tiles in launches of
    // whole models ----
    std::vector<std::vector<int>> own;
    std::vector<int> tileModel;
    auto cut_all = [&](int target) -> bool {
        own.clear();
        tileModel.clear();
        for (size_t q = 0; q < models.size(); ++q) {
            const int nv = models[q].hi - models[q].lo;
            int k = std::max(1, (nv + target - 1) / target);
            const size_t first = own.size();
            bool done = false;
            for (int tries = 0; tries < 64 && !done; ++tries) {
                own.resize(first);
                done = cut_model(H, models[q], k, cut_slices, own);
                if (!done) k += 1 + k / 16;
            }
            if (!done) return false;
            tileModel.resize(own.size(), (int)q);
        }
        return true;
    };
    const int sms = lim.sms, one_row = lim.max_warps * kLanes;
    int most_tiles = ns <= one_row / 10 * 9 * sms ? sms : lim.co_resident;
    int target = std::min(max_rows, std::max(lim.min_rows, (ns + most_tiles - 1) / most_tiles));
    if (ns <= one_row && models.size() == 1) target = one_row;  // one tile: no exchange at all
    bool fits = false;
    // few rows: the tiles of one cluster, a row per thread
    if (lim.cluster > 0 && ns > lim.cluster_min && ns <= lim.cluster * lim.cluster_rows) {
        for (int t = (ns + lim.cluster - 1) / lim.cluster; !P.cluster && t <= lim.cluster_rows; t += std::max(4, t / 16)) {
            if (!cut_all(t)) return;
            P.cluster = (int)own.size() <= lim.cluster;
            for (const auto& o : own) P.cluster = P.cluster && (int)o.size() <= one_row;
        }
        fits = P.cluster;
    }
    while (!fits) {
        if (!cut_all(target)) return;
        if ((int)own.size() <= most_tiles) {
            fits = true;
            break;
        }
        if (target >= (most_tiles < lim.co_resident ? one_row : max_rows)) {
            if (most_tiles == lim.co_resident) break;
            most_tiles = lim.co_resident;
            target = std::max(lim.min_rows, (ns + most_tiles - 1) / most_tiles);
            continue;
        }
        target = std::min(max_rows, target + std::max(8, target / 16));
    }
    if (!fits && (models.size() < 2 || H.ntet > 0)) return;
    P.pairs = pairs && most_tiles == lim.co_resident;
    for (const Model& m : models) P.pairs = P.pairs && m.stride > 0;
    if (pairs && !P.pairs) return;
    const int nt = (int)own.size();

    // ---- launches: runs of whole models ----
    {
        const int cap = std::min(lim.co_resident, lim.group_cap);
        int lo = 0;
        while (lo < nt) {
            int hi = lo;  // exclusive
            while (hi < nt) {
                int e = hi;
                while (e < nt && tileModel[e] == tileModel[hi]) ++e;
                if (e - lo > cap) break;
                hi = e;
            }
            if (hi == lo) return;
            P.groups.push_back(TileGroup{lo, hi - 1});
            lo = hi;
        }
        if (P.groups.size() > 1 && H.ntet > 0) return;
    }

    std::vector<int> tileOf(ns, -1), cls(ns, 0), modelOf(P.pairs ? ns : 0);
    if (P.pairs)
        for (size_t q = 0; q < models.size(); ++q)
            std::fill(modelOf.begin() + models[q].lo, modelOf.begin() + models[q].hi, (int)q);
    for (int t = 0; t < nt; ++t)
        for (int v : own[t]) tileOf[v] = t;
    for (const Model& m : models)
        if (m.stride > 0)
            for (int v = m.lo; v < m.hi; ++v) cls[v] = (((v - m.lo) / m.stride) + ((v - m.lo) % m.stride)) & 1;

    // ---- exchange relations: halos (columns of the matrix rows and stencils),
    // closed so that whoever reads a tile is read by it, and the tiles to wait
    // for (tets too) ----
    std::vector<std::vector<int>> halo(nt), nbr(nt);
    {
        std::vector<int> stamp(ns, -1);
        for (int t = 0; t < nt; ++t)
            for (int v : own[t]) {
                auto see = [&](int c) {
                    if (tileOf[c] == t || stamp[c] == t) return;
                    stamp[c] = t;
                    halo[t].push_back(c);
                    nbr[t].push_back(tileOf[c]);
                };
                for (int e = H.nPtr[v]; e < H.nPtr[v + 1]; ++e) see(H.nCol[e]);
                for (int e = H.lPtr[v] + 1; e < H.lPtr[v + 1]; ++e) see(H.lNbr[e]);
            }
        auto reads = [&](int t, int u) {
            for (int c : halo[t])
                if (tileOf[c] == u) return true;
            return false;
        };
        std::vector<std::vector<int>> from(nt);
        for (int t = 0; t < nt; ++t) {
            for (int c : halo[t]) from[t].push_back(tileOf[c]);
            std::sort(from[t].begin(), from[t].end());
            from[t].erase(std::unique(from[t].begin(), from[t].end()), from[t].end());
        }
        for (int t = 0; t < nt; ++t)
            for (int u : from[t])
                if (!std::binary_search(from[u].begin(), from[u].end(), t) && !reads(u, t))
                    halo[u].push_back(own[t][0]);
        for (int e = 0; e < H.ntet; ++e)
            for (int a = 0; a < 4; ++a)
                for (int b = 0; b < 4; ++b) {
                    const int va = H.tets[4 * (size_t)e + a], vb = H.tets[4 * (size_t)e + b];
                    if (va >= 0 && vb >= 0 && tileOf[va] != tileOf[vb]) nbr[tileOf[va]].push_back(tileOf[vb]);
                }
        for (int t = 0; t < nt; ++t)
            for (size_t q = 0, n = nbr[t].size(); q < n; ++q)
                if (q == 0 || nbr[t][q] != nbr[t][q - 1]) nbr[nbr[t][q]].push_back(t);
        for (int t = 0; t < nt; ++t) {
            std::sort(nbr[t].begin(), nbr[t].end());
            nbr[t].erase(std::unique(nbr[t].begin(), nbr[t].end()), nbr[t].end());
        }
    }
    std::vector<uint8_t> pub(ns, 0);
    for (int t = 0; t < nt; ++t)
        for (int c : halo[t]) pub[c] = 1;

    std::vector<std::vector<int>> tetsOf(H.ntet > 0 ? nt : 0);
    for (int e = 0; e < H.ntet; ++e) tetsOf[tileOf[H.tets[4 * (size_t)e]]].push_back(e);

    int patW = 2;
    for (int i = 0; i < ns; ++i) patW = std::max(patW, H.nPtr[i + 1] - H.nPtr[i]);
    if (patW > 255) return;
    P.pat_stride = P.pairs ? kPairEntries : (patW + 7) / 8 * 8;
    // the other row of v's pair: its neighbour in the grid row, of the same tile and
    // in the same block of the summation order; -1: none
    auto partner = [&](int v) {
        const Model& m = models[modelOf[v]];
        const int x = (v - m.lo) % m.stride, u = x % 2 ? v - 1 : v + 1;
        if (u >= m.hi || (x % 2 == 0 && x + 1 >= m.stride) || tileOf[u] != tileOf[v]) return -1;
        return order_block > 0 && u / order_block != v / order_block ? -1 : u;
    };

    // ---- tables, tile by tile, each by itself (several threads), then joined ----
    const int G = 16 / lim.value_bytes;
    auto build = [&](int t, std::vector<int>& pos, TilePlan& Q) -> bool {
        std::vector<int> ext, ent(patW);
        std::vector<int16_t> o(P.pat_stride);
        TileInfo T{};
        auto order = [&](int a, int b) { return cls[a] != cls[b] ? cls[a] < cls[b] : a < b; };
        ext = own[t];
        ext.insert(ext.end(), halo[t].begin(), halo[t].end());
        std::sort(ext.begin(), ext.end(), order);
        for (size_t q = 0; q < ext.size(); ++q) pos[ext[q]] = (int)q;
        T.nloc = (int)ext.size();
        if (T.nloc > 32767) return false;
        // slices: runs of own rows of one parity; kept within 32 consecutive
        // places of the local vectors (no two lanes in one bank) when that
        // costs at most 15% more slices
        // (of pairs: the first rows, in the order of the grid)
        std::vector<int> rows;
        for (int v : own[t]) {
            const int u = P.pairs ? partner(v) : -1;
            if (u < 0 || order(v, u)) rows.push_back(v);
        }
        if (!P.pairs) std::sort(rows.begin(), rows.end(), order);
        const int per = P.pairs ? 2 : 1;  // slices of a run
        std::vector<int> beg;  // first row of each slice
        for (int span = 1; span >= 0; --span) {
            std::vector<int> b;
            for (int q = 0; q < (int)rows.size(); ++q) {
                const bool brk = b.empty() || q - b.back() >= kLanes ||
                                 (!P.pairs && cls[rows[q]] != cls[rows[b.back()]]) ||
                                 (span && std::abs(pos[rows[q]] - pos[rows[b.back()]]) >= kLanes);
                if (brk) b.push_back(q);
            }
            if (span) {
                beg = b;
            } else if ((int)beg.size() * per > max_slices || beg.size() * 100 > b.size() * 115) {
                beg = b;
            }
        }
        if ((int)beg.size() * per > max_slices) return false;
        T.model = tileModel[t];
        T.nslice = (int)beg.size() * per;
        T.slot0 = (int)Q.slots.size();
        T.slice0 = (int)Q.slices.size();
        T.ent0 = (int)Q.val.size();
        T.pat0 = (int)(Q.pat.size() / P.pat_stride);
        std::unordered_map<uint64_t, std::vector<int>> seen;  // hash of the offsets -> pattern ids
        int npat = 0;
        auto pattern = [&]() {  // of the offsets o
            uint64_t h = 1469598103934665603ull;
            for (int16_t v : o) h = (h ^ (uint16_t)v) * 1099511628211ull;
            for (int c : seen[h])
                if (std::memcmp(&Q.pat[(size_t)(T.pat0 + c) * P.pat_stride], o.data(), sizeof(int16_t) * P.pat_stride) == 0)
                    return c;
            seen[h].push_back(npat);
            Q.pat.insert(Q.pat.end(), o.begin(), o.end());
            return npat++;
        };
        // entry e's part in the order of row r's sum: own block, below it, above it
        auto part = [&](int r, int e) {
            if (order_block <= 0) return 0;
            const int lo = r / order_block * order_block;
            return H.nCol[e] < lo ? 1 : H.nCol[e] < lo + order_block ? 0 : 2;
        };
        for (int s = 0; s < (int)beg.size(); ++s) {
            const int q0 = beg[s], q1 = s + 1 < (int)beg.size() ? beg[s + 1] : (int)rows.size();
            const size_t base = Q.val.size();
            if (P.pairs) {
                std::vector<TileSlot> second(kLanes, TileSlot{-1, 0, 0, 0});
                std::vector<double> v(2 * kPairEntries * kLanes, 0.0);  // by entry, lane, row
                int len = 0;
                TileSlot last{-1, 0, 0, 0};
                for (int lane = 0; lane < kLanes; ++lane) {
                    if (q0 + lane >= q1) {  // an empty lane sums zeros at valid places
                        Q.slots.push_back(last);
                        second[lane] = last;
                        continue;
                    }
                    const int r = rows[q0 + lane], u = partner(r);
                    struct Entry {
                        int part, col;
                        double v[2];
                    };
                    std::vector<Entry> m;
                    for (int w = 0; w < (u < 0 ? 1 : 2); ++w)
                        for (int row = w ? u : r, e = H.nPtr[row]; e < H.nPtr[row + 1]; ++e) {
                            Entry x{part(row, e), H.nCol[e], {0.0, 0.0}};
                            x.v[w] = H.nVal[e];
                            m.push_back(x);
                        }
                    std::sort(m.begin(), m.end(), [](const Entry& x, const Entry& y) {
                        return x.part != y.part ? x.part < y.part : x.col < y.col;
                    });
                    int n = 0, ka = 0, kb = 0;
                    for (size_t q = 0; q < m.size(); ++q) {
                        if (n > 0 && m[n - 1].col == m[q].col && m[n - 1].part == m[q].part) {
                            for (int w = 0; w < 2; ++w) m[n - 1].v[w] += m[q].v[w];  // one of the two is zero
                        } else {
                            m[n++] = m[q];
                        }
                    }
                    if (n > kPairEntries) return false;
                    for (int k = 0; k < n; ++k) {
                        ka += order_block > 0 && m[k].part == 0;
                        kb += order_block > 0 && m[k].part < 2;
                        for (int w = 0; w < 2; ++w) v[2 * (kLanes * k + lane) + w] = m[k].v[w];
                    }
                    len = std::max(len, n);
                    for (int k = 0; k < P.pat_stride; ++k)
                        o[k] = n > 0 ? (int16_t)(pos[m[std::min(k, n - 1)].col] - pos[r]) : (int16_t)0;
                    const int pat = pattern() * P.pat_stride, parts = (ka << 8) | (kb << 16);
                    Q.slots.push_back(TileSlot{r, pos[r], pat, pub[r] | parts});
                    last = TileSlot{-1, pos[r], pat, parts};
                    second[lane] = u < 0 ? last : TileSlot{u, pos[u], pat, pub[u] | parts};
                }
                Q.slots.insert(Q.slots.end(), second.begin(), second.end());
                len = (len + 3) / 4 * 4;
                Q.slices.push_back(TileSlice{(int)(base - T.ent0), len});
                Q.slices.push_back(TileSlice{(int)(base - T.ent0), 0});
                Q.val.resize(base + 2 * (size_t)len * kLanes);
                for (int k = 0; k < len; ++k)
                    for (int q = 0; q < 2 * kLanes; ++q)
                        Q.val[base + 128 * (size_t)(k / 2) + 4 * (q / 2) + 2 * (k % 2) + q % 2] = v[2 * kLanes * (size_t)k + q];
                continue;
            }
            int len = 0;
            for (int q = q0; q < q1; ++q) len = std::max(len, H.nPtr[rows[q] + 1] - H.nPtr[rows[q]]);
            len = (len + 3) / 4 * 4;
            Q.slices.push_back(TileSlice{(int)(base - T.ent0), len});
            Q.val.resize(base + (size_t)len * kLanes, 0.0);
            for (int lane = 0; lane < kLanes; ++lane) {
                if (q0 + lane >= q1) {
                    Q.slots.push_back(TileSlot{-1, 0, 0, 0});
                    continue;
                }
                const int r = rows[q0 + lane], b = H.nPtr[r], n = H.nPtr[r + 1] - b;
                for (int k = 0; k < n; ++k) ent[k] = b + k;
                int ka = 0, kb = 0;
                if (order_block > 0) {  // own block first, then the columns below it, then those above
                    std::stable_sort(ent.begin(), ent.begin() + n, [&](int x, int y) { return part(r, x) < part(r, y); });
                    for (int k = 0; k < n; ++k) {
                        ka += part(r, ent[k]) == 0;
                        kb += part(r, ent[k]) < 2;
                    }
                }
                std::fill(o.begin(), o.end(), (int16_t)0);
                for (int k = 0; k < P.pat_stride; ++k)
                    o[k] = n > 0 ? (int16_t)(pos[H.nCol[ent[std::min(k, n - 1)]]] - pos[r]) : (int16_t)0;
                for (int k = 0; k < n; ++k) Q.val[base + (size_t)kLanes * G * (k / G) + (size_t)G * lane + k % G] = H.nVal[ent[k]];
                Q.slots.push_back(TileSlot{r, pos[r], pattern() * P.pat_stride, pub[r] | (ka << 8) | (kb << 16)});
            }
        }
        for (int s = 0; s < T.nslice; ++s) {
            TileSlot* sl = &Q.slots[T.slot0 + (size_t)kLanes * s];
            int len = 0;
            for (int lane = 0; lane < kLanes; ++lane)
                if (sl[lane].row >= 0) len = std::max(len, H.lPtr[sl[lane].row + 1] - H.lPtr[sl[lane].row] - 1);
            const size_t base = Q.st_pos.size(), n = base + (size_t)len * kLanes;
            Q.stencil.push_back((int)base);
            Q.st_pos.resize(n, 0);
            Q.st_rest.resize(n, 0.0);
            Q.st_lbo.resize(n, 0.0);
            Q.st_bend.resize(n, 0.0);
            for (int lane = 0; lane < kLanes; ++lane) {
                const int r = sl[lane].row;
                if (r < 0) continue;
                const int nst = H.lPtr[r + 1] - H.lPtr[r] - 1;
                if (nst > 127) return false;
                sl[lane].pub |= nst << 24;
                for (int e = H.lPtr[r] + 1, k = 0; e < H.lPtr[r + 1]; ++e, ++k) {
                    const size_t q = base + (size_t)kLanes * k + lane;
                    Q.st_pos[q] = (int16_t)(pos[H.lNbr[e]] - pos[r]);
                    Q.st_rest[q] = H.lRest[e];
                    Q.st_lbo[q] = H.lLbo[e];
                    Q.st_bend[q] = H.lBendT[e];
                }
            }
        }
        T.npat = npat;
        T.nent = (int)Q.val.size() - T.ent0;
        if (T.nent >= 1 << 20 || npat * P.pat_stride > 65535) return false;  // packed in the kernel
        T.halo0 = (int)Q.halo.size();
        T.nhalo = (int)halo[t].size();
        std::sort(halo[t].begin(), halo[t].end());
        for (int c : halo[t]) Q.halo.push_back(TileHalo{c, pos[c]});
        T.nbr0 = (int)Q.nbr.size();
        T.nnbr = (int)nbr[t].size();
        Q.nbr.insert(Q.nbr.end(), nbr[t].begin(), nbr[t].end());
        T.tet0 = (int)Q.tet.size();
        if (H.ntet > 0) {
            T.ntet = (int)tetsOf[t].size();
            Q.tet.insert(Q.tet.end(), tetsOf[t].begin(), tetsOf[t].end());
        }
        Q.tiles.push_back(T);
        return true;
    };
    std::vector<TilePlan> piece(nt);
    {
        std::atomic<int> next{0};
        std::atomic<bool> ok{true};
        auto work = [&]() {
            try {
                std::vector<int> pos(ns, 0);
                for (int t; ok && (t = next++) < nt;)
                    if (!build(t, pos, piece[t])) ok = false;
            } catch (const std::bad_alloc&) {  // no plan
                ok = false;
            }
        };
        std::vector<std::thread> team;
        for (int k = std::min({nt / 16, 7, (int)std::thread::hardware_concurrency() - 1}); k > 0; --k) {
            try {
                team.emplace_back(work);
            } catch (const std::exception&) {  // no thread or no memory for one (those that run are joined below)
                break;
            }
        }
        work();
        for (std::thread& th : team) th.join();
        if (!ok) return;
    }
    int most = 0;
    size_t most3 = 0;
    for (TilePlan& Q : piece) {
        TileInfo T = Q.tiles[0];
        T.slot0 = (int)P.slots.size();
        T.slice0 = (int)P.slices.size();
        T.ent0 = (int)P.val.size();
        T.pat0 = (int)(P.pat.size() / P.pat_stride);
        T.halo0 = (int)P.halo.size();
        T.nbr0 = (int)P.nbr.size();
        T.tet0 = (int)P.tet.size();
        for (int& q : Q.stencil) q += (int)P.st_pos.size();
        auto join = [](auto& to, auto& from) {
            to.insert(to.end(), from.begin(), from.end());
            from.clear();
            from.shrink_to_fit();
        };
        join(P.slots, Q.slots);
        join(P.slices, Q.slices);
        join(P.val, Q.val);
        join(P.pat, Q.pat);
        join(P.stencil, Q.stencil);
        join(P.st_pos, Q.st_pos);
        join(P.st_rest, Q.st_rest);
        join(P.st_lbo, Q.st_lbo);
        join(P.st_bend, Q.st_bend);
        join(P.halo, Q.halo);
        join(P.nbr, Q.nbr);
        join(P.tet, Q.tet);
        most = std::max(most, T.nslice);
        const size_t sm = tile_smem_bytes(T, P.pat_stride, lim.value_bytes, 2, lim.slot_rhs, P.pairs);
        if (lim.vectors > 2)
            most3 = std::max(most3,
                             tile_smem_bytes(T, P.pat_stride, lim.value_bytes, lim.vectors, lim.slot_rhs, P.pairs));
        if (sm > lim.smem) return;
        P.smem_bytes = std::max(P.smem_bytes, sm);
        P.tiles.push_back(T);
    }
    for (const TileInfo& T : P.tiles) P.nloc_max = std::max(P.nloc_max, T.nloc);
    if (P.cluster) {
        // whom each row goes to; the vectors are laid out alike in every tile
        std::unordered_map<int, int> slotOf;
        for (size_t q = 0; q < P.slots.size(); ++q)
            if (P.slots[q].row >= 0) slotOf[P.slots[q].row] = (int)q;
        P.push.assign(4 * P.slots.size(), -1);
        for (int t = 0; t < nt && P.cluster; ++t)
            for (int h = 0; h < P.tiles[t].nhalo; ++h) {
                const TileHalo& q = P.halo[P.tiles[t].halo0 + h];
                int* d = &P.push[4 * (size_t)slotOf[q.row]];
                int k = 0;
                while (k < 4 && d[k] >= 0) ++k;
                if (k == 4) P.cluster = false;  // a fifth reader
                else d[k] = t << 16 | q.pos;
            }
        size_t sm = 0;
        for (const TileInfo& T : P.tiles) {
            TileInfo u = T;
            u.nloc = P.nloc_max;
            sm = std::max(sm, tile_smem_bytes(u, P.pat_stride, lim.value_bytes, lim.vectors, lim.slot_rhs));
        }
        if (sm > lim.smem || most > lim.max_warps) P.cluster = false;
        if (!P.cluster) {  // larger tiles have fewer readers
            TileLimits l = lim;
            l.cluster = lim.cluster >= 8 ? lim.cluster / 2 : 0;
            P = TilePlan();
            try_plan(H, l, order_block, pairs, spare, P);
            return;
        }
        P.smem_bytes = sm;
        most3 = sm;
    }
    P.rows_per_thread = P.pairs ? 2 : (most + lim.max_warps - 1) / lim.max_warps;
    P.threads = (most + P.rows_per_thread - 1) / P.rows_per_thread * kLanes;
    if (lim.vectors > 2 && most3 <= lim.smem) {
        P.vectors = lim.vectors;
        P.smem_bytes = most3;
    }
    P.ok = !P.pairs || P.vectors == lim.vectors;
}

}  // namespace

void build_tile_plan(const HostTables& H, const TileLimits& lim, int order_block, TilePlan& P) {
    if (lim.pairs && H.ntet == 0 && H.nsim > lim.pair_rows * lim.co_resident)
        for (int spare = 0; spare <= 6; spare += 2) {
            P = TilePlan();
            try_plan(H, lim, order_block, true, spare, P);
            if (P.ok || !P.pairs) break;
        }
    if (P.ok && P.pairs) return;
    P = TilePlan();
    try_plan(H, lim, order_block, false, 0, P);
}

}  // namespace pdipc
