// Checks the tile partition (tile_plan.h) of several meshes against the host
// tables it was built from: every row in exactly one slot, every matrix entry
// and stencil neighbour found at its place with its value, in the stated order,
// halos of the same model owned by a tile that is waited for and reads back,
// launches of whole models within the limits.  Prints "ok" or what failed.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <numeric>
#include <random>
#include <set>

#include "tile_plan.h"

using namespace pdipc;

static ModelInput grid(int nx, int ny, double y, bool shuffle) {
    ModelInput m;
    m.nv = nx * ny;
    std::mt19937 g(nx * 131 + ny);
    std::uniform_real_distribution<double> u(-1e-4, 1e-4);
    std::vector<int> id(m.nv);
    std::iota(id.begin(), id.end(), 0);
    if (shuffle) std::shuffle(id.begin(), id.end(), g);
    m.X.resize(3 * m.nv);
    for (int r = 0; r < ny; ++r)
        for (int c = 0; c < nx; ++c) {
            const int v = id[r * nx + c];
            m.X[3 * v] = 0.01 * c + u(g);
            m.X[3 * v + 1] = y + u(g);
            m.X[3 * v + 2] = 0.01 * r + u(g);
        }
    for (int r = 0; r + 1 < ny; ++r)
        for (int c = 0; c + 1 < nx; ++c) {
            const int a = id[r * nx + c], b = id[r * nx + c + 1], d = id[(r + 1) * nx + c], e = id[(r + 1) * nx + c + 1];
            if ((r + c) & 1) m.F.insert(m.F.end(), {a, d, b, b, d, e});
            else m.F.insert(m.F.end(), {a, d, e, a, e, b});
        }
    m.nf = (int)m.F.size() / 3;
    m.density = 0.1;
    m.k_stretch = 1e4;
    m.k_bend = 1e-3;
    m.k_pin = 1e6;
    m.pins = {0};
    return m;
}

#define FAIL(...)            \
    do {                     \
        printf(__VA_ARGS__); \
        printf("\n");        \
        return false;        \
    } while (0)

static bool check(const HostTables& H, const TileLimits& L, int block) {
    TilePlan P;
    build_tile_plan(H, L, block, P);
    if (!P.ok) FAIL("no plan for %d rows", H.nsim);
    const int G = 16 / L.value_bytes;
    std::vector<int> owner(H.nsim, -1);
    for (size_t t = 0; t < P.tiles.size(); ++t)
        for (int q = 0; q < P.tiles[t].nslice * 32; ++q) {
            const int r = P.slots[P.tiles[t].slot0 + q].row;
            if (r < 0) continue;
            if (owner[r] >= 0) FAIL("row %d twice", r);
            owner[r] = (int)t;
        }
    for (int r = 0; r < H.nsim; ++r)
        if (owner[r] < 0) FAIL("row %d in no tile", r);
    size_t smem = 0;
    for (size_t t = 0; t < P.tiles.size(); ++t) {
        const TileInfo& T = P.tiles[t];
        if (T.nslice > P.rows_per_thread * P.threads / 32) FAIL("tile %zu: too many slices", t);
        TileInfo room = T;  // a cluster's vectors are laid out alike
        if (P.cluster) room.nloc = P.nloc_max;
        smem = std::max(smem, tile_smem_bytes(room, P.pat_stride, L.value_bytes, P.vectors, L.slot_rhs, P.pairs));
        std::vector<int> at(T.nloc, -1);
        auto place = [&](int pos, int row) {
            if (pos < 0 || pos >= T.nloc || at[pos] != -1) return false;
            at[pos] = row;
            return true;
        };
        std::set<int> nbr(P.nbr.begin() + T.nbr0, P.nbr.begin() + T.nbr0 + T.nnbr);
        for (int q = 0; q < T.nslice * 32; ++q) {
            const TileSlot& S = P.slots[T.slot0 + q];
            if (S.row >= 0 && !place(S.pos, S.row)) FAIL("tile %zu: place of row %d", t, S.row);
            if (P.pairs && S.row < 0 && (S.pos < 0 || S.pos >= T.nloc)) FAIL("tile %zu: place of an empty lane", t);
        }
        for (int h = 0; h < T.nhalo; ++h) {
            const TileHalo& q = P.halo[T.halo0 + h];
            const int u = owner[q.row];
            if (!place(q.pos, q.row)) FAIL("tile %zu: place of halo row %d", t, q.row);
            if (u == (int)t || !nbr.count(u) || P.tiles[u].model != T.model) FAIL("tile %zu: halo owner", t);
            bool back = false;
            for (int k = 0; k < P.tiles[u].nhalo; ++k) back = back || owner[P.halo[P.tiles[u].halo0 + k].row] == (int)t;
            if (!back) FAIL("tile %zu reads %d, which does not read it", t, u);
            bool pub = false;
            for (int k = 0; k < P.tiles[u].nslice * 32; ++k) {
                const TileSlot& S = P.slots[P.tiles[u].slot0 + k];
                if (S.row == q.row) pub = S.pub & 1;
            }
            if (!pub) FAIL("halo row %d not published", q.row);
        }
        for (int s = 0; s < T.nslice; ++s) {
            const int w = P.pairs ? s & 1 : 0;
            const TileSlice& sc = P.slices[T.slice0 + s - w];
            if (P.pairs && sc.len > kPairEntries) FAIL("tile %zu: union too long", t);
            if (P.pairs ? sc.len % 4 || sc.off % 128 || sc.off + 64 * sc.len > T.nent : sc.len % 4 || sc.off % (32 * G) || sc.off + 32 * sc.len > T.nent) FAIL("slice range");
            for (int l = 0; l < 32; ++l) {
                const TileSlot& S = P.slots[T.slot0 + 32 * s + l];
                auto val = [&](int k) {
                    if (P.pairs) return P.val[(size_t)T.ent0 + sc.off + 128 * (k / 2) + 4 * l + 2 * (k % 2) + w];
                    return P.val[(size_t)T.ent0 + sc.off + 32 * G * (k / G) + G * l + k % G];
                };
                auto col = [&](int k) {
                    const int p = P.slots[T.slot0 + 32 * (s - w) + l].pos + P.pat[((size_t)T.pat0) * P.pat_stride + S.pat + k];
                    return p < 0 || p >= T.nloc ? -1 : at[p];
                };
                if (P.pairs)  // every lane reads within the tile, whatever it sums
                    for (int k = 0; k < sc.len; ++k)
                        if (col(k) < 0) FAIL("tile %zu: lane outside", t);
                if (S.row < 0) continue;
                const int r = S.row, b = H.nPtr[r], n = H.nPtr[r + 1] - b, ka = (S.pub >> 8) & 255, kb = (S.pub >> 16) & 255;
                if (n > sc.len) FAIL("row %d cut", r);
                int ne = n;  // of the union: what either row of the pair has
                if (P.pairs) {
                    const int q = P.slots[T.slot0 + 32 * (s ^ 1) + l].row;
                    std::set<int> cols(H.nCol.begin() + b, H.nCol.begin() + b + n);
                    if (q >= 0) cols.insert(H.nCol.begin() + H.nPtr[q], H.nCol.begin() + H.nPtr[q + 1]);
                    if (q >= 0 && (std::abs(q - r) != 1 || (block > 0 && q / block != r / block))) FAIL("row %d: pair", r);
                    ne = (int)cols.size();
                }
                for (int k = ne; k < sc.len; ++k)
                    if (val(k) != 0.0 || col(k) < 0) FAIL("row %d padding", r);
                // stored order: [0, ka) own block, [ka, kb) below, the rest above; in
                // the order (ka..kb), (0..ka), (kb..) the columns ascend
                std::vector<int> ord;
                for (int k = ka; k < kb; ++k) ord.push_back(k);
                for (int k = 0; k < ka; ++k) ord.push_back(k);
                for (int k = kb; k < ne; ++k) ord.push_back(k);
                if (P.pairs)  // the partner's own columns weigh nothing
                    for (size_t q = ord.size(); q-- > 0;)
                        if (!std::binary_search(H.nCol.begin() + b, H.nCol.begin() + b + n, col(ord[q]))) {
                            if (val(ord[q]) != 0.0) FAIL("row %d: weight of its partner's column", r);
                            ord.erase(ord.begin() + q);
                        }
                if ((int)ord.size() != n) FAIL("row %d: %d of %d entries", r, (int)ord.size(), n);
                if (block == 0 && (ka || kb)) FAIL("row %d: parts without a block", r);
                for (int k = 0; k < n; ++k) {
                    if (col(ord[k]) != H.nCol[b + k] || val(ord[k]) != H.nVal[b + k]) FAIL("row %d entry %d", r, k);
                    const bool own = block > 0 && H.nCol[b + k] / block == r / block;
                    if (block > 0 && own != (ord[k] < ka)) FAIL("row %d entry %d: part", r, k);
                }
                const int nst = H.lPtr[r + 1] - H.lPtr[r] - 1;
                if ((S.pub >> 24) != nst) FAIL("row %d: stencil count", r);
                for (int k = 0; k < nst; ++k) {
                    const size_t q = (size_t)P.stencil[T.slice0 + s] + 32 * k + l;
                    const int e = H.lPtr[r] + 1 + k;
                    if (at[S.pos + P.st_pos[q]] != H.lNbr[e] || P.st_rest[q] != H.lRest[e] || P.st_lbo[q] != H.lLbo[e] ||
                        P.st_bend[q] != H.lBendT[e])
                        FAIL("row %d stencil %d", r, k);
                }
            }
        }
    }
    if (P.cluster) {  // every halo place is written once, by its row's owner, and nothing else is
        if ((int)P.tiles.size() > L.cluster || P.rows_per_thread != 1 || P.groups.size() != 1) FAIL("cluster shape");
        std::set<std::pair<int, int>> want, got;
        for (size_t t = 0; t < P.tiles.size(); ++t)
            for (int h = 0; h < P.tiles[t].nhalo; ++h) {
                const TileHalo& q = P.halo[P.tiles[t].halo0 + h];
                want.insert({(int)t << 16 | q.pos, q.row});
            }
        for (size_t q = 0; q < P.push.size(); ++q)
            if (P.push[q] >= 0 && !got.insert({P.push[q], P.slots[q / 4].row}).second) FAIL("written twice");
        if (P.push.size() != 4 * P.slots.size() || want != got) FAIL("cluster readers");
    }
    if (smem != P.smem_bytes || smem > L.smem) FAIL("shared memory");
    int next = 0;
    for (const TileGroup& g : P.groups) {
        if (g.lo != next || g.hi - g.lo + 1 > std::min(L.co_resident, L.group_cap)) FAIL("launch range");
        if (g.lo > 0 && P.tiles[g.lo - 1].model == P.tiles[g.lo].model) FAIL("a launch splits a model");
        next = g.hi + 1;
    }
    if (next != (int)P.tiles.size()) FAIL("launches miss tiles");
    return true;
}

int main() {
    auto run = [](std::vector<ModelInput> ms, int block, int value_bytes, int cap, int cluster = 0, bool pairs = false) {
        HostTables H;
        const std::string e = build_host_tables(ms, -9.8, H);
        if (!e.empty()) {
            printf("%s\n", e.c_str());
            return false;
        }
        TileLimits L;
        L.value_bytes = value_bytes;
        L.vectors = value_bytes == 4 ? 3 : 2;
        if (value_bytes == 8) {  // as the FP64 solve asks
            L.max_warps = 9;
            L.max_rows_per_thread = 1;
            L.min_rows = 32;
            L.co_resident = L.sms;
            L.slot_rhs = true;
            L.smem = 226 * 1024;
        }
        if (cap) L.group_cap = cap;
        L.cluster = cluster;
        if (pairs) {  // as on four SMs
            L.pairs = true;
            L.sms = 4;
            L.co_resident = 8;
            TilePlan P;
            build_tile_plan(H, L, block, P);
            if (!P.ok || !P.pairs) {
                printf("no pairs for %d rows\n", H.nsim);
                return false;
            }
        }
        L.cluster_min = 320;
        L.cluster_rows = 272;
        return check(H, L, block);
    };
    bool ok = true;
    for (int n : {2, 3, 5, 21, 22, 37, 64, 97}) ok = ok && run({grid(n, n, 0, false)}, 0, 4, 0);
    for (int n : {22, 65}) ok = ok && run({grid(n, n, 0, false)}, 64, 4, 0) && run({grid(n, n, 0, false)}, 192, 8, 0);
    ok = ok && run({grid(200, 3, 0, false)}, 64, 4, 0) && run({grid(3, 200, 0, false)}, 64, 8, 0);  // strips
    ok = ok && run({grid(40, 31, 0, true)}, 64, 4, 0);                                              // shuffled numbering
    ok = ok && run({grid(20, 20, 0, false), grid(48, 40, 1, false), grid(7, 9, 2, true)}, 64, 4, 0);
    ok = ok && run({grid(20, 20, 0, false), grid(48, 40, 1, false), grid(33, 33, 2, false)}, 64, 4, 16);
    ok = ok && run({grid(170, 170, 0, false)}, 0, 8, 0) && run({grid(64, 64, 0, false)}, 0, 8, 0);
    ok = ok && run({grid(400, 340, 0, false)}, 0, 4, 0);  // two CTAs per SM, two rows per thread
    for (int n : {18, 25, 33, 49, 65, 66}) ok = ok && run({grid(n, n, 0, false)}, 64, 4, 0, 16);
    ok = ok && run({grid(40, 31, 0, true)}, 64, 4, 0, 16) && run({grid(300, 3, 0, false)}, 0, 4, 0, 16);
    ok = ok && run({grid(20, 20, 0, false), grid(18, 40, 1, false), grid(7, 9, 2, true)}, 64, 4, 0, 16);
    for (int n : {48, 57, 64, 80}) ok = ok && run({grid(n, n, 0, false)}, 0, 4, 0, 0, true) && run({grid(n, n, 0, false)}, 70, 4, 0, 0, true);
    ok = ok && run({grid(41, 60, 0, false), grid(37, 33, 0, false), grid(20, 51, 0, false)}, 93, 4, 0, 0, true);
    ok = ok && run({grid(64, 64, 0, false), grid(64, 64, 0, false), grid(64, 64, 0, false)}, 0, 4, 0, 0, true);  // launches
    if (ok) printf("ok\n");
    return ok ? 0 : 1;
}
