// tile_plan.h — partition of the simulated rows into tiles for the tiled
// persistent solve (pd_tile.cu, pd_tile3.cu) and every table a tile reads.  Host only.
#pragma once

#include <cstdint>
#include <vector>

#include "host_tables.h"

namespace pdipc {

// One tile: the rows one CTA updates.  All first/count pairs index the
// concatenated tables of TilePlan.
struct TileInfo {
    int slot0, nslice;   // its slots: 32 per slice
    int slice0;          // first slice record
    int ent0, nent;      // matrix entries by slice
    int pat0, npat;      // column-offset patterns
    int halo0, nhalo;    // rows of other tiles its rows' matrix entries and stencils read
    int nloc;            // own rows + halo: length of its local vectors
    int nbr0, nnbr;      // tiles it exchanges anything with
    int tet0, ntet;      // tets it projects
    int model;           // the simulated model its rows belong to
    int pad;
};
struct TileSlot {
    int row;  // -1: an empty lane
    int pos;  // place in the tile's local vectors
    int pat;  // first element of its offsets in the tile's pattern table
    int pub;  // bit 0: some other tile reads the row; bits 8-15 and 16-23: entries [0, a) lie in the
              // row's own block, [a, b) below it, [b, ...) above (b <= 255); bits 24-30: neighbours
              // in its stencil
};
struct TileSlice {
    int off;  // first entry, relative to ent0; entry k of lane l at off + 32 G (k / G) + G l + k % G
              // (G = 16 / value_bytes: a lane's G consecutive entries are one 16-byte load)
    int len;  // entries per row, a multiple of 4
};
struct TileHalo {
    int row;  // owned by another tile of the same model
    int pos;
};
// One launch: whole models, tiles [lo, hi].
struct TileGroup {
    int lo = 0, hi = -1;
};

struct TileLimits {
    int value_bytes = 4;
    int vectors = 2;          // vectors of the local vertices a tile holds; 3: where they fit
    int max_warps = 14;       // row warps a CTA can have
    int max_rows_per_thread = 2;
    int min_rows = 128;       // rows of a tile at least, where the mesh has them
    int sms = 152;
    int co_resident = 304;    // CTAs one cooperative launch holds: one or two per SM
    int cluster = 0;          // CTAs of a cluster at most (0: none),
    int cluster_min = 0;      // where there are more rows than this,
    int cluster_rows = 0;     // and no more than this many per CTA
    bool pairs = false;       // a thread may sum two neighbours of a grid row together, where the
    int pair_rows = 0;        // tiles of one launch would hold more rows than this each
    bool slot_rhs = false;    // a tile also holds three values per slot (pd_tile3.cu)
    int group_cap = 1 << 30;  // pdipc_params.pd_group_ctas
    size_t smem = 113 * 1024; // per CTA
};

struct TilePlan {
    bool ok = false;
    int rows_per_thread = 1;
    int threads = 0;
    int pat_stride = 0;  // elements of one pattern, a multiple of 8 (16 bytes)
    size_t smem_bytes = 0;
    int vectors = 2;
    // the tiles form one thread-block cluster: vectors at the start of shared
    // memory, nloc_max places each, and up to four readers of every slot's row,
    // tile << 16 | place there (-1: none)
    bool cluster = false;
    int nloc_max = 0;
    std::vector<int> push;
    // slices 2u and 2u + 1 hold, lane by lane, two neighbours of a grid row whose
    // sums run together over the union of their columns (places relative to the
    // first row's; parts [0, a) [a, b) [b, ...) of the union).  Only slice 2u has
    // entries: k of lane l for the first and second row at off + 128 (k / 2) + 4 l +
    // 2 (k % 2), + 1 (zero where the row has no such column).  Values stay outside
    // of shared memory.
    bool pairs = false;
    std::vector<TileInfo> tiles;
    std::vector<TileSlot> slots;
    std::vector<TileSlice> slices;
    std::vector<double> val;
    std::vector<int16_t> pat;
    // the rows' local-step stencils, SELL-32 by slot (one record per slice)
    std::vector<int> stencil;         // first element
    std::vector<int16_t> st_pos;      // neighbour's place relative to the row's
    std::vector<double> st_rest, st_lbo, st_bend;
    std::vector<TileHalo> halo;
    std::vector<int> nbr;
    std::vector<int> tet;
    std::vector<TileGroup> groups;
};

// Shared memory of one tile: values, patterns and the vectors of its local
// vertices.
size_t tile_smem_bytes(const TileInfo& t, int pat_stride, int value_bytes, int vectors, bool slot_rhs,
                       bool pairs = false);
constexpr int kPairEntries = 32;  // of a union at most: 64 values of a slice's pairs per lane

// order_block > 0: a row sums its entries in the order [columns of its own block
// of order_block rows][lower columns][higher columns], each part ascending;
// 0: ascending columns.  Leaves out.ok false when no partition fits the limits.
void build_tile_plan(const HostTables& H, const TileLimits& lim, int order_block, TilePlan& out);

}  // namespace pdipc
