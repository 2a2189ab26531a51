// tile.h — arguments and launch of the tiled persistent PD solve (pd_tile.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "common.cuh"
#include "persistent.h"
#include "tile_plan.h"

namespace pdipc {

// Pairs (FP32 arithmetic on a grid, no tets): a thread sums two neighbours of a grid
// row over the union of their columns, 28 in place of 24 + 20, so that a place of the
// iterate is read once for both; the values, two per entry, lie in tensor memory (a
// warp's 32 pairs take 64 of the columns of its quarter of the lanes), where reading
// them takes nothing of shared memory's bandwidth, which bounded these sums.  A
// kernel that uses tensor memory runs one CTA per SM: it is two tiles, half of the
// threads each, and takes all 512 columns.
// One sweep of a mixed solve, before -> with pairs: 512x512 4.47 -> 3.73 us, four
// 256x256 4.84 -> 3.65; one solve 3.24 -> 2.90 ms and 3.49 -> 2.93, 40 cloths of 16^2
// to 126^2 1.93 -> 1.74, 430x430 1.40 -> 1.30 (FP32 1.17 -> 1.11).  Up to kPairRows
// rows per tile the sweeps wait for each other's words rather than for the sums, and
// half the threads take longer (333x333: 1.32, 1.44 with pairs; 380x380: 1.25, 1.20).
constexpr int kPairColumns = 512, kPairTiles = 2, kPairRows = 400;
constexpr int kTileMaxWarps = 14;  // row warps per CTA; two CTAs share an SM (72 registers per thread)

// A published value: 16 bytes read and written as one, the phase's tag in the
// last word.  A vertex is one word in FP32 (x, y, z, tag) and three in FP64
// ((value, tag) per component).
struct alignas(16) TileWord {
    unsigned long long lo, hi;
};

// T: solver scalar; S: state scalar (T in the direct form, double in the
// correction form).
template <typename T, typename S>
struct TileArgs {
    int nsim;
    int lg;
    int cheby;
    T relax;
    T omega[kMaxCheby];
    long long timeout;  // limit of a poll in clock cycles (a cluster polls nothing)
    // state, as in PersistArgs
    V4<S>* P;
    V4<T>* Ph;
    V4<T>* Pl;
    const V4<S>* Pold;
    const V4<S>* Xrest;
    const V4<S>* Rhs0;
    const V4<T>* CollRhs;
    const V4<T>* PinRhs;
    const T* Delastic;
    const T* Dinert;
    const T* CollDiag;
    const int* PinFlag;
    const T* PinK;
    const T* Strain;
    const T* CurvNorm;
    const T* tBend0;
    const T* tLbo0;
    // tets (as in PersistArgs; tile t projects tet[tet0 .. tet0 + ntet))
    const int4* Tets;
    const T* TetIdm;
    const T* TetW;
    V4<T>* TetOut;
    const int* vtPtr;
    const int* vtIdx;
    const int* tet;
    // tiles
    const TileInfo* tiles;
    const TileSlot* slots;
    const TileSlice* slices;
    const T* val;
    const int16_t* pat;
    const TileHalo* halo;
    int patStride;
    // stencils by slot: neighbour k of a row of slice s at stencil[s] + 32 k +
    // lane (place relative to the row's own, weights)
    const int* stencil;
    const int16_t* stPos;
    const T* stRest;  // spring rest length
    const T* stLbo;
    const T* stBend;  // transposed bending weight
    // exchange: ex[(parity * kWords + w) * nsim + row], tags from epoch0 + 1
    TileWord* ex;
    unsigned epoch0;
    // tets only: phase counts of the tiles and the tiles each waits for
    unsigned* flags;
    const int* nbr;
    unsigned flag0;
    unsigned* err;
    const OuterGate* gate;
    const unsigned* instStop;  // per-instance stopping: tiles of a stopped model return at entry
    V4<T>* tape;               // direct form: the positions at the start of every local-global iteration, or null
    int lo, hi;                // tiles of this launch
    int partSmem;              // pairs: shared memory of one of a CTA's tiles
    const int4* push;          // cluster: the readers of every slot's row (TilePlan::push)
    int nlocMax;               // cluster: places of each vector
    int third;                 // correction form: the tiles hold a third vector
    int keptFirst;             // correction form: which product of a sweep's update is rounded (jacobi)
};

// Words of one vertex in a phase: the correction form publishes the two halves
// of its positions in the same phase.
template <typename T, typename S>
constexpr int kTileWords = sizeof(T) == 8 ? 3 : sizeof(S) == 8 ? 2 : 1;
// Entries of a row whose values lie together (16 bytes).
template <typename T>
constexpr int kTileGroup = 16 / (int)sizeof(T);
// Tags and flags one launch uses at most.
inline unsigned tile_phases(int lg, int cheby) { return (unsigned)(lg * (2 * cheby + 1) + 2); }

// Residents: CTAs of the variant one cooperative launch can hold (0: no such variant).
template <typename T, typename S>
int tile_residents(int rows_per_thread, bool tets, bool pairs, int threads, size_t smem, int sms);
template <typename T, typename S>
cudaError_t launch_pd_tile(const TileArgs<T, S>& args, int tiles, int rows_per_thread, bool tets, bool pairs, int threads,
                           size_t smem, cudaStream_t s);
// The tiles as one thread-block cluster (FP32 arithmetic, a row per thread): a
// thread writes its new vector into the shared memory of the tiles that read it,
// and the cluster's barrier ends the sweep, in place of words in global memory that
// the readers poll; one CTA per SM, so a thread takes 120 registers (20x20 0.377 ->
// 0.352 ms, 64x64 0.437 -> 0.428; the words' kernels are no faster with more than
// 72).  One solve of 10 x (local step + 30 sweeps), mixed, words -> cluster: 20x20
// 0.50 -> 0.35 ms, 32x32 0.46 -> 0.36, 48x48 0.49 -> 0.44, 64x64 0.50 -> 0.43; FP32
// 0.42 -> 0.31, 0.39 -> 0.31, 0.45 -> 0.37, 0.46 -> 0.38.
// Up to kTileClusterMin rows one tile alone is as fast (16x16 0.340 ms, 0.344 in a
// cluster; FP32 0.285, 0.307); beyond kTileClusterRows rows per CTA the sums of so
// few SMs cost more than the words of many (66x66: 0.550, 0.552 in a cluster).  With
// tets their projection wants the SMs (block of 8^3 cubes: 0.74, 0.81 in a cluster).
constexpr int kTileCluster = 16, kTileClusterMin = 320, kTileClusterRows = 272;
// Whether the device holds such a cluster, and the launch.
template <typename T, typename S>
bool tile_cluster_fits(int tiles, int threads, size_t smem);
template <typename T, typename S>
cudaError_t launch_pd_tile_cluster(const TileArgs<T, S>& args, int tiles, int threads, size_t smem, cudaStream_t s);

// FP64 with three warps per slice, one component each (pd_tile3.cu); no tets.
// threads: 96 per slice.  Up to kTile3Rows rows per SM: one solve of 10 local-global
// iterations, a component against a row per thread, 0.99 / 1.66 ms at 64x64 (27
// rows per SM), 1.56 / 1.77 at 128x128 (108), 2.28 / 2.56 at 180x180 (213); beyond,
// a tile per SM no longer holds the rows.
constexpr int kTile3Warps = 9;  // slices of a tile
constexpr int kTile3Rows = 216;
int tile3_residents(int threads, size_t smem, int sms);
cudaError_t launch_pd_tile3(const TileArgs<double, double>& args, int tiles, int threads, size_t smem, cudaStream_t s);

}  // namespace pdipc
