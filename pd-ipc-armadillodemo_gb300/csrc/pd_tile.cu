// pd_tile.cu — the whole projective-dynamics solve of an outer iteration
// (lg x [local step + Chebyshev-accelerated R2 steps as weighted-Jacobi
// sweeps]) in one cooperative launch over compact tiles of rows.
//
// What bounds the solve is not bandwidth but the 31 data exchanges of every
// local-global iteration.  So:
//   * a tile is a compact block of rows (tile_plan.cpp): only the rows within
//     the stencil's reach of its edge are exchanged, and most tiles' rows need
//     nothing from outside;
//   * an exchanged vertex is one 16-byte word that carries the phase's tag, so
//     a reader polls the data itself: one L2 write and one L2 read per phase
//     instead of data, a release of a flag, polls of the flag and a copy;
//   * few tiles form one thread-block cluster (kCl) and write their boundary rows
//     straight into the readers' shared memory;
//   * many rows are summed in pairs with their values in tensor memory (kPairs);
//   * otherwise two CTAs share an SM, so one tile sums while the other waits;
//   * matrix values, column offsets and both copies of the iterate stay in
//     shared memory for the launch; the local step's neighbour differences come
//     from the same memory (positions, or their high and low halves, occupy the
//     two copies while no iterate does), and right-hand sides, inverse diagonals
//     and the Chebyshev history in registers.
//
// Measured (GB300, one solve, before: the row-block launches of pd_persistent.cuh
// or, FP64, one launch per sweep): mixed 16x16 0.97 -> 0.34 ms, 64x64 0.96 -> 0.42,
// 181x181 1.31 -> 0.67, 512x512 4.35 -> 2.90, four 256x256 10.6 -> 2.93; FP32 96x96
// 1.34 -> 0.45; FP64 257x257 9.2 -> 8.0 (smaller FP64 meshes: pd_tile3.cu).
//
// Double buffering of the exchange: in phase p a tile writes its boundary rows
// to parity p & 1 and then reads its halo there.  It overwrites that parity in
// phase p + 2, after it has read every neighbour's phase p + 1, which a
// neighbour publishes only after a CTA barrier that follows its own reads of
// phase p (the plan makes reading mutual).  In a cluster no tile starts a phase
// before all have ended the one before, so two copies of the iterate do.
//
// Every poll of a word or a count is clock-bounded: past the limit it raises
// kErrBarrier, the tile leaves together at its next barrier, and the others' waits end
// on the error or their own limit.  A cluster polls nothing and has no such limit: its
// CTAs run together, each comes to every barrier, and none leaves before the last.
#include <algorithm>
#include <type_traits>

#include "smem_limit.h"
#include "tet_element.cuh"
#include "tile_device.cuh"

namespace pdipc {

namespace {

// How rows exchange and sum: words in global memory; a cluster's shared memory;
// words, with two neighbours of a grid row summed together by one thread.
enum TileForm { kWords, kCluster, kPairs };

template <typename T, typename S, bool kCorr, bool kTets, int R, TileForm kForm>
__global__ void __launch_bounds__(kTileMaxWarps * (kForm == kPairs ? 64 : 32), kForm == kWords ? 2 : 1)
    k_pd_tile(const __grid_constant__ TileArgs<T, S> a) {
    constexpr int kW = kTileWords<T, S>;
    constexpr int kG = kTileGroup<T>;
    constexpr bool kCl = kForm == kCluster, kPair = kForm == kPairs;
    constexpr int kUnroll = R == 1 ? 2 : 1;  // two rows per thread leave no registers for more
    extern __shared__ __align__(16) unsigned char smem[];
    if (outer_stopped(a.gate)) return;
    // pairs: a CTA is several tiles, of as many threads each, with barriers of their own
    const int nthr = kPair ? (int)blockDim.x / kPairTiles : (int)blockDim.x, part = kPair ? (int)threadIdx.x / nthr : 0;
    const int tid = (int)threadIdx.x - part * nthr;
    const int tile = a.lo + (kPair ? kPairTiles * (int)blockIdx.x + part : (int)blockIdx.x);
    unsigned tmem = 0;
    __shared__ unsigned tmem_base;
    auto finish = [&]() {  // every way out from here on
        if constexpr (kPair) {
            tmem_fence_before();
            __syncthreads();
            tmem_fence_after();
            if (threadIdx.x < 32) tmem_free(tmem_base, kPairColumns);
        }
    };
    if constexpr (kPair) {
        if (threadIdx.x < 32) tmem_alloc(&tmem_base, kPairColumns);
        tmem_fence_before();
        __syncthreads();
        tmem_fence_after();
        const unsigned w = threadIdx.x >> 5;
        tmem = tmem_base + ((w & 3u) << 21) + 2u * kPairEntries * (w >> 2);
        if (tile > a.hi) return finish();
    }
    const TileInfo ti = a.tiles[tile];
    if (a.instStop && a.instStop[ti.model]) return finish();
    auto sync = [&]() {  // of the tile's threads
        if constexpr (kPair) half_sync(1 + part, nthr);
        else __syncthreads();
    };
    auto sync_or = [&](bool v) -> bool {
        if constexpr (kPair) return half_sync_or(1 + part, nthr, v);
        else return __syncthreads_or(v);
    };
    const int warp = tid >> 5, lane = tid & 31, nw = nthr >> 5;

    // ---- shared memory: values, offset patterns, two vectors of the local
    // vertices as (x, y) pairs and z ----
    auto a16 = [](size_t b) { return (b + 15) / 16 * 16; };
    // (in a cluster the vectors come first and are laid out alike in every CTA)
    const int nl = kCl ? a.nlocMax : ti.nloc;
    const int vecBytes = (int)a16(3 * (size_t)nl * sizeof(T));
    unsigned char* tab = smem + part * (size_t)a.partSmem + (kCl ? (kCorr ? 3 : 2) * (size_t)vecBytes : 0);
    T* sval = reinterpret_cast<T*>(tab);
    int16_t* spat = reinterpret_cast<int16_t*>(tab + (kPair ? 0 : a16((size_t)ti.nent * sizeof(T))));
    unsigned char* vec0 =
        kCl ? smem : reinterpret_cast<unsigned char*>(spat) + a16((size_t)ti.npat * a.patStride * sizeof(int16_t));
    auto XY = [&](int b) { return reinterpret_cast<Pair<T>*>(vec0 + b * vecBytes); };
    auto Z = [&](int b) { return reinterpret_cast<T*>(XY(b) + nl); };
    if constexpr (!kPair)
        for (int q = tid; q < ti.nent; q += nthr) sval[q] = __ldg(a.val + ti.ent0 + q);
    for (int q = tid; q < ti.npat * a.patStride; q += nthr)
        spat[q] = __ldg(a.pat + (size_t)ti.pat0 * a.patStride + q);

    // ---- this thread's rows: slice r nw + warp, this lane.  Packed, two rows per
    // thread leave few registers: gp = row (negative: none), bit 30: published;
    // lpe = place | pattern's first element << 16; eol = first entry | entries
    // per row << 20 ----
    int gp[R];
    unsigned lpe[R], eol[R];
    T id[R];
    auto slice = [&](int r) { return kPair ? 2 * warp + r : r * nw + warp; };
    auto slot = [&](int r) { return ti.slot0 + 32 * slice(r) + lane; };
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int s = slice(r);
        gp[r] = -1;
        lpe[r] = eol[r] = 0u;
        id[r] = T(0);
        if (s < ti.nslice) {
            const TileSlot sl = a.slots[slot(r)];
            const TileSlice sc = a.slices[ti.slice0 + s];
            if (kPair || sl.row >= 0) {  // (pairs: an empty lane takes part in its warp's sums)
                lpe[r] = (unsigned)sl.pos | ((unsigned)sl.pat << 16);
                eol[r] = (unsigned)(sc.off + kG * lane) | ((unsigned)sc.len << 20);
            }
            if (sl.row >= 0) {
                gp[r] = sl.row | ((sl.pub & 1) << 30);
                id[r] = T(1) / ((a.Delastic[sl.row] + a.Dinert[sl.row]) + a.CollDiag[sl.row]);
            }
        }
    }
    auto live = [&](int r) { return gp[r] >= 0; };
    auto row = [&](int r) { return gp[r] & 0x3fffffff; };
    auto pub = [&](int r) { return gp[r] >= 0x40000000; };
    auto lp = [&](int r) { return (int)(lpe[r] & 0xffffu); };
    auto pe = [&](int r) { return (int)(lpe[r] >> 16); };
    auto eo = [&](int r) { return (int)(eol[r] & 0xfffffu); };
    auto el = [&](int r) { return (int)(eol[r] >> 20); };
    // the first halo row this thread polls (others through the table)
    const TileHalo h0 = tid < ti.nhalo ? a.halo[ti.halo0 + tid] : TileHalo{-1, 0};

    auto put = [&](int b, int q, T x, T y, T z) {
        XY(b)[q] = Pair<T>{x, y};
        Z(b)[q] = z;
    };
    auto own = [&](int b, int r, T& x, T& y, T& z) {
        const Pair<T> p = XY(b)[lp(r)];
        x = p.x;
        y = p.y;
        z = Z(b)[lp(r)];
    };
    unsigned tag = a.epoch0;  // of the last phase published
    auto words = [&](int w) { return a.ex + ((size_t)(tag & 1u) * kW + w) * a.nsim; };
    // publish one vector of row g under the current tag (slot w of the phase's words)
    auto publish = [&](int w, int g, T x, T y, T z) {
        if constexpr (sizeof(T) == 4) {
            st_word(words(w) + g, pack2(__float_as_uint(x), __float_as_uint(y)), pack2(__float_as_uint(z), tag));
        } else {
            st_word(words(0) + g, (unsigned long long)__double_as_longlong(x), tag);
            st_word(words(1) + g, (unsigned long long)__double_as_longlong(y), tag);
            st_word(words(2) + g, (unsigned long long)__double_as_longlong(z), tag);
        }
    };
    // cluster: the row's readers, whose shared memory this thread writes
    int4 to = make_int4(-1, -1, -1, -1);
    if constexpr (kCl)
        if (live(0)) to = __ldg(a.push + slot(0));
    auto push = [&](int b, int d, T x, T y, T z) {
        if (d < 0) return;
        const int q = d & 0xffff;
        st_remote(remote_addr(XY(b) + q, (unsigned)d >> 16), x, y);
        st_remote(remote_addr(Z(b) + q, (unsigned)d >> 16), z);
    };
    // row r's new vector (place b; word w of the phase) to whoever reads it
    auto send = [&](int w, int b, int r, T x, T y, T z) {
        if (!pub(r)) return;
        if constexpr (kCl) {
            push(b, to.x, x, y, z);
            push(b, to.y, x, y, z);
            push(b, to.z, x, y, z);
            push(b, to.w, x, y, z);
        } else {
            publish(w, row(r), x, y, z);
        }
    };
    // every CTA that might write here, or be written to, is at the same point
    auto sync_all = [&]() {
        if constexpr (kCl) cluster_sync();
        else sync();
    };
    // wait for the word at p to carry the current tag
    auto wait_word = [&](const TileWord* p, TileWord& w) -> bool {
        w = ld_word(p);
        auto there = [&]() { return sizeof(T) == 4 ? (unsigned)(w.hi >> 32) == tag : (unsigned)w.hi == tag; };
        if (there()) return true;
        const long long t0 = clock64();
        for (int n = 1;; ++n) {
            w = ld_word(p);
            if (there()) return true;
            if (clock64() - t0 > a.timeout) {
                atomicOr(a.err, (unsigned)kErrBarrier);
                return false;
            }
            if ((n & 15) == 0 && (ld_acquire(a.err) & kErrBarrier)) return false;
        }
    };
    // the halo of the current phase into vector b (and the second half into b2)
    auto fetch_one = [&](int row, int pos, int b, int b2) -> bool {
        TileWord w;
        if constexpr (sizeof(T) == 4) {
            if (!wait_word(words(0) + row, w)) return false;
            put(b, pos, __uint_as_float((unsigned)w.lo), __uint_as_float((unsigned)(w.lo >> 32)),
                __uint_as_float((unsigned)w.hi));
            if (b2 >= 0) {
                if (!wait_word(words(kW - 1) + row, w)) return false;
                put(b2, pos, __uint_as_float((unsigned)w.lo), __uint_as_float((unsigned)(w.lo >> 32)),
                    __uint_as_float((unsigned)w.hi));
            }
        } else {
            TileWord wy, wz;
            if (!wait_word(words(0) + row, w) || !wait_word(words(1) + row, wy) || !wait_word(words(2) + row, wz))
                return false;
            put(b, pos, __longlong_as_double((long long)w.lo), __longlong_as_double((long long)wy.lo),
                __longlong_as_double((long long)wz.lo));
        }
        return true;
    };
    auto fetch = [&](int b, int b2) -> bool {
        bool ok = h0.row < 0 || fetch_one(h0.row, h0.pos, b, b2);
        for (int h = tid + nthr; ok && h < ti.nhalo; h += nthr) {
            const TileHalo q = a.halo[ti.halo0 + h];
            ok = fetch_one(q.row, q.pos, b, b2);
        }
        return ok;
    };
    // end of a phase: the halo is in, every own value is written; false: the launch ends
    auto arrive = [&](int b, int b2 = -1) -> bool {
        if constexpr (kCl) {
            cluster_sync();
            return true;
        }
        if (ti.nhalo == 0) {
            sync();
            return true;
        }
        return !sync_or(!fetch(b, b2));
    };
    // tets only: what neighbours wrote to global memory before their same call
    // is visible after it (release and acquire of the tiles' phase counts)
    unsigned fl = a.flag0;
    auto global_sync = [&]() -> bool {
        sync();
        ++fl;
        if (tid == 0) st_release(a.flags + tile, fl);
        bool ok = true;
        const long long t0 = clock64();
        for (int q = tid; ok && q < ti.nnbr; q += nthr) {
            const int n = a.nbr[ti.nbr0 + q];
            while ((int)(ld_acquire(a.flags + n) - fl) < 0) {
                if (clock64() - t0 > a.timeout || (ld_acquire(a.err) & kErrBarrier)) {
                    atomicOr(a.err, (unsigned)kErrBarrier);
                    ok = false;
                    break;
                }
            }
        }
        return !sync_or(!ok);
    };

    // pairs: the values of a warp's 32 pairs go to 64 columns of tensor memory
    if constexpr (kPair) {
        const float4* vp = reinterpret_cast<const float4*>(a.val + ti.ent0 + eo(0));
        __syncwarp();
        for (int k = 0; k < el(0); k += 2) tmem_store4(tmem + 2 * k, __ldg(vp + 16 * k));
        tmem_store_wait();
    }
    // the same sums of both rows of a pair: each place is read once for the two,
    // each with its own values (zero where a row has no such column)
    auto pair_sum = [&](int b, T (&s)[R][3]) {
        if constexpr (kPair) {
#pragma unroll
            for (int r = 0; r < R; ++r) s[r][0] = s[r][1] = s[r][2] = T(0);
            const uint2* pp = reinterpret_cast<const uint2*>(spat + pe(0));
            const Pair<T>* xy = XY(b) + lp(0);
            const T* z = Z(b) + lp(0);
            __syncwarp();
            for (int k = 0; k < el(0); k += 4) {
                unsigned v[8];
                tmem_load8(tmem + 2 * k, v);
                const uint2 o2 = pp[k >> 2];
                const unsigned o[2] = {o2.x, o2.y};
                Pair<T> p[4];
                T q[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int j = (e & 1) ? (int)o[e >> 1] >> 16 : (int)(short)(o[e >> 1] & 0xffffu);
                    p[e] = xy[j];
                    q[e] = z[j];
                }
                tmem_wait8(v);
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        s[r][0] = fma_(__uint_as_float(v[2 * e + r]), p[e].x, s[r][0]);
                        s[r][1] = fma_(__uint_as_float(v[2 * e + r]), p[e].y, s[r][1]);
                        s[r][2] = fma_(__uint_as_float(v[2 * e + r]), q[e], s[r][2]);
                    }
            }
        }
    };
    // sum_k N_ik z_k of owned row r over vector b, in the stored order.  Batches
    // of entries whose loads are all in flight before the first sum: a 16-byte
    // load brings eight offsets (one address in most warps), another the values
    // of kG entries.
    auto row_sum = [&](int r, int b, T& s0, T& s1, T& s2) {
        s0 = T(0);
        s1 = T(0);
        s2 = T(0);
        const Group<T>* vp = reinterpret_cast<const Group<T>*>(sval + eo(r));
        const uint2* pp = reinterpret_cast<const uint2*>(spat + pe(r));
        const Pair<T>* xy = XY(b) + lp(r);
        const T* z = Z(b) + lp(r);
        auto batch = [&](auto nc, const unsigned* o, const T* v) {
            constexpr int n = decltype(nc)::value;
            Pair<T> p[n];
            T q[n];
#pragma unroll
            for (int k = 0; k < n; ++k) {
                const int j = (k & 1) ? (int)o[k >> 1] >> 16 : (int)(short)(o[k >> 1] & 0xffffu);
                p[k] = xy[j];
                q[k] = z[j];
            }
#pragma unroll
            for (int k = 0; k < n; ++k) {
                s0 = fma_(v[k], p[k].x, s0);
                s1 = fma_(v[k], p[k].y, s1);
                s2 = fma_(v[k], q[k], s2);
            }
        };
        int k = 0;
        if constexpr (kG == 4 && R == 1) {
            for (; k + 8 <= el(r); k += 8) {
                const uint4 o4 = *reinterpret_cast<const uint4*>(pp + (k >> 2));
                const unsigned o[4] = {o4.x, o4.y, o4.z, o4.w};
                const Group<T> va = vp[(k >> 2) * 32], vb = vp[(k >> 2) * 32 + 32];
                T v[8];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    v[q] = va.v[q];
                    v[4 + q] = vb.v[q];
                }
                batch(std::integral_constant<int, 8>(), o, v);
            }
        }
#pragma unroll(kUnroll)
        for (; k < el(r); k += 4) {
            const uint2 o2 = pp[k >> 2];
            const unsigned o[2] = {o2.x, o2.y};
            T v[4];
#pragma unroll
            for (int g = 0; g < 4 / kG; ++g) {
                const Group<T> va = vp[(k / kG + g) * 32];
#pragma unroll
                for (int q = 0; q < kG; ++q) v[g * kG + q] = va.v[q];
            }
            batch(std::integral_constant<int, 4>(), o, v);
        }
    };
    auto sum_of = [&](int r, int b, const T (&ps)[R][3], T& s0, T& s1, T& s2) {
        if constexpr (kPair) {
            s0 = ps[r][0];
            s1 = ps[r][1];
            s2 = ps[r][2];
        } else {
            row_sum(r, b, s0, s1, s2);
        }
    };
    const T w = a.relax, om1 = T(1) - a.relax;
    const bool kept_first = kCorr && (kCl || a.keptFirst);  // known in a cluster, whose sweeps it would lengthen by 3%

    // ---- positions of the local vertices: own rows and halo ----
    auto load_pos = [&](int row, int pos) {
        if constexpr (kCorr) {
            const V4<T> h = ldg_state(a.Ph, row), l = ldg_state(a.Pl, row);
            put(0, pos, h.x, h.y, h.z);
            put(1, pos, l.x, l.y, l.z);
        } else {
            const V4<S> x = ldg_state(a.P, row);
            put(0, pos, x.x, x.y, x.z);
        }
    };
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (live(r)) load_pos(row(r), lp(r));
    for (int h = tid; h < ti.nhalo; h += nthr) {
        const TileHalo q = a.halo[ti.halo0 + h];
        load_pos(q.row, q.pos);
    }
    sync_all();  // also: every CTA of a cluster runs before its shared memory is written

    const bool third = kCl || kPair || a.third;
    int cur = 0;  // the vector that holds the positions (direct form) at the start of an iteration
    for (int lg = 0; lg < a.lg; ++lg) {
        if constexpr (kTets) {
            for (int q = tid; q < ti.ntet; q += nthr)
                tet_element<S, kCorr>(a.tet[ti.tet0 + q], a.Tets, a.TetIdm, a.TetW, a.P, a.Ph, a.Pl, a.TetOut);
            if (!global_sync()) return finish();
        }
        // correction form: the residual's matrix part of owned row r, in column
        // order (the entries below the row's own block, those in it, those above)
        auto matrix_part = [&](int r, Acc& r0, Acc& r1, Acc& r2) {
            const T* vp = sval + eo(r);
            const int16_t* pp = spat + pe(r);
            const Pair<T>*hp = XY(0) + lp(r), *lpp = XY(1) + lp(r);
            const T *hz = Z(0) + lp(r), *lz = Z(1) + lp(r);
            const T h0x = hp[0].x, h0y = hp[0].y, h0z = hz[0], l0x = lpp[0].x, l0y = lpp[0].y, l0z = lz[0];
            auto part = [&](int k0, int k1) {
#pragma unroll 4
                for (int k = k0; k < k1; ++k) {
                    const T v = vp[32 * (k & ~(kG - 1)) + (k & (kG - 1))];
                    const int j = pp[k];
                    const Pair<T> p = hp[j], q = lpp[j];
                    r0.add(v, diff_ff(p.x, q.x, h0x, l0x));
                    r1.add(v, diff_ff(p.y, q.y, h0y, l0y));
                    r2.add(v, diff_ff(hz[j], lz[j], h0z, l0z));
                }
            };
            const int parts = __ldg(&a.slots[slot(r)].pub), ka = (parts >> 8) & 255, kb = (parts >> 16) & 255;
            part(ka, kb);
            part(0, ka);
            part(kb, el(r));
        };
        // the same for both rows of a pair.  The parts' bounds differ between lanes only
        // near a block's edge: the warp runs over all its lanes' ranges, each lane
        // adding its own.
        auto pair_matrix = [&](Acc (&ac)[kCorr ? R : 1][3]) {
            if constexpr (kPair && kCorr) {
                const int16_t* pp = spat + pe(0);
                const Pair<T>*hp = XY(0) + lp(0), *lpp = XY(1) + lp(0);
                const T *hz = Z(0) + lp(0), *lz = Z(1) + lp(0);
                T h[R][3], l[R][3];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    own(0, r, h[r][0], h[r][1], h[r][2]);
                    own(1, r, l[r][0], l[r][1], l[r][2]);
                }
                auto range = [&](int k0, int k1, int lo, int hi) {
                    for (int k = k0; k < k1; ++k) {
                        unsigned v[2];
                        tmem_load2(tmem + 2 * k, v);
                        const int j = pp[k];
                        const Pair<T> p = hp[j], q = lpp[j];
                        const T pz = hz[j], qz = lz[j];
                        tmem_wait2(v);
                        if (k >= lo && k < hi) {
#pragma unroll
                            for (int r = 0; r < R; ++r) {
                                const T vr = __uint_as_float(v[r]);
                                if (vr == T(0)) continue;  // its partner's column
                                ac[r][0].add(vr, diff_ff(p.x, q.x, h[r][0], l[r][0]));
                                ac[r][1].add(vr, diff_ff(p.y, q.y, h[r][1], l[r][1]));
                                ac[r][2].add(vr, diff_ff(pz, qz, h[r][2], l[r][2]));
                            }
                        }
                        __syncwarp();
                    }
                };
                const int n = el(0);
                if (n == 0) return;  // no slice
                const int parts = __ldg(&a.slots[slot(0)].pub), ka = (parts >> 8) & 255, kb = (parts >> 16) & 255;
                __syncwarp();
                range(__reduce_min_sync(~0u, ka), __reduce_max_sync(~0u, kb), ka, kb);
                range(0, __reduce_max_sync(~0u, ka), 0, ka);
                range(__reduce_min_sync(~0u, kb), n, kb, n);
            }
        };
        // ---- local step: curvature vectors, springs and (correction form without
        // a third vector) the matrix part of the residual, all from shared memory ----
        T aq[R][3], rh[R][3], px[R][3];
        Acc acc[kCorr ? R : 1][3];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            aq[r][0] = aq[r][1] = aq[r][2] = T(0);
            rh[r][0] = rh[r][1] = rh[r][2] = T(0);
            px[r][0] = px[r][1] = px[r][2] = T(0);
            if (!live(r)) continue;
            const int i = row(r);
            const int st = __ldg(a.stencil + ti.slice0 + slice(r)) + lane, nst = __ldg(&a.slots[slot(r)].pub) >> 24;
            const T strain = a.Strain[i];
            T a0, a1, a2;
            if constexpr (kCorr) {
                Acc r0, r1, r2;
                const V4<S> x = ldg_state(a.P, i);
                {
                    const V4<S> y = ldg_state(a.Rhs0, i);
                    const T di = a.Dinert[i];
                    r0.add(di, (T)(y.x - x.x));
                    r1.add(di, (T)(y.y - x.y));
                    r2.add(di, (T)(y.z - x.z));
                }
                const int pf = a.PinFlag[i];
                if (pf >= 0) {
                    const V4<S> xr = ldg_state(a.Xrest, i);
                    const T k = a.PinK[pf];
                    r0.add(k, (T)(xr.x - x.x));
                    r1.add(k, (T)(xr.y - x.y));
                    r2.add(k, (T)(xr.z - x.z));
                }
                {
                    const T dc = a.CollDiag[i];
                    if (dc != T(0)) {  // else both terms are zero
                    const V4<T> c = ldg_state(a.CollRhs, i);
                    const V4<S> xo = ldg_state(a.Pold, i);
                    r0.add(c.x);
                    r0.add(dc, (T)(xo.x - x.x));
                    r1.add(c.y);
                    r1.add(dc, (T)(xo.y - x.y));
                    r2.add(c.z);
                    r2.add(dc, (T)(xo.z - x.z));
                    }
                }
                const Pair<T>*hp = XY(0) + lp(r), *lpp = XY(1) + lp(r);
                const T *hz = Z(0) + lp(r), *lz = Z(1) + lp(r);
                const T h0x = hp[0].x, h0y = hp[0].y, h0z = hz[0], l0x = lpp[0].x, l0y = lpp[0].y, l0z = lz[0];
                a0 = a1 = a2 = T(0);
#pragma unroll 4
                for (int k = 0; k < nst; ++k) {
                    const int j = __ldg(a.stPos + st + 32 * k);
                    const Pair<T> hj = hp[j], lj = lpp[j];
                    const T hjz = hz[j], ljz = lz[j];
                    const T d0 = diff_ff(h0x, l0x, hj.x, lj.x), d1 = diff_ff(h0y, l0y, hj.y, lj.y),
                            d2 = diff_ff(h0z, l0z, hjz, ljz);
                    const T wl = __ldg(a.stLbo + st + 32 * k);
                    a0 = fma_(wl, -d0, a0);
                    a1 = fma_(wl, -d1, a1);
                    a2 = fma_(wl, -d2, a2);
                    const T cl = dsqrt(norm2(d0, d1, d2));
                    const T rc = strain * (__ldg(a.stRest + st + 32 * k) / cl);
                    r0.add(rc, d0);
                    r1.add(rc, d1);
                    r2.add(rc, d2);
                }
                if (!third) matrix_part(r, r0, r1, r2);
                acc[r][0] = r0;
                acc[r][1] = r1;
                acc[r][2] = r2;
            } else {
                const Pair<T>* xp = XY(cur) + lp(r);
                const T* xz = Z(cur) + lp(r);
                const T x0 = xp[0].x, x1 = xp[0].y, x2 = xz[0];
                const T l0 = a.tLbo0[i];
                a0 = x0 * l0;
                a1 = x1 * l0;
                a2 = x2 * l0;
                T t0 = T(0), t1 = T(0), t2 = T(0);
#pragma unroll 4
                for (int k = 0; k < nst; ++k) {
                    const int j = __ldg(a.stPos + st + 32 * k);
                    const Pair<T> xj = xp[j];
                    const T xjz = xz[j];
                    const T l = __ldg(a.stLbo + st + 32 * k);
                    a0 = fma_(xj.x, l, a0);
                    a1 = fma_(xj.y, l, a1);
                    a2 = fma_(xjz, l, a2);
                    const T d0 = x0 - xj.x, d1 = x1 - xj.y, d2 = x2 - xjz;
                    const T cl = dsqrt(norm2(d0, d1, d2));
                    const T rc = strain * (__ldg(a.stRest + st + 32 * k) / cl);
                    t0 = fma_(rc, d0, t0);
                    t1 = fma_(rc, d1, t1);
                    t2 = fma_(rc, d2, t2);
                }
                rh[r][0] = t0;
                rh[r][1] = t1;
                rh[r][2] = t2;
                if (a.tape) a.tape[(size_t)lg * a.nsim + i] = V4<T>{x0, x1, x2, T(0)};
            }
            const T nrm = dsqrt(norm2(a0, a1, a2));
            if (nrm >= T(1e-10)) {
                const T c = a.CurvNorm[i] / nrm;
                a0 *= c;
                a1 *= c;
                a2 *= c;
            }
            aq[r][0] = a0;
            aq[r][1] = a1;
            aq[r][2] = a2;
        }
        // ---- the curvature vectors go into the third vector, or where the
        // positions' high halves were (correction form), or into the free vector
        // (direct form) ----
        const int qb = kCorr ? (third ? 2 : 0) : cur ^ 1;
        if (kCorr && !third) sync_all();
        ++tag;
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (live(r)) {
                send(0, qb, r, aq[r][0], aq[r][1], aq[r][2]);
                put(qb, lp(r), aq[r][0], aq[r][1], aq[r][2]);
            }
        if (!arrive(qb)) return finish();
        // ---- bending, then the right-hand side (direct) or residual (correction) ----
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (!live(r)) continue;
            const int i = row(r);
            const int st = __ldg(a.stencil + ti.slice0 + slice(r)) + lane, nst = __ldg(&a.slots[slot(r)].pub) >> 24;
            const Pair<T>* qp = XY(qb) + lp(r);
            const T* qz = Z(qb) + lp(r);
            const T b0 = a.tBend0[i];
            if constexpr (kCorr) {
                Acc r0 = acc[r][0], r1 = acc[r][1], r2 = acc[r][2];
                r0.add(b0, aq[r][0]);
                r1.add(b0, aq[r][1]);
                r2.add(b0, aq[r][2]);
#pragma unroll 4
                for (int k = 0; k < nst; ++k) {
                    const int j = __ldg(a.stPos + st + 32 * k);
                    const T bt = __ldg(a.stBend + st + 32 * k);
                    r0.add(bt, qp[j].x);
                    r1.add(bt, qp[j].y);
                    r2.add(bt, qz[j]);
                }
                if constexpr (kTets)
                    for (int q = a.vtPtr[i]; q < a.vtPtr[i + 1]; ++q) {
                        const float4 t = __ldcg((const float4*)a.TetOut + a.vtIdx[q]);
                        r0.add(t.x);
                        r1.add(t.y);
                        r2.add(t.z);
                    }
                if constexpr (kPair) {
                    acc[r][0] = r0;
                    acc[r][1] = r1;
                    acc[r][2] = r2;
                    continue;
                }
                if (third) matrix_part(r, r0, r1, r2);
                rh[r][0] = r0.value();
                rh[r][1] = r1.value();
                rh[r][2] = r2.value();
            } else {
                T t0 = rh[r][0], t1 = rh[r][1], t2 = rh[r][2];
                t0 = fma_(b0, aq[r][0], t0);
                t1 = fma_(b0, aq[r][1], t1);
                t2 = fma_(b0, aq[r][2], t2);
                const V4<S> q0 = ldg_state(a.Rhs0, i);
                T u0 = q0.x + t0, u1 = q0.y + t1, u2 = q0.z + t2;
#pragma unroll 4
                for (int k = 0; k < nst; ++k) {
                    const int j = __ldg(a.stPos + st + 32 * k);
                    const T bt = __ldg(a.stBend + st + 32 * k);
                    u0 = fma_(bt, qp[j].x, u0);
                    u1 = fma_(bt, qp[j].y, u1);
                    u2 = fma_(bt, qz[j], u2);
                }
                if constexpr (kTets)
                    for (int q = a.vtPtr[i]; q < a.vtPtr[i + 1]; ++q) {
                        const float4 t = __ldcg((const float4*)a.TetOut + a.vtIdx[q]);
                        u0 += t.x;
                        u1 += t.y;
                        u2 += t.z;
                    }
                const V4<T> cr = ldg_state(a.CollRhs, i);
                u0 += cr.x;
                u1 += cr.y;
                u2 += cr.z;
                const V4<T> pn = ldg_state(a.PinRhs, i);
                u0 += pn.x;
                u1 += pn.y;
                u2 += pn.z;
                rh[r][0] = u0;
                rh[r][1] = u1;
                rh[r][2] = u2;
            }
        }

        if constexpr (kPair && kCorr) {
            pair_matrix(acc);
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (live(r)) {
                    rh[r][0] = acc[r][0].value();
                    rh[r][1] = acc[r][1].value();
                    rh[r][2] = acc[r][2].value();
                }
        }

        // ---- Chebyshev-accelerated R2 iteration as two J sweeps per step ----
        // direct form: on x from the positions; correction form: on delta from 0
        ++tag;
        {
            T y[R][3], ps[R][3];
            if (kPair && !kCorr) pair_sum(cur, ps);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                T s0 = T(0), s1 = T(0), s2 = T(0);
                T c0 = T(0), c1 = T(0), c2 = T(0);
                if (!kCorr) {
                    sum_of(r, cur, ps, s0, s1, s2);
                    own(cur, r, c0, c1, c2);
                }
                y[r][0] = jacobi(om1, c0, w, s0, rh[r][0], id[r], kept_first);
                y[r][1] = jacobi(om1, c1, w, s1, rh[r][1], id[r], kept_first);
                y[r][2] = jacobi(om1, c2, w, s2, rh[r][2], id[r], kept_first);
                if (!kCl && pub(r)) publish(0, row(r), y[r][0], y[r][1], y[r][2]);
            }
            // the curvature vectors (direct form), or the positions, have been read
            if (!kCorr || third) sync_all();
            cur = kCorr ? 1 : cur ^ 1;
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (live(r)) {
                    if (kCl) send(0, cur, r, y[r][0], y[r][1], y[r][2]);
                    put(cur, lp(r), y[r][0], y[r][1], y[r][2]);
                }
        }
        if (!arrive(cur)) return finish();
        for (int it = 0; it < a.cheby; ++it) {
            const bool last = it == a.cheby - 1;
            const T om = a.omega[it];
            // x = S(y), Chebyshev-combined with the step before the last
            ++tag;
            T ps[R][3];
            pair_sum(cur, ps);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                T s0, s1, s2, n[3];
                sum_of(r, cur, ps, s0, s1, s2);
                T c0, c1, c2;
                own(cur, r, c0, c1, c2);
                n[0] = jacobi(om1, c0, w, s0, rh[r][0], id[r], kept_first);
                n[1] = jacobi(om1, c1, w, s1, rh[r][1], id[r], kept_first);
                n[2] = jacobi(om1, c2, w, s2, rh[r][2], id[r], kept_first);
                if (it > 0) {
                    n[0] = fma_(om, add_(n[0], -px[r][0]), px[r][0]);
                    n[1] = fma_(om, add_(n[1], -px[r][1]), px[r][1]);
                    n[2] = fma_(om, add_(n[2], -px[r][2]), px[r][2]);
                }
                // the next step's step before last: the other vector still holds this
                // row's current x (the correction starts from zero)
                if (kCorr && last) {
                    px[r][0] = n[0];
                    px[r][1] = n[1];
                    px[r][2] = n[2];
                } else if (!kCorr || it > 0) {
                    own(cur ^ 1, r, px[r][0], px[r][1], px[r][2]);
                }
                if (!live(r)) continue;
                if (!(kCorr && last)) {
                    send(0, cur ^ 1, r, n[0], n[1], n[2]);
                    put(cur ^ 1, lp(r), n[0], n[1], n[2]);
                }
                if (!kCorr && last && (kTets || lg == a.lg - 1)) a.P[row(r)] = V4<S>{n[0], n[1], n[2], S(0)};
            }
            if (last) break;
            cur ^= 1;
            if (!arrive(cur)) return finish();
            // y = S(x)
            ++tag;
            pair_sum(cur, ps);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                T s0, s1, s2;
                sum_of(r, cur, ps, s0, s1, s2);
                T c0, c1, c2;
                own(cur, r, c0, c1, c2);
                const T y0 = jacobi(om1, c0, w, s0, rh[r][0], id[r], kept_first);
                const T y1 = jacobi(om1, c1, w, s1, rh[r][1], id[r], kept_first);
                const T y2 = jacobi(om1, c2, w, s2, rh[r][2], id[r], kept_first);
                if (!live(r)) continue;
                send(0, cur ^ 1, r, y0, y1, y2);
                put(cur ^ 1, lp(r), y0, y1, y2);
            }
            cur ^= 1;
            if (!arrive(cur)) return finish();
        }
        // ---- the new positions ----
        if constexpr (kCorr) {
            sync_all();  // both vectors have been read
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (!live(r)) continue;
                const V4<S> x = ldg_state(a.P, row(r));
                const S q0 = x.x + (S)px[r][0], q1 = x.y + (S)px[r][1], q2 = x.z + (S)px[r][2];
                a.P[row(r)] = V4<S>{q0, q1, q2, S(0)};
                float hx, lx, hy, ly, hz, lz;
                split_ff(q0, hx, lx);
                split_ff(q1, hy, ly);
                split_ff(q2, hz, lz);
                if (kTets || lg == a.lg - 1) {
                    a.Ph[row(r)] = V4<T>{hx, hy, hz, T(0)};
                    a.Pl[row(r)] = V4<T>{lx, ly, lz, T(0)};
                }
                send(0, 0, r, hx, hy, hz);
                send(1, 1, r, lx, ly, lz);
                put(0, lp(r), hx, hy, hz);
                put(1, lp(r), lx, ly, lz);
            }
            if (lg == a.lg - 1) break;
            if (!arrive(0, 1)) return finish();
        } else {
            cur ^= 1;
            if (lg == a.lg - 1) break;
            if (!arrive(cur)) return finish();
        }
        if constexpr (kTets)
            if (!global_sync()) return finish();
    }
    if constexpr (kCl) cluster_sync();  // nobody leaves while another may write to its shared memory
    finish();
}

template <typename T, typename S>
const void* tile_kernel(int R, bool tets, bool pairs) {
    constexpr bool kCorr = !std::is_same<T, S>::value;
    if constexpr (sizeof(T) == 8) {
        return tets || pairs || R != 1 ? nullptr : (const void*)k_pd_tile<T, S, kCorr, false, 1, kWords>;
    } else {
        if (R != 1 && R != 2) return nullptr;
        if (pairs) return tets || R != 2 ? nullptr : (const void*)k_pd_tile<T, S, kCorr, false, 2, kPairs>;
        if (tets) return R == 1 ? (const void*)k_pd_tile<T, S, kCorr, true, 1, kWords> : (const void*)k_pd_tile<T, S, kCorr, true, 2, kWords>;
        return R == 1 ? (const void*)k_pd_tile<T, S, kCorr, false, 1, kWords> : (const void*)k_pd_tile<T, S, kCorr, false, 2, kWords>;
    }
}

// Pairs: the CTA's tiles, and more than half of an SM's shared memory: the CTA takes all
// columns of tensor memory, so another launch's must not share the SM.
size_t cta_smem(bool pairs, size_t smem) {
    return pairs ? std::max(kPairTiles * smem, (size_t)(116 * 1024)) : smem;
}

}  // namespace

template <typename T, typename S>
int tile_residents(int R, bool tets, bool pairs, int threads, size_t smem, int sms) {
    const void* f = tile_kernel<T, S>(R, tets, pairs);
    if (!f || threads > kTileMaxWarps * 32) return 0;
    smem = cta_smem(pairs, smem);
    if (allow_smem(f, smem) != cudaSuccess) return 0;
    int per_sm = 0;
    const int per_cta = pairs ? kPairTiles : 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, threads * per_cta, smem) != cudaSuccess)
        return 0;
    return per_sm * sms * per_cta;
}

template <typename T, typename S>
cudaError_t launch_pd_tile(const TileArgs<T, S>& args, int tiles, int R, bool tets, bool pairs, int threads, size_t smem,
                           cudaStream_t s) {
    const void* f = tile_kernel<T, S>(R, tets, pairs);
    if (!f || tiles < 1) return cudaErrorInvalidConfiguration;
    void* params[] = {(void*)&args};
    const int per_cta = pairs ? kPairTiles : 1;
    return cudaLaunchCooperativeKernel(f, dim3((tiles + per_cta - 1) / per_cta), dim3(threads * per_cta), params,
                                       cta_smem(pairs, smem), s);
}

namespace {

template <typename T, typename S>
const void* cluster_kernel() {
    return (const void*)k_pd_tile<T, S, !std::is_same<T, S>::value, false, 1, kCluster>;
}
cudaLaunchConfig_t cluster_config(int tiles, int threads, size_t smem, cudaStream_t s, cudaLaunchAttribute* at) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(tiles);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = tiles;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = 1;
    return c;
}

}  // namespace

template <typename T, typename S>
bool tile_cluster_fits(int tiles, int threads, size_t smem) {
    if constexpr (sizeof(T) == 8) {
        return false;
    } else {
        const void* f = cluster_kernel<T, S>();
        if (threads > kTileMaxWarps * 32 || tiles > kTileCluster) return false;
        if (allow_smem(f, smem) != cudaSuccess) return false;
        if (cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return false;
        cudaLaunchAttribute at;
        const cudaLaunchConfig_t c = cluster_config(tiles, threads, smem, nullptr, &at);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, f, &c) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return n > 0;
    }
}

template <typename T, typename S>
cudaError_t launch_pd_tile_cluster(const TileArgs<T, S>& args, int tiles, int threads, size_t smem,
                                   cudaStream_t s) {
    if constexpr (sizeof(T) == 8) {
        return cudaErrorInvalidConfiguration;
    } else {
        cudaLaunchAttribute at;
        const cudaLaunchConfig_t c = cluster_config(tiles, threads, smem, s, &at);
        void* params[] = {(void*)&args};
        return cudaLaunchKernelExC(&c, cluster_kernel<T, S>(), params);
    }
}

#define PDIPC_INST_TILE(T, S)                                                                     \
    template int tile_residents<T, S>(int, bool, bool, int, size_t, int);                         \
    template bool tile_cluster_fits<T, S>(int, int, size_t);                                      \
    template cudaError_t launch_pd_tile_cluster<T, S>(const TileArgs<T, S>&, int, int, size_t,    \
                                                      cudaStream_t);                              \
    template cudaError_t launch_pd_tile<T, S>(const TileArgs<T, S>&, int, int, bool, bool, int, size_t, \
                                              cudaStream_t);
PDIPC_INST_TILE(float, float)
PDIPC_INST_TILE(float, double)
PDIPC_INST_TILE(double, double)

}  // namespace pdipc
