// pd_tile3.cu — the tiled PD solve (pd_tile.cu) in FP64, one component of a row
// per thread.
//
// FP64 instructions are what bounds it: a warp's takes its scheduler's FP64 unit
// for 64 cycles, so a row of 24 entries costs a thread that does all three
// components at least 2.5 us a sweep, whatever the size of the tile.  Here the
// tile's warps come in three groups, one per component, each over all of the
// tile's slices: a third of the chain per thread, three times the warps, the same
// number of FP64 instructions.  The local step, whose norms need all three
// components, is dealt out by slices instead, and hands its right-hand sides over
// in shared memory.  One tile per SM: past a few hundred rows the FP64 units are
// busy throughout and a second tile would only add halo.
//
// Every component goes through the operations of pd_tile.cu in the same order.
#include <algorithm>
#include <type_traits>

#include "smem_limit.h"
#include "tile_device.cuh"

namespace pdipc {

namespace {

using F = double;

__global__ void __launch_bounds__(kTile3Warps * 96, 1) k_pd_tile3(const __grid_constant__ TileArgs<F, F> a) {
    extern __shared__ __align__(16) unsigned char smem[];
    if (outer_stopped(a.gate)) return;
    const int tile = (int)blockIdx.x + a.lo;
    const TileInfo ti = a.tiles[tile];
    if (a.instStop && a.instStop[ti.model]) return;
    const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31;
    const int nw = nth / 96;              // warps per component
    const int comp = (tid >> 5) / nw, warp = (tid >> 5) % nw;

    // ---- shared memory: values, offset patterns, two vectors of the local
    // vertices in three planes, right-hand sides by slot ----
    auto a16 = [](size_t b) { return (b + 15) / 16 * 16; };
    F* sval = reinterpret_cast<F*>(smem);
    int16_t* spat = reinterpret_cast<int16_t*>(smem + a16((size_t)ti.nent * sizeof(F)));
    F* vec = reinterpret_cast<F*>(smem + a16((size_t)ti.nent * sizeof(F)) +
                                  a16((size_t)ti.npat * a.patStride * sizeof(int16_t)));
    const int nl = ti.nloc;
    auto plane = [&](int b, int c) { return vec + (size_t)(3 * b + c) * nl; };
    F* srhs = vec + 6 * (size_t)nl;
    const int nslot = 32 * ti.nslice;
    for (int q = tid; q < ti.nent; q += nth) sval[q] = __ldg(a.val + ti.ent0 + q);
    for (int q = tid; q < ti.npat * a.patStride; q += nth)
        spat[q] = __ldg(a.pat + (size_t)ti.pat0 * a.patStride + q);

    // ---- this thread's row (component comp): slice warp, this lane ----
    int row = -1, pos = 0, el = 0;
    bool pub = false;
    const F* mv = sval;         // its entries' values
    const int16_t* mp = spat;   // and offsets
    F id = 0.0;
    if (warp < ti.nslice) {
        const TileSlot sl = a.slots[ti.slot0 + 32 * warp + lane];
        const TileSlice sc = a.slices[ti.slice0 + warp];
        if (sl.row >= 0) {
            row = sl.row;
            pos = sl.pos;
            el = sc.len;
            pub = sl.pub & 1;
            mv = sval + sc.off + 2 * lane;
            mp = spat + sl.pat;
            id = 1.0 / ((a.Delastic[row] + a.Dinert[row]) + a.CollDiag[row]);
        }
    }

    unsigned tag = a.epoch0;  // of the last phase published
    auto words = [&](int w) { return a.ex + ((size_t)(tag & 1u) * 3 + w) * a.nsim; };
    auto publish = [&](int c, int g, F v) { st_word(words(c) + g, (unsigned long long)__double_as_longlong(v), tag); };
    // the halo of the current phase into vector b, a component of a row per item
    auto fetch = [&](int b) -> bool {
        for (int q = tid; q < 3 * ti.nhalo; q += nth) {
            const int c = q / ti.nhalo;
            const TileHalo h = a.halo[ti.halo0 + q - c * ti.nhalo];
            const TileWord* p = words(c) + h.row;
            TileWord w = ld_word(p);
            if ((unsigned)w.hi != tag) {
                const long long t0 = clock64();
                for (int n = 1;; ++n) {
                    w = ld_word(p);
                    if ((unsigned)w.hi == tag) break;
                    if (clock64() - t0 > a.timeout) {
                        atomicOr(a.err, (unsigned)kErrBarrier);
                        return false;
                    }
                    if ((n & 15) == 0 && (ld_acquire(a.err) & kErrBarrier)) return false;
                }
            }
            plane(b, c)[h.pos] = __longlong_as_double((long long)w.lo);
        }
        return true;
    };
    // end of a phase: the halo is in, every own value is written; false: the launch ends
    auto arrive = [&](int b) -> bool {
        if (ti.nhalo == 0) {
            __syncthreads();
            return true;
        }
        return !__syncthreads_or(!fetch(b));
    };

    // sum_k N_ik z_k of this thread's row and component over vector b: batches of
    // entries whose loads are all in flight before the first sum
    auto row_sum = [&](int b) -> F {
        F s = 0.0;
        const Group<F>* vp = reinterpret_cast<const Group<F>*>(mv);
        const uint2* pp = reinterpret_cast<const uint2*>(mp);
        const F* z = plane(b, comp) + pos;
#pragma unroll 2
        for (int k = 0; k < el; k += 4) {
            const uint2 o = pp[k >> 2];
            const Group<F> va = vp[(k >> 1) * 32], vb = vp[(k >> 1) * 32 + 32];
            const F z0 = z[(int)(short)(o.x & 0xffffu)], z1 = z[(int)o.x >> 16];
            const F z2 = z[(int)(short)(o.y & 0xffffu)], z3 = z[(int)o.y >> 16];
            s = fma_(va.v[0], z0, s);
            s = fma_(va.v[1], z1, s);
            s = fma_(vb.v[0], z2, s);
            s = fma_(vb.v[1], z3, s);
        }
        return s;
    };
    const F w = a.relax, om1 = 1.0 - a.relax;

    // ---- positions of the local vertices ----
    auto load_pos = [&](int g, int pos) {
        const V4<F> x = a.P[g];
        plane(0, 0)[pos] = x.x;
        plane(0, 1)[pos] = x.y;
        plane(0, 2)[pos] = x.z;
    };
    for (int q = tid; q < nslot; q += nth) {
        const TileSlot sl = a.slots[ti.slot0 + q];
        if (sl.row >= 0) load_pos(sl.row, sl.pos);
    }
    for (int h = tid; h < ti.nhalo; h += nth) {
        const TileHalo q = a.halo[ti.halo0 + h];
        load_pos(q.row, q.pos);
    }
    __syncthreads();

    int cur = 0;
    for (int lg = 0; lg < a.lg; ++lg) {
        // ---- local step, all components, by slices: warp k takes slice k (there are
        // three times as many warps) ----
        const int s = tid >> 5;
        TileSlot sl{-1, 0, 0, 0};
        if (s < ti.nslice) sl = a.slots[ti.slot0 + 32 * s + lane];
        const int i = sl.row, nst = sl.pub >> 24;
        const int st = sl.row >= 0 ? __ldg(a.stencil + ti.slice0 + s) + lane : 0;
        F t0 = 0.0, t1 = 0.0, t2 = 0.0, a0 = 0.0, a1 = 0.0, a2 = 0.0;
        ++tag;
        if (sl.row >= 0) {
            const F strain = a.Strain[i], l0 = a.tLbo0[i];
            const F *X = plane(cur, 0) + sl.pos, *Y = plane(cur, 1) + sl.pos, *Z = plane(cur, 2) + sl.pos;
            const F x0 = X[0], x1 = Y[0], x2 = Z[0];
            a0 = mul_(x0, l0);
            a1 = mul_(x1, l0);
            a2 = mul_(x2, l0);
#pragma unroll 4
            for (int k = 0; k < nst; ++k) {
                const int j = __ldg(a.stPos + st + 32 * k);
                const F y0 = X[j], y1 = Y[j], y2 = Z[j], lb = __ldg(a.stLbo + st + 32 * k);
                a0 = fma_(y0, lb, a0);
                a1 = fma_(y1, lb, a1);
                a2 = fma_(y2, lb, a2);
                const F d0 = add_(x0, -y0), d1 = add_(x1, -y1), d2 = add_(x2, -y2);
                const F cl = dsqrt(norm2(d0, d1, d2));
                const F rc = mul_(strain, __ldg(a.stRest + st + 32 * k) / cl);
                t0 = fma_(rc, d0, t0);
                t1 = fma_(rc, d1, t1);
                t2 = fma_(rc, d2, t2);
            }
            const F nrm = dsqrt(norm2(a0, a1, a2));
            if (nrm >= 1e-10) {
                const F c = a.CurvNorm[i] / nrm;
                a0 = mul_(a0, c);
                a1 = mul_(a1, c);
                a2 = mul_(a2, c);
            }
            if (sl.pub & 1) {
                publish(0, i, a0);
                publish(1, i, a1);
                publish(2, i, a2);
            }
            plane(cur ^ 1, 0)[sl.pos] = a0;
            plane(cur ^ 1, 1)[sl.pos] = a1;
            plane(cur ^ 1, 2)[sl.pos] = a2;
            if (a.tape) a.tape[(size_t)lg * a.nsim + i] = V4<F>{x0, x1, x2, 0.0};
        }
        if (!arrive(cur ^ 1)) return;
        if (sl.row >= 0) {
            const F *X = plane(cur ^ 1, 0) + sl.pos, *Y = plane(cur ^ 1, 1) + sl.pos, *Z = plane(cur ^ 1, 2) + sl.pos;
            const F b0 = a.tBend0[i];
            const V4<F> q0 = a.Rhs0[i], cr = a.CollRhs[i], pn = a.PinRhs[i];
            F u0 = add_(q0.x, fma_(b0, a0, t0)), u1 = add_(q0.y, fma_(b0, a1, t1)), u2 = add_(q0.z, fma_(b0, a2, t2));
#pragma unroll 4
            for (int k = 0; k < nst; ++k) {
                const int j = __ldg(a.stPos + st + 32 * k);
                const F bt = __ldg(a.stBend + st + 32 * k);
                u0 = fma_(bt, X[j], u0);
                u1 = fma_(bt, Y[j], u1);
                u2 = fma_(bt, Z[j], u2);
            }
            srhs[32 * s + lane] = add_(add_(u0, cr.x), pn.x);
            srhs[nslot + 32 * s + lane] = add_(add_(u1, cr.y), pn.y);
            srhs[2 * nslot + 32 * s + lane] = add_(add_(u2, cr.z), pn.z);
        }
        // ---- first sweep; its sums read the positions, which stay ----
        ++tag;
        F y = row_sum(cur), rh = 0.0, px = 0.0;
        __syncthreads();  // the right-hand sides are there, and the curvature vectors have been read
        if (row >= 0) {
            rh = srhs[comp * nslot + 32 * warp + lane];
            y = jacobi(om1, plane(cur, comp)[pos], w, y, rh, id, false);
            if (pub) publish(comp, row, y);
            plane(cur ^ 1, comp)[pos] = y;
        }
        cur ^= 1;
        if (!arrive(cur)) return;
        for (int it = 0; it < a.cheby; ++it) {
            const bool last = it == a.cheby - 1;
            const F om = a.omega[it];
            ++tag;
            F n = jacobi(om1, plane(cur, comp)[pos], w, row_sum(cur), rh, id, false);
            if (it > 0) n = fma_(om, add_(n, -px), px);
            px = plane(cur ^ 1, comp)[pos];  // still this row's current x
            if (row >= 0) {
                if (pub) publish(comp, row, n);
                plane(cur ^ 1, comp)[pos] = n;
                if (last && lg == a.lg - 1) reinterpret_cast<F*>(a.P + row)[comp] = n;
            }
            cur ^= 1;
            if (last) break;
            if (!arrive(cur)) return;
            ++tag;
            const F v = jacobi(om1, plane(cur, comp)[pos], w, row_sum(cur), rh, id, false);
            if (row >= 0) {
                if (pub) publish(comp, row, v);
                plane(cur ^ 1, comp)[pos] = v;
            }
            cur ^= 1;
            if (!arrive(cur)) return;
        }
        if (lg == a.lg - 1) break;
        if (!arrive(cur)) return;
    }
}

}  // namespace

int tile3_residents(int threads, size_t smem, int sms) {
    const void* f = (const void*)k_pd_tile3;
    if (threads > kTile3Warps * 96) return 0;
    if (allow_smem(f, smem) != cudaSuccess) return 0;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, threads, smem) != cudaSuccess) return 0;
    return per_sm * sms;
}

cudaError_t launch_pd_tile3(const TileArgs<double, double>& args, int tiles, int threads, size_t smem, cudaStream_t s) {
    if (tiles < 1) return cudaErrorInvalidConfiguration;
    void* params[] = {(void*)&args};
    return cudaLaunchCooperativeKernel((const void*)k_pd_tile3, dim3(tiles), dim3(threads), params, smem, s);
}

}  // namespace pdipc
