// Checks of csrc/geometry.cuh, compiled for the host.  Prints "ok" or what failed.
//   * The closest-point distances where their weights degenerate: parallel, collinear,
//     coincident and zero-length edges, triangles without area, NaN.  The weights go in
//     poisoned and must come out set, in [0, 1] for finite input, with the distance of
//     the best end (edge) in long double.
//   * The FP32 exit of the time-of-impact filters on rounded coordinates: wherever it
//     says 1, the FP64 test must return 1, near its margins, far from the origin, on
//     parallel edges, parted along an axis or a diagonal, with conservative steps and
//     without.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>

#include "host_cuda.h"
#include "geometry.cuh"

using namespace pdipc;
typedef long double LD;

static LD seg(const LD* p, const LD* a, const LD* b) {  // squared distance point - segment
    LD ab[3], t = 0, n = 0, s = 0;
    for (int k = 0; k < 3; ++k) {
        ab[k] = b[k] - a[k];
        t += (p[k] - a[k]) * ab[k];
        n += ab[k] * ab[k];
    }
    t = n > 0 ? std::fmin(std::fmax(t / n, (LD)0), (LD)1) : 0;
    for (int k = 0; k < 3; ++k) s += (p[k] - a[k] - t * ab[k]) * (p[k] - a[k] - t * ab[k]);
    return s;
}

// extent 1 coordinates on a dyadic lattice, so that the degeneracy survives rounding:
// the distance's own arithmetic is then within 64 roundings of the exact square
template <typename R>
static bool distances() {
    const LD tol = 64 * (LD)std::numeric_limits<R>::epsilon();
    const R poison = R(1e30);
    std::mt19937 g(7);
    auto lat = [&](int n) { return (R)((int)(g() % (2 * n + 1)) - n) / R(8); };
    for (int trial = 0; trial < 20000; ++trial) {
        R x[4][3], dir[3], d[3];
        for (int k = 0; k < 3; ++k) dir[k] = lat(8);
        const int kind = trial % 4;
        const R la = kind == 2 ? R(0) : lat(4), lb = kind == 3 ? R(0) : lat(4);  // lengths along dir: zero ones too
        for (int k = 0; k < 3; ++k) {
            x[0][k] = lat(8);
            x[1][k] = x[0][k] + la * dir[k];
            x[2][k] = kind == 1 ? x[0][k] + R(0.5) * dir[k] : lat(8);  // 1: collinear edges
            x[3][k] = x[2][k] + lb * dir[k];
        }
        LD y[4][3];
        for (int j = 0; j < 4; ++j)
            for (int k = 0; k < 3; ++k) y[j][k] = x[j][k];
        R r = poison, s = poison;
        const R e = geo::edge_edge_sq(x[0], x[1], x[2], x[3], &r, &s, d);
        LD best = std::fmin(std::fmin(seg(y[0], y[2], y[3]), seg(y[1], y[2], y[3])),
                            std::fmin(seg(y[2], y[0], y[1]), seg(y[3], y[0], y[1])));
        if (!(r >= 0 && r <= 1 && s >= 0 && s <= 1) || std::fabs((LD)e - best) > tol * 12) {
            printf("edges, trial %d: r %g s %g d2 %.9g, %.9Lg expected\n", trial, (double)r, (double)s, (double)e, best);
            return false;
        }
        // a triangle without area: its corners on one line (or one point)
        R a = poison, b = poison, c = poison, t[3][3];
        const R l1 = kind == 2 ? R(0) : lat(4), l2 = kind == 3 ? l1 : lat(4);
        for (int k = 0; k < 3; ++k) {
            t[0][k] = x[2][k];
            t[1][k] = x[2][k] + l1 * dir[k];
            t[2][k] = x[2][k] + l2 * dir[k];
        }
        for (int j = 0; j < 3; ++j)
            for (int k = 0; k < 3; ++k) y[1 + j][k] = t[j][k];
        const R f = geo::vtx_tri(x[0], t[0], t[1], t[2], &a, &b, &c, d);
        best = std::fmin(seg(y[0], y[1], y[2]), std::fmin(seg(y[0], y[2], y[3]), seg(y[0], y[1], y[3])));
        if (!(a >= 0 && a <= 1 && b >= 0 && b <= 1 && c >= 0 && c <= 1) || std::fabs((LD)f - best) > tol * 12) {
            printf("triangle, trial %d: %g %g %g d2 %.9g, %.9Lg expected\n", trial, (double)a, (double)b, (double)c,
                   (double)f, best);
            return false;
        }
        x[trial % 4][trial % 3] = std::numeric_limits<R>::quiet_NaN();
        r = s = a = b = c = poison;
        geo::edge_edge_sq(x[0], x[1], x[2], x[3], &r, &s, d);
        geo::vtx_tri(x[0], x[1], x[2], x[3], &a, &b, &c, d);
        if (r == poison || s == poison || a == poison || b == poison || c == poison) {
            printf("NaN, trial %d: a weight was not set\n", trial);
            return false;
        }
    }
    return true;
}

template <bool kPT>
static bool filter() {
    std::mt19937 g(11);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    int settled[2] = {0, 0};
    for (int trial = 0; trial < 200000; ++trial) {
        const double far = trial % 3 == 0 ? 0.0 : trial % 3 == 1 ? 10.0 : 1000.0, size = 0.01;
        double o[3], dir[3] = {0, 0, 0}, x0[4][3], x1[4][3];
        for (double& v : o) v = far * u(g);
        // the second primitive is moved along an axis or a diagonal by about the
        // distance at which the exit begins, or less
        const int k = g() % 3, diag = g() % 3;
        dir[k] = 1.0;
        if (diag) dir[(k + 1) % 3] = diag == 1 ? 1.0 : -1.0;
        const double move = size * 0.5, gap = move * u(g) * 8.0;
        const bool flat = g() % 2;  // parallel edges, motion without a spread of its own
        for (int j = 0; j < 4; ++j) {
            const bool second = kPT ? j > 0 : j > 1;
            for (int c = 0; c < 3; ++c) {
                x0[j][c] = o[c] + (flat ? (j & 1) * (c == (k + 2) % 3) * size : size * 0.2 * u(g)) + second * gap * dir[c];
                x1[j][c] = x0[j][c] + move * (second ? -0.3 : 0.3) * dir[c] + 0.1 * move * u(g);
            }
        }
        float xh[4][3], dh[4][3], m = 0.f;
        for (int j = 0; j < 4; ++j)
            for (int c = 0; c < 3; ++c) {  // as toi_maybe (collision_kernels.cu) forms them
                xh[j][c] = (float)x0[j][c] - (float)x0[0][c];
                dh[j][c] = (float)x1[j][c] - (float)x0[j][c];
                m = std::fmax(m, std::fmax(std::fabs((float)x0[j][c]), std::fabs((float)x1[j][c])));
            }
        const float eps = m / 1048576.f;
        for (int steps = 0; steps < 2; ++steps) {
            if (!geo::ccd_trivial_approx<float, kPT>(xh, dh, 4 * eps, 8 * eps, steps != 0)) continue;
            ++settled[steps];
            double x[4][3], dx[4][3];
            for (int j = 0; j < 4; ++j)
                for (int c = 0; c < 3; ++c) {
                    x[j][c] = x0[j][c];
                    dx[j][c] = x1[j][c] - x0[j][c];
                }
            const int it = steps ? 10 : 0;
            const double toi = kPT ? geo::ccd_pt<double>(x, dx, 0.1, it) : geo::ccd_ee<double>(x, dx, 0.1, it);
            if (toi != 1.0) {
                printf("filter %d, trial %d, steps %d: the exact test gives %.17g\n", kPT, trial, steps, toi);
                return false;
            }
        }
    }
    if (settled[0] < 1000 || settled[1] < settled[0] + 100) {  // the cases reach both exits
        printf("filter %d: %d and %d settled\n", kPT, settled[0], settled[1]);
        return false;
    }
    return true;
}

int main() {
    if (!distances<float>() || !distances<double>()) return 1;
    if (!filter<true>() || !filter<false>()) return 1;
    printf("ok\n");
    return 0;
}
