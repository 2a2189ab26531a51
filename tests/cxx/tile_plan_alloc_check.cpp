// Every allocation of the thread that builds a tile plan fails once: the build must
// end in no plan, a plan, or std::bad_alloc, with its other threads joined.  Prints
// "ok" or what failed.
#include <cstdio>
#include <cstdlib>
#include <new>
#include <thread>

#include "tile_plan.h"

static thread_local long long countdown = -1;  // allocations until the one that fails; < 0: none does

void* operator new(std::size_t n) {
    if (countdown >= 0 && countdown-- == 0) throw std::bad_alloc();
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

using namespace pdipc;

int main() {
    const int nx = 24, ny = 20, models = 4;
    std::vector<ModelInput> in(models);
    for (int q = 0; q < models; ++q) {
        ModelInput& m = in[q];
        m.nv = nx * ny;
        for (int r = 0; r < ny; ++r)
            for (int c = 0; c < nx; ++c) m.X.insert(m.X.end(), {0.01 * c, (double)q, 0.01 * r});
        for (int r = 0; r + 1 < ny; ++r)
            for (int c = 0; c + 1 < nx; ++c) {
                const int a = r * nx + c;
                m.F.insert(m.F.end(), {a, a + nx, a + nx + 1, a, a + nx + 1, a + 1});
            }
        m.nf = (int)m.F.size() / 3;
        m.density = 0.1;
        m.k_stretch = 1e4;
        m.k_bend = 1e-3;
        m.pins = {0};
    }
    HostTables H;
    if (!build_host_tables(in, -9.8, H).empty()) return 1;
    TileLimits lim;
    lim.min_rows = 16;
    lim.sms = 64;  // enough tiles for several threads
    int plans = 0, none = 0, thrown = 0;
    for (long long k = 0;; ++k) {
        TilePlan P;
        bool failed = true;
        try {
            countdown = k;
            build_tile_plan(H, lim, 0, P);
            failed = countdown < 0;
            countdown = -1;
            ++(P.ok ? plans : none);
        } catch (const std::bad_alloc&) {
            countdown = -1;
            ++thrown;
        }
        if (!failed) {
            if (!P.ok || P.tiles.size() < 48) {
                printf("no plan of several threads with all of its memory\n");
                return 1;
            }
            break;  // past the last allocation
        }
    }
    if ((std::thread::hardware_concurrency() > 1 && plans < 2) || thrown < 2) {  // a thread that does not start costs nothing; a table that does not fit ends it
        printf("%d plans, %d without, %d thrown\n", plans, none, thrown);
        return 1;
    }
    printf("ok\n");
    return 0;
}
