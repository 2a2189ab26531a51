// Checks csrc/host_copy.h: copies of all sizes around the threads' parts, and that
// mapping a buffer's pages leaves its bytes.  Prints "ok" or what failed.
#include <cstdio>
#include <cstring>
#include <vector>

#include "host_copy.h"

int main() {
    for (size_t mb = 0; mb < 8; ++mb)
        for (int off : {-9, -1, 0, 1, 8}) {
            const long long n = (long long)(mb << 20) / 8 + off;
            if (n < 0) continue;
            std::vector<double> a(n + 2), b(n + 2, -1.0);
            for (long long i = 0; i < n + 2; ++i) a[i] = ((double)i + 1.0) / 3.0;
            pdipc::copy_host(b.data() + 1, a.data() + 1, 8 * (size_t)n);
            if (std::memcmp(b.data() + 1, a.data() + 1, 8 * (size_t)n) || b[0] != -1.0 || b[n + 1] != -1.0) {
                printf("copy of %lld doubles\n", n);
                return 1;
            }
            const std::vector<double> was = b;
            pdipc::map_pages(b.data() + 1, 8 * (size_t)n);  // unaligned, and not past the end
            if (std::memcmp(b.data(), was.data(), 8 * was.size())) {
                printf("pages of %lld doubles: the bytes changed\n", n);
                return 1;
            }
        }
    printf("ok\n");
    return 0;
}
