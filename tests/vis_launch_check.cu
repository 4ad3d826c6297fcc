// The launch shape of a visibility batch at every edge of its rule and at the
// largest counts, built by tests/test_vis_launch.py with the undefined-behaviour
// sanitizer.  Prints the number of counts looked at.
#include <climits>
#include <cstdio>

#include "rg_internal.h"

int main() {
    const int units = 152 * 8;
    const int edges[] = {1, 4 * units, 32 * units, 128 * units, 512 * units, INT_MAX - 512, INT_MAX - units, INT_MAX};
    int looked = 0;
    for (int e : edges)
        for (long long v = (long long)e - 2; v <= (long long)e + 2; ++v) {
            if (v < 1 || v > INT_MAX) continue;
            const int n = (int)v;
            const VisLaunch l = vis_launch(n);
            const bool small = n <= 32 * units;
            const int lo = small ? 4 : 128, hi = small ? 32 : 512;
            const long long all = (long long)l.blocks * l.chunk;
            if (l.threads != (small ? 32 : 128) || l.chunk < lo || l.chunk > hi || all < n || all - l.chunk >= n) {
                printf("n %d: threads %d chunk %d blocks %u\n", n, l.threads, l.chunk, l.blocks);
                return 1;
            }
            if (l.chunk > lo && l.chunk < hi && l.blocks > (unsigned)units) return 2;
            ++looked;
        }
    printf("%d\n", looked);
    return 0;
}
