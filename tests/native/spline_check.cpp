// CPU check of the statistics' lines per block (gkm-dns_b200/csrc/gks_limits.h):
// every block fits an SM, and two of them do up to the line lengths stated at
// spline_lines.  Prints "ok" and exits 0, or names the violations and exits 1.
#include "gks_limits.h"

#include <cstdio>

int main()
{
    int fails = 0;
    for (int axis = 0; axis < 3; ++axis)
        for (int nt = 10; nt <= gks::kSplineNtMax; ++nt) {
            const int lines = gks::spline_lines(axis, nt);
            const size_t block = gks::spline_bytes(axis, lines, nt) + gks::kSmemPerBlock;
            const bool one = block <= gks::kSmemPerSm, two = 2 * block <= gks::kSmemPerSm;
            const bool want16 = nt <= 289, want2 = nt <= (axis == 2 ? 555 : 556);
            if (!one || two != want2 || (lines == 16) != want16) {
                std::printf("FAIL axis %d nt %d: %d lines, %zu bytes\n", axis, nt, lines, block);
                ++fails;
            }
        }
    if (fails) return 1;
    std::printf("ok\n");
    return 0;
}
