// Every row of arrays at each 4-byte boundary: the loads that row_loads names
// cover its coordinates and stay within the array; all rows have them but those
// at its ends.
#include <cstdio>

#include "kernels.cuh"

int main() {
    for (uint64_t base = 4096; base < 4096 + 16; base += 4)
        for (uint32_t words = 4; words <= 6; words += 2)
            for (uint64_t n = 1; n <= 40; n++) {
                const uint64_t w = words + 1, end = base + 4 * n * w;
                for (uint64_t i = 0; i < n; i++) {
                    const uint64_t b = base + 4 * i * w;
                    const pbig::RowLoads r = pbig::row_loads(b, words, base, end);
                    const uint64_t first = b - 4 * r.before, last = first + 16 * r.count;
                    const bool inside = first >= base && last <= end, covers = first % 16 == 0 && last >= b + 4 * words;
                    const bool at_an_end = i * w < 4 || (n - i) * w < words + 4;
                    if (r.before > 3 || r.count > 3 || (r.count ? !(inside && covers) : !at_an_end)) {
                        printf("base %llu words %u row %llu of %llu\n", (unsigned long long)base, words, (unsigned long long)i,
                               (unsigned long long)n);
                        return 1;
                    }
                }
            }
    return 0;
}
