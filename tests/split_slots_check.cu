// Host check of the members the split inflater takes (split_slots.cuh), built and run by tests/test_split_slots_host.py:
// every size it takes is counted without loss in the 32 bits its kernels count in, and every size a BGZF file may hold
// is taken.
#include <cstdio>

#include "../cubam_b200/csrc/split_slots.cuh"

using namespace cb::split;

static int failures = 0;

int main() {
    for (int bit = 0; bit < 32; bit++) {
        for (int k = -70; k <= 70; k++) {
            const uint32_t n = (1u << bit) + (uint32_t)k;
            if (in_reach(n, 100) && 8ull * n + 15 * 8 + 512 > BITS && failures++ < 10) printf("FAIL input of %u bytes\n", n);
            if (!in_reach(100, n)) continue;
            const unsigned long long slot = slot_bytes(n), out = 127ull + n + 258;  // from the output's first line on
            if ((uint32_t)slot != slot && failures++ < 10) printf("FAIL slot of %u bytes\n", n);
            if ((uint32_t)out != out && failures++ < 10) printf("FAIL output of %u bytes\n", n);
            if (slot < 4ull * n / 3 && failures++ < 10) printf("FAIL symbols of %u bytes\n", n);
        }
    }
    if (!in_reach(65535, 65536)) failures++;
    if (in_reach(3u << 20, 3u << 30)) failures++;  // 3 GB of zeros
    printf("%d failures\n", failures);
    return failures != 0;
}
