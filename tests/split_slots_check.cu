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
    // a workspace made for some output has the scratch for it and leaves the arena whole; a larger one no less of either
    for (long long n : {1LL, 2LL, 39LL, 5327LL, 5328LL, 5329LL, 200'000LL, 10'000'000LL}) {
        if (in_flight(n) > n || in_flight(n) > FLIGHT) failures++;
        for (unsigned long long mean : {0ull, 1ull, 100ull, 1023ull, 1024ull, 1025ull, 4096ull, 16384ull, 16385ull, 65280ull, 1ull << 26}) {
            for (unsigned long long more : {0ull, 1ull, 5ull}) {
                const unsigned long long out = mean * n + more, need = arena_and_scratch(n, out);
                for (unsigned long long k : {0ull, 1ull, 15ull, 16ull, 4095ull, 1ull << 20, 1ull << 40}) {
                    const uint32_t s = scratch_for(n, need + k);
                    const bool ok = s >= scratch_bytes(n, out) && (k > 16 || s == scratch_bytes(n, out)) &&
                                    s % 4096 == 0 && s <= SCRATCH_MAX && need + k - (unsigned long long)in_flight(n) * s >= 2 * out;
                    if (!ok && failures++ < 10) printf("FAIL %lld members, %llu bytes, %llu more: %u\n", n, out, k, s);
                }
                // a smaller one keeps room for what it holds
                const unsigned long long less = need / 3;
                if ((unsigned long long)in_flight(n) * scratch_for(n, less) > less && failures++ < 10) printf("FAIL %lld, %llu\n", n, less);
            }
        }
    }
    printf("%d failures\n", failures);
    return failures != 0;
}
