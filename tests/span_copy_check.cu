// Host check of the span copy's lanes (spans.cuh), built and run by tests/test_span_copy_host.py: sources and
// destinations of every alignment lie at both ends of a page whose neighbours may not be touched (a read or write of
// a word that holds no byte of a span ends the program), and only the span's bytes are written.
#include <cstdio>
#include <cstring>
#include <sys/mman.h>
#include <vector>

#include "../cubam_b200/csrc/spans.cuh"

static int failures = 0;

// A page between two that may not be touched.
static uint8_t* page() {
    uint8_t* m = (uint8_t*)mmap(nullptr, 3 * 4096, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    mprotect(m + 4096, 4096, PROT_READ | PROT_WRITE);
    return m + 4096;
}

template <uint32_t LANES, bool LONG> static void copy_of(uint8_t* src, uint8_t* dst, int so, int d, int len) {
    std::vector<uint8_t> want(4096, 0xA5);
    memset(dst, 0xA5, 4096);
    if (len > 0) memcpy(want.data() + d, src + so, len);
    for (uint32_t l = 0; l < LANES; l++)
        LONG ? cb::copy_long<LANES, 2>(src + so, dst + d, len, l) : cb::copy_words<LANES>(src + so, dst + d, len, l);
    if (memcmp(dst, want.data(), 4096) && failures++ < 10) printf("FAIL lanes %u long %d from %d to %d, %d bytes\n", LANES, LONG, so, d, len);
}

int main() {
    uint8_t *src = page(), *dst = page();
    for (int i = 0; i < 4096; i++) src[i] = (uint8_t)(i * 131 + (i >> 8) * 7 + 1);
    for (int len : {-3, -1, 0, 1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 33, 63, 64, 65, 255, 511, 512, 513, 700, 2049, 4096}) {
        const int n = len > 0 ? len : 0;
        for (int a = 0; a < 20 && a + n <= 4096; a++)
            for (int b = 0; b < 20 && b + n <= 4096; b++)
                for (int end = 0; end < 4; end++) {  // each at the page's start or its end
                    const int so = end & 1 ? 4096 - n - a : a, d = end & 2 ? 4096 - n - b : b;
                    copy_of<4, false>(src, dst, so, d, len);
                    copy_of<32, false>(src, dst, so, d, len);
                    copy_of<32, true>(src, dst, so, d, len);
                }
    }
    printf("%d failures\n", failures);
    return failures != 0;
}
