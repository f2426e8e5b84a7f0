// The host's XXH32 as the frame decoder uses it: a digest held in memory,
// against one thread's registers. Test infrastructure only.
#include <chrono>

#include "xxhash32.h"

namespace {
template <class Fn>
double best(Fn fn) {
    double b = 1e9;
    for (int k = 0; k < 40; ++k) {
        const auto t = std::chrono::steady_clock::now();
        fn();
        const std::chrono::duration<double> s = std::chrono::steady_clock::now() - t;
        if (s.count() < b) b = s.count();
    }
    return b;
}
}  // namespace

// The digest of n bytes given in parts of `part` stripes.
extern "C" __attribute__((noinline)) uint32_t xxh_parts(cdb::Xxh32* h, const unsigned char* p,
                                                        size_t n, size_t part) {
    size_t at = 0;
    for (; n - at >= 16 * part; at += 16 * part) h->stripes(p + at, part);
    const size_t rest = (n - at) / 16;
    h->stripes(p + at, rest);
    return h->finish(p + n / 16 * 16, n % 16);
}
extern "C" uint32_t xxh_digest(const unsigned char* p, size_t n, size_t part) {
    cdb::Xxh32 h;
    return xxh_parts(&h, p, n, part);
}
// Time of a digest in memory over that of four scalar accumulators.
extern "C" double xxh_pace(const unsigned char* p, size_t n) {
    volatile uint32_t sink = 0;
    const double mem = best([&] { sink = sink + xxh_digest(p, n, n / 16); });
    const double reg = best([&] {
        uint32_t v[4] = {1, 2, 3, 4};
        for (size_t i = 0; i + 16 <= n; i += 16)
            for (int k = 0; k < 4; ++k) {
                v[k] = cdb::xxh_rotl(v[k] + cdb::xxh_read32(p + i + 4 * k) * cdb::kXxhP2, 13) *
                       cdb::kXxhP1;
                asm("" : "+r"(v[k]));
            }
        sink = sink + v[0] + v[1] + v[2] + v[3];
    });
    return mem / reg;
}
