// Host emulation of the warp-per-page GDeflate decoder (cudec_b200/csrc/
// gdeflate_page.cuh): the device source itself, its lanes run by cuda_emul.h.
// Test infrastructure only.
#include "cuda_emul.h"

#include "gdeflate_page.cuh"

extern "C" int gdeflate_emulate(const uint8_t* src, uint64_t n, uint8_t* dst, uint64_t cap,
                                uint64_t seed, uint64_t* written) {
    static cdb::gdf::Tables* s = new cdb::gdf::Tables();
    std::memset(static_cast<void*>(s), 0x5C, sizeof *s);  // stale state must not matter
    std::vector<int> st(32, -2);
    std::vector<uint64_t> out(32, 0);
    const bool ok = emul::run(32, seed, [&] {
        const uint32_t t = threadIdx.x;
        uint64_t w = 0;
        st[t] = cdb::gdf::decode_page(src, n, dst, cap, *s, t, &w);
        out[t] = w;
    });
    for (uint32_t t = 1; ok && t < 32; ++t)
        if (st[t] != st[0] || out[t] != out[0]) return -3;  // lanes disagree
    *written = ok && st[0] == 0 ? out[0] : 0;
    return ok ? st[0] : -1;
}
