// Host emulation of the CTA-per-frame Zstd decoder (cudec_b200/csrc/
// zstd_frame.cuh): the device source itself, its warps and barriers run by
// cuda_emul.h. Test infrastructure only.
#include "cuda_emul.h"

#include "zstd_frame.cuh"

// One chunk; multi: a frame sequence. Returns the status, -1 when the CTA
// deadlocks or its lanes meet different collectives. `slot`: kLitSlot bytes.
extern "C" int zstd_emulate(int multi, const uint8_t* src, uint64_t n, uint8_t* dst, uint64_t cap,
                            uint8_t* slot, uint64_t seed, uint64_t* written) {
    static cdb::zstd::TeamSmem* s = new cdb::zstd::TeamSmem();
    std::memset(static_cast<void*>(s), 0x5C, sizeof *s);  // stale state must not matter
    cdb::zstd::smem_lo() = reinterpret_cast<const char*>(s);
    cdb::zstd::smem_hi() = cdb::zstd::smem_lo() + sizeof *s;
    std::vector<int> st(cdb::zstd::kTeam, -2);
    std::vector<uint64_t> out(cdb::zstd::kTeam, 0);
    const bool ok = emul::run(cdb::zstd::kTeam, seed, [&] {
        const uint32_t t = threadIdx.x;
        uint64_t w = 0;
        const int r = multi ? cdb::zstd::decode_frames(src, n, dst, cap, *s, slot, &w)
                            : cdb::zstd::decode_frame(src, n, dst, cap, *s, slot, &w);
        st[t] = r;
        out[t] = w;
    });
    for (uint32_t t = 1; ok && t < cdb::zstd::kTeam; ++t)
        if (st[t] != st[0] || out[t] != out[0]) return -3;  // threads disagree
    *written = ok && st[0] == 0 ? out[0] : 0;
    if (!ok) std::fprintf(stderr, "emulation: %s\n", emul::cta()->bad);
    return ok ? st[0] : -1;
}
