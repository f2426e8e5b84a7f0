// Host emulation of the CTA-per-chunk LZ decoder's device path
// (cudec_b200/csrc/lz_cta_kernel.cuh): the source itself with its warps and
// barriers run by cuda_emul.h, at each of the kernel's widths. Test
// infrastructure only.
#include "cuda_emul.h"

#include "lz_cta_kernel.cuh"

namespace {

template <class F, uint32_t T>
int run(const uint8_t* src, uint64_t S, uint8_t* dst, uint64_t cap, uint64_t seed,
        uint64_t* written) {
    using Shm = cdb::lzc::Shm<F, T>;
    static Shm* shm = new Shm();
    std::memset(static_cast<void*>(shm), 0x5C, sizeof *shm);  // stale state must not matter
    emul_ldgs() = 0;
    std::vector<int> st(T, -2);
    std::vector<uint64_t> out(T, 0);
    const bool ok = emul::run(T, seed, [&] {
        const uint32_t t = threadIdx.x;
        cdb::lzc::Chunk<F, T> ch{*shm, src, S, dst, cap, 0};
        uint64_t w = 0;
        st[t] = ch.run(&w);
        out[t] = w;
    });
    for (uint32_t t = 1; ok && t < T; ++t)
        if (st[t] != st[0] || (st[0] == 0 && out[t] != out[0])) return -3;  // threads disagree
    *written = ok && st[0] == 0 ? out[0] : 0;
    return ok ? st[0] : -1;
}

template <class F>
int widths(uint32_t threads, const uint8_t* src, uint64_t S, uint8_t* dst, uint64_t cap,
           uint64_t seed, uint64_t* written) {
    return threads == 128   ? run<F, 128>(src, S, dst, cap, seed, written)
           : threads == 256 ? run<F, 256>(src, S, dst, cap, seed, written)
                            : run<F, 512>(src, S, dst, cap, seed, written);
}

// A batch's capacities, their reads counted.
struct Caps {
    const size_t* p;
    size_t n;
    uint64_t* reads;
    size_t operator[](size_t i) const {
        if (i >= n) std::abort();
        ++*reads;
        return p[i];
    }
};

}  // namespace

// Barriers that the CTA of the last run met, and thread 0's loads of input past
// the staged bytes.
extern "C" uint32_t lz_barriers() { return emul::cta()->bars[0].gen; }
extern "C" uint64_t lz_ldgs() { return emul_ldgs(); }

// The large chunks of a batch, as the wide kernel's `wide` CTAs pick them
// (chunk[0, *count): its index, one per CTA) and as the narrow CTAs of the m
// chunks at `ask` find them (is[0, m)); reads: capacities that those m read.
// -1: the CTA deadlocks.
extern "C" int lz_large(const size_t* caps, size_t n, uint32_t wide, uint64_t seed,
                        uint64_t* chunk, uint32_t* count, const uint64_t* ask, size_t m,
                        uint8_t* is, uint64_t* reads) {
    uint64_t other = 0;
    *reads = 0;
    const Caps w{caps, n, &other}, c{caps, n, reads};
    if (!emul::run(256, seed, [&] {
            uint32_t cnt = 0;
            const uint32_t k = cdb::lzc::large_from<256>(w, n, wide, &cnt);
            if (threadIdx.x == 0) *count = cnt;
            for (uint32_t i = 0; i < cnt; ++i) {
                const size_t at = cdb::lzc::large_chunk<256>(w, n, k, i);
                __syncthreads();
                if (threadIdx.x == 0) chunk[i] = at;
            }
        }))
        return -1;
    const bool ok = emul::run(128, seed, [&] {
        for (size_t i = 0; i < m; ++i) {
            const bool large = cdb::lzc::is_large<128>(c, n, wide, ask[i]);
            if (threadIdx.x == 0) is[i] = large;
        }
    });
    return ok ? 0 : -1;
}

// fmt 0 = LZ4, 1 = Snappy; -1: the CTA deadlocks or its lanes meet different
// collectives.
extern "C" int lz_emulate(int fmt, uint32_t threads, const uint8_t* src, uint64_t n, uint8_t* dst,
                          uint64_t cap, uint64_t seed, uint64_t* written) {
    return fmt == 0 ? widths<cdb::lzc::Lz4F>(threads, src, n, dst, cap, seed, written)
                    : widths<cdb::lzc::SnappyF>(threads, src, n, dst, cap, seed, written);
}
