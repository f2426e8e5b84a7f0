// A CUDA CTA on the host, for the CPU tests of device code written with warp
// collectives and barriers: every thread is a fiber, run one at a time, that
// gives way where it meets a collective or a barrier, an arrival without a
// wait included. A collective completes when all 32 lanes have reached it, a
// barrier when its thread count has; if every fiber waits, the CTA has
// deadlocked and run() returns false, as it does where a thread meets a
// barrier twice before it completes or threads state different counts for it.
// The order in which runnable fibers are taken is drawn from the seed, and a
// seed can name a warp that only runs when no other can, so that code which
// leans on an order or a pace that CUDA does not give shows it. Test
// infrastructure only.
#pragma once

#include <ucontext.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <vector>

#define CDB_EMULATE 1
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__ inline
#define __constant__
#define __align__(n) alignas(n)
#define __shared__ static

namespace emul {

struct Fiber {
    ucontext_t ctx;
    bool done = false;
    const uint32_t* gen = nullptr;  // what it waits for: *gen to differ from `at`
    uint32_t at = 0;
    bool runnable() const { return !done && (gen == nullptr || *gen != at); }
};

struct Warp {
    uint64_t value[2][32];
    uint32_t arrived = 0, gen = 0;
    int op = 0;
};

struct Barrier {
    uint32_t arrived = 0, gen = 0, count = 0;
    std::vector<uint32_t> seen;  // per thread: 1 + the generation it last arrived in
};

struct Cta {
    static constexpr size_t kStack = 256 << 10;
    uint32_t threads = 0;
    std::vector<Fiber> fibers;
    std::vector<Warp> warps;
    Barrier bars[16];
    ucontext_t main_ctx;
    uint32_t cur = 0;
    const char* bad = nullptr;
    std::function<void()> body;
};

inline Cta*& cta() {
    static Cta* c = nullptr;
    return c;
}

// Back to the scheduler until *gen differs from `at` (null: until its turn).
inline void give_way(const uint32_t* gen = nullptr, uint32_t at = 0) {
    Cta* c = cta();
    Fiber& f = c->fibers[c->cur];
    f.gen = gen;
    f.at = at;
    swapcontext(&f.ctx, &c->main_ctx);
}

inline void fail(const char* why) {
    cta()->bad = why;
    give_way();  // for good
}

inline void entry() {
    Cta* c = cta();
    c->body();
    c->fibers[c->cur].done = true;
    swapcontext(&c->fibers[c->cur].ctx, &c->main_ctx);
}

// The seed whose order is `order` (below 256; 0: by thread number) and that
// starves warp `warp`.
constexpr uint64_t starving(uint64_t order, uint32_t warp) {
    return order | static_cast<uint64_t>(warp + 1) << 8;
}

// Runs `body` as `threads` threads; false when they deadlock or misuse a
// collective or a barrier.
inline bool run(uint32_t threads, uint64_t seed, std::function<void()> body) {
    static std::vector<std::unique_ptr<char[]>> pool;
    static Cta c;
    c = Cta();
    c.threads = threads;
    c.body = std::move(body);
    c.fibers.resize(threads);
    c.warps.resize(threads / 32);
    for (Barrier& b : c.bars) b.seen.assign(threads, 0);
    cta() = &c;
    while (pool.size() < threads) pool.emplace_back(new char[Cta::kStack]);
    for (uint32_t t = 0; t < threads; ++t) {
        Fiber& f = c.fibers[t];
        getcontext(&f.ctx);
        f.ctx.uc_stack.ss_sp = pool[t].get();
        f.ctx.uc_stack.ss_size = Cta::kStack;
        f.ctx.uc_link = nullptr;
        makecontext(&f.ctx, entry, 0);
    }
    const uint64_t order = seed & 255;
    const uint32_t starved = static_cast<uint32_t>(seed >> 8);  // 1 + the warp
    uint64_t rng = order * 0x9E3779B97F4A7C15ull + 1;
    for (;;) {
        rng = rng * 6364136223846793005ull + 1442695040888963407ull;
        const uint32_t start = order ? static_cast<uint32_t>(rng >> 33) % threads : 0;
        const bool down = order && (rng >> 62 & 1);
        bool ran = false;
        // the starved warp in a turn of its own, when no other thread can run
        for (int turn = 0; turn < 2 && !ran; ++turn)
            for (uint32_t k = 0; k < threads; ++k) {
                const uint32_t t = (start + (down ? threads - k : k)) % threads;
                if ((turn == 1) != (t / 32 + 1 == starved) || !c.fibers[t].runnable()) continue;
                ran = true;
                c.cur = t;
                swapcontext(&c.main_ctx, &c.fibers[t].ctx);
                if (c.bad) return false;
            }
        if (ran) continue;
        for (uint32_t t = 0; t < threads; ++t)
            if (!c.fibers[t].done) {
                c.bad = "deadlock";
                return false;
            }
        return true;
    }
}

// All 32 lanes' values of a collective.
inline const uint64_t* collect(int op, uint64_t v) {
    Cta* c = cta();
    Warp& w = c->warps[c->cur / 32];
    const uint32_t lane = c->cur % 32, gen = w.gen;
    if (w.arrived == 0) w.op = op;
    if (w.op != op) fail("lanes of a warp at different collectives");
    uint64_t* slot = w.value[gen & 1];
    slot[lane] = v;
    if (++w.arrived == 32) {
        w.arrived = 0;
        ++w.gen;
    } else {
        give_way(&w.gen, gen);
    }
    return slot;
}

inline void bar(int id, uint32_t n, bool wait) {
    Cta* c = cta();
    Barrier& b = c->bars[id];
    const uint32_t gen = b.gen;
    if (b.arrived != 0 && b.count != n) fail("threads state different counts for a barrier");
    if (b.seen[c->cur] == gen + 1) fail("a thread meets a barrier twice before it completes");
    b.count = n;
    b.seen[c->cur] = gen + 1;
    if (++b.arrived == n) {
        b.arrived = 0;
        ++b.gen;
    }
    if (!wait) give_way();
    else if (b.gen == gen) give_way(&b.gen, gen);
}

struct Idx {
    struct X {
        operator uint32_t() const { return cta()->cur; }
    } x;
};

}  // namespace emul

static emul::Idx threadIdx;

inline void __syncwarp() { (void)emul::collect(1, 0); }
inline void __syncthreads() { emul::bar(0, emul::cta()->threads, true); }
template <class T>
T __shfl_sync(unsigned, T v, uint32_t from) {
    uint64_t x = 0;
    std::memcpy(&x, &v, sizeof v);
    x = emul::collect(2, x)[from & 31];
    std::memcpy(&v, &x, sizeof v);
    return v;
}
template <class T>
T __shfl_up_sync(unsigned, T v, uint32_t d) {
    uint64_t x = 0;
    std::memcpy(&x, &v, sizeof v);
    const uint32_t lane = emul::cta()->cur & 31;
    x = emul::collect(3, x)[lane >= d ? lane - d : lane];
    std::memcpy(&v, &x, sizeof v);
    return v;
}
template <class T>
T __shfl_xor_sync(unsigned, T v, uint32_t d) {
    uint64_t x = 0;
    std::memcpy(&x, &v, sizeof v);
    const uint32_t lane = emul::cta()->cur & 31;
    x = emul::collect(4, x)[(lane ^ d) & 31];
    std::memcpy(&v, &x, sizeof v);
    return v;
}
inline unsigned __ballot_sync(unsigned, bool p) {
    const uint64_t* v = emul::collect(5, p);
    unsigned m = 0;
    for (int k = 0; k < 32; ++k) m |= static_cast<unsigned>(v[k] & 1) << k;
    return m;
}
inline bool __any_sync(unsigned, bool p) { return __ballot_sync(0, p) != 0; }
inline bool __all_sync(unsigned, bool p) { return __ballot_sync(0, p) == 0xffffffffu; }
inline unsigned __match_any_sync(unsigned, uint32_t x) {
    const uint64_t* v = emul::collect(6, x);
    unsigned m = 0;
    for (int k = 0; k < 32; ++k) m |= (v[k] == x ? 1u : 0u) << k;
    return m;
}
inline float __fdividef(float a, float b) { return a / b; }
inline int __clz(uint32_t x) { return x ? __builtin_clz(x) : 32; }
inline int __clzll(long long x) { return x ? __builtin_clzll(static_cast<uint64_t>(x)) : 64; }
inline int __ffs(uint32_t x) { return __builtin_ffs(static_cast<int>(x)); }
inline int __ffsll(long long x) { return __builtin_ffsll(x); }
inline int __popc(uint32_t x) { return __builtin_popcount(x); }
inline int __popcll(uint64_t x) { return __builtin_popcountll(x); }
inline uint32_t __brev(uint32_t x) {
    uint32_t r = 0;
    for (int k = 0; k < 32; ++k) r |= ((x >> k) & 1u) << (31 - k);
    return r;
}
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) {
    return static_cast<uint32_t>((static_cast<uint64_t>(hi) << 32 | lo) >> (s & 31));
}
inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t s) {
    return static_cast<uint32_t>((static_cast<uint64_t>(hi) << 32 | lo) << (s & 31) >> 32);
}
inline uint32_t __funnelshift_rc(uint32_t lo, uint32_t hi, uint32_t s) {
    return s >= 32 ? hi : __funnelshift_r(lo, hi, s);
}
inline uint32_t __funnelshift_lc(uint32_t lo, uint32_t hi, uint32_t s) {
    return s >= 32 ? lo : __funnelshift_l(lo, hi, s);
}
// Thread 0's loads through the read-only path.
inline uint64_t& emul_ldgs() {
    static uint64_t n = 0;
    return n;
}
template <class T>
T __ldg(const T* p) {
    emul_ldgs() += emul::cta()->cur == 0;
    return *p;
}

inline uint32_t atomicAdd(uint32_t* a, uint32_t v) {
    const uint32_t old = *a;
    *a += v;
    return old;
}
inline uint32_t atomicOr(uint32_t* a, uint32_t v) {
    const uint32_t old = *a;
    *a |= v;
    return old;
}
inline uint32_t atomicMin(uint32_t* a, uint32_t v) {
    const uint32_t old = *a;
    if (v < old) *a = v;
    return old;
}

// the device code's shared memory accesses by address
namespace cdb {
namespace zstd {
using SAddr = uintptr_t;
inline const char*& smem_lo() {
    static const char* p = nullptr;
    return p;
}
inline const char*& smem_hi() {
    static const char* p = nullptr;
    return p;
}
inline void in_smem(SAddr a, size_t n) {
    if (a < reinterpret_cast<SAddr>(smem_lo()) || a + n > reinterpret_cast<SAddr>(smem_hi())) {
        std::fprintf(stderr, "emulation: address outside shared memory\n");
        std::abort();
    }
}
inline SAddr saddr(const void* p) { return reinterpret_cast<SAddr>(p); }
inline uint32_t lds(SAddr a) {
    in_smem(a, 4);
    return *reinterpret_cast<const uint32_t*>(a);
}
inline void sts4_first(SAddr a, uint32_t x, uint32_t y, uint32_t z, uint32_t w, uint32_t lane) {
    if (lane) return;
    in_smem(a, 16);
    uint32_t* p = reinterpret_cast<uint32_t*>(a);
    p[0] = x, p[1] = y, p[2] = z, p[3] = w;
}
}  // namespace zstd
}  // namespace cdb

// named barriers of the device code (bar.sync / bar.arrive)
namespace cdb {
inline void bar_sync(int id, int n) { emul::bar(id, static_cast<uint32_t>(n), true); }
inline void bar_arrive(int id, int n) { emul::bar(id, static_cast<uint32_t>(n), false); }
}  // namespace cdb
