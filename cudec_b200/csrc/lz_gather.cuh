// Output by gathering: the map from output bytes to the tokens of a batch,
// and the way from an output byte to the byte it copies. Shared by the
// LZ4/Snappy and the Zstd decoders; compiled for the host too (the CPU tests
// emulate the decoders).
//
// A batch is a run of consecutive tokens (a literal run, then a match). Its
// output positions are relative to the aligned 32-byte sector of the
// destination that holds its first byte, and kWindow of them are mapped at a
// time: per sector one start bit per byte and the number of tokens that
// start before it. A byte's token is that count plus the start bits up to
// the byte, less one.
#pragma once

#include <cstdint>

#ifndef CDB_HD
#if defined(__CUDACC__)
#define CDB_HD __host__ __device__ __forceinline__
#else
#define CDB_HD inline
#endif
#endif

// Code for a CTA's threads: on the device, and where a test runs them as one.
#if defined(__CUDA_ARCH__) || defined(CDB_EMULATE)
#define CDB_DEVICE_CODE 1
#else
#define CDB_DEVICE_CODE 0
#endif

namespace cdb {
namespace lzg {

constexpr uint32_t kWindow = 4096;  // output bytes mapped at a time
constexpr uint32_t kSectors = kWindow / 32;

// One token of a batch (output positions).
struct alignas(16) Rec {
    uint32_t out;  // first byte
    uint32_t le;   // end of the literal run: the match starts here
    uint32_t dl;   // a literal byte's index in the literal source = its position + dl
    uint32_t off;  // match offset
};

struct alignas(8) Sector {
    uint32_t starts, before;
};

#if CDB_DEVICE_CODE
__device__ __forceinline__ void at_or(uint32_t* a, uint32_t v) { atomicOr(a, v); }
__device__ __forceinline__ uint32_t pop32(uint32_t v) { return __popc(v); }
#else
inline void at_or(uint32_t* a, uint32_t v) { *a |= v; }
inline uint32_t pop32(uint32_t v) { return static_cast<uint32_t>(__builtin_popcount(v)); }
#endif

// m mod d for m below 2^12, 1 <= d <= m. Exact on the device: (m + 1/2) / d
// lies at least 1/(2 d) from an integer, and the quotient's error is below
// m / d * 2^-20.
CDB_HD uint32_t small_mod(uint32_t m, uint32_t d) {
#if defined(__CUDA_ARCH__)
    const uint32_t q = static_cast<uint32_t>(
        __fdividef(static_cast<float>(m) + 0.5f, static_cast<float>(d)));
    return m - q * d;
#else
    return m % d;
#endif
}

// Token i, output [y0, y1), into the window at W (its start bits zeroed and
// published before).
CDB_HD void map_token(Sector* map, uint32_t i, uint32_t y0, uint32_t y1, uint32_t W) {
    if (y0 >= W && y0 < W + kWindow) at_or(&map[(y0 - W) >> 5].starts, 1u << (y0 & 31));
    // the sectors that begin in (y0, y1]
    const uint32_t from = y0 < W ? 0 : (y0 - W) / 32 + 1;
    for (uint32_t k = from; k < kSectors && W + 32 * k <= y1; ++k) map[k].before = i + 1;
}

// Where a byte of the output comes from: a literal's index in the literal
// source, or a window position before the window's first byte of the batch
// (down to -2^31).
struct Source {
    int32_t at;
    bool lit;
    bool ok;  // the byte is one of the batch's
};

#if defined(__CUDA_ARCH__)
#define LZG_UNROLL _Pragma("unroll")
#else
#define LZG_UNROLL
#endif

// The sources of lane's byte in the sectors k, k + step, ... (N of them) of
// the window at W, for bytes [lo, hi) of it; kRecs: records, a power of two.
// A source inside the window is followed through the map, past whole periods
// of an overlapping match, so each match costs one hop at most (matches are
// shorter than 2^12 bytes, see small_mod; offsets are below 2^31). The loads
// of all N run together; the bytes that need another hop go on in a loop
// that most groups skip.
template <uint32_t N, uint32_t kRecs>
CDB_HD void sources(const Sector* map, const Rec* rec, uint32_t k, uint32_t step, uint32_t lane,
                    uint32_t lo, uint32_t hi, uint32_t W, Source (&src)[N]) {
    const uint32_t upto = 0xffffffffu >> (31 - lane);
    uint32_t le[N], off[N];
    bool any = false;
    LZG_UNROLL
    for (uint32_t j = 0; j < N; ++j) {
        // past the window or the batch: any record, the byte is not used
        const Sector sc = map[(k + j * step) % kSectors];
        const Rec r = rec[(sc.before + pop32(sc.starts & upto) - 1) % kRecs];
        le[j] = r.le;
        off[j] = r.off;
        src[j].at = static_cast<int32_t>(r.dl);
    }
    LZG_UNROLL
    for (uint32_t j = 0; j < N; ++j) {
        const uint32_t x = 32 * (k + j * step) + lane;
        const uint32_t m = x + W - le[j];  // position in the match; wraps in the literals
        src[j].lit = static_cast<int32_t>(m) < 0;
        src[j].at = static_cast<int32_t>(src[j].lit ? x + W + static_cast<uint32_t>(src[j].at)
                                                    : x - off[j]);
        src[j].ok = x - lo < hi - lo;
        any = any || (src[j].ok && !src[j].lit && (m >= off[j] || off[j] <= x - lo));
    }
#if CDB_DEVICE_CODE
    if (!__any_sync(0xffffffffu, any)) return;
#else
    if (!any) return;
#endif
    LZG_UNROLL
    for (uint32_t j = 0; j < N; ++j) {
        uint32_t x = 32 * (k + j * step) + lane;
        if (src[j].lit || !src[j].ok) continue;
        uint32_t end = le[j], by = off[j];
        for (;;) {
            const uint32_t m = x + W - end;
            if (m >= by) by += m - small_mod(m, by);
            if (by > x - lo) {
                src[j].at = static_cast<int32_t>(x - by);
                break;
            }
            x -= by;
            const Sector sc = map[x >> 5];
            const Rec r = rec[sc.before + pop32(sc.starts & (0xffffffffu >> (31 - (x & 31)))) - 1];
            if (static_cast<int32_t>(x + W - r.le) < 0) {
                src[j].at = static_cast<int32_t>(x + W + r.dl);
                src[j].lit = true;
                break;
            }
            end = r.le;
            by = r.off;
        }
    }
}

CDB_HD uint32_t fsr(uint32_t lo, uint32_t hi, uint32_t sh) {  // funnel shift right, sh < 32
#if defined(__CUDA_ARCH__)
    return __funnelshift_r(lo, hi, sh);
#else
    return sh ? (lo >> sh) | (hi << (32 - sh)) : lo;
#endif
}

struct alignas(16) V16 {
    uint32_t w[4];
};

// 16 bytes at global address p, read as the aligned words holding them (no
// word past the last wanted byte is touched).
CDB_HD V16 gload16(const uint8_t* p) {
    const uintptr_t ad = reinterpret_cast<uintptr_t>(p);
    const uint32_t s4 = static_cast<uint32_t>(ad & 3), sh = 8 * s4;
    const uint32_t* q = reinterpret_cast<const uint32_t*>(ad - s4);
    const uint32_t w0 = q[0], w1 = q[1], w2 = q[2], w3 = q[3];
    const uint32_t w4 = s4 ? q[4] : 0;
    return V16{{fsr(w0, w1, sh), fsr(w1, w2, sh), fsr(w2, w3, sh), fsr(w3, w4, sh)}};
}
CDB_HD void put16(uint8_t* p, const V16& v) { *reinterpret_cast<V16*>(p) = v; }  // p aligned

// Thread t's share, of T threads, of a copy of n bytes (no byte of the source
// being written meanwhile): destination-aligned 16-byte blocks, two in flight.
CDB_HD void copy_share(uint8_t* to, const uint8_t* src, uint64_t n, uint32_t t, uint32_t T) {
    uint64_t head = (16 - (reinterpret_cast<uintptr_t>(to) & 15)) & 15;
    if (head > n) head = n;
    const uint64_t body = head + ((n - head) & ~15ull), step = 16ull * T;
    if (t < head) to[t] = src[t];
    uint64_t q = head + 16ull * t;
    for (; q + step < body; q += 2 * step) {
        const V16 a = gload16(src + q), b = gload16(src + q + step);
        put16(to + q, a);
        put16(to + q + step, b);
    }
    if (q < body) put16(to + q, gload16(src + q));
    if (body + t < n) to[body + t] = src[body + t];
}

// Thread t's share of n bytes that repeat the period[0, f) in shared memory.
CDB_HD void period_share(uint8_t* to, const uint8_t* period, uint32_t f, uint64_t n, uint32_t t,
                         uint32_t T) {
    uint64_t head = (16 - (reinterpret_cast<uintptr_t>(to) & 15)) & 15;
    if (head > n) head = n;
    const uint64_t body = head + ((n - head) & ~15ull);
    if (t < head) to[t] = period[t % f];
    uint32_t ph = static_cast<uint32_t>((head + 16ull * t) % f);
    const uint32_t adv = static_cast<uint32_t>((16ull * T) % f);
    for (uint64_t q = head + 16ull * t; q < body; q += 16ull * T) {
        V16 v{{0, 0, 0, 0}};
        uint32_t h = ph;
        for (uint32_t j = 0; j < 16; ++j) {
            v.w[j >> 2] |= static_cast<uint32_t>(period[h]) << (8 * (j & 3));
            h = h + 1 == f ? 0 : h + 1;
        }
        put16(to + q, v);
        ph += adv;
        if (ph >= f) ph -= f;
    }
    if (body + t < n) to[body + t] = period[(body + t) % f];
}

}  // namespace lzg
}  // namespace cdb
