// A warp's queued matches, executed a match per lane (the GDeflate decoder's).
//
// A lane moves 16 bytes per piece, read as the aligned words that hold them
// and written as the destination's aligned words, with the bytes of a shared
// word apart; two pieces are in flight where the second does not read the
// first. Matches a lane would take long over are written by the whole warp.
// The LZ4, Snappy and Zstd CTA decoders gather byte by byte instead
// (lz_gather.cuh): there four warps and more wait for the slowest lane's
// match, and pieces measured 656 us against 447 for 1,024 LZ4 chunks of
// 64 KiB, 16.6 ms against 10.5 for 512 Zstd frames of 1 MiB.
//
// The lanes' parts compile for the host too (the CPU tests emulate the
// decoder).
#pragma once

#include <cstdint>

#include "lz_gather.cuh"

namespace cdb {
namespace lanes {

constexpr uint32_t kLaneMax = 128;  // longer matches are copied by the whole warp
constexpr uint32_t kPeriod = 512;   // bytes of scratch of warp_match

using lzg::fsr;
CDB_HD uint32_t fsl(uint32_t lo, uint32_t hi, uint32_t sh) {  // (hi:lo) << sh, high word, sh < 32
#if defined(__CUDA_ARCH__)
    return __funnelshift_l(lo, hi, sh);
#else
    return static_cast<uint32_t>((static_cast<uint64_t>(hi) << 32 | lo) << sh >> 32);
#endif
}

struct P16 {
    uint32_t w[4];
};

// m (1..16) bytes at p, from the aligned words that hold them.
CDB_HD P16 get(const uint8_t* p, uint32_t m) {
    const uint32_t s4 = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p) & 3), sh = 8 * s4;
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p - s4);
    const uint32_t n = s4 + m;  // bytes from q on
    const uint32_t w0 = q[0];
    const uint32_t w1 = n > 4 ? q[1] : 0u, w2 = n > 8 ? q[2] : 0u;
    const uint32_t w3 = n > 12 ? q[3] : 0u, w4 = n > 16 ? q[4] : 0u;
    return P16{{fsr(w0, w1, sh), fsr(w1, w2, sh), fsr(w2, w3, sh), fsr(w3, w4, sh)}};
}

// The first m (1..16) bytes of v at p.
CDB_HD void put(uint8_t* p, const P16& v, uint32_t m) {
    const uint32_t a = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p) & 3), sh = 8 * a;
    uint8_t* b = p - a;
    uint32_t* q = reinterpret_cast<uint32_t*>(b);
    const uint32_t end = a + m;  // 1..19
    const uint32_t x0 = v.w[0] << sh, x1 = fsl(v.w[0], v.w[1], sh);
    const uint32_t x2 = fsl(v.w[1], v.w[2], sh);
    const uint32_t x3 = fsl(v.w[2], v.w[3], sh);
    const uint32_t x4 = fsl(v.w[3], 0u, sh);
    if (a == 0 && end >= 4) {
        q[0] = x0;
    } else {
        if (a == 0) b[0] = static_cast<uint8_t>(x0);
        if (a <= 1 && end > 1) b[1] = static_cast<uint8_t>(x0 >> 8);
        if (a <= 2 && end > 2) b[2] = static_cast<uint8_t>(x0 >> 16);
        if (end > 3) b[3] = static_cast<uint8_t>(x0 >> 24);
    }
    if (end >= 8) q[1] = x1;
    if (end >= 12) q[2] = x2;
    if (end >= 16) q[3] = x3;
    const uint32_t i = end >> 2, r = end & 3;  // a last word in part
    if (i && r) {
        const uint32_t x = i == 1 ? x1 : i == 2 ? x2 : i == 3 ? x3 : x4;
        b[4 * i] = static_cast<uint8_t>(x);
        if (r > 1) b[4 * i + 1] = static_cast<uint8_t>(x >> 8);
        if (r > 2) b[4 * i + 2] = static_cast<uint8_t>(x >> 16);
    }
}

CDB_HD uint32_t piece(uint32_t n, uint32_t k) {
    return n - k < 16 ? n - k : 16u;
}

// n bytes from d back (d >= 16), two pieces at a time where the second does
// not read the first.
CDB_HD void copy_back(uint8_t* to, const uint8_t* from, uint32_t n, bool apart) {
    for (uint32_t k = 0; k < n;) {
        const bool two = apart && k + 16 < n;
        const P16 x = get(from + k, piece(n, k));
        P16 y = x;
        if (two) y = get(from + k + 16, piece(n, k + 16));
        put(to + k, x, piece(n, k));
        k += 16;
        if (two) {
            put(to + k, y, piece(n, k));
            k += 16;
        }
    }
}

// A match of n bytes from `off` back, every byte before it written. An offset
// under 16 is a period: the match's first bytes are put one by one up to the
// first multiple of it past 16, after which it continues that far back.
CDB_HD void match(uint8_t* to, uint32_t n, uint32_t off) {
    uint32_t d = off, k = 0;
    if (off < 16) {
        while (d < 16) d += off;
        const uint32_t head = n < d ? n : d;
        const uint8_t* from = to - off;
        uint32_t j = 0;
        for (; k < head; ++k) {
            to[k] = from[j];
            j = j + 1 == off ? 0 : j + 1;
        }
    }
    copy_back(to + k, to + k - d, n - k, d >= 32);
}

#if defined(__CUDACC__) || defined(CDB_EMULATE)
// The warp copies n bytes (source and destination apart).
__device__ __forceinline__ void warp_copy(uint8_t* to, const uint8_t* from, uint64_t n,
                                          uint32_t lane) {
    lzg::copy_share(to, from, n, lane, 32);
    __syncwarp();
}

// The warp writes a match of n bytes; scratch: kPeriod bytes of shared memory.
__device__ __forceinline__ void warp_match(uint8_t* to, uint64_t n, uint64_t off,
                                           uint8_t* scratch, uint32_t lane) {
    if (off >= kPeriod) {
        // waves that never read their own output
        for (uint64_t k = 0; k < n; k += off)
            warp_copy(to + k, to + k - off, n - k < off ? n - k : off, lane);
    } else {
        const uint32_t f = static_cast<uint32_t>(off);
        for (uint32_t j = lane; j < f; j += 32)
            scratch[j] = to[static_cast<int64_t>(j) - static_cast<int64_t>(f)];
        __syncwarp();
        lzg::period_share(to, scratch, f, n, lane, 32);
        __syncwarp();
    }
}

// The lanes' matches (pend: a match of n bytes at position at, from off back;
// at ascends with the lane, from b0 on), each once no other pending match's
// output overlaps the bytes its source reads past b0 (everything else there
// is written). Matches start in lane order, so the pending ones starting
// below a source's end are among a prefix of the lanes, and the last of them
// ending by its start clears it; the lowest pending match always goes.
__device__ __forceinline__ void match_rounds(uint8_t* base, bool pend, uint64_t at, uint32_t n,
                                             uint64_t off, uint64_t b0, uint8_t* scratch,
                                             uint32_t lane) {
    const uint32_t rms = pend || n ? static_cast<uint32_t>(at - b0) : ~0u;
    const uint32_t rme = rms + n;
    uint32_t rs = 0, re = 0;
    if (pend) {
        const uint64_t s0 = at - off;
        const uint64_t e0 = s0 + n < at ? s0 + n : at;
        rs = s0 > b0 && s0 <= at ? static_cast<uint32_t>(s0 - b0) : 0u;
        re = e0 > b0 && e0 <= at ? static_cast<uint32_t>(e0 - b0) : 0u;
    }
    for (;;) {
        const unsigned pm = __ballot_sync(0xffffffffu, pend);
        if (!pm) break;
        uint32_t l = 0;  // the last lane whose match starts below re
#pragma unroll
        for (uint32_t st = 16; st; st >>= 1) {
            const uint32_t c = l + st;
            if (__shfl_sync(0xffffffffu, rms, c & 31) < re) l = c;
        }
        const bool below = __shfl_sync(0xffffffffu, rms, 0) < re;
        const unsigned cand = below ? pm & (l == 31 ? 0xffffffffu : ((2u << l) - 1)) : 0u;
        const uint32_t last = cand ? 31 - __clz(cand) : 0u;
        const uint32_t last_end = __shfl_sync(0xffffffffu, rme, last);
        const bool ready = pend && (re <= rs || cand == 0 || last_end <= rs);
        if (ready && n <= kLaneMax) {
            match(base + at, n, static_cast<uint32_t>(off));
            pend = false;
        }
        for (unsigned m = __ballot_sync(0xffffffffu, ready && pend); m; m &= m - 1) {
            const int k = __ffs(m) - 1;
            warp_match(base + __shfl_sync(0xffffffffu, at, k), __shfl_sync(0xffffffffu, n, k),
                       __shfl_sync(0xffffffffu, off, k), scratch, lane);
            if (lane == static_cast<uint32_t>(k)) pend = false;
        }
        __syncwarp();
    }
}

#endif

}  // namespace lanes
}  // namespace cdb
