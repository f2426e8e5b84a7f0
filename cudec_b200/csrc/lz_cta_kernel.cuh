// CTA-per-chunk decoder for the byte-oriented LZ formats (LZ4 block, raw
// Snappy): the chunk's token chain is found by every thread of the CTA
// walking a stretch of the input speculatively, tokens are parsed one per
// thread, and the output is produced one byte per lane by gathering.
//
// A chunk is decoded tile by tile. A tile is the kTile input positions that
// start at a known token (the chunk's first, then each tile's exit):
//
//   1. stage: the tile's input bytes (plus kLook bytes past it) land in
//      shared memory by cp.async, in aligned 16-byte blocks, while the tile
//      before runs;
//   2. steps and exits: the distance to the next token from every position
//      (the format's step, without branches, four positions at a time), and
//      from every position of a region (kReg positions, one region per
//      thread) the distance to the first chain position past the region,
//      computed backwards;
//   3. the regions' entries: region t is entered at region t - 1's exit. LZ
//      chains started anywhere merge after a few tokens, which two ways use:
//      settle (CTAs up to kSettle threads): every region starts from the exit
//      of its first position, so most are right at once. In a round, the
//      first region f whose entry is not its neighbour's exit takes it
//      (everything before f is right), a region that the chain leaving f - 1
//      passes over takes that exit too, and any other region takes its
//      neighbour's exit where that lies inside it; each looks its own exit
//      up. Only region f takes an uncommon step (a long extension, the
//      chunk's end). After kRounds rounds one thread follows the chain
//      through the rest, a look-up per region;
//      chase (wider ones, whose rounds are more and dearer): a warp's 32
//      regions are followed from each of their first 32 positions at once, one
//      lane each; lane 0 notes where it enters each region. One thread then
//      follows the tile's chain from warp to warp: the warp's entry is mostly
//      one of those 32 positions (or past the warp); otherwise it goes region
//      by region until it meets the chain of lane 0. Each thread then finds
//      its region's entry the same way, from its warp's;
//   4. list: each thread walks its region from its entry; a scan of the
//      counts gives every token its index, and the tokens' positions go to a
//      list;
//   5. batches of kThreads tokens, one per thread: parse (the format's fast
//      form, the exact ladder of lz_ladder.cuh where it declines), a scan of
//      the output lengths, the ladder's conditions at the token's output
//      offset (the first failing or terminal token decides the chunk as the
//      serial parser would, since the steps equal the ladder's next position
//      for every token the ladder accepts), and a map of the batch's output:
//      one start bit per output byte and the token count before each aligned
//      32-byte sector;
//   6. copy: a warp writes whole 32-byte sectors of the destination, one
//      byte per lane. A byte's token is the sector's count plus a popcount
//      of the start bits up to it; a literal byte comes from the staged
//      input, a match byte from the destination. A match byte whose source
//      lies in the same window is followed through the map (a period is
//      taken modulo its length, so a match costs one hop) until a literal
//      or a byte before the window is met, so no byte waits for another.
//      A token longer than kBig is copied by the whole CTA, 16 bytes per
//      thread at a time: an LZ4 one in its place between the batch's other
//      tokens, whose parse still holds; Snappy's (literals, and rare) and those
//      that only the ladder can read end the batch. When each ended it, and a
//      match from less than 16 bytes per thread back was always written from
//      its period, 100 chunks of 64 KiB of matches of 1,100 to 4,000 bytes took
//      269 us, 16 of 4 MiB 12,816; now 119 and 4,443.
//
// What bounds it: instruction issue and the waits between barriers (65 % of the
// issue slots at seven CTAs per SM; 254,000 warp instructions per 64 KiB chunk
// of 5,250 tokens; per issued instruction 2.2 warps wait out fixed latencies,
// 1.8 at a barrier, 0.8 for global memory). The decoder before this one
// computed chain exits by the format's branching step, merged 16-byte pieces
// per token into a shared-memory ring with atomics, and spent 568,000. 1,024
// chunks of 64 KiB on a B200: LZ4 0.943 -> 0.411 ms (163 GB/s out), Snappy
// 1.149 -> 0.432.
//
// Every phase is per-thread code between CTA barriers, driven through an
// executor: on the device each phase runs once per thread followed by
// __syncthreads(); the host executor runs the phases for every thread in
// turn, which emulates the CTA exactly (no phase reads what another thread
// writes in the same phase, except through atomics whose order does not
// change the result). The host emulation is what the CPU tests run.
//
// Statuses follow the reference ladders exactly: LZ4 iderex/cudec
// src/lz4_block.h:95-258, Snappy src/snappy_block.h:172-435.
#pragma once

#include <cstdint>
#include <cstring>

#include "cudec.h"
#include "lz_gather.cuh"
#include "lz_ladder.cuh"

namespace cdb {
namespace lzc {

constexpr uint32_t kThreads = 128;  // threads per CTA unless a chunk gets more
constexpr uint32_t kReg = 52;       // positions per region: at most 64 (a mask), an odd number of
                                    // words (no bank conflicts where the regions are walked)
constexpr uint32_t kLook = 512;     // staged bytes past the tile
using lzg::kSectors;
using lzg::kWindow;
using lzg::Rec;
using lzg::Sector;
constexpr uint32_t kBig = 1024;                    // longer tokens: whole-CTA copies
constexpr uint32_t kExtCap = 16;                   // extension bytes a fast parse reads

// What follows from the CTA's width.
template <uint32_t T>
struct Width {
    static constexpr uint32_t kWarps = T / 32;
    static constexpr uint32_t kTile = T * kReg;  // positions per tile: a region per thread
    static constexpr uint32_t kInBytes = (kTile + kLook + 32 + 15) / 16 * 16;  // staged input
    static constexpr uint32_t kUnroll = T == 128 ? 3 : 2;      // sectors in flight per warp
    static constexpr uint32_t kPart = 32 * kWarps * kUnroll;  // output bytes between barriers
    // resident CTAs per SM that the registers are compiled for
    static constexpr int kPerSm = T == 128 ? 7 : T == 256 ? 3 : 1;
};

static_assert(kReg <= 64 && kReg % 8 == 4, "a region's mask is one word; odd in 4-byte words");

// Region exits: positions relative to the tile's entry, or
constexpr uint32_t kExitEnd = 0xFFFFFFFFu;   // the chain ends (its last token is noted)
constexpr uint32_t kExitFar = 0xFFFFFFFEu;   // 2^31 or further: s.far
constexpr uint32_t kExitOpen = 0xFFFFFFFDu;  // a step left open: not known to be on the chain
constexpr uint32_t kExitMax = 0x80000000u;   // positions are below this

// Step results (absolute positions otherwise).
constexpr uint64_t kStepEnd = ~0ull;
constexpr uint64_t kLenMax = 65536;  // a batch clamps longer tokens, which are its last
constexpr uint32_t kSlowRel = 0xFFFFFFFFu;  // a fast step declines: the generic step decides
constexpr uint32_t kStepSlow = 255;         // no short step from this position
// Widest CTA whose regions are settled in rounds rather than chased. Us with
// rounds / chased: 512 threads, 148 LZ4 chunks of 64 KiB 168 / 136, 16 of 4 MiB
// 9,151 / 6,050 (few tokens per region: 13 rounds and a serial rest per tile);
// 128 threads, 1,024 Snappy chunks of 64 KiB 430 / 438, 8,192 LZ4 chunks of
// 8 KiB 453 / 471.
constexpr uint32_t kSettle = 128;
constexpr uint32_t kRounds = 12;            // settling rounds before the serial finish

// ---------------------------------------------------------------------------
// Portable primitives (device: the real thing; host: the sequential
// emulation's plain operations).
#if CDB_DEVICE_CODE
#define LZC_LDG(p) __ldg(p)
__device__ __forceinline__ void at_min(uint32_t* a, uint32_t v) { atomicMin(a, v); }
__device__ __forceinline__ uint32_t pop64(uint64_t v) { return __popcll(v); }
__device__ __forceinline__ uint32_t ctz64(uint64_t v) { return __ffsll(v) - 1; }
#else
#define LZC_LDG(p) (*(p))
inline void at_min(uint32_t* a, uint32_t v) {
    if (v < *a) *a = v;
}
inline uint32_t pop64(uint64_t v) { return static_cast<uint32_t>(__builtin_popcountll(v)); }
inline uint32_t ctz64(uint64_t v) { return static_cast<uint32_t>(__builtin_ctzll(v)); }
#endif

// Profiling builds (-DCDB_PHASE_TIMING) accumulate, from thread 0 of every
// CTA, the SM cycles of each phase and event counts over a launch. Cycles:
// 0 stage, 1 steps, 2 exits and entries, 3 list, 4 parse and scan, 5 check and map,
// 6 copy, 7 whole-CTA tokens. Events: 0 tiles, 1 tokens, 2 settle rounds or
// regions chased, 3 batches, 4 whole-CTA tokens, 5 windows.
#if defined(CDB_PHASE_TIMING) && defined(__CUDACC__)
__device__ unsigned long long lzc_cycles[16];
__device__ unsigned long long lzc_events[16];
#endif
#if defined(CDB_PHASE_TIMING) && defined(__CUDA_ARCH__)
#define LZC_PHASE(i)                                                                    \
    do {                                                                                \
        if (threadIdx.x == 0) {                                                         \
            const long long n_ = clock64();                                             \
            atomicAdd(&lzc_cycles[i], static_cast<unsigned long long>(n_ - tl));        \
            tl = n_;                                                                    \
        }                                                                               \
    } while (0)
#define LZC_EVENT(i, n)                                                                 \
    do {                                                                                \
        if (threadIdx.x == 0) atomicAdd(&lzc_events[i], static_cast<unsigned long long>(n)); \
    } while (0)
#define LZC_START() tl = clock64()
#else
#define LZC_PHASE(i) \
    do {             \
    } while (0)
#define LZC_EVENT(i, n) \
    do {                \
    } while (0)
#define LZC_START() \
    do {            \
    } while (0)
#endif

#if defined(__CUDACC__)
#define LZC_APART __host__ __device__ __noinline__
#else
#define LZC_APART inline
#endif

// ---------------------------------------------------------------------------
// Phases. each(fn): fn(tid) for every thread of the CTA, then a barrier (on
// the host: every thread in turn). The host forms emulate the CTA
// sequentially.
template <uint32_t kThreads, class Fn>
CDB_HD void each(Fn fn) {
#if CDB_DEVICE_CODE
    fn(threadIdx.x);
    __syncthreads();
#else
    for (uint32_t t = 0; t < kThreads; ++t) fn(t);
#endif
}

// The same without the barrier.
template <uint32_t kThreads, class Fn>
CDB_HD void each_free(Fn fn) {
#if CDB_DEVICE_CODE
    fn(threadIdx.x);
#else
    for (uint32_t t = 0; t < kThreads; ++t) fn(t);
#endif
}

// each(), with the threads whose call returned true as a bit each in words.
template <uint32_t kThreads, class Fn>
CDB_HD void vote(uint32_t* words, Fn fn) {
#if CDB_DEVICE_CODE
    const uint32_t b = __ballot_sync(0xffffffffu, fn(threadIdx.x));
    if ((threadIdx.x & 31) == 0) words[threadIdx.x >> 5] = b;
    __syncthreads();
#else
    for (uint32_t t = 0; t < kThreads; ++t) {
        if (t % 32 == 0) words[t / 32] = 0;
        if (fn(t)) words[t / 32] |= 1u << (t % 32);
    }
#endif
}

// A value that each thread keeps from phase to phase: a register on the
// device, one slot per thread on the host.
template <class V, uint32_t kThreads>
struct Priv {
#if CDB_DEVICE_CODE
    V v;
    __device__ __forceinline__ V& operator[](uint32_t) { return v; }
#else
    V v[kThreads];
    V& operator[](uint32_t t) { return v[t]; }
#endif
};

// 16 bytes global -> shared (an aligned block); completed by land().
CDB_HD void copy16_async(uint8_t* d, const uint8_t* src) {
#if defined(__CUDA_ARCH__)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(d))),
                 "l"(src)
                 : "memory");
#else
    std::memcpy(d, src, 16);
#endif
}
CDB_HD void land_async() {
#if defined(__CUDA_ARCH__)
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_all;" ::: "memory");
#endif
}
// ---------------------------------------------------------------------------
// Formats: the exact ladder plus the step of the walk and the fast parse.

// The staged bytes by position relative to the tile's entry.
struct Staged {
    const uint8_t* in;  // the staging buffer, 16-byte aligned
    uint32_t at0;       // the entry's index in it
    CDB_HD uint32_t at(uint32_t r) const { return in[at0 + r]; }
    CDB_HD uint32_t word(uint32_t r) const {  // the four bytes from r
        const uint32_t i = at0 + r;
        const uint32_t* w = reinterpret_cast<const uint32_t*>(in) + (i >> 2);
        return lzg::fsr(w[0], w[1], 8 * (i & 3));
    }
};

// A token's fields as the fast parse reads them; positions relative to the
// tile's entry.
struct Tok {
    uint32_t lit, ml, off;
    uint32_t ls;  // position of the literal run
};

// LZ4: next = the ladder's next position for every token it accepts as
// non-terminal; kStepEnd when the token can have no successor (the ladder
// then answers terminal or reject).
struct Lz4F : lzl::Lz4Ladder {
    static constexpr uint32_t kMinStep = 3;  // tokens with a successor span >= 3 bytes
    static constexpr bool kSnappy = false;

    // kLen: only *olen is asked for, and above kLenMax only that it is.
    template <bool kLen = false, class R>
    CDB_HD static uint64_t step(const R& in, uint64_t S, uint64_t P, uint64_t* olen) {
        if (P >= S) return kStepEnd;
        const uint32_t tok = in.at(P);
        uint64_t q = P + 1;
        uint64_t lit = tok >> 4;
        uint32_t b;
        if (lit == 15) {
            do {
                if (q >= S) return kStepEnd;
                b = in.at(q++);
                lit += b;
            } while (b == 255 && !(kLen && lit > kLenMax));
        }
        *olen = lit;
        if (kLen && lit > kLenMax) return kStepEnd;
        if (lit > S - q || S - q - lit < kSrcSlack) return kStepEnd;
        q += lit + 2;
        uint64_t ml = (tok & 15) + 4;
        if ((tok & 15) == 15) {
            do {
                if (q >= S) return kStepEnd;
                b = in.at(q++);
                ml += b;
            } while (b == 255 && !(kLen && ml > kLenMax));
        }
        *olen = lit + ml;
        return q;
    }

    // The step over the staged bytes without branches, for a token whose
    // header (with at most one extension byte per length, below 255) lies
    // well inside them and well before the chunk's end: word(in, r) are the
    // four bytes from position r, lim = min(staged bytes, rest), rest = bytes
    // to the chunk's end. kSlowRel: the other forms decide.
    static constexpr uint32_t kMargin = 2 * kExtCap + 2 + kSrcSlack;
    CDB_HD static uint32_t hop_rel(const Staged& in, uint32_t r, uint32_t lim, uint32_t) {
        if (r + kMargin > lim) return kSlowRel;
        const uint32_t u = in.word(r);
        uint32_t lit = (u >> 4) & 15;
        const uint32_t x1 = (u >> 8) & 255, e = lit == 15;
        lit += e ? x1 : 0;
        const uint32_t q = r + 1 + e + lit;  // the offset's position
        if (q + 2 + kExtCap + kSrcSlack > lim) return kSlowRel;
        const bool m = (u & 15) == 15;
        const bool far = (e && x1 == 255) || (m && in.at(q + 2) == 255);
        return far ? kSlowRel : q + 2 + m;
    }
    // hop_rel's distances from positions r..r+3 (r a multiple of 4), a byte
    // each, all four at once; kStepSlow where it declines or the distance is
    // longer than 146.
    CDB_HD static uint32_t steps_rel(const Staged& in, uint32_t r, uint32_t lim) {
        if (r + 3 + 160 + kMargin > lim) return steps_end(in, r, lim);
        const uint32_t u = in.word(r), x1 = lzg::fsr(u, in.word(r + 4), 8);
        constexpr uint32_t k1 = 0x01010101u;
        const uint32_t lit = (u >> 4) & 0x0f0f0f0fu;
        const uint32_t e = ((lit + k1) >> 4) & k1;                // an extended literal length
        const uint32_t m = (((u & 0x0f0f0f0fu) + k1) >> 4) & k1;  // an extended match length
        const uint32_t x = x1 & (e * 255);
        uint32_t slow = ((x >> 7) & k1) * 255;  // extension bytes from 128 up
        const uint32_t n = lit + 3 * k1 + e + (x & 0x7f7f7f7fu);  // past the offset: 3..146
        if (m) {  // declined where the match's extension byte is 255
            LZG_UNROLL
            for (uint32_t j = 0; j < 4; ++j)
                if (((m >> (8 * j)) & 1) && in.at(r + j + ((n >> (8 * j)) & 255)) == 255)
                    slow |= 255u << (8 * j);
        }
        return (n + m) | slow;
    }
    CDB_HD static uint32_t steps_end(const Staged& in, uint32_t r, uint32_t lim) {
        uint32_t out = 0;
        for (uint32_t j = 0; j < 4; ++j) {
            const uint32_t n = hop_rel(in, r + j, lim, 0);
            out |= (n != kSlowRel && n - r - j < kStepSlow ? n - r - j : kStepSlow) << (8 * j);
        }
        return out;
    }
    CDB_HD static bool ext_rel(const Staged& in, uint32_t* q, uint32_t* len) {
        for (uint32_t k = 0; k < kExtCap; ++k) {
            const uint32_t x = in.at((*q)++);
            *len += x;
            if (x != 255) return true;
        }
        return false;
    }
    // The token's fields: with at most one extension byte per length without
    // branches, with up to kExtCap in loops. Returns the next token's
    // position; kSlowRel: the generic forms decide.
    CDB_HD static uint32_t parse_rel(const Staged& in, uint32_t r, uint32_t lim, Tok* t) {
        if (r + kMargin > lim) return kSlowRel;
        const uint32_t u = in.word(r);
        uint32_t lit = (u >> 4) & 15, ml = (u & 15) + 4;
        const uint32_t x1 = (u >> 8) & 255, e = lit == 15, m = ml == 19;
        lit += e ? x1 : 0;
        uint32_t q = r + 1 + e + lit;
        if (q + 2 + kExtCap + kSrcSlack <= lim) {
            const uint32_t v = in.word(q), x2 = (v >> 16) & 255;
            if (!(e && x1 == 255) && !(m && x2 == 255)) {
                t->ls = r + 1 + e;
                t->lit = lit;
                t->off = v & 0xffff;
                t->ml = ml + (m ? x2 : 0);
                return q + 2 + m;
            }
        }
        q = r + 1;
        lit = (u >> 4) & 15;
        if (lit == 15 && !ext_rel(in, &q, &lit)) return kSlowRel;
        t->ls = q;
        t->lit = lit;
        q += lit;
        if (q + 2 + kExtCap + kSrcSlack > lim) return kSlowRel;
        t->off = in.at(q) | (in.at(q + 1) << 8);
        q += 2;
        if (ml == 19 && !ext_rel(in, &q, &ml)) return kSlowRel;
        t->ml = ml;
        return q;
    }
    // Whether the ladder accepts such a token as non-terminal, `out` bytes
    // into a batch that has `have` bytes before it and room for `room` (both
    // clamped below 2^31): its conditions (src/lz4_block.h:139-258) on the
    // final lengths (the extension loops' running checks only fail when the
    // final values fail them); false: the full ladder decides.
    CDB_HD static bool admit(const Tok& t, uint32_t out, uint32_t have, uint32_t room) {
        const uint32_t used = out + t.lit;
        return used + kMfLimit <= room && t.off - 1 < have + used &&
               used + t.ml + kLastLiterals <= room;
    }
};

// Raw Snappy: one element per step; an element that ends at S steps to S
// (the chunk's end: Snappy's finish decides there).
struct SnappyF : lzl::SnappyLadder {
    static constexpr uint32_t kMinStep = 2;  // elements span >= 2 bytes
    static constexpr bool kSnappy = true;

    template <bool kLen = false, class R>
    CDB_HD static uint64_t step(const R& in, uint64_t S, uint64_t P, uint64_t* olen) {
        if (P >= S) return kStepEnd;
        const uint32_t tag = in.at(P);
        const uint32_t kind = tag & 3;
        if (kind == 0) {
            const uint32_t l6 = tag >> 2;
            uint64_t hdr = 1, n = l6;
            if (l6 >= 60) {
                const uint32_t extra = l6 - 59;
                if (extra > S - P - 1) return kStepEnd;
                n = 0;
                for (uint32_t i = 0; i < extra; ++i)
                    n |= static_cast<uint64_t>(in.at(P + 1 + i)) << (8 * i);
                hdr += extra;
            }
            n += 1;
            const uint64_t q = P + hdr;
            *olen = n;
            if (n > S - q) return kStepEnd;
            return q + n;
        }
        const uint64_t hdr = kind == 1 ? 2 : (kind == 2 ? 3 : 5);
        *olen = kind == 1 ? 4 + ((tag >> 2) & 7) : (tag >> 2) + 1;
        if (hdr > S - P) return kStepEnd;
        return P + hdr;
    }

    // The fast forms (see Lz4F): every element but a literal with a four-byte
    // length.
    CDB_HD static uint32_t fields(const Staged& in, uint32_t r, uint32_t* len, uint32_t* u) {
        *u = in.word(r);
        const uint32_t kind = *u & 3, l6 = (*u >> 2) & 63;
        const uint32_t ext = l6 >= 60 ? l6 - 59 : 0;  // bytes of the literal's length
        const uint32_t n = (ext ? (*u >> 8) & (0xffffffu >> (24 - 8 * (ext & 3))) : l6) + 1;
        *len = kind == 0 ? n : kind == 1 ? 4 + (l6 & 7) : l6 + 1;
        if (kind == 0) return ext == 4 ? kSlowRel : r + 1 + ext + n;
        return r + (kind == 3 ? 5 : 1 + kind);
    }
    CDB_HD static uint32_t steps_rel(const Staged& in, uint32_t r, uint32_t lim) {
        if (r + 70 > lim) return 0xffffffffu;  // lim <= the chunk's end
        const uint32_t u = in.word(r);
        constexpr uint32_t k1 = 0x01010101u;
        const uint32_t kind = u & 3 * k1, l6 = (u >> 2) & 63 * k1;
        const uint32_t lit = (((kind | (kind >> 1)) & k1) ^ k1) * 255;  // literals
        const uint32_t copy = kind + k1 + ((kind >> 1) & kind & k1);    // 2, 3, 5
        const uint32_t slow = (((l6 + 4 * k1) >> 6) & k1) * 255;        // a length of its own
        return (lit & ((l6 + 2 * k1) | slow)) | (copy & ~lit);
    }
    CDB_HD static uint32_t hop_rel(const Staged& in, uint32_t r, uint32_t lim, uint32_t rest) {
        if (r + 5 > lim) return kSlowRel;
        uint32_t len, u;
        const uint32_t nx = fields(in, r, &len, &u);
        return nx <= rest ? nx : kSlowRel;  // may lie past the staged bytes
    }
    CDB_HD static uint32_t parse_rel(const Staged& in, uint32_t r, uint32_t lim, Tok* t) {
        if (r + 5 > lim) return kSlowRel;
        uint32_t len, u;
        const uint32_t nx = fields(in, r, &len, &u);
        if (nx > lim) return kSlowRel;
        const uint32_t kind = u & 3;
        if (kind == 0) {
            t->ls = nx - len;
            t->lit = len;
            t->ml = 0;
            t->off = 1;
        } else {
            t->ls = r;
            t->lit = 0;
            t->ml = len;
            t->off = kind == 1   ? ((u & 0xe0) << 3) | ((u >> 8) & 255)
                     : kind == 2 ? (u >> 8) & 0xffff
                                 : (u >> 8) | (in.at(r + 4) << 24);
        }
        return nx;
    }
    // Whether the ladder (src/snappy_block.h:249-435) accepts such an element
    // (see Lz4F); false: the full ladder decides.
    CDB_HD static bool admit(const Tok& t, uint32_t out, uint32_t have, uint32_t room) {
        return out + t.lit + t.ml <= room && (t.ml == 0 || t.off - 1 < have + out);
    }
};

// ---------------------------------------------------------------------------
// What ends a batch early, its first event: a failing or terminal token, or one
// whose lengths only the ladder tells. And the batch's first long token.
struct Cut {
    uint32_t event, big;
};
// An event token's code: its status when it fails, or
constexpr int32_t kEnd = CUDEC_OK;    // terminal, executed with the batch
constexpr int32_t kFar = INT32_MIN;   // copied by exec_far()

// Shared memory of one CTA. The input is staged in two buffers in turn: the
// next tile's bytes land while this one's tokens run.
template <class F, uint32_t kThreads = lzc::kThreads>
struct Shm : Width<kThreads> {
    using Width<kThreads>::kTile, Width<kThreads>::kInBytes, Width<kThreads>::kWarps;
    static constexpr uint32_t kMaxTok = kTile / F::kMinStep + 3;  // tokens of a tile
    alignas(16) uint8_t in[2][kInBytes];
    union {
        struct {  // finding the tile's tokens
            uint32_t step[kTile / 4];   // bytes: distance to the next token, kStepSlow
            uint32_t exit[kTile / 4];   // bytes: distance to the region's exit, kStepSlow
        } w;
        struct {  // executing them
            Rec rec[kThreads];
            Sector map[kSectors];
            uint16_t pos[kMaxTok];   // the tile's tokens, relative to its entry
            uint8_t period[16 * kThreads];  // whole-CTA copies: a short match's period
        } e;
    } u;
    // settle: where each region is left and (finish) entered, which of them
    // are, and the threads whose region is not settled (in the batches: whose
    // token is long); chase: where the chain
    // from a warp's position number `lane` leaves the warp's regions, where
    // lane 0's enters each of them, where the tile's chain enters the warp's
    // and leaves the tile
    uint32_t exit[kThreads], entry[kThreads];
    uint32_t entered[kWarps], votes[kWarps];
    uint32_t tile_exit;
    int32_t event[kThreads];    // an event token's code
    uint32_t wsum[2][kWarps];   // scans: per-warp totals, used in turn
    Cut cut[2];                 // batches in turn
    uint64_t far;               // the successor past 2^31, see kExitFar
};

// Input reader over the staged tile with the chunk's global bytes behind it
// (the ladders read only positions below S).
struct Reader {
    const uint8_t* g;
    const uint8_t* buf;
    uint64_t ibase;
    uint32_t staged;
    CDB_HD uint32_t at(uint64_t q) const {
        const uint64_t r = q - ibase;
        return r < staged ? buf[r] : LZC_LDG(g + q);
    }
};

// ---------------------------------------------------------------------------
// The chunk decoder (every thread of the CTA runs it; control flow depends
// only on values that every thread holds or that a barrier published).
template <class F, uint32_t kThreads = lzc::kThreads>
struct Chunk {
    using W_ = Width<kThreads>;
    static constexpr uint32_t kWarps = W_::kWarps, kTile = W_::kTile, kInBytes = W_::kInBytes;
    static constexpr uint32_t kUnroll = W_::kUnroll, kPart = W_::kPart;
    static constexpr uint32_t kMaxTok = Shm<F, kThreads>::kMaxTok;
    template <class V>
    using Priv = lzc::Priv<V, kThreads>;
    template <class Fn>
    CDB_HD static void each(Fn fn) {
        lzc::each<kThreads>(fn);
    }
    template <class Fn>
    CDB_HD static void each_free(Fn fn) {
        lzc::each_free<kThreads>(fn);
    }
    template <class Fn>
    CDB_HD static void vote(uint32_t* words, Fn fn) {
        lzc::vote<kThreads>(words, fn);
    }

    Shm<F, kThreads>& s;
    const uint8_t* g;  // compressed chunk
    uint64_t S;
    uint8_t* dst;
    uint64_t cap;
    uint64_t limit;      // LZ4: capacity; Snappy: declared length
    uint64_t e = 0;      // tile entry (absolute input position)
    uint64_t ibase = 0;  // staged input base (absolute position)
    uint64_t d = 0;      // output bytes produced
    uint32_t buf = 0;    // the staging buffer of this tile
    uint32_t turn = 0, cut_turn = 0;  // which of the alternating buffers are in use
    long long tl = 0;    // profiling builds: thread 0's last phase mark

    CDB_HD Reader reader() const { return Reader{g, s.in[buf], ibase, kInBytes}; }
    // The staged bytes from the tile entry on, and how many of them the fast
    // forms may read (also bounded by the chunk's end).
    CDB_HD uint32_t staged_at() const { return static_cast<uint32_t>(e - ibase); }
    CDB_HD uint32_t staged_lim() const {
        const uint32_t avail = kInBytes - staged_at();
        const uint64_t rest = S > e ? S - e : 0;
        return rest < avail ? static_cast<uint32_t>(rest) : avail;
    }

    // Exclusive scan of v over the CTA; returns the total. One barrier.
    CDB_HD uint32_t scan(Priv<uint32_t>& v, Priv<uint32_t>& excl) {
        uint32_t total = 0;
#if CDB_DEVICE_CODE
        const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        uint32_t* ws = s.wsum[turn];
        turn ^= 1;
        uint32_t x = v.v;
#pragma unroll
        for (uint32_t k = 1; k < 32; k <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, k);
            if (lane >= k) x += y;
        }
        if (lane == 31) ws[w] = x;
        __syncthreads();
        uint32_t before = 0;
#pragma unroll
        for (uint32_t k = 0; k < kWarps; ++k) {
            const uint32_t y = ws[k];
            if (k < w) before += y;
            total += y;
        }
        excl.v = before + x - v.v;
#else
        for (uint32_t t = 0; t < kThreads; ++t) {
            excl[t] = total;
            total += v[t];
        }
#endif
        return total;
    }

    // ---- 1. stage the input of the tile at `from` in buffer `to`: aligned
    // blocks holding at least one byte of [0, S) only; landed by land().
    CDB_HD static uint64_t base_of(const uint8_t* g, uint64_t from) {
        return from - ((reinterpret_cast<uintptr_t>(g) + from) & 15);  // may wrap below zero
    }
    CDB_HD void stage(uint64_t from, uint32_t to) {
        const int64_t ib = static_cast<int64_t>(base_of(g, from));
        each_free([&](uint32_t t) {
            for (uint32_t b = 16 * t; b < kInBytes; b += 16 * kThreads) {
                const int64_t q = ib + b;
                if (q + 16 <= 0 || q >= static_cast<int64_t>(S)) continue;
                copy16_async(s.in[to] + b, g + q);
            }
        });
    }
    CDB_HD void land() {
        each([&](uint32_t) { land_async(); });
    }

    // The distances to the next token from every position of the tile, by
    // the format's step (bytes of s.u.w.step; kStepSlow: hop() looks closer).
    CDB_HD void steps(uint32_t lim) {
        const Staged in{s.in[buf], staged_at()};
        each([&](uint32_t t) {
            for (uint32_t i = t; i < kTile / 4; i += kThreads)
                s.u.w.step[i] = F::steps_rel(in, 4 * i, lim);
        });
    }

    // Region t's exits: from each of its positions the distance to the first
    // chain position past the region (bytes of s.u.w.exit; kStepSlow where a
    // step on the way is, or the distance is longer). Backwards, kMinStep
    // positions at a time: none of them leads to another.
    CDB_HD void exits(uint32_t t) {
        const uint8_t* step = reinterpret_cast<const uint8_t*>(s.u.w.step);
        uint8_t* ex = reinterpret_cast<uint8_t*>(s.u.w.exit);
        const uint32_t lo = t * kReg, hi = lo + kReg;
        constexpr uint32_t G = F::kMinStep;
        static_assert(kReg % G == 0 || kReg % G == 1, "whole groups, one position at most left");
        uint32_t p = hi;
        while (p >= lo + G) {
            uint32_t d[G], e[G];
            LZG_UNROLL
            for (uint32_t j = 0; j < G; ++j) d[j] = step[p - 1 - j];
            LZG_UNROLL
            for (uint32_t j = 0; j < G; ++j) {
                const uint32_t n = p - 1 - j + d[j];
                e[j] = n < hi ? ex[n] : 0u;
            }
            LZG_UNROLL
            for (uint32_t j = 0; j < G; ++j) {
                const uint32_t x = d[j] + e[j];
                ex[p - 1 - j] = static_cast<uint8_t>(x < kStepSlow ? x : kStepSlow);
            }
            p -= G;
        }
        if (p > lo) {
            const uint32_t d = step[lo], n = lo + d, x = d + (n < hi ? ex[n] : 0u);
            ex[lo] = static_cast<uint8_t>(x < kStepSlow ? x : kStepSlow);
        }
    }

    // The step from position p (relative to the tile's entry), which is on
    // the chain: the next token's relative position or an exit code.
    CDB_HD uint32_t hop(uint32_t lim, uint32_t rest, uint32_t p) const {
        const uint32_t d = reinterpret_cast<const uint8_t*>(s.u.w.step)[p];
        if (d != kStepSlow) return p + d;
        const Staged in{s.in[buf], staged_at()};
        const uint32_t n = F::hop_rel(in, p, lim, rest);
        if (n != kSlowRel) return n;
        const uint64_t P = e + p;
        if (P >= S) return kExitEnd;
        uint64_t ol = 0;
        const uint64_t nx = F::step(reader(), S, P, &ol);
        if (nx == kStepEnd) return kExitEnd;
        if (nx - e < kExitMax) return static_cast<uint32_t>(nx - e);
        s.far = nx;  // every later region is passed over
        return kExitFar;
    }

    // Where the tile's chain, which is at p in region r, leaves the region.
    CDB_HD uint32_t leave(uint32_t lim, uint32_t rest, uint32_t r, uint32_t p) const {
        const uint32_t d = reinterpret_cast<const uint8_t*>(s.u.w.exit)[p];
        if (d != kStepSlow) return p + d;
        while (p < (r + 1) * kReg) p = hop(lim, rest, p);
        return p;
    }

    // Not `sure`: p may not be on the chain, so a way with an uncommon step is
    // left open.
    CDB_HD uint32_t leave_if_sure(uint32_t lim, uint32_t rest, uint32_t r, uint32_t p,
                                  bool sure) const {
        const uint32_t d = reinterpret_cast<const uint8_t*>(s.u.w.exit)[p];
        return d != kStepSlow ? p + d : sure ? leave(lim, rest, r, p) : kExitOpen;
    }

    // The chain from region f on, entered at `sure`: one thread follows it
    // from region to region.
    CDB_HD void finish(uint32_t lim, uint32_t rest, uint32_t f, uint32_t sure,
                       Priv<uint32_t>& entry) {
        each([&](uint32_t t) {
            if (t < kWarps) s.entered[t] = 0;  // (votes are still being read)
        });
        each([&](uint32_t t) {
            if (t != 0) return;
            uint32_t p = sure;
            while (p < kTile) {
                const uint32_t r = p / kReg;
                s.entry[r] = p;
                s.entered[r / 32] |= 1u << (r % 32);
                p = leave(lim, rest, r, p);
            }
            s.tile_exit = p;
        });
        each_free([&](uint32_t t) {
            if (t >= f) entry[t] = (s.entered[t / 32] >> (t % 32)) & 1 ? s.entry[t] : kExitEnd;
        });
    }

    // The regions' entries and the tile's exit by rounds of neighbours.
    CDB_HD void settle(uint32_t lim, uint32_t rest, Priv<uint32_t>& entry) {
        Priv<uint32_t> next;
        each([&](uint32_t t) {
            entry[t] = t * kReg;
            s.exit[t] = leave_if_sure(lim, rest, t, t * kReg, t == 0);
        });
        for (uint32_t round = 0;; ++round) {
            LZC_EVENT(2, 1);
            vote(s.votes, [&](uint32_t t) {
                next[t] = t ? s.exit[t - 1] : 0;
                return next[t] != entry[t] || s.exit[t] == kExitOpen;
            });
            uint32_t f = kThreads;  // the first region that is not settled
            for (uint32_t w = kWarps; w-- > 0;)
                if (s.votes[w]) f = 32 * w + ctz64(s.votes[w]);
            if (f == kThreads) {
                each([&](uint32_t t) {
                    if (t == kThreads - 1) s.tile_exit = s.exit[t];
                });
                return;
            }
            const uint32_t sure = f ? s.exit[f - 1] : 0;
            if (round == kRounds) {
                return finish(lim, rest, f, sure, entry);
            }
            each([&](uint32_t t) {
                const uint32_t hi = (t + 1) * kReg;
                uint32_t p = next[t];
                if (t < f) return;
                if (t > f) {
                    if (sure >= hi) p = sure;
                    else if (p >= hi) return;
                    if (p == entry[t]) return;
                }
                entry[t] = p;
                s.exit[t] = p < hi ? leave_if_sure(lim, rest, t, p, t == f) : p;
            });
        }
    }

    // The chain from position t % 32 of its warp's regions to past them. Where
    // a region's exit is not noted, by the format's steps in the staged bytes
    // (merged lanes take them together).
    CDB_HD void follow(uint32_t lim, uint32_t rest, uint32_t t) {
        constexpr uint32_t kSpan = 32 * kReg;  // positions of a warp
        const uint8_t* step = reinterpret_cast<const uint8_t*>(s.u.w.step);
        const uint8_t* ex = reinterpret_cast<const uint8_t*>(s.u.w.exit);
        const Staged in{s.in[buf], staged_at()};
        const uint32_t lane = t % 32, lo = t / 32 * kSpan, hi = lo + kSpan;
        uint32_t p = lo + lane;
        while (p < hi) {
            if (lane == 0) s.entry[p / kReg] = p;
            const uint32_t d = ex[p];
            if (d != kStepSlow) {
                p += d;
                continue;
            }
            const uint32_t end = (p / kReg + 1) * kReg;
            while (p < end) {
                const uint32_t h = step[p];
                p = h != kStepSlow ? p + h : F::hop_rel(in, p, lim, rest);
                if (p == kSlowRel) p = kExitOpen;
            }
        }
        s.exit[t] = p;
    }

    // The tile's chain from warp to warp (one thread).
    CDB_HD void chase(uint32_t lim, uint32_t rest) {
        constexpr uint32_t kSpan = 32 * kReg;
        uint32_t p = 0;
        for (uint32_t w = 0; w < kWarps; ++w) {
            const uint32_t lo = w * kSpan, hi = lo + kSpan;
            s.entered[w] = p;
            if (p >= hi) continue;
            uint32_t to = p - lo < 32 ? s.exit[32 * w + p - lo] : kExitOpen;
            while (to == kExitOpen && p < hi) {
                LZC_EVENT(2, 1);
                const uint32_t r = p / kReg;
                if (s.entry[r] == p) to = s.exit[32 * w];
                if (to == kExitOpen) p = leave(lim, rest, r, p);
            }
            if (to != kExitOpen) p = to;
        }
        s.tile_exit = p;
    }

    // Where the tile's chain enters region t (past it: it does not).
    CDB_HD uint32_t enter(uint32_t lim, uint32_t rest, uint32_t t) const {
        uint32_t p = s.entered[t / 32];
        while (p < t * kReg) {
            const uint32_t r = p / kReg;
            if (s.entry[r] == p && s.exit[t & ~31u] != kExitOpen) return s.entry[t];
            p = leave(lim, rest, r, p);
        }
        return p;
    }

    // ---- 2.-5. the tile's tokens: their positions in s.u.e.pos, their count,
    // and the tile's exit (absolute; kStepEnd when the chain ends).
    CDB_HD uint32_t find_tokens(uint64_t* exit) {
        const uint32_t lim = staged_lim();
        const uint64_t left = S - e;
        const uint32_t rest = left < kExitMax ? static_cast<uint32_t>(left) : kExitMax - 1;
        steps(lim);
        LZC_PHASE(1);
        Priv<uint32_t> entry;
        if constexpr (kThreads <= kSettle) {
            each_free([&](uint32_t t) { exits(t); });
            settle(lim, rest, entry);
        } else {
            each([&](uint32_t t) {
                exits(t);
                s.entry[t] = kExitEnd;
            });
            each([&](uint32_t t) { follow(lim, rest, t); });
            each([&](uint32_t t) {
                if (t == 0) chase(lim, rest);
            });
            each_free([&](uint32_t t) { entry[t] = enter(lim, rest, t); });
        }
        LZC_PHASE(2);
        const uint32_t x = s.tile_exit;
        *exit = x == kExitEnd ? kStepEnd : x == kExitFar ? s.far : e + x;
        if (*exit < S) stage(*exit, buf ^ 1);  // lands while this tile's tokens run
        Priv<uint64_t> mask;
        each_free([&](uint32_t t) {
            const uint32_t lo = t * kReg;
            mask[t] = 0;
            for (uint32_t p = entry[t]; p < lo + kReg; p = hop(lim, rest, p))
                mask[t] |= 1ull << (p - lo);
        });
        Priv<uint32_t> cnt, at;
        each_free([&](uint32_t t) { cnt[t] = pop64(mask[t]); });
        const uint32_t ntok = scan(cnt, at);
        if (ntok <= kMaxTok)
            each([&](uint32_t t) {
                uint32_t i = at[t];
                for (uint64_t m = mask[t]; m; m &= m - 1)
                    s.u.e.pos[i++] = static_cast<uint16_t>(t * kReg + ctz64(m));
            });
        LZC_PHASE(3);
        return ntok;
    }

    // The ladder's answer for the token at P with dt bytes before it.
    CDB_HD int ladder_at(uint64_t P, uint64_t dt, lzl::Seq* sq) const {
        *sq = lzl::Seq{};
        if (F::kSnappy && P == S) {
            sq->done = true;
            return F::finish(dt, limit);
        }
        return F::parse(reader(), S, limit, P, dt, sq);
    }

    // ---- 6. write the batch's output bytes [y0, y1) that lie in the window
    // at W (both relative to the batch's first sector, at base), kPart bytes
    // at a time: kUnroll sectors per warp, then a barrier, so that only the
    // sources inside a part have to be followed through the map.
    CDB_HD void copy_window(uint8_t* base, uint32_t y0, uint32_t y1, uint32_t W) {
        const uint32_t begin = y0 > W ? y0 - W : 0;
        const uint32_t hi = y1 - W < kWindow ? y1 - W : kWindow;
        uint8_t* wb = base + W;
        const uint8_t* in = s.in[buf];
        for (uint32_t part = begin / kPart * kPart; part < hi; part += kPart) {
            const uint32_t lo = part > begin ? part : begin;
            each([&](uint32_t t) {
                const uint32_t lane = t % 32, k = part / 32 + t / 32;
                if (32 * k >= hi) return;
                lzg::Source src[kUnroll];
                lzg::sources<kUnroll, kThreads>(s.u.e.map, s.u.e.rec, k, kWarps, lane, lo, hi, W,
                                                src);
                // literal and match bytes in registers of their own: with one
                // for both, the second load would wait for the first
                uint32_t a[kUnroll], m[kUnroll];
                LZG_UNROLL
                for (uint32_t j = 0; j < kUnroll; ++j) {
                    a[j] = m[j] = 0;
                    if (src[j].ok && !src[j].lit) m[j] = wb[src[j].at];
                    if (src[j].ok && src[j].lit) a[j] = in[src[j].at];
                }
                uint8_t* y = wb + 32 * k + lane;
                LZG_UNROLL
                for (uint32_t j = 0; j < kUnroll; ++j)
                    if (src[j].ok) y[32 * j * kWarps] = static_cast<uint8_t>(a[j] | m[j]);
            });
        }
    }

    // A match of ml bytes at `to`, every byte before it written, by the whole
    // CTA: in waves that never read their own output, or from its period.
    CDB_HD void copy_match(uint8_t* to, uint64_t ml, uint64_t off) {
        if (off >= 16 * kThreads || ml <= off) {
            for (uint64_t k = 0; k < ml; k += off)
                each([&](uint32_t t) {
                    lzg::copy_share(to + k, to + k - off, ml - k < off ? ml - k : off, t,
                                    kThreads);
                });
        } else {
            const uint32_t f = static_cast<uint32_t>(off);
            each([&](uint32_t t) {
                for (uint32_t j = t; j < f; j += kThreads)
                    s.u.e.period[j] = (to - off)[j];
            });
            each([&](uint32_t t) {
                lzg::period_share(to, s.u.e.period, f, ml, t, kThreads);
            });
        }
    }

    // A long token of a batch (its first sector at base), output [r.out, end).
    CDB_HD void exec_long(uint8_t* base, const Rec& r, uint32_t end) {
        if (r.le != r.out)
            each([&](uint32_t t) {
                lzg::copy_share(base + r.out, s.in[buf] + (r.out + r.dl), r.le - r.out, t,
                                kThreads);
            });
        if (end != r.le) copy_match(base + r.le, end - r.le, r.off);
        LZC_PHASE(7);
        LZC_EVENT(4, 1);
    }

    // The token at input position P, which the ladder has accepted: copied by
    // the whole CTA, its exact 64-bit lengths from the ladder. Returns whether
    // it is the chunk's last.
    CDB_HD bool exec_far(uint64_t P) {
        lzl::Seq sq;
        (void)ladder_at(P, d, &sq);
        if (sq.lit)
            each([&](uint32_t t) {
                lzg::copy_share(dst + d, g + sq.lit_src, sq.lit, t, kThreads);
            });
        if (sq.ml) copy_match(dst + d + sq.lit, sq.ml, sq.off);
        d += sq.lit + sq.ml;
        LZC_PHASE(7);
        LZC_EVENT(4, 1);
        return sq.done;
    }

    // Tokens [i, j) of a batch, none of them long, output [y, z) past base;
    // `mapped`: the map holds them for the window at 0.
    CDB_HD void gather(uint8_t* base, uint32_t i, uint32_t j, uint32_t y, uint32_t z,
                       bool mapped) {
        for (uint32_t W = mapped ? 0 : y & ~31u; W < z; W += kWindow) {
            if (W || !mapped) {
                each([&](uint32_t t) {
                    for (uint32_t k = t; k < kSectors; k += kThreads) s.u.e.map[k].starts = 0;
                });
                each([&](uint32_t t) {
                    if (t >= i && t < j)
                        lzg::map_token(s.u.e.map, t, s.u.e.rec[t].out,
                                       t + 1 < j ? s.u.e.rec[t + 1].out : z, W);
                    if (t == i && W <= y) s.u.e.map[0].before = i;
                });
            }
            copy_window(base, y, z, W);
            LZC_EVENT(5, 1);
        }
    }

    // The first long token of [i, m), or m.
    CDB_HD uint32_t next_long(uint32_t i, uint32_t m) const {
        for (; i < m; i = (i | 31) + 1) {
            const uint32_t v = s.votes[i / 32] >> (i % 32);
            if (v != 0) {
                i += ctz64(v);
                return i < m ? i : m;
            }
        }
        return m;
    }

    // Tokens [0, m) of a batch, output up to y1, some of them long: the runs
    // between those are gathered.
    CDB_HD void exec_longs(uint8_t* base, uint32_t m, uint32_t y1) {
        vote(s.votes, [&](uint32_t t) {
            if (t >= m) return false;
            const Rec r = s.u.e.rec[t];
            return (t + 1 < m ? s.u.e.rec[t + 1].out : y1) - r.out > kBig || r.off >> 31;
        });
        for (uint32_t i = 0; i < m;) {
            const uint32_t j = next_long(i, m);
            const uint32_t y = s.u.e.rec[i].out, z = j < m ? s.u.e.rec[j].out : y1;
            if (z > y) gather(base, i, j, y, z, i == 0);
            LZC_PHASE(6);
            if (j < m) exec_long(base, s.u.e.rec[j], j + 1 < m ? s.u.e.rec[j + 1].out : y1);
            i = j + 1;
        }
    }

    // The same out of line, so that it does not weigh on the registers and the
    // code of batches without long tokens.
    LZC_APART static void run_longs(Shm<F, kThreads>& s, uint32_t buf, uint8_t* base, uint32_t m,
                                    uint32_t y1) {
        Chunk c{s, nullptr, 0, nullptr, 0, 0};
        c.buf = buf;
        c.exec_longs(base, m, y1);
    }

    // Tokens [0, ntok) of the tile. Returns a status, and in *done whether
    // the chunk's terminal token was among them.
    CDB_HD int run_tokens(uint32_t ntok, bool* done) {
        const uint32_t lim = staged_lim();
        const uint32_t at0 = staged_at();
        const Staged in{s.in[buf], at0};
        for (uint32_t b0 = 0; b0 < ntok;) {
            const uint32_t n = ntok - b0 < kThreads ? ntok - b0 : kThreads;
            uint8_t* const base = dst + d - ((reinterpret_cast<uintptr_t>(dst) + d) & 31);
            const uint32_t y0 = static_cast<uint32_t>((reinterpret_cast<uintptr_t>(dst) + d) & 31);
            constexpr uint32_t kClamp = 0x7fffffffu;
            const uint32_t have = d < kClamp ? static_cast<uint32_t>(d) : kClamp;
            const uint32_t room = limit - d < kClamp ? static_cast<uint32_t>(limit - d) : kClamp;
            Priv<Tok> tok;
            Priv<bool> fast;
            Priv<uint32_t> olen, out;
            // parse; the map starts empty
            each_free([&](uint32_t t) {
                for (uint32_t i = t; i < kSectors; i += kThreads) s.u.e.map[i].starts = 0;
                olen[t] = 0;
                fast[t] = false;
                tok[t] = Tok{0, 0, 0, 0};
                if (t >= n) return;
                const uint32_t p = s.u.e.pos[b0 + t];
                if (F::parse_rel(in, p, lim, &tok[t]) != kSlowRel) {
                    fast[t] = true;
                    olen[t] = tok[t].lit + tok[t].ml;
                } else {
                    // clamped: such a token ends the batch
                    uint64_t ol = 0;
                    (void)F::template step<true>(reader(), S, e + p, &ol);
                    olen[t] = static_cast<uint32_t>(ol > kLenMax ? kLenMax : ol);
                }
            });
            const uint32_t total = scan(olen, out);
            LZC_PHASE(4);
            Cut& ct = s.cut[cut_turn];
            Cut& other = s.cut[cut_turn ^ 1];
            cut_turn ^= 1;
            each([&](uint32_t t) {
                if (t == 0) other = Cut{~0u, ~0u};
                if (t >= n) return;
                Tok& tk = tok[t];
                uint32_t ls = tk.ls, off = tk.off, lit = tk.lit, ml = tk.ml;
                if (!fast[t] || !F::admit(tk, out[t], have, room)) {
                    lzl::Seq sq;
                    const uint64_t P = e + s.u.e.pos[b0 + t];
                    const int st = ladder_at(P, d + out[t], &sq);
                    // the chain's next token is the ladder's (or past the tile)
                    const bool lost = b0 + t + 1 < ntok && e + s.u.e.pos[b0 + t + 1] != sq.next;
                    const bool far =
                        sq.lit > kBig || sq.ml > kBig ||
                        (sq.lit && (sq.lit_src - e > lim || sq.lit > lim - (sq.lit_src - e)));
                    if (st != CUDEC_OK || sq.done || far || lost) {
                        s.event[t] = st != CUDEC_OK          ? st
                                     : lost && !sq.done ? CUDEC_ERR_CUDA  // cannot happen
                                     : far              ? kFar
                                                        : kEnd;
                        at_min(&ct.event, t);
                    }
                    lit = far ? 0 : static_cast<uint32_t>(sq.lit);
                    ml = far ? 0 : static_cast<uint32_t>(sq.ml);
                    off = sq.off;
                    ls = static_cast<uint32_t>(sq.lit_src - e);
                }
                const uint32_t y = y0 + out[t];
                const uint32_t le = y + lit;
                s.u.e.rec[t] = Rec{y, le, at0 + ls - y, off};
                if (lit + ml > kBig || off >> 31) {  // the gather's limits
                    // (code for long ones costs Snappy batches without them 2 %)
                    if (F::kSnappy) s.event[t] = kFar;
                    at_min(F::kSnappy ? &ct.event : &ct.big, t);
                } else lzg::map_token(s.u.e.map, t, y, le + ml, 0);
                if (t == 0) s.u.e.map[0].before = 0;
            });
            const uint32_t ev = ct.event, bg = ct.big;
            LZC_PHASE(5);
            LZC_EVENT(3, 1);
            // tokens [0, k), then the event
            const uint32_t k = ev < n ? ev : n;
            const int32_t code = k < n ? s.event[k] : kFar;
            if (code != kEnd && code != kFar) return code;
            const bool last = code == kEnd;
            const uint32_t m = k + last;
            const uint32_t y1 = last ? s.u.e.rec[k].le : k < n ? s.u.e.rec[k].out : y0 + total;
            if (F::kSnappy || bg >= m) {
                if (y1 > y0) gather(base, 0, m, y0, y1, true);
            } else {
                run_longs(s, buf, base, m, y1);
            }
            LZC_PHASE(6);
            d += y1 - y0;
            if (last) {
                *done = true;
                return CUDEC_OK;
            }
            if (k < n) {
                const uint64_t P = e + s.u.e.pos[b0 + k];
                if (exec_far(P)) {
                    *done = true;
                    return CUDEC_OK;
                }
                b0 += k + 1;
            } else {
                b0 += n;
            }
        }
        return CUDEC_OK;
    }

    // ---- the chunk
    CDB_HD int run(uint64_t* written) {
        const int st = decode(written);
        // a chunk may end with the next tile's copies in flight
        each_free([&](uint32_t) { land_async(); });
        return st;
    }
    CDB_HD int decode(uint64_t* written) {
        uint64_t first = 0, lim = 0;
        const int st = F::begin(Reader{g, s.in[0], ~0ull >> 1, 0}, S, cap, &first, &lim);
        if (st != CUDEC_OK) return st;
        limit = lim;
        e = first;
        each_free([&](uint32_t t) {  // published by the first tile's barriers
            if (t == 0) s.cut[0] = s.cut[1] = Cut{~0u, ~0u};
        });
        // every tile holds at least one token and consumes at least one
        // position, so the chunk's tiles number at most S + 1
        uint64_t fuel = S == ~0ull ? ~0ull : S + 1;
        LZC_START();
        stage(e, 0);
        for (;;) {
            ibase = base_of(g, e);
            land();
            LZC_PHASE(0);
            uint64_t exit = 0;
            const uint32_t ntok = find_tokens(&exit);
            if (ntok > kMaxTok) return CUDEC_ERR_CUDA;  // unreachable (tile bounds)
            LZC_EVENT(0, 1);
            LZC_EVENT(1, ntok);
            bool done = false;
            const int rt = run_tokens(ntok, &done);
            if (rt != CUDEC_OK) return rt;
            if (done) break;
            if (exit == kStepEnd || fuel-- == 0) return CUDEC_ERR_CORRUPT_INPUT;
            e = exit;
            buf ^= 1;
        }
        *written = d;
        return CUDEC_OK;
    }
};

// ---------------------------------------------------------------------------
// A batch's large chunks. In a batch of many chunks a few large ones would run
// on alone at the narrow CTAs' pace: those are left to a CTA each of the wide
// kernel that runs beside. Large: a capacity of 2^k bytes or more, for the
// smallest k from kLargeLog on that leaves no more of them than the wide kernel
// has CTAs (a batch of many large chunks has the SMs busy to its end anyway).
// Measured:
// 8,000 uneven Snappy chunks (256 bytes to 4 MiB, median 16 KiB) 7,997 us
// without the wide kernel, 4,950 with it; 2,000 of them 4,084 and 2,610;
// 30,000 uneven LZ4 chunks 5,901 and 3,811, with kLargeLog 19 4,022, with 17
// the same.
//
// `Caps` is the batch's capacities (the CPU tests count the reads).
#if defined(__CUDACC__) || defined(CDB_EMULATE)
constexpr uint32_t kLargeLog = 18, kLogs = 16;

// Size class of a capacity: 0 below 2^kLargeLog, then one per power of two up
// to kLogs.
__device__ __forceinline__ uint32_t large_class(uint64_t cap) {
    const uint64_t c = cap >> kLargeLog;
    const uint32_t k = c ? 64 - __clzll(static_cast<long long>(c)) : 0;
    return k < kLogs ? k : kLogs;
}
// Whether a capacity is of class k (1 or more) or a higher one.
__device__ __forceinline__ bool from_class(uint64_t cap, uint32_t k) {
    return (cap >> (kLargeLog + k - 1)) != 0;
}

// The class from which on the batch's chunks are large (above kLogs: none is),
// by the whole CTA of T threads; count: the large chunks. A warp adds the
// chunks of a class in one go: a batch's capacities are often all alike.
template <uint32_t T, class Caps>
__device__ __forceinline__ uint32_t large_from(const Caps& caps, size_t n, uint32_t wide,
                                               uint32_t* count) {
    __shared__ uint32_t hist[kLogs + 1];
    const uint32_t t = threadIdx.x, lane = t & 31;
    if (t <= kLogs) hist[t] = 0;
    __syncthreads();
    constexpr uint32_t U = 8;
    for (size_t i0 = 0; i0 < n; i0 += T * U) {
        uint64_t c[U];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const size_t i = i0 + u * T + t;
            c[u] = i < n ? caps[i] : 0;
        }
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            if (!__any_sync(0xffffffffu, (c[u] >> kLargeLog) != 0)) continue;
            const uint32_t k = large_class(c[u]);
            const unsigned same = __match_any_sync(0xffffffffu, k);
            if ((same >> lane) == 1u) atomicAdd(&hist[k], __popc(same));
        }
    }
    __syncthreads();
    uint32_t k = kLogs + 1, sum = 0;
    while (k > 1 && hist[k - 1] <= wide - sum) sum += hist[--k];
    __syncthreads();  // read by every thread before the next use
    *count = sum;
    return sum ? k : kLogs + 1;
}

// Whether chunk c (of class 1 or more) is one of the large ones, by the whole
// CTA of T threads: at most `wide` chunks are of its class or a higher one.
// The chunks are read from c on, round the end, until more than `wide` of them
// are known, at first 2 per thread between barriers, then twice as many each
// time. So all the calls of a launch for one class read no more than some
// 2 (wide + 1) n capacities together, wherever its chunks lie in the batch, and
// 2 T each where all capacities are alike. Us for LZ4 pages of 4 KiB in slots of
// 1 MiB, when each narrow CTA counted the whole batch, and now; in slots of
// 4 KiB: 8,192 pages 434, 329; 319. 100,000 pages 19,558, 3,781; 3,610.
template <uint32_t T, class Caps>
__device__ __forceinline__ bool is_large(const Caps& caps, size_t n, uint32_t wide, size_t c) {
    __shared__ uint32_t found;
    const uint32_t t = threadIdx.x, lane = t & 31;
    if (t == 0) found = 0;
    __syncthreads();
    const uint32_t k = large_class(caps[c]);
    uint32_t seen = 0;
    constexpr uint32_t U = 2, kMost = 16;
    uint32_t per = U;
    for (size_t at = 0; at < n && seen <= wide; at += static_cast<size_t>(T) * per) {
        if (at != 0 && per < kMost) per *= 2;
        uint32_t mine = 0;
        for (uint32_t u0 = 0; u0 < per; u0 += U) {
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const size_t q = at + (u0 + u) * T + t;
                size_t i = c + q;
                if (i >= n) i -= n;
                mine += q < n && from_class(caps[i], k);
            }
        }
#pragma unroll
        for (uint32_t d = 16; d; d >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, d);
        if (lane == 0 && mine) atomicAdd(&found, mine);
        __syncthreads();
        seen = found;
        __syncthreads();  // read by every thread before the next addition
    }
    return seen <= wide;
}

// The index of chunk number w of class k or higher (threads' shares in turn),
// by the whole CTA of T threads; w < their count.
template <uint32_t T, class Caps>
__device__ __forceinline__ size_t large_chunk(const Caps& caps, size_t n, uint32_t k,
                                              uint32_t w) {
    __shared__ uint32_t sums[T / 32];
    __shared__ size_t found;
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t mine = 0;
#pragma unroll 4
    for (size_t i = t; i < n; i += T) mine += from_class(caps[i], k);
    uint32_t before = mine;  // then inclusive over the warp
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, before, d);
        if (lane >= d) before += v;
    }
    if (lane == 31) sums[warp] = before;
    __syncthreads();
    for (uint32_t i = 0; i < warp; ++i) before += sums[i];
    if (w < before && w >= before - mine) {
        uint32_t left = w - (before - mine);
        size_t i = t;
        while (!from_class(caps[i], k) || left-- != 0) i += T;
        found = i;
    }
    __syncthreads();
    return found;
}
#endif

// ---------------------------------------------------------------------------
// The batch kernels. Dynamic shared memory: sizeof(Shm).
#if defined(__CUDACC__)
template <class F, uint32_t kThreads>
__device__ __forceinline__ void decode_chunk(size_t c, const void* const* src_ptrs,
                                             const size_t* src_sizes, void* const* dst_ptrs,
                                             const size_t* dst_caps, cudec_chunk_result* results) {
    extern __shared__ __align__(16) uint8_t lzc_smem[];
    Shm<F, kThreads>& s = *reinterpret_cast<Shm<F, kThreads>*>(lzc_smem);
    Chunk<F, kThreads> ch{s, static_cast<const uint8_t*>(src_ptrs[c]), src_sizes[c],
                          static_cast<uint8_t*>(dst_ptrs[c]), dst_caps[c], 0};
    uint64_t written = 0;
    const int st = ch.run(&written);
    if (threadIdx.x == 0) {
        results[c].status = st;
        results[c].reserved = 0;
        results[c].bytes_written = st == CUDEC_OK ? written : 0;
    }
    __syncthreads();  // the next chunk reuses the shared state
}

// One CTA per chunk. wide: the wide kernel's CTAs (0: it does not run).
template <class F, uint32_t kThreads>
__global__ void __launch_bounds__(kThreads, Width<kThreads>::kPerSm)
    lz_cta_kernel(const void* const* src_ptrs, const size_t* src_sizes, void* const* dst_ptrs,
                  const size_t* dst_caps, size_t n, cudec_chunk_result* results, uint32_t wide) {
    for (size_t c = blockIdx.x; c < n; c += gridDim.x) {
        if (wide && large_class(dst_caps[c]) && is_large<kThreads>(dst_caps, n, wide, c))
            continue;  // a wide CTA's
        decode_chunk<F, kThreads>(c, src_ptrs, src_sizes, dst_ptrs, dst_caps, results);
    }
    // the two kernels end together: this one is launched without waiting for
    // the wide one, which has all its CTAs running or done by now
    if (wide && blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class F, uint32_t kThreads>
__global__ void __launch_bounds__(kThreads, Width<kThreads>::kPerSm)
    lz_wide_kernel(const void* const* src_ptrs, const size_t* src_sizes, void* const* dst_ptrs,
                   const size_t* dst_caps, size_t n, cudec_chunk_result* results) {
    uint32_t count;
    const uint32_t k = large_from<kThreads>(dst_caps, n, gridDim.x, &count);
    // a CTA without work leaves first, so that the narrow ones spread evenly
    if (blockIdx.x >= count) return;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    decode_chunk<F, kThreads>(large_chunk<kThreads>(dst_caps, n, k, blockIdx.x), src_ptrs,
                              src_sizes, dst_ptrs, dst_caps, results);
}
#endif

}  // namespace lzc
}  // namespace cdb
