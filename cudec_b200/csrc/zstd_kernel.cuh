// Zstd decode on sm_100a: tables and bit readers, each used by one warp of the
// CTA that decodes a frame (zstd_frame.cuh has the frame loop and the roles
// of the CTA's warps).
//
// Semantics follow the reference's v1 subset and reject ladder
// (iderex/cudec src/zstd_frame.h:196-409, src/zstd_bitstream.h:481-638,
// src/zstd_fse.h:259-676, src/zstd_huf.h:198-460, src/zstd_literals.h:211-547,
// src/zstd_seq.h:320-676, src/zstd_repcode.h:98-184) and the status mapping
// of its frame driver (tests/zstd_twin_driver.h:178-390): a literal, table,
// sequence, repeat-offset or window fault is CUDEC_ERR_CORRUPT_INPUT; the
// declared content size above the capacity, or output past it, is
// CUDEC_ERR_OUTPUT_TOO_SMALL; skippable frames, dictionary ids, frames
// without a content size and windows above 8 MB are CUDEC_ERR_UNSUPPORTED.
//
//  * table descriptions are staged in shared memory and read by 32-bit
//    windows; the tables are built lane-parallel (cells in order, each
//    symbol's next state by its rank among the cells of the same symbol);
//  * a Huffman stream decodes in several lanes at once (huf_streams);
//  * the windowed reads keep the reference's strictness (a read of more bits
//    than remain is a reject, a peek past the end reads zeros) by testing the
//    position, which goes negative on an over-read.
#pragma once

#include <cstdint>

#include "cudec.h"

namespace cdb {
namespace zstd {

constexpr uint32_t kLitSlot = 128 * 1024;   // literal slot per frame in flight (block maximum)
constexpr uint64_t kMaxWindow = 8ull << 20;
// Frame sequences (decode_frames): the largest window log libzstd's
// one-shot decoder takes (ZSTD_WINDOWLOG_MAX on 64-bit hosts). The window
// costs nothing here (matches read the destination), and offsets stay below
// 2^32 (an offset code is at most 31).
constexpr uint32_t kMaxWindowLogSeq = 31;

constexpr uint32_t kFseCells = 512;  // FSE decode cells per field (table log <= 9)
constexpr uint32_t kDescWords = 36;  // a staged description: 2 words of zeros, 128 bytes, 2 spare
constexpr uint32_t kMergeMax = 32;   // positions a Huffman lane notes for its neighbour

// Scratch of one table-building warp.
struct __align__(16) Scratch {
    uint32_t desc[kDescWords];
    int16_t counts[64];
    uint16_t next[64];
    uint8_t slot[kFseCells];  // symbol of each table slot, in spread order
};

__device__ __forceinline__ unsigned hibit32(uint32_t v) { return 31u - __clz(v); }

__device__ __forceinline__ uint64_t rd_le(const uint8_t* p, unsigned n) {
    uint64_t v = 0;
    for (unsigned i = 0; i < n; ++i) v |= static_cast<uint64_t>(p[i]) << (8 * i);
    return v;
}

// Shared memory by its 32-bit address, so that a warp's serial loops pay
// neither generic addressing nor 64-bit arithmetic.
#ifndef CDB_EMULATE
using SAddr = uint32_t;
__device__ __forceinline__ SAddr saddr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t lds(SAddr a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
// Lane 0 stores four words (predicated: no branch in a serial loop).
__device__ __forceinline__ void sts4_first(SAddr a, uint32_t x, uint32_t y, uint32_t z, uint32_t w,
                                           uint32_t lane) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %5, 0;\n\t"
        "@p st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n\t}" ::"r"(a), "r"(x), "r"(y), "r"(z),
        "r"(w), "r"(lane)
        : "memory");
}
#endif

// Backward bitstream read by absolute position: bits [0, bp) of the stream
// (little-endian bit order, bit i = byte i/8 >> i%8) remain and the next
// bits are the highest, as BitIn reads them. window() returns the 64 bits
// below bp (bit 63 = stream bit bp - 1) as hi:lo, bits outside the stream
// reading as zeros; field() takes k (<= 31) of them counted from the top.
// No state but bp: a sequence's fields come from one window and bp drops by
// their total, with no refill and no per-read checks (bp < 0 is an
// over-read, tested by the caller).
struct BitWin {
    const uint8_t* s;
    int64_t size;
    const uint32_t* abase;  // s rounded down to a 4-byte boundary
    uint32_t boff;          // bit offset of s within that word

    __device__ __forceinline__ void init(const uint8_t* src, uint64_t n) {
        s = src;
        size = static_cast<int64_t>(n);
        abase = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(src) & ~uintptr_t{3});
        boff = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(src) & 3) * 8;
    }
    __device__ __forceinline__ void window(int32_t bp, uint32_t* hi, uint32_t* lo) const {
        if (bp >= 96) {
            // three aligned words hold the 64 bits; each holds a stream byte
            // (the third is read only when the bits reach into it)
            const uint32_t t = boff + static_cast<uint32_t>(bp) - 64;
            const uint32_t* p = abase + (t >> 5);
            const uint32_t sh = t & 31;
            const uint32_t w0 = __ldg(p), w1 = __ldg(p + 1);
            const uint32_t w2 = sh ? __ldg(p + 2) : 0u;
            *lo = __funnelshift_r(w0, w1, sh);
            *hi = __funnelshift_r(w1, w2, sh);
            return;
        }
        // near (or past) the stream's start: byte by byte
        const int64_t low = static_cast<int64_t>(bp) - 64;
        uint64_t x = 0;
        for (int64_t q = low >> 3; q <= (static_cast<int64_t>(bp) - 1) >> 3; ++q) {
            if (q < 0 || q >= size) continue;
            const int64_t at = 8 * q - low;  // byte q's bit 0 within the window, in (-8, 64)
            const uint64_t b = s[q];
            x |= at >= 0 ? b << at : b >> (-at);
        }
        *lo = static_cast<uint32_t>(x);
        *hi = static_cast<uint32_t>(x >> 32);
    }
    __device__ __forceinline__ static uint32_t field(uint32_t hi, uint32_t lo, uint32_t at,
                                                     uint32_t k) {
        const uint32_t t = at < 32 ? __funnelshift_lc(lo, hi, at) : __funnelshift_lc(0u, lo, at - 32);
        return __funnelshift_rc(t, 0u, 32 - k);
    }
};

// Stage up to 128 bytes of a description at src (zeros past `size`), after
// two words of zeros. One warp.
__device__ __forceinline__ void stage_desc(Scratch& sc, const uint8_t* src, uint64_t size,
                                           uint32_t lane) {
    __syncwarp();
    uint32_t v = 0;
    for (uint32_t k = 0; k < 4; ++k)
        if (4 * lane + k < size) v |= static_cast<uint32_t>(src[4 * lane + k]) << (8 * k);
    sc.desc[2 + lane] = v;
    if (lane < 2) sc.desc[lane] = sc.desc[34 + lane] = 0;
    __syncwarp();
}

// The 32 bits from bit position bp of the staged bytes on (bp >= -64).
__device__ __forceinline__ uint32_t desc_bits(const Scratch& sc, int32_t bp) {
    const uint32_t t = static_cast<uint32_t>(bp + 64);
    return __funnelshift_r(sc.desc[t >> 5], sc.desc[(t >> 5) + 1], t & 31);
}

// FSE description (src/zstd_fse.h ZstdFseReadNCount) into sc.counts. At most
// 53 symbols of at most 10 bits and 2 bits per three skipped symbols: inside
// the staged 128 bytes. Returns false on reject.
__device__ inline bool fse_ncount(const uint8_t* src, uint64_t size, unsigned max_sym,
                                  unsigned max_log, Scratch& sc, uint32_t lane, unsigned* out_max,
                                  unsigned* out_log, uint64_t* used) {
    if (size == 0) return false;
    const unsigned nsym = max_sym + 1;
    stage_desc(sc, src, size, lane);
    for (unsigned s = lane; s < 64; s += 32) sc.counts[s] = 0;
    __syncwarp();
    const int32_t bits = size < 128 ? static_cast<int32_t>(8 * size) : 1024;
    int32_t bp = 4;
    if (bp > bits) return false;
    const unsigned log = (sc.desc[2] & 15) + 5;
    if (log > max_log) return false;
    int32_t remaining = static_cast<int32_t>(1u << log) + 1;
    int32_t threshold = static_cast<int32_t>(1u << log);
    unsigned nbits = log + 1, sym = 0;
    bool prev0 = false;
    for (unsigned it = 0; it < nsym; ++it) {
        if (prev0) {
            bool open = true;
            for (unsigned step = 0; step < nsym && open; ++step) {
                if (bp + 2 > bits) return false;
                const unsigned rep = desc_bits(sc, bp) & 3;
                bp += 2;
                sym += rep;
                if (rep != 3) open = false;
                if (sym >= nsym) return false;
            }
            if (open) return false;
            prev0 = false;
        }
        const int32_t small = (2 * threshold - 1) - remaining;
        const uint32_t pk = desc_bits(sc, bp);
        const int32_t narrow = static_cast<int32_t>(pk & static_cast<uint32_t>(threshold - 1));
        int32_t prob;
        unsigned w;
        if (narrow < small) {
            prob = narrow;
            w = nbits - 1;
        } else {
            prob = static_cast<int32_t>(pk & static_cast<uint32_t>(2 * threshold - 1));
            if (prob >= threshold) prob -= small;
            w = nbits;
        }
        bp += static_cast<int32_t>(w);
        if (bp > bits) return false;
        --prob;
        remaining -= prob < 0 ? -prob : prob;
        if (lane == 0) sc.counts[sym] = static_cast<int16_t>(prob);
        ++sym;
        prev0 = prob == 0;
        if (remaining < threshold) {
            if (remaining <= 1) break;
            nbits = hibit32(static_cast<uint32_t>(remaining)) + 1;
            threshold = static_cast<int32_t>(1u << (nbits - 1));
        }
        if (sym >= nsym) break;
    }
    __syncwarp();
    if (remaining != 1) return false;
    *out_max = sym - 1;
    *out_log = log;
    *used = static_cast<uint64_t>(bp + 7) / 8;
    return true;
}

// An FSE cell: next-state base << 22 | symbol << 16 | extra bits << 8 | state
// bits, so that the low halves of a sequence's three cells add up to its
// state bits and extra bits.
__device__ __forceinline__ uint32_t cell_of(uint32_t next, uint32_t sym, uint32_t xbits,
                                            uint32_t nbits) {
    return next << 22 | sym << 16 | xbits << 8 | nbits;
}

// Extra bits of a code: field 0 literal lengths, 1 offsets, 2 match lengths,
// 3 none (Huffman weights).
__device__ __forceinline__ uint32_t extra_bits(unsigned field, uint32_t sym);

// Table spread and cells (src/zstd_fse.h ZstdFseBuildDTable) from sc.counts,
// by one warp. The reference visits positions 0, step, 2 step, ... (mod size),
// skipping those the low-probability symbols took at the top; visit i's slot
// is therefore its rank among the kept visits.
__device__ inline bool fse_build(unsigned max_sym, unsigned log, uint32_t* cells, unsigned field,
                                 Scratch& sc, uint32_t lane) {
    const uint32_t size = 1u << log, lt = (1u << lane) - 1;
    __syncwarp();
    // two symbols per lane: slots claimed, low-probability symbols, slot starts
    uint32_t low_rank = 0, claimed = 0;
    bool ok = true;
    uint32_t nlow = 0;
    for (uint32_t i = lane; i < size; i += 32) sc.slot[i] = 0xff;
    __syncwarp();
    for (unsigned s0 = 0; s0 < 64; s0 += 32) {
        const unsigned s = s0 + lane;
        const int32_t p = s <= max_sym ? sc.counts[s] : 0;
        ok = ok && p >= -1;
        const unsigned lows = __ballot_sync(0xffffffffu, p < 0);
        const uint32_t pos_cnt = p > 0 ? static_cast<uint32_t>(p) : 0u;
        uint32_t incl = pos_cnt;
#pragma unroll
        for (uint32_t k = 1; k < 32; k <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, incl, k);
            if (lane >= k) incl += o;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        low_rank = nlow + __popc(lows & lt);
        if (p < 0 && low_rank < size) cells[size - 1 - low_rank] = s << 16;
        const uint32_t at = claimed + incl - pos_cnt;
        if (pos_cnt && at < size) sc.slot[at] = static_cast<uint8_t>(s);
        sc.next[s] = static_cast<uint16_t>(p < 0 ? 1 : p);
        nlow += __popc(lows);
        claimed += total;
    }
    if (!__all_sync(0xffffffffu, ok) || claimed + nlow != size) return false;
    __syncwarp();
    // every slot's symbol: the last start at or before it
    uint32_t carry = 0;
    for (uint32_t i0 = 0; i0 < size; i0 += 32) {
        const uint32_t m = sc.slot[i0 + lane];
        const unsigned set = __ballot_sync(0xffffffffu, m != 0xff) & (lt | (1u << lane));
        const uint32_t near = __shfl_sync(0xffffffffu, m, set ? 31 - __clz(set) : 0);
        const uint32_t v = set ? near : carry;
        sc.slot[i0 + lane] = static_cast<uint8_t>(v);
        carry = __shfl_sync(0xffffffffu, v, 31);
    }
    __syncwarp();
    const uint32_t mask = size - 1, step = (size >> 1) + (size >> 3) + 3;
    const uint32_t kept = size - nlow;  // positions below this are spread to
    uint32_t slots = 0;
    for (uint32_t i0 = 0; i0 < size; i0 += 32) {
        const uint32_t pos = ((i0 + lane) * step) & mask;
        const bool keep = pos < kept;
        const unsigned km = __ballot_sync(0xffffffffu, keep);
        if (keep) cells[pos] = static_cast<uint32_t>(sc.slot[slots + __popc(km & lt)]) << 16;
        slots += __popc(km);
    }
    __syncwarp();
    for (uint32_t i0 = 0; i0 < size; i0 += 32) {
        const uint32_t s = (cells[i0 + lane] >> 16) & 0x3f;
        const unsigned same = __match_any_sync(0xffffffffu, s);
        const uint32_t ns = sc.next[s] + __popc(same & lt);
        __syncwarp();
        if ((same >> lane) == 1u) sc.next[s] = static_cast<uint16_t>(ns + 1);  // the last of them
        const uint32_t b = log - hibit32(ns);
        cells[i0 + lane] = cell_of((ns << b) - size, s, extra_bits(field, s), b);
        __syncwarp();
    }
    return true;
}

// Shared memory of the literals warp.
struct __align__(16) HufSmem {
    uint16_t cells[1 << 11];  // symbol | bits << 8
    uint32_t wcells[64];      // the weights' FSE table
    uint8_t weights[260];
    uint16_t merge[kMergeMax][32];  // [i][lane]: bits used before a lane's i-th symbol
    Scratch sc;
};

// Huffman weights (src/zstd_huf.h ZstdHufReadWeights, literals cap 11).
__device__ inline bool huf_weights(const uint8_t* src, uint64_t size, HufSmem& h, uint32_t lane,
                                   unsigned* count, unsigned* table_log, uint64_t* used) {
    if (size == 0) return false;
    const unsigned hdr = src[0];
    unsigned written = 0;
    uint8_t* wt = h.weights;
    __syncwarp();
    if (hdr >= 128) {
        written = hdr - 127;
        const uint64_t pay = (written + 1u) / 2u;
        if (pay + 1 > size) return false;
        if (written + 1 > 256) return false;
        for (unsigned i = lane; i < written; i += 32) {
            const unsigned b = src[1 + i / 2];
            wt[i] = static_cast<uint8_t>((i % 2) == 0 ? (b >> 4) : (b & 15));
        }
        *used = pay + 1;
    } else {
        const uint64_t pay = hdr;
        if (pay + 1 > size) return false;
        unsigned fmax, flog;
        uint64_t desc;
        if (!fse_ncount(src + 1, pay, 12, 6, h.sc, lane, &fmax, &flog, &desc)) return false;
        if (!fse_build(fmax, flog, h.wcells, 3, h.sc, lane)) return false;
        // the backward stream after the description: at most 127 bytes
        const uint64_t n = pay - desc;
        if (n == 0) return false;
        const uint32_t last = src[pay];
        if (last == 0) return false;
        stage_desc(h.sc, src + 1 + desc, n, lane);
        int32_t bp = static_cast<int32_t>((n - 1) * 8 + hibit32(last));
        auto take = [&](uint32_t k) {  // the k (<= 6) highest remaining bits
            const uint32_t v = desc_bits(h.sc, bp - static_cast<int32_t>(k)) & ((1u << k) - 1);
            bp -= static_cast<int32_t>(k);
            return v;
        };
        if (static_cast<int32_t>(2 * flog) > bp) return false;
        uint32_t act = take(flog), oth = take(flog);
        const uint32_t cap = 255;
        uint32_t produced = 0;
        bool done = false;
        while (produced < cap) {
            const uint32_t cell = h.wcells[act];
            if (lane == 0) wt[produced] = static_cast<uint8_t>((cell >> 16) & 0x3f);
            ++produced;
            const uint32_t nb = cell & 0xff;
            if (static_cast<int32_t>(nb) > bp) {
                if (produced == cap) return false;
                if (lane == 0) wt[produced] = static_cast<uint8_t>((h.wcells[oth] >> 16) & 0x3f);
                ++produced;
                done = true;
                break;
            }
            const uint32_t nx = (cell >> 22) + take(nb);
            act = oth;
            oth = nx;
        }
        if (!done) return false;
        written = produced;
        *used = pay + 1;
    }
    __syncwarp();
    uint32_t total = 0, ones = 0;
    bool ok = true;
    for (unsigned i = lane; i < written; i += 32) {
        ok = ok && wt[i] <= 11;
        total += (1u << (wt[i] & 31)) >> 1;
        ones += wt[i] == 1;
    }
    if (!__all_sync(0xffffffffu, ok)) return false;
#pragma unroll
    for (uint32_t k = 16; k; k >>= 1) {
        total += __shfl_xor_sync(0xffffffffu, total, k);
        ones += __shfl_xor_sync(0xffffffffu, ones, k);
    }
    if (total == 0) return false;
    const unsigned tl = hibit32(total) + 1;
    if (tl > 11) return false;
    const uint32_t rest = (1u << tl) - total;
    const unsigned last = hibit32(rest) + 1;
    if ((1u << (last - 1)) != rest) return false;
    if (lane == 0) wt[written] = static_cast<uint8_t>(last);
    __syncwarp();
    if (ones + (last == 1) < 2) return false;
    *count = written + 1;
    *table_log = tl;
    return true;
}

// Decoding table from weights (src/zstd_huf.h ZstdHufBuildDTable): symbols in
// weight order, each weight-w symbol spans 2^(w-1) cells of tl+1-w bits. Each
// symbol's first cell is marked, then every cell takes the last mark before
// it. The weights' spans fill the table exactly (huf_weights).
__device__ inline void huf_build(HufSmem& h, unsigned count, unsigned tl, uint32_t lane) {
    const uint8_t* wt = h.weights;
    const uint32_t size = 1u << tl, lt = (1u << lane) - 1;
    uint16_t* start = h.sc.next;  // the next cell of each weight
    __syncwarp();
    uint32_t cnt = 0;  // lane k: symbols of weight k
    for (unsigned i = 0; i < count; ++i) cnt += wt[i] == lane;
    const uint32_t span_all = lane >= 1 && lane <= tl ? cnt << (lane - 1) : 0u;
    uint32_t incl = span_all;
#pragma unroll
    for (uint32_t k = 1; k < 32; k <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, incl, k);
        if (lane >= k) incl += o;
    }
    start[lane] = static_cast<uint16_t>(incl - span_all);
    for (uint32_t i = lane; i < size; i += 32) h.cells[i] = 0;
    __syncwarp();
    for (unsigned s0 = 0; s0 < count; s0 += 32) {
        const unsigned s = s0 + lane;
        const unsigned k = s < count ? wt[s] : 0;
        const unsigned same = __match_any_sync(0xffffffffu, k);
        const uint32_t span = (1u << k) >> 1;
        const uint32_t at = start[k] + span * __popc(same & lt);
        __syncwarp();
        if (k) {
            h.cells[at] = static_cast<uint16_t>(s | ((tl + 1 - k) << 8));
            if ((same >> lane) == 1u) start[k] = static_cast<uint16_t>(at + span);
        }
        __syncwarp();
    }
    uint32_t carry = 0;
    for (uint32_t i0 = 0; i0 < size; i0 += 32) {
        const uint32_t m = i0 + lane < size ? h.cells[i0 + lane] : 0u;
        const unsigned set = __ballot_sync(0xffffffffu, m != 0) & (lt | (1u << lane));
        const uint32_t near = __shfl_sync(0xffffffffu, m, set ? 31 - __clz(set) : 0);
        const uint32_t v = set ? near : carry;
        if (i0 + lane < size) h.cells[i0 + lane] = static_cast<uint16_t>(v);
        carry = __shfl_sync(0xffffffffu, v, 31);
    }
    __syncwarp();
}

// Decode symbols from bit position *bp down while it is above `end` and fewer
// than `most` have been decoded; returns their number. put(i, symbol) takes
// each, note(i, bp) each position before its symbol. Five symbols per window
// (5 x 11 <= 55 bits, 11 the largest table log). kWhole: without a test per
// symbol while all five are wanted whatever their lengths. One warp of a frame's
// CTA decodes its literals, so frames of little else wait for these loops. Us
// with the tests everywhere; without them in the eight lanes' first pass and
// for a lane alone; in their writing pass too: 4,096 frames of 16 KiB that are
// nearly all literals 1,282, 1,223, 1,246; 96 of 260,000 bytes at level 19
// 1,774, 1,590, 1,591; 8,000 of 8,000 bytes 1,450, 1,349, 1,339; 512 of 1 MiB
// 7,683, 7,565, 7,719; 2,048 of them 26,916, 26,769, 27,248.
template <bool kWhole, class Put, class Note>
__device__ __forceinline__ uint32_t huf_run(const BitWin& bw, const uint16_t* cells, unsigned tl,
                                            int32_t* bp, int32_t end, uint32_t most, Put put,
                                            Note note) {
    uint32_t n = 0;
    int32_t p = *bp;
    // windows whose five symbols are all wanted, whatever their lengths
    while (kWhole && p - end > 5 * 11 && most - n >= 5) {
        uint32_t hi, lo;
        bw.window(p, &hi, &lo);
        uint32_t at = 0;
#pragma unroll
        for (uint32_t j = 0; j < 5; ++j) {
            const uint32_t cell = cells[BitWin::field(hi, lo, at, tl)];
            note(n + j, p - static_cast<int32_t>(at));
            put(n + j, cell & 0xff);
            at += cell >> 8;
        }
        p -= static_cast<int32_t>(at);
        n += 5;
    }
    while (p > end && n < most) {
        uint32_t hi, lo;
        bw.window(p, &hi, &lo);
        uint32_t at = 0;
        const int32_t p0 = p;
#pragma unroll
        for (uint32_t j = 0; j < 5; ++j) {
            if (p > end && n < most) {
                const uint32_t cell = cells[BitWin::field(hi, lo, at, tl)];
                note(n, p);
                put(n, cell & 0xff);
                at += cell >> 8;
                p = p0 - static_cast<int32_t>(at);
                ++n;
            }
        }
    }
    *bp = p;
    return n;
}

constexpr int32_t kHufSplit = 3200;  // bits of a stream from which eight lanes share it

// `count` literals from one Huffman stream (streams == 1) or four (their
// sizes in the payload's first six bytes), by one warp. A stream is accepted
// only when exactly all its bits give exactly its symbols, which is what
// per-symbol checks plus a final "all bits used" check amount to.
//
// Eight lanes share a stream of kHufSplit bits or more. Each first decodes
// its eighth of the bits from wherever it falls: Huffman codes fall into step
// after a few symbols, so the position where it leaves is (checked below) the
// true start of the next lane's part. Each lane then decodes from its true
// start until it meets a position it noted the first time, which gives its
// true symbol count and so every lane's place in the output, and decodes its
// part again, writing. Where a lane does not fall into step within kMergeMax
// symbols, one lane decodes the stream alone (as it does a short stream).
// Four lanes alone took 0.76 M cycles for 21,000 literals.
__device__ inline bool huf_streams(const uint8_t* pay, uint64_t psize, unsigned streams,
                                   uint64_t count, HufSmem& h, unsigned tl, uint8_t* dst,
                                   uint32_t lane) {
    const uint32_t per = streams == 1 ? 32u : 8u;  // lanes of a stream
    const uint32_t q = lane / per, j = lane % per;
    const uint8_t* src = pay;
    uint64_t size = psize, want = count;
    uint8_t* out = dst;
    if (streams != 1) {
        if (psize < 10 || count < 6) return false;
        const uint64_t c0 = rd_le(pay, 2), c1 = rd_le(pay + 2, 2), c2 = rd_le(pay + 4, 2);
        const uint64_t sb = psize - 6;
        if (c0 + c1 + c2 >= sb) return false;
        const uint64_t seg = (count + 3) / 4;
        size = q == 0 ? c0 : q == 1 ? c1 : q == 2 ? c2 : sb - c0 - c1 - c2;
        src = pay + 6 + (q == 0 ? 0 : q == 1 ? c0 : q == 2 ? c0 + c1 : c0 + c1 + c2);
        want = q < 3 ? seg : count - 3 * seg;
        out = dst + q * seg;
    }
    const uint32_t last = size ? src[size - 1] : 0u;
    if (!__all_sync(0xffffffffu, last != 0)) return false;  // empty, or no padding marker
    const int32_t T = static_cast<int32_t>((size - 1) * 8 + hibit32(last));  // size <= 128 KiB
    BitWin bw;
    bw.init(src, size);
    const uint32_t n_want = static_cast<uint32_t>(want);
    auto no_note = [](uint32_t, int32_t) {};
    auto no_put = [](uint32_t, uint32_t) {};
    bool split = __all_sync(0xffffffffu, T >= kHufSplit);
    if (split) {
        const int32_t part = T / static_cast<int32_t>(per);
        const int32_t from = T - static_cast<int32_t>(j) * part;
        const int32_t end = j + 1 == per ? 0 : from - part;
        int32_t x = from;
        const uint32_t n1 = huf_run<true>(bw, h.cells, tl, &x, end, ~0u, no_put,
                                          [&](uint32_t i, int32_t p) {
                                              if (i < kMergeMax)
                                                  h.merge[i][lane] =
                                                      static_cast<uint16_t>(from - p);
                                          });
        // the true start, and the symbols up to the first noted position
        int32_t start = __shfl_up_sync(0xffffffffu, x, 1);
        if (j == 0) start = T;
        int32_t p = start;
        uint32_t nt = 0, g = 0;
        int32_t gp = from;
        bool merged = true;
        while (p != gp) {
            if (gp > p) {
                if (++g >= kMergeMax || g >= n1) {
                    merged = false;
                    break;
                }
                gp = from - h.merge[g][lane];
            } else {
                nt += huf_run<false>(bw, h.cells, tl, &p, p - 1, 1, no_put, no_note);
            }
        }
        split = __all_sync(0xffffffffu, merged);
        if (split) {
            const uint32_t n = nt + (n1 - g);
            uint32_t incl = n;
            for (uint32_t k = 1; k < per; k <<= 1) {
                const uint32_t o = __shfl_up_sync(0xffffffffu, incl, k);
                if (j >= k) incl += o;
            }
            // the last lane's end and count are the stream's
            const bool ok = j + 1 != per || (x == 0 && incl == n_want);
            if (!__all_sync(0xffffffffu, ok)) return false;
            uint8_t* o = out + (incl - n);
            (void)huf_run<false>(
                bw, h.cells, tl, &start, -(1 << 30), n,
                [&](uint32_t i, uint32_t sym) { o[i] = static_cast<uint8_t>(sym); }, no_note);
            __syncwarp();
            return true;
        }
    }
    bool ok = true;
    if (j == 0) {
        int32_t p = T;
        (void)huf_run<true>(
            bw, h.cells, tl, &p, -(1 << 30), n_want,
            [&](uint32_t i, uint32_t sym) { out[i] = static_cast<uint8_t>(sym); }, no_note);
        ok = p == 0;
    }
    ok = __all_sync(0xffffffffu, ok);
    __syncwarp();
    return ok;
}

// Baseline | extra-bit count << 24 per code, one constant read per field.
static __constant__ uint32_t kLLCode[36] = {
    0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15,
    16 | 1u << 24, 18 | 1u << 24, 20 | 1u << 24, 22 | 1u << 24, 24 | 2u << 24, 28 | 2u << 24,
    32 | 3u << 24, 40 | 3u << 24, 48 | 4u << 24, 64 | 6u << 24, 128 | 7u << 24,
    256 | 8u << 24, 512 | 9u << 24, 1024 | 10u << 24, 2048 | 11u << 24, 4096 | 12u << 24,
    8192 | 13u << 24, 16384 | 14u << 24, 32768 | 15u << 24, 65536 | 16u << 24};
static __constant__ uint32_t kMLCode[53] = {
    3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18,
    19, 20, 21, 22, 23, 24, 25, 26, 27, 28, 29, 30, 31, 32, 33, 34,
    35 | 1u << 24, 37 | 1u << 24, 39 | 1u << 24, 41 | 1u << 24, 43 | 2u << 24, 47 | 2u << 24,
    51 | 3u << 24, 59 | 3u << 24, 67 | 4u << 24, 83 | 4u << 24, 99 | 5u << 24,
    131 | 7u << 24, 259 | 8u << 24, 515 | 9u << 24, 1027 | 10u << 24, 2051 | 11u << 24,
    4099 | 12u << 24, 8195 | 13u << 24, 16387 | 14u << 24, 32771 | 15u << 24,
    65539 | 16u << 24};
static __constant__ int16_t kPreLL[36] = {4, 3, 2, 2, 2, 2, 2, 2, 2, 2, 2, 2, 2, 1, 1, 1, 2, 2,
                                   2, 2, 2, 2, 2, 2, 2, 3, 2, 1, 1, 1, 1, 1, -1, -1, -1, -1};
static __constant__ int16_t kPreOF[29] = {1, 1, 1, 1, 1, 1, 2, 2, 2, 1, 1, 1, 1, 1, 1,
                                   1, 1, 1, 1, 1, 1, 1, 1, 1, -1, -1, -1, -1, -1};
static __constant__ int16_t kPreML[53] = {1, 4, 3, 2, 2, 2, 2, 2, 2, 1, 1, 1, 1, 1, 1, 1, 1, 1,
                                   1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1,
                                   1, 1, 1, 1, 1, 1, 1, 1, 1, 1, -1, -1, -1, -1, -1, -1, -1};

__device__ __forceinline__ uint32_t extra_bits(unsigned field, uint32_t sym) {
    return field == 0 ? kLLCode[sym] >> 24 : field == 1 ? sym : field == 2 ? kMLCode[sym] >> 24 : 0u;
}

// The sequence tables' state across a frame's blocks (the tables themselves
// stay in shared memory for the repeat mode).
struct Tables {
    unsigned log[3];
    bool present[3];
};

// Sequence table load (src/zstd_seq.h ZstdSeqLoadTable), by one warp.
__device__ inline bool seq_table(uint32_t (*fse)[kFseCells], Scratch& sc, Tables& t,
                                 unsigned field, unsigned mode, const uint8_t* src, uint64_t size,
                                 uint64_t* used, uint32_t lane) {
    const unsigned symmax = field == 0 ? 35 : field == 1 ? 31 : 52;
    const unsigned logmax = field == 1 ? 8 : 9;
    *used = 0;
    if (mode == 3) return t.present[field];
    if (mode == 1) {
        if (size == 0) return false;
        const unsigned s = src[0];
        if (s > symmax) return false;
        __syncwarp();
        if (lane == 0) fse[field][0] = cell_of(0, s, extra_bits(field, s), 0);
        __syncwarp();
        t.log[field] = 0;
        t.present[field] = true;
        *used = 1;
        return true;
    }
    unsigned dmax, log;
    if (mode == 0) {
        const int16_t* pre = field == 0 ? kPreLL : field == 1 ? kPreOF : kPreML;
        dmax = field == 0 ? 35 : field == 1 ? 28 : 52;
        log = field == 1 ? 5 : 6;
        __syncwarp();
        for (unsigned s = lane; s <= dmax; s += 32) sc.counts[s] = pre[s];
        __syncwarp();
    } else {
        if (!fse_ncount(src, size, symmax, logmax, sc, lane, &dmax, &log, used)) return false;
    }
    if (!fse_build(dmax, log, fse[field], field, sc, lane)) {
        *used = 0;
        return false;
    }
    t.log[field] = log;
    t.present[field] = true;
    return true;
}

}  // namespace zstd
}  // namespace cdb
