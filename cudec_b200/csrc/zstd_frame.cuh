// One Zstd frame decoded by one CTA of six warps (RFC 8878 subset of the
// reference, statuses as iderex/cudec tests/zstd_twin_driver.h:178-390 maps
// them). Shared by the Zstd batch entry and the mixed-format kernel.
//
// A frame's serial part is the sequences' state chain: a sequence's three
// states come out of the bits that the sequence before it left. Everything
// else follows from the block headers, so the warps take parts of the frame:
//
//   * warp 0 walks the blocks, builds the sequence tables and runs the state
//     chain, noting per sequence its three cells and its bit position, kItem
//     sequences at a time;
//   * warp 1 decodes the blocks' Huffman literals into the frame's slot of
//     the workspace, a block ahead where two blocks' literals fit the slot,
//     and hashes the finished blocks of a frame with a checksum;
//   * warps 2 to 5 execute: one sequence per thread for its values (their
//     bits read at the noted position), the repeat offsets (a scan of
//     functions of the three offsets), positions and the reference's checks,
//     then the output by gathering (lz_gather.cuh).
//
// With one warp doing all of this in turn a sequence cost about 490 cycles in
// the state chain (every lane repeating the whole decode) and 356 in
// execution; the chain alone is some 170 cycles with four frames on an SM, and
// the rest hides behind it. What bounds a launch now is latency: a frame takes
// about as long alone as among four on its SM, execution waiting for the match
// bytes of each part and for its barriers, then the state chain. With 256
// frames of 1 MiB a quarter of the issue slots are used, and per issued
// instruction 3.4 warps wait at a barrier and 1.4 for global memory. Measured,
// L2 flushed: 512 frames of 1 MiB at level 3 25,825 us before, 7,565 now; six
// of 128 KiB 4,250 and 850; the mixed plan's batch of uneven chunks of all
// formats 31,882 and 8,240. Slower than before: many small frames of few long
// sequences (4,096 frames of 16 KiB: matches of 200 to 900 bytes 213 and 279,
// literal runs and copies of 300 to 3,000 200 and 265, nearly all literals
// 1,118 and 1,223): four frames on an SM, not sixteen and more, to hide each
// other's waits.
//
// The warps meet at named barriers, every arrival matched by a wait:
//   kBarItem   warps 0, 2-5: item i is in its buffer (two buffers in turn,
//              so warp 0 is at most one item ahead);
//   kBarReady  (2, by the block's parity) warp 1 arrives, warps 2-5 wait:
//              the block's literals are in the slot, or the block is faulty;
//   kBarFree   (2) warps 2-5 arrive, warp 1 waits: the block is executed;
//   kBarExec   warps 2-5.
// Warp 1 arrives at a block's kBarReady only after its wait at the kBarFree of
// the block two before, which the block's own kBarFree shares: so warps 2-5
// wait at the kBarReady of every block that they begin, a faulty one
// included, before they arrive at its kBarFree. Without that a warp 1 that is
// late would be overtaken at that barrier and the CTA would not end.
// A fault found by warp 0 travels as an item, one found by warp 1 as the
// block's literal fault, so that warps 2-5 meet everything in the serial
// decoder's order and alone decide the frame's status. The one that ends the
// frame is block `stop`: warp 0 leaves after the item barrier, warp 1 after
// that block's kBarFree; a literals arrival that nothing waited for is waited
// for at the end.
#pragma once

#include <cstdint>

#include "cudec.h"
#include "lz_gather.cuh"
#include "zstd_kernel.cuh"

namespace cdb {
namespace zstd {

constexpr uint32_t kExecWarps = 4;
constexpr uint32_t kExec = 32 * kExecWarps;  // executing threads
constexpr uint32_t kTeam = 64 + kExec;       // threads of a frame's CTA
constexpr uint32_t kItem = kExec;     // sequences per item: one per executing thread
constexpr uint32_t kBigCopy = 1024;   // longer sequences are copied by all of them together
// output sectors in flight per warp (512 frames of 1 MiB: 2, 7.68 ms; 3, 7.70;
// 4, 7.84; 8,000 frames of 8,000 bytes: 1.45, 1.56, 1.63)
constexpr uint32_t kUnroll = 2;
constexpr uint32_t kPart = kExec * kUnroll;  // output bytes between barriers

constexpr int kBarItem = 1, kBarReady = 2, kBarFree = 4, kBarExec = 6;
constexpr int kItemCount = 32 + kExec, kLitCount = 32 + kExec;

#ifndef CDB_EMULATE
__device__ __forceinline__ void bar_sync(int id, int n) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int n) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}
#endif

// Profiling builds (-DCDB_PHASE_TIMING) accumulate SM cycles over all frames
// of a launch: 0 sequence tables, 1 state chain, 2 warp 0 waiting for an item
// buffer, 3 literals, 4 hash, 5 warps 2-5 waiting for an item, 6 waiting
// for literals, 7 executing. Events: 0 blocks, 1 sequences, 2 literals,
// 3 items.
#ifdef CDB_PHASE_TIMING
__device__ unsigned long long zs_cycles[8];
__device__ unsigned long long zs_events[8];
#define ZS_T(v) const long long v = clock64()
#define ZS_ADD(i, t0)            \
    if ((threadIdx.x & 31) == 0) \
    atomicAdd(&zs_cycles[i], static_cast<unsigned long long>(clock64() - (t0)))
#define ZS_EV(i, n)              \
    if ((threadIdx.x & 31) == 0) \
    atomicAdd(&zs_events[i], static_cast<unsigned long long>(n))
#else
#define ZS_T(v)
#define ZS_ADD(i, t0)
#define ZS_EV(i, n)
#endif

// What warp 0 hands to the executing warps.
enum : uint32_t { kSequences = 0, kRaw = 1, kRle = 2, kFault = 3 };
enum : uint32_t { kFirst = 1, kLast = 2, kEnd = 4 };  // of its block; of the frame
struct Item {
    uint32_t kind, flags;
    uint32_t n;          // sequences
    uint32_t size;       // raw, RLE: bytes out; sequences: bytes of the bitstream
    const uint8_t* src;  // raw, RLE: the block's body; sequences: the bitstream
    const uint8_t* lit;  // raw, RLE literals (null: warp 1's)
    uint32_t regen;      // literals of the block
    uint32_t rle;        // literals are one byte repeated
    int32_t shift;       // sequences: the Raw positions' excess over the bitstream's
};

// A sequence as the state chain leaves it: the three cells and the bit
// position below which its extra bits lie (Item::shift past the bitstream's).
struct __align__(16) Raw {
    uint32_t ll, of, ml;
    int32_t bp;
};

// The effect of some sequences on the three repeat offsets: each is either a
// value or an offset before them less `v` (not below zero).
struct Reps {
    uint32_t v[3];
    uint32_t from;  // 2 bits each: 0-2 which one, 3 a value
};

constexpr uint32_t kBitWords = 512;  // staged bitstream: more than an item's (128 x 89 bits)
constexpr uint32_t kItemBits = kItem * 89 + 96;  // most bits an item's chain looks at

struct __align__(16) TeamSmem {
    uint32_t fse[3][kFseCells];
    uint32_t bits[kBitWords + 4];  // warp 0's stretch of the bitstream
    HufSmem huf;
    Scratch sc;  // warp 0's
    Item item[2];
    Raw raw[2][kItem];
    lzg::Rec rec[kItem];
    lzg::Sector map[lzg::kSectors];
    uint32_t lcode[36], mcode[53];  // kLLCode, kMLCode
    uint8_t period[16 * kExec];
    Reps reps[kExecWarps];    // an item's effect, per executing warp
    uint32_t lsum[kExecWarps], tsum[kExecWarps];  // literal and output bytes of its sequences
    uint32_t big[kExecWarps];  // sequences copied by all of them
    int32_t fail[kExecWarps];  // first failing sequence's verdict
    uint32_t lit_at[2];       // a block's literals in the slot
    uint64_t out_at[2];       // output after a block
    uint32_t lit_fault;       // first block with a literal fault
    uint32_t ready;           // literal arrivals made
    uint32_t stop, leave;     // the block that ended the frame early; the item
                              // whose barrier is warp 0's last then
    uint32_t waited;          // literal arrivals waited for
    int32_t status;
    uint32_t hash_bad;
    uint64_t out, end;        // output bytes; position after the last block
};

// ---------------------------------------------------------------------------
// Headers.
struct Frame {
    const uint8_t* f;
    uint64_t N;
    uint8_t* dst;
    uint64_t cap;
    uint64_t head, fcs, window, bmax;
    bool has_fcs, csum;
};

// The frame header (src/zstd_frame.h:196-290).
template <bool Wide>
__device__ inline int frame_head(Frame& F) {
    const uint8_t* f = F.f;
    const uint64_t N = F.N;
    if (N < 4) return CUDEC_ERR_CORRUPT_INPUT;
    const uint32_t magic = static_cast<uint32_t>(rd_le(f, 4));
    if (magic != 0xFD2FB528u) {
        if (magic >= 0x184D2A50u && magic <= 0x184D2A5Fu) return CUDEC_ERR_UNSUPPORTED;
        return CUDEC_ERR_CORRUPT_INPUT;
    }
    if (N < 5) return CUDEC_ERR_CORRUPT_INPUT;
    const unsigned d = f[4], fcs_flag = d >> 6, single = (d >> 5) & 1;
    F.csum = (d >> 2) & 1;
    if (d & 8) return CUDEC_ERR_CORRUPT_INPUT;
    if (d & 3) return CUDEC_ERR_UNSUPPORTED;
    const unsigned fcs_size = fcs_flag == 0 ? (single ? 1 : 0)
                            : fcs_flag == 1 ? 2 : fcs_flag == 2 ? 4 : 8;
    F.has_fcs = fcs_size != 0;  // single segment implies a content size
    if (!F.has_fcs && !Wide) return CUDEC_ERR_UNSUPPORTED;
    const unsigned wbytes = single ? 0 : 1;
    F.head = 5 + wbytes + fcs_size;
    if (N < F.head) return CUDEC_ERR_CORRUPT_INPUT;
    F.fcs = F.has_fcs ? rd_le(f + 5 + wbytes, fcs_size) : 0;
    if (fcs_size == 2) F.fcs += 256;
    if (single) {
        F.window = F.fcs;
    } else {
        const uint64_t e = f[5] >> 3, m = f[5] & 7, base = 1ull << (10 + e);
        F.window = base + (base / 8) * m;
        if (!Wide && F.window > kMaxWindow) return CUDEC_ERR_UNSUPPORTED;
        if (Wide && 10 + e > kMaxWindowLogSeq) return CUDEC_ERR_UNSUPPORTED;
    }
    if (F.has_fcs && F.fcs > F.cap) return CUDEC_ERR_OUTPUT_TOO_SMALL;
    F.bmax = F.window < kLitSlot ? F.window : kLitSlot;
    return CUDEC_OK;
}

struct Block {
    const uint8_t* b;
    uint32_t type, size, body;
    bool last;
};

__device__ __forceinline__ bool block_head(const Frame& F, uint64_t pos, Block* k) {
    if (F.N - pos < 3) return false;
    const uint32_t raw = static_cast<uint32_t>(rd_le(F.f + pos, 3));
    k->last = raw & 1;
    k->type = (raw >> 1) & 3;
    k->size = raw >> 3;
    if (k->type == 3 || k->size > F.bmax) return false;
    k->body = k->type == 1 ? 1 : k->size;
    if (F.N - pos < 3ull + k->body) return false;
    k->b = F.f + pos + 3;
    return true;
}

// The literals section's header (src/zstd_literals.h:357-547).
struct Lits {
    unsigned type, streams;
    uint32_t head, regen, csize;
    uint32_t used;  // bytes of the section
};

__device__ __forceinline__ bool lit_head(const Frame& F, const Block& k, Lits* l) {
    const uint8_t* b = k.b;
    if (k.body == 0) return false;
    const unsigned fmt = (b[0] >> 2) & 3;
    l->type = b[0] & 3;
    l->csize = 0;
    l->streams = 0;
    if (l->type < 2) {
        const unsigned hs = fmt == 1 ? 2 : fmt == 3 ? 3 : 1;
        if (k.body < hs) return false;
        l->regen = static_cast<uint32_t>(rd_le(b, hs)) >> (hs == 1 ? 3 : 4);
        l->head = hs;
    } else {
        const unsigned hs = fmt == 2 ? 4 : fmt == 3 ? 5 : 3;
        const unsigned fb = fmt == 2 ? 14 : fmt == 3 ? 18 : 10;
        if (k.body < hs) return false;
        const uint64_t rw = rd_le(b, hs), msk = (1ull << fb) - 1;
        l->regen = static_cast<uint32_t>((rw >> 4) & msk);
        l->csize = static_cast<uint32_t>((rw >> (4 + fb)) & msk);
        l->head = hs;
        l->streams = fmt == 0 ? 1 : 4;
    }
    if (l->regen > F.bmax) return false;
    const uint32_t after = k.body - l->head;
    const uint32_t need = l->type == 0 ? l->regen : l->type == 1 ? 1u : l->csize;
    if (need > after) return false;
    l->used = l->head + need;
    return true;
}

// ---------------------------------------------------------------------------
// Warp 0: blocks, sequence tables, the state chain.
struct SeqRole {
    const Frame& F;
    TeamSmem& s;
    uint32_t lane;
    uint32_t item = 0;

    __device__ __forceinline__ Item& slot() { return s.item[item & 1]; }
    // Item `item` is in its buffer; false once the frame is decided.
    __device__ __forceinline__ bool emit() {
        ZS_T(t0);
        __syncwarp();
        bar_sync(kBarItem, kItemCount);
        const bool go = s.leave != item;
        ++item;
        ZS_ADD(2, t0);
        ZS_EV(3, 1);
        return go;
    }
    __device__ __forceinline__ void fault(uint32_t flags) {
        if (lane == 0) slot() = Item{kFault, flags, 0, 0, nullptr, nullptr, 0, 0, 0};
        (void)emit();
    }

    // The sequences of a block with tables t; false when the role ends here.
    __device__ __forceinline__ bool sequences(const Tables& t, const uint8_t* sec, uint32_t size,
                                              uint32_t nseq, const Lits& l, const uint8_t* lit,
                                              uint32_t end_flags) {
        const uint32_t lastb = sec[size - 1];
        if (lastb == 0) {
            fault(kFirst);
            return false;
        }
        int32_t bp = static_cast<int32_t>((size - 1) * 8 + hibit32(lastb));  // at most 8 x 128 KiB
        BitWin bw;
        bw.init(sec, size);
        const unsigned l0 = t.log[0], l1 = t.log[1], l2 = t.log[2];
        if (static_cast<int32_t>(l0 + l1 + l2) > bp) {
            fault(kFirst);
            return false;
        }
        uint32_t hi, lo;
        bw.window(bp, &hi, &lo);
        uint32_t sl = __funnelshift_rc(hi, 0u, 32 - l0);
        uint32_t so = BitWin::field(hi, lo, l0, l1);
        uint32_t sm = BitWin::field(hi, lo, l0 + l1, l2);
        bp -= static_cast<int32_t>(l0 + l1 + l2);
        uint32_t flags = kFirst;
        // states as addresses of their cells; positions as bits of s.bits
        const SAddr tl = saddr(s.fse[0]), to = saddr(s.fse[1]), tm = saddr(s.fse[2]);
        const SAddr bits = saddr(s.bits);
        SAddr al = tl + 4 * sl, ao = to + 4 * so, am = tm + 4 * sm;
        int32_t low = bp;   // stream bits from here on up are staged
        int32_t shift = 0;  // staged bit of stream bit 0
        for (uint32_t i0 = 0; i0 < nseq; i0 += kItem) {
            ZS_T(t0);
            const uint32_t cnt = nseq - i0 < kItem ? nseq - i0 : kItem;
            const bool tail = i0 + cnt == nseq;
            if (bp - low < static_cast<int32_t>(kItemBits)) {
                // stage the words that end with bit bp - 1's; before the
                // stream's first word, zeros
                const int32_t top = (static_cast<int32_t>(bw.boff) + bp + 31) >> 5;  // past it
                const int32_t w0 = top - static_cast<int32_t>(kBitWords);
                __syncwarp();
                for (uint32_t k = lane; k < kBitWords; k += 32) {
                    const int32_t w = w0 + static_cast<int32_t>(k);
                    s.bits[k] = w >= 0 ? __ldg(bw.abase + w) : 0u;
                }
                __syncwarp();
                shift = static_cast<int32_t>(bw.boff) - 32 * w0;
                low = -shift;
            }
            const SAddr raw = saddr(s.raw[item & 1]);
            // States stay below their table's size and codes within their
            // field's range by construction (seq_table checks the symbols,
            // a cell's next base + its bits is below the table size). A
            // position that goes negative is an over-read, tested once per
            // item (an item looks at kItemBits at most, and at least those
            // are staged, zeros before the stream's start): a stream fault
            // is a reject whatever the execution verdicts were.
            int32_t t = bp + shift;
            const uint32_t chain = tail ? cnt - 1 : cnt;  // the last one reads no state bits
            uint32_t k = 0;
            for (; k < chain; ++k) {
                const uint32_t cl = lds(al), co = lds(ao), cm = lds(am);
                const uint32_t sum = cl + co + cm;
                const uint32_t xb = (sum >> 8) & 0xff, sb = sum & 0xff;  // at most 63 and 26
                sts4_first(raw + 16 * k, cl, co, cm, static_cast<uint32_t>(t), lane);
                // the 32 bits below the extra bits hold the state bits
                const uint32_t u = static_cast<uint32_t>(t) - xb;
                const SAddr ua = bits + (((u - 32) >> 5) << 2);
                const uint32_t w0 = lds(ua), w1 = lds(ua + 4);
                t -= static_cast<int32_t>(xb + sb);
                hi = __funnelshift_r(w0, w1, u);
                const uint32_t lb = cl & 0xff, mb = cm & 0xff, ob = co & 0xff;
                const uint32_t h1 = hi << lb;  // at most 9 bits each
                al = tl + 4 * ((cl >> 22) + __funnelshift_rc(hi, 0u, 32 - lb));
                am = tm + 4 * ((cm >> 22) + __funnelshift_rc(h1, 0u, 32 - mb));
                ao = to + 4 * ((co >> 22) + __funnelshift_rc(h1 << mb, 0u, 32 - ob));
            }
            if (tail) {
                const uint32_t cl = lds(al), co = lds(ao), cm = lds(am);
                sts4_first(raw + 16 * k, cl, co, cm, static_cast<uint32_t>(t), lane);
                t -= static_cast<int32_t>(((cl + co + cm) >> 8) & 0xff);
            }
            bp = t - shift;
            ZS_ADD(1, t0);
            if (bp < 0 || (tail && bp != 0)) {
                fault(flags);
                return false;
            }
            if (lane == 0)
                slot() = Item{kSequences, flags | (tail ? kLast | end_flags : 0u), cnt, size, sec,
                              lit, l.regen, l.type == 1, shift};
            if (!emit()) return false;
            flags = 0;
        }
        return true;
    }

    __device__ void run() {
        Tables t;
        for (int k = 0; k < 3; ++k) {
            t.log[k] = 0;
            t.present[k] = false;
        }
        uint64_t pos = F.head;
        for (;;) {
            Block k;
            if (!block_head(F, pos, &k)) return fault(kFirst);
            ZS_EV(0, 1);
            const uint32_t end_flags = k.last ? kEnd : 0u;
            if (k.last && lane == 0) s.end = pos + 3 + k.body;
            if (k.type != 2) {
                if (lane == 0)
                    slot() = Item{k.type == 0 ? kRaw : kRle, kFirst | kLast | end_flags, 0, k.size,
                                  k.b, nullptr, 0, 0, 0};
                if (!emit()) return;
            } else {
                Lits l;
                if (!lit_head(F, k, &l)) return fault(kFirst);
                // ---- sequences section (src/zstd_seq.h:320-676)
                const uint8_t* lit = l.type < 2 ? k.b + l.head : nullptr;
                const uint8_t* sec = k.b + l.used;
                uint32_t rem = k.body - l.used;
                if (rem == 0) return fault(kFirst);
                uint32_t nseq, cnum = 1;
                if (sec[0] < 128) {
                    nseq = sec[0];
                } else if (sec[0] < 255) {
                    if (rem < 2) return fault(kFirst);
                    nseq = ((static_cast<uint32_t>(sec[0]) - 128) << 8) + sec[1];
                    cnum = 2;
                } else {
                    if (rem < 3) return fault(kFirst);
                    nseq = static_cast<uint32_t>(sec[1]) + (static_cast<uint32_t>(sec[2]) << 8) +
                           0x7F00u;
                    cnum = 3;
                }
                if (nseq == 0) {
                    if (lane == 0)
                        slot() = Item{kSequences, kFirst | kLast | end_flags, 0, 0, nullptr, lit,
                                      l.regen, l.type == 1, 0};
                    if (!emit()) return;
                } else {
                    if (nseq > F.bmax / 3 || rem <= cnum) return fault(kFirst);
                    const unsigned modes = sec[cnum++];
                    if (modes & 3) return fault(kFirst);
                    sec += cnum;
                    rem -= cnum;
                    ZS_T(t0);
                    for (unsigned fld = 0; fld < 3; ++fld) {
                        uint64_t u;
                        if (!seq_table(s.fse, s.sc, t, fld, (modes >> (6 - 2 * fld)) & 3, sec, rem,
                                       &u, lane))
                            return fault(kFirst);
                        sec += u;
                        rem -= static_cast<uint32_t>(u);
                    }
                    ZS_ADD(0, t0);
                    ZS_EV(1, nseq);
                    if (rem == 0) return fault(kFirst);
                    if (!sequences(t, sec, rem, nseq, l, lit, end_flags)) return;
                }
            }
            if (k.last) return;
            pos += 3 + k.body;
        }
    }
};

// ---------------------------------------------------------------------------
// Warp 1: literals, and the content checksum.

// XXH64 (public xxHash specification, seed 0) of output that grows: the four
// accumulators live in lanes mod 4, 256 bytes per step.
struct Hash {
    uint64_t acc = 0, done = 0;
    static constexpr uint64_t P1 = 11400714785074694791ull, P2 = 14029467366897019727ull,
                              P3 = 1609587929392839161ull, P4 = 9650029242287828579ull,
                              P5 = 2870177450012600261ull;
    __device__ __forceinline__ static uint64_t rotl(uint64_t x, int r) {
        return (x << r) | (x >> (64 - r));
    }
    // 8 bytes at p from the aligned words holding them
    __device__ __forceinline__ static uint64_t rd8(const uint8_t* p) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(p);
        const uint32_t* q = reinterpret_cast<const uint32_t*>(a & ~uintptr_t{3});
        const uint32_t sh = 8 * static_cast<uint32_t>(a & 3);
        const uint32_t w0 = q[0], w1 = q[1], w2 = sh ? q[2] : 0u;
        return static_cast<uint64_t>(__funnelshift_r(w1, w2, sh)) << 32 |
               __funnelshift_r(w0, w1, sh);
    }
    __device__ __forceinline__ static uint64_t shfl(uint64_t v, uint32_t from) {
        const uint32_t lo = __shfl_sync(0xffffffffu, static_cast<uint32_t>(v), from);
        const uint32_t hi = __shfl_sync(0xffffffffu, static_cast<uint32_t>(v >> 32), from);
        return static_cast<uint64_t>(hi) << 32 | lo;
    }
    __device__ __forceinline__ void begin(uint32_t lane) {
        const uint32_t a = lane & 3;
        acc = a == 0 ? P1 + P2 : a == 1 ? P2 : a == 2 ? 0 : 0 - P1;
    }
    // stripes of 32 bytes, at most eight
    __device__ __forceinline__ void stripes(const uint8_t* p, uint32_t n, uint32_t lane) {
        const uint64_t m = lane < 4 * n ? rd8(p + 8 * lane) * P2 : 0;
        for (uint32_t k = 0; k < n; ++k)
            acc = rotl(acc + shfl(m, 4 * k + (lane & 3)), 31) * P1;
    }
    // whole steps of p[done, end)
    __device__ __forceinline__ void grow(const uint8_t* p, uint64_t end, uint32_t lane) {
        for (; done + 256 <= end; done += 256) stripes(p + done, 8, lane);
    }
    __device__ __forceinline__ uint64_t digest(const uint8_t* p, uint64_t n, uint32_t lane) {
        grow(p, n, lane);
        const uint32_t rest = static_cast<uint32_t>((n - done) / 32);
        stripes(p + done, rest, lane);
        done += 32ull * rest;
        uint64_t h;
        if (n >= 32) {
            const uint64_t v1 = shfl(acc, 0), v2 = shfl(acc, 1), v3 = shfl(acc, 2),
                           v4 = shfl(acc, 3);
            h = rotl(v1, 1) + rotl(v2, 7) + rotl(v3, 12) + rotl(v4, 18);
            for (uint64_t v : {v1, v2, v3, v4}) h = (h ^ (rotl(v * P2, 31) * P1)) * P1 + P4;
        } else {
            h = P5;
        }
        h += n;
        uint64_t i = done;
        for (; i + 8 <= n; i += 8)
            h = rotl(h ^ (rotl(rd_le(p + i, 8) * P2, 31) * P1), 27) * P1 + P4;
        if (i + 4 <= n) {
            h = rotl(h ^ (rd_le(p + i, 4) * P1), 23) * P2 + P3;
            i += 4;
        }
        for (; i < n; ++i) h = rotl(h ^ (p[i] * P5), 11) * P1;
        h = (h ^ (h >> 33)) * P2;
        h = (h ^ (h >> 29)) * P3;
        return h ^ (h >> 32);
    }
};

struct LitRole {
    const Frame& F;
    TeamSmem& s;
    uint8_t* slot;
    uint32_t lane;
    unsigned huf_log = 0;
    bool huf_present = false;
    uint32_t freed = 0;  // blocks known executed
    Hash hash;

    // Waits for block `freed`; false when it ended the frame.
    __device__ __forceinline__ bool next_free() {
        bar_sync(kBarFree + static_cast<int>(freed & 1), kLitCount);
        const uint64_t out = s.out_at[freed & 1];
        const bool stop = s.stop == freed;
        ++freed;
        if (stop) return false;
        ZS_T(t0);
        if (F.csum) hash.grow(F.dst, out, lane);
        ZS_ADD(4, t0);
        return true;
    }

    // A compressed block's Huffman literals to slot + at.
    __device__ __forceinline__ bool literals(const Block& k, const Lits& l, uint32_t at) {
        const uint8_t* pay = k.b + l.head;
        uint64_t psize = l.csize;
        if (l.type == 2) {
            unsigned cnt, tl;
            uint64_t used;
            if (!huf_weights(pay, psize, s.huf, lane, &cnt, &tl, &used)) return false;
            huf_build(s.huf, cnt, tl, lane);
            huf_log = tl;
            huf_present = true;
            pay += used;
            psize -= used;
        } else if (!huf_present) {
            return false;
        }
        if (psize == 0) return false;
        return huf_streams(pay, psize, l.streams, l.regen, s.huf, huf_log, slot + at, lane);
    }

    __device__ void run() {
        if (F.csum) hash.begin(lane);
        uint64_t pos = F.head;
        uint32_t before = 0;  // slot bytes of the previous block's literals
        uint32_t i = 0;
        bool go = true;
        for (;; ++i) {
            Block k;
            Lits l;
            bool ok = block_head(F, pos, &k);
            uint32_t need = 0;
            if (ok && k.type == 2) {
                ok = lit_head(F, k, &l);
                if (ok && l.type >= 2) need = (l.regen + 15) & ~15u;
            }
            // blocks up to i - 2 are executed, and i - 1 too where the two
            // blocks' literals do not fit the slot together (odd blocks'
            // literals end the slot)
            const uint32_t want = need && before + need > kLitSlot ? i : i ? i - 1 : 0;
            while (go && freed < want) go = next_free();
            if (!go) return;
            const uint32_t at = i & 1 ? kLitSlot - need : 0;
            ZS_T(t0);
            if (need) ok = literals(k, l, at);
            ZS_ADD(3, t0);
            ZS_EV(2, need);
            if (lane == 0) {
                s.lit_at[i & 1] = at;
                s.ready = i + 1;
                if (!ok) s.lit_fault = i;
            }
            __syncwarp();
            bar_arrive(kBarReady + static_cast<int>(i & 1), kLitCount);
            if (!ok || k.last) break;
            before = need;
            pos += 3 + k.body;
        }
        while (freed <= i)
            if (!next_free()) return;
        if (F.csum) {
            // the frame ran to its end: s.out and s.end are its own
            const uint64_t out = s.out_at[i & 1], end = s.end;
            ZS_T(t0);
            const uint32_t h = static_cast<uint32_t>(hash.digest(F.dst, out, lane));
            ZS_ADD(4, t0);
            const bool bad = F.N - end < 4 || h != static_cast<uint32_t>(rd_le(F.f + end, 4));
            if (lane == 0 && bad) s.hash_bad = 1;
        }
    }
};

// ---------------------------------------------------------------------------
// Warps 2 to 5: execution.

// One sequence's effect on the repeat offsets (src/zstd_repcode.h:98-184).
__device__ __forceinline__ Reps reps_of(uint32_t ov, uint32_t ll) {
    if (ov > 3) return Reps{{ov - 3, 0, 0}, 3u | 0u << 2 | 1u << 4};
    const uint32_t tk = ll != 0 ? ov - 1 : ov;
    return tk == 0 ? Reps{{0, 0, 0}, 0u | 1u << 2 | 2u << 4}
         : tk == 1 ? Reps{{0, 0, 0}, 1u | 0u << 2 | 2u << 4}
         : tk == 2 ? Reps{{0, 0, 0}, 2u | 0u << 2 | 1u << 4}
                   : Reps{{1, 0, 0}, 0u | 0u << 2 | 1u << 4};
}
__device__ __forceinline__ uint32_t less(uint32_t a, uint32_t b) { return a > b ? a - b : 0; }
// `b` after `a`.
__device__ __forceinline__ Reps reps_join(const Reps& a, const Reps& b) {
    Reps r;
    r.from = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const uint32_t j = (b.from >> (2 * k)) & 3;
        const uint32_t av = j == 0 ? a.v[0] : j == 1 ? a.v[1] : a.v[2];
        const uint32_t af = (a.from >> (2 * (j & 3))) & 3;
        const bool value = j == 3;
        // an offset of a's result: a value less b's, or an older offset less both
        r.v[k] = value ? b.v[k] : af == 3 ? less(av, b.v[k]) : av + b.v[k];
        r.from |= (value ? 3u : af) << (2 * k);
    }
    return r;
}
// Offset k after a, the three before it being p.
__device__ __forceinline__ uint32_t reps_at(const Reps& a, int k, const uint32_t* p) {
    const uint32_t j = (a.from >> (2 * k)) & 3;
    return j == 3 ? a.v[k] : less(j == 0 ? p[0] : j == 1 ? p[1] : p[2], a.v[k]);
}

struct ExecRole {
    const Frame& F;
    TeamSmem& s;
    const uint8_t* slot;
    uint32_t c;  // executing thread
    uint64_t out = 0;
    uint32_t rep[3] = {1, 4, 8};
    uint32_t block = 0, waited = 0;

    __device__ __forceinline__ void sync() const { bar_sync(kBarExec, kExec); }

    __device__ __forceinline__ void fill(uint64_t at, uint8_t b, uint64_t n) {
        const uint32_t w = 0x01010101u * b;
        uint8_t* to = F.dst + at;
        uint64_t head = (16 - (reinterpret_cast<uintptr_t>(to) & 15)) & 15;
        if (head > n) head = n;
        const uint64_t body = head + ((n - head) & ~15ull);
        if (c < head) to[c] = b;
        for (uint64_t q = head + 16ull * c; q < body; q += 16ull * kExec)
            lzg::put16(to + q, lzg::V16{{w, w, w, w}});
        if (body + c < n) to[body + c] = b;
    }
    __device__ __forceinline__ void copy(uint64_t at, const uint8_t* src, uint64_t n) {
        lzg::copy_share(F.dst + at, src, n, c, kExec);
    }

    // Output [y0, y1) (of the batch whose first sector is at base) of the
    // mapped window at W, kPart bytes at a time (see lz_cta_kernel.cuh).
    __device__ __forceinline__ void gather(uint8_t* base, uint32_t y0, uint32_t y1, uint32_t W,
                                           const uint8_t* lit, uint32_t lit_mask) {
        const uint32_t begin = y0 > W ? y0 - W : 0;
        const uint32_t hi = y1 - W < lzg::kWindow ? y1 - W : lzg::kWindow;
        const uint32_t lane = c & 31;
        uint8_t* wb = base + W;
        for (uint32_t part = begin / kPart * kPart; part < hi; part += kPart) {
            const uint32_t lo = part > begin ? part : begin;
            const uint32_t k = part / 32 + c / 32;
            if (32 * k < hi) {
                lzg::Source src[kUnroll];
                lzg::sources<kUnroll, kItem>(s.map, s.rec, k, kExecWarps, lane, lo, hi, W, src);
                uint32_t v[kUnroll];
#pragma unroll
                for (uint32_t j = 0; j < kUnroll; ++j) {
                    const uint8_t* p = src[j].lit
                                           ? lit + (static_cast<uint32_t>(src[j].at) & lit_mask)
                                           : wb + src[j].at;
                    v[j] = 0;
                    if (src[j].ok) v[j] = *p;
                }
                uint8_t* y = wb + 32 * k + lane;
#pragma unroll
                for (uint32_t j = 0; j < kUnroll; ++j)
                    if (src[j].ok) y[kExec * j] = static_cast<uint8_t>(v[j]);
            }
            sync();
        }
    }

    // A long sequence: literals, then the match, by all executing threads.
    __device__ __forceinline__ void big(uint64_t at, const uint8_t* lit, bool rle, uint32_t ll,
                                        uint32_t ml, uint32_t off) {
        if (rle) fill(at, lit[0], ll);
        else copy(at, lit, ll);
        sync();
        const uint64_t ms = at + ll;
        if (off >= 16 * kExec) {
            // waves that never read their own output
            for (uint64_t k = 0; k < ml; k += off) {
                copy(ms + k, F.dst + ms + k - off, ml - k < off ? ml - k : off);
                sync();
            }
        } else {
            for (uint32_t j = c; j < off; j += kExec) s.period[j] = F.dst[ms - off + j];
            sync();
            lzg::period_share(F.dst + ms, s.period, off, ml, c, kExec);
            sync();
        }
    }

    // The sequences of an item. Returns the first failing one's verdict, and
    // then executes none of them.
    __device__ __forceinline__ int sequences(const Item& it, const Raw* raw, const uint8_t* lit,
                                             uint32_t& lp) {
        const uint32_t lane = c & 31, q = c >> 5;
        const bool have = c < it.n;
        for (uint32_t k = c; k < lzg::kSectors; k += kExec) s.map[k].starts = 0;
        uint32_t ll = 0, ml = 0, ov = 4;
        Reps rp = Reps{{0, 0, 0}, 0u | 1u << 2 | 2u << 4};
        if (have) {
            const Raw r = raw[c];
            BitWin bw;
            bw.init(it.src, it.size);
            // offset, match length and literal length extras, from the top
            const uint32_t co = (r.of >> 16) & 0x1f;
            const uint32_t mcode = s.mcode[(r.ml >> 16) & 0x3f], lcode = s.lcode[(r.ll >> 16) & 0x3f];
            const uint32_t mlb = mcode >> 24, llb = lcode >> 24;
            uint32_t hi, lo;
            bw.window(r.bp - it.shift, &hi, &lo);
            const uint32_t eo = __funnelshift_rc(hi, 0u, 32 - co);
            const uint32_t em = __funnelshift_rc(__funnelshift_lc(lo, hi, co), 0u, 32 - mlb);
            const uint32_t el = BitWin::field(hi, lo, co + mlb, llb);
            // values fit 32 bits: a code below 32 plus its extra bits,
            // lengths below 2^17 + 2^16
            ml = (mcode & 0xffffffu) + em;
            ll = (lcode & 0xffffffu) + el;
            ov = (1u << co) + eo;
            rp = reps_of(ov, ll);
        }
        uint32_t lsum = ll, tsum = ll + ml;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t a = __shfl_up_sync(0xffffffffu, lsum, d);
            const uint32_t b = __shfl_up_sync(0xffffffffu, tsum, d);
            if (lane >= d) {
                lsum += a;
                tsum += b;
            }
        }
        // the repeat offsets: where no sequence of the warp uses one, the
        // state after it is its last three offsets; otherwise a scan
        if (!__any_sync(0xffffffffu, have && ov <= 3) && it.n >= 32 * q + 32) {
            const uint32_t mine = ov - 3;
            rp.v[0] = mine;
            rp.v[1] = __shfl_up_sync(0xffffffffu, mine, 1);
            rp.v[2] = __shfl_up_sync(0xffffffffu, mine, 2);
            rp.from = 3u | 3u << 2 | 3u << 4;  // used of lane 31 alone, but for v[0]
        } else {
#pragma unroll 1
            for (uint32_t d = 1; d < 32; d <<= 1) {
                Reps o;
                o.v[0] = __shfl_up_sync(0xffffffffu, rp.v[0], d);
                o.v[1] = __shfl_up_sync(0xffffffffu, rp.v[1], d);
                o.v[2] = __shfl_up_sync(0xffffffffu, rp.v[2], d);
                o.from = __shfl_up_sync(0xffffffffu, rp.from, d);
                if (lane >= d) rp = reps_join(o, rp);
            }
        }
        if (lane == 31) {
            s.reps[q] = rp;
            s.lsum[q] = lsum;
            s.tsum[q] = tsum;
        }
        sync();
        // the offsets before this warp's sequences, and after all of them;
        // likewise the sums
        uint32_t p[3] = {rep[0], rep[1], rep[2]};
        uint32_t litn = 0, total = 0, lbase = 0, tbase = 0;
#pragma unroll
        for (uint32_t w = 0; w < kExecWarps; ++w) {
            const Reps r = s.reps[w];
            const uint32_t a0 = reps_at(r, 0, rep), a1 = reps_at(r, 1, rep), a2 = reps_at(r, 2, rep);
            rep[0] = a0, rep[1] = a1, rep[2] = a2;
            litn += s.lsum[w];
            total += s.tsum[w];
            if (w < q) {
                p[0] = a0, p[1] = a1, p[2] = a2;
                lbase = litn;
                tbase = total;
            }
        }
        const uint32_t off = reps_at(rp, 0, p);
        lsum += lbase;
        tsum += tbase;
        // the reference driver's checks, each in its order
        const uint32_t lsrc = lp + lsum - ll;
        const uint64_t cur = out + (tsum - ml);  // output before the match
        const int v = !have ? CUDEC_OK
                    : static_cast<uint64_t>(lsrc) + ll > it.regen ? CUDEC_ERR_CORRUPT_INPUT
                    : off == 0 ? CUDEC_ERR_CORRUPT_INPUT
                    : (off > cur || off > F.window) ? CUDEC_ERR_CORRUPT_INPUT
                    : (cur > F.cap || ml > F.cap - cur) ? CUDEC_ERR_OUTPUT_TOO_SMALL
                    : CUDEC_OK;
        uint8_t* const to = F.dst + out;
        const uint32_t y0 = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(to) & 31);
        uint8_t* const base = to - y0;
        const uint32_t y = y0 + tsum - ll - ml, le = y + ll;
        const bool isbig = have && (ll + ml > kBigCopy || off >> 31);  // the gather's limits
        s.rec[c] = lzg::Rec{y, le, lsrc - y, off};
        if (have && !isbig) lzg::map_token(s.map, c, y, le + ml, 0);
        if (c == 0) s.map[0].before = 0;
        const unsigned fails = __ballot_sync(0xffffffffu, v != CUDEC_OK);
        const unsigned bigs = __ballot_sync(0xffffffffu, isbig);
        const int first = __shfl_sync(0xffffffffu, v, fails ? __ffs(fails) - 1 : 0);
        if (lane == 0) {
            s.fail[q] = fails ? first : CUDEC_OK;
            s.big[q] = bigs;
        }
        sync();
        for (uint32_t w = 0; w < kExecWarps; ++w)
            if (s.fail[w] != CUDEC_OK) return s.fail[w];
        uint32_t bigm[kExecWarps];
#pragma unroll
        for (uint32_t w = 0; w < kExecWarps; ++w) bigm[w] = s.big[w];
        const uint32_t mask = it.rle ? 0u : ~0u;
        uint32_t i0 = 0;
        for (;;) {
            uint32_t k = it.n;  // the next long one
#pragma unroll
            for (uint32_t w = kExecWarps; w-- > 0;) {
                const uint32_t from = i0 > 32 * w ? i0 - 32 * w : 0;
                const uint32_t m = from < 32 ? bigm[w] & (~0u << from) : 0u;
                if (m) k = 32 * w + __ffs(m) - 1;
            }
            if (k > i0) {
                const uint32_t a = s.rec[i0].out, z = k < it.n ? s.rec[k].out : y0 + total;
                for (uint32_t W = i0 ? a & ~31u : 0u; W < z; W += lzg::kWindow) {
                    if (i0 || W) {
                        for (uint32_t m = c; m < lzg::kSectors; m += kExec) s.map[m].starts = 0;
                        sync();
                        if (c >= i0 && c < k) lzg::map_token(s.map, c, y, le + ml, W);
                        if (c == i0 && W <= a) s.map[0].before = i0;
                        sync();
                    }
                    gather(base, a, z, W, lit, mask);
                }
            }
            if (k == it.n) break;
            const lzg::Rec r = s.rec[k];
            const uint32_t e = k + 1 < it.n ? s.rec[k + 1].out : y0 + total;
            big(out + (r.out - y0), lit + ((r.out + r.dl) & mask), it.rle != 0, r.le - r.out,
                e - r.le, r.off);
            i0 = k + 1;
            if (i0 == it.n) break;
        }
        lp += litn;
        out += total;
        return CUDEC_OK;
    }

    // Block `block` is executed, or has decided the frame.
    __device__ __forceinline__ void finish_block(bool stop) {
        if (c == 0) {
            s.out_at[block & 1] = out;
            if (stop) s.stop = block;
        }
        sync();
        bar_arrive(kBarFree + static_cast<int>(block & 1), kLitCount);
        ++block;
    }

    __device__ void run() {
        int exec = CUDEC_OK;  // the block's first execution verdict
        uint32_t lp = 0;      // its literals consumed
        const uint8_t* lit = nullptr;
        for (uint32_t i = 0;; ++i) {
            ZS_T(t0);
            bar_sync(kBarItem, kItemCount);
            ZS_ADD(5, t0);
            const Item it = s.item[i & 1];
            int st = CUDEC_OK;   // ends the frame here
            bool over = false;   // warp 0 makes no further item
            if (it.flags & kFirst) {
                ZS_T(t1);
                bar_sync(kBarReady + static_cast<int>(block & 1), kLitCount);
                ZS_ADD(6, t1);
                ++waited;
            }
            if (it.kind == kFault) {
                st = CUDEC_ERR_CORRUPT_INPUT;
                over = true;
            } else {
                over = (it.flags & kEnd) != 0;
                if (it.flags & kFirst) {
                    exec = CUDEC_OK;
                    lp = 0;
                    lit = it.lit != nullptr ? it.lit : slot + s.lit_at[block & 1];
                    if (s.lit_fault == block) st = CUDEC_ERR_CORRUPT_INPUT;
                }
                ZS_T(t2);
                if (st != CUDEC_OK) {
                } else if (it.kind == kSequences) {
                    if (it.n && exec == CUDEC_OK) exec = sequences(it, s.raw[i & 1], lit, lp);
                    if (it.flags & kLast) {
                        const uint32_t tail = it.regen - lp;
                        if (exec != CUDEC_OK) st = exec;
                        else if (out > F.cap || tail > F.cap - out) st = CUDEC_ERR_OUTPUT_TOO_SMALL;
                        else {
                            if (it.rle) fill(out, lit[0], tail);
                            else copy(out, lit + lp, tail);
                            out += tail;
                        }
                    }
                } else if (it.size > F.cap - out) {
                    st = CUDEC_ERR_OUTPUT_TOO_SMALL;
                } else {
                    if (it.kind == kRaw) copy(out, it.src, it.size);
                    else fill(out, it.src[0], it.size);
                    out += it.size;
                }
                ZS_ADD(7, t2);
            }
            if (st != CUDEC_OK) {
                if (c == 0) {
                    s.status = st;
                    s.leave = i + 1;
                }
                finish_block(true);
                if (!over) bar_sync(kBarItem, kItemCount);  // warp 0 learns of it
                break;
            }
            if (it.flags & kLast) finish_block(false);
            if (over) break;
        }
        if (c == 0) {
            s.out = out;
            s.waited = waited;
        }
    }
};

// Decode the frame at the start of f[0, N) by the whole CTA (kTeam threads);
// every thread returns the same status, *written and *consumed (the frame's
// bytes). Bytes after the frame are not looked at. Wide: the frame-sequence
// reading, which also takes a frame without a content size (its output
// bounded by cap alone) and any window whose log is at most kMaxWindowLogSeq;
// otherwise the reference's subset.
template <bool Wide>
__device__ inline int decode_frame_part(const uint8_t* f, uint64_t N, uint8_t* dst, uint64_t cap,
                                        TeamSmem& s, uint8_t* slot, uint64_t* written,
                                        uint64_t* consumed) {
    *written = 0;
    *consumed = 0;
    Frame F{f, N, dst, cap, 0, 0, 0, 0, false, false};
    const int h = frame_head<Wide>(F);
    if (h != CUDEC_OK) return h;
    const uint32_t t = threadIdx.x;
    if (t == 0) {
        s.lit_fault = s.stop = s.leave = ~0u;
        s.ready = s.waited = 0;
        s.status = CUDEC_OK;
        s.hash_bad = 0;
    }
    if (t < 36) s.lcode[t] = kLLCode[t];
    if (t < 53) s.mcode[t] = kMLCode[t];
    __syncthreads();
    if (t < 32) {
        SeqRole{F, s, t}.run();
    } else if (t < 64) {
        LitRole{F, s, slot, t - 32}.run();
    } else {
        ExecRole{F, s, slot, t - 64}.run();
    }
    __syncthreads();
    // literal arrivals that nothing waited for (the frame ended early)
    if (t >= 64)
        for (uint32_t r = s.waited; r < s.ready; ++r)
            bar_sync(kBarReady + static_cast<int>(r & 1), kLitCount);
    const int st = s.status;
    const uint64_t out = s.out, end = s.end;
    const bool bad = s.hash_bad != 0;
    __syncthreads();  // the next frame writes them
    if (st != CUDEC_OK) return st;
    if (F.has_fcs && out != F.fcs) return CUDEC_ERR_CORRUPT_INPUT;
    if (bad) return CUDEC_ERR_CORRUPT_INPUT;
    *written = out;
    *consumed = end + (F.csum ? 4 : 0);
    return CUDEC_OK;
}

// One frame per chunk, the reference's rule (src/zstd_frame.h:196-409):
// bytes after the frame are CORRUPT_INPUT, a skippable frame UNSUPPORTED.
__device__ inline int decode_frame(const uint8_t* f, uint64_t N, uint8_t* dst, uint64_t cap,
                                   TeamSmem& s, uint8_t* slot, uint64_t* written) {
    uint64_t out = 0, used = 0;
    *written = 0;
    const int st = decode_frame_part<false>(f, N, dst, cap, s, slot, &out, &used);
    if (st != CUDEC_OK) return st;
    if (used != N) return CUDEC_ERR_CORRUPT_INPUT;
    *written = out;
    return CUDEC_OK;
}

// A chunk of concatenated frames, as libzstd's ZSTD_decompress reads a
// buffer with its default limits (the reference's subset ladder,
// docs/MASTERPLAN.md:1286-1296, rungs 1-3 up to that limit): skippable
// frames (magic 0x184D2A50-5F, 4-byte size) are skipped, and each Zstd frame
// decodes after the previous one's output, with or without a content size,
// with any window up to a log of kMaxWindowLogSeq (a dictionary id stays
// UNSUPPORTED); fewer than 4 bytes left, or a skippable frame running past
// the chunk, is CORRUPT_INPUT.
__device__ inline int decode_frames(const uint8_t* f, uint64_t N, uint8_t* dst, uint64_t cap,
                                    TeamSmem& s, uint8_t* slot, uint64_t* written) {
    *written = 0;
    uint64_t pos = 0, out = 0;
    while (pos < N) {
        if (N - pos < 4) return CUDEC_ERR_CORRUPT_INPUT;
        const uint32_t magic = static_cast<uint32_t>(rd_le(f + pos, 4));
        if (magic >= 0x184D2A50u && magic <= 0x184D2A5Fu) {
            if (N - pos < 8) return CUDEC_ERR_CORRUPT_INPUT;
            const uint64_t sz = rd_le(f + pos + 4, 4);
            if (sz > N - pos - 8) return CUDEC_ERR_CORRUPT_INPUT;
            pos += 8 + sz;
            continue;
        }
        uint64_t fo = 0, used = 0;
        const int st = decode_frame_part<true>(f + pos, N - pos, dst + out, cap - out, s, slot,
                                               &fo, &used);
        if (st != CUDEC_OK) return st;
        out += fo;
        pos += used;
    }
    *written = out;
    return CUDEC_OK;
}

}  // namespace zstd
}  // namespace cdb
