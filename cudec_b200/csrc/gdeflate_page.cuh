// One GDeflate page decoded by one warp: the 32 substreams are the 32 lanes.
//
// Each lane keeps its substream's bit buffer (64 bits) and occupancy in
// registers; the word cursor is warp-uniform. A round is one operation per
// lane on its own bits, then the refill: every lane below 32 buffered bits
// takes the next word, in lane order (word = cursor + the number of lower
// lanes that also refill) - the schedule of iderex/cudec
// src/gdeflate_schedule.h:129-165 executed for all 32 lanes at once. Block
// headers, table descriptions, stored bytes and symbols follow the round
// structure documented in oracle_gdeflate_decode (the CPU restatement this
// kernel is checked against): the draft's sections 5-11 and divergences
// D1-D6 from RFC 1951, with the open points decided there.
//
// Symbols: a 10-bit lookup table per code (litlen, distance) in shared
// memory, canonical decoding for longer codes; the precode has a complete
// 7-bit table. End-of-block quiesce is a ballot: lanes after the first lane
// that read end-of-block (and have no distance pending) do not consume.
// Output positions come from a warp scan of the round's item lengths. A
// literal goes straight to the destination; a match is queued once its
// distance is known, and the queue is executed a match per lane when it holds
// 32 (lane_copy.cuh): a round yields some three matches, which on their own
// left most lanes idle while the warp waited for memory once per 16 bytes of
// the longest. Shared memory holds only the tables and the queue, so many
// pages decode per SM: staging the page in shared memory measured 5x slower
// for lack of resident warps.
//
// Bound by instruction issue and, in small batches, by one page's chain of
// rounds; memory is far from it. 4,096 pages of 64 KiB took 2,241 us with
// copies made in each round, the input refilled by per-lane loads, serial
// table builds and long codes walked bit by bit; 1,820 with the queue, the
// refill from a register window, lane-parallel builds and long codes found by
// five compares. 24 pages: 999 and 885 us.
//
// Errors are reported in serial order: an operation's error at lane l
// precedes lane l's refill, which precedes lane l+1's operation.
#pragma once

#include <cstdint>

#include "cudec.h"
#include "lane_copy.cuh"

namespace cdb {
namespace gdf {

constexpr uint32_t kPageMax = 65536;
constexpr uint32_t kTabBits = 10;
constexpr uint32_t kNoEvent = 64;  // event index when none (2 * lane + phase otherwise)

constexpr uint32_t kQueue = 64;      // queued matches: up to a round's 32 past half of it

// Per-warp shared memory: decode tables, then what building them needs, or
// the match queue and its map.
struct __align__(16) Tables {
    // symbol | length << 9, 0: longer than the table (or no code)
    uint16_t ltab[1 << kTabBits];
    uint16_t dtab[1 << kTabBits];
    uint16_t count[16];  // symbols per length during a table build
    uint16_t lsym[288], dsym[32];
    uint32_t base[64];  // lengths' (from 0) and distances' (from 32) base | extra bits << 24
    union {
        struct {
            uint16_t ptab[128];
            uint16_t next[16], place[16];
            uint8_t lens[320];
            uint8_t plen[20];
        } b;
        struct {
            uint32_t at[kQueue], len[kQueue], off[kQueue];
            uint8_t period[lanes::kPeriod];  // a long match's period
        } q;
    } u;
    // codes longer than the table: see Long
    struct Long {
        uint16_t limit[5];  // of length kTabBits + 1 + k, left-aligned in 15 bits: past its codes
        uint16_t from[5];   // its first code, left-aligned the same
        uint16_t index[5];  // its first symbol's place in sym
    } llong, dlong;
};

static __constant__ uint16_t kLBase[29] = {3,  4,  5,  6,  7,  8,  9,  10,  11,  13,
                                    15, 17, 19, 23, 27, 31, 35, 43,  51,  59,
                                    67, 83, 99, 115, 131, 163, 195, 227, 3};
static __constant__ uint8_t kLExtra[29] = {0, 0, 0, 0, 0, 0, 0, 0, 1, 1, 1, 1, 2, 2, 2,
                                    2, 3, 3, 3, 3, 4, 4, 4, 4, 5, 5, 5, 5, 16};
static __constant__ uint32_t kDBase[32] = {1,     2,     3,     4,     5,     7,    9,    13,
                                    17,    25,    33,    49,    65,    97,   129,  193,
                                    257,   385,   513,   769,   1025,  1537, 2049, 3073,
                                    4097,  6145,  8193,  12289, 16385, 24577, 32769, 49153};
static __constant__ uint8_t kDExtra[32] = {0, 0, 0, 0, 1, 1, 2, 2, 3,  3,  4,  4,  5,  5,  6,  6,
                                    7, 7, 8, 8, 9, 9, 10, 10, 11, 11, 12, 12, 13, 13, 14, 14};
static __constant__ uint8_t kPerm[19] = {16, 17, 18, 0, 8, 7, 9, 6, 10, 11, 12, 13, 14, 15, 5, 4, 3, 2, 1};

struct Lane {
    uint64_t bb;
    uint32_t left;
    // the words ahead: lane l holds words l and 32 + l of the 64 from the
    // cursor's group on, so a refill is two shuffles and the loads run 32
    // words ahead of their use
    uint32_t at;          // the cursor within the group, below 32
    uint32_t w0, w1;
    const uint8_t* next;  // the word that lane 0 loads next
    uint64_t avail;       // words from the cursor on
    bool aligned;

    // The word `lane` words past `next`; `off` words past the cursor.
    __device__ __forceinline__ uint32_t word(uint32_t lane, uint32_t off) const {
        if (off >= avail) return 0;
        const uint8_t* p = next + 4 * lane;
        if (aligned) return __ldg(reinterpret_cast<const uint32_t*>(p));
        return static_cast<uint32_t>(__ldg(p)) | (static_cast<uint32_t>(__ldg(p + 1)) << 8) |
               (static_cast<uint32_t>(__ldg(p + 2)) << 16) |
               (static_cast<uint32_t>(__ldg(p + 3)) << 24);
    }
    // The first 32 of the page's n words are the lanes' first bits.
    __device__ __forceinline__ void begin(const uint8_t* page, uint64_t n, uint32_t lane) {
        next = page;
        aligned = (reinterpret_cast<uintptr_t>(page) & 3) == 0;
        avail = n;
        at = 0;
        left = 32;
        bb = word(lane, lane);
        avail -= 32;
        next += 128;
        w0 = word(lane, lane);
        next += 128;
        w1 = word(lane, 32 + lane);
        next += 128;
    }
    __device__ __forceinline__ void consume(uint32_t n) {
        bb >>= n;
        left -= n;
    }
    // The refill turn of every lane; returns the event index of the first
    // lane with no word left (2 * lane + 1), else kNoEvent.
    __device__ __forceinline__ uint32_t refill(uint32_t lane) {
        const bool need = left < 32;
        const unsigned m = __ballot_sync(0xffffffffu, need);
        const uint32_t rank = __popc(m & ((1u << lane) - 1));
        const uint32_t want = __popc(m), i = at + rank;
        const uint32_t v0 = __shfl_sync(0xffffffffu, w0, i & 31);
        const uint32_t v1 = __shfl_sync(0xffffffffu, w1, i & 31);
        if (need && rank < avail) {
            bb |= static_cast<uint64_t>(i < 32 ? v0 : v1) << left;
            left += 32;
        }
        uint32_t ev = kNoEvent;
        if (want > avail) {
            // the lane whose rank equals avail is the first that finds no word
            const unsigned short_lanes = __ballot_sync(0xffffffffu, need && rank >= avail);
            ev = 2 * (__ffs(short_lanes) - 1) + 1;
            at += static_cast<uint32_t>(avail);
            avail = 0;
        } else {
            at += want;
            avail -= want;
        }
        if (at >= 32) {
            at -= 32;
            w0 = w1;
            w1 = word(lane, 32 - at + lane);
            next += 128;
        }
        return ev;
    }
};

// Table from code lengths (sorted symbols for the longer codes and a lookup
// table of tbits bits), 32 symbols at a time: a symbol's place among those of
// its length is its rank in the group (a match over the lanes) past the
// earlier groups'. Returns false (all lanes) when the code is
// over-subscribed.
static __device__ __noinline__ bool build_code(Tables& sm, const uint8_t* lens, uint32_t n,
                                           uint16_t* tab, uint16_t* sym, uint32_t tbits,
                                           Tables::Long* big, uint32_t lane) {
    const uint32_t lt = (1u << lane) - 1;
    uint16_t* next = sm.u.b.next;    // per length: the next code,
    uint16_t* place = sm.u.b.place;  // and the next place in sym
    uint16_t* count = sm.count;
    __syncwarp();
    if (lane < 16) count[lane] = 0;
    __syncwarp();
    for (uint32_t s0 = 0; s0 < n; s0 += 32) {
        const uint32_t l = s0 + lane < n ? lens[s0 + lane] : 0u;
        const unsigned same = __match_any_sync(0xffffffffu, l);
        if (l && (same >> lane) == 1u) count[l] = static_cast<uint16_t>(count[l] + __popc(same));
        __syncwarp();
    }
    // every lane walks the lengths; lane b keeps length b's first code and place
    int leftk = 1;
    bool ok = true;
    uint32_t c = 0, at = 0, prev = 0;
    for (uint32_t b = 1; b < 16; ++b) {
        const uint32_t k = count[b];
        leftk = (leftk << 1) - static_cast<int>(k);
        ok = ok && leftk >= 0;
        c = (c + prev) << 1;
        if (lane == b) {
            next[b] = static_cast<uint16_t>(c);
            place[b] = static_cast<uint16_t>(at);
        }
        if (lane == b && b > kTabBits && big) {
            // a valid code's limits fit: c + k is at most 2^b
            const uint32_t end = (c + k) << (15 - b);
            big->limit[b - kTabBits - 1] = static_cast<uint16_t>(end < 0xffff ? end : 0xffff);
            big->from[b - kTabBits - 1] = static_cast<uint16_t>(c << (15 - b));
            big->index[b - kTabBits - 1] = static_cast<uint16_t>(at);
        }
        at += k;
        prev = k;
    }
    if (!ok) return false;
    const uint32_t size = 1u << tbits;
    for (uint32_t i = lane; i < size; i += 32) tab[i] = 0;
    __syncwarp();
    for (uint32_t s0 = 0; s0 < n; s0 += 32) {
        const uint32_t s = s0 + lane;
        const uint32_t l = s < n ? lens[s] : 0u;
        const unsigned same = __match_any_sync(0xffffffffu, l);
        const uint32_t rank = __popc(same & lt);
        const uint32_t code = next[l] + rank, to = place[l] + rank;  // unused for l = 0
        __syncwarp();
        if (l) {
            sym[to] = static_cast<uint16_t>(s);
            if ((same >> lane) == 1u) {
                next[l] = static_cast<uint16_t>(code + 1);
                place[l] = static_cast<uint16_t>(to + 1);
            }
            if (l <= tbits) {
                const uint32_t rc = __brev(code) >> (32 - l);
                const uint16_t e = static_cast<uint16_t>(s | (l << 9));
                for (uint32_t i = rc; i < size; i += 1u << l) tab[i] = e;
            }
        }
        __syncwarp();
    }
    return true;
}

// Decode a code from the low bits of bb: symbol and length, or false. Codes
// of up to kTabBits bits come from the lookup table. A longer one (a few per
// cent of the symbols, so most rounds have one in some lane) is read
// left-aligned in 15 bits: canonical codes ascend with their length, so its
// length is the first whose limit lies above it, five comparisons without a
// loop.
__device__ __forceinline__ bool decode_sym(uint64_t bb, const uint16_t* tab, const uint16_t* sym,
                                           const Tables::Long& big, uint32_t* s, uint32_t* len) {
    const uint16_t e = tab[bb & ((1u << kTabBits) - 1)];
    if (e) {
        *s = e & 511;
        *len = e >> 9;
        return true;
    }
    const uint32_t code = __brev(static_cast<uint32_t>(bb)) >> 17;
    uint32_t k = 0;
#pragma unroll
    for (uint32_t j = 0; j < 5; ++j) k += code >= big.limit[j];
    if (k == 5) return false;
    *len = kTabBits + 1 + k;
    *s = sym[big.index[k] + ((code - big.from[k]) >> (4 - k))];
    return true;
}

// The first event of a round: op errors (phase 0, status in st) against the
// refill's first failure (phase 1, CORRUPT). Returns CUDEC_OK when none.
__device__ __forceinline__ int first_event(bool err, int st, uint32_t refill_ev, uint32_t lane) {
    const unsigned em = __ballot_sync(0xffffffffu, err);
    const uint32_t op_ev = em ? 2 * (__ffs(em) - 1) : kNoEvent;
    if (op_ev == kNoEvent && refill_ev == kNoEvent) return CUDEC_OK;
    if (op_ev < refill_ev) return __shfl_sync(0xffffffffu, st, op_ev / 2);
    return CUDEC_ERR_CORRUPT_INPUT;
}

// Execute the first n (at most 32) of the queued matches: their positions
// ascend, and every other byte before the last one's end is written.
__device__ __forceinline__ void flush_queue(uint8_t* out, Tables& sm, uint32_t n,
                                            uint32_t lane) {
    __syncwarp();
    const bool mine = lane < n;
    const uint32_t at = mine ? sm.u.q.at[lane] : 0u, len = mine ? sm.u.q.len[lane] : 0u;
    const uint32_t off = mine ? sm.u.q.off[lane] : 0u;
    const uint32_t b0 = __shfl_sync(0xffffffffu, at, 0);
    lanes::match_rounds(out, mine, at, len, off, b0, sm.u.q.period, lane);
}

// Decode one page; every lane returns the same status and *written. Output
// goes straight to dst (its bytes are only ever read back by this warp's own
// copies, ordered by __syncwarp), so a warp needs only its tables in shared
// memory and many warps share an SM.
__device__ __forceinline__ int decode_page(const uint8_t* pg, uint64_t N, uint8_t* dst,
                                           uint64_t cap, Tables& sm, uint32_t lane,
                                           uint64_t* written) {
    *written = 0;
    uint8_t* const out = dst;
    if (N % 4 != 0 || N / 4 < 32) return CUDEC_ERR_CORRUPT_INPUT;
    Lane ln;
    ln.begin(pg, N / 4, lane);
    __syncwarp();
    if (lane < 29) sm.base[lane] = kLBase[lane] | static_cast<uint32_t>(kLExtra[lane]) << 24;
    sm.base[32 + lane] = kDBase[lane] | static_cast<uint32_t>(kDExtra[lane]) << 24;
    uint32_t pos = 0;
    const uint64_t room = cap;
    bool final = false;
    while (!final) {
        // ---- block header round (lane 0) ----
        const uint32_t hb = __shfl_sync(0xffffffffu, static_cast<uint32_t>(ln.bb & 7), 0);
        final = hb & 1;
        const uint32_t btype = hb >> 1;
        if (lane == 0) ln.consume(3);
        if (ln.refill(lane) != kNoEvent) return CUDEC_ERR_CORRUPT_INPUT;
        if (btype == 3) return CUDEC_ERR_CORRUPT_INPUT;
        if (btype == 0) {
            const uint32_t len = __shfl_sync(0xffffffffu, static_cast<uint32_t>(ln.bb & 0xFFFF), 0);
            if (lane == 0) ln.consume(16);
            if (ln.refill(lane) != kNoEvent) return CUDEC_ERR_CORRUPT_INPUT;
            for (uint32_t r = 0; r * 32 < len; ++r) {
                const bool act = r * 32 + lane < len;
                const uint32_t p = pos + r * 32 + lane;
                const uint8_t b = static_cast<uint8_t>(ln.bb);
                int st = CUDEC_OK;
                if (act) {
                    ln.consume(8);
                    if (p >= kPageMax) st = CUDEC_ERR_CORRUPT_INPUT;
                    else if (p >= room) st = CUDEC_ERR_OUTPUT_TOO_SMALL;
                    else out[p] = b;
                }
                const uint32_t rev = ln.refill(lane);
                const int s = first_event(st != CUDEC_OK, st, rev, lane);
                if (s != CUDEC_OK) return s;
            }
            pos += len;
            continue;
        }
        // ---- tables ----
        uint32_t hlit = 288, hdist = 32;
        if (btype == 1) {
            for (uint32_t s = lane; s < 320; s += 32)
                sm.u.b.lens[s] = s < 144 ? 8 : s < 256 ? 9 : s < 280 ? 7 : s < 288 ? 8 : 5;
            __syncwarp();
        } else {
            const uint32_t h = __shfl_sync(0xffffffffu, static_cast<uint32_t>(ln.bb & 0x3FFF), 0);
            hlit = (h & 31) + 257;
            hdist = ((h >> 5) & 31) + 1;
            const uint32_t hclen = (h >> 10) + 4;
            if (lane == 0) ln.consume(14);
            if (ln.refill(lane) != kNoEvent) return CUDEC_ERR_CORRUPT_INPUT;
            if (hlit > 288 || hdist > 32) return CUDEC_ERR_CORRUPT_INPUT;
            if (lane < 19) sm.u.b.plen[kPerm[lane]] = 0;
            __syncwarp();
            if (lane < hclen) {
                sm.u.b.plen[kPerm[lane]] = static_cast<uint8_t>(ln.bb & 7);
                ln.consume(3);
            }
            if (ln.refill(lane) != kNoEvent) return CUDEC_ERR_CORRUPT_INPUT;
            // precode: complete 7-bit table (its codes are at most 7 bits)
            if (!build_code(sm, sm.u.b.plen, 19, sm.u.b.ptab, sm.lsym, 7, nullptr, lane))
                return CUDEC_ERR_CORRUPT_INPUT;
            const uint32_t total = hlit + hdist;
            uint32_t have = 0;
            uint32_t prev_last = 0;  // the last length written so far
            while (have < total) {
                const uint16_t e = sm.u.b.ptab[ln.bb & 127];
                const bool valid = e != 0;
                const uint32_t sym = e & 511, clen = e >> 9;
                uint32_t rep = 1, xb = 0, val = sym;
                if (valid && sym >= 16) {
                    xb = sym == 16 ? 2 : sym == 17 ? 3 : 7;
                    const uint32_t x = static_cast<uint32_t>(ln.bb >> clen) & ((1u << xb) - 1);
                    rep = (sym == 16 ? 3 : sym == 17 ? 3 : 11) + x;
                    val = sym == 16 ? 0xFFFFu : 0;
                }
                // lane l is active while fewer than `total` lengths are known
                uint32_t incl = rep;
#pragma unroll
                for (uint32_t k = 1; k < 32; k <<= 1) {
                    const uint32_t o = __shfl_up_sync(0xffffffffu, incl, k);
                    if (lane >= k) incl += o;
                }
                const uint32_t excl = incl - rep;
                // activity needs the decoded count of earlier lanes; an
                // invalid code stops the count (its lane errors if active)
                const unsigned badm = __ballot_sync(0xffffffffu, !valid);
                const uint32_t first_bad = badm ? __ffs(badm) - 1 : 32;
                const bool act = have + excl < total && lane <= first_bad;
                int st = CUDEC_OK;
                if (act) {
                    if (!valid) st = CUDEC_ERR_CORRUPT_INPUT;
                    else if (sym == 16 && have + excl == 0) st = CUDEC_ERR_CORRUPT_INPUT;
                    else if (have + incl > total) st = CUDEC_ERR_CORRUPT_INPUT;
                }
                // value of code 16 runs: the nearest earlier length
                uint32_t v = act ? val : 0xFFFFu;
#pragma unroll
                for (uint32_t k = 1; k < 32; k <<= 1) {
                    const uint32_t o = __shfl_up_sync(0xffffffffu, v, k);
                    if (v == 0xFFFFu && lane >= k) v = o;
                }
                if (v == 0xFFFFu) v = prev_last;
                if (act && st == CUDEC_OK) {
                    ln.consume(clen + xb);
                    for (uint32_t k = 0; k < rep; ++k) sm.u.b.lens[have + excl + k] = static_cast<uint8_t>(v);
                }
                const uint32_t rev = ln.refill(lane);
                const int s = first_event(st != CUDEC_OK, st, rev, lane);
                if (s != CUDEC_OK) return s;
                const unsigned am = __ballot_sync(0xffffffffu, act);
                const uint32_t last = 31 - __clz(am);
                prev_last = __shfl_sync(0xffffffffu, v, last);
                have += __shfl_sync(0xffffffffu, incl, last);
                __syncwarp();
            }
            if (sm.u.b.lens[256] == 0) return CUDEC_ERR_CORRUPT_INPUT;
        }
        if (!build_code(sm, sm.u.b.lens, hlit, sm.ltab, sm.lsym, kTabBits, &sm.llong, lane))
            return CUDEC_ERR_CORRUPT_INPUT;
        if (!build_code(sm, sm.u.b.lens + hlit, hdist, sm.dtab, sm.dsym, kTabBits, &sm.dlong,
                        lane))
            return CUDEC_ERR_CORRUPT_INPUT;
        // ---- data rounds ----
        bool pend = false, eob = false;
        uint32_t ppos = 0, plen = 0;
        uint32_t queued = 0;
        __syncwarp();  // the queue takes the place of what built the tables
        for (;;) {
            const bool want_dist = pend;
            const bool want_lit = !pend && !eob;
            uint32_t sym = 0, clen = 0;
            bool valid = true;
            // one decode for both kinds of lane (the code chosen per lane),
            // so the warp does not run the two in turn
            if (want_dist || want_lit) {
                const bool dd = want_dist;
                valid = decode_sym(ln.bb, dd ? sm.dtab : sm.ltab, dd ? sm.dsym : sm.lsym,
                                   dd ? sm.dlong : sm.llong, &sym, &clen);
            }
            const unsigned eobm = __ballot_sync(0xffffffffu, want_lit && valid && sym == 256);
            const uint32_t e = eobm ? __ffs(eobm) - 1 : 32;
            // a bad code stops the round at its lane if that lane would act:
            // distance lanes always, literal lanes before end-of-block
            const unsigned badm =
                __ballot_sync(0xffffffffu, !valid && (want_dist || (want_lit && lane < e)));
            const uint32_t first_bad = badm ? __ffs(badm) - 1 : 32;
            const bool act = (want_dist || (want_lit && lane <= e)) && lane <= first_bad;
            uint32_t L = 0, xb = 0, d = 0;
            int st = CUDEC_OK;
            if (act) {
                if (!valid || (!want_dist && sym > 285)) {
                    st = CUDEC_ERR_CORRUPT_INPUT;
                } else if (!want_dist && sym < 256) {
                    L = 1;
                } else if (want_dist || sym > 256) {
                    const uint32_t bx = sm.base[want_dist ? 32 + sym : sym - 257];
                    xb = bx >> 24;
                    const uint32_t v = (bx & 0xffffff) +
                                       (static_cast<uint32_t>(ln.bb >> clen) & ((1u << xb) - 1));
                    if (want_dist) d = v;
                    else L = v;
                }
            }
            uint32_t incl = L;
#pragma unroll
            for (uint32_t k = 1; k < 32; k <<= 1) {
                const uint32_t o = __shfl_up_sync(0xffffffffu, incl, k);
                if (lane >= k) incl += o;
            }
            const uint32_t p = pos + incl - L;
            if (act && st == CUDEC_OK) {
                if (L) {
                    if (p + L > kPageMax) st = CUDEC_ERR_CORRUPT_INPUT;
                    else if (p + L > room) st = CUDEC_ERR_OUTPUT_TOO_SMALL;
                }
                if (want_dist && d > ppos) st = CUDEC_ERR_CORRUPT_INPUT;
            }
            if (act && st == CUDEC_OK) ln.consume(clen + xb);
            const uint32_t rev = ln.refill(lane);
            const int s = first_event(st != CUDEC_OK, st, rev, lane);
            if (s != CUDEC_OK) return s;
            // literals of this round
            if (act && want_lit && sym < 256) out[p] = static_cast<uint8_t>(sym);
            // matches whose distance arrived
            const bool ready = act && want_dist;
            const unsigned rm = __ballot_sync(0xffffffffu, ready);
            if (ready) {
                const uint32_t i = queued + __popc(rm & ((1u << lane) - 1));
                sm.u.q.at[i] = ppos;
                sm.u.q.len[i] = plen;
                sm.u.q.off[i] = d;
            }
            queued += __popc(rm);
            if (act && want_dist) pend = false;
            if (act && want_lit && sym > 256) {
                pend = true;
                ppos = p;
                plen = L;
            }
            pos += __shfl_sync(0xffffffffu, incl, 31);
            if (e < 32) eob = true;
            const bool done = eob && !__any_sync(0xffffffffu, pend);
            while (queued >= 32 || (done && queued)) {
                const uint32_t n = queued < 32 ? queued : 32u;
                flush_queue(out, sm, n, lane);
                queued -= n;
                if (lane < queued) {
                    sm.u.q.at[lane] = sm.u.q.at[32 + lane];
                    sm.u.q.len[lane] = sm.u.q.len[32 + lane];
                    sm.u.q.off[lane] = sm.u.q.off[32 + lane];
                }
                __syncwarp();
            }
            if (done) break;
        }
    }
    if (ln.avail != 0) return CUDEC_ERR_CORRUPT_INPUT;
    __syncwarp();
    *written = pos;
    return CUDEC_OK;
}

}  // namespace gdf
}  // namespace cdb
