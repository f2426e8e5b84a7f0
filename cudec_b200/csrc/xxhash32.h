// XXH32 (seed 0 by default), written from the published xxHash specification
// (xxhash.com, "xxHash fast digest algorithm", 32-bit variant): four 32-bit
// accumulators over 16-byte stripes, then the 4-byte and 1-byte tails and the
// final avalanche. Used for the LZ4 frame's header, block and content
// checksums (lz4 frame format, "Header Checksum" / "Block checksum" /
// "Content checksum"). Host-only.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstring>

namespace cdb {

constexpr uint32_t kXxhP1 = 0x9E3779B1u;
constexpr uint32_t kXxhP2 = 0x85EBCA77u;
constexpr uint32_t kXxhP3 = 0xC2B2AE3Du;
constexpr uint32_t kXxhP4 = 0x27D4EB2Fu;
constexpr uint32_t kXxhP5 = 0x165667B1u;

inline uint32_t xxh_rotl(uint32_t x, int r) { return (x << r) | (x >> (32 - r)); }

inline uint32_t xxh_read32(const unsigned char* p) {
    uint32_t v;
    std::memcpy(&v, p, 4);  // little-endian hosts
    return v;
}

// The digest of data that arrives in parts: stripes() takes whole 16-byte
// stripes, finish() the rest.
class Xxh32 {
  public:
    explicit Xxh32(uint32_t seed = 0)
        : seed_(seed), v_{seed + kXxhP1 + kXxhP2, seed + kXxhP2, seed, seed - kXxhP1} {}

    void stripes(const unsigned char* p, size_t n) {  // n stripes
        len_ += 16 * static_cast<uint64_t>(n);
        uint32_t a = v_[0], b = v_[1], c = v_[2], d = v_[3];
        for (; n != 0; --n, p += 16) {
            a = xxh_rotl(a + xxh_read32(p) * kXxhP2, 13) * kXxhP1;
            b = xxh_rotl(b + xxh_read32(p + 4) * kXxhP2, 13) * kXxhP1;
            c = xxh_rotl(c + xxh_read32(p + 8) * kXxhP2, 13) * kXxhP1;
            d = xxh_rotl(d + xxh_read32(p + 12) * kXxhP2, 13) * kXxhP1;
        }
        // One register each: seen as one vector (they leave for one array), the
        // four took 32-bit vector products without hardware for them, 2.5 GB/s
        // instead of 5.1.
        asm("" : "+r"(a), "+r"(b), "+r"(c), "+r"(d));
        v_[0] = a, v_[1] = b, v_[2] = c, v_[3] = d;
    }

    uint32_t finish(const unsigned char* p, size_t rest) {  // rest < 16
        uint32_t h = len_ != 0 ? xxh_rotl(v_[0], 1) + xxh_rotl(v_[1], 7) + xxh_rotl(v_[2], 12) +
                                     xxh_rotl(v_[3], 18)
                               : seed_ + kXxhP5;
        h += static_cast<uint32_t>(len_ + rest);
        const unsigned char* const end = p + rest;
        for (; p + 4 <= end; p += 4) h = xxh_rotl(h + xxh_read32(p) * kXxhP3, 17) * kXxhP4;
        for (; p < end; ++p) h = xxh_rotl(h + (*p) * kXxhP5, 11) * kXxhP1;
        h ^= h >> 15;
        h *= kXxhP2;
        h ^= h >> 13;
        h *= kXxhP3;
        h ^= h >> 16;
        return h;
    }

  private:
    uint32_t seed_;
    uint32_t v_[4];
    uint64_t len_ = 0;
};

inline uint32_t xxh32(const void* data, size_t len, uint32_t seed = 0) {
    const unsigned char* p = static_cast<const unsigned char*>(data);
    Xxh32 h(seed);
    h.stripes(p, len / 16);
    return h.finish(p + len / 16 * 16, len % 16);
}

}  // namespace cdb
