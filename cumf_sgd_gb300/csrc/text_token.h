// text_token.h - byte-parallel conversion of short rating-text tokens.
//
// Most tokens of a rating text are short: ids of up to 7 digits and ratings such as "4" or
// "3.5".  Such a token is converted from one 64-bit little-endian window of the text (byte 0 =
// the token's first character) with arithmetic on all 8 bytes at once.  The result equals what
// the general parsers of text_parse.cu give for the same token (%d, and %f correctly rounded);
// every token this path does not take (a sign, an exponent, inf/nan, 8 or more characters,
// any byte other than a digit or one '.', a '.' in an id) is left to them, and so are all
// errors.
//
// Shared by the device parser and host tests, so it uses no CUDA-only calls except the
// correctly rounded division, which is IEEE division on the host too.
#pragma once
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define CUMF_HD __host__ __device__ __forceinline__
#else
#define CUMF_HD inline
#endif

namespace cumf {
namespace text_token {

constexpr uint64_t kOnes = 0x0101010101010101ull;
constexpr uint64_t kHigh = 0x8080808080808080ull;

CUMF_HD int lowest_byte(uint64_t high_bits) {  // index of the lowest byte whose bit 7 is set
#ifdef __CUDA_ARCH__
    return (__ffsll((long long)high_bits) - 8) >> 3;
#else
    return __builtin_ctzll(high_bits) >> 3;
#endif
}

CUMF_HD bool space_byte(uint32_t c) { return c == 32u || (c - 9u) <= 4u; }

// Bit 7 of byte i is set iff byte i of x is zero.
CUMF_HD uint64_t zero_bytes(uint64_t x) { return ~(((x & ~kHigh) + ~kHigh) | x | ~kHigh); }

CUMF_HD float div_rn(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fdiv_rn(a, b);
#else
    return a / b;
#endif
}

// Bit 7 of byte i is set iff byte i of x is a space (' ', '\t', '\n', '\v', '\f', '\r').
CUMF_HD uint64_t space_bytes(uint64_t x) {
    const uint64_t ascii = ~x & kHigh;
    const uint64_t ge9 = (x | kHigh) - 0x09ull * kOnes;      // bit 7: b >= 9
    const uint64_t gt13 = (x & ~kHigh) + 0x72ull * kOnes;    // bit 7: b >= 14
    return (zero_bytes(x ^ (0x20ull * kOnes)) | (ge9 & ~gt13 & ascii)) & kHigh;
}

// The bit 7 flags of the 8 bytes (as space_bytes gives them) -> an 8-bit mask, bit i = byte i.
CUMF_HD uint32_t byte_flags(uint64_t high_bits) { return (uint32_t)(((high_bits >> 7) * 0x0102040810204080ull) >> 56); }

// 4 digit values (0-9) in the bytes of a word, the most significant in byte 0 -> their number.
CUMF_HD uint32_t digits4(uint32_t d) {
    d = (d * 10u + (d >> 8)) & 0x00ff00ffu;  // byte 2j <- 10*b[2j] + b[2j+1]
    return (d * 100u + (d >> 16)) & 0xffffu;
}

// Four characters that are all digits: their low halves; *ok is cleared otherwise.  (The test that
// simdjson's number parser is known for: a byte is a digit iff its high half is 3 and adding 6
// leaves it 3; a carry into the next byte comes only from a byte that is none.)
CUMF_HD uint32_t digit_values(uint32_t y, bool *ok) {
    *ok &= ((y & 0xf0f0f0f0u) | (((y + 0x06060606u) & 0xf0f0f0f0u) >> 4)) == 0x33333333u;
    return y & 0x0f0f0f0fu;
}

// The number of the first n (0..7) characters of x, all digits; *ok is cleared otherwise.  They
// are moved to the end of 8 characters, '0' before them.
CUMF_HD uint32_t digits_value(uint64_t x, int n, bool *ok) {
    const uint64_t y = n ? (x << (64 - 8 * n)) | ((0x30ull * kOnes) >> (8 * n)) : 0x30ull * kOnes;
    const uint32_t hi = digit_values((uint32_t)y, ok), lo = digit_values((uint32_t)(y >> 32), ok);
    return digits4(hi) * 10000u + digits4(lo);
}

// x: the 8 bytes starting at a token's first character; n (1..7): its length, byte n of x
// being a space.  is_rating: the token is the third field of a record (%f) rather than an id
// (%d).  Returns true and the 32-bit field (the id, or the float's bits) when the token is
// taken here.
CUMF_HD bool convert_n(uint64_t x, int n, bool is_rating, uint32_t *word) {
    bool ok = true;
    if (!is_rating) {
        *word = digits_value(x, n, &ok);  // < 10^7
        return ok;
    }
    int frac = 0;
    const uint64_t dots = n > 1 ? zero_bytes(x ^ (0x2eull * kOnes)) & ((1ull << (8 * n)) - 1) & kHigh : 0;
    if (dots) {  // drop the first '.' (a second one is not a digit)
        const int at = lowest_byte(dots);
        const uint64_t below = (1ull << (8 * at)) - 1;  // the bytes before it
        x = (x & below) | ((x >> 8) & ~below);
        frac = --n - at;
    }
    // value < 10^7 < 2^24 and 10^frac (frac <= 6) are exact floats: one rounded division is
    // the correctly rounded value of value * 10^-frac (the general parser's first case does
    // the same).
    float f = (float)digits_value(x, n, &ok);
    if (frac) f = div_rn(f, ((frac & 1) ? 10.f : 1.f) * ((frac & 2) ? 100.f : 1.f) * ((frac & 4) ? 10000.f : 1.f));
#ifdef __CUDA_ARCH__
    *word = __float_as_uint(f);
#else
    memcpy(word, &f, 4);
#endif
    return ok;
}

// The same, finding the token's end in x itself (the first byte below 0x21 must be a space;
// a token of 8 or more characters is not taken).
CUMF_HD bool convert(uint64_t x, bool is_rating, uint32_t *word) {
    const uint64_t ctl = ~((x | kHigh) - 0x21ull * kOnes) & ~x & kHigh;
    const uint64_t end = ctl & (0ull - ctl);
    if (end == 0 || end == 0x80u || !(end & space_bytes(x))) return false;
    return convert_n(x, lowest_byte(end), is_rating, word);
}

}  // namespace text_token
}  // namespace cumf
