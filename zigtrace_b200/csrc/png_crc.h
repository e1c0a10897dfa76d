/*
 * png_crc.h -- arithmetic of the PNG chunk checksum (CRC-32, ISO-HDLC:
 * reflected polynomial 0xEDB88320, register preset to all ones, result
 * complemented) and the powers of x by which output.cu joins the shares of a
 * file's slices.  Polynomials over GF(2) are held bit-reflected: bit 31 is
 * the coefficient of x^0.  Plain C++, so that the host can check it.
 */
#ifndef ZT_PNG_CRC_H
#define ZT_PNG_CRC_H

#include <stdint.h>

#if defined(__CUDACC__)
#define ZT_CRC_HD __host__ __device__
#else
#define ZT_CRC_HD
#endif

namespace zt {

constexpr uint32_t kCrcPoly = 0xEDB88320u;
constexpr uint32_t kCrcOne = 1u << 31; /* x^0 */

/* a * b mod P. */
ZT_CRC_HD constexpr uint32_t crc_mulmod(uint32_t a, uint32_t b) {
  uint32_t p = 0;
  for (int i = 0; i < 32; ++i) {
    p ^= b & (0u - (a >> 31));
    a <<= 1;
    b = (b >> 1) ^ (kCrcPoly & (0u - (b & 1u))); /* b *= x */
  }
  return p;
}

/* Register update for one input byte. */
ZT_CRC_HD constexpr uint32_t crc_byte(uint32_t i) {
  uint32_t c = i;
  for (int k = 0; k < 8; ++k) c = (c >> 1) ^ (kCrcPoly & (0u - (c & 1u)));
  return c;
}

constexpr int kPngThreads = 256;
constexpr uint32_t kPngSeg = 32;                       /* bytes per thread */
constexpr uint32_t kPngSlice = kPngThreads * kPngSeg;  /* 8 KB per block */

/* Largest file: 41 bytes before the zlib stream, at most 2^31 - 1 of it
 * (png.zig:32), its CRC and the IEND chunk; it may start anywhere in a
 * segment. */
constexpr uint64_t kPngMaxSlices = (41 + 0x7FFFFFFFull + 4 + 12 + kPngSeg - 1 + kPngSlice - 1) / kPngSlice;
constexpr int kPngDigits = 4;
static_assert(kPngMaxSlices - 1 < (1ull << (6 * kPngDigits)), "every count of following slices has its digits");

/* Powers of x: seg[t] = x^(8 * kPngSeg * (kPngThreads - 1 - t)), what follows
 * a thread's segment in its slice; slice[d][k] = x^(8 * kPngSlice * k *
 * 64^d), the digits base 64 of the number of slices that follow. */
struct CrcPowers {
  uint32_t seg[kPngThreads];
  uint32_t slice[kPngDigits][64];
  uint32_t tab[256][4]; /* tab[i][j]: register update of byte i followed by j zero bytes */
};
constexpr CrcPowers make_crc_powers() {
  CrcPowers P{};
  uint32_t x = kCrcOne >> 1; /* x^1 */
  for (uint32_t n = 1; n < 8 * kPngSeg; n <<= 1) x = crc_mulmod(x, x);
  uint32_t r = kCrcOne;
  for (int t = kPngThreads - 1; t >= 0; --t) {
    P.seg[t] = r;
    r = crc_mulmod(r, x);
  }
  for (int d = 0; d < kPngDigits; ++d) { /* r = x^(8 * kPngSlice * 64^d) */
    uint32_t q = kCrcOne;
    for (int k = 0; k < 64; ++k) {
      P.slice[d][k] = q;
      q = crc_mulmod(q, r);
    }
    r = q;
  }
  for (uint32_t i = 0; i < 256; ++i) {
    uint32_t c = i;
    for (int j = 0; j < 4; ++j) {
      c = j == 0 ? crc_byte(c) : (c >> 8) ^ crc_byte(c & 255u);
      P.tab[i][j] = c;
    }
  }
  return P;
}

/* x^(8 * bytes of n slices), by its digits base 64; mul is the product mod P. */
template <typename Mul>
ZT_CRC_HD inline uint32_t crc_slices_power(const CrcPowers& P, uint32_t n, const Mul& mul) {
  uint32_t r = P.slice[0][n & 63u];
  for (int d = 1; d < kPngDigits && (n >>= 6) != 0; ++d) r = mul(r, P.slice[d][n & 63u]);
  return r;
}

}  // namespace zt

#endif /* ZT_PNG_CRC_H */
