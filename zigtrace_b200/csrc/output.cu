/*
 * output.cu -- the output stage on the device: Image.toRgb8 / Output.encode
 * (src/image.zig:14-73) and png.writePng (src/png.zig:10-117).
 *
 * Both are byte work.  The encode maps each f64 channel to a byte in one
 * pass.  The PNG takes two launches:
 *   k_png_slices  one block per 8 KB of the file, one thread per 32 bytes:
 *                 generates the bytes (signature, IHDR, zlib header,
 *                 stored-block headers, the filter byte of each row, the RGB
 *                 rows, IEND), writes them, and reduces the slice's share of
 *                 the Adler-32 sums and of the CRC-32;
 *   k_png_sums    adds up the slices' shares and writes the two checksums.
 * The checksums are linear in the bytes, so a slice's share depends on its
 * own bytes and position only: Adler-32 as two modular sums (A = 1 + sum
 * d_i, B = n + sum (n - i) d_i, mod 65521), CRC-32 as the sum over GF(2) of
 * each segment's register times x^(8 bytes that follow it) modulo the CRC
 * polynomial.
 * The bytes are exactly those of the reference's writer for the same RGB8
 * input (same block split, same headers, same checksums).
 */
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <string>
#include <vector>

#include "output.cuh"
#include "png_crc.h"
#include "scene_host.h"

namespace zt {

static zt_status out_cuda_fail(cudaError_t e, const char* what) {
  return fail(ZT_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

/* ------------------------------------------------------------- encode ---- */
/* Output.encode, image.zig:31-37, with Tonemap.apply, image.zig:14-21: the
 * same f64 operations as the host zt_image_to_rgb8. */
__device__ __forceinline__ uint8_t encode_value(double linear, uint32_t tonemap, double gamma, double exposure) {
  const double v = isnan(linear) ? 0.0 : linear;
  const double x = fmax(v * exposure, 0.0);
  double m;
  if (tonemap == 0) m = x;
  else if (tonemap == 1) m = x / (1.0 + x);
  else m = (x * (2.51 * x + 0.03)) / (x * (2.43 * x + 0.59) + 0.14);
  /* std.math.clamp: a NaN gives 1, as @min(NaN, 1) = 1.  Spelled out: nvcc
   * may turn fmax(0, fmin(x, 1)) into a saturating operation that maps NaN
   * to 0 (inf / (1 + inf) in the Reinhard curve, for one). */
  const double mapped = isnan(m) ? 1.0 : fmax(0.0, fmin(m, 1.0));
  const double corrected = pow(mapped, 1.0 / gamma);
  const double c = isnan(corrected) ? 1.0 : fmax(0.0, fmin(corrected, 1.0));
  return (uint8_t)round(c * 255.0);
}

/* encode_value as a call: the encode kernels reach it for the few values
 * that encode_fast leaves. */
__device__ __noinline__ uint8_t encode_value_called(double linear, uint32_t tonemap, double gamma, double exposure) {
  return encode_value(linear, tonemap, gamma, exposure);
}

/* Output.encode's constants for the single-precision estimate: `margin` is
 * an upper bound on |estimate - exact| of c * 255, or above 1/2 when the
 * estimate is not to be used. */
struct EncodeFast {
  float exposure, inv_gamma, margin;
};

/* The byte of one channel from a single-precision estimate of c * 255; true
 * when the estimate is further than `margin` from where the rounding changes,
 * else encode_value has to decide.  Its pow() is what bounded the encode
 * (1920x1080: 83 us, 0.68 TB/s); the estimate takes three instructions of the
 * special-function unit instead.
 * Error bound, u = 2^-24: x = v * exposure has three roundings, 3u.  The
 * curves are quotients N / D of sums of positive terms, whose relative error
 * is what x's error becomes (3u times the curve's elasticity: at most 1, for
 * ACES 1.5, N's being in [1, 2] and D's rising with it) plus the operations'
 * own: E at most 3u (none), 10u (Reinhard: a sum, a division of 2 ulp and a
 * product) and 4.5u + 3u (N) + 4u (D) + 5u = 17u (ACES, its constants
 * rounded too).  With L = log2(mapped)
 * from lg2.approx (2^-22 of max(1, |L|)), y = L / gamma (two roundings) and
 * c = 2^y from ex2.approx (2^-22):
 *   |dc| <= c ln2 (|y| (2^-22 + 2u) + (2^-22 + E / ln2) / gamma) + 2^-22 c,
 * and c |y| = 2^-|y| |y| <= 0.54.  The host takes 1.5 times that, times 255,
 * for 0.1 <= 1 / gamma <= 4.  Below x = 1e-30 (negative values, NaN and zero
 * among them, which all count as 0) the byte is 0 and the estimate of
 * c * 255 below 0.26, flushed subnormals included; above 1e15 every curve
 * gives 255, as the f64 curves do (inf / inf counts as 1).
 * The rounding adds 1.5 * 2^23, whose sum's low bits are the integer. */
template <uint32_t kTonemap>
__device__ __forceinline__ bool encode_fast(double v, const EncodeFast& f, uint32_t& byte) {
  const float x = fminf(fmaxf((float)v * f.exposure, 0.0f), 1e15f);
  float m;
  if (kTonemap == 0) m = x;
  else if (kTonemap == 1) m = __fdividef(x, 1.0f + x);
  else m = __fdividef(x * fmaf(2.51f, x, 0.03f), fmaf(x, fmaf(2.43f, x, 0.59f), 0.14f));
  float l, c;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(fminf(m, 1.0f)));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(c) : "f"(l * f.inv_gamma));
  const float r = fmaf(c, 255.0f, 12582912.0f);
  byte = __float_as_uint(r) & 255u;
  return fabsf(fmaf(c, 255.0f, 12582912.0f - r)) < 0.5f - f.margin;
}

static EncodeFast encode_fast_setup(uint32_t tonemap, double gamma, double exposure) {
  const double inv = 1.0 / gamma, u = ldexp(1.0, -24);
  EncodeFast f{(float)exposure, (float)inv, 1.0f}; /* margin 1: never sure */
  if (!(inv >= 0.1 && inv <= 4.0) || !(fabs(exposure) >= 1e-10 && fabs(exposure) <= 1e10)) return f;
  const double e = (tonemap == 0 ? 3 : tonemap == 1 ? 10 : 17) * u, ln2 = 0.6931471805599453;
  const double dc = ln2 * (0.54 * (4 * u + 2 * u) + inv * (4 * u + e / ln2)) + 4 * u;
  f.margin = (float)(1.5 * 255 * dc + 1e-6); /* c * 255 + 1.5 * 2^23 rounds to an integer; the remainder's rounding */
  return f;
}

/* kEncodePairs pairs of channels per thread, a 16-byte load and a 2-byte
 * store each, both coalesced across the warp; the loads are issued before
 * any value is used.  1920x1080: 14.8 us, 3.8 TB/s (at the copy peak 8.6 us;
 * issue slots bound it), against 83 us with encode_value for every channel. */
constexpr int kEncodePairs = 4;
template <uint32_t kTonemap>
__global__ void __launch_bounds__(256) k_encode_rgb8(const double2* __restrict__ px, uint64_t pairs, EncodeFast f,
                                                     double gamma, double exposure, uchar2* __restrict__ out) {
  const uint64_t base = (uint64_t)blockIdx.x * (256 * kEncodePairs) + threadIdx.x;
  double v[2 * kEncodePairs];
#pragma unroll
  for (int k = 0; k < kEncodePairs; ++k) {
    const double2 p = base + 256 * k < pairs ? __ldcs(px + base + 256 * k) : make_double2(0.0, 0.0);
    v[2 * k] = p.x;
    v[2 * k + 1] = p.y;
  }
  uint32_t e[2 * kEncodePairs], left = 0;
#pragma unroll
  for (int k = 0; k < 2 * kEncodePairs; ++k) left |= encode_fast<kTonemap>(v[k], f, e[k]) ? 0u : 1u << k;
  if (left) { /* one branch for all values */
#pragma unroll
    for (int k = 0; k < 2 * kEncodePairs; ++k)
      if (left >> k & 1u) e[k] = encode_value_called(v[k], kTonemap, gamma, exposure);
  }
#pragma unroll
  for (int k = 0; k < kEncodePairs; ++k)
    if (base + 256 * k < pairs) out[base + 256 * k] = make_uchar2((uint8_t)e[2 * k], (uint8_t)e[2 * k + 1]);
}

/* One value per thread, for the last value of an odd number and for buffers
 * without 16- and 2-byte alignment. */
template <uint32_t kTonemap>
__global__ void __launch_bounds__(256) k_encode_rgb8_scalar(const double* __restrict__ px, uint64_t n, EncodeFast f,
                                                            double gamma, double exposure,
                                                            uint8_t* __restrict__ out) {
  const uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  uint32_t e;
  if (!encode_fast<kTonemap>(px[i], f, e)) e = encode_value_called(px[i], kTonemap, gamma, exposure);
  out[i] = (uint8_t)e;
}

template <uint32_t kTonemap>
static void launch_encode(const double* d_px, uint64_t n, double gamma, double exposure, uint8_t* d_out,
                          cudaStream_t stream) {
  const EncodeFast f = encode_fast_setup(kTonemap, gamma, exposure);
  const bool aligned = ((uintptr_t)d_px % 16 == 0) && ((uintptr_t)d_out % 2 == 0);
  const uint64_t pairs = aligned ? n / 2 : 0, rest = n - 2 * pairs;
  if (pairs)
    k_encode_rgb8<kTonemap>
        <<<(unsigned)((pairs + 256 * kEncodePairs - 1) / (256 * kEncodePairs)), 256, 0, stream>>>(
            reinterpret_cast<const double2*>(d_px), pairs, f, gamma, exposure, reinterpret_cast<uchar2*>(d_out));
  if (rest)
    k_encode_rgb8_scalar<kTonemap><<<(unsigned)((rest + 255) / 256), 256, 0, stream>>>(
        d_px + 2 * pairs, rest, f, gamma, exposure, d_out + 2 * pairs);
}

zt_status launch_encode_rgb8(const double* d_px, uint64_t n_values, uint32_t tonemap, double gamma, double exposure,
                             uint8_t* d_out, cudaStream_t stream) {
  if (tonemap == 0) launch_encode<0>(d_px, n_values, gamma, exposure, d_out, stream);
  else if (tonemap == 1) launch_encode<1>(d_px, n_values, gamma, exposure, d_out, stream);
  else launch_encode<2>(d_px, n_values, gamma, exposure, d_out, stream);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ZT_OK : out_cuda_fail(e, "launch k_encode_rgb8");
}

/* ---------------------------------------------------------------- CRC ---- */
/* x^n mod P; x has order 2^32 - 1, so x^-n is x^(2^32 - 1 - n). */
struct CrcSquares {
  uint32_t v[64]; /* x^(2^k) */
};
constexpr CrcSquares make_crc_squares() {
  CrcSquares s{};
  uint32_t b = kCrcOne >> 1;
  for (int k = 0; k < 64; ++k) {
    s.v[k] = b;
    b = crc_mulmod(b, b);
  }
  return s;
}
static uint32_t crc_xpow(uint64_t n) {
  static constexpr CrcSquares sq = make_crc_squares();
  uint32_t r = kCrcOne;
  for (int k = 0; n != 0; n >>= 1, ++k)
    if (n & 1u) r = crc_mulmod(r, sq.v[k]);
  return r;
}

struct CrcTable {
  uint32_t byte[256];
};
static CrcTable make_crc_table() {
  CrcTable T;
  for (uint32_t i = 0; i < 256; ++i) T.byte[i] = crc_byte(i);
  return T;
}

static __device__ __align__(16) const CrcPowers c_crc_powers = make_crc_powers();

static uint32_t crc32_host(const uint8_t* p, size_t n, const CrcTable& T, uint32_t c = 0xFFFFFFFFu) {
  for (size_t i = 0; i < n; ++i) c = T.byte[(c ^ p[i]) & 0xffu] ^ (c >> 8);
  return c;
}

/* ---------------------------------------------------------------- PNG ---- */
constexpr uint32_t kMaxStoredBlock = 65535; /* png.zig:8 */
constexpr uint32_t kHeadBytes = 41;         /* signature 8 + IHDR chunk 25 + IDAT length 4 + "IDAT" 4 */

PngLayout png_layout(uint64_t width, uint64_t height) {
  PngLayout L;
  memset(&L, 0, sizeof L);
  const uint64_t max31 = 0x7FFFFFFFull;
  if (width == 0 || height == 0 || width > max31 || height > max31) return L; /* png.zig:12-13 */
  const uint64_t raw_len = (width * 3 + 1) * height;                          /* png.zig:29 */
  const uint64_t blocks = (raw_len + kMaxStoredBlock - 1) / kMaxStoredBlock;
  const uint64_t zlib_len = 2 + raw_len + 5 * blocks + 4;
  if (zlib_len > max31) return L; /* png.zig:32 */
  L.width = (uint32_t)width;
  L.height = (uint32_t)height;
  L.row_bytes = (uint32_t)(3 * width);
  L.raw_len = (uint32_t)raw_len;
  L.blocks = (uint32_t)blocks;
  L.zlib_len = (uint32_t)zlib_len;
  L.idat_data = kHeadBytes;
  const uint64_t total = kHeadBytes + zlib_len + 4 /* IDAT CRC */ + 12 /* IEND chunk */;
  if (total > 0xFFFFFFFFull) return PngLayout{};
  L.total = (uint32_t)total;
  return L;
}

static void put_be32(uint8_t* p, uint32_t v) {
  p[0] = (uint8_t)(v >> 24);
  p[1] = (uint8_t)(v >> 16);
  p[2] = (uint8_t)(v >> 8);
  p[3] = (uint8_t)v;
}

/* Signature, IHDR chunk, IDAT length and type (png.zig:15-38); IEND chunk. */
struct PngFrame {
  uint8_t head[kHeadBytes];
  uint8_t tail[12];
};

static PngFrame png_frame(const PngLayout& L, const CrcTable& T) {
  PngFrame F;
  static const uint8_t sig[8] = {0x89, 'P', 'N', 'G', '\r', '\n', 0x1a, '\n'};
  memcpy(F.head, sig, 8);
  uint8_t* ihdr = F.head + 8;
  put_be32(ihdr, 13);
  memcpy(ihdr + 4, "IHDR", 4);
  put_be32(ihdr + 8, L.width);
  put_be32(ihdr + 12, L.height);
  ihdr[16] = 8; /* bit depth */
  ihdr[17] = 2; /* truecolour */
  ihdr[18] = 0; /* deflate */
  ihdr[19] = 0; /* filter method */
  ihdr[20] = 0; /* no interlace */
  put_be32(ihdr + 21, ~crc32_host(ihdr + 4, 17, T));
  put_be32(F.head + 33, L.zlib_len);
  memcpy(F.head + 37, "IDAT", 4);
  put_be32(F.tail, 0);
  memcpy(F.tail + 4, "IEND", 4);
  put_be32(F.tail + 8, ~crc32_host(F.tail + 4, 4, T));
  return F;
}

/* Where a position of the raw stream sits: stored block, offset in it, row
 * and column (column 0 is the filter byte). */
struct PngCursor {
  uint32_t block, off; /* off counts the block's 5 header bytes */
  uint32_t raw;        /* index of the next raw byte */
  uint32_t y, c;
};
__device__ __forceinline__ PngCursor png_cursor(const PngLayout& L, uint32_t r) { /* r: bytes after the zlib header */
  PngCursor p;
  p.block = r / (kMaxStoredBlock + 5);
  p.off = r - p.block * (kMaxStoredBlock + 5);
  p.raw = p.block * kMaxStoredBlock + (p.off < 5 ? 0 : p.off - 5);
  p.y = p.raw / (L.row_bytes + 1);
  p.c = p.raw - p.y * (L.row_bytes + 1);
  return p;
}

/* Four bytes into the register. */
__device__ __forceinline__ uint32_t crc_word(const uint32_t (*tab)[256], uint32_t c) {
  return tab[3][c & 255u] ^ tab[2][(c >> 8) & 255u] ^ tab[1][(c >> 16) & 255u] ^ tab[0][c >> 24];
}

/* a * b mod P without the 32-step loop: the carry-less product from integer
 * products of operands split so that every fourth bit is kept (a column sums
 * at most 8 terms, which its 4 bits hold; the multiplication of T. Pornin's
 * constant-time GHASH), then one table step for the half at and above x^32. */
__device__ __forceinline__ uint32_t crc_mulmod_tab(const uint32_t (*tab)[256], uint32_t a, uint32_t b) {
  uint32_t x[4], y[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[i] = a & (0x11111111u << i);
    y[i] = b & (0x11111111u << i);
  }
  unsigned long long q = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) { /* bits i mod 4 of the product */
    unsigned long long z = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) z ^= (unsigned long long)x[j] * y[(i - j) & 3];
    q |= z & (0x1111111111111111ull << i);
  }
  q <<= 1; /* bit 63 is x^0 */
  return (uint32_t)(q >> 32) ^ crc_word(tab, (uint32_t)q);
}

/* One block per slice of kPngSlice output bytes, aligned to kPngSeg in
 * memory (slice 0 starts `lead` bytes before the file): a thread generates
 * its 32 bytes in registers, writes them as two 16-byte stores and keeps
 * them for the checksums, so the file is written once and never read back.
 * Away from block headers the bytes are a run of the RGB image at any
 * alignment, with one zero (a row's filter byte) inserted where a row begins:
 * words with a funnel shift, and the run delayed by a byte behind the zero.
 * sums: per slice its Adler-32 shares A and B (mod 65521) and its CRC share.
 * What bounds it is the latency of one block's chain (loads, 8 table steps,
 * one polynomial product a thread, two more for the slice): all blocks of a
 * full-HD file are resident at once.  1920x1080 (6.2 MB in, 6.2 MB out):
 * 14.8 us with the second launch, against 120 us for a byte-per-thread
 * gather, two checksum passes over its output and three small launches. */
__global__ void __launch_bounds__(kPngThreads) k_png_slices(const uint8_t* __restrict__ rgb, PngLayout L,
                                                            const __grid_constant__ PngFrame F, uint32_t lead,
                                                            uint8_t* __restrict__ png, uint32_t* __restrict__ sums) {
  __shared__ uint32_t tab[4][256];
  __shared__ uint32_t part[3][kPngThreads / 32];
  const int t = threadIdx.x;
  cudaTriggerProgrammaticLaunchCompletion(); /* k_png_sums may take its place and wait */
  const uint4 row = *reinterpret_cast<const uint4*>(c_crc_powers.tab[t]);
  const uint32_t after_me = c_crc_powers.seg[t];
  const uint32_t raw_at = L.idat_data + 2, adler_at = L.idat_data + L.zlib_len - 4, crc_at = adler_at + 4;
  const int64_t q0 = (int64_t)blockIdx.x * kPngSlice + (int64_t)t * kPngSeg - lead; /* file position */
  uint32_t w[kPngSeg / 4 + 1];
  uint32_t sum = 0, crc = 0;
  unsigned long long sum_b = 0;
  bool run = q0 >= raw_at && q0 + kPngSeg <= adler_at && L.row_bytes >= kPngSeg;
  PngCursor p{};
  if (run) {
    p = png_cursor(L, (uint32_t)q0 - raw_at);
    run = p.off >= 5 && p.off + kPngSeg <= kMaxStoredBlock + 5;
  }
  const uint8_t* src = rgb + (size_t)p.y * L.row_bytes + (p.c == 0 ? 0 : p.c - 1);
  const uint32_t shift = (uint32_t)((uintptr_t)src & 3u);
  const uint32_t* words = reinterpret_cast<const uint32_t*>(src - shift);
  /* the words around the run must lie inside the image */
  run = run && src - shift >= rgb && src - shift + kPngSeg + 4 <= rgb + (size_t)L.row_bytes * L.height;
  if (run) {
#pragma unroll
    for (int k = 0; k <= (int)kPngSeg / 4; ++k) w[k] = __ldg(words + k);
  }
  tab[0][t] = row.x;
  tab[1][t] = row.y;
  tab[2][t] = row.z;
  tab[3][t] = row.w;
  if (run) {
    const uint32_t zero_at = p.c == 0 ? 0 : L.row_bytes + 1 - p.c; /* byte of the run that is the filter byte */
#pragma unroll
    for (int k = 0; k < (int)kPngSeg / 4; ++k) w[k] = __funnelshift_r(w[k], w[k + 1], 8 * shift);
    if (zero_at < kPngSeg) {
      uint32_t before = 0;
#pragma unroll
      for (int k = 0; k < (int)kPngSeg / 4; ++k) {
        const uint32_t now = w[k], late = __funnelshift_l(before, now, 8); /* one byte later */
        before = now;
        const int z = (int)zero_at - 4 * k; /* < 0: behind the zero, > 3: before it */
        const uint32_t head = z >= 4 ? 0xFFFFFFFFu : z <= 0 ? 0u : (1u << (8 * z)) - 1u;
        const uint32_t tail = z < 0 ? 0xFFFFFFFFu : z >= 3 ? 0u : 0xFFFFFFFFu << (8 * z + 8);
        w[k] = (now & head) | (late & tail);
      }
    }
    uint32_t weighted = 0;
#pragma unroll
    for (int k = 0; k < (int)kPngSeg / 4; ++k) {
      sum = __dp4a(w[k], 0x01010101u, sum);
      weighted = __dp4a(w[k], 0x03020100u + 0x04040404u * (uint32_t)k, weighted);
    }
    sum_b = (unsigned long long)(L.raw_len - p.raw) * sum - weighted;
    uint4* o = reinterpret_cast<uint4*>(png + q0);
    o[0] = make_uint4(w[0], w[1], w[2], w[3]);
    o[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
  /* Block headers, the file's head and tail, narrow images: the warp puts
   * such a segment together with a byte per lane (one thread taking its 32
   * bytes one after the other held its block up for 11 us). */
  const uint32_t lane = t & 31;
  for (unsigned left = __ballot_sync(0xffffffffu, !run); left != 0; left &= left - 1) {
    const uint32_t owner = __ffs(left) - 1;
    const int64_t q = q0 + (int64_t)kPngSeg * ((int)owner - (int)lane) + lane;
    uint32_t v = 0, d = 0, db = 0;
    if (q < 0) {
    } else if (q < kHeadBytes) {
      v = F.head[q];
    } else if (q < raw_at) {
      v = q == L.idat_data ? 0x78 : 0x01; /* zlib header, png.zig:40 */
    } else if (q < adler_at) {
      const PngCursor c = png_cursor(L, (uint32_t)q - raw_at);
      if (c.off < 5) { /* stored block header, png.zig:103-110 */
        const uint32_t remaining = L.raw_len - c.block * kMaxStoredBlock;
        const uint32_t len = remaining < kMaxStoredBlock ? remaining : kMaxStoredBlock;
        const uint32_t bits = c.off == 0 ? (len == remaining ? 1u : 0u) : c.off < 3 ? len : ~len;
        v = c.off == 0 ? bits : (bits >> (c.off & 1u ? 0 : 8)) & 0xFFu;
      } else { /* the raw stream: a 0 filter byte, then the row (png.zig:42-46) */
        if (c.c != 0) v = __ldg(rgb + (size_t)c.y * L.row_bytes + (c.c - 1));
        d = v;
        db = (uint32_t)((unsigned long long)(L.raw_len - c.raw) * v % 65521u);
      }
    } else if (q >= crc_at + 4 && q < L.total) {
      v = F.tail[q - (crc_at + 4)];
    }
    if (q >= 0 && q < L.total && !(q >= adler_at && q < crc_at + 4)) png[q] = (uint8_t)v;
    /* the CRC covers the chunk type and the data */
    uint32_t word = q >= (int64_t)L.idat_data - 4 && q < adler_at ? v << (8 * (lane & 3)) : 0u;
    word |= __shfl_xor_sync(0xffffffffu, word, 1);
    word |= __shfl_xor_sync(0xffffffffu, word, 2);
    d = __reduce_add_sync(0xffffffffu, d);
    db = __reduce_add_sync(0xffffffffu, db);
#pragma unroll
    for (int k = 0; k < (int)kPngSeg / 4; ++k) {
      const uint32_t x = __shfl_sync(0xffffffffu, word, 4 * k);
      if (lane == owner) w[k] = x;
    }
    if (lane == owner) {
      sum = d;
      sum_b = db;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < (int)kPngSeg / 4; ++k) crc = crc_word(tab, crc ^ w[k]);
  crc = crc_mulmod_tab(tab, crc, after_me);
  uint32_t b = (uint32_t)(sum_b % 65521u); /* 256 of them, and of sums of 32 bytes, fit 32 bits */
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
    crc ^= __shfl_xor_sync(0xffffffffu, crc, o);
  }
  if ((t & 31) == 0) {
    part[0][t / 32] = sum;
    part[1][t / 32] = b;
    part[2][t / 32] = crc;
  }
  __syncthreads();
  if (t == 0) {
    const uint32_t follow = crc_slices_power(c_crc_powers, gridDim.x - 1 - blockIdx.x, [&](uint32_t a, uint32_t b) {
      return crc_mulmod_tab(tab, a, b);
    });
    uint32_t s0 = 0, s1 = 0, s2 = 0;
    for (int k = 0; k < kPngThreads / 32; ++k) {
      s0 += part[0][k];
      s1 += part[1][k];
      s2 ^= part[2][k];
    }
    sums[3 * (size_t)blockIdx.x + 0] = s0 % 65521u;
    sums[3 * (size_t)blockIdx.x + 1] = s1 % 65521u;
    sums[3 * (size_t)blockIdx.x + 2] = crc_mulmod_tab(tab, s2, follow);
  }
}

/* Adds up the slices and writes Adler-32 (png.zig:47-50) and the chunk CRC,
 * both big-endian.  The CRC register after the data and the four Adler bytes
 * is (sum + preset') x^32-shifted: `undo` takes the zero bytes out that the
 * last slice holds after the data and appends four (x^(32 - 8n)); `preset` is
 * the all-ones start of the register carried past the data and the four
 * bytes; the Adler bytes themselves enter times x^32. */
__global__ void __launch_bounds__(1024) k_png_sums(const uint32_t* __restrict__ sums, uint32_t n_slices, PngLayout L,
                                                   uint32_t undo, uint32_t preset, uint8_t* __restrict__ png) {
  __shared__ uint32_t part[3][32];
  const int t = threadIdx.x;
  cudaGridDependencySynchronize(); /* launched while k_png_slices still runs */
  unsigned long long a = 0, b = 0;
  uint32_t c = 0;
  for (uint32_t s = t; s < n_slices; s += 1024) {
    a += sums[3 * (size_t)s + 0];
    b += sums[3 * (size_t)s + 1];
    c ^= sums[3 * (size_t)s + 2];
  }
  uint32_t a32 = (uint32_t)(a % 65521u), b32 = (uint32_t)(b % 65521u); /* 1024 of them fit 32 bits */
  auto reduce = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a32 += __shfl_xor_sync(0xffffffffu, a32, o);
      b32 += __shfl_xor_sync(0xffffffffu, b32, o);
      c ^= __shfl_xor_sync(0xffffffffu, c, o);
    }
  };
  reduce();
  if ((t & 31) == 0) {
    part[0][t / 32] = a32;
    part[1][t / 32] = b32;
    part[2][t / 32] = c;
  }
  __syncthreads();
  if (t >= 32) return;
  a32 = part[0][t];
  b32 = part[1][t];
  c = part[2][t];
  reduce();
  const uint32_t A = (1 + a32) % 65521u;
  const uint32_t B = (L.raw_len % 65521u + b32) % 65521u;
  const uint32_t adler = __byte_perm((B << 16) | A, 0, 0x0123); /* as the four file bytes lie in memory */
  /* lane 0: the slices' sum; lane 1: the Adler bytes */
  uint32_t crc = crc_mulmod(t == 0 ? c : adler, t == 0 ? undo : kCrcPoly /* x^32 mod P */);
  crc = ~(crc ^ __shfl_xor_sync(0xffffffffu, crc, 1) ^ preset);
  uint8_t* o = png + L.idat_data + L.zlib_len - 4;
  if (t < 4) o[t] = (uint8_t)(adler >> (8 * t));
  crc = __shfl_sync(0xffffffffu, crc, 0);
  if (t >= 4 && t < 8) o[t] = (uint8_t)(crc >> (24 - 8 * (t - 4)));
}

/* Slices that cover a file of L.total bytes starting anywhere in a segment. */
static uint32_t png_slices(const PngLayout& L) { return (uint32_t)((L.total + kPngSeg - 1 + kPngSlice - 1) / kPngSlice); }

size_t png_scratch_bytes(const PngLayout& L) { return (size_t)png_slices(L) * 3 * sizeof(uint32_t); }

zt_status launch_png(const uint8_t* d_rgb, const PngLayout& L, uint8_t* d_png, void* d_scratch, cudaStream_t stream) {
  static const CrcTable T = make_crc_table();
  const PngFrame F = png_frame(L, T);
  uint32_t* sums = static_cast<uint32_t*>(d_scratch);
  const uint32_t ns = png_slices(L), lead = (uint32_t)((uintptr_t)d_png % kPngSeg);
  const uint64_t adler_at = (uint64_t)L.idat_data + L.zlib_len - 4;
  const uint64_t after = (uint64_t)ns * kPngSlice - lead - adler_at; /* bytes of the slices past the data */
  const uint64_t order = 0xFFFFFFFFull;
  const uint32_t undo = crc_xpow((32 + order - (8 * after) % order) % order);
  const uint32_t preset = crc_mulmod(0xFFFFFFFFu, crc_xpow(8 * (adler_at + 4 - (L.idat_data - 4))));
  k_png_slices<<<ns, kPngThreads, 0, stream>>>(d_rgb, L, F, lead, d_png, sums);
  cudaError_t e = cudaGetLastError();
  cudaLaunchAttribute overlap;
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = 1;
  cfg.blockDim = 1024;
  cfg.stream = stream;
  cfg.attrs = &overlap;
  cfg.numAttrs = 1;
  if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, k_png_sums, (const uint32_t*)sums, ns, L, undo, preset, d_png);
  return e == cudaSuccess ? ZT_OK : out_cuda_fail(e, "launch png kernels");
}

/* png.writePng on the host, sequentially (the same bytes). */
static void png_host(const uint8_t* rgb, const PngLayout& L, uint8_t* out) {
  static const CrcTable T = make_crc_table();
  const PngFrame F = png_frame(L, T);
  memcpy(out, F.head, kHeadBytes);
  uint8_t* z = out + L.idat_data;
  size_t w = 0;
  z[w++] = 0x78;
  z[w++] = 0x01;
  uint32_t remaining = L.raw_len, block_left = 0, a = 1, b = 0;
  auto put = [&](uint8_t byte) {
    if (block_left == 0) { /* StoredDeflate.startBlock, png.zig:103-111 */
      const uint32_t len = remaining < kMaxStoredBlock ? remaining : kMaxStoredBlock;
      z[w++] = (uint8_t)(len == remaining ? 1 : 0);
      z[w++] = (uint8_t)(len & 0xFF);
      z[w++] = (uint8_t)(len >> 8);
      z[w++] = (uint8_t)(~len & 0xFF);
      z[w++] = (uint8_t)((~len >> 8) & 0xFF);
      block_left = len;
    }
    z[w++] = byte;
    a = (a + byte) % 65521u;
    b = (b + a) % 65521u;
    --block_left;
    --remaining;
  };
  for (uint32_t y = 0; y < L.height; ++y) {
    put(0);
    for (uint32_t c = 0; c < L.row_bytes; ++c) put(rgb[(size_t)y * L.row_bytes + c]);
  }
  put_be32(z + w, (b << 16) | a);
  w += 4;
  put_be32(z + w, ~crc32_host(out + L.idat_data - 4, 4 + L.zlib_len, T));
  memcpy(z + w + 4, F.tail, 12);
}

}  // namespace zt

using namespace zt;

extern "C" {

zt_status zt_png_size(uint64_t width, uint64_t height, uint64_t* bytes_out) {
  if (!bytes_out) return fail(ZT_ERR_INVALID_ARGUMENT, "zt_png_size: NULL output");
  const PngLayout L = png_layout(width, height);
  *bytes_out = L.total;
  if (L.total == 0) {
    if (width == 0 || height == 0 || width > 0x7FFFFFFFull || height > 0x7FFFFFFFull)
      return fail(ZT_ERR_INVALID_ARGUMENT, "InvalidDimensions: width and height must be in 1 .. 2^31-1");
    return fail(ZT_ERR_INVALID_ARGUMENT, "ImageTooLarge: the zlib stream would exceed 2^31-1 bytes");
  }
  return ZT_OK;
}

zt_status zt_png_encode(const uint8_t* rgb, uint64_t width, uint64_t height, uint8_t* out, uint64_t out_capacity) {
  uint64_t need = 0;
  const zt_status rc = zt_png_size(width, height, &need);
  if (rc != ZT_OK) return rc;
  if (!rgb || !out) return fail(ZT_ERR_INVALID_ARGUMENT, "zt_png_encode: NULL argument");
  if (out_capacity < need) return fail(ZT_ERR_INVALID_ARGUMENT, "zt_png_encode: output smaller than zt_png_size");
  png_host(rgb, png_layout(width, height), out);
  return ZT_OK;
}

zt_status zt_png_encode_device(const uint8_t* d_rgb, uint64_t width, uint64_t height, uint8_t* d_out,
                               uint64_t out_capacity, void* stream) {
  uint64_t need = 0;
  const zt_status rc = zt_png_size(width, height, &need);
  if (rc != ZT_OK) return rc;
  if (!d_rgb || !d_out) return fail(ZT_ERR_INVALID_ARGUMENT, "zt_png_encode_device: NULL argument");
  if (out_capacity < need) return fail(ZT_ERR_INVALID_ARGUMENT, "zt_png_encode_device: output smaller than zt_png_size");
  const PngLayout L = png_layout(width, height);
  cudaStream_t s = (cudaStream_t)stream;
  void* scratch = nullptr;
  const zt_status rc2 = pool_alloc(&scratch, png_scratch_bytes(L), s, "zt_png_encode_device: scratch");
  if (rc2 != ZT_OK) return rc2;
  const zt_status r = launch_png(d_rgb, L, d_out, scratch, s);
  const cudaError_t e = cudaFreeAsync(scratch, s);
  if (r != ZT_OK) return r;
  return e == cudaSuccess ? ZT_OK : out_cuda_fail(e, "zt_png_encode_device: free scratch");
}

zt_status zt_image_to_rgb8_device(const double* d_pixels, uint64_t n_pixels, uint32_t tonemap, double gamma,
                                  double exposure, uint8_t* d_rgb_out, void* stream) {
  if ((!d_pixels || !d_rgb_out) && n_pixels) return fail(ZT_ERR_INVALID_ARGUMENT, "zt_image_to_rgb8_device: NULL argument");
  if (tonemap > 2) return fail(ZT_ERR_INVALID_ARGUMENT, "tonemap must be 0 (none), 1 (reinhard) or 2 (aces)");
  return launch_encode_rgb8(d_pixels, 3 * n_pixels, tonemap, gamma, exposure, d_rgb_out, (cudaStream_t)stream);
}

}  /* extern "C" */
