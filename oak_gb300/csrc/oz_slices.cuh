// Shared pieces of the exact slice products on the FP16 tensor cores (zone_gram_oz.cu,
// zone_isqrt_oz.cu): tcgen05 / mbarrier instructions, the K-major operand tile layout, and the
// balanced base-256 digits of a 54-bit fixed-point number.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace oakg {

namespace {

constexpr int kWaitPolls = 1 << 22;  // bound of every mbarrier wait
// F + kDigitBias has the digits d_p = byte (6 - p) - 128 of F = sum_p d_p 256^(6 - p)
constexpr int kDigits = 7;
constexpr unsigned long long kDigitBias = 0x80808080808080ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);  // start address
  d |= (uint64_t)1 << 16;                   // leading byte offset (unused: K fits one swizzle row)
  d |= (uint64_t)(1024u >> 4) << 32;        // stride byte offset
  d |= (uint64_t)1 << 46;                   // descriptor version
  d |= (uint64_t)2 << 61;                   // 128-byte swizzle
  return d;
}

// instruction descriptor: D F32, A and B FP16, both K-major, M = 128, N = n
__device__ __forceinline__ constexpr uint32_t idesc_f16(uint32_t n) {
  return (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                        uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %3, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %4, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(accum), "r"(idesc));
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   mbar)
               : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
  for (int i = 0; i < kWaitPolls; i++) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

__device__ __forceinline__ void fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// 8 consecutive accumulator columns of this warp's 32 tensor-memory lanes
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}

// byte offset of the 16-byte chunk `chunk` (8 observations) of operand row `row` in a slice
__device__ __forceinline__ uint32_t tile_off(int row, int chunk) {
  return (uint32_t)((row >> 3) * 1024 + (row & 7) * 128 + ((chunk ^ (row & 7)) << 4));
}

// The seven digits of two biased fixed-point numbers (F + kDigitBias) as packed FP16 pairs, a in
// the low half: out[p] holds digit p = byte (6 - p) - 128. 0x6400 | byte is the FP16 number
// 1024 + byte, and subtracting 1152 is exact: five instructions for two digits of a pair,
// where a conversion through FP32 takes eighteen.
__device__ __forceinline__ void digit_pairs(unsigned long long a, unsigned long long b,
                                            uint32_t (&out)[7]) {
  const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32), bl = (uint32_t)b,
                 bh = (uint32_t)(b >> 32);
  const __half2 bias = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));
  auto pair = [&](uint32_t m, uint32_t sel) {
    const uint32_t w = __byte_perm(m, 0x64646464u, sel);
    const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&w), bias);
    return *reinterpret_cast<const uint32_t*>(&h);
  };
  // bytes 0 (then 1) of a and b side by side, bytes 2 and 3 likewise
  const uint32_t l01 = __byte_perm(al, bl, 0x5140), l23 = __byte_perm(al, bl, 0x7362);
  const uint32_t h01 = __byte_perm(ah, bh, 0x5140), h23 = __byte_perm(ah, bh, 0x7362);
  out[6] = pair(l01, 0x4140);
  out[5] = pair(l01, 0x4342);
  out[4] = pair(l23, 0x4140);
  out[3] = pair(l23, 0x4342);
  out[2] = pair(h01, 0x4140);
  out[1] = pair(h01, 0x4342);
  out[0] = pair(h23, 0x4140);
}

// vt 2^e2 rounded to nearest even, by integer operations (the conversion and scaling FP64
// instructions avoided), over FP64's whole range; |vt| < 2^63.
__device__ __forceinline__ double scaled_i64(long long vt, int e2) {
  if (vt == 0) return 0.0;
  const unsigned long long sgn = vt < 0 ? (1ull << 63) : 0ull;
  const unsigned long long m = vt < 0 ? (unsigned long long)(-vt) : (unsigned long long)vt;
  const int lz = __clzll((long long)m);
  const int be = 63 - lz + e2 + 1023;
  const unsigned long long mm = m << lz;  // leading one at bit 63
  if (be < 1) {                           // subnormal: in units of 2^-1074
    const int sh = 12 - be;
    if (sh > 64) return __longlong_as_double((long long)sgn);
    const unsigned long long q = sh < 64 ? mm >> sh : 0ull;
    const unsigned long long rem = sh < 64 ? mm << (64 - sh) : mm, half = 1ull << 63;
    return __longlong_as_double(
        (long long)(sgn | (q + ((rem > half || (rem == half && (q & 1ull))) ? 1ull : 0ull))));
  }
  if (be > 2046) return __longlong_as_double((long long)(sgn | 0x7FF0000000000000ull));
  const unsigned long long mant = (mm >> 11) & 0xFFFFFFFFFFFFFull;
  const unsigned long long rem = mm & 0x7FFull;
  const unsigned long long up = (rem > 0x400ull || (rem == 0x400ull && (mant & 1ull))) ? 1ull : 0ull;
  return __longlong_as_double((long long)(sgn | (((unsigned long long)be << 52) + mant + up)));
}

// 8 consecutive K elements (54-bit fixed point) of an operand row as digit slices
// of SLICE bytes; false where seven digits do not hold one (from 2^55 - 2^47 units on)
template <uint32_t SLICE>
__device__ __forceinline__ bool stage_digits(const long long (&F)[8], unsigned char* slices,
                                             uint32_t off) {
  uint32_t d[4][kDigits];
  unsigned long long all = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const unsigned long long a = (unsigned long long)F[2 * i] + kDigitBias,
                             b = (unsigned long long)F[2 * i + 1] + kDigitBias;
    all |= a | b;
    digit_pairs(a, b, d[i]);
  }
#pragma unroll
  for (int p = 0; p < kDigits; p++)
    *reinterpret_cast<uint4*>(slices + p * SLICE + off) =
        make_uint4(d[0][p], d[1][p], d[2][p], d[3][p]);
  return (all >> 56) == 0;  // the byte past the digits, 0xFF below -2^55
}

// round(x 2^(B - E)) for |x| < 2^E, B = 54 or 62, by integer operations: the 64-bit conversion
// instructions run at the FP64 pipe's rate
template <int B>
__device__ __forceinline__ long long fixed_of(double x, int E) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  int e = (int)((b >> 52) & 0x7FFu);
  unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  if (e == 0) {  // a subnormal: no leading one
    m ^= 0x10000000000000ull;
    e = 1;
  }
  const int s = e - 1075 + B - E;  // x 2^(B - E) = m 2^s
  unsigned long long F;
  if (s >= 0)
    F = m << (s < 10 ? s : 10);
  else
    F = s > -55 ? (m + (1ull << (-s - 1))) >> (-s) : 0ull;
  return (b >> 63) ? -(long long)F : (long long)F;
}

// This thread's half (even or odd digits of the first operand) of 8 product columns: the
// levels' sum in units of 2^(E_row + F_col - 60 + SH). Level L's even part lies in column block L
// (W columns each), its odd part in block L - 1; ta: the first of the columns in block 0, in this
// warp's lanes.
template <uint32_t W, int SH>
__device__ __forceinline__ void read_levels(uint32_t ta, bool odd, long long (&v)[8]) {
  uint32_t r[64];
#pragma unroll
  for (int L = 0; L < 8; L++) {
    // odd digits: level L is in block L - 1 (level 0 has none; block 0 is read in its place)
    const uint32_t col = odd ? (L > 0 ? W * (L - 1) : 0u) : W * L;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r[8 * L]), "=r"(r[8 * L + 1]), "=r"(r[8 * L + 2]), "=r"(r[8 * L + 3]),
          "=r"(r[8 * L + 4]), "=r"(r[8 * L + 5]), "=r"(r[8 * L + 6]), "=r"(r[8 * L + 7])
        : "r"(ta + col));
  }
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int q = 0; q < 64; q += 16)
    asm volatile(""
                 : "+r"(r[q]), "+r"(r[q + 1]), "+r"(r[q + 2]), "+r"(r[q + 3]), "+r"(r[q + 4]),
                   "+r"(r[q + 5]), "+r"(r[q + 6]), "+r"(r[q + 7]), "+r"(r[q + 8]),
                   "+r"(r[q + 9]), "+r"(r[q + 10]), "+r"(r[q + 11]), "+r"(r[q + 12]),
                   "+r"(r[q + 13]), "+r"(r[q + 14]), "+r"(r[q + 15])
                 :
                 : "memory");
  // a level sum x is an integer below 2^22: the bits of x + 1.5 2^23 are kB + x
  constexpr uint32_t kB = 0x4B400000u, kB2 = kB * 257u;
  auto biased = [](uint32_t x) { return __float_as_uint(__uint_as_float(x) + 12582912.f); };
#pragma unroll
  for (int t = 0; t < 8; t++) {
    const uint32_t x0 = odd ? kB : biased(r[t]);
    const int32_t a = (int32_t)((x0 << 8) + biased(r[8 + t]) - kB2);
    const int32_t b = (int32_t)((biased(r[16 + t]) << 8) + biased(r[24 + t]) - kB2);
    const int32_t c = (int32_t)((biased(r[32 + t]) << 8) + biased(r[40 + t]) - kB2);
    const int32_t d = (int32_t)((biased(r[48 + t]) << 8) + biased(r[56 + t]) - (kB2 - (128u << SH)));
    // modulo 2^64; the product's value fits
    long long u = (long long)c * (256 >> SH) + (long long)(d >> (8 + SH));
    u = (long long)b * (16777216 >> SH) + u;
    v[t] = (long long)((unsigned long long)u + ((unsigned long long)((uint32_t)a << (8 - SH)) << 32));
  }
}

}  // namespace

}  // namespace oakg
