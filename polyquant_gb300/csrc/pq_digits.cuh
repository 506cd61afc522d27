// FP64 numbers as eight signed base-256 digits held in FP16, so that products of FP64 matrices run on the tensor
// cores without rounding (the error-free splitting of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 2012, here
// with digits of one common exponent): x = 2^(e - 6) sum_i d_i 256^-i for a common exponent e of a row with |x| < 2^e.
//
// A number becomes the integer t = round(x 2^(62 - e)), |t| <= 2^62, and its balanced bytes d_i in [-128, 127]
// (|d_0| <= 64).  A product of two rows is sum_l 256^-l a_l with a_l = sum_{i + j = l} sum_k d_i d'_j.  For K <= 256
// the sums of orders 0 .. 4 stay at or below 2^24, so their FP32 accumulation is exact, and a rounding of order
// l >= 5 is below 2^-59 of the largest possible product.  Orders 0 .. 7 are kept (36 digit products): what is left
// out is below 2^-62 of the two row maxima for each of the K terms, where an FP64 product rounds each term at 2^-53.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace pq {
namespace digits {

constexpr int N = 8;            // digits, and orders kept
constexpr int CHUNK = 32;       // K values whose digits lie together: [chunk][digit][32]
constexpr int BAD = 1 << 28;    // exponent of a row that holds an infinity or a NaN

// row length in FP16 of K values
__host__ __device__ constexpr int64_t row_len(int64_t k) { return (k + CHUNK - 1) / CHUNK * CHUNK * N; }

// exponent e with |x| < 2^e for every x whose high word (sign removed) is at most hi
__device__ __forceinline__ int exponent_of(uint32_t hi) {
  const int ex = (int)(hi >> 20);
  return ex == 0x7ff ? BAD : ex - 1022;
}

// round(x 2^(BITS - e)) for |x| < 2^e, by integer arithmetic (the FP64 pipe runs at 1/64 of the integer rate)
template <int BITS = 62> __device__ __forceinline__ int64_t fixed_point(double x, int e) {
  const uint64_t b = (uint64_t)__double_as_longlong(x);
  const int ex = (int)((b >> 52) & 0x7ff);
  const uint64_t mant = (b & 0xfffffffffffffULL) | (ex ? 1ULL << 52 : 0ULL);
  const int sh = (ex ? ex : 1) - e - 1075 + BITS;  // <= BITS - 53
  uint64_t t;
  if (sh >= 0)
    t = mant << sh;
  else
    t = sh > -54 ? (mant + (1ULL << (-sh - 1))) >> -sh : 0ULL;
  const int64_t s = (int64_t)b >> 63;
  return ((int64_t)t ^ s) - s;
}

// the eight digits of t as FP16, four packed pairs (d_0, d_1), (d_2, d_3), ...: with 0x80 added to every byte each
// byte is a digit plus 128, and 1024 + byte has the byte as its FP16 mantissa
__device__ __forceinline__ void to_half(int64_t t, __half2 (&d)[4]) {
  const uint64_t u = (uint64_t)t + 0x8080808080808080ULL;
  const uint32_t w[2] = {(uint32_t)(u >> 32), (uint32_t)u};
  const __half2 off = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));  // 1152
#pragma unroll
  for (int i = 0; i < 4; i++) {
    // bytes 3 and 2 (i even) or 1 and 0 (i odd) of the word, most significant digit first
    const uint32_t p = (i & 1) ? __byte_perm(w[i >> 1], 0x64646464u, 0x4041) : __byte_perm(w[i >> 1], 0x64646464u, 0x4243);
    d[i] = __hsub2(*reinterpret_cast<const __half2 *>(&p), off);
  }
}

__device__ __forceinline__ int64_t mad_wide(int a, int b, int64_t c) {
  int64_t d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}

// sum_l 256^(7 - l) a_l as hi 2^32 + lo; a_0 is below 2^21 and a_1 below 2^23, so 256 a_0 + a_1 stays in 32 bits
__device__ __forceinline__ void combine(const float (&a)[N], int64_t &hi, int64_t &lo) {
  int v[N];
#pragma unroll
  for (int l = 0; l < N; l++) v[l] = __float2int_rn(a[l]);
  hi = mad_wide(v[0] * 256 + v[1], 65536, mad_wide(v[2], 256, v[3]));
  lo = (mad_wide(v[4], 256, v[5]) << 16) + mad_wide(v[6], 256, v[7]);
}

// (hi 2^32 + lo) 2^e rounded to FP64, by integer arithmetic
__device__ __forceinline__ double to_double(int64_t hi, int64_t lo, int e) {
  hi += lo >> 32;
  uint32_t l = (uint32_t)lo;
  const int64_t sgn = hi >> 63;
  uint64_t h = (uint64_t)(hi ^ sgn);
  l ^= (uint32_t)sgn;
  if (sgn) h += ++l == 0;  // two's complement of the 96-bit magnitude
  if (h == 0) {
    h = l;
    l = 0;
    e -= 32;
  }
  if (h == 0) return 0.0;
  const int lz = __clzll((long long)h);
  // the top 64 bits; what lies below is under 2^-63 of the value
  const uint64_t m = (h << lz) | (lz ? ((uint64_t)l << 32) >> (64 - lz) : 0ULL);
  const uint64_t r = (m >> 11) + ((m >> 10) & 1ULL);  // 2^52 .. 2^53
  const int ex = 1118 - lz + e;                       // the value is r 2^(ex - 1075)
  if (ex < 1 || ex > 2045) return (sgn ? -1.0 : 1.0) * scalbn((double)r, ex - 1075);
  return __longlong_as_double((long long)(((uint64_t)(ex - 1) << 52) + r) | (sgn & (long long)0x8000000000000000ULL));
}

}  // namespace digits

// The same with seven signed base-512 digits (|d_0| <= 128, the others <= 256, exact in FP16) and eight orders, 34
// digit products, for sums of at most 80 products: t = round(x 2^(61 - e)) = sum_i d_i 512^(6 - i).  Orders 0 .. 3 stay
// below 2^24 for 80 terms, a rounding of order l >= 4 is below 2^-55 of the largest possible sum; the products left
// out are below 2^-67 of the two maxima each.
namespace digits9 {

constexpr int N = 7, ORDERS = 8, BITS = 61;

// the seven digits of t as FP16 bits
__device__ __forceinline__ void to_half(int64_t t, unsigned short (&d)[N]) {
  uint64_t off = 0;
#pragma unroll
  for (int k = 0; k < N; k++) off |= 256ULL << (9 * k);
  const uint64_t u = (uint64_t)t + off;
#pragma unroll
  for (int i = 0; i < N; i++) {
    const unsigned f = (unsigned)(u >> (9 * (N - 1 - i))) & 511u;
    d[i] = __half_as_ushort(__hsub(__ushort_as_half((unsigned short)(0x6400u | f)), __ushort_as_half((unsigned short)0x6500)));
  }
}

// sum_l 512^(7 - l) a_l as hi 2^36 + lo; 512 a_0 + a_1 stays in 32 bits
__device__ __forceinline__ void combine(const float (&a)[ORDERS], int64_t &hi, int64_t &lo) {
  int v[ORDERS];
#pragma unroll
  for (int l = 0; l < ORDERS; l++) v[l] = __float2int_rn(a[l]);
  hi = digits::mad_wide(v[0] * 512 + v[1], 1 << 18, digits::mad_wide(v[2], 512, v[3]));
  lo = (digits::mad_wide(v[4], 512, v[5]) << 18) + digits::mad_wide(v[6], 512, v[7]);
}

// The same for sums below 2^22 by multiply-adds alone: conversions run at an eighth and integer logic and adds at half
// of their rate.  1.5 2^23 + a_l has a_l in its low bits, so hi and lo come with the constants HI and LO added.  `far`
// collects squares: from 2^44 on some sum may have been too large.
constexpr uint32_t MAGIC = 0x4b400000u;  // bits of 1.5 2^23
constexpr uint64_t HI = (uint64_t)MAGIC * 513u, LO = (uint64_t)MAGIC * 513u * ((1u << 18) + 1u);
constexpr float FAR = 17592186044416.0f;  // 2^44
__device__ __forceinline__ void combine_small(const float (&a)[ORDERS], uint64_t &hi, uint64_t &lo, float &far) {
  uint32_t v[ORDERS];
#pragma unroll
  for (int l = 0; l < ORDERS; l++) {
    v[l] = __float_as_uint(a[l] + 12582912.0f);
    far = fmaf(a[l], a[l], far);
  }
  auto wide = [](uint32_t x, uint32_t m, uint64_t y) {
    uint64_t d;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(x), "r"(m), "l"(y));
    return d;
  };
  const int top = (int)(v[0] * 512u + v[1] - MAGIC * 513u);
  hi = (uint64_t)digits::mad_wide(top, 1 << 18, (int64_t)wide(v[2], 512u, v[3]));
  const uint64_t x = wide(v[4], 512u, v[5]), y = wide((uint32_t)x, 1u << 18, wide(v[6], 512u, v[7]));
  lo = y + ((uint64_t)((uint32_t)(x >> 32) << 18) << 32);
}

}  // namespace digits9
}  // namespace pq
