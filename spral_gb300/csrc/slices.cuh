// FP64 operands as eight balanced base-256 digits (exact in FP16), and the
// way back from exact digit-product sums to FP64: shared by the kernels that
// form FP64 products on the tensor cores (the method is described in
// slice_gemm.cu).  Integer instructions only: an FP64 instruction issues some
// 70 times slower on GB300.
#pragma once
#include <climits>
#include <cstdint>
#include <cuda_runtime.h>

namespace ssids300 {

// exponent of a row with Inf or NaN: the products of the row become NaN
constexpr int kSliceNonFinite = 1 << 19;
// exponent of a row of zeros
constexpr int kEmptyExponent = -(1 << 18);

// biased exponent of an entry after its column's balance 2^h
__device__ __forceinline__ int slice_exponent(unsigned long long bits, int h) {
  const int e = (int)((bits >> 52) & 0x7ff);
  return e == 0x7ff ? kSliceNonFinite : max(e, 1) + h;
}

// exponent of |v|, far below all others for a zero
__device__ __forceinline__ int slice_log2(double v) {
  const int e = (int)(((unsigned)__double2hiint(v) >> 20) & 0x7ff);
  return e ? e - 1023 : -4096;
}
// Column balance 2^h of pivot column c from D^{-1} (dlast ends the pivots), h
// half the exponent of the largest entry in the column of D, so that the
// columns of L 2^h and of L D 2^-h are of one size: 1 / d of a 1x1 pivot; of a
// 2x2 pivot with D^{-1} = [a b; b d], det = a d - b^2, the larger of d / det (a /
// det in its second column) and b / det, by exponents: no 2x2 pivot's det is
// much smaller than the larger of its products.  (The off-diagonal entry alone
// is no measure: threshold pivoting takes 2x2 pivots with any entry there.)
__device__ __forceinline__ int slice_balance(const double* D, int c, int dlast) {
  const long long inf = 0x7ff0000000000000LL;
  // all loads at once
  const double v0 = D[2 * c], v1 = D[2 * c + 1];
  const double p0 = c > 0 ? D[2 * c - 2] : 0.0, p1 = c > 0 ? D[2 * c - 1] : 0.0;
  const double n0 = c + 1 < dlast ? D[2 * c + 2] : 0.0, n1 = c + 1 < dlast ? D[2 * c + 3] : 0.0;
  const bool second = __double_as_longlong(v0) == inf;
  int h = -slice_log2(v0);
  if (second || __double_as_longlong(n0) == inf) {
    const int a = slice_log2(second ? p0 : v0), b = slice_log2(second ? p1 : v1);
    const int d = slice_log2(second ? v1 : n1);
    h = max(second ? a : d, b) - max(a + d, 2 * b);
  }
  return h > -2048 && h < 2048 ? h >> 1 : 0;
}

// The eight balanced digits of an entry (exponent e after the balance, row
// exponent em) as bytes, biased by 128, the leading digit in the top byte.
__device__ __forceinline__ unsigned long long slice_digits(unsigned long long bits, int e, int em) {
  const unsigned hi = (unsigned)(bits >> 32), lo = (unsigned)bits;
  const unsigned m = (hi & 0xfffffu) | ((hi & 0x7ff00000u) ? 0x100000u : 0u);
  // |value| 2^62 / 2^(em - 1022), truncated; the mantissa's 53 bits start at
  // bit 61 for the row's largest exponent.  (A zero's exponent may exceed em;
  // entries of a row with Inf or NaN have no meaning.)
  const unsigned long long M =
      ((unsigned long long)__funnelshift_l(lo, m, 9) << 32) | (unsigned long long)(lo << 9);
  const unsigned long long X = M >> min(max(em - e, 0), 63);
  // balanced digits: the bytes of +-X + 0x8080808080808080, minus 128
  const long long sg = (long long)((int)hi >> 31);
  return (X ^ (unsigned long long)sg) + (0x8080808080808080ULL - (unsigned long long)sg);
}
// byte `byte` of two words as a pair of FP16 digits: 1024 + byte, minus 1152
__device__ __forceinline__ unsigned slice_pair(unsigned x, unsigned y, int byte) {
  const unsigned t = __byte_perm(
      x, y, (unsigned)(byte | (byte << 4) | ((4 + byte) << 8) | ((4 + byte) << 12)));
  unsigned w;
  asm("{\n .reg .b32 t;\n lop3.b32 t, %1, 0x00ff00ff, 0x64006400, 0xea;\n"
      " sub.rn.f16x2 %0, t, %2;\n}\n"
      : "=r"(w)
      : "r"(t), "r"(0x64806480u));
  return w;
}

// Digits of eight consecutive columns of one row (entries b, exponents e after
// the balance, row exponent em): slice s (0 the leading digit) goes to the 16
// bytes at d + s * stride, as eight FP16 values.
__device__ __forceinline__ void slice_store(const unsigned long long (&b)[8], const int (&e)[8],
                                            int em, char* d, int64_t stride) {
  unsigned zl[8], zh[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const unsigned long long Z = slice_digits(b[q], e[q], em);
    zl[q] = (unsigned)Z;
    zh[q] = (unsigned)(Z >> 32);
  }
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    unsigned w[4];
#pragma unroll
    for (int p = 0; p < 4; ++p)
      w[p] = slice_pair(s < 4 ? zh[2 * p] : zl[2 * p], s < 4 ? zh[2 * p + 1] : zl[2 * p + 1],
                        (7 - s) & 3);
    *reinterpret_cast<uint4*>(d + s * stride) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// The FP64 number nearest to (w2 2^64 + w1 2^32 + w0) 2^e, a 96-bit integer in
// two's complement
__device__ __forceinline__ double fixed_to_double(int w2, unsigned w1, unsigned w0, int e) {
  const unsigned sg = (unsigned)(w2 >> 31);
  // magnitude
  unsigned long long lo = ((unsigned long long)(w1 ^ sg) << 32) | (unsigned long long)(w0 ^ sg);
  const unsigned c = sg & 1u;
  lo += c;
  unsigned hi = ((unsigned)w2 ^ sg) + ((lo < (unsigned long long)c) ? 1u : 0u);
  if (hi == 0) {
    hi = (unsigned)(lo >> 32);
    lo <<= 32;
    e -= 32;
  }
  if (hi == 0) {
    hi = (unsigned)(lo >> 32);
    lo <<= 32;
    e -= 32;
    if (hi == 0) {
      hi = (unsigned)(lo >> 32);
      lo = 0;
      e -= 32;
      if (hi == 0) return 0.0;
    }
  }
  const int z = __clz(hi);
  const unsigned t1 = __funnelshift_l((unsigned)(lo >> 32), hi, z);
  const unsigned t0 = __funnelshift_l((unsigned)lo, (unsigned)(lo >> 32), z);
  // 53 bits, to nearest on the next one (the bits below it cannot matter by
  // more than 2^-11 of a unit)
  const unsigned long long q =
      ((((unsigned long long)t1 << 32) | t0) >> 11) + (unsigned long long)((t0 >> 10) & 1u);
  const int E = e + 95 - z + 1023;
  const unsigned long long sign = (unsigned long long)(sg & 0x80000000u) << 32;
  if (E <= 0 || E >= 2046) {  // outside the normal range: rare
    const double v = ldexp((double)q, E - 1023 - 52);
    return sg ? -v : v;
  }
  // a carry of the rounding runs into the exponent, as it should
  return __longlong_as_double((long long)((((unsigned long long)(E - 1)) << 52) + q + sign));
}
// (H 2^32 + L) 2^e with |H|, |L| < 2^62
__device__ __forceinline__ double fixed_to_double(long long H, long long L, int e) {
  const unsigned long long l = (unsigned long long)L;
  const unsigned long long lo = ((unsigned long long)H << 32) + l;
  const int hi = (int)(H >> 32) + (int)(L >> 63) + (lo < l ? 1 : 0);
  return fixed_to_double(hi, (unsigned)(lo >> 32), (unsigned)lo, e);
}

// Exponent of two for fixed_to_double of a product sum of rows with exponents
// er and ec: X_A X_B = T 2^56, each X = value 2^62 / 2^(exponent - 1022)
__device__ __forceinline__ int slice_product_exponent(int er, int ec) {
  return er + ec - 2044 - 68;
}

// ---- mma.sync on digits (small tiles, operands used once) ----
// digits of four entries as MMA registers: v[s][0] holds entries 0, 1 of digit
// s, v[s][1] entries 2, 3 (FP16 pairs)
__device__ __forceinline__ void slice_quad(const unsigned long long (&b)[4], const int (&h)[4],
                                           int em, unsigned (&v)[8][2]) {
  unsigned zl[4], zh[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const unsigned long long Z = slice_digits(b[q], slice_exponent(b[q], h[q]), em);
    zl[q] = (unsigned)Z;
    zh[q] = (unsigned)(Z >> 32);
  }
#pragma unroll
  for (int s = 0; s < 8; ++s)
#pragma unroll
    for (int w = 0; w < 2; ++w)
      v[s][w] = slice_pair(s < 4 ? zh[2 * w] : zl[2 * w], s < 4 ? zh[2 * w + 1] : zl[2 * w + 1],
                           (7 - s) & 3);
}
__device__ __forceinline__ void ldsm_x4(unsigned (&v)[4], const char* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"((unsigned)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm_x2(unsigned (&v)[2], const char* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
               : "=r"(v[0]), "=r"(v[1])
               : "r"((unsigned)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const unsigned (&a)[4],
                                         const unsigned (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// eight levels of exact digit products (each |v| <= 2^22) added to H 2^32 + L
__device__ __forceinline__ void levels_add(const float (&v)[8], long long& H, long long& L) {
  // an integer |i| <= 2^22 plus 1.5 * 2^23 has i in its low mantissa bits; two
  // levels make one 32-bit integer (below 2^30 + 2^22), modulo 2^32 throughout
  int p[4];
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const unsigned i0 = __float_as_uint(v[2 * l] + 12582912.0f);
    const unsigned i1 = __float_as_uint(v[2 * l + 1] + 12582912.0f);
    p[l] = (int)(i0 * 256u + i1 - 257u * 0x4B400000u);
  }
  H += (long long)p[0] * 65536 + p[1];
  L += (long long)p[2] * 65536 + p[3];
}
// their sum as FP64, times 2^e
__device__ __forceinline__ double levels_to_double(const float (&v)[8], int e) {
  long long H = 0, L = 0;
  levels_add(v, H, L);
  return fixed_to_double(H, L, e);
}

// Tiles of 2 TN x TN of the lower trapezoid M x N: row ti of tiles holds
// tile columns 0 .. min(tn, 2 ti + 2) - 1.
template <int TN>
__host__ __device__ inline int trapezoid_tiles(int M, int N) {
  const int tm = (M + 2 * TN - 1) / (2 * TN), tn = (N + TN - 1) / TN;
  const int q = tn / 2 < tm ? tn / 2 : tm;
  return q * (q + 1) + (tm - q) * tn;
}
template <int TN>
__device__ __forceinline__ void trapezoid_tile(int t, int N, int& ti, int& tj) {
  const int tn = (N + TN - 1) / TN;
  const int q = tn / 2;
  if (t >= q * (q + 1)) {
    const int s = t - q * (q + 1);
    ti = q + s / tn;
    tj = s % tn;
    return;
  }
  int i = (int)((sqrtf(4.0f * t + 1.0f) - 1.0f) * 0.5f);
  while (i > 0 && i * (i + 1) > t) --i;
  while ((i + 1) * (i + 2) <= t) ++i;
  ti = i;
  tj = t - i * (i + 1);
}

}  // namespace ssids300
