// Residue arithmetic of the exact tensor-core products (crt_gemm.cu,
// crt_step.cu): the moduli and their tables, balanced residues of scaled
// float64 values, and the reconstruction of a float64 from the residues of an
// integer product.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace slu {
namespace crt {
namespace {

constexpr int NM = 16;   // moduli
struct Tables {
  int p[NM];
  float pf[NM], inv[NM];
  uint32_t ca[2][NM], cb[2][NM];   // balanced 2^(8 i) mod p (A), times (P/p)^-1 (B), packed bytes
  int ba[NM], bb[NM];              // -(2^59) mod p (A), times (P/p)^-1 (B)
  uint32_t w[15][NM / 4];          // byte i of P/p_l, four moduli packed
  int p16[8];                      // P in 16-bit pieces
  float top;                       // 2^112 / P
};

constexpr unsigned long long mod_pow2(int e, int p) {
  unsigned long long r = 1;
  for (int i = 0; i < e; ++i) r = r * 2 % p;
  return r;
}
constexpr int balanced(int v, int p) { return 2 * v > p ? v - p : v; }

constexpr Tables make_tables() {
  Tables T{};
  const int p[NM] = {256, 253, 251, 249, 247, 245, 241, 239, 233, 229, 227, 223, 211, 199, 197, 193};
  unsigned __int128 P = 1;
  for (int l = 0; l < NM; ++l) P *= (unsigned)p[l];
  for (int l = 0; l < NM; ++l) {
    T.p[l] = p[l];
    T.pf[l] = (float)p[l];
    T.inv[l] = 1.0f / (float)p[l];
    const unsigned __int128 W = P / (unsigned)p[l];
    const int wm = (int)(W % (unsigned)p[l]);
    int m = 1;   // inverse of P/p modulo p
    while (m * wm % p[l] != 1) ++m;
    for (int i = 0; i < 8; ++i) {
      const int c = (int)mod_pow2(8 * i, p[l]);
      // p = 256: 128 is its own balanced form's limit; store -128
      int a = balanced(c, p[l]), b = balanced(c * m % p[l], p[l]);
      if (a == 128) a = -128;
      if (b == 128) b = -128;
      T.ca[i / 4][l] |= (uint32_t)(uint8_t)a << (8 * (i % 4));
      T.cb[i / 4][l] |= (uint32_t)(uint8_t)b << (8 * (i % 4));
    }
    const int h = (int)mod_pow2(59, p[l]);
    T.ba[l] = -h;
    T.bb[l] = -(h * m % p[l]);
    for (int i = 0; i < 15; ++i)
      T.w[i][l / 4] |= (uint32_t)(uint8_t)(W >> (8 * i)) << (8 * (l % 4));
  }
  for (int i = 0; i < 8; ++i) T.p16[i] = (int)(uint16_t)(P >> (16 * i));
  T.top = (float)(5192296858534827628530496329220096.0 / (double)P);   // 2^112 / P
  return T;
}
__constant__ Tables c_tab = make_tables();

// Largest |a'| exponent for products of depth K: |X| <= K 2^(2t) <= 2^123 < P / 4,
// and at most the 59 bits that `scaled` shifts by (depths of 8 and less).
constexpr int kMaxBits = 59;
constexpr int bits_for(int K) {
  int lg = 0;
  while ((1LL << lg) < K) ++lg;
  return (123 - lg) / 2 < kMaxBits ? (123 - lg) / 2 : kMaxBits;
}
constexpr bool bits_fit() {
  for (int K = 1; K <= 8192; ++K) {
    int lg = 0;
    while ((1 << lg) < K) ++lg;
    if (bits_for(K) > kMaxBits || lg + 2 * bits_for(K) > 123) return false;
  }
  return true;
}
static_assert(bits_fit(), "scaled operands must fit the shift and the moduli");

// dp4a of unsigned bytes of a with signed bytes of b, and the reverse
__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ int dp4a_su(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp4a.s32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}


__device__ __forceinline__ uint32_t hi32(double v) { return (uint32_t)__double2hiint(v); }

// A float64 (its bits) d powers of two below the largest of its row as a t-bit
// integer (t <= kMaxBits), rounded to nearest and shifted by 2^59 to be non-negative
// (the tables take the shift off again); ok = false gives zero.
__device__ __forceinline__ void scaled_by(uint32_t hi, uint32_t lo, int d, int t, bool ok,
                                          uint32_t& zlo, uint32_t& zhi) {
  const int fe = (int)((hi >> 20) & 0x7ff);
  // the mantissa from bit 63 down: |a'| = m 2^-(s + 1), rounded half away
  const uint32_t mh = (__funnelshift_l(lo, hi, 11) & 0x7fffffffu) | (fe ? 0x80000000u : 0u);
  const uint32_t ml = lo << 11;
  const int s = ok ? 63 - t + d : 64;
  const uint32_t ql = s < 32 ? __funnelshift_r(ml, mh, s) : (s < 64 ? mh >> (s - 32) : 0u);
  const uint32_t qh = s < 32 ? mh >> s : 0u;
  const unsigned long long q = (((unsigned long long)qh << 32 | ql) + 1) >> 1;
  const unsigned long long sg = (long long)(int)hi >> 63;
  const unsigned long long z = (q ^ sg) + ((1ULL << 59) - sg);
  zlo = (uint32_t)z;
  zhi = (uint32_t)(z >> 32);
}
// The same where the largest exponent field of the row is F (>= 1)
__device__ __forceinline__ void scaled(uint32_t hi, uint32_t lo, int F, int t, bool ok,
                                       uint32_t& zlo, uint32_t& zhi) {
  scaled_by(hi, lo, F - max((int)((hi >> 20) & 0x7ff), 1), t, ok, zlo, zhi);
}

// Balanced residue modulo p (ip = 1 / p) of the shifted integer, from the byte
// weights c0, c1 and the bias (table entry + 0x4B400000): |s| < 2^19 is exact
// as the low bits of a float of magnitude 1.5 2^23.
__device__ __forceinline__ float residue(uint32_t zlo, uint32_t zhi, uint32_t c0, uint32_t c1,
                                         int bias, float p, float ip) {
  const int s = dp4a_us(zlo, c0, dp4a_us(zhi, c1, bias));
  const float g = __int_as_float(s) - 12582912.f;
  const float q = fmaf(g, ip, 12582912.f) - 12582912.f;
  return fmaf(-p, q, g);
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// An exact product sum (|x| < 2^24 + 2^8) reduced modulo p: the residue in the
// low byte.
__device__ __forceinline__ uint32_t reduced(float x, float p, float ip) {
  const float k = fmaf(x, ip, 12582912.f) - 12582912.f;
  return __float_as_uint(fmaf(-p, k, x) + 12582912.f);
}

// The magnitude c3:c2:c1:c0 times 2^e, rounded to nearest even, with a sign
__device__ __forceinline__ double to_double(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                            int e, uint32_t neg) {
  unsigned long long lo = (unsigned long long)c1 << 32 | c0, hi = (unsigned long long)c3 << 32 | c2;
  if (!(lo | hi)) return 0.0;
  const int lz = hi ? __clzll(hi) : 64 + __clzll(lo);
  if (lz >= 64) {
    hi = lo << (lz - 64);
    lo = 0;
  } else if (lz > 0) {
    hi = hi << lz | lo >> (64 - lz);
    lo <<= lz;
  }
  // value = hi.lo 2^(64 - lz) with the top bit of hi set: 53 bits kept
  unsigned long long m = hi >> 11;
  const unsigned long long rest = (hi & 0x7ff) << 1 | (lo != 0);
  m += rest > 0x800 || (rest == 0x800 && (m & 1));
  // m in [2^52, 2^53]; value m 2^(75 - lz + e)
  const int field = 75 - lz + e + 1075;
  double v;
  if (field >= 1 && field <= 2045) {
    v = __longlong_as_double((long long)(((unsigned long long)field << 52) +
                                         (m - (1ULL << 52))));
  } else {
    v = ldexp((double)m, 75 - lz + e);
  }
  return __hiloint2double(__double2hiint(v) | (int)(neg << 31), __double2loint(v));
}

// X 2^e for the integer product X with residues r (one byte per modulus, four
// moduli per word): X = sum_l y_l P/p_l - k P, byte position by byte position
// (__dp4a sums four moduli), then 16-bit pieces and 32-bit words with carries.
__device__ __forceinline__ double combine(uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3,
                                          int e) {
  int s[16];
#pragma unroll
  for (int b = 0; b < 15; ++b)
    s[b] = dp4a_su(r3, c_tab.w[b][3],
                   dp4a_su(r2, c_tab.w[b][2],
                           dp4a_su(r1, c_tab.w[b][1], dp4a_su(r0, c_tab.w[b][0], 0))));
  s[15] = 0;
  // k = nearest integer to (sum of y_l P / p_l) / P; the product is below P / 4
  const float f = fmaf((float)s[12], 1.0f / 65536.0f,
                       fmaf((float)s[13], 1.0f / 256.0f, (float)s[14]));
  const int k = __float2int_rn(f * c_tab.top);
  long long w[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int u0 = s[4 * a] + (s[4 * a + 1] << 8) - k * c_tab.p16[2 * a];
    const int u1 = s[4 * a + 2] + (s[4 * a + 3] << 8) - k * c_tab.p16[2 * a + 1];
    w[a] = (long long)u1 * 65536 + u0;
  }
  w[1] += w[0] >> 32;
  w[2] += w[1] >> 32;
  w[3] += w[2] >> 32;
  uint32_t x0 = (uint32_t)w[0], x1 = (uint32_t)w[1], x2 = (uint32_t)w[2], x3 = (uint32_t)w[3];
  // nearly always the magnitude is 2^96 or more and the result a normal number
  const uint32_t neg = x3 >> 31;
  if (neg) {
    x0 = ~x0 + 1;
    x1 = ~x1 + (x0 == 0);
    x2 = ~x2 + ((x0 | x1) == 0);
    x3 = ~x3 + ((x0 | x1 | x2) == 0);
  }
  const int lz = __clz(x3), field = 1023 + 127 + e - lz;
  if (x3 == 0 || field < 1 || field > 2045)
    return to_double(x0, x1, x2, x3, e, neg);
  // the top bit to bit 31 of a; what is below b as its lowest bit
  const uint32_t a = __funnelshift_l(x2, x3, lz);
  const uint32_t b = __funnelshift_l(x1, x2, lz) | ((x1 << lz | x0) != 0);
  const uint32_t lo = __funnelshift_r(b, a, 11);
  const uint32_t up = (b & 0x7ff) + (lo & 1) > 0x400;
  // m in [2^52, 2^53]; value m 2^(field - 1075)
  const unsigned long long m = ((unsigned long long)(a >> 11) << 32 | lo) + up;
  return __longlong_as_double(
      (long long)((((unsigned long long)(field - 1) << 52) + m) | (unsigned long long)neg << 63));
}

}  // namespace
}  // namespace crt
}  // namespace slu
