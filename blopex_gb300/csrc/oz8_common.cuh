// oz8_common.cuh -- the digits of the FP64-accurate split-operand kernels
// oz_xc64.cu and oz_gram64.cu (the error-free splitting of oz_common.cuh with
// seven 8-bit digits in fp16, levels 0-7 of their products).
#pragma once
#include "oz_common.cuh"

// ---------------------------------------- seven 8-bit digits (55 fraction bits)
// The digits of the FP64-accurate kernels: |v| < 2^(E - 1022) in fixed point
// with 55 fraction bits (a value within two binades of its group's largest
// keeps all 53 bits of its significand; smaller ones are truncated), cut into
// seven balanced digits: of the magnitude, the top one in [0, 128], the others
// in [-128, 127], then all with the value's sign.  With the levels 0-7 of
// the digit products a product of two values is off by at most ~2^-54 of the
// product of their groups' scales, one rounding of FP64.
//
// The integer (ALU) pipe issues at half the rate of the FMA pipe and is the
// busiest of these kernels (52 to 54%): hence the truncation, the sign applied by
// the packed FMA that also takes the bias out of the digits, and the constant byte in
// the fixed point word that one byte permutation turns into fp16 numbers.
#define OZ8_S 7
#define OZ8_F 55

// the exponent word to hand to oz8_fixed (a group of zeros, E = 0, cuts to 0)
static __device__ __forceinline__ uint32_t oz8_scale(int E)
{
  return E ? ((uint32_t)E << 20) | 0xFFFFFu : 0xFFFFFFFFu;
}

// The exponent word the kernels keep of a group: its largest biased exponent E,
// or OZ8_UNSAFE when the digits cannot carry it: infinities or NaN (2047), or
// only values so small (below 2^-960) that subnormals would matter; 0: zeros
#define OZ8_UNSAFE 0x10000
static __device__ __forceinline__ int oz8_code(int E) { return E == 2047 || (E != 0 && E < 64) ? OZ8_UNSAFE : E; }
// the sum of two groups' words: products that the fast conversion can scale from
// |T| >= 2^32 on (also at the weight 2^-56 of a Gram's last row block) without
// leaving FP64's normal range
static __device__ __forceinline__ bool oz8_ordinary(int e2) { return (unsigned)(e2 - 1120) <= 1900u; }
// products to be summed with FP64 FMAs: unusable digits, or so small that the
// roundings of subnormal sums would show (above the ordinary range the general
// conversion is right)
static __device__ __forceinline__ bool oz8_direct(int ex, int ey)
{
  return ((ex | ey) & OZ8_UNSAFE) || (ex && ey && ex + ey < 1120);
}

// |v| (v's bits hi:lo) in fixed point against its group's scale, as the bytes
// digit 0, digits 1-6 + 128 (from the top down, below a byte 0x64)
static __device__ __forceinline__ void oz8_fixed(uint32_t lo, uint32_t hi, uint32_t es, uint32_t& vlo, uint32_t& vhi)
{
  const uint32_t sh = min((es - (hi & 0x7FFFFFFFu)) >> 20, 63u);  // 55 bits >> 63 = 0: far below the scale
  const uint32_t mh = (hi & 0xFFFFFu) | 0x100000u;
  const uint64_t m = ((uint64_t)__funnelshift_l(lo, mh, 2) << 32) | (lo << 2);
  const uint64_t v = (m >> sh) + 0x6400808080808080ull;
  vlo = (uint32_t)v;
  vhi = (uint32_t)(v >> 32);
}

static __device__ __forceinline__ uint32_t oz8_hfma2(uint32_t a, uint32_t b, uint32_t c)
{
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
static __device__ __forceinline__ uint32_t oz8_hmul2(uint32_t a, uint32_t b)
{
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// the fp16 digits of two values (fixed point words a, b of oz8_fixed; ha, hb
// the values' high words): d[t] holds digit t of both.  0x6400 | f is the fp16
// 1024 + f; (1024 + f) s - (1024 + bias) s = s (f - bias) exactly.
static __device__ __forceinline__ void oz8_digits2(uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi, uint32_t ha,
                                                   uint32_t hb, uint32_t (&d)[OZ8_S])
{
  const uint32_t s = (__byte_perm(ha, hb, 0x7632) & 0x80008000u) | 0x3C003C00u;  // +-1
  const uint32_t c0 = oz8_hmul2(s, 0xE400E400u), c = oz8_hmul2(s, 0xE480E480u);    // -1024 s, -1152 s
  const uint32_t al = (alo & 0x00FFFFFFu) | 0x64000000u, bl = (blo & 0x00FFFFFFu) | 0x64000000u;
  d[0] = oz8_hfma2(__byte_perm(ahi, bhi, 0x7632), s, c0);
  d[1] = oz8_hfma2(__byte_perm(ahi, bhi, 0x7531), s, c);
  d[2] = oz8_hfma2(__byte_perm(ahi, bhi, 0x7430), s, c);
  d[3] = oz8_hfma2((__byte_perm(alo, blo, 0x0703) & 0x00FF00FFu) | 0x64006400u, s, c);
  d[4] = oz8_hfma2(__byte_perm(al, bl, 0x7632), s, c);
  d[5] = oz8_hfma2(__byte_perm(al, bl, 0x7531), s, c);
  d[6] = oz8_hfma2(__byte_perm(al, bl, 0x7430), s, c);
}

// the digits of eight values: pk[t][k] holds digit t of values 2k and 2k + 1
static __device__ __forceinline__ void oz8_digits8(const uint32_t* lo, const uint32_t* hi, uint32_t es,
                                                   uint32_t (&pk)[OZ8_S][4])
{
#pragma unroll
  for (int k = 0; k < 4; k++) {
    uint32_t al, ah, bl, bh, d[OZ8_S];
    oz8_fixed(lo[2 * k], hi[2 * k], es, al, ah);
    oz8_fixed(lo[2 * k + 1], hi[2 * k + 1], es, bl, bh);
    oz8_digits2(al, ah, bl, bh, hi[2 * k], hi[2 * k + 1], d);
#pragma unroll
    for (int t = 0; t < OZ8_S; t++) pk[t][k] = d[t];
  }
}

// the magnitudes of the top digits of eight values (their four words), and these
// added up into two FP16 numbers: integers, exact up to 2048
static __device__ __forceinline__ uint32_t oz8_hadd2(uint32_t a, uint32_t b)
{
  uint32_t d;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
static __device__ __forceinline__ uint32_t oz8_magnitudes(const uint32_t (&d)[4], uint32_t (&m)[4])
{
#pragma unroll
  for (int k = 0; k < 4; k++) m[k] = d[k] & 0x7FFF7FFFu;
  return oz8_hadd2(oz8_hadd2(m[0], m[1]), oz8_hadd2(m[2], m[3]));
}
static __device__ __forceinline__ float oz8_both(uint32_t h2)
{
  float lo, hi;
  asm("{\n .reg .b16 l, h;\n mov.b32 {l, h}, %2;\n cvt.f32.f16 %0, l;\n cvt.f32.f16 %1, h;\n}\n"
      : "=f"(lo), "=f"(hi)
      : "r"(h2));
  return lo + hi;
}

// The exact integer T = sum_L S_L 256^(7 - L) of the eight level sums, in
// units of 2^15 (rounded once, at 2^-55 of the scales' product): |S_0..3| <=
// 2^22, the others up to 2^23.  FP32 to integer by adding 1.5 2^23 (exact to
// 2^22); the larger levels 4-6 by adding 1.5 2^24, which gives the nearest even
// integer, the odd unit left over moving down a level as 256; of level 7 only
// the leading bits count.  (Conversion instructions run at a sixteenth of the
// additions' rate.)  The product of the two values is T 2^(Ex + Ey - 2099).
//
// Factors are below 1 but for a top digit rounded up to 128 (and, where the
// slices of a row block are 0 and 4, the digit 4 beside it), so that R rows or
// columns give |T| < R 2^55 (1 + 2^-32): 2^62 and a little for the 64 columns of
// an update and the 128 rows of a Gram group, but just above 2^63 for 256 rows of
// values next to a power of two.  HALF drops a bit of T for those (the product is
// T 2^(Ex + Ey - 2098)); the one-instruction normalisation of oz8_scaled_fast
// needs |T| < 2^63 too.
#define OZ8_BASE 2099
template <bool HALF>
static __device__ __forceinline__ long long oz8_combine(uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3,
                                                        uint32_t s4, uint32_t s5, uint32_t s6, uint32_t s7)
{
  const float m23 = 12582912.0f, m24 = 25165824.0f;
  const uint32_t b23 = 0x4B400000u, b24 = 0x4BC00000u;
  const uint32_t i0 = __float_as_uint(__fadd_rn(__uint_as_float(s0), m23));
  const uint32_t i1 = __float_as_uint(__fadd_rn(__uint_as_float(s1), m23));
  const uint32_t i2 = __float_as_uint(__fadd_rn(__uint_as_float(s2), m23));
  const uint32_t i3 = __float_as_uint(__fadd_rn(__uint_as_float(s3), m23));
  const float f4 = __uint_as_float(s4);
  const float y4 = __fadd_rn(f4, m24);
  const float f5 = fmaf(__fsub_rn(f4, __fsub_rn(y4, m24)), 256.0f, __uint_as_float(s5));
  const float y5 = __fadd_rn(f5, m24);
  const float f6 = fmaf(__fsub_rn(f5, __fsub_rn(y5, m24)), 256.0f, __uint_as_float(s6));
  const uint32_t i6 = __float_as_uint(__fadd_rn(f6, m24));
  const uint32_t i7 = __float_as_uint(__fadd_rn(__uint_as_float(s7), m24));
  const int a0 = (int)(i0 * 256u + i1 - b23 * 257u);
  const int a1 = (int)(i2 * 256u + i3 - b23 * 257u);
  const int a4 = (int)(__float_as_uint(y4) - b24), a5 = (int)(__float_as_uint(y5) - b24);
  const int a6 = (int)(i6 * 256u + i7 - b24 * 257u + 8192u) >> 14;
  const long long t = (long long)a1 * 131072 + ((long long)a4 * 1024 + (long long)(a5 * 4 + a6));
  // (an odd t to the even half: always up, the sums over many groups drifted)
  return HALF ? ((t + ((t >> 1) & 1)) >> 1) + ((long long)a0 << 32) : t + ((long long)a0 << 33);
}

// FP64 nearest to T 2^base, |T| < 2^63, from integer operations only (ties
// away from zero): the FP64 pipe's conversion of a 64-bit integer takes longer
// than all of these.  Fast form: |T| >= 2^32 and an ordinary sum of exponents.
static __device__ __forceinline__ double oz8_scaled_fast(long long T, int base)
{
  const uint64_t sg = (uint64_t)(T >> 63);
  const uint64_t A = ((uint64_t)T ^ sg) - sg;
  const uint32_t ah = (uint32_t)(A >> 32), al = (uint32_t)A;
  uint32_t p;  // A's leading bit is 32 + p
  asm("bfind.u32 %0, %1;" : "=r"(p) : "r"(ah));
  const uint32_t ls = 30u - p;
  const uint64_t m = ((((uint64_t)__funnelshift_l(al, ah, ls) << 32) | (al << ls)) + 0x200u) >> 10;
  const uint32_t rh = (uint32_t)(m >> 32) + (uint32_t)((int)p + base + 1054) * 0x100000u;
  return __hiloint2double((int)(rh | ((uint32_t)sg & 0x80000000u)), (int)(uint32_t)m);
}
// any T and base: below the normal range 0, above it infinity
static __device__ __noinline__ double oz8_scaled(long long T, int base)
{
  if (T == 0) return 0.0;
  const uint64_t A = T < 0 ? (uint64_t)0 - (uint64_t)T : (uint64_t)T;
  const int lz = __clzll((long long)A);  // >= 1
  const uint64_t m = ((A << (lz - 1)) + 0x200u) >> 10;
  const int e = 1085 - lz + base;  // biased exponent less 1
  uint64_t bits = m + ((uint64_t)(uint32_t)e << 52);
  if ((unsigned)e >= 2046u) bits = e > 0 ? 0x7FF0000000000000ull : 0ull;
  return __longlong_as_double((long long)(bits | ((uint64_t)T & 0x8000000000000000ull)));
}
// instruction descriptor of tcgen05.mma.kind::f16: D = F32, A = B = FP16,
// both K-major, M x N (type code 0)
static __host__ __device__ constexpr uint32_t f16_idesc(int M, int N)
{
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
