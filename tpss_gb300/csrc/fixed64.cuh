// fixed64.cuh -- 64-bit contractions on the integer pipe.
//
// GB300 issues 2 FP64 multiply-adds per clock and SM but 27 32 x 32 + 64 bit integer ones
// (IMAD.WIDE; both measured on all SMs in 5 x 5 pairs of contractions, the pipe's limit is 32), and
// three of these do the product of an FP64 multiply-add to 58 bits: 17.6 clocks per warp and value
// of such a contraction against 81. The kernels that include this file keep the values of a block (a patch, a
// cell) as 64-bit integers with one exponent per block (block floating point):
//   value = x 2^e,  |x| < 2^59,  coefficient = c 2^-F,  sum_j |c_ij| <= 2^62 in every row i.
// With signed 32-bit limbs x = xh 2^32 + xl, c = ch 2^32 + cl (xl, cl in [-2^31, 2^31)) a row's
// sum is  sum_j c_ij x_j / 2^64 = sum ch xh + (sum ch xl + cl xh) / 2^32 + sum cl xl / 2^64:
// three IMAD.WIDE per product without the last sum, four with it, and the accumulators cannot overflow
// (|sum ch xh| < 2^60, |sum ch xl + cl xh| < 2^63 for up to 16 terms).
//
// Error of a row of n terms, in units 2^(e+64-F): 1/2 from the rounding, and without the low products up to n/4
// (each is a quarter unit at most; random rows of 5 to 16 terms are off by 1.2 to 1.4 at worst). The largest
// |x| is 2^58 units and more, a row sum of |c| 2^61 to 2^62 (of the largest row), so that this is (n + 2) 2^-57 at most
// of (largest row sum of |c|) x (largest |x| of the block). An FP64 chain makes up to n 2^-53 sum_j |c_ij x_j|. The two
// differ in kind: this one is relative to the block's largest value and the matrix' largest row, and beats FP64's where all of a
// block's values enter a row with coefficients of one magnitude. So a block holds no values that its rows do not contract,
// and the C0IP bands, whose coefficients differ by up to 1e5, and the transfers keep the low products (LOW).
// After every contraction the block is shifted up again to 59 bits by the headroom its largest value leaves.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace tpss
{
namespace fx
{
// Exponents of a block's largest value that the kernels cover whose matrices have entries within 2^(+-kTableRange): a
// result's unit 2^(e - 58 + 64 - F), |F - 62| <= kTableRange, stays a normal number
constexpr int kRange = 800, kTableRange = 150;

// 64-bit accumulator of 32 x 32-bit products. add() is one IMAD.WIDE: it is written with the carry
// flag because ptxas splits the accumulation of mad.wide chains into products and separate 64-bit
// additions (43 instead of 30 instructions per value of a 5 x 5 pair of contractions, 19.6 instead of
// 17.6 clocks per warp)
struct Acc
{
  unsigned lo;
  int hi;
  __device__ __forceinline__ explicit Acc(unsigned l = 0) : lo(l), hi(0) {}
  __device__ __forceinline__ void add(int a, int b)
  {
    asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\tmadc.hi.s32 %1, %2, %3, %1;" : "+r"(lo), "+r"(hi) : "r"(a), "r"(b));
  }
  // the first product of a sum (from a zero accumulator add() would be two instructions)
  __device__ __forceinline__ void start(int a, int b)
  {
    asm("{.reg .b64 t;\n\tmul.wide.s32 t, %2, %3;\n\tmov.b64 {%0, %1}, t;}" : "=r"(lo), "=r"(hi) : "r"(a), "r"(b));
  }
  __device__ __forceinline__ int64_t value() const { return (int64_t)((uint64_t)(unsigned)hi << 32 | lo); }
};

__device__ __forceinline__ int hi32(int64_t x) { return (int)(x >> 32); }

// signed limbs of x
__device__ __forceinline__ void split(int64_t x, int &h, int &l)
{
  l = (int)x;
  h = (int)(x >> 32) + (int)((unsigned)l >> 31);
}

// x >> s and x << s with s >= 64 giving 0 (or the sign): PTX clamps the amounts
__device__ __forceinline__ uint64_t shr_u(uint64_t x, int s)
{
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
  return r;
}
__device__ __forceinline__ int64_t shr_s(int64_t x, int s)
{
  int64_t r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
  return r;
}
__device__ __forceinline__ int64_t shl(int64_t x, int s)
{
  int64_t r;
  asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
  return r;
}
// x 2^s for either sign of s (|x| 2^s must fit)
__device__ __forceinline__ int64_t shift(int64_t x, int s) { return shr_s(shl(x, max(s, 0)), max(-s, 0)); }

// bits of |x| in the high word (|x| or |x| - 1): ORed over a block, their highest set bit gives the
// block's headroom
__device__ __forceinline__ unsigned mag_hi(int64_t x)
{
  const int h = (int)(x >> 32);
  return (unsigned)(h ^ (h >> 31));
}

// shift that brings a block whose high-word magnitudes OR to m (< 2^27) to 59 bits
__device__ __forceinline__ int headroom(unsigned m) { return __clz(m | 1u) - 5; }

// double -> integer with unit 2^(emax - 1023 - 58), emax the block's largest biased exponent
// (truncated toward zero beyond the 59 bits; zeros and denormals give 0 for emax >= 64)
__device__ __forceinline__ int64_t from_double(double v, int emax)
{
  const int hi = __double2hiint(v);
  const unsigned lo = (unsigned)__double2loint(v);
  const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
  const int e = (int)(((unsigned)hi >> 20) & 0x7ffu);
  const uint64_t m = (((uint64_t)mh << 32) | lo) << 6;
  const int64_t a = (int64_t)shr_u(m, emax - e);
  const int64_t s = (int64_t)(hi >> 31);
  return (a ^ s) - s;
}

// y 2^ex as a double (ex keeps the result in the normal range). The conversion instruction is an FP64
// one (64 clocks of a warp's FP64 pipe); to_double_alu does it in about 20 integer operations (40
// clocks of another pipe), rounding half up. Kernels split their results between the two.
__device__ __forceinline__ double to_double(int64_t y, int ex)
{
  const double d = __ll2double_rn(y);
  const int hi = y == 0 ? 0 : __double2hiint(d) + ex * (1 << 20);
  return __hiloint2double(hi, __double2loint(d));
}

__device__ __forceinline__ double to_double_alu(int64_t y, int ex)
{
  const int64_t s = y >> 63;
  const uint64_t a = (uint64_t)((y ^ s) - s);
  const int up = __clzll((long long)a) - 1;  // leading bit to bit 62
  const uint64_t m = ((a << (up & 63)) + 0x200) >> 10;  // leading bit at 52, or 53 after a carry
  const int hi = (int)(m >> 32) + ((ex + 1084 - up) << 20);
  return a == 0 ? 0.0 : __hiloint2double(hi | (int)((unsigned)(s >> 32) & 0x80000000u), (int)m);
}

// 2^e as a double, e in [-1022, 1023]
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }

// positive normal double r = m 2^q with 2^60 <= m < 2^61, m in signed limbs
__device__ __forceinline__ void split_positive(double r, int &mh, int &ml, int &q)
{
  const int hi = __double2hiint(r);
  const unsigned lo = (unsigned)__double2loint(r);
  const uint64_t m = (((uint64_t)(((unsigned)hi & 0xfffffu) | 0x100000u) << 32) | lo) << 8;
  split((int64_t)m, mh, ml);
  q = (int)((unsigned)hi >> 20) - 1023 - 60;
}

// 1/d = m 2^q with 2^60 <= m <= 2^61, in the form of split_positive: Newton's iteration r <- r + r (1 - d r) from a
// single-precision start, twice (24 to 48 to 61 bits). An FP64 division keeps a warp's FP64 pipe busy for
// some 10 instructions of 64 clocks (Richardson step on 20^3 distorted cells, k = 3: 432 -> 424 us). What is not in (2^-900, 2^900) is divided in FP64.
__device__ __forceinline__ void reciprocal(double d, int &mh, int &ml, int &q)
{
  const int hi = __double2hiint(d), e = hi >> 20;
  if(e < 1023 - 900 || e > 1023 + 900)
  {
    split_positive(1.0 / d, mh, ml, q);
    return;
  }
  // d = x 2^(e - 1022), x = D / 2^64 in [1/2, 1); r in units of 2^-61
  const uint64_t D = (((uint64_t)(((unsigned)hi & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(d)) << 11;
  const float x = (float)(unsigned)(D >> 32) * 0x1p-32f;
  int64_t r = (int64_t)(unsigned)(__frcp_rn(x) * 0x1p23f) << 38;
#pragma unroll
  for(int i = 0; i < 2; ++i)
  {
    const int64_t rest = (int64_t)(1ull << 61) - (int64_t)__umul64hi(D, (uint64_t)r);
    r += __mul64hi(r, rest << 3);
  }
  split(r >> 1, mh, ml);
  q = -60 - (e - 1022);
}

// x m / 2^61 (|x| < 2^60, m as above): |result| <= |x|, error below 3 units
__device__ __forceinline__ int64_t mul_m61(int64_t x, int mh, int ml)
{
  int xh, xl;
  split(x, xh, xl);
  Acc M(1u << 28), S;
  M.add(xl, mh);
  M.add(xh, ml);
  S.start(xh, mh);
  return (S.value() << 3) + (M.value() >> 29);
}

// ---- coefficient rows: int2 (x: low limb, y: high limb), read as pairs
// sum_j c_j x_j / 2^64 of one row of H coefficients for the first H of L values x in limbs. LOW: with the
// products of the low limbs, less their last 4 bits, so that up to 31 terms fit
template<int H, bool LOW = false, int L>
__device__ __forceinline__ int64_t row_dot(const int2 *__restrict__ row, const int (&xh)[L], const int (&xl)[L])
{
  Acc M, S, Q;
  const int4 *row4 = reinterpret_cast<const int4 *>(row);
#pragma unroll
  for(int j2 = 0; j2 < (H + 1) / 2; ++j2)
  {
    const int4 c = row4[j2];
    if constexpr(LOW)
    {
      if(j2 == 0) Q.start(c.x, xl[0] >> 4);
      else Q.add(c.x, xl[2 * j2] >> 4);
    }
    if(j2 == 0) M.start(c.y, xl[0]);
    else M.add(c.y, xl[2 * j2]);
    M.add(c.x, xh[2 * j2]);
    if(j2 == 0) S.start(c.y, xh[0]);
    else S.add(c.y, xh[2 * j2]);
    if(2 * j2 + 1 < H)
    {
      const int j = 2 * j2 + 1 < H ? 2 * j2 + 1 : 0;
      if constexpr(LOW) Q.add(c.z, xl[j] >> 4);
      M.add(c.w, xl[j]);
      M.add(c.z, xh[j]);
      S.add(c.w, xh[j]);
    }
  }
  // rounded to the nearest unit from M's low word (which also keeps its last product one instruction)
  if constexpr(LOW) return S.value() + ((M.value() + (Q.value() >> 28) + (1ll << 31)) >> 32);
  else return S.value() + (M.hi + (int)(M.lo >> 31));
}
}  // namespace fx
}  // namespace tpss
