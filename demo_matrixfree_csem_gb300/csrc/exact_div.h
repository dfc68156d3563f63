// Correctly rounded complex128 quotients by integer arithmetic.
//
// The complex128 kernels give the reference's results bit for bit, so each of their
// divisions has to be the IEEE quotient rounded to nearest. GB300 issues two FP64
// operations per SM and cycle (one warp instruction in 16 cycles, measured: 523 G add, mul
// or fma per second), and an IEEE division costs 7 of them, 20 when a numerator is zero
// (73 and 26 G per second measured), while the integer units stand idle. So a quotient
// a / d whose divisor is known beforehand is formed on the integer units, about 35
// instructions and no FP64 operation:
//
//   with the 53-bit integer significands ma and md of a and d, and R = floor(2^116 / md)
//   (one 64-bit word per divisor), h = floor(2^11 ma R / 2^64) is at most 2 below
//   2^63 ma / md. Its upper 53 bits are the quotient's significand q rounded down, or one
//   less (then the true quotient exceeds q + 1 by less than 2^-8); the remainder
//   r = ma 2^s - q md is exact in 64 bits, and q is rounded up where 2 r > md (2 r = md
//   would be a tie, which a quotient of two 53-bit significands never is).
//
// The range is limited so that no exponent leaves the normal numbers; zero numerators are
// taken through; for everything else (subnormals, infinities, NaN, exponents beyond the
// range) `bad` is set and the caller repeats the point with the / operator.
#pragma once
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define CSEM_HD __host__ __device__ __forceinline__
#else
#define CSEM_HD static inline
#endif

namespace csem {

// numerators and divisors whose exponent fields lie in [XD_LO, XD_HI) keep the quotient
// normal: 2^+-383 over 2^+-383
constexpr uint32_t XD_LO = 640u << 20, XD_HI = 1407u << 20;

CSEM_HD uint64_t xd_bits(double a)
{
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(a);
#else
  uint64_t u;
  memcpy(&u, &a, 8);
  return u;
#endif
}

CSEM_HD double xd_double(uint64_t u)
{
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double a;
  memcpy(&a, &u, 8);
  return a;
#endif
}

CSEM_HD uint64_t xd_mulhi(uint64_t a, uint64_t b)
{
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

CSEM_HD bool xd_in_range(uint32_t hi) { return (hi & 0x7fffffffu) - XD_LO < XD_HI - XD_LO; }

// R of a divisor: floor(2^116 / md), all ones for a power of two (2^64 - 1 for 2^64, which
// the bounds above allow); 0 for a divisor outside the range
inline uint64_t xd_recip(double d)
{
  const uint64_t u = xd_bits(d);
  if (!xd_in_range((uint32_t)(u >> 32))) return 0;
  const uint64_t m = (u & 0xfffffffffffffull) | (1ull << 52);
  if (m == 1ull << 52) return ~0ull;
#ifdef __CUDA_ARCH__
  return 0;  // made on the host only
#else
  return (uint64_t)((((unsigned __int128)1) << 116) / m);
#endif
}

// a / d for a divisor d > 0 in range with R = xd_recip(d)
CSEM_HD double xd_div(double a, double d, uint64_t R, uint32_t& bad)
{
  const uint64_t u = xd_bits(a), v = xd_bits(d);
  const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u, dh = (uint32_t)(v >> 32);
  const uint64_t ma = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
  const uint64_t md = ((uint64_t)((dh & 0xfffffu) | 0x100000u) << 32) | (uint32_t)v;
  const uint64_t h = xd_mulhi(ma << 11, R);
  const uint32_t top = (uint32_t)(h >> 63);  // 1: ma >= md, the quotient's leading bit is bit 63
  const uint64_t q = h >> (10 + top);
  const uint64_t r = ((uint64_t)(lo << (21 - top)) << 32) - q * md;  // ma 2^(53 - top) - q md, exact
  const uint64_t qr = q + (r > (md >> 1) ? 1 : 0);
  // exponent field of the quotient less one (q's leading bit adds it), a's sign kept
  const uint32_t e = (hi & 0xfff00000u) - (dh & 0x7ff00000u) + (1021u << 20) + (top << 20);
  const uint64_t res = qr + ((uint64_t)e << 32);
  const bool zero = ((hi << 1) | lo) == 0;
  bad |= (zero || xd_in_range(hi)) ? 0u : 1u;
  return zero ? a : xd_double(res);
}

// The same for a divisor that is only known now, of either sign: R by Newton's iteration on
// integers, from a single precision reciprocal (23 bits; 44 after one step, 60 after two). q is
// off by at most one either way, and the remainder is signed. 30 integer instructions; the FP64
// unit's own reciprocal costs it 9 operations, in a chain.
struct XdDen {
  double d;
  uint64_t R;
};
CSEM_HD XdDen xd_den(double d, uint32_t& bad)
{
  XdDen n;
  n.d = d;
  const uint64_t u = xd_bits(d);
  const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u;
  bad |= xd_in_range(hi) ? 0u : 1u;
  const uint64_t D = (((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | lo) << 11;  // 2^63 times 1 <= d' < 2
  const uint32_t f = 0x3f800000u | (hi & 0xfffffu) << 3 | lo >> 29;
#ifdef __CUDA_ARCH__
  float r = __fdividef(1.f, __uint_as_float(f));
  r = fminf(fmaxf(r, 0.5f), 0.99999994f);
  const uint32_t x = (__float_as_uint(r) << 8) | 0x80000000u;  // 2^32 / d'
#else
  float g, r;
  memcpy(&g, &f, 4);
  r = 1.f / g;
  r = r < 0.5f ? 0.5f : (r > 0.99999994f ? 0.99999994f : r);
  uint32_t x;
  memcpy(&x, &r, 4);
  x = (x << 8) | 0x80000000u;
#endif
  // y ~ 2^63 / d', and 2^62 - D y / 2^64 the error times 2^62
  uint64_t y = (uint64_t)x << 31;
  const int64_t e = (int64_t)(1ull << 62) - (int64_t)xd_mulhi(D, y);  // below 2^41 in size
  y += (uint64_t)(((int64_t)x * (int32_t)(e >> 10)) >> 21);
  const int64_t e1 = (int64_t)(1ull << 62) - (int64_t)xd_mulhi(D, y);  // below 2^20
  y += (uint64_t)(((int64_t)(uint32_t)(y >> 32) * (int32_t)e1) >> 30);
  n.R = (u << 12) == 0 || y >> 63 ? ~0ull : y << 1;
  return n;
}
CSEM_HD double xd_div2(double a, double d, uint64_t R, uint32_t& bad)
{
  const uint64_t u = xd_bits(a), v = xd_bits(d);
  const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u, dh = (uint32_t)(v >> 32);
  const uint64_t ma = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
  const uint64_t md = ((uint64_t)((dh & 0xfffffu) | 0x100000u) << 32) | (uint32_t)v;
  const uint64_t h = xd_mulhi(ma << 11, R);
  const uint32_t top = (uint32_t)(h >> 63);
  const uint64_t q = h >> (10 + top);
  const int64_t r = (int64_t)(((uint64_t)(lo << (21 - top)) << 32) - q * md);
  // q + n with n = round(r / md): r / md lies in (-1.1, 2.1), ties excluded as above
  const int64_t hmd = (int64_t)(md >> 1);
  const uint64_t qr = q + (r > hmd ? 1 : 0) + (r - (int64_t)md > hmd ? 1 : 0) - (r < -hmd ? 1 : 0);
  const uint32_t e = ((hi ^ (dh & 0x80000000u)) & 0xfff00000u) - (dh & 0x7ff00000u) + (1021u << 20) + (top << 20);
  const uint64_t res = qr + ((uint64_t)e << 32);
  const bool zero = ((hi << 1) | lo) == 0;
  bad |= (zero || xd_in_range(hi)) ? 0u : 1u;
  return zero ? a : xd_double(res);
}

}  // namespace csem
