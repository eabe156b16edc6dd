// terms.cuh -- DFT terms in pairs: the unmasked instances of both tiled kernels and the
// reconstruction's REF instance.
#pragma once
#include "viss_internal.cuh"

namespace viss {

// Two FP32 values in one 64-bit register pair; sm_103a's packed operations round each half as
// the single ones do.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// sin and cos of two angles (half a turn added), weighted into packed sums.
__device__ __forceinline__ void sincos2(f32x2 x, f32x2 c, f32x2& fr, f32x2& fi) {
  float xa, xb, sa, ca, sb, cb;
  unpack2(x, xa, xb);
  __sincosf(xa, &sa, &ca);
  __sincosf(xb, &sb, &cb);
  fr = fma2(c, pack2(ca, cb), fr);
  fi = fma2(c, pack2(sa, sb), fi);
}

// Two terms without the SFU, for phases that are all fixed point (integer uvw): the top bit of
// the phase (shifted by a quarter turn) is the sign of the term, the next 23 bits the
// angle r in half turns, |r| <= 1/2, and sin(pi r) and cos(pi r) are polynomials in r^2 (least
// maximum error by iteratively reweighted least squares; in FP32 they are off by 6e-8 rms,
// the SFU's values with their angle by 2.6e-7).
constexpr uint32_t POLY_BIAS = 128u + 0xC0000000u - (uint32_t)PHASE_BIAS;  // on top of the phase bias
__device__ __forceinline__ void poly2(uint32_t qa, uint32_t qb, f32x2 c, f32x2& fr, f32x2& fi) {
  qa += POLY_BIAS;
  qb += POLY_BIAS;
  // bit 23 of q >> 8 falls on a bit that is set in 1.0f
  const f32x2 r = add2(pack2(__uint_as_float((qa >> 8) | 0x3f800000u), __uint_as_float((qb >> 8) | 0x3f800000u)),
                       pack2(-1.5f, -1.5f));
  float ca, cb;
  unpack2(c, ca, cb);
  const f32x2 cs = pack2(__uint_as_float(__float_as_uint(ca) ^ (qa & 0x80000000u)),
                         __uint_as_float(__float_as_uint(cb) ^ (qb & 0x80000000u)));
  const f32x2 y = mul2(r, r);
  f32x2 s = fma2(y, pack2(0.0772222504f, 0.0772222504f), pack2(-0.598046422f, -0.598046422f));
  f32x2 k = fma2(y, pack2(0.219696805f, 0.219696805f), pack2(-1.33188021f, -1.33188021f));
  s = fma2(y, s, pack2(2.55003166f, 2.55003166f));
  k = fma2(y, k, pack2(4.05841208f, 4.05841208f));
  s = fma2(y, s, pack2(-5.16770697f, -5.16770697f));
  k = fma2(y, k, pack2(-4.934793f, -4.934793f));
  s = fma2(y, s, pack2(3.1415925f, 3.1415925f));
  k = fma2(y, k, pack2(0.99999994f, 0.99999994f));
  fr = fma2(cs, k, fr);
  fi = fma2(cs, mul2(r, s), fi);
}

// Two of the thread's terms: fixed-point coordinates A, B, C and FP32 ones X, Y, Z (lo: lx, ly, lz) of
// its two rows or pixels against the other side's, which stand in shared memory: s = {A, B, C, -}
// and the FP32 parts twice, {x, x, y, y}, {z, z, c, c}, as packed operands.  bias: the row's,
// one for each term.  POLY: without the SFU (integer uvw only).
template <bool FRAC, bool COMP, bool POLY>
__device__ __forceinline__ void term2(const int4& s, const ulonglong2& sxy, f32x2 sz, const float4& slo, f32x2 c, const int* A,
                                      const int* B, const int* C, int bias0, int bias1, f32x2 X, f32x2 Y, f32x2 Z,
                                      f32x2 lx, f32x2 ly, f32x2 lz, f32x2& fr, f32x2& fi) {
  const uint32_t q[2] = {(uint32_t)s.x * (uint32_t)A[0] + (uint32_t)s.y * (uint32_t)B[0] + (uint32_t)s.z * (uint32_t)C[0] +
                             (uint32_t)bias0,
                         (uint32_t)s.x * (uint32_t)A[1] + (uint32_t)s.y * (uint32_t)B[1] + (uint32_t)s.z * (uint32_t)C[1] +
                             (uint32_t)bias1};
  if (POLY) {
    poly2(q[0], q[1], c, fr, fi);
    return;
  }
  f32x2 e = pack2(KM3PI, KM3PI);
  if (FRAC) e = fma2(sxy.x, X, fma2(sxy.y, Y, fma2(sz, Z, e)));
  if (COMP)
    e = fma2(pack2(slo.x, slo.x), lx, fma2(pack2(slo.y, slo.y), ly, fma2(pack2(slo.z, slo.z), lz, e)));
  const f32x2 f = pack2(__uint_as_float((q[0] >> 9) | 0x3f800000u), __uint_as_float((q[1] >> 9) | 0x3f800000u));
  sincos2(fma2(f, pack2(K2PI, K2PI), e), c, fr, fi);
}

}  // namespace viss
