// Device helpers shared by the quantisation kernels: packed absmax, the exact per-token scale and the division-free
// quantisation of a 16-byte chunk.
//
// Arithmetic contract (bit-exact with torch on CPU; deploy/int8_exec.py:508-509 and :83-101):
//   scale = max(absmax, 1e-8) / 127        IEEE fp32 division
//   q     = round_half_even(x / scale)     IEEE fp32 division, clamp to [-127, 127]
#pragma once
#include "common.cuh"

namespace pq {
namespace {

// Running maximum of |x| over packed 16-bit floats, kept as two packed magnitudes.  Clearing the sign bits leaves
// non-negative bf16 / fp16 bit patterns, whose order as unsigned 16-bit integers is their order as numbers, so the
// maximum is an integer one: two masked words and the running value per three-input halfword maximum.  (The
// floating-point packed abs / max instructions of these types issue on the slow special-function pipe.)
template <typename T>
__device__ __forceinline__ uint32_t absmax_chunk(uint32_t acc, const uint4& v) {
  constexpr uint32_t kMag = 0x7FFF7FFFu;
  acc = __vimax3_u16x2(acc, v.x & kMag, v.y & kMag);
  acc = __vimax3_u16x2(acc, v.z & kMag, v.w & kMag);
  return acc;
}

// Quantisation of one 16-byte chunk (8 elements) to 8 int8 codes (two 32-bit words).
//
// Exact contract: code = round_half_even(fl(x / scale)) with the IEEE quotient.  With inv = fl(1 / scale) correctly
// rounded, q0 = fl(x * inv), the residual r = fl(x - q0 * scale) and q = fl(q0 + r * inv) give the correctly rounded quotient
// (Markstein's correction step) short of underflow, where the code is 0 either way; adding 1.5 * 2^23 rounds it to the
// nearest integer, half to even, and leaves that integer in the low mantissa bits.  The tests compare the codes with the
// division's for every significand of the absmax and every value of the type that can give a code other than 0: no difference.
// (Not finite: the residual of absmax / 127 is inf - inf, so a row with an infinity gets scale NaN and every code is the low byte
// of a NaN, -1.)
// Four packed operations per pair of elements and no branch.  (Bracketing the quotient between two products and redoing
// a chunk with divisions when they disagree costs the same four operations, but every |x| = absmax / 2 is a rounding tie
// and took that path: a third of all warp-wide chunks of normally distributed bf16 data.)  No conversion instructions
// are used: those run on a slow pipe.  Codes never leave [-127, 127] because |x| <= absmax.
struct QuantScale {
  float scale;       // absmax / 127 (or the 1e-8 floor / 127)
  float inv;         // 1 / scale
};
__device__ __forceinline__ QuantScale make_quant_scale(float amax) {
  QuantScale qs;
  // absmax / 127, correctly rounded, without the generic division routine: quotient estimate with the rounded
  // reciprocal, exact residual, one correction.  absmax is a bf16 or fp16 value (or the 1e-8 floor): the sequence
  // was checked against the IEEE quotient for every such value on the host and is checked again for all of them
  // on the device by the tests.
  const float a = fmaxf(amax, 1e-8f);
  const float r127 = 0.007874015718698502f;           // RN(1/127)
  const float q0 = __fmul_rn(a, r127);
  const float rem = __fmaf_rn(-q0, 127.0f, a);
  qs.scale = __fmaf_rn(rem, r127, q0);
  qs.inv = __frcp_rn(qs.scale);                        // correctly rounded reciprocal = IEEE 1 / scale
  return qs;
}

template <typename T>
__device__ __forceinline__ float2 unpack2(uint32_t w) {
  T tag{};
  return make_float2(lo_f32(w, tag), hi_f32(w, tag));
}

template <typename T>
__device__ __forceinline__ void quant_chunk(const uint4& v, const QuantScale& qs, uint32_t& lo, uint32_t& hi) {
  const float2 magic = make_float2(12582912.0f, 12582912.0f);
  const float2 inv = make_float2(qs.inv, qs.inv), neg_scale = make_float2(-qs.scale, -qs.scale);
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint32_t m[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = unpack2<T>(w[i]);
    const float2 q0 = __fmul2_rn(f, inv);
    const float2 r = __ffma2_rn(q0, neg_scale, f);
    const float2 q = __fadd2_rn(__ffma2_rn(r, inv, q0), magic);
    m[2 * i] = __float_as_uint(q.x); m[2 * i + 1] = __float_as_uint(q.y);
  }
  // low bytes of the eight integers -> two words
  lo = __byte_perm(__byte_perm(m[0], m[1], 0x0040), __byte_perm(m[2], m[3], 0x0040), 0x5410);
  hi = __byte_perm(__byte_perm(m[4], m[5], 0x0040), __byte_perm(m[6], m[7], 0x0040), 0x5410);
}

template <typename T>
__device__ __forceinline__ float amax_of_packed(uint32_t acc) {
  T tag{};
  return fmaxf(lo_f32(acc, tag), hi_f32(acc, tag));
}

}  // namespace
}  // namespace pq
