// Row arithmetic of the bulk paths, on top of quant_row.cuh.  A header of its own because of the constant table: the modules of
// the decode step's kernels include quant_row.cuh, and while the table stood there their graphed step was 0.4 % to 2 %
// slower (22 layers of a small model: 429 against 417 us) without any of them using it.
#pragma once

#include "f32x2.cuh"
#include "quant_row.cuh"

namespace skv {

// ---- groups of eight consecutive elements per lane -----------------------------------------------------------------------
// The bulk paths (append of a prompt, rows moved by a reallocation) give a lane two such groups, so that several rows
// share a warp's instructions, and run everything per element on two elements at once (fma.rn.f32x2; element i is paired
// with i + 4) and on the multiply-add pipe: those kernels are bound by issue slots and by the half-rate integer pipe that
// compares, selects and byte permutes go through.
//   * rint(x / s) is the add of 1.5 * 2^23 inside x * (1/s) + magic, done with the reciprocal a 2^-20 too large and again
//     a 2^-20 too small.  The approximate reciprocal and the division's own rounding are off by less than 2^-22, so
//     where both give the same integer it is the rounded quotient's; the squared differences are summed and tested once
//     per lane (a NaN does not pass either).
//   * codes are joined as a polynomial in 2^bits, whose values stay below 2^17 and are therefore exact.
constexpr float kRoundMagic = 12582912.f;  // 1.5 * 2^23 = 0x4B400000

// What the arithmetic needs to know about a bucket's width, one constant load each instead of a chain of selects.
struct WidthConst {
  float levels, rlevels;  // 2^(bits-1) - 1 (at least 1) and its rounded reciprocal
  float base;             // 2^bits
  float bias;             // 2^23 + 2^(bits-1): a stored code in the significand of 2^23 minus this is the code's value
  uint32_t off;           // (2 to 4 bits) 2^(bits-1) * (1 + 2^bits + 2^2bits + 2^3bits) + the bits of kRoundMagic
  int bits;
};
static __constant__ WidthConst kWidthConst[kNumBuckets] = {
    {1.f, 1.f, 4.f, 8388610.f, 2u * 85u + 0x4B400000u, 2},
    {3.f, 1.f / 3.f, 8.f, 8388612.f, 4u * 585u + 0x4B400000u, 3},
    {7.f, 1.f / 7.f, 16.f, 8388616.f, 8u * 4369u + 0x4B400000u, 4},
    {127.f, 1.f / 127.f, 256.f, 8388736.f, 0u, 8},
};

// Quantises the row held by LPR lanes (G groups of 8 elements each; `amax`: this lane's largest magnitude) at the width of
// `bucket`.  Returns the row's scale, and of each group the packed field of 8 * bits bits: (lo, hi) at 8 bits, lo otherwise.
// Bit-exact with scale_of / quantize_vals; a lane with a near-tie, a NaN or a scale outside the normal range redoes its values
// with the division, as those do.
template <int LPR, int G>
__device__ __forceinline__ float quantize_groups(const float (&x)[G][8], float amax, int bucket, uint32_t (&lo)[G], uint32_t (&hi)[G]) {
  const WidthConst& wc = kWidthConst[bucket];
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  float scale;
  if (amax >= 1e-30f && amax <= 1e30f) {
    const float q0 = __fmul_rn(amax, wc.rlevels);
    scale = __fmaf_rn(__fmaf_rn(-q0, wc.levels, amax), wc.rlevels, q0);
  } else {
    scale = __fdiv_rn(amax, wc.levels);
    if (scale == 0.f) scale = 1.f;
  }
  const float rc = rcp_approx(scale);
  const float up = rc * (1.f + 0x1p-20f), dn = rc * (1.f - 0x1p-20f);
  const uint64_t up2 = f32x2(up, up), dn2 = f32x2(dn, dn), magic2 = f32x2(kRoundMagic, kRoundMagic), neg2 = f32x2(-1.f, -1.f);
  uint64_t nq[G][4], diff = 0ull;  // the negated codes of elements i and i + 4, as floats
#pragma unroll
  for (int j = 0; j < G; ++j) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint64_t x2 = f32x2(x[j][i], x[j][i + 4]);
      const uint64_t m = f32x2_fma(x2, up2, magic2), d = f32x2_fma(f32x2_fma(x2, dn2, magic2), neg2, m);
      diff = f32x2_fma(d, d, diff);
      nq[j][i] = f32x2_fma(m, neg2, magic2);
    }
  }
  const float2 dd = f32x2_parts(diff);
  const bool exact = !(scale >= 1e-30f && scale <= 1e30f && dd.x + dd.y == 0.f);
  if (exact) {
    const float fhi = wc.levels, flo = -fhi - 1.f;
#pragma unroll
    for (int j = 0; j < G; ++j) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        nq[j][i] = f32x2(-fminf(fmaxf(rintf(__fdiv_rn(x[j][i], scale)), flo), fhi),
                         -fminf(fmaxf(rintf(__fdiv_rn(x[j][i + 4], scale)), flo), fhi));
    }
  }
  const uint64_t base2 = f32x2(wc.base, wc.base);
#pragma unroll
  for (int j = 0; j < G; ++j) {
    const uint64_t (&n)[4] = nq[j];
    if (bucket == 3) {  // two's complement bytes: pairs of codes joined, offset so that no byte borrows from the next, flipped back
      const float2 a = f32x2_parts(f32x2_add(f32x2_fma(n[1], base2, n[0]), magic2));
      const float2 b = f32x2_parts(f32x2_add(f32x2_fma(n[3], base2, n[2]), magic2));
      constexpr uint32_t m = 0x4B400000u, o = 0x80808080u;
      lo[j] = ((m + o - __float_as_uint(a.x)) + ((m - __float_as_uint(b.x)) << 16)) ^ o;
      hi[j] = ((m + o - __float_as_uint(a.y)) + ((m - __float_as_uint(b.y)) << 16)) ^ o;
    } else {  // four codes each as a polynomial in 2^bits, made non-negative by the offset of every code, then joined
      const float2 poly = f32x2_parts(f32x2_add(
          f32x2_fma(f32x2_fma(f32x2_fma(n[3], base2, n[2]), base2, n[1]), base2, n[0]), magic2));
      lo[j] = (wc.off - __float_as_uint(poly.x)) + ((wc.off - __float_as_uint(poly.y)) << (4 * wc.bits));
      hi[j] = 0u;
    }
  }
  return scale;
}
// Stores the packed fields of a lane that holds two neighbouring groups (lane l of the row's head_dim / 16; whole warp, `next` =
// lo[0] of the next lane) at the row's address.
__device__ __forceinline__ void store_field16(uint8_t* row, int bucket, int l, const uint32_t (&lo)[2], const uint32_t (&hi)[2],
                                              uint32_t next) {
  uint32_t* out = reinterpret_cast<uint32_t*>(row);
  if (bucket == 3) {
    uint2* w = reinterpret_cast<uint2*>(out) + 2 * l;  // a store is asked for no more than 8-byte alignment here
    w[0] = make_uint2(lo[0], hi[0]);
    w[1] = make_uint2(lo[1], hi[1]);
  } else if (bucket == 2) {
    reinterpret_cast<uint2*>(out)[l] = make_uint2(lo[0], lo[1]);
  } else if (bucket == 0) {
    out[l] = lo[0] | (lo[1] << 16);
  } else {  // 3 bits: two lanes' 48 bits make three words
    uint32_t* w = out + 3 * (l >> 1);
    if (l & 1) {
      w[2] = (lo[0] >> 16) | (lo[1] << 8);
    } else {
      w[0] = lo[0] | (lo[1] << 24);
      w[1] = (lo[1] >> 8) | (next << 16);
    }
  }
}

// The 8 values code * scale of a lane's field.  The code goes into the significand of 2^23 and the offset comes off in the
// same subtraction, so no int->float conversion is needed; 8-bit rows hold two's complement, which flipping the top bit
// turns into the offset form of the other widths.
__device__ __forceinline__ void dequantize8(uint32_t lo, uint32_t hi, int bucket, float scale, float (&x)[8]) {
  const WidthConst& wc = kWidthConst[bucket];
  const int bits = wc.bits;
  const uint32_t fm = (1u << bits) - 1u, flip = bucket == 3 ? 0x80808080u : 0u;
  const uint64_t nb2 = f32x2(-wc.bias, -wc.bias), s2 = f32x2(scale, scale);
  lo ^= flip;
  hi = bucket == 3 ? hi ^ flip : lo >> (4 * bits);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t a = ((lo >> (bits * i)) & fm) | 0x4B000000u, b = ((hi >> (bits * i)) & fm) | 0x4B000000u;
    const float2 v = f32x2_parts(f32x2_mul(f32x2_add(f32x2(__uint_as_float(a), __uint_as_float(b)), nb2), s2));
    x[i] = v.x;
    x[i + 4] = v.y;
  }
}

}  // namespace skv
