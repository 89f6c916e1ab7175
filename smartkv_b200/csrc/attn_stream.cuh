// Tile arithmetic of the fp16-query decode-attention kernel (decode_attention_f16.cu): where the rows of a 16-key tile
// lie in shared memory, and the P.V product on unpacked codes.  lane = 4*g + t throughout; the score side (element orders,
// integer products) is attn_frag.cuh's.
//
// Layout.  A tile's K rows and V rows are copied in 16-byte chunks (cp.async), and the chunk's place is free.  In every
// 128-byte line the chunk index is XORed with a function of the line (swizzle below), so that both the 16-byte slice loads
// of K and the 8-row ldmatrix loads of V touch every bank once.  Rows of 3-bit codes (48 or 24 bytes) stay linear.
//
// V.  ldmatrix.trans on 16-bit columns hands lane (g,t) bytes 2g, 2g+1 of one 16-byte chunk for the keys 2t and 2t+1 side
// by side: the byte permutes that pairing two rows takes otherwise come with the load.  The fields become fp16 as in
// attn_frag.cuh (one logic operation, one packed multiply-add, exact).  Cheaper forms lose accuracy and were taken back: a
// masked field is an fp16 subnormal as it stands, but the tensor core aligns products by the operand's nominal exponent, so
// small fields lose up to 10 of the accumulator's bits (2-bit cache, 8192 keys: output error 2.0e-3 against 2.7e-4).
#pragma once

#include "attn_frag.cuh"

namespace skv {

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&d)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm_x2_trans(uint32_t (&d)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];" : "=r"(d[0]), "=r"(d[1]) : "r"(addr) : "memory");
}

// ---- chunk places ---------------------------------------------------------------------------------------
// XOR applied to the chunk index inside 128-byte line `line` of a tile, rows of `row_bytes` bytes.
__host__ __device__ constexpr int chunk_swizzle(int row_bytes, int line) {
  return row_bytes == 128 ? (line & 7) : row_bytes == 64 ? (line & 3) : row_bytes == 32 ? (line & 1) : 0;
}
// byte offset of 16-byte chunk c of row r
__host__ __device__ constexpr int chunk_place(int row_bytes, int r, int c) {
  const int linear = r * row_bytes + 16 * c, line = linear >> 7;
  return (line << 7) | ((((linear >> 4) & 7) ^ chunk_swizzle(row_bytes, line)) << 4);
}

// This lane's K slice of row g starts here; the slice of row g + 8 lies 8 rows further (a whole number of swizzle periods).
template <int D, int BITS>
__device__ __forceinline__ int kslice_place(int lane) {
  constexpr int RB = D * BITS / 8, SB = RB / 4;
  const int g = lane >> 2, t = lane & 3;
  if constexpr (BITS == 3) return g * RB + t * SB;
  else if constexpr (SB >= 16) return chunk_place(RB, g, t * (SB / 16));
  else return chunk_place(RB, g, t * SB / 16) + (t * SB) % 16;
}
// Raw K slice from `p` = tile + kslice_place (+ 8 rows); the second chunk of a 32-byte slice is the XOR neighbour.
template <int D, int BITS>
__device__ __forceinline__ void load_kslice_sw(const uint8_t* tile, int place, uint32_t (&w)[SliceWords<D, BITS>::K]) {
  constexpr int SB = D * BITS / 32;
  static_assert(BITS != 3, "3-bit rows are linear: load_kslice");
  if constexpr (SB >= 16) {
#pragma unroll
    for (int i = 0; i < SB / 16; ++i) {
      const uint4 v = *reinterpret_cast<const uint4*>(tile + (place ^ (16 * i)));
      w[4 * i + 0] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
    }
  } else if constexpr (SB == 8) {
    const uint2 v = *reinterpret_cast<const uint2*>(tile + place);
    w[0] = v.x; w[1] = v.y;
  } else {
    w[0] = *reinterpret_cast<const uint32_t*>(tile + place);
  }
}

// The row address this lane gives to ldmatrix: matrices 0, 1 = keys 0..7, 8..15 of chunk c, matrices 2, 3 of chunk c + 1
// (c even: XOR 16 * c gives the other chunk pairs).
template <int D, int BITS>
__device__ __forceinline__ int vmatrix_place(int lane) {
  constexpr int RB = D * BITS / 8;
  const int m = lane >> 3, r = lane & 7;
  return chunk_place(RB, (m & 1) * 8 + r, RB == 16 ? 0 : (m >> 1));
}

// Integer scores of one n-tile from zero (qk_ntile_i8 of attn_frag.cuh without an accumulator to set up first).
template <bool B_UNSIGNED>
__device__ __forceinline__ void mma_i8_first(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (B_UNSIGNED) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
  } else {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
  }
}
template <int D, int BITS>
__device__ __forceinline__ void qk_stream(const uint32_t (&k)[SliceWords<D, BITS>::K], const uint32_t (&qa)[D / 32][4], int (&acc)[4]) {
  uint32_t b[D / 16];
  unpack_kslice_i8<D, BITS>(k, b);
  mma_i8_first<BITS != 8>(acc, qa[0], b[0], b[1]);
#pragma unroll
  for (int s = 1; s < D / 32; ++s) mma_i8_16832<BITS != 8>(acc, qa[s], b[2 * s], b[2 * s + 1]);
}

// ---- P.V -------------------------------------------------------------------------------------------------
// Bit position of the field that row half hi (0: rows g, 1: rows g + 8) of output tile j multiplies.
template <int BITS>
__host__ __device__ constexpr int vfield_pos(int j, int hi) {
  constexpr int pos2[8] = {0, 2, 4, 6, 8, 0, 2, 4}, pos3[8] = {0, 3, 6, 1, 4, 7, 2, 5};
  return BITS == 8 ? 0 : BITS == 4 ? 4 * hi : BITS == 2 ? pos2[2 * (j % 4) + hi] : pos3[2 * (j % 4) + hi];
}
// Output tile j, row g is head element vdim(j, g); row g + 8 the one after it.
template <int D, int BITS>
__device__ __forceinline__ int vdim(int j, int g) {
  if constexpr (BITS == 8) return 16 * j + 2 * g;
  else if constexpr (BITS == 4) return 32 * (j / 2) + 4 * g + 2 * (j % 2);
  else if constexpr (BITS == 2) return 64 * (j / 4) + 8 * g + 2 * (j % 4);
  else return g * (D / 8) + 2 * j;
}

// (field at bit P of both halves - offset) * 2^P
template <int P, int W>
__device__ __forceinline__ uint32_t vfield(uint32_t x) {
  constexpr uint32_t m = ((1u << W) - 1u) << P;
  constexpr uint32_t add = h2c(-(1024.0 + (double)(1 << (W - 1)) * (1 << P)));
  return hadd2_bits(lop_and_or(x, m | (m << 16), kMagic), add);
}
// The fields of one 16-bit column pair x in tile order: f[2 * i + hi] belongs to row half hi of tile i of the column's tiles.
template <int BITS>
__device__ __forceinline__ void vfields(uint32_t x, uint32_t* f) {
  if constexpr (BITS == 8) {  // two's complement: 1024 + (code ^ 0x80), less 1152
    constexpr uint32_t add = h2c(-1152.0);
    f[0] = hadd2_bits(lop_and_xor(x, 0x00ff00ffu, 0x64806480u), add);
    f[1] = hadd2_bits(lop_and_xor(x >> 8, 0x00ff00ffu, 0x64806480u), add);
  } else if constexpr (BITS == 4) {
    const uint32_t y = x >> 8;
    f[0] = vfield<0, 4>(x);
    f[1] = vfield<4, 4>(x);
    f[2] = vfield<0, 4>(y);
    f[3] = vfield<4, 4>(y);
  } else {
    static_assert(BITS == 2, "3-bit rows: vfields3");
    const uint32_t y = x >> 10;
    f[0] = vfield<0, 2>(x);
    f[1] = vfield<2, 2>(x);
    f[2] = vfield<4, 2>(x);
    f[3] = vfield<6, 2>(x);
    f[4] = vfield<8, 2>(x);
    f[5] = vfield<0, 2>(y);
    f[6] = vfield<2, 2>(y);
    f[7] = vfield<4, 2>(y);
  }
}
// 3-bit: one 24-bit group (8 fields) of two rows; x0 = bytes 0,1 of both, x1 = bytes 1,2, x2 = byte 2 (upper byte unused)
__device__ __forceinline__ void vfields3(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t* f) {
  f[0] = vfield<0, 3>(x0);
  f[1] = vfield<3, 3>(x0);
  f[2] = vfield<6, 3>(x0);
  f[3] = vfield<1, 3>(x1);
  f[4] = vfield<4, 3>(x1);
  f[5] = vfield<7, 3>(x1);
  f[6] = vfield<2, 3>(x2);
  f[7] = vfield<5, 3>(x2);
}
// 3-bit rows A (words a) and B: all D/8 fields of this lane's slice
template <int D>
__device__ __forceinline__ void vpair3(const uint32_t (&a)[2], const uint32_t (&b)[2], int g, uint32_t* f) {
  if constexpr (D == 128) {  // 6 bytes, 0 or 2 bytes into the words: two groups of 3 bytes
    const uint32_t lo = (g & 1) ? 0x5432u : 0x3210u, hi = (g & 1) ? 0x7654u : 0x5432u;
    const uint32_t a0 = prmt(a[0], a[1], lo), b0 = prmt(b[0], b[1], lo);  // bytes 0..3
    const uint32_t a1 = prmt(a[0], a[1], hi), b1 = prmt(b[0], b[1], hi);  // bytes 2..5
    vfields3(prmt(a0, b0, 0x5410), prmt(a0, b0, 0x6521), prmt(a0, b0, 0x7632), f);
    vfields3(prmt(a1, b1, 0x6521), prmt(a1, b1, 0x7632), prmt(a1, b1, 0x7733), f + 8);
  } else {  // 3 bytes at byte offset 3g of the row
    const int sh = ((g * 3) & 3) * 8;
    const uint32_t a0 = __funnelshift_r(a[0], a[1], sh), b0 = __funnelshift_r(b[0], b[1], sh);
    vfields3(prmt(a0, b0, 0x5410), prmt(a0, b0, 0x6521), prmt(a0, b0, 0x7632), f);
  }
}

// o += V^T P of one 16-key tile, in code units times 2^vfield_pos (the V scale is in P).  pb0 / pb1: P^T fragments of the keys (2t, 2t+1) and
// (2t+8, 2t+9).  vm: this lane's ldmatrix address.
template <int D, int BITS>
__device__ __forceinline__ void pv_stream(uint32_t vm, uint32_t pb0, uint32_t pb1, float (&o)[D / 16][4]) {
  constexpr int NCH = D * BITS / 128;  // 16-byte chunks of a row
  constexpr int MT = 8 / BITS;         // output tiles of a chunk
#pragma unroll
  for (int ch = 0; ch < NCH; ch += 2) {
    uint32_t x[4];
    if constexpr (NCH == 1) ldsm_x2_trans(x, vm);
    else ldsm_x4_trans(x, vm ^ (16 * ch));
#pragma unroll
    for (int e = 0; e < (NCH == 1 ? 1 : 2); ++e) {
      uint32_t f0[2 * MT], f1[2 * MT];
      vfields<BITS>(x[2 * e], f0);
      vfields<BITS>(x[2 * e + 1], f1);
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const uint32_t a[4] = {f0[2 * i], f0[2 * i + 1], f1[2 * i], f1[2 * i + 1]};
        mma_16816(o[(ch + e) * MT + i], a, pb0, pb1);
      }
    }
  }
}
// the same for 3-bit rows: vr = this lane's raw slices of the keys 2t, 2t+1, 2t+8, 2t+9
template <int D>
__device__ __forceinline__ void pv_stream3(const uint32_t (&vr)[4][2], int g, uint32_t pb0, uint32_t pb1, float (&o)[D / 16][4]) {
  uint32_t f0[D / 8], f1[D / 8];
  vpair3<D>(vr[0], vr[1], g, f0);
  vpair3<D>(vr[2], vr[3], g, f1);
#pragma unroll
  for (int j = 0; j < D / 16; ++j) {
    const uint32_t a[4] = {f0[2 * j], f0[2 * j + 1], f1[2 * j], f1[2 * j + 1]};
    mma_16816(o[j], a, pb0, pb1);
  }
}

// The accumulators as [head][kAccStride] floats in shared memory, in code units, and back (the order of the elements over the
// lanes and their powers of two depend on the width).  A stride of D + 4 floats spreads the 64-bit stores over the banks and makes 8 heads exactly one tile slot.
__host__ __device__ constexpr float pow2f(int e) {
  float v = 1.f;
  for (int i = 0; i < e; ++i) v *= 2.f;
  for (int i = 0; i > e; --i) v *= 0.5f;
  return v;
}
template <int D>
constexpr int kAccStride = D + 4;
template <int D, int BITS>
__device__ __forceinline__ void store_acc(float* buf, int lane, const float (&o)[D / 16][4]) {
  const int g = lane >> 2, t = lane & 3;
  float* r0 = buf + 2 * t * kAccStride<D> + vdim<D, BITS>(0, g);
#pragma unroll
  for (int j = 0; j < D / 16; ++j) {
    const int d = vdim<D, BITS>(j, 0);
    const float u0 = pow2f(-vfield_pos<BITS>(j, 0)), u1 = pow2f(-vfield_pos<BITS>(j, 1));
    *reinterpret_cast<float2*>(r0 + d) = make_float2(o[j][0] * u0, o[j][2] * u1);
    *reinterpret_cast<float2*>(r0 + kAccStride<D> + d) = make_float2(o[j][1] * u0, o[j][3] * u1);
  }
}
template <int D, int BITS>
__device__ __forceinline__ void load_acc(const float* buf, int lane, float (&o)[D / 16][4]) {
  const int g = lane >> 2, t = lane & 3;
  const float* r0 = buf + 2 * t * kAccStride<D> + vdim<D, BITS>(0, g);
#pragma unroll
  for (int j = 0; j < D / 16; ++j) {
    const int d = vdim<D, BITS>(j, 0);
    const float2 x = *reinterpret_cast<const float2*>(r0 + d), y = *reinterpret_cast<const float2*>(r0 + kAccStride<D> + d);
    const float u0 = pow2f(vfield_pos<BITS>(j, 0)), u1 = pow2f(vfield_pos<BITS>(j, 1));
    o[j][0] = x.x * u0;
    o[j][2] = x.y * u1;
    o[j][1] = y.x * u0;
    o[j][3] = y.y * u1;
  }
}

// ---- query -------------------------------------------------------------------------------------------------
// 4 x 4 byte transpose: out[e] = byte e of the four words
__device__ __forceinline__ void transpose4(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, uint32_t* out) {
  const uint32_t a = prmt(w0, w1, 0x5140), b = prmt(w2, w3, 0x5140), c = prmt(w0, w1, 0x7362), d = prmt(w2, w3, 0x7362);
  out[0] = prmt(a, b, 0x5410);
  out[1] = prmt(a, b, 0x7632);
  out[2] = prmt(c, d, 0x5410);
  out[3] = prmt(c, d, 0x7632);
}
// One limb of a head's query slice (elements t*D/4 ..) in the order kelem_i8<BITS> of the key registers.
template <int D, int BITS>
__device__ __forceinline__ void query_slice(const int8_t* limb, int t, uint32_t (&r)[D / 16]) {
  uint32_t w[D / 16];
  const uint4* p = reinterpret_cast<const uint4*>(limb + t * (D / 4));
#pragma unroll
  for (int i = 0; i < D / 64; ++i) {
    const uint4 v = p[i];
    w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
  }
  if constexpr (BITS == 8) {
#pragma unroll
    for (int i = 0; i < D / 16; ++i) r[i] = w[i];
  } else if constexpr (BITS == 4) {
#pragma unroll
    for (int s = 0; s < D / 32; ++s) {
      r[2 * s] = prmt(w[2 * s], w[2 * s + 1], 0x6420);
      r[2 * s + 1] = prmt(w[2 * s], w[2 * s + 1], 0x7531);
    }
  } else if constexpr (BITS == 2) {
#pragma unroll
    for (int h = 0; h < D / 64; ++h) transpose4(w[4 * h], w[4 * h + 1], w[4 * h + 2], w[4 * h + 3], r + 4 * h);
  } else {
    static_assert(D == 128, "3-bit rows of head_dim 64 use the fp16 path");
    transpose4(w[0], w[2], w[4], w[6], r);
    transpose4(w[1], w[3], w[5], w[7], r + 4);
  }
}

}  // namespace skv
