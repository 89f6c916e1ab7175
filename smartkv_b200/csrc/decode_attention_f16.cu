// Fused packed-KV decode attention for fp16 queries (q_len == 1, GQA group <= 8): the mma.sync kernel in which every warp
// streams its own tiles.
//
// Partition.  A CTA (one per SM) owns the runs the plan gives it (attn_sched.cuh); its tile string is cut once more, by the
// same tile costs, into one contiguous slice per warp.  A slice lies in one or two buckets as a rule, so at any time the
// warps of an SM work on all widths: the byte-bound 8-bit tiles and the arithmetic-bound narrow ones overlap.
// Pipeline.  Each warp copies its tiles into a ring of its own (cp.async, 16 bytes a lane), STAGES - 1 tiles
// ahead, and waits for nothing but its own copies: no producer warp, no barrier between warps while streaming.
// (The L2 evict-first hint of the bulk copies is left out: cp.async with an L2 cache hint raised "an illegal instruction".)
// Merge.  The pieces of one run that end in different warps are folded through shared memory once per eight runs, in warp
// order, so a run leaves two partials (attn_params.cuh) where per-warp partials left eleven.
//
// Replaces smartkv/csrc/quantized_attention.cu:460-828 (per-bucket kernel, one CTA per head walking the whole context);
// numerics follow the CPU streaming path smartkv/core/fused_cpu.py:70-113 (dequantise, q.k/sqrt(d), online softmax).
//
// Bound: HBM while streaming (16 x 8192 keys at a budget of 0.35: 188 MB in 41.4 us a launch back to back, some 30 of them at
// 6.3 TB/s); the rest is the start (plan, first copies, query: 5 us), the merge and the spread of the warps' ends.  Before (one
// producer warp with bulk copies, 11 consumer warps on shared blocks, partials per warp; see decode_attention.cu, which keeps
// that form for fp32 queries) and now, us a launch back to back: 43.5 / 41.4 (16 x 8192), 38.2 / 33.3 (1 x 131072), 50.8 / 46.1
// (64 x 16384, one KV head), 11.1 / 7.6 (8 x 770, head_dim 64); a decode step, whose combine now folds one partial a run:
// 1763 / 1589, 1740 / 1304, 1640 / 1249, 418 / 274.
#include <atomic>
#include <cstdio>
#include <type_traits>

#include "attn_params.cuh"
#include "attn_stream.cuh"
#include "post_attention.cuh"

extern std::atomic<int> g_dependent_launch;  // decode_attention.cu

namespace skv {

constexpr int kGroupRuns = kPlanFirstRuns;  // runs a CTA handles between two merges: 8 runs x 4 buckets = one lane each
static_assert(kGroupRuns * kNumBuckets == 32, "one lane per (run, bucket)");
// The running maximum is raised when a score exceeds it by this much (log2 units).  p * v_scale is rounded to fp16, and for the key
// that sets the maximum p is exactly 1, which at 2 bits makes the product exact; how many rows' largest key that holds for
// depends on it and on how the keys are cut into streams.  Root-mean-square output error against 64 bits over eleven
// shapes (384 query sets each), relative to the block pipeline of decode_attention.cu with this kernel's operands and 8: at 8 1.004
// (0.980 to 1.018 by shape), at 4 0.983 (0.918 to 1.006), at 0 0.974.  Time of eight layers, us at 8 / 4 / 0: 16 x 8192 keys 421.3 /
// 421.5 / 423.3, 1 x 131072 402.8 / 402.6 / 401.2, head_dim 64: 16 x 4096 183.2 / 184.0 / 188.3, 1 x 32768 141.5 / 142.3 / 144.6.
constexpr float kLazyTau = 4.0f;

// Warps of a CTA.  head_dim 128: twelve, 168 registers each; sixteen at 128 end later for all their work in flight, because
// every warp brings its start, its share of the merge and a rounding to whole tiles (steps of 16 x 8192 keys 1610 us
// against 1658, 64 x 16384 1253 against 1288, 1 x 131072 the same; eight warps 1687, 1317 and 1487 against 1358; all with the
// combine of two partials a run).  head_dim 64, whose contexts are short: sixteen (8 x 770 keys 303 us a step, twelve 316).
template <int D>
struct StreamShape {
  static constexpr int WARPS = D == 128 ? 12 : 16;
  static constexpr int SLOT = 16 * (2 * D + 8);  // one 16-key tile at the widest: K rows, V rows, scales
  static constexpr int V_AT = 16 * D, S_AT = 32 * D;
  static constexpr int STAGES = D == 128 ? 3 : 6;
  static constexpr int RING = STAGES * SLOT;
  static_assert(8 * kAccStride<D> * 4 <= SLOT, "the accumulators of 8 heads must fit a slot");
};

// What the CTA's warps share besides their rings.
template <int D>
struct __align__(16) StreamShared {
  static constexpr int WARPS = StreamShape<D>::WARPS;
  int8_t limb[kGroupRuns][2][8][D];                    // query of a run: int8 limbs (radix 128), most significant first
  __half qh[D == 64 ? kGroupRuns : 1][D == 64 ? 8 : 1][D];  // fp16 rows, for the 3-bit keys of head_dim 64
  float sq[kGroupRuns][8];                             // limb step per head: q = sq * (128 * limb0 + limb1)
  int sum[kGroupRuns][8];                              // 128 * sum(limb0) + sum(limb1)
  float tail_m[WARPS][8], tail_l[WARPS][8];          // (max, sum) of every warp's last piece
  float weight[WARPS][8];                             // its weight in the merged partial
  int tail_run[WARPS];                                // run (of the group) of that piece, -1: the warp had no tile
  int has_first[kGroupRuns], has_second[kGroupRuns];   // partials of a run written by a warp alone
};

struct SoftState {
  float m;  // running reference maximum (log2 units); head lane >> 2
  float l;  // this lane's share of the running sum
};

// The query row of one head of a run by one warp (same limbs as the fp32-query kernel's).
template <int D>
__device__ __forceinline__ void prep_query(StreamShared<D>& sh, int rr, int gq, const __half* row, int lane) {
  constexpr int EPL = D / 32;
  float q[EPL];
  float amax = 0.f;
#pragma unroll
  for (int e = 0; e < EPL; ++e) {
    const __half h = row[lane * EPL + e];
    if (D == 64) sh.qh[rr][gq][lane * EPL + e] = h;
    q[e] = __half2float(h);
    amax = fmaxf(amax, fabsf(q[e]));
  }
  amax = warp_max(amax);
  const float range = 127.f * 128.f;
  const float step = amax > 0.f ? amax / range : 1.f;
  const float inv = 1.f / step;
  int sum0 = 0, sum1 = 0;
#pragma unroll
  for (int e = 0; e < EPL; ++e) {
    const float rem = fminf(fmaxf(rintf(q[e] * inv), -range), range);
    const float hi = rintf(rem * (1.f / 128.f));
    const int l0 = (int)hi, l1 = (int)(rem - hi * 128.f);
    sh.limb[rr][0][gq][lane * EPL + e] = (int8_t)l0;
    sh.limb[rr][1][gq][lane * EPL + e] = (int8_t)l1;
    sum0 += l0;
    sum1 += l1;
  }
  int sum = 128 * sum0 + sum1;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  if (lane == 0) {
    sh.sq[rr][gq] = step;
    sh.sum[rr][gq] = sum;
  }
}

// floor(x / cost of a tile of bucket bk) for x < 2^30, as a multiplication (the error of the rounded-up reciprocal, less than
// the cost, stays below 2^38 / 2^30)
__device__ __forceinline__ unsigned tiles_in(unsigned x, int D, int bk) {
  unsigned m = 0;
#pragma unroll
  for (int i = 0; i < kNumBuckets; ++i) {
    const unsigned c = (unsigned)tile_cost_for(D, bucket_bits(i), kPlanModelFrag);
    if (bk == i) m = (unsigned)(((1ull << 38) + c - 1) / c);
  }
  return __umulhi(x, m) >> 6;
}

// A warp's copies: the tiles of its pieces in order, one commit group a tile (empty groups after the last).
struct TileFeed {
  const uint8_t *k, *v, *s;  // next tile of the piece, this lane's 16 bytes
  int left;                  // tiles of the piece still to be issued
  int chunks;                // 16-byte chunks of a tile's K rows
  int place0, flip;          // place of this lane's chunk; XOR for every other 512 bytes
  unsigned pieces;           // lanes holding pieces not begun
  uint32_t slot;             // shared-memory address the next tile goes to
};

// HALF: at most four query heads per KV head.  The score rows of heads 4..7 then repeat heads 0..3, so that lanes g < 4 take
// the first eight keys of a tile through the softmax and lanes g >= 4 the other eight, instead of idling.
template <int D, bool MASKED, bool HALF>
__global__ void __launch_bounds__(StreamShape<D>::WARPS * 32, 1) decode_attn_f16_kernel(const AttnParams p) {
  using S = StreamShape<D>;
  constexpr int WARPS = S::WARPS;
  extern __shared__ __align__(128) uint8_t smem[];
  StreamShared<D>& sh = *reinterpret_cast<StreamShared<D>*>(smem + WARPS * S::RING);
  const StoreGeom& g = p.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lg = lane >> 2, t = lane & 3;
  const int gq = HALF ? lg & 3 : lg;  // scores: head gq; accumulators: heads 2t, 2t+1
  const int G = p.group, Hkv = g.num_kv_heads;
  uint8_t* ring = smem + warp * S::RING;
  const uint32_t ring_at = smem_u32(ring);

  if (tid < kGroupRuns * 8) {  // heads that do not exist score zero whatever their limbs hold
    sh.sq[tid >> 3][tid & 7] = 0.f;
    sh.sum[tid >> 3][tid & 7] = 0;
  }
  if constexpr (D == 64) {
    for (int i = tid; i < kGroupRuns * 8 * D / 2; i += WARPS * 32) reinterpret_cast<uint32_t*>(&sh.qh[0][0][0])[i] = 0u;
  }
  __syncthreads();
  // What is read before pdl_wait() -- the plan and this layer's rows -- was written by kernels that completed long before a
  // dependent launch of this kernel can start; the query and everything written here come after it.
  pdl_launch_dependents();
  const PlanView pv = plan_view(const_cast<int*>(p.plan), p.num_ctas, g.num_seqs * Hkv);
  const int run_begin = pv.cta_begin[blockIdx.x], run_end = pv.cta_begin[blockIdx.x + 1];
  if (run_begin >= run_end) {  // still, no CTA of a dependent launch leaves before its predecessor ended
    pdl_wait();
    return;
  }
  const int tile_mul = pv.header[3] == 128 ? 8 : 1;  // a plan cut in 128-key tiles is read in 16-key tiles

  for (int r0 = run_begin; r0 < run_end; r0 += kGroupRuns) {
    const int nr = (run_end - r0) < kGroupRuns ? (run_end - r0) : kGroupRuns;
    // ---- lane = (run of the group, bucket): this warp's slice of the lane's tiles ------------------------------------
    const int rr = lane >> 2, bk = lane & 3;
    int ka = 0, n = 0, cnt = 0, seq = 0, head = 0;
    {
      const RunDesc* d = r0 == run_begin ? pv.first + blockIdx.x * kPlanFirstRuns + rr : pv.runs + r0 + (rr < nr ? rr : 0);
      seq = d->seq;
      head = d->head;
      cnt = d->cnt[bk];
      ka = d->ka[bk];
      const int kb = d->kb[bk], nt = (cnt + 15) >> 4;
      n = (kb * tile_mul < nt ? kb * tile_mul : nt);
      ka = ka * tile_mul < nt ? ka * tile_mul : nt;
      n -= ka;
      if (rr >= nr) seq = head = cnt = ka = n = 0;  // a record of no run
    }
    // cost units before and after this lane's tiles; a string too long for 30 bits counts tiles instead
    const bool by_count = __any_sync(0xffffffffu, n >= 1 << 17);
    const unsigned cost = by_count ? 1u : (unsigned)tile_cost_for(D, bucket_bits(bk), kPlanModelFrag);
    const unsigned own = (unsigned)n * cost;
    unsigned end = own;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned x = __shfl_up_sync(0xffffffffu, end, off);
      if (lane >= off) end += x;
    }
    const unsigned total = __shfl_sync(0xffffffffu, end, 31), start = end - own;
    auto first_tile = [&](int w) -> int {  // first tile of this lane whose cost begins in slice w or a later one
      const unsigned at = (unsigned)(((unsigned long long)total * w + WARPS - 1) / WARPS);
      if (at <= start) return 0;
      if (at >= end) return n;
      return (int)(by_count ? at - start : tiles_in(at - start + cost - 1, D, bk));
    };
    const int a = first_tile(warp), b = first_tile(warp + 1);
    // the run of this lane in the whole warp (its four lanes): does this warp's slice hold all of it?
    const unsigned mine = __ballot_sync(0xffffffffu, a < b);
    const unsigned missing = __ballot_sync(0xffffffffu, a > 0 || b < n);
    const int tail = mine ? (31 - __clz(mine)) >> 2 : -1;
    TileFeed f;
    f.left = 0;
    f.pieces = mine;
    f.slot = ring_at;
    auto issue = [&]() {
      if (f.left == 0 && f.pieces != 0) {  // next piece
        const int src = __ffs(f.pieces) - 1;
        f.pieces &= f.pieces - 1;
        const int fseq = __shfl_sync(0xffffffffu, seq, src), fhead = __shfl_sync(0xffffffffu, head, src), fb = src & 3;
        const uint8_t* arena = arena_ptr(g, p.store, p.layer, fseq) + lane * 16;
        const long long row = (long long)fhead * g.cap[fb] + __shfl_sync(0xffffffffu, ka + a, src) * 16;
        f.k = arena + g.k_off[fb] + row * g.row_bytes[fb];
        f.v = arena + g.v_off[fb] + row * g.row_bytes[fb];
        f.s = arena + g.sc_off[fb] + row * 8;
        f.left = __shfl_sync(0xffffffffu, b - a, src);
        const int rb = g.row_bytes[src & 3], line = lane >> 3;
        f.chunks = rb;  // 16 rows of rb bytes
        f.place0 = (line << 7) | (((lane & 7) ^ chunk_swizzle(rb, line)) << 4);
        f.flip = rb == 128 ? 64 : 0;
      }
      if (f.left > 0) {
#pragma unroll
        for (int i = 0; i < D / 32; ++i) {
          if (32 * i < f.chunks) {
            if (32 * i + lane < f.chunks) {
              const uint32_t dst = f.slot + 512 * i + ((i & 1) ? f.place0 ^ f.flip : f.place0);
              cp_async16(dst, f.k + 512 * i);
              cp_async16(dst + S::V_AT, f.v + 512 * i);
            }
          }
        }
        if (lane < 8) cp_async16(f.slot + S::S_AT + lane * 16, f.s);
        f.k += f.chunks * 16;
        f.v += f.chunks * 16;
        f.s += 128;
        --f.left;
        f.slot = f.slot + S::SLOT == ring_at + S::RING ? ring_at : f.slot + S::SLOT;
      }
      cp_async_commit();
    };
    // the same inside a piece whose rows have row_bytes_tag bytes
    auto issue_more = [&](auto row_bytes_tag) {
      constexpr int RB = decltype(row_bytes_tag)::value;
#pragma unroll
      for (int i = 0; 32 * i < RB; ++i) {
        if (32 * i + 32 <= RB || lane < RB - 32 * i) {
          const uint32_t dst = f.slot + 512 * i + ((i & 1) ? f.place0 ^ (RB == 128 ? 64 : 0) : f.place0);
          cp_async16(dst, f.k + 512 * i);
          cp_async16(dst + S::V_AT, f.v + 512 * i);
        }
      }
      if (lane < 8) cp_async16(f.slot + S::S_AT + lane * 16, f.s);
      f.k += RB * 16;
      f.v += RB * 16;
      f.s += 128;
      --f.left;
      f.slot = f.slot + S::SLOT == ring_at + S::RING ? ring_at : f.slot + S::SLOT;
      cp_async_commit();
    };
#pragma unroll
    for (int i = 0; i < S::STAGES - 1; ++i) issue();

    // ---- query rows of the group's runs, one head a warp at a time ------------------------------------------------------
    if (r0 == run_begin) pdl_wait();  // the first copies are in flight
    int guard_flag = 0;  // the (layer, sequence) arena holds a V scale above kVScaleGuard
    if (rr < nr) guard_flag = *arena_flags(g, arena_ptr(g, p.store, p.layer, seq));
    if (tid < kGroupRuns) sh.has_first[tid] = sh.has_second[tid] = 0;
    for (int i = warp; i < nr * G; i += WARPS) {
      const int qr = i / G, h = i - qr * G;
      const int qseq = __shfl_sync(0xffffffffu, seq, 4 * qr), qhead = __shfl_sync(0xffffffffu, head, 4 * qr);
      prep_query<D>(sh, qr, h, static_cast<const __half*>(p.query) + ((long long)qseq * p.num_q_heads + qhead * G + h) * D, lane);
    }
    const unsigned guards = __ballot_sync(0xffffffffu, guard_flag != 0);
    __syncthreads();

    // ---- this warp's pieces -----------------------------------------------------------------------------------------
    SoftState st = {-INFINITY, 0.f};
    float o[D / 16][4];
    int at = 0;                    // offset of the current tile's slot
    const float* carry = nullptr;  // accumulators of the run so far, left by its previous piece
    unsigned todo = mine;

    auto piece = [&](auto bits_tag, int src) {
      constexpr int BITS = decltype(bits_tag)::value;
      constexpr int RB = D * BITS / 8;
      constexpr bool I8 = BITS != 3 || D == 128;  // 3-bit keys of head_dim 64 keep the fp16 score path
      const int prr = src >> 2, bucket = src & 3;
      const int pa = __shfl_sync(0xffffffffu, ka + a, src), pn = __shfl_sync(0xffffffffu, b - a, src);
      const int pseq = __shfl_sync(0xffffffffu, seq, src), phead = __shfl_sync(0xffffffffu, head, src);
      int keys = __shfl_sync(0xffffffffu, cnt, src) - pa * 16;  // live keys from the current tile on
      if (carry != nullptr) {
        load_acc<D, BITS>(carry, lane, o);
      } else {
#pragma unroll
        for (int j = 0; j < D / 16; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
      }

      // query fragments in this width's element order
      uint32_t qa[I8 ? D / 32 : D / 16][4];
      float qs;
      int init = 0;
      if constexpr (I8) {
        uint32_t l0[D / 16], l1[D / 16];
        query_slice<D, BITS>(&sh.limb[prr][0][gq][0], t, l0);
        query_slice<D, BITS>(&sh.limb[prr][1][gq][0], t, l1);
#pragma unroll
        for (int s = 0; s < D / 32; ++s) {
          qa[s][0] = l0[2 * s];
          qa[s][1] = l1[2 * s];
          qa[s][2] = l0[2 * s + 1];
          qa[s][3] = l1[2 * s + 1];
        }
        qs = sh.sq[prr][gq] * p.scale_log2;
        if (BITS != 8) init = -(1 << (BITS - 1)) * sh.sum[prr][gq];  // the offset of the stored codes
      } else {
        gather_qa_f16<D, BITS>(&sh.qh[prr][0][0], false, 4 * gq + t, qa);
        qs = p.scale_log2;
      }
      const long long slot0 = g.bucket_base[bucket] + (long long)pa * 16;
      float* lrow = nullptr;  // logits of head gq, keys 2t.. of the current tile
      if (p.logits != nullptr && gq < G)
        lrow = p.logits + ((long long)pseq * p.num_q_heads + phead * G + gq) * g.slots + slot0 + 2 * t + (HALF ? 2 * (lg & 4) : 0);
      [[maybe_unused]] const int32_t* tok = MASKED ? p.slot_token + (long long)pseq * g.slots + slot0 : nullptr;
      [[maybe_unused]] const float* mrow = MASKED ? p.mask + (long long)pseq * p.mask_stride : nullptr;
      const int kplace = kslice_place<D, BITS>(lane), vplace = BITS == 3 ? 0 : vmatrix_place<D, BITS>(lane);

      auto tiles = [&](auto guard_tag) {
        constexpr bool GUARD = decltype(guard_tag)::value;
#pragma unroll 1
        for (int i = 0; i < pn; ++i) {
          cp_async_wait<S::STAGES - 2>();
          __syncwarp();  // every lane's copies have landed, and every lane is done with the slot the next copies take
          if (i + S::STAGES - 1 < pn) issue_more(std::integral_constant<int, RB>{}); else issue();
          const uint8_t* cs = ring + at;
          // ---- every shared-memory load of the scores up front -----------------------------------------------
          uint32_t kr0[SliceWords<D, BITS>::K], kr1[SliceWords<D, BITS>::K];
          [[maybe_unused]] uint32_t vr[4][2];
          if constexpr (BITS == 3) {
            load_kslice<D, BITS>(cs, lg, t, kr0);
            load_kslice<D, BITS>(cs, lg + 8, t, kr1);
            load_vrow<D, BITS>(cs + S::V_AT, 2 * t, lg, vr[0]);
            load_vrow<D, BITS>(cs + S::V_AT, 2 * t + 1, lg, vr[1]);
            load_vrow<D, BITS>(cs + S::V_AT, 2 * t + 8, lg, vr[2]);
            load_vrow<D, BITS>(cs + S::V_AT, 2 * t + 9, lg, vr[3]);
          } else {
            load_kslice_sw<D, BITS>(cs, kplace, kr0);
            load_kslice_sw<D, BITS>(cs + 8 * RB, kplace, kr1);
          }
          // ---- scores of head gq (log2 units).  x[0], x[1]: keys k0, k0 + 1; x[2], x[3]: keys k0 + 8, k0 + 9 (HALF: lanes
          // of the lower and of the upper row half hold one pair each)
          constexpr int NX = HALF ? 2 : 4;
          const int k0 = 2 * t + (HALF ? 2 * (lg & 4) : 0);
          const float4* sc = reinterpret_cast<const float4*>(cs + S::S_AT) + t + (HALF ? (lg & 4) : 0);
          float x[NX], vs[NX];
          if constexpr (I8) {
            int c0[4], c1[4];
            qk_stream<D, BITS>(kr0, qa, c0);
            qk_stream<D, BITS>(kr1, qa, c1);
            if constexpr (HALF) {
#pragma unroll
              for (int e = 0; e < 4; ++e) c0[e] = (lg & 4) ? c1[e] : c0[e];
            } else {
              x[2] = (float)(c1[0] * 128 + c1[2] + init);
              x[3] = (float)(c1[1] * 128 + c1[3] + init);
            }
            x[0] = (float)(c0[0] * 128 + c0[2] + init);
            x[1] = (float)(c0[1] * 128 + c0[3] + init);
          } else {
            float c0[4], c1[4];
            qk_ntile_f16<D, BITS>(kr0, t, qa, c0);
            qk_ntile_f16<D, BITS>(kr1, t, qa, c1);
            if constexpr (HALF) {
              x[0] = (lg & 4) ? c1[0] : c0[0];
              x[1] = (lg & 4) ? c1[1] : c0[1];
            } else {
              x[0] = c0[0];
              x[1] = c0[1];
              x[2] = c1[0];
              x[3] = c1[1];
            }
          }
#pragma unroll
          for (int e = 0; e < NX; e += 2) {
            const float4 s2 = sc[2 * e];  // (ks, vs) of two keys
            x[e] *= s2.x * qs;
            x[e + 1] *= s2.z * qs;
            vs[e] = s2.y;
            vs[e + 1] = s2.w;
          }
          if constexpr (MASKED) {
            // additive mask, indexed by the key's token id as the reference indexes it by the key's global slot
            // (smartkv/csrc/quantized_attention.cu:570-575); natural-log units -> log2 units
            constexpr float kLog2e = 1.4426950408889634f;
#pragma unroll
            for (int e = 0; e < NX; ++e) {
              const int key = k0 + (e & 1) + 4 * (e & 2);
              if (key < keys) {
                const int id = tok[key];
                if (id >= 0) x[e] = fmaf(mrow[id], kLog2e, x[e]);
              }
            }
            tok += 16;
          }
          if (keys < 16) {  // last tile of a bucket: rows past its end may hold anything, scales included
#pragma unroll
            for (int e = 0; e < NX; ++e) {
              if (k0 + (e & 1) + 4 * (e & 2) >= keys) {
                x[e] = -INFINITY;
                vs[e] = 0.f;
              }
            }
          }
          keys -= 16;
          if (lrow != nullptr) {
            *reinterpret_cast<float2*>(lrow) = make_float2(x[0], x[1]);
            if constexpr (!HALF) *reinterpret_cast<float2*>(lrow + 8) = make_float2(x[2], x[3]);
            lrow += 16;
          }
          float mx = fmaxf(x[0], x[1]);
          if constexpr (!HALF) mx = fmaxf(mx, fmaxf(x[2], x[3]));
          // The P operand of the P.V product is p * v_scale in fp16.  With p <= 2^kLazyTau it stays in range as long as the
          // V scale does not exceed kVScaleGuard; every kernel that writes a V scale records in the arena's footer when
          // one does, and only runs over such an arena pay for the test (GUARD), which raises the running maximum far
          // enough for the product to fit.
          bool slow = mx > st.m + kLazyTau;
          if constexpr (GUARD) {
#pragma unroll
            for (int e = 0; e < NX; ++e) slow = slow || vs[e] > kVScaleGuard;
          }
          if (__any_sync(0xffffffffu, slow)) {
            auto head_max = [&](float v) {
              v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
              v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
              if constexpr (HALF) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 16));
              return v;
            };
            float nm = fmaxf(st.m, head_max(mx));
            if constexpr (GUARD) {
              const float mu2 = (nm == -INFINITY) ? 0.f : nm;
              float am = 0.f;
#pragma unroll
              for (int e = 0; e < NX; ++e) am = fmaxf(am, ex2f(x[e] - mu2) * vs[e]);
              am = head_max(am);
              if (am > 16384.f) nm += ceilf(log2f(am)) - 14.f;  // am > 0 needs a finite score, so nm is finite here
            }
            const float alpha = (nm == -INFINITY) ? 1.f : ex2f(st.m - nm);
            st.l *= alpha;
            st.m = nm;
            // the accumulators of this lane belong to heads 2t and 2t+1, whose lanes are 8t.. and 8t+4..
            const float a0 = __shfl_sync(0xffffffffu, alpha, 8 * t), a1 = __shfl_sync(0xffffffffu, alpha, 8 * t + 4);
#pragma unroll
            for (int j = 0; j < D / 16; ++j) {
              o[j][0] *= a0;
              o[j][2] *= a0;
              o[j][1] *= a1;
              o[j][3] *= a1;
            }
          }
          const float mu = (st.m == -INFINITY) ? 0.f : st.m;
#pragma unroll
          for (int e = 0; e < NX; ++e) x[e] = ex2f(x[e] - mu);
          // P^T B fragments: keys (2t, 2t+1) and (2t+8, 2t+9) of head lg.  HALF: the lane 16 away holds the other pair;
          // columns 4..7 multiply it with the wrong keys and are never read.
          uint32_t pb0 = h2_bits(__floats2half2_rn(x[0] * vs[0], x[1] * vs[1])), pb1;
          if constexpr (HALF) {
            st.l += x[0] + x[1];
            pb1 = __shfl_xor_sync(0xffffffffu, pb0, 16);
          } else {
            st.l += (x[0] + x[1]) + (x[2] + x[3]);
            pb1 = h2_bits(__floats2half2_rn(x[2] * vs[2], x[3] * vs[3]));
          }
          if constexpr (BITS == 3) pv_stream3<D>(vr, lg, pb0, pb1, o);
          else pv_stream<D, BITS>(ring_at + at + S::V_AT + vplace, pb0, pb1, o);
          at = at + S::SLOT == S::RING ? 0 : at + S::SLOT;
        }
      };
      if ((guards >> (4 * prr)) & 1u) tiles(std::true_type{}); else tiles(std::false_type{});
      // The slot of the last tile is free until the next tile is issued: the accumulators go through it to the next width's
      // order or to the run's partial; those of the warp's last piece wait for the merge at the start of the ring (nothing is in
      // flight then).
      uint8_t* acc_at = ring + (todo == 0 ? 0 : at == 0 ? S::RING - S::SLOT : at - S::SLOT);
      __syncwarp();
      store_acc<D, BITS>(reinterpret_cast<float*>(acc_at), lane, o);
      __syncwarp();
      carry = reinterpret_cast<const float*>(acc_at);
    };

    while (todo != 0) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      switch (src & 3) {
        case 0: piece(std::integral_constant<int, 2>{}, src); break;
        case 1: piece(std::integral_constant<int, 3>{}, src); break;
        case 2: piece(std::integral_constant<int, 4>{}, src); break;
        default: piece(std::integral_constant<int, 8>{}, src); break;
      }
      const int prr = src >> 2;
      if (todo != 0 && (__ffs(todo) - 1) >> 2 == prr) continue;  // the run goes on in the next bucket
      float lsum = st.l;
      lsum += __shfl_xor_sync(0xffffffffu, lsum, 1);
      lsum += __shfl_xor_sync(0xffffffffu, lsum, 2);
      if constexpr (HALF) lsum += __shfl_xor_sync(0xffffffffu, lsum, 16);
      if (prr == tail) {
        if (t == 0 && lg == gq) {
          sh.tail_m[warp][gq] = st.m;
          sh.tail_l[warp][gq] = lsum;
        }
      } else {
        // the run ends here and this warp goes on: its piece is the run's second partial, or all of the run
        const bool whole = ((missing >> (4 * prr)) & 15u) == 0;
        float* out = p.partials + ((long long)(r0 + prr) * kF16PartialsPerRun + (whole ? 0 : 1)) * partial_stride(G, D);
        if (t == 0 && lg < G) *reinterpret_cast<float2*>(out + gq * (D + 2)) = make_float2(st.m, lsum);
        for (int h = 0; h < G; ++h)
          for (int d = 2 * lane; d < D; d += 64)
            *reinterpret_cast<float2*>(out + h * (D + 2) + 2 + d) = *reinterpret_cast<const float2*>(carry + h * kAccStride<D> + d);
        if (lane == 0) (whole ? sh.has_first : sh.has_second)[prr] = 1;
      }
      carry = nullptr;
      st.m = -INFINITY;
      st.l = 0.f;
      __syncwarp();
    }
    if (lane == 0) sh.tail_run[warp] = tail;
    cp_async_wait<0>();
    __syncthreads();

    // ---- merge: the warps whose last piece belongs to one run, in warp order ------------------------------------------------
    if (tid < WARPS * 8) {
      const int w = tid >> 3, h = tid & 7, run = sh.tail_run[w];
      float mi[WARPS], M = -INFINITY, L = 0.f, own = 0.f;
      int leader = WARPS;
#pragma unroll
      for (int i = 0; i < WARPS; ++i) {
        mi[i] = sh.tail_run[i] == run ? sh.tail_m[i][h] : -INFINITY;
        if (sh.tail_run[i] == run && i < leader) leader = i;
        M = fmaxf(M, mi[i]);
      }
#pragma unroll
      for (int i = 0; i < WARPS; ++i) {
        const float f = mi[i] == -INFINITY ? 0.f : ex2f(mi[i] - M);
        if (i == w) own = f;
        L += f == 0.f ? 0.f : sh.tail_l[i][h] * f;
      }
      if (run >= 0 && h < G && leader == w)
        *reinterpret_cast<float2*>(p.partials + (long long)(r0 + run) * kF16PartialsPerRun * partial_stride(G, D) + h * (D + 2)) =
            make_float2(M, L);
      sh.weight[w][h] = own;
      // A piece that does not count may hold anything (masked keys with an infinite V scale): it is cleared here, which is rare,
      // so that the sum below need not select (20 layers of 64 query heads on 8 KV heads, 15 x 930 keys: 520 us a step with a
      // select, 515 so; one that waits for the weight before it loads, 16 x 8192 keys: 1612 us against 1587).
      if (own == 0.f && run >= 0 && h < G) {
        float* acc = reinterpret_cast<float*>(smem + w * S::RING) + h * kAccStride<D>;
#pragma unroll 1
        for (int d = 0; d < D; ++d) acc[d] = 0.f;
      }
    }
    __syncthreads();
    const int tr = lane < WARPS ? sh.tail_run[lane] : -1;
    for (int run = 0; run < nr; ++run) {
      const unsigned who = __ballot_sync(0xffffffffu, tr == run);
      float* out = p.partials + (long long)(r0 + run) * kF16PartialsPerRun * partial_stride(G, D);
      if (who != 0) {
        for (int e = tid; e < G * D; e += WARPS * 32) {
          const int h = e / D, d = e - h * D;
          const float* acc_at = reinterpret_cast<const float*>(smem) + h * kAccStride<D> + d;
          float acc = 0.f;
#pragma unroll
          for (int w = 0; w < WARPS; ++w)
            if ((who >> w) & 1u) acc = fmaf(sh.weight[w][h], acc_at[w * (S::RING / 4)], acc);
          out[h * (D + 2) + 2 + d] = acc;
        }
      }
      // partials nobody wrote are marked empty
      for (int e = tid; e < kF16PartialsPerRun * G; e += WARPS * 32) {
        const int s = e / G, h = e - s * G;
        const bool written = s == 0 ? (who != 0 || sh.has_first[run]) : s == 1 ? sh.has_second[run] != 0 : false;
        if (!written) *reinterpret_cast<float2*>(out + (long long)s * partial_stride(G, D) + h * (D + 2)) = make_float2(-INFINITY, 0.f);
      }
    }
    if (r0 + kGroupRuns < run_end) __syncthreads();  // the rings and the query rows are used again
  }
}

template <int D, bool MASKED, bool HALF>
static int launch_f16(const AttnParams& p, cudaStream_t st) {
  static bool configured[64] = {};  // per template instance and device: the attribute belongs to the device's context
  constexpr int WARPS = StreamShape<D>::WARPS;
  constexpr size_t smem = (size_t)WARPS * StreamShape<D>::RING + sizeof(StreamShared<D>);
  static_assert(smem <= 232448, "more shared memory than a CTA can have");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return SKV_ERR_CUDA;
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    const cudaError_t rc =
        cudaFuncSetAttribute(decode_attn_f16_kernel<D, MASKED, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (rc != cudaSuccess) {
      fprintf(stderr, "skv_decode_attention: cannot reserve %zu bytes of shared memory: %s\n", smem, cudaGetErrorString(rc));
      return SKV_ERR_CUDA;
    }
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  const int mode = g_dependent_launch.load();
  launch_maybe_dependent(decode_attn_f16_kernel<D, MASKED, HALF>, dim3(p.num_ctas), dim3(WARPS * 32), smem, st, p,
                         p.dependent != 0 && (mode == 1 || mode == 2));
  const cudaError_t rc = cudaGetLastError();
  if (rc != cudaSuccess) {
    fprintf(stderr, "skv_decode_attention: launch failed: %s\n", cudaGetErrorString(rc));
    return SKV_ERR_CUDA;
  }
  return SKV_OK;
}

template <int D>
static int launch_f16_head_dim(const AttnParams& p, cudaStream_t st) {
  if (p.group <= 4) return p.mask != nullptr ? launch_f16<D, true, true>(p, st) : launch_f16<D, false, true>(p, st);
  return p.mask != nullptr ? launch_f16<D, true, false>(p, st) : launch_f16<D, false, false>(p, st);
}
int launch_attn_f16(const AttnParams& p, cudaStream_t st) {
  return p.g.head_dim == 128 ? launch_f16_head_dim<128>(p, st) : launch_f16_head_dim<64>(p, st);
}

}  // namespace skv
