// Causal self-attention over the unquantised prompt (more than one query token against an empty
// cache), with the per-key attention mass the importance tracker needs -- without ever writing the
// [batch, heads, queries, keys] probability tensor to memory.
//
//   pass 1 (prefill_fwd_kernel): streaming softmax, S = Q K^T, running max / sum, O += P V; writes O
//       (fp16) and, per query row, the log-sum-exp in base-2 units.
//   pass 2 (prefill_mass_kernel): the transposed product S^T = K Q^T per (128-key tile, KV head,
//       sequence) over every query tile at or after the key tile and every query head of the group;
//       with the row normalisers of pass 1, p = exp2(s - lse[q]) is final, and its sum over the
//       queries, weighted by the head weight, is the key's mass.  One value per (sequence, KV head,
//       key) is written; the caller adds the KV heads (a fixed order, so the result is reproducible).
//
// What bounds both: the exponentials.  A 128 x 128 tile has 16384 of them, 1024 cycles of an SM's 16-a-cycle
// unit; its products take 1024 cycles (pass 1, head_dim 128), 512 (pass 1 at 64, pass 2 at 128) or 256 cycles of the
// tensor core.  So the products run on tcgen05 (fp16 in, fp32 accumulators in tensor memory) from TMA-fetched
// tiles, issued by one lane, and a thread is left with half a query row (pass 2: a key row): no shuffle, no
// shared-memory traffic for S or P.  P goes back to tensor memory as the A operand of P V (fp16, as everywhere
// here), over the columns its S came from.
//
// Both kernels are persistent, one CTA per SM: four softmax warpgroups, one loading warp, one warp that issues the MMAs.
// A warp's own work is a chain (wait, read S, maximum, exponentials, write P), so it takes four warps per scheduler to
// keep the exponential unit busy.  While O was still rescaled only when a maximum had grown by 2^8, at 8192 tokens: with two warps,
// each thread owning a whole row, the unit was 44 % busy in pass 1 (651 us) and 76 % in pass 2 (389 us), with four 51 %
// (577 us) and 86 % (357 us).  One warp issues the MMAs of both tiles in turn; in those
// builds, with one per tile both waited for the tensor core and then both for the exponential unit (pass 1 792 us), and 64-key
// blocks with scores two blocks ahead ended up in the same lockstep (770 us).  Part of the exponentials as a polynomial on
// the multiply-add pipe costs more issue time than it saves (10 to 20 % slower).
// Pass 1 gives each pair of warpgroups its own 128-query tile, 64 keys to a thread, so that one pair computes exponentials
// while the tensor core works for the other: two query heads of one KV head at the same positions where the group is
// even (they share every K and V tile and have the same causal range), otherwise two neighbouring query tiles of one
// head.  Pass 2 hands the query tiles of the stream to the warpgroups in turn, each with its own accumulator.  Units of
// work are dealt longest first, back and forth over the CTAs, because a causal unit's length is proportional to its position.
//
// Both passes together, B200: one sequence of 8192 tokens, 32 / 8 heads, head_dim 128: 1004 us (4315 us with 64 x 64 tiles on
// mma.sync); 8 x 512 tokens, 32 / 4 heads, head_dim 64: 64 us (223 us).  Pass 1 alone, 3 x 1391 tokens, 32 / 8 heads,
// head_dim 128: 78 us (289 us).
#include <cuda_fp16.h>

#include "f32x2.cuh"
#include "tc05.cuh"

namespace skv {

constexpr int kPfTile = 128;                 // queries per tile and keys per streamed tile
constexpr int kPfSoftmaxThreads = 512;       // four warpgroups
constexpr int kPfLoadWarp = kPfSoftmaxThreads / 32, kPfMmaWarp = kPfLoadWarp + 1;
constexpr int kPfThreads = kPfSoftmaxThreads + 64;  // + the loading warp and the MMA warp
constexpr uint32_t kPfTmemCols = 512;

struct PrefillTensor {
  const __half* base;
  long long sb, st, sh;  // element strides of batch, token, head (head_dim is contiguous)
  int mul_h, mul_b;      // 0: the map has no such dimension (one entry, or the same data for all of them)
  int by_rows;           // the map cannot express the strides: the loading warp copies row by row
};

struct PrefillParams {
  PrefillTensor q, k, v;
  __half* out;                 // [batch][tokens][q heads][head_dim]
  float* lse;                  // [batch][q heads][tokens], base-2
  const float* head_w;         // [batch][q heads] or null
  float* mass;                 // [batch][kv heads][tokens]
  int batch, tokens, num_q_heads, num_kv_heads;
  int tiles;                   // 128-token tiles of a sequence
  int units;
  float scale_log2;
  unsigned wait_cycles;        // limit of every wait, at most 2^31
  int32_t* err;                // set to 1 when a wait runs out (may be null)
};

template <int D>
struct PfCfg {
  static constexpr int kTileBytes = kPfTile * D * 2;
  static constexpr int kStages = D == 128 ? 4 : 6;
  static constexpr uint32_t kFwdSmem = (kStages + 2) * kTileBytes + 1024 + 2 * 2 * 2 * kPfTile * 4 + 256;
  static constexpr uint32_t kMassSmem = (kStages + 1) * kTileBytes + 1024 + 8 * 136 * 4 + 2 * 3 * kPfTile * 4 + 448;
};

__device__ __forceinline__ float pf_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pf_pack_half2(float lo, float hi) {
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}
// max(a, b, c); a NaN loses against a number, as in fmaxf
__device__ __forceinline__ float pf_max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ uint64_t pf_exp2_pair(uint64_t x2) {
  const float2 x = f32x2_parts(x2);
  return f32x2(pf_exp2(x.x), pf_exp2(x.y));
}

// Bounded wait: the thread is suspended inside try_wait; after the limit, or once another role gave up, it returns false.  A CTA that
// gives up sets the error flag, writes NaN to the rows it still owed, waits for its copies and MMAs in flight, frees its tensor
// memory and ends.  With a limit of no cycles the MMA warp does so on the first tile that is not there at once.
struct PfGiveUp {  // in shared memory, so that the call takes no registers from the callers
  int32_t* err;
  unsigned cycles;
  int flag;
};
__device__ __noinline__ bool pf_wait_slow(uint64_t* bar, uint32_t parity, PfGiveUp* give_up) {
  if (mbar_test_wait(bar, parity)) return true;
  volatile int* flag = &give_up->flag;
  const unsigned t0 = (unsigned)clock();
  while ((unsigned)clock() - t0 < give_up->cycles) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*flag) return false;
  }
  *flag = 1;
  if (give_up->err) atomicExch(give_up->err, 1);
  return false;
}
__device__ __forceinline__ bool pf_wait(uint64_t* bar, uint32_t parity, PfGiveUp* give_up) {
  return mbar_try_wait(bar, parity) || pf_wait_slow(bar, parity, give_up);
}
__device__ __forceinline__ bool pf_wait_unit(uint64_t* bar, uint32_t parity, PfGiveUp* give_up, unsigned cycles) {
  return (cycles > 0 && mbar_try_wait(bar, parity)) || pf_wait_slow(bar, parity, give_up);
}

// Waits, bounded, for what this CTA itself has in flight, whatever the limit of the other waits.
__device__ __forceinline__ void pf_drain(uint64_t* bar, uint32_t parity) {
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity) && clock64() - t0 < 1000000000ll) {}
}

// The unit a CTA takes in its `round`-th turn (-1: none left): back and forth, so that whoever got the longest unit of
// one round gets the shortest of the next.
__device__ __forceinline__ int pf_unit(int round, int units) {
  const int grid = (int)gridDim.x, c = (int)blockIdx.x;
  const long long u = (long long)round * grid + ((round & 1) ? grid - 1 - c : c);
  return u < units ? (int)u : -1;
}

// One 128-row tile of a strided [tokens][D] matrix into shared memory as K-major 128-byte swizzled blocks of 64 columns
// ([D / 64][128 rows][128 B], rows at or beyond `tokens` zero).  Whole warp; `bar` must have been armed for the bytes when
// the tile goes through the map.
template <int D>
__device__ __forceinline__ void pf_load_tile(uint8_t* dst, const CUtensorMap* map, const PrefillTensor& t, int row0, int h, int b,
                                             int tokens, uint64_t* bar, int lane) {
  if (!t.by_rows) {
    if (lane == 0) {
#pragma unroll
      for (int c = 0; c < D / 64; ++c)
        tma_load_4d(dst + c * (kPfTile * 128), map, c * 64, row0, h * t.mul_h, b * t.mul_b, bar);
    }
    return;
  }
  constexpr int CH = D / 8;  // 16-byte chunks per row
  const __half* src = t.base + b * t.sb + h * t.sh;
  for (int i = lane; i < kPfTile * CH; i += 32) {
    const int r = i / CH, c = i % CH;
    uint4 val = make_uint4(0u, 0u, 0u, 0u);
    if (row0 + r < tokens) val = *reinterpret_cast<const uint4*>(src + (long long)(row0 + r) * t.st + c * 8);
    *reinterpret_cast<uint4*>(dst + (c >> 3) * (kPfTile * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = val;
  }
  fence_proxy_async();  // the MMAs read the tile through the async proxy
  __syncwarp();
}
template <int D>
__device__ __forceinline__ uint32_t pf_tile_tx(const PrefillTensor& t) {
  return t.by_rows ? 0u : (uint32_t)PfCfg<D>::kTileBytes;
}

// Low words of the matrix descriptors: start address in 16-byte units, below the leading byte offset (unused by K-major
// swizzled tiles; between the 64-column blocks of a V tile).  The high word is the same for all tiles here.
__device__ __forceinline__ uint32_t pf_desc_k(uint32_t smem_addr) { return (smem_addr >> 4) | (1u << 16); }
__device__ __forceinline__ uint32_t pf_desc_v(uint32_t smem_addr) { return (smem_addr >> 4) | ((uint32_t)(kPfTile * 128 / 16) << 16); }

// S = A B^T over head_dim, both K-major: one 16-column step per instruction
template <int D>
__device__ __forceinline__ void pf_issue_scores(uint32_t d_tmem, uint32_t a_desc, uint32_t b_desc) {
  constexpr uint32_t idesc = idesc_f16(0, 0, 128, 128);
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) {
    const uint32_t off = ((kk / 4) * (kPfTile * 128) + (kk % 4) * 32) >> 4;
    if (kk == 0) mma_f16_ss_sw128<false>(d_tmem, a_desc + off, b_desc + off, idesc);
    else mma_f16_ss_sw128<true>(d_tmem, a_desc + off, b_desc + off, idesc);
  }
}

// Of the tile's rows 32 g .. 32 g + 31, those before row 16 kk, as a bit mask.
__device__ __forceinline__ constexpr uint32_t pf_rows_before(int kk, int g) {
  return kk >= 2 * g + 2 ? 0xffffffffu : kk == 2 * g + 1 ? 0x0000ffffu : 0u;
}

struct PfFwdUnit {
  int tile[2], head[2], blocks[2];  // per warpgroup: query tile, query head, key tiles (0: nothing to do)
  int hk, b;
};
__device__ __forceinline__ PfFwdUnit pf_fwd_unit(const PrefillParams& p, int u) {
  PfFwdUnit r;
  const int G = p.num_q_heads / p.num_kv_heads;
  if ((G & 1) == 0) {
    const int pairs = p.num_q_heads >> 1, per = pairs * p.batch;
    const int t = p.tiles - 1 - u / per, rest = u % per;
    r.b = rest / pairs;
    const int h = 2 * (rest % pairs);
    r.tile[0] = r.tile[1] = t;
    r.head[0] = h;
    r.head[1] = h + 1;
    r.blocks[0] = r.blocks[1] = t + 1;
    r.hk = h / G;
  } else {
    const int per = p.num_q_heads * p.batch;
    const int t = (p.tiles + 1) / 2 - 1 - u / per, rest = u % per;
    r.b = rest / p.num_q_heads;
    const int h = rest % p.num_q_heads;
    r.tile[0] = 2 * t;
    r.tile[1] = 2 * t + 1;
    r.head[0] = r.head[1] = h;
    r.blocks[0] = 2 * t + 1;
    r.blocks[1] = 2 * t + 1 < p.tiles ? 2 * t + 2 : 0;
    r.hk = h / G;
  }
  return r;
}

struct PfFwdBars {
  uint64_t full[6], empty[6];
  uint64_t qfull, qempty;
  uint64_t sfull[2], pready[2], oready[2];
  uint64_t drain;
  uint32_t tmem_base;
  PfGiveUp give_up;
};

template <int D>
__global__ void __launch_bounds__(kPfThreads, 1)
    prefill_fwd_kernel(const __grid_constant__ PrefillParams p, const __grid_constant__ CUtensorMap qmap,
                       const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap) {
  using Cfg = PfCfg<D>;
  constexpr int NS = Cfg::kStages, TB = Cfg::kTileBytes;
  extern __shared__ uint8_t pf_smem_raw[];
  uint8_t* smem = pf_smem_raw + ((1024u - (smem_u32(pf_smem_raw) & 1023u)) & 1023u);  // swizzle atoms are 1024 bytes
  uint8_t* ring = smem;                    // [NS][TB]: K and V tiles in the order they are used
  uint8_t* qs = ring + NS * TB;            // [2][TB]
  float* xch = reinterpret_cast<float*>(qs + 2 * TB);  // [2 (step)][2 (tile)][2 (half)][128]: what the halves of a row tell each other
  PfFwdBars& br = *reinterpret_cast<PfFwdBars*>(xch + 8 * kPfTile);
  static_assert(sizeof(PfFwdBars) <= 256, "barrier block");
  PfGiveUp* give_up = &br.give_up;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);

  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      mbar_init(&br.full[s], 1);
      mbar_init(&br.empty[s], 1);
    }
    mbar_init(&br.qfull, 1);
    mbar_init(&br.qempty, 1);
    for (int w = 0; w < 2; ++w) {
      mbar_init(&br.sfull[w], 1);
      mbar_init(&br.pready[w], 8);  // one arrival per warp
      mbar_init(&br.oready[w], 1);
    }
    mbar_init(&br.drain, 1);
    br.give_up = {p.err, p.wait_cycles, 0};
    mbar_fence_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(&br.tmem_base, kPfTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, br.tmem_base, 0);  // columns: S_0 S_1 (128 each), O_0 O_1 (D each)

  if (warp == kPfLoadWarp) {
    // ================================ loading warp ================================
    int i = 0, last_unit = -1;
    bool ok = true;
    auto stage = [&](const CUtensorMap* map, const PrefillTensor& t, int row0, int h, int b) {
      const int s = i % NS;
      ok = pf_wait(&br.empty[s], ((i / NS) & 1) ^ 1u, give_up);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return;
      const uint32_t tx = pf_tile_tx<D>(t);
      if (tx && lane == 0) mbar_expect_tx(&br.full[s], tx);
      pf_load_tile<D>(ring + s * TB, map, t, row0, h, b, p.tokens, &br.full[s], lane);
      if (!tx && lane == 0) mbar_arrive(&br.full[s]);
      ++i;
    };
    for (int round = 0; ok; ++round) {
      const int u = pf_unit(round, p.units);
      if (u < 0) break;
      const PfFwdUnit un = pf_fwd_unit(p, u);
      ok = __all_sync(0xffffffffu, pf_wait(&br.qempty, (round & 1) ^ 1u, give_up));
      if (!ok) break;
      const int nq = un.blocks[1] > 0 ? 2 : 1;
      const uint32_t tx = pf_tile_tx<D>(p.q) * nq;
      if (tx && lane == 0) mbar_expect_tx(&br.qfull, tx);
      for (int w = 0; w < nq; ++w)
        pf_load_tile<D>(qs + w * TB, &qmap, p.q, un.tile[w] * kPfTile, un.head[w], un.b, p.tokens, &br.qfull, lane);
      if (!tx && lane == 0) mbar_arrive(&br.qfull);
      last_unit = round;
      const int blocks = max(un.blocks[0], un.blocks[1]);
      for (int j = 0; ok && j < blocks; ++j) {
        stage(&kmap, p.k, j * kPfTile, un.hk, un.b);
        if (ok) stage(&vmap, p.v, j * kPfTile, un.hk, un.b);
      }
    }
    // No copy in flight may outlive the shared memory it targets.  Usually every copy has been waited for by whoever uses it, but
    // another role may have given up after this one issued its last.
    for (int s = 0; s < NS; ++s) {
      const int cnt = i > s ? (i - 1 - s) / NS + 1 : 0;
      if (cnt > 0) pf_drain(&br.full[s], (cnt - 1) & 1);
    }
    if (last_unit >= 0) pf_drain(&br.qfull, last_unit & 1);
  } else if (warp == kPfMmaWarp) {
    // ================================ MMA warp ================================
    // The whole warp walks the loop and one elected lane issues, so that addresses and descriptors are warp-uniform values:
    // computed by a single lane they cost the issuing thread more than the instruction itself.
    int base = 0;                 // ring index of the unit's first K tile
    int pc[2] = {0, 0};           // P blocks taken from each tile so far
    bool ok = true;
    const uint32_t ring_d = smem_u32(ring) >> 4, qs_a = smem_u32(qs);
    constexpr uint32_t pv_idesc = idesc_f16(0, 1, 128, D);
    for (int round = 0; ok; ++round) {
      const int u = pf_unit(round, p.units);
      if (u < 0) break;
      const PfFwdUnit un = pf_fwd_unit(p, u);
      const int blocks = max(un.blocks[0], un.blocks[1]);
      ok = __all_sync(0xffffffffu, pf_wait_unit(&br.qfull, round & 1, give_up, p.wait_cycles));
      // step j: P V of block j-1, then the scores of block j, for one tile and then the other
      for (int j = 0; ok && j <= blocks; ++j) {
        const int ik = base + 2 * j, iv = ik - 1;
        const int sk = ik % NS, sv = (iv + NS) % NS;
        if (j < blocks) ok = pf_wait(&br.full[sk], (ik / NS) & 1, give_up);
        if (ok && j > 0) ok = pf_wait(&br.full[sv], (iv / NS) & 1, give_up);
        ok = __all_sync(0xffffffffu, ok);
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          if (ok && j > 0 && j - 1 < un.blocks[w]) {
            ok = __all_sync(0xffffffffu, pf_wait(&br.pready[w], pc[w] & 1, give_up));
            if (!ok) break;
            ++pc[w];
            tc_fence_after();
            if (elect_one()) {
              const uint32_t vd = pf_desc_v((ring_d << 4) + sv * TB);
              const uint32_t od = tmem + 256 + w * D, pd = tmem + w * 128;
              auto p_at = [&](int kk) { return pd + (kk / 4) * 64 + (kk % 4) * 8; };
              // V rows are the contraction: MN-major, 64-column blocks 16 KB apart
              if (j > 1) mma_f16_ts_sw128<true>(od, pd, vd, pv_idesc);
              else mma_f16_ts_sw128<false>(od, pd, vd, pv_idesc);
              if (j < un.blocks[w]) {
#pragma unroll
                for (int kk = 1; kk < kPfTile / 16; ++kk) mma_f16_ts_sw128<true>(od, p_at(kk), vd + kk * 128, pv_idesc);
              } else {
                // In the diagonal block the queries before a step's 16 keys leave it out: their P there is zero, but zero times an
                // infinite or NaN value is not.
#pragma unroll
                for (int kk = 1; kk < kPfTile / 16; ++kk)
                  mma_f16_ts_sw128_lanes(od, p_at(kk), vd + kk * 128, pv_idesc, pf_rows_before(kk, 0), pf_rows_before(kk, 1),
                                         pf_rows_before(kk, 2), pf_rows_before(kk, 3));
                mma_commit(&br.oready[w]);
              }
            }
            __syncwarp();
          }
          if (ok && j < un.blocks[w]) {
            // the S columns hold P of the block before; its P V was issued first by this warp's one lane, and MMAs run in order
            if (elect_one()) {
              pf_issue_scores<D>(tmem + w * 128, pf_desc_k(qs_a + w * TB), pf_desc_k((ring_d << 4) + sk * TB));
              mma_commit(&br.sfull[w]);
            }
            __syncwarp();
          }
        }
        if (!ok) break;
        if (elect_one()) {
          if (j > 0) mma_commit(&br.empty[sv]);
          if (j < blocks) mma_commit(&br.empty[sk]);
          if (j == blocks - 1) mma_commit(&br.qempty);
        }
        __syncwarp();
      }
      base += 2 * blocks;
    }
    if (elect_one()) {
      mma_commit(&br.drain);
      pf_drain(&br.drain, 0);
    }
    __syncwarp();
  } else {
    // ================================ softmax warpgroups: half a query row per thread ================================
    const int wg = warp >> 3, half = (warp >> 2) & 1, wq = warp & 3;  // tile, half of the keys, lane quarter of tensor memory
    const uint32_t lanes = (uint32_t)(wq * 32) << 16;
    const uint32_t ts = tmem + wg * 128 + lanes, to = tmem + 256 + wg * D + half * (D / 2) + lanes;
    const float sc = p.scale_log2;
    const uint64_t sc2 = f32x2(sc, sc);
    const int n = p.tokens;
    int sn = 0, on = 0, xp = 0;  // score tiles / outputs received so far; parity of the exchange buffer
    bool ok = true;
    // the other half's value of the same row (all 256 threads of the tile)
    auto exchange = [&](float v) -> float {
      float* x = xch + ((xp * 2 + wg) * 2) * kPfTile + wq * 32 + lane;
      x[half * kPfTile] = v;
      if (wg == 0) asm volatile("bar.sync 1, 256;" ::: "memory");
      else asm volatile("bar.sync 2, 256;" ::: "memory");
      xp ^= 1;
      return x[(half ^ 1) * kPfTile];
    };
    // The two tiles compute their exponentials in turn (tile 0 first): left alone they drift into step, both at the
    // exponential unit and then both waiting for the tensor core (both passes at 8192 tokens, together with the MMA warp's uniform
    // addresses and while O was rescaled at 2^8: 985 us, 949 with the turns).
    // Each turn is one pass of both through two named barriers, the same number for both tiles whatever they have to do.
    auto turn_wait = [&] {
      if (wg == 0) asm volatile("bar.sync 3, 512;" ::: "memory");
      else asm volatile("bar.sync 4, 512;" ::: "memory");
    };
    auto turn_pass = [&] {
      if (wg == 0) asm volatile("bar.arrive 4, 512;" ::: "memory");
      else asm volatile("bar.arrive 3, 512;" ::: "memory");
    };
    if (wg == 1) turn_pass();
    for (int round = 0;; ++round) {
      const int u = pf_unit(round, p.units);
      if (u < 0) break;
      const PfFwdUnit un = pf_fwd_unit(p, u);
      const int blocks = un.blocks[wg], turns = max(un.blocks[0], un.blocks[1]);
      const int row = un.tile[wg] * kPfTile + wq * 32 + lane;
      float m = -INFINITY, l = 0.f;  // the row's maximum and sum so far
      for (int j = 0; j < turns; ++j) {
        if (j >= blocks) {  // the other tile's longer unit
          turn_wait();
          turn_pass();
          continue;
        }
        if (ok) ok = __all_sync(0xffffffffu, pf_wait(&br.sfull[wg], sn & 1, give_up));
        ++sn;
        // In the diagonal block a warp's rows see nothing of the 32-key chunks after its own and, in its own, the keys up to
        // the row's position (keys beyond the prompt lie behind those).
        const bool diag = j == blocks - 1;
        const int own = diag ? wq - 2 * half : 2;  // chunks of this half before it are visible in full, the one at it in part
        tc_fence_after();
        // 64 values would not fit beside everything else in the 96 registers a thread has, so the second 32 are read twice, 16 at a
        // time: for the maximum, and again for the exponentials.
        uint32_t s0[16], s1[16], t[16];
        float bm = -INFINITY;
        auto mask_own = [&](uint32_t (&s)[16], int first) {
#pragma unroll
          for (int e = 0; e < 16; ++e)
            if (first + e > lane) s[e] = 0xff800000u;
        };
        auto piece_max = [&](const uint32_t (&s)[16]) {
          float b0 = -INFINITY;
#pragma unroll
          for (int e = 0; e < 16; e += 4) {
            b0 = pf_max3(b0, __uint_as_float(s[e]), __uint_as_float(s[e + 1]));
            bm = pf_max3(bm, __uint_as_float(s[e + 2]), __uint_as_float(s[e + 3]));
          }
          bm = fmaxf(bm, b0);
        };
        const uint32_t th = ts + half * 64;
        if (ok) {
          tmem_ld16(th + 32, t);
          tmem_ld16(th, s0);
          tmem_ld16(th + 16, s1);
          tmem_ld_wait(t);
          tmem_ld_wait(s0);
          tmem_ld_wait(s1);
          if (own >= 1) {
            if (own == 1) mask_own(t, 0);
            piece_max(t);
          }
          tmem_ld16(th + 48, t);
          if (own >= 0) {
            if (own == 0) {
              mask_own(s0, 0);
              mask_own(s1, 16);
            }
            piece_max(s0);
            piece_max(s1);
          }
          tmem_ld_wait(t);
          if (own >= 1) {
            if (own == 1) mask_own(t, 16);
            piece_max(t);
          }
        }
        bm = fmaxf(bm, exchange(bm));
        if (!ok) {  // the other warps still need this one at the barriers
          turn_wait();
          turn_pass();
          continue;
        }
        if (j == 0) {
          m = bm;
        } else {
          // O is rescaled whenever a row's maximum grows, however little.  Waiting until it has grown by 2^8 is 4 % faster
          // (949 against 991 us when it was changed, both passes at 8192 tokens), but then the row's largest P is no longer exactly 1, and its
          // rounding to fp16 (it is the weight that counts) makes the output's error against 64 bits 10 % larger.  Both
          // halves of a row decide alike; the round trip of O mostly fits in the wait for the turn.
          const bool need = bm > m;
          if (__any_sync(0xffffffffu, need)) {
            // the exponentials are taken against the maximum times the scale rounded to fp32, so the factor is that of the rounded
            // numbers (and the log-sum-exp below uses it): otherwise the key mass is off by up to 2^-24 of the logit
            const float f = need ? pf_exp2(__fmul_rn(m, sc) - __fmul_rn(bm, sc)) : 1.f;
            if (need) m = bm;
            l *= f;
#pragma unroll 1
            for (int c = 0; c < D / 64; ++c) {  // P V of the block before is complete: this block's scores came after it
              uint32_t o[32];
              tmem_ld32(to + c * 32, o);
              tmem_ld_wait(o);
#pragma unroll
              for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
              tmem_st32(to + c * 32, o);
            }
          }
        }
        turn_wait();
        const float msc = m == -INFINITY ? 0.f : __fmul_rn(m, sc);
        const uint64_t nm2 = f32x2(-msc, -msc);
        uint64_t l2a = 0, l2b = 0;
        // P of a half lies over that half's own S columns, of which the ones written have been read.
        auto piece_exp = [&](const uint32_t (&s)[16], bool seen, uint32_t to_col) {
          uint32_t pk[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            if (!seen) {  // this warp's rows see none of these keys
              pk[e] = 0u;
              continue;
            }
            const uint64_t x2 = f32x2_fma(f32x2(__uint_as_float(s[2 * e]), __uint_as_float(s[2 * e + 1])), sc2, nm2);
            const uint64_t p2 = pf_exp2_pair(x2);
            if (e & 1) l2b = f32x2_add(l2b, p2);
            else l2a = f32x2_add(l2a, p2);
            const float2 x = f32x2_parts(p2);
            pk[e] = pf_pack_half2(x.x, x.y);
          }
          tmem_st8(to_col, pk);
        };
        tmem_ld16(th + 32, t);
        piece_exp(s0, own >= 0, th);
        tmem_ld_wait(t);
        if (own == 1) mask_own(t, 0);
        tmem_ld16(th + 48, s0);
        piece_exp(s1, own >= 0, th + 8);
        piece_exp(t, own >= 1, th + 16);
        tmem_ld_wait(s0);
        if (own == 1) mask_own(s0, 16);
        piece_exp(s0, own >= 1, th + 24);
        turn_pass();
        const float2 l2 = f32x2_parts(f32x2_add(l2a, l2b));
        l += l2.x + l2.y;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&br.pready[wg]);
      }
      if (blocks == 0) continue;
      l += exchange(l);
      float inv = l > 0.f ? 1.f / l : 0.f, ls = __fadd_rn(__fmul_rn(m, sc), log2f(l));
      if (ok) ok = __all_sync(0xffffffffu, pf_wait(&br.oready[wg], on & 1, give_up));
      ++on;
      tc_fence_after();
      if (!ok) inv = ls = __int_as_float(0x7fffffff);
      if (row < n && half == 0) p.lse[((long long)un.b * p.num_q_heads + un.head[wg]) * n + row] = ls;
      __half* ob = p.out + (((long long)un.b * n + row) * p.num_q_heads + un.head[wg]) * D + half * (D / 2);
#pragma unroll
      for (int c = 0; c < D / 64; ++c) {
        uint32_t o[32];
        tmem_ld32(to + c * 32, o);
        tmem_ld_wait(o);
        if (row < n) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            uint4 w4;
            w4.x = pf_pack_half2(__uint_as_float(o[8 * e]) * inv, __uint_as_float(o[8 * e + 1]) * inv);
            w4.y = pf_pack_half2(__uint_as_float(o[8 * e + 2]) * inv, __uint_as_float(o[8 * e + 3]) * inv);
            w4.z = pf_pack_half2(__uint_as_float(o[8 * e + 4]) * inv, __uint_as_float(o[8 * e + 5]) * inv);
            w4.w = pf_pack_half2(__uint_as_float(o[8 * e + 6]) * inv, __uint_as_float(o[8 * e + 7]) * inv);
            *reinterpret_cast<uint4*>(ob + c * 32 + e * 8) = w4;
          }
        }
      }
      tc_fence_before();  // O has been read: the arrival on the next unit's first P orders it before the next P V
    }
    if (wg == 0) turn_wait();  // the last turn handed back
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, kPfTmemCols);
}

constexpr int kPfLseSlots = 8;
constexpr int kPfAcc = 4;  // score accumulators in tensor memory, one per warpgroup

struct PfMassBars {
  uint64_t full[6], empty[6];
  uint64_t kfull, kempty;
  uint64_t sfull[kPfAcc], sempty[kPfAcc];
  uint64_t lfull[kPfLseSlots], lempty[kPfLseSlots];
  uint64_t drain;
  uint32_t tmem_base;
  PfGiveUp give_up;
};

struct PfMassUnit {
  int kt, hk, b, count;  // key tile, KV head, sequence, query tiles in the stream
};
__device__ __forceinline__ PfMassUnit pf_mass_unit(const PrefillParams& p, int u) {
  PfMassUnit r;
  const int per = p.num_kv_heads * p.batch, rest = u % per;
  r.kt = u / per;  // the first key tile sees the most queries
  r.b = rest / p.num_kv_heads;
  r.hk = rest % p.num_kv_heads;
  r.count = (p.tiles - r.kt) * (p.num_q_heads / p.num_kv_heads);
  return r;
}

template <int D>
__global__ void __launch_bounds__(kPfThreads, 1)
    prefill_mass_kernel(const __grid_constant__ PrefillParams p, const __grid_constant__ CUtensorMap qmap,
                        const __grid_constant__ CUtensorMap kmap) {
  using Cfg = PfCfg<D>;
  constexpr int NS = Cfg::kStages, TB = Cfg::kTileBytes, LS = 136;  // floats per lse slot: 128 + the head weight, 16-byte rows
  extern __shared__ uint8_t pf_smem_raw[];
  uint8_t* smem = pf_smem_raw + ((1024u - (smem_u32(pf_smem_raw) & 1023u)) & 1023u);
  uint8_t* ring = smem;                                            // [NS][TB]: query tiles
  uint8_t* ks = ring + NS * TB;                                    // the unit's key tile
  float* lse_s = reinterpret_cast<float*>(ks + TB);                // [kPfLseSlots][LS], negated
  float* red = lse_s + kPfLseSlots * LS;                           // [2][3][128]: the sums of the warpgroups but the first
  PfMassBars& br = *reinterpret_cast<PfMassBars*>(red + 2 * 3 * kPfTile);
  static_assert(sizeof(PfMassBars) <= 448, "barrier block");
  PfGiveUp* give_up = &br.give_up;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int G = p.num_q_heads / p.num_kv_heads, n = p.tokens;

  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      mbar_init(&br.full[s], 1);
      mbar_init(&br.empty[s], 1);
    }
    mbar_init(&br.kfull, 1);
    mbar_init(&br.kempty, 1);
    for (int s = 0; s < kPfAcc; ++s) {
      mbar_init(&br.sfull[s], 1);
      mbar_init(&br.sempty[s], 4);  // one arrival per warp of the warpgroup that takes the tile
    }
    for (int s = 0; s < kPfLseSlots; ++s) {
      mbar_init(&br.lfull[s], 1);
      mbar_init(&br.lempty[s], 4);
    }
    mbar_init(&br.drain, 1);
    br.give_up = {p.err, p.wait_cycles, 0};
    mbar_fence_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(&br.tmem_base, kPfTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, br.tmem_base, 0);

  if (warp == kPfLoadWarp) {
    // ================================ loading warp ================================
    int i = 0, last_unit = -1;
    bool ok = true;
    for (int round = 0; ok; ++round) {
      const int u = pf_unit(round, p.units);
      if (u < 0) break;
      const PfMassUnit un = pf_mass_unit(p, u);
      ok = __all_sync(0xffffffffu, pf_wait(&br.kempty, (round & 1) ^ 1u, give_up));
      if (!ok) break;
      const uint32_t ktx = pf_tile_tx<D>(p.k), qtx = pf_tile_tx<D>(p.q);
      if (ktx && lane == 0) mbar_expect_tx(&br.kfull, ktx);
      pf_load_tile<D>(ks, &kmap, p.k, un.kt * kPfTile, un.hk, un.b, n, &br.kfull, lane);
      if (!ktx && lane == 0) mbar_arrive(&br.kfull);
      last_unit = round;
      int qt = un.kt, h = un.hk * G;
      for (int j = 0; j < un.count; ++j, ++i) {
        const int s = i % NS, ls = i % kPfLseSlots;
        // the row normalisers are on their way while the warp waits for a free stage; a query beyond the prompt gets
        // -inf (negated lse), which makes its probability zero
        const float* lse = p.lse + ((long long)un.b * p.num_q_heads + h) * n;
        float nl[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int q = qt * kPfTile + e * 32 + lane;
          nl[e] = q < n ? -lse[q] : -INFINITY;
        }
        const float w = p.head_w != nullptr ? p.head_w[(long long)un.b * p.num_q_heads + h] : 1.f;
        ok = pf_wait(&br.empty[s], ((i / NS) & 1) ^ 1u, give_up);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (qtx && lane == 0) mbar_expect_tx(&br.full[s], qtx);
        pf_load_tile<D>(ring + s * TB, &qmap, p.q, qt * kPfTile, h, un.b, n, &br.full[s], lane);
        if (!qtx && lane == 0) mbar_arrive(&br.full[s]);
        ok = __all_sync(0xffffffffu, pf_wait(&br.lempty[ls], ((i / kPfLseSlots) & 1) ^ 1u, give_up));
        if (!ok) {
          ++i;  // this stage's copy is in flight
          break;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) lse_s[ls * LS + e * 32 + lane] = nl[e];
        if (lane == 0) lse_s[ls * LS + 128] = w;
        __syncwarp();
        if (lane == 0) mbar_arrive(&br.lfull[ls]);
        if (++qt == p.tiles) {
          qt = un.kt;
          ++h;
        }
      }
    }
    // No copy in flight may outlive the shared memory it targets.  Usually every copy has been waited for by whoever uses it, but
    // another role may have given up after this one issued its last.
    for (int s = 0; s < NS; ++s) {
      const int cnt = i > s ? (i - 1 - s) / NS + 1 : 0;
      if (cnt > 0) pf_drain(&br.full[s], (cnt - 1) & 1);
    }
    if (last_unit >= 0) pf_drain(&br.kfull, last_unit & 1);
  } else if (warp == kPfMmaWarp) {
    // ================================ MMA warp ================================
    int i = 0;
    bool ok = true;
    const uint32_t ring_d = smem_u32(ring), ks_d = pf_desc_k(smem_u32(ks));
    for (int round = 0; ok; ++round) {
      const int u = pf_unit(round, p.units);
      if (u < 0) break;
      const PfMassUnit un = pf_mass_unit(p, u);
      ok = __all_sync(0xffffffffu, pf_wait_unit(&br.kfull, round & 1, give_up, p.wait_cycles));
      for (int j = 0; ok && j < un.count; ++j, ++i) {
        const int s = i % NS, a = i % kPfAcc;
        ok = pf_wait(&br.full[s], (i / NS) & 1, give_up) && pf_wait(&br.sempty[a], ((i / kPfAcc) & 1) ^ 1u, give_up);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          pf_issue_scores<D>(tmem + a * 128, ks_d, pf_desc_k(ring_d + s * TB));
          mma_commit(&br.sfull[a]);
          mma_commit(&br.empty[s]);
          if (j == un.count - 1) mma_commit(&br.kempty);
        }
        __syncwarp();
      }
    }
    if (elect_one()) {
      mma_commit(&br.drain);
      pf_drain(&br.drain, 0);
    }
    __syncwarp();
  } else {
    // ================================ four warpgroups: one key row per thread ================================
    const int wg = warp >> 2, wq = warp & 3, wt = tid & 127;
    const uint32_t lanes = (uint32_t)(wq * 32) << 16;
    const uint64_t sc2 = f32x2(p.scale_log2, p.scale_log2);
    int i0 = 0;  // stream index of the unit's first query tile
    bool ok = true;
    for (int round = 0;; ++round) {
      const int u = pf_unit(round, p.units);
      if (u < 0) break;
      const PfMassUnit un = pf_mass_unit(p, u);
      const int per_head = p.tiles - un.kt;
      float acc = 0.f;
      for (int j = (wg - i0) & 3; ok && j < un.count; j += kPfAcc) {
        const int i = i0 + j, a = i % kPfAcc, ls = i % kPfLseSlots;
        const bool diag = j % per_head == 0;
        ok = pf_wait(&br.sfull[a], (i / kPfAcc) & 1, give_up) && pf_wait(&br.lfull[ls], (i / kPfLseSlots) & 1, give_up);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const float* nl = lse_s + ls * LS;
        uint64_t t0 = 0, t1 = 0;
        const uint32_t ta0 = tmem + a * 128 + lanes;
        auto add4 = [&](float4 q4, uint32_t sa, uint32_t sb, uint32_t sc, uint32_t sd) {
          const uint64_t xa = f32x2_fma(f32x2(__uint_as_float(sa), __uint_as_float(sb)), sc2, f32x2(q4.x, q4.y));
          const uint64_t xb = f32x2_fma(f32x2(__uint_as_float(sc), __uint_as_float(sd)), sc2, f32x2(q4.z, q4.w));
          t0 = f32x2_add(t0, pf_exp2_pair(xa));
          t1 = f32x2_add(t1, pf_exp2_pair(xb));
        };
        auto chunk_sum = [&](int c, uint32_t (&s)[32]) {
          if (!diag || c > wq) {
#pragma unroll
            for (int e = 0; e < 32; e += 4)
              add4(*reinterpret_cast<const float4*>(nl + c * 32 + e), s[e], s[e + 1], s[e + 2], s[e + 3]);
          } else if (c == wq) {
            // Queries before the row's key do not see it: all of the chunks before the warp's own, and here the first `lane`.  Their
            // normalisers become -inf too: the negated one of a query without a finite score is +inf or NaN, which a score of -inf
            // does not absorb.
            const uint32_t none = 0xff800000u;
#pragma unroll
            for (int e = 0; e < 32; e += 4) {
              float4 q4 = *reinterpret_cast<const float4*>(nl + c * 32 + e);
              q4.x = e < lane ? -INFINITY : q4.x;
              q4.y = e + 1 < lane ? -INFINITY : q4.y;
              q4.z = e + 2 < lane ? -INFINITY : q4.z;
              q4.w = e + 3 < lane ? -INFINITY : q4.w;
              add4(q4, e < lane ? none : s[e], e + 1 < lane ? none : s[e + 1], e + 2 < lane ? none : s[e + 2],
                   e + 3 < lane ? none : s[e + 3]);
            }
          }
        };
        uint32_t s0[32], s1[32];
        tmem_ld32(ta0, s0);
        tmem_ld_wait(s0);
        tmem_ld32(ta0 + 32, s1);
        chunk_sum(0, s0);
        tmem_ld_wait(s1);
        tmem_ld32(ta0 + 64, s0);
        chunk_sum(1, s1);
        tmem_ld_wait(s0);
        tmem_ld32(ta0 + 96, s1);
        chunk_sum(2, s0);
        tmem_ld_wait(s1);
        tc_fence_before();  // the accumulator has been read
        __syncwarp();
        if (lane == 0) mbar_arrive(&br.sempty[a]);
        chunk_sum(3, s1);
        const float2 t2 = f32x2_parts(f32x2_add(t0, t1));
        acc = fmaf(nl[128], t2.x + t2.y, acc);
        __syncwarp();
        if (lane == 0) mbar_arrive(&br.lempty[ls]);
      }
      i0 += un.count;
      if (!ok) acc = __int_as_float(0x7fffffff);
      // the warpgroups hand their sums to the first; the buffer alternates, so the barrier of the next unit protects it
      float* rd = red + (round & 1) * 3 * kPfTile + wt;
      if (wg != 0) rd[(wg - 1) * kPfTile] = acc;
      asm volatile("bar.sync 1, 512;" ::: "memory");
      if (wg == 0) {
        const int key = un.kt * kPfTile + wt;
        if (key < n)
          p.mass[((long long)un.b * p.num_kv_heads + un.hk) * n + key] = ((acc + rd[0]) + rd[kPfTile]) + rd[2 * kPfTile];
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, kPfTmemCols);
}

// ---- host ---------------------------------------------------------------------------------------------------
// A map of {head_dim, token, head, batch}, box = 128 tokens x 64 columns.  A dimension with one entry, or one that repeats the
// same data (stride 0), is left at extent 1 and its coordinate stays 0.  What no map can hold (every token the same row, or a
// stride beyond 2^40 bytes) is copied row by row in the kernel.
static bool make_map(CUtensorMap* map, PrefillTensor& t, int head_dim, int tokens, int heads, int batch) {
  constexpr long long kMaxStride = 1ll << 39;  // elements; 2^40 bytes
  t.mul_h = heads > 1 && t.sh != 0;
  t.mul_b = batch > 1 && t.sb != 0;
  auto fits = [](long long s) { return s > 0 && s < kMaxStride; };
  t.by_rows = (tokens > 1 && !fits(t.st)) || (t.mul_h && !fits(t.sh)) || (t.mul_b && !fits(t.sb));
  if (t.by_rows) return true;
  EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  const cuuint64_t gdim[4] = {(cuuint64_t)head_dim, (cuuint64_t)tokens, (cuuint64_t)(t.mul_h ? heads : 1),
                              (cuuint64_t)(t.mul_b ? batch : 1)};
  const cuuint64_t row = (cuuint64_t)head_dim * 2;
  const cuuint64_t gstr[3] = {tokens > 1 ? (cuuint64_t)t.st * 2 : row, t.mul_h ? (cuuint64_t)t.sh * 2 : row,
                              t.mul_b ? (cuuint64_t)t.sb * 2 : row};
  const cuuint32_t box[4] = {64, kPfTile, 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<__half*>(t.base), gdim, gstr, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int D>
static int launch_prefill(PrefillParams& p, bool want_mass, cudaStream_t st) {
  using Cfg = PfCfg<D>;
  CUtensorMap qmap = {}, kmap = {}, vmap = {};
  if (!make_map(&qmap, p.q, D, p.tokens, p.num_q_heads, p.batch) || !make_map(&kmap, p.k, D, p.tokens, p.num_kv_heads, p.batch) ||
      !make_map(&vmap, p.v, D, p.tokens, p.num_kv_heads, p.batch))
    return SKV_ERR_CUDA;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return SKV_ERR_CUDA;
  static bool configured[64] = {};  // the attribute belongs to the device's context
  if (dev >= 64 || !configured[dev]) {
    if (cudaFuncSetAttribute(prefill_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::kFwdSmem) != cudaSuccess ||
        cudaFuncSetAttribute(prefill_mass_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::kMassSmem) !=
            cudaSuccess)
      return SKV_ERR_CUDA;
    if (dev < 64) configured[dev] = true;
  }
  const int G = p.num_q_heads / p.num_kv_heads;
  const long long fwd_units = (long long)p.batch * (G % 2 == 0 ? (long long)p.tiles * (p.num_q_heads / 2)
                                                               : (long long)((p.tiles + 1) / 2) * p.num_q_heads);
  const long long mass_units = (long long)p.batch * p.tiles * p.num_kv_heads;
  if (fwd_units > 0x7fffffffll || mass_units > 0x7fffffffll) return SKV_ERR_UNSUPPORTED;
  p.units = (int)fwd_units;
  prefill_fwd_kernel<D><<<p.units < sms ? p.units : sms, kPfThreads, Cfg::kFwdSmem, st>>>(p, qmap, kmap, vmap);
  if (want_mass) {
    p.units = (int)mass_units;
    prefill_mass_kernel<D><<<p.units < sms ? p.units : sms, kPfThreads, Cfg::kMassSmem, st>>>(p, qmap, kmap);
  }
  return cudaGetLastError() == cudaSuccess ? SKV_OK : SKV_ERR_CUDA;
}

}  // namespace skv

using namespace skv;

extern "C" int skv_prefill_attention_checked(const void* q, const void* k, const void* v, int dtype, int batch, int tokens,
                                             int num_q_heads, int num_kv_heads, int head_dim, const int64_t* q_strides,
                                             const int64_t* k_strides, const int64_t* v_strides, const float* head_weights,
                                             void* out, float* lse, float* key_mass, int32_t* err_flag, void* stream) {
  if (!q || !k || !v || !out || !lse || !q_strides || !k_strides || !v_strides) return SKV_ERR_INVALID;
  if (dtype != SKV_DTYPE_F16) return SKV_ERR_UNSUPPORTED;
  if (head_dim != 64 && head_dim != 128) return SKV_ERR_UNSUPPORTED;
  if (batch <= 0 || tokens <= 0 || num_kv_heads <= 0 || num_q_heads % num_kv_heads != 0) return SKV_ERR_INVALID;
  if (batch > 65535 || num_q_heads > 65535) return SKV_ERR_UNSUPPORTED;
  for (int i = 0; i < 3; ++i)  // 16-byte pieces of every row
    if (q_strides[i] % 8 || k_strides[i] % 8 || v_strides[i] % 8) return SKV_ERR_INVALID;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15) return SKV_ERR_INVALID;
  auto tensor = [](const void* base, const int64_t* s) {
    return PrefillTensor{static_cast<const __half*>(base), s[0], s[1], s[2], 0, 0, 0};
  };
  PrefillParams p = {};
  p.q = tensor(q, q_strides);
  p.k = tensor(k, k_strides);
  p.v = tensor(v, v_strides);
  p.out = static_cast<__half*>(out);
  p.lse = lse;
  p.head_w = head_weights;
  p.mass = key_mass;
  p.batch = batch;
  p.tokens = tokens;
  p.num_q_heads = num_q_heads;
  p.num_kv_heads = num_kv_heads;
  p.tiles = (tokens + kPfTile - 1) / kPfTile;
  p.scale_log2 = 1.4426950408889634f / sqrtf((float)head_dim);
  const unsigned polls = wait_polls();
  p.wait_cycles = polls >= 1u << 24 ? 1u << 31 : polls >> 4 << 11;  // 128 cycles a poll, none below 16 polls
  p.err = err_flag;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return head_dim == 64 ? launch_prefill<64>(p, key_mass != nullptr, st) : launch_prefill<128>(p, key_mass != nullptr, st);
}

extern "C" int skv_prefill_attention(const void* q, const void* k, const void* v, int dtype, int batch, int tokens,
                                     int num_q_heads, int num_kv_heads, int head_dim, const int64_t* q_strides,
                                     const int64_t* k_strides, const int64_t* v_strides, const float* head_weights,
                                     void* out, float* lse, float* key_mass, void* stream) {
  return skv_prefill_attention_checked(q, k, v, dtype, batch, tokens, num_q_heads, num_kv_heads, head_dim, q_strides, k_strides,
                                       v_strides, head_weights, out, lse, key_mass, nullptr, stream);
}
