// Requantise / repack after a reallocation.
//
// Replaces SmartKVCache._requantize_tokens / _requantize_single / _write_quantized_slot
// (smartkv/core/cache.py:806-926) and the bucket bookkeeping around them (swap-with-last
// delete :1121-1161, append :1046-1083): a Python loop over every (layer, changed token).
//
// A token whose width changed is dequantised from its stored codes (code * scale, fp32),
// quantised again at the new width (cache.py:819-844: from the dequantised codes, not from
// the original values) and moved to the bucket of the new width.  Buckets stay dense: the
// positions a bucket loses are refilled first by its own rows that now lie beyond the new
// count, then by the arriving rows, so only changed rows and a few tail rows are touched.
// Which row of a bucket a token occupies is not observable (attention is a sum over keys).
//
// Three steps, every one stream-ordered:
//   skv_repack_plan     one block per sequence: the list of moves (source -> destination
//                       storage index), the same for every layer
//   skv_requant_repack  per layer range: all moved rows -> staging (requantised where the
//                       width changed), then staging -> destination, so that every read of the
//                       old layout precedes every write of the new one.  Rows of different
//                       (layer, sequence, KV head) never touch, so one CTA or a cluster takes one
//                       of those at a time and its own barrier is the only order needed.
//   skv_repack_meta     the per-token arrays kept in storage order follow the same moves.
#include <cooperative_groups.h>

#include <cub/block/block_scan.cuh>

#include "quant_bulk.cuh"

namespace skv {

namespace cg = cooperative_groups;

constexpr int kPlanThreads = 1024;
constexpr int kStageRowBytes = 136;  // 16 bytes for each of up to 8 lanes, the fp32 scale, padding
constexpr int kMaxSeqsRepack = 1024;

__device__ __forceinline__ int bucket_of_slot(const StoreGeom& g, int s) {
  int b = 0;
#pragma unroll
  for (int i = 1; i < kNumBuckets; ++i)
    if (s >= g.bucket_base[i]) b = i;
  return b;
}

// ---- the moves ----------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kPlanThreads)
    repack_plan_kernel(StoreGeom g, const int32_t* counts, const uint8_t* new_bits, int32_t* move_src,
                       int32_t* move_dst, int32_t* n_moves, int32_t* counts_new, int32_t* scratch, int32_t* err) {
  const int b = blockIdx.x, tid = threadIdx.x, T = g.slots;
  using Scan = cub::BlockScan<int, kPlanThreads>;
  __shared__ typename Scan::TempStorage tmp;
  __shared__ int s_new[kNumBuckets], s_free[kNumBuckets], s_tail[kNumBuckets], s_off[kNumBuckets + 1];
  __shared__ int s_run[2];
  const uint8_t* nb = new_bits + (long long)b * T;
  int32_t* free_pos = scratch + (long long)b * 2 * T;  // [T], bucket w's list at [bucket_base[w] ...)
  int32_t* tail_src = free_pos + T;                     // [T]
  int32_t* msrc = move_src + (long long)b * T;
  int32_t* mdst = move_dst + (long long)b * T;
  int cnt[kNumBuckets];
#pragma unroll
  for (int i = 0; i < kNumBuckets; ++i) cnt[i] = counts[b * kNumBuckets + i];
  if (tid < kNumBuckets) s_new[tid] = 0;
  __syncthreads();

  // new counts
  for (int w = 0; w < kNumBuckets; ++w) {
    for (int pos = tid; pos < cnt[w]; pos += kPlanThreads) {
      const int nbk = bits_bucket(nb[g.bucket_base[w] + pos]);
      if (nbk >= 0) atomicAdd(&s_new[nbk], 1);
      else if (err) atomicExch(err, 4);  // a live token without a width
    }
  }
  __syncthreads();
  bool over = false;
#pragma unroll
  for (int i = 0; i < kNumBuckets; ++i) over |= s_new[i] > g.cap[i];
  if (over) {
    if (tid == 0) {
      if (err) atomicExch(err, 3);  // a bucket would overflow: nothing moves
      n_moves[b] = 0;
      for (int i = 0; i < kNumBuckets; ++i) counts_new[b * kNumBuckets + i] = cnt[i];
    }
    return;
  }

  // per bucket: free positions (ascending) and own rows beyond the new count (ascending)
  for (int w = 0; w < kNumBuckets; ++w) {
    const int c_old = cnt[w], c_new = s_new[w], base = g.bucket_base[w], width = bucket_bits(w);
    const int span = c_old > c_new ? c_old : c_new;
    if (tid == 0) s_run[0] = s_run[1] = 0;
    __syncthreads();
    for (int p0 = 0; p0 < span; p0 += kPlanThreads) {
      const int pos = p0 + tid;
      const bool live = pos < c_old;
      const bool stays = live && nb[base + pos] == width;
      const int is_free = (pos < c_new && !stays) ? 1 : 0;
      const int is_tail = (stays && pos >= c_new) ? 1 : 0;
      int packed = is_free | (is_tail << 16), excl, total;
      Scan(tmp).ExclusiveSum(packed, excl, total);
      const int rf = s_run[0] + (excl & 0xffff), rt = s_run[1] + (excl >> 16);
      if (is_free) free_pos[base + rf] = pos;
      if (is_tail) tail_src[base + rt] = base + pos;
      __syncthreads();
      if (tid == 0) {
        s_run[0] += total & 0xffff;
        s_run[1] += total >> 16;
      }
      __syncthreads();
    }
    if (tid == 0) {
      s_free[w] = s_run[0];
      s_tail[w] = s_run[1];
    }
    __syncthreads();
  }
  if (tid == 0) {
    int off = 0;
    for (int w = 0; w < kNumBuckets; ++w) {
      s_off[w] = off;
      off += s_free[w];
    }
    s_off[kNumBuckets] = off;
    n_moves[b] = off;
    for (int i = 0; i < kNumBuckets; ++i) counts_new[b * kNumBuckets + i] = s_new[i];
  }
  __syncthreads();

  // arrivals of every bucket in ascending source storage index, after the bucket's tail rows
  __shared__ int s_arr[kNumBuckets];
  if (tid < kNumBuckets) s_arr[tid] = 0;
  __syncthreads();
  for (int ws = 0; ws < kNumBuckets; ++ws) {
    const int base = g.bucket_base[ws], width = bucket_bits(ws);
    for (int p0 = 0; p0 < cnt[ws]; p0 += kPlanThreads) {
      const int pos = p0 + tid;
      int to = -1;
      if (pos < cnt[ws]) {
        const int nw = nb[base + pos];
        if (nw != width) to = bits_bucket(nw);
      }
      // a chunk can send up to 1024 rows to one bucket: two scans of two 16-bit fields each
      int pa = (to == 0 ? 1 : 0) | ((to == 1 ? 1 : 0) << 16);
      int pb = (to == 2 ? 1 : 0) | ((to == 3 ? 1 : 0) << 16);
      int ea, ta, eb, tb;
      Scan(tmp).ExclusiveSum(pa, ea, ta);
      __syncthreads();
      Scan(tmp).ExclusiveSum(pb, eb, tb);
      if (to >= 0) {
        const int rank = to == 0 ? (ea & 0xffff) : to == 1 ? (ea >> 16) : to == 2 ? (eb & 0xffff) : (eb >> 16);
        msrc[s_off[to] + s_tail[to] + s_arr[to] + rank] = base + pos;
      }
      __syncthreads();
      if (tid == 0) {
        s_arr[0] += ta & 0xffff;
        s_arr[1] += ta >> 16;
        s_arr[2] += tb & 0xffff;
        s_arr[3] += tb >> 16;
      }
      __syncthreads();
    }
  }
  // destinations and the tail sources
  for (int w = 0; w < kNumBuckets; ++w) {
    const int base = g.bucket_base[w];
    if (tid == 0 && s_tail[w] + s_arr[w] != s_free[w] && err) atomicExch(err, 5);  // bookkeeping broken
    for (int k = tid; k < s_free[w]; k += kPlanThreads) mdst[s_off[w] + k] = base + free_pos[base + k];
    for (int k = tid; k < s_tail[w]; k += kPlanThreads) msrc[s_off[w] + k] = tail_src[base + k];
  }
}

// ---- moving the rows ------------------------------------------------------------------------------------
struct RowMoveParams {
  StoreGeom g;
  uint8_t* store;
  int layer_begin, layer_end;
  const int32_t* move_src;
  const int32_t* move_dst;
  const int32_t* n_moves;
  uint8_t* staging;
  long long staging_rows;
  int32_t* err;
};

// prefix of the per-sequence move counts into shared memory (at least one warp per block); returns the total
__device__ __forceinline__ int load_move_prefix(const int32_t* n_moves, int B, int* s_prefix) {
  if (threadIdx.x < 32) {
    int carry = 0;
    if (threadIdx.x == 0) s_prefix[0] = 0;
    for (int b0 = 0; b0 < B; b0 += 32) {
      const int b = b0 + (int)threadIdx.x;
      int v = b < B ? n_moves[b] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, v, o);
        if ((int)threadIdx.x >= o) v += up;
      }
      if (b < B) s_prefix[b + 1] = carry + v;
      carry += __shfl_sync(0xffffffffu, v, 31);
    }
  }
  __syncthreads();
  return s_prefix[B];
}
__device__ __forceinline__ int find_seq(const int* s_prefix, int B, int m) {
  int lo = 0, hi = B - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (s_prefix[mid] <= m) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// CTAs of 512 threads that work at once: two per SM of a B200 (the staging size depends on it, so it is no question to a device).
constexpr int kRowThreads = 512;
constexpr int kRowCtas = 296;

// One item = the moves of one (layer, KV head, sequence).  Phase 0 reads the source rows, requantises where the width changes
// and leaves every lane's packed field and the scale in staging; after the cluster's barrier phase 1 writes the
// destinations.  Staging is written and read back by the same few CTAs, so it lives in L2.
//
// The staging buffer is divided among the workers that have an item in hand, by the moves there are and not by the moves there could be.
// A worker is a single CTA, or a cluster where that ends sooner: where there are fewer items than CTAs, or room for few slots.  So a
// buffer sized by a budget serves all layers in one launch: what it limits is how many items are in hand at once.  With a launch per as many layers as the worst case allows, 1 x 131072 tokens, 32 layers, 8 heads with 1 GiB
// took 4377 us a reallocation, now 2720 us.
//
// What bounds it: the rows are scattered pieces of 32 to 128 bytes, so the memory system needs many of them in flight
// (a warp issues the loads of four moves first), and the quantiser's instructions.  As two grid-wide kernels per
// layer range, each with one row per half-warp and a staging buffer in HBM, 16 sequences of 8192 tokens, 32 layers, 8 heads
// took 2330 us for 13,000 moves (2.9 GB of DRAM traffic: a row is two or three 32-byte sectors and its scale one); with 8 elements
// a lane 1360 us.  A lane holds 16 elements, so that twice as many rows share the instructions that are done once per lane or
// row: a whole reallocation 1677 -> 1403 us (two moves in flight 1517).
// A row's place inside its (arena, KV head): bucket and position in one word, so that a warp passes it round in one shuffle.
// Positions stay below 2^30 (a store has fewer than 2^31 / 3 storage indices), so all ones is no place.
constexpr uint32_t kNoPlace = 0xffffffffu;
__device__ __forceinline__ uint32_t row_place(const StoreGeom& g, int slot) {
  const int b = bucket_of_slot(g, slot);
  return ((uint32_t)b << 30) | (uint32_t)(slot - g.bucket_base[b]);
}

template <int D, int CS>
__global__ void __launch_bounds__(kRowThreads, 2) repack_rows_kernel(const __grid_constant__ RowMoveParams p) {
  constexpr int LPR = D / 16;             // lanes per row
  constexpr int PPP = 32 / (2 * LPR);     // moves side by side in a warp: the K and the V row of each
  constexpr int RB = 4 / PPP;        // row groups whose loads a warp has in flight
  constexpr int MB = RB * PPP;            // moves whose rows a warp has in flight
  constexpr int MC = 8;                   // moves a warp looks up at a time: lanes 0-7 the sources, 8-15 the destinations
  const StoreGeom& g = p.g;
  __shared__ int s_prefix[kMaxSeqsRepack + 1];
  __shared__ int s_max;
  __shared__ uint8_t* s_base[3][kNumBuckets];  // of the item: K rows, V rows, scale pairs of every bucket
  if (threadIdx.x == 0) s_max = 0;
  const int B = g.num_seqs, total = load_move_prefix(p.n_moves, B, s_prefix);
  for (int b = threadIdx.x; b < B; b += kRowThreads) atomicMax(&s_max, s_prefix[b + 1] - s_prefix[b]);
  __syncthreads();
  const int longest = s_max, Hkv = g.num_kv_heads, nl = p.layer_end - p.layer_begin;
  if (longest == 0) return;
  const int items = nl * Hkv * B;  // the host has checked that it fits
  // a place for every row, or else a slot of `longest` moves for each worker; the same decisions in every CTA
  const bool places = (long long)total * nl * Hkv * 2 <= p.staging_rows;
  const long long room = p.staging_rows / (2ll * longest);
  if (!places && room == 0) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && p.err) atomicExch(p.err, 6);  // staging too small: nothing moves
    return;
  }
  auto workers_of = [&](int n) -> int {
    const int w = items < n ? items : n;
    return places || w < room ? w : (int)room;
  };
  auto turns_of = [&](int n) -> int { return (items - 1) / n + 1; };
  const bool share = CS > 1 && turns_of(workers_of((int)gridDim.x / CS)) < CS * turns_of(workers_of((int)gridDim.x));
  const int per = share ? CS : 1, workers = workers_of((int)gridDim.x / per), worker = (int)blockIdx.x / per;
  if (worker >= workers) return;  // the whole cluster, where one shares
  const bool slots = room >= workers;
  const int lane = threadIdx.x & 31, l = lane & (LPR - 1), which = (lane / LPR) & 1, sub = lane / (2 * LPR);
  const int cw = ((int)blockIdx.x % per) * (kRowThreads / 32) + (threadIdx.x >> 5), cwarps = per * (kRowThreads / 32);
  auto sync = [&] {
    if (CS == 1 || !share) __syncthreads();
    else cg::this_cluster().sync();
  };
  for (int it = worker; it < items; it += workers) {
    const int lh = it / B, seq = it - lh * B, li = lh / Hkv, h = lh - li * Hkv;
    const int moves = s_prefix[seq + 1] - s_prefix[seq];
    if (moves == 0) continue;  // the same for the whole worker
    uint8_t* arena = arena_ptr(g, p.store, p.layer_begin + li, seq);
    const int32_t* msrc = p.move_src + (long long)seq * g.slots;
    const int32_t* mdst = p.move_dst + (long long)seq * g.slots;
    uint8_t* stage = p.staging + (slots ? (long long)worker * longest * 2 : ((long long)lh * total + s_prefix[seq]) * 2) * kStageRowBytes +
                     which * kStageRowBytes;
    if (threadIdx.x < 3 * kNumBuckets) {
      const int what = threadIdx.x / kNumBuckets, b = threadIdx.x % kNumBuckets;
      const long long first = (long long)h * g.cap[b];
      s_base[what][b] = arena + (what == 0   ? g.k_off[b] + first * g.row_bytes[b]
                                 : what == 1 ? g.v_off[b] + first * g.row_bytes[b]
                                             : g.sc_off[b] + first * 8);
    }
    __syncthreads();
    auto look_up = [&](int c0) -> uint32_t {
      const int m = c0 + (lane & (MC - 1));
      return lane < 2 * MC && m < moves ? row_place(g, (lane < MC ? msrc : mdst)[m]) : kNoPlace;
    };
    auto row_ptr = [&](uint32_t place) -> uint8_t* {
      const int b = (int)(place >> 30);
      return s_base[which][b] + (long long)(place & 0x3fffffffu) * (D / 8 * kWidthConst[b].bits);
    };
    auto scale_ptr = [&](uint32_t place) -> float* {
      return reinterpret_cast<float*>(s_base[2][place >> 30]) + 2ll * (place & 0x3fffffffu) + which;
    };

    for (int c0 = cw * MC; c0 < moves; c0 += cwarps * MC) {
      const uint32_t mine = look_up(c0);
#pragma unroll 1
      for (int m0 = 0; m0 < MC && c0 + m0 < moves; m0 += MB) {
        uint4 w[RB];
        float sc[RB];
        int bs[RB];
#pragma unroll
        for (int u = 0; u < RB; ++u) {
          const uint32_t at = __shfl_sync(0xffffffffu, mine, m0 + u * PPP + sub);
          bs[u] = at == kNoPlace ? 0 : (int)(at >> 30);
          w[u] = make_uint4(0u, 0u, 0u, 0u);
          sc[u] = 0.f;
          if (at == kNoPlace) continue;
          // a lane's 16 * bits bits: one word, at 3 bits two words of which every other lane's begins halfway, two, or four
          const uint32_t* rp = reinterpret_cast<const uint32_t*>(row_ptr(at)) + ((l * kWidthConst[bs[u]].bits) >> 1);
          if (bs[u] == 3) {
            const uint2 a = reinterpret_cast<const uint2*>(rp)[0], b = reinterpret_cast<const uint2*>(rp)[1];
            w[u] = make_uint4(a.x, a.y, b.x, b.y);
          } else {
            w[u].x = rp[0];
            if (bs[u] != 0) w[u].y = rp[1];
          }
          sc[u] = *scale_ptr(at);
        }
#pragma unroll
        for (int u = 0; u < RB; ++u) {
          const uint32_t to = __shfl_sync(0xffffffffu, mine, MC + m0 + u * PPP + sub);
          if (__all_sync(0xffffffffu, to == kNoPlace)) break;
          const int b_from = bs[u], b_to = to == kNoPlace ? 0 : (int)(to >> 30);
          uint32_t lo[2], hi[2] = {w[u].y, w[u].w};  // of each group of 8 elements; hi at 8 bits only
          if (b_from == 3) {
            lo[0] = w[u].x;
            lo[1] = w[u].z;
          } else if (b_from == 2) {
            lo[0] = w[u].x;
            lo[1] = w[u].y;
          } else if (b_from == 1) {
            const int sh = (l & 1) * 16;
            const uint32_t v = __funnelshift_r(w[u].x, w[u].y, sh);
            lo[0] = v & 0x00ffffffu;
            lo[1] = (v >> 24) | (((w[u].y >> sh) & 0xffffu) << 8);
          } else {
            lo[0] = w[u].x & 0xffffu;
            lo[1] = w[u].x >> 16;
          }
          float scale = sc[u];
          if (__any_sync(0xffffffffu, b_from != b_to)) {
            float x[2][8], amax = 0.f;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              dequantize8(lo[j], hi[j], b_from, scale, x[j]);
#pragma unroll
              for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(x[j][i]));
            }
            uint32_t nlo[2], nhi[2];
            const float ns = quantize_groups<LPR, 2>(x, amax, b_to, nlo, nhi);
            if (b_from != b_to) {
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                lo[j] = nlo[j];
                hi[j] = nhi[j];
              }
              scale = ns;
            }
          }
          if (to != kNoPlace) {
            uint8_t* st = stage + (long long)(c0 + m0 + u * PPP + sub) * 2 * kStageRowBytes;
            uint2* f = reinterpret_cast<uint2*>(st) + 2 * l;  // staged rows lie on 8-byte boundaries
            f[0] = make_uint2(lo[0], hi[0]);
            f[1] = make_uint2(lo[1], hi[1]);
            if (l == 0) *reinterpret_cast<float*>(st + 16 * LPR) = scale;
          }
        }
      }
    }
    sync();
    for (int c0 = cw * MC; c0 < moves; c0 += cwarps * MC) {
      const uint32_t mine = look_up(c0);
#pragma unroll 1
      for (int m0 = 0; m0 < MC && c0 + m0 < moves; m0 += MB) {
        uint2 f[RB][2];
        float sc[RB];
#pragma unroll
        for (int u = 0; u < RB; ++u) {
          f[u][0] = f[u][1] = make_uint2(0u, 0u);
          sc[u] = 0.f;
          if (c0 + m0 + u * PPP + sub < moves) {
            const uint8_t* st = stage + (long long)(c0 + m0 + u * PPP + sub) * 2 * kStageRowBytes;
            f[u][0] = reinterpret_cast<const uint2*>(st)[2 * l];
            f[u][1] = reinterpret_cast<const uint2*>(st)[2 * l + 1];
            if (l == 0) sc[u] = *reinterpret_cast<const float*>(st + 16 * LPR);
          }
        }
#pragma unroll
        for (int u = 0; u < RB; ++u) {
          const uint32_t at = __shfl_sync(0xffffffffu, mine, MC + m0 + u * PPP + sub);
          const int b = (int)(at >> 30);
          const uint32_t lo[2] = {f[u][0].x, f[u][1].x}, hi[2] = {f[u][0].y, f[u][1].y};
          const uint32_t next = __shfl_down_sync(0xffffffffu, lo[0], 1);
          if (at == kNoPlace) continue;
          store_field16(row_ptr(at), b, l, lo, hi, next);
          if (l == 0) {
            *scale_ptr(at) = sc[u];
            if (which) note_v_scale(g, arena, sc[u]);
          }
        }
      }
    }
    sync();  // the slot is free for the next item
  }
}

// CTAs that share an item (up to 8, the portable cluster size): enough to keep them all busy when there are few items, or when the
// staging buffer has room for few slots of the most moves there can be.
static int row_cluster(long long items, long long room) {
  int cs = items * 2 > kRowCtas ? 1 : items * 4 > kRowCtas ? 2 : items * 8 > kRowCtas ? 4 : 8;
  while (cs < 8 && room < (items < kRowCtas / cs ? items : kRowCtas / cs)) cs *= 2;
  return cs;
}

template <int D, int CS>
static cudaError_t launch_rows(const RowMoveParams& p, long long items, cudaStream_t st) {
  // No more clusters than run at once (items are dealt in advance, so a second wave would wait for the first: 1554 instead of 1162 us
  // for the rows of 1 x 131072 tokens in 32 layers): a cluster lies in one GPC, so 71 of 4 CTAs and 33 of 8 do.
  constexpr long long fit = CS <= 2 ? kRowCtas / CS : 256 / CS;
  const long long clusters = items < fit ? items : fit;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * CS));
  cfg.blockDim = dim3(kRowThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CS > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, repack_rows_kernel<D, CS>, p);
}

// ---- per-token arrays -----------------------------------------------------------------------------------
struct MetaParams {
  StoreGeom g;
  const int32_t* move_src;
  const int32_t* move_dst;
  const int32_t* n_moves;
  int32_t* counts;
  const int32_t* counts_new;
  int32_t* slot_token;
  double* cumulative;
  double* rank_pct;
  int8_t* rank_streak;
  float* layer_ema;
  uint8_t* touched;
  uint8_t* staging;
  long long staging_moves;
  int32_t* err;
};

constexpr int kMetaCtas = 296;  // two per SM: a move and layer per thread, a few turns at most in a settled store

__host__ __device__ inline long long meta_move_bytes(int num_layers) { return 24 + 8LL * num_layers; }

template <int PHASE>
__global__ void repack_meta_kernel(const MetaParams p) {
  const StoreGeom& g = p.g;
  __shared__ int s_prefix[kMaxSeqsRepack + 1];
  const int total = load_move_prefix(p.n_moves, g.num_seqs, s_prefix);
  if (total > p.staging_moves) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && p.err) atomicExch(p.err, 6);
    return;
  }
  const int L = g.num_layers, T = g.slots, B = g.num_seqs;
  // staging arrays, one entry per move
  double* st_cum = reinterpret_cast<double*>(p.staging);
  double* st_pct = st_cum + p.staging_moves;
  int32_t* st_tok = reinterpret_cast<int32_t*>(st_pct + p.staging_moves);
  float* st_ema = reinterpret_cast<float*>(st_tok + p.staging_moves);             // [L][moves]
  uint8_t* st_tch = reinterpret_cast<uint8_t*>(st_ema + (long long)L * p.staging_moves);  // [L][moves]
  int8_t* st_str = reinterpret_cast<int8_t*>(st_tch + (long long)L * p.staging_moves);
  // one (move, layer) per thread, moves innermost; "layer" L stands for the arrays that have none
  const long long nthreads = (long long)gridDim.x * blockDim.x, pairs = (long long)total * (L + 1);
  for (long long it = (long long)blockIdx.x * blockDim.x + threadIdx.x; it < pairs; it += nthreads) {
    const int l = (int)(it / total), m = (int)(it - (long long)l * total);
    const int b = find_seq(s_prefix, B, m);
    const int k = m - s_prefix[b];
    const long long si = (long long)b * T + p.move_src[(long long)b * T + k];
    const long long di = (long long)b * T + p.move_dst[(long long)b * T + k];
    const long long sl = (long long)l * p.staging_moves + m, la = (long long)l * B * T;
    if (PHASE == 0) {
      if (l == L) {
        st_cum[m] = p.cumulative[si];
        st_pct[m] = p.rank_pct[si];
        st_tok[m] = p.slot_token[si];
        st_str[m] = p.rank_streak[si];
      } else {
        st_ema[sl] = p.layer_ema[la + si];
        st_tch[sl] = p.touched[la + si];
      }
    } else {
      if (l == L) {
        p.cumulative[di] = st_cum[m];
        p.rank_pct[di] = st_pct[m];
        p.slot_token[di] = st_tok[m];
        p.rank_streak[di] = st_str[m];
      } else {
        p.layer_ema[la + di] = st_ema[sl];
        p.touched[la + di] = st_tch[sl];
      }
    }
  }
}

// indices a bucket gave up hold no token any more: a later append must find fresh state there
__global__ void repack_meta_clear_kernel(const MetaParams p) {
  const StoreGeom& g = p.g;
  const int b = blockIdx.y, L = g.num_layers, T = g.slots, B = g.num_seqs;
  for (int w = 0; w < kNumBuckets; ++w) {
    const int c_old = p.counts[b * kNumBuckets + w], c_new = p.counts_new[b * kNumBuckets + w];
    for (int pos = c_new + blockIdx.x * blockDim.x + threadIdx.x; pos < c_old; pos += gridDim.x * blockDim.x) {
      const long long i = (long long)b * T + g.bucket_base[w] + pos;
      p.cumulative[i] = 0.0;
      p.rank_pct[i] = 0.0;
      p.rank_streak[i] = -1;
      p.slot_token[i] = -1;
      for (int l = 0; l < L; ++l) {
        p.layer_ema[(long long)l * B * T + i] = 0.f;
        p.touched[(long long)l * B * T + i] = 0;
      }
    }
  }
}
__global__ void repack_commit_counts_kernel(int32_t* counts, const int32_t* counts_new, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) counts[i] = counts_new[i];
}

}  // namespace skv

using namespace skv;

extern "C" int64_t skv_repack_plan_workspace_bytes(const SkvStoreDesc* desc) {
  if (!desc || desc->num_seqs <= 0 || desc->slots <= 0) return SKV_ERR_INVALID;
  return (int64_t)desc->num_seqs * desc->slots * 2 * (int64_t)sizeof(int32_t);
}

extern "C" int skv_repack_plan(const SkvStoreDesc* desc, const int32_t* counts, const uint8_t* new_bits,
                               int32_t* move_src, int32_t* move_dst, int32_t* n_moves, int32_t* counts_new,
                               void* workspace, int32_t* err_flag, void* stream) {
  if (!desc || !counts || !new_bits || !move_src || !move_dst || !n_moves || !counts_new || !workspace)
    return SKV_ERR_INVALID;
  if (desc->num_seqs > kMaxSeqsRepack) return SKV_ERR_UNSUPPORTED;
  repack_plan_kernel<<<desc->num_seqs, kPlanThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      make_geom(*desc), counts, new_bits, move_src, move_dst, n_moves, counts_new, static_cast<int32_t*>(workspace),
      err_flag);
  return cudaGetLastError() == cudaSuccess ? SKV_OK : SKV_ERR_CUDA;
}

extern "C" int64_t skv_requant_staging_bytes(const SkvStoreDesc* desc, int64_t max_moves, int num_layers) {
  if (!desc || max_moves < 0 || num_layers <= 0) return SKV_ERR_INVALID;
  // a place for every row, or one slot per CTA for the moves of one sequence, whichever is less
  const int64_t rows = max_moves * num_layers * desc->num_kv_heads * 2;
  const int64_t slots = (max_moves < desc->slots ? max_moves : (int64_t)desc->slots) * 2 * kRowCtas;
  return (rows < slots ? rows : slots) * (int64_t)kStageRowBytes;
}

extern "C" int64_t skv_requant_min_staging_bytes(const SkvStoreDesc* desc, int64_t max_moves) {
  if (!desc || max_moves < 0) return SKV_ERR_INVALID;
  return (max_moves < desc->slots ? max_moves : (int64_t)desc->slots) * 2 * kStageRowBytes;
}

extern "C" int skv_requant_repack(const SkvStoreDesc* desc, void* store, int layer_begin, int layer_end,
                                  const int32_t* move_src, const int32_t* move_dst, const int32_t* n_moves,
                                  void* staging, int64_t staging_bytes, int32_t* err_flag, void* stream) {
  if (!desc || !store || !move_src || !move_dst || !n_moves || !staging) return SKV_ERR_INVALID;
  if (layer_begin < 0 || layer_end > desc->num_layers || layer_begin >= layer_end) return SKV_ERR_INVALID;
  if (desc->head_dim != 64 && desc->head_dim != 128) return SKV_ERR_UNSUPPORTED;
  if (desc->num_seqs > kMaxSeqsRepack) return SKV_ERR_UNSUPPORTED;
  RowMoveParams p;
  p.g = make_geom(*desc);
  p.store = static_cast<uint8_t*>(store);
  p.layer_begin = layer_begin;
  p.layer_end = layer_end;
  p.move_src = move_src;
  p.move_dst = move_dst;
  p.n_moves = n_moves;
  p.staging = static_cast<uint8_t*>(staging);
  p.staging_rows = staging_bytes / kStageRowBytes;
  p.err = err_flag;
  if (desc->slots >= (1 << 30)) return SKV_ERR_UNSUPPORTED;  // row_place
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const long long items = (long long)(layer_end - layer_begin) * desc->num_kv_heads * desc->num_seqs;
  if (items > (1 << 30)) return SKV_ERR_UNSUPPORTED;
  const int cs = row_cluster(items, p.staging_rows / (2ll * desc->slots));
  const bool d128 = desc->head_dim == 128;
  const cudaError_t rc = cs == 1   ? (d128 ? launch_rows<128, 1>(p, items, st) : launch_rows<64, 1>(p, items, st))
                         : cs == 2 ? (d128 ? launch_rows<128, 2>(p, items, st) : launch_rows<64, 2>(p, items, st))
                         : cs == 4 ? (d128 ? launch_rows<128, 4>(p, items, st) : launch_rows<64, 4>(p, items, st))
                                   : (d128 ? launch_rows<128, 8>(p, items, st) : launch_rows<64, 8>(p, items, st));
  if (rc != cudaSuccess) return SKV_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? SKV_OK : SKV_ERR_CUDA;
}

extern "C" int64_t skv_repack_meta_staging_bytes(const SkvStoreDesc* desc, int64_t max_moves) {
  if (!desc || max_moves < 0) return SKV_ERR_INVALID;
  return max_moves * meta_move_bytes(desc->num_layers) + 256;
}

extern "C" int skv_repack_meta(const SkvStoreDesc* desc, const int32_t* move_src, const int32_t* move_dst,
                               const int32_t* n_moves, int32_t* counts, const int32_t* counts_new,
                               int32_t* slot_token, double* cumulative, double* rank_pct, int8_t* rank_streak,
                               float* layer_ema, uint8_t* touched, void* staging, int64_t staging_bytes,
                               int32_t* err_flag, void* stream) {
  if (!desc || !move_src || !move_dst || !n_moves || !counts || !counts_new || !slot_token || !cumulative ||
      !rank_pct || !rank_streak || !layer_ema || !touched || !staging)
    return SKV_ERR_INVALID;
  if (desc->num_seqs > kMaxSeqsRepack) return SKV_ERR_UNSUPPORTED;
  MetaParams p;
  p.g = make_geom(*desc);
  p.move_src = move_src;
  p.move_dst = move_dst;
  p.n_moves = n_moves;
  p.counts = counts;
  p.counts_new = counts_new;
  p.slot_token = slot_token;
  p.cumulative = cumulative;
  p.rank_pct = rank_pct;
  p.rank_streak = rank_streak;
  p.layer_ema = layer_ema;
  p.touched = touched;
  p.staging = static_cast<uint8_t*>(staging);
  p.staging_moves = (staging_bytes - 256) / meta_move_bytes(desc->num_layers);
  p.staging_moves &= ~7LL;  // keeps every staging array 8-byte aligned
  p.err = err_flag;
  if (p.staging_moves <= 0) return SKV_ERR_CAPACITY;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  repack_meta_kernel<0><<<kMetaCtas, 256, 0, st>>>(p);
  repack_meta_kernel<1><<<kMetaCtas, 256, 0, st>>>(p);
  repack_meta_clear_kernel<<<dim3(8, desc->num_seqs), 256, 0, st>>>(p);
  repack_commit_counts_kernel<<<(desc->num_seqs * kNumBuckets + 255) / 256, 256, 0, st>>>(counts, counts_new,
                                                                                        desc->num_seqs * kNumBuckets);
  return cudaGetLastError() == cudaSuccess ? SKV_OK : SKV_ERR_CUDA;
}
