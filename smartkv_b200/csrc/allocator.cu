// Budgeted bit allocation on the device.
//
// Replaces SmartKVCache.allocate_precision / _solve_allocation
// (smartkv/core/cache.py:281-351, 353-601), a Python heap loop over every cached
// token, for all sequences of the batch at once.
//
// The heap pops (token, step) items by (gain-per-bit desc, token id asc); an item is
// pushed only after the token's previous step was accepted.  Give every item the
// *effective key* min(own score, effective key of the token's previous step): sorted
// by (effective key desc, token id asc, step asc) the items come out in exactly the
// heap's pop order.  The walk over the sorted items then has two phases:
//   1. while the memory ratio is below 0.85 * budget nothing is gated and (for all but
//      tiny caches) every step is affordable, so everything is accepted: the payload
//      is a prefix sum and the phase ends at the first position c1 whose prefix
//      reaches 0.85 * budget (cache.py:468-472: a token accepted past the gate is not
//      pushed again);
//   2. after c1 a token can be accepted once more, and only if its previous step lies
//      before c1; those items are accepted greedily while they fit, skipping items that
//      do not (cache.py:502-505).  Step costs take at most three values, and once an
//      item of some cost fails every later item of that or a larger cost fails too, so
//      the walk is a few prefix sums with cut points instead of a serial loop.
// Caches so small that a single step can jump from below the gate to above the budget
// are walked serially by one thread with the same rules.
// The rank-percentile / streak state of the hysteresis (cache.py:423-450) is kept per
// token in storage order, and the high-priority post-pass (cache.py:522-591) is a serial
// loop that returns at once when it has nothing to do (the usual case).
//
// One cluster of CTAs per sequence does all of it in one launch.  What bounds it is latency: a few
// thousand tokens per sequence are sorted twice (by id, by score) and their steps once, and every
// sort is a chain of passes over data that sits in L2.  The general device-wide sorts this
// replaces ran over the whole capacity of the store (four times the live tokens, two sorts each to keep
// the sequences apart, about 40 launches); a cluster knows its sequence's live count, skips digits
// that all keys share, and its passes are separated by a hardware barrier.  A whole reallocation of 16 x 8256 tokens went
// from 2889 to 2774 us with it, a batch of 8 generations (512 + 16 tokens, 26 reallocations) from 44.5 to 38.2 ms.
//
// All score arithmetic is fp64 in the reference's operation order; the powers
// bits^alpha come from the host so that they are the host libm's values.
#include <cooperative_groups.h>

#include <climits>
#include <cmath>
#include <cub/block/block_scan.cuh>

#include "common.cuh"

namespace skv {

namespace cg = cooperative_groups;

constexpr int kAllocThreads = 512;
constexpr int kAllocWarps = kAllocThreads / 32;
constexpr int kStepsMax = 3;  // steps between the (up to) four widths

struct AllocCfgDev {
  int num_heads, head_dim;
  int nb;            // number of available widths
  int bits[4];       // ascending
  double util[4];    // bits^alpha
  double budget, floor_, rank_thr, high_frac, high_boost;
  int intervals, min_high, scale_bits, critical_window;
  int nprot;
  int prot[SKV_ALLOC_MAX_PROTECTED];
};

struct SeqInfo {
  int n_prot;    // protected tokens (max bits, not ranked)
  int n_scored;  // unprotected tokens with a finite positive score
  int pad_[2];
};

// Workspace carved out of one caller buffer; every array but the last holds T (tok_*, rank_src) or 3T entries per sequence.
struct AllocWs {
  uint64_t *k64a, *k64b;
  uint32_t *v32a, *v32b;
  uint32_t* tok_slot;   // id order -> storage index
  uint32_t* rank_src;   // rank order -> id-order index
  int32_t* posof;       // item index -> walk position
  double* tok_score;
  uint8_t* tok_flags;   // bit0 protected, bit1 high, bit2 blocked (serial walk), bit3 reset streak
  int32_t* tok_acc;     // accepted steps
  uint8_t* item_valid;
  SeqInfo* info;        // [B]
};

__host__ __device__ inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

struct AllocParams {
  StoreGeom g;
  AllocCfgDev c;
  int T;  // slots
  const int32_t* counts;
  const int32_t* slot_token;
  const double* scores;
  const double* recency;
  double* rank_pct;
  int8_t* rank_streak;
  uint8_t* new_bits;
  int32_t* new_counts;
  int32_t* changed;
  AllocWs w;
};

__device__ __forceinline__ uint64_t desc_key(double x) {
  uint64_t u = (uint64_t)__double_as_longlong(x);
  u = (u >> 63) ? ~u : (u | 0x8000000000000000ull);  // ascending-sortable
  return ~u;                                         // descending
}

__device__ __forceinline__ bool is_protected(const AllocCfgDev& c, int id) {
  if (id < c.critical_window) return true;
  for (int i = 0; i < c.nprot; ++i)
    if (c.prot[i] == id) return true;
  return false;
}
__device__ __forceinline__ bool in_protected_list(const AllocCfgDev& c, int id) {
  for (int i = 0; i < c.nprot; ++i)
    if (c.prot[i] == id) return true;
  return false;
}

// ratio(payload) of cache.py:374-388 for n tokens
__device__ __forceinline__ double mem_ratio(const AllocCfgDev& c, int n, long long payload_bits) {
  const double elements = (double)(2 * c.num_heads * c.head_dim);
  const double scale_total = (double)((long long)n * 2 * c.num_heads * c.scale_bits);
  const double fp16_total = (double)n * elements * 16.0;
  return fp16_total > 0.0 ? ((double)payload_bits + scale_total) / fp16_total : 0.0;
}

__device__ __forceinline__ int slot_bucket(const StoreGeom& g, int s) {
  int b = 0;
#pragma unroll
  for (int i = 1; i < kNumBuckets; ++i)
    if (s >= g.bucket_base[i]) b = i;
  return b;
}

// ---- one sequence, one cluster --------------------------------------------------------------------------------
struct AllocShared {
  uint32_t hist[kAllocWarps][256];  // per warp: digit counts, then the next free position of every digit
  uint32_t digit_tot[2][256];       // this CTA's counts; double buffered, the other CTAs of the cluster read them
  typename cub::BlockScan<int, kAllocThreads>::TempStorage scan;
  int walk_tot[2], ev_pos[2], ev_cost[2], ev_incl[2];  // double buffered like digit_tot
  int need, bucket_hist[kNumBuckets], changed;
};

template <int CS>
__device__ __forceinline__ void cluster_sync() {
  if constexpr (CS == 1) __syncthreads();
  else cg::this_cluster().sync();
}
template <int CS>
__device__ __forceinline__ int cluster_rank() {
  return CS == 1 ? 0 : (int)cg::this_cluster().block_rank();
}
template <int CS, class X>
__device__ __forceinline__ X* cluster_peer(X* mine, int rank) {
  if constexpr (CS == 1) return mine;
  else return cg::this_cluster().map_shared_rank(mine, rank);
}

// Stable least-significant-digit radix sort of m (key, value) pairs by the low `bits` bits of the key, all CTAs of the cluster,
// between the buffers a and b (in L2); the pointers are swapped so that the result is in ka / va.  Each warp owns a
// contiguous piece of the input: it counts its digits, a scan over (digit, CTA, warp) turns the counts into positions, and a
// second sweep moves the pairs.  Digits on which all keys agree cost the count only.
template <int CS>
__device__ void cluster_radix_sort(uint64_t*& ka, uint32_t*& va, uint64_t*& kb, uint32_t*& vb, int m, int bits, int& parity,
                                   AllocShared& sh) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = cluster_rank<CS>();
  const int gw = rank * kAllocWarps + warp;
  const int lo = (int)((long long)m * gw / (CS * kAllocWarps)), hi = (int)((long long)m * (gw + 1) / (CS * kAllocWarps));
  for (int shift = 0; shift < bits; shift += 8, parity ^= 1) {
    for (int i = tid; i < kAllocWarps * 256; i += kAllocThreads) (&sh.hist[0][0])[i] = 0;
    __syncthreads();
    for (int i = lo + lane; i < hi; i += 32) atomicAdd(&sh.hist[warp][(uint32_t)(ka[i] >> shift) & 255u], 1u);
    __syncthreads();
    uint32_t mine = 0;
    if (tid < 256) {
#pragma unroll
      for (int w = 0; w < kAllocWarps; ++w) mine += sh.hist[w][tid];
      sh.digit_tot[parity][tid] = mine;
    }
    cluster_sync<CS>();
    uint32_t total = 0, lower = 0;
    if (tid < 256) {
#pragma unroll
      for (int c = 0; c < CS; ++c) {
        const uint32_t v = *cluster_peer<CS>(&sh.digit_tot[parity][tid], c);
        total += v;
        lower += c < rank ? v : 0u;
      }
    }
    if (__syncthreads_or(tid < 256 && (int)total == m)) continue;  // one digit for all
    int base;
    cub::BlockScan<int, kAllocThreads>(sh.scan).ExclusiveSum((int)total, base);
    if (tid < 256) {
      uint32_t at = (uint32_t)base + lower;
#pragma unroll
      for (int w = 0; w < kAllocWarps; ++w) {
        const uint32_t c = sh.hist[w][tid];
        sh.hist[w][tid] = at;
        at += c;
      }
    }
    __syncthreads();
    for (int i0 = lo; i0 < hi; i0 += 32) {
      const int i = i0 + lane;
      const bool in = i < hi;
      const uint64_t key = in ? ka[i] : 0ull;
      const uint32_t val = in ? va[i] : 0u;
      const uint32_t d = in ? (uint32_t)(key >> shift) & 255u : 256u;
      const uint32_t peers = __match_any_sync(0xffffffffu, d);
      const int before = __popc(peers & ((1u << lane) - 1u));
      uint32_t at = 0;
      if (in) at = sh.hist[warp][d] + before;
      __syncwarp();
      if (in && before == 0) sh.hist[warp][d] += __popc(peers);
      __syncwarp();
      if (in) {
        kb[at] = key;
        vb[at] = val;
      }
    }
    cluster_sync<CS>();
    uint64_t* tk = ka; ka = kb; kb = tk;
    uint32_t* tv = va; va = vb; vb = tv;
  }
}

// High-priority post-pass (cache.py:522-591), one CTA.  Usually nothing to do: the top-ranked tokens reach the widest width
// in phase 1.  When one of them did not, one thread replays the reference's loop literally.
__device__ void alloc_highpass(const AllocParams& p, int b, int n, int n_prot, int want, long long P, const uint32_t* rank,
                               const uint32_t* tok_slot, const double* tok_score, uint8_t* tok_flags, int32_t* tok_acc,
                               int32_t* undo, AllocShared& sh) {
  const int tid = threadIdx.x;
  const AllocCfgDev& c = p.c;
  const int nb = c.nb, hi = c.bits[nb - 1];
  if (tid == 0) sh.need = 0;
  __syncthreads();
  for (int r = tid; r < want; r += kAllocThreads) {
    const int i = (int)rank[r];
    if ((tok_flags[i] & 2) && c.bits[tok_acc[i]] < hi) sh.need = 1;
  }
  __syncthreads();
  if (!sh.need || tid != 0) return;

  const int n_ranked = n - n_prot;
  const long long elements = 2LL * c.num_heads * c.head_dim;
  const double limit = c.budget + 1e-6;
  for (int r = 0; r < want; ++r) {
    const int gt = (int)rank[r];
    if (!(tok_flags[gt] & 2)) continue;
    const int cur = c.bits[tok_acc[gt]];
    if (cur >= hi) continue;
    const long long delta = (long long)(hi - cur) * elements;
    double cand = mem_ratio(c, n, P + delta);
    if (cand > limit) {
      int n_undo = 0;
      bool fits = false;
      // victims in ascending score, equal scores in ascending id: walk the ranking from its tail,
      // each run of equal scores front to back; then the window-protected tokens (score +inf)
      auto try_victim = [&](int gc) -> bool {
        const uint8_t f = tok_flags[gc];
        if ((f & 2) || gc == gt) return false;
        // tokens on the protected list are never victims; a token protected only by the
        // critical window can be (cache.py:541-546 filters on the list alone)
        if ((f & 1) && in_protected_list(c, p.slot_token[(long long)b * p.T + tok_slot[gc]])) return false;
        const int acc = tok_acc[gc];
        if (acc <= 0) return false;
        const long long give = (long long)(c.bits[acc] - c.bits[acc - 1]) * elements;
        tok_acc[gc] = acc - 1;
        P -= give;
        undo[n_undo++] = gc;
        cand = mem_ratio(c, n, P + delta);
        return cand <= limit;
      };
      int r2 = n_ranked - 1;
      while (r2 >= 0 && !fits) {
        int g0 = r2;
        const double sc = tok_score[rank[r2]];
        while (g0 > 0 && tok_score[rank[g0 - 1]] == sc) --g0;
        for (int q = g0; q <= r2 && !fits; ++q) fits = try_victim((int)rank[q]);
        r2 = g0 - 1;
      }
      for (int q = n_ranked; q < n && !fits; ++q) fits = try_victim((int)rank[q]);
      if (!fits) {
        for (int u = n_undo - 1; u >= 0; --u) {
          const int gc = undo[u];
          const int acc = tok_acc[gc];
          P += (long long)(c.bits[acc + 1] - c.bits[acc]) * elements;
          tok_acc[gc] = acc + 1;
        }
        continue;
      }
      for (int u = 0; u < n_undo; ++u) tok_flags[undo[u]] |= 8;
    }
    tok_acc[gt] = nb - 1;
    P += delta;
    tok_flags[gt] |= 8;
  }
}

template <int CS>
__global__ void __launch_bounds__(kAllocThreads) alloc_kernel(const __grid_constant__ AllocParams p) {
  __shared__ AllocShared sh;
  const int rank = cluster_rank<CS>(), b = (int)blockIdx.x / CS, tid = threadIdx.x, T = p.T;
  const int ct = rank * kAllocThreads + tid;      // thread of the cluster
  constexpr int NT = CS * kAllocThreads;
  const AllocCfgDev& c = p.c;
  const long long t1 = (long long)b * T, t3 = 3 * t1;
  uint64_t *ka = p.w.k64a + t3, *kb = p.w.k64b + t3;
  uint32_t *va = p.w.v32a + t3, *vb = p.w.v32b + t3;
  uint32_t* tok_slot = p.w.tok_slot + t1;
  uint32_t* rank_src = p.w.rank_src + t1;
  int32_t* posof = p.w.posof + t3;
  double* tok_score = p.w.tok_score + t1;
  uint8_t* tok_flags = p.w.tok_flags + t1;
  int32_t* tok_acc = p.w.tok_acc + t1;
  uint8_t* item_valid = p.w.item_valid + t3;
  SeqInfo* info = p.w.info + b;
  int cnt[kNumBuckets], n = 0;
#pragma unroll
  for (int i = 0; i < kNumBuckets; ++i) {
    cnt[i] = p.counts[b * kNumBuckets + i];
    n += cnt[i];
  }
  int parity = 0;

  // ---- 1. live tokens, sorted by id; results start empty ----
  for (int s = ct; s < T; s += NT) p.new_bits[t1 + s] = 0;
  if (ct < kNumBuckets) p.new_counts[b * kNumBuckets + ct] = 0;
  if (ct == 0) {
    p.changed[b] = 0;
    info->n_prot = 0;
    info->n_scored = 0;
  }
  if (tid < kNumBuckets) sh.bucket_hist[tid] = 0;
  if (tid == 0) sh.changed = 0;
  if (n == 0) return;  // the same for every CTA of the cluster
  for (int j = ct; j < n; j += NT) {
    int rem = j, s = 0;
#pragma unroll
    for (int i = 0; i < kNumBuckets; ++i) {
      if (rem >= 0 && rem < cnt[i]) s = p.g.bucket_base[i] + rem;
      rem -= cnt[i];
      if (rem < 0) rem = -(1 << 30);
    }
    ka[j] = (uint64_t)(uint32_t)p.slot_token[t1 + s];
    va[j] = (uint32_t)s;
  }
  cluster_sync<CS>();
  cluster_radix_sort<CS>(ka, va, kb, vb, n, 32, parity, sh);

  // ---- 2. scores -> descending sort keys ----
  // (key, value) pairs of the ranking go to the other buffers: this loop reads va
  for (int j = ct; j < n; j += NT) {
    const uint32_t s = va[j];
    const int id = p.slot_token[t1 + s];
    double score = p.scores[t1 + s];
    if (p.recency) score *= p.recency[t1 + s];
    const bool prot = is_protected(c, id);
    if (prot) score = INFINITY;
    tok_slot[j] = s;
    tok_score[j] = score;
    tok_flags[j] = prot ? 1 : 0;
    tok_acc[j] = prot ? c.nb - 1 : 0;  // protected tokens sit at the widest width (cache.py:364-368)
    kb[j] = prot ? ~0ull : desc_key(score);
    vb[j] = (uint32_t)j;
    if (prot) atomicAdd(&info->n_prot, 1);
    const uint32_t active = __activemask();
    const uint32_t scored = __ballot_sync(active, !prot && isfinite(score) && score > 0.0);
    if ((tid & 31) == __ffs(active) - 1 && scored) atomicAdd(&info->n_scored, __popc(scored));
  }
  cluster_sync<CS>();
  cluster_radix_sort<CS>(kb, vb, ka, va, n, 64, parity, sh);
  for (int r = ct; r < n; r += NT) rank_src[r] = vb[r];
  cluster_sync<CS>();

  // ---- 3. ranks, hysteresis state, high-priority set, item keys ----
  const int n_prot = info->n_prot, n_scored = info->n_scored;
  const int n_ranked = n - n_prot, n_items = 3 * n;
  const int lo = c.bits[0], hi = c.bits[c.nb - 1];
  const long long elements = 2LL * c.num_heads * c.head_dim;
  int want = 0;
  if ((c.high_frac > 0.0 || c.min_high > 0) && n_scored > 0) {
    const int byfrac = (int)ceil((double)n_scored * c.high_frac);
    want = c.min_high > byfrac ? c.min_high : byfrac;
    if (want > n_scored) want = n_scored;
  }
  const long long payload0 = (long long)n_ranked * lo * elements + (long long)n_prot * hi * elements;
  const bool gated0 = mem_ratio(c, n, payload0) >= c.budget * 0.85;
  int max_cost = 0, min_cost = 1 << 30;
  for (int i = 0; i + 1 < c.nb; ++i) {
    max_cost = max(max_cost, c.bits[i + 1] - c.bits[i]);
    min_cost = min(min_cost, c.bits[i + 1] - c.bits[i]);
  }
  // a single step may carry the ratio from below the gate past the budget: walk serially
  const double step_ratio = (double)max_cost / ((double)n * 16.0);
  const bool serial = !(step_ratio * 1.0000001 + 1e-9 < 0.15 * c.budget - 1e-6);

  for (int r = ct; r < n; r += NT) {
    const int i = (int)rank_src[r];
    uint64_t key[kStepsMax] = {~0ull, ~0ull, ~0ull};
    uint8_t valid[kStepsMax] = {0, 0, 0};
    const long long gs = t1 + tok_slot[i];
    uint8_t flags = tok_flags[i];
    int8_t streak = p.rank_streak[gs];
    if (flags & 1) {
      // cache.py:448-450: an unranked token without state gets the neutral record
      if (streak < 0) {
        p.rank_pct[gs] = 1.0;
        p.rank_streak[gs] = (int8_t)c.intervals;
      }
    } else {
      // rank percentile and streak (cache.py:423-446)
      const int den = (n_ranked - 1) > 1 ? (n_ranked - 1) : 1;
      const double pct = n_ranked == 1 ? 0.0 : (double)r / (double)den;
      if (streak < 0) {
        streak = (int8_t)c.intervals;
      } else {
        const bool moved = fabs(pct - p.rank_pct[gs]) >= c.rank_thr;
        streak = moved ? (int8_t)((streak + 1) < c.intervals ? (streak + 1) : c.intervals) : (int8_t)0;
      }
      p.rank_pct[gs] = pct;
      p.rank_streak[gs] = streak;
      const bool high = r < want;  // positive finite scores sort first, so rank < want implies both
      if (high) flags |= 2;
      tok_flags[i] = flags;

      // items (cache.py:455-482); gated from the start and not moving: not even the first step is pushed
      double imp = tok_score[i];
      if (!isfinite(imp)) imp = c.floor_ > 0.0 ? c.floor_ : 0.0;
      if (imp <= 0.0) imp = c.floor_ > 0.0 ? c.floor_ : 0.0;
      if (imp > 0.0 && !(gated0 && streak < c.intervals)) {
        double eff = INFINITY;
#pragma unroll
        for (int k = 0; k < kStepsMax; ++k) {
          if (k + 1 >= c.nb) break;
          const int cur = c.bits[k], nxt = c.bits[k + 1];
          double v = imp;
          if (high && nxt >= hi) v *= c.high_boost;
          const double gain = c.util[k + 1] - c.util[k];
          if (gain <= 0.0 || nxt - cur <= 0) break;
          const double own = (v * gain) / (double)(nxt - cur);
          eff = own < eff ? own : eff;
          key[k] = desc_key(eff);
          valid[k] = 1;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kStepsMax; ++k) {
      ka[3 * i + k] = key[k];
      va[3 * i + k] = (uint32_t)(3 * i + k);
      item_valid[3 * i + k] = valid[k];
    }
  }
  cluster_sync<CS>();
  cluster_radix_sort<CS>(ka, va, kb, vb, n_items, 64, parity, sh);
  for (int pos = ct; pos < n_items; pos += NT) posof[va[pos]] = pos;
  cluster_sync<CS>();

  // ---- 4. the walk ----
  const double gate = c.budget * 0.85, limit = c.budget + 1e-6;
  long long P = payload0;
  if (serial) {
    // tiny cache: the literal walk (accept iff the token sits at the step's width, is not
    // gate-blocked and the step fits)
    if (rank == 0 && tid == 0) {
      for (int pos = 0; pos < n_items; ++pos) {
        const int it = (int)va[pos];
        if (!item_valid[it]) continue;
        const int i = it / 3, step = it - 3 * i;
        if (tok_acc[i] != step || (tok_flags[i] & 4)) continue;
        const long long delta = (long long)(c.bits[step + 1] - c.bits[step]) * elements;
        if (mem_ratio(c, n, P + delta) > limit) continue;
        tok_acc[i] = step + 1;
        P += delta;
        tok_flags[i] |= 8;
        if (mem_ratio(c, n, P) >= gate) tok_flags[i] |= 4;
      }
    }
  } else {
    int phase = gated0 ? 2 : 1;  // 1 = before the gate, 2 = after it
    int c1 = -1;                 // position of the accept that reached the gate (-1: gated from the start)
    int dead = 1 << 30;          // steps of this cost or more no longer fit
    int start = 0, par = 0;
    // Every turn finds the next event (the gate reached, or a step that does not fit) by prefix sums over the thread's, the
    // CTA's and the cluster's pieces of the walk, and accepts what lies before it: at most one turn per distinct cost and
    // one for the gate.
    const int seg_lo = (int)((long long)n_items * ct / NT), seg_hi = (int)((long long)n_items * (ct + 1) / NT);
    auto cost_at = [&](int pos, int& item) -> int {  // 0: not eligible
      item = (int)va[pos];
      if (!item_valid[item]) return 0;
      const int step = item % 3, cost = c.bits[step + 1] - c.bits[step];
      return (phase == 1 || (cost < dead && (step == 0 || posof[item - 1] < c1))) ? cost : 0;
    };
    auto hits = [&](long long units) -> bool {
      const double ratio = mem_ratio(c, n, P + units * elements);
      return phase == 1 ? ratio >= gate : ratio > limit;
    };
    while (start < n_items) {
      if (tid == 0) sh.ev_pos[par] = INT_MAX;
      const int from = max(seg_lo, start);
      int sum = 0, item;
      for (int pos = from; pos < seg_hi; ++pos) sum += cost_at(pos, item);
      int excl, tot;
      cub::BlockScan<int, kAllocThreads>(sh.scan).ExclusiveSum(sum, excl, tot);
      if (tid == 0) sh.walk_tot[par] = tot;
      cluster_sync<CS>();
      int before = excl, all = 0;
#pragma unroll
      for (int q = 0; q < CS; ++q) {
        const int v = *cluster_peer<CS>(&sh.walk_tot[par], q);
        all += v;
        before += q < rank ? v : 0;
      }
      // the first event of the walk lies with the thread whose items carry the sum across the line
      if (sum > 0 && hits(before + sum) && !(before > 0 && hits(before))) {
        int incl = before;
        for (int pos = from; pos < seg_hi; ++pos) {
          const int cost = cost_at(pos, item);
          incl += cost;
          if (cost > 0 && hits(incl)) {
            sh.ev_pos[par] = pos;
            sh.ev_cost[par] = cost;
            sh.ev_incl[par] = incl;
            break;
          }
        }
      }
      cluster_sync<CS>();
      int ev = INT_MAX, ev_cost = 0, ev_incl = 0;
#pragma unroll
      for (int q = 0; q < CS; ++q) {
        const int v = *cluster_peer<CS>(&sh.ev_pos[par], q);
        if (v < ev) {
          ev = v;
          ev_cost = *cluster_peer<CS>(&sh.ev_cost[par], q);
          ev_incl = *cluster_peer<CS>(&sh.ev_incl[par], q);
        }
      }
      // phase 1: the item that reaches the gate is itself accepted; phase 2: the failing item is not
      const int until = min(seg_hi, phase == 1 && ev != INT_MAX ? ev + 1 : ev);
      for (int pos = from; pos < until; ++pos) {
        if (cost_at(pos, item) == 0) continue;
        const int i = item / 3;
        atomicMax(&tok_acc[i], item - 3 * i + 1);
        tok_flags[i] |= 8;  // two steps of one token may set the same bit at once: same value either way
      }
      if (ev == INT_MAX) {
        P += (long long)all * elements;
        break;
      }
      start = ev + 1;
      if (phase == 1) {
        P += (long long)ev_incl * elements;
        phase = 2;
        c1 = ev;
      } else {
        P += (long long)(ev_incl - ev_cost) * elements;
        dead = ev_cost;
        if (ev_cost <= min_cost) break;
      }
      par ^= 1;
    }
  }
  cluster_sync<CS>();

  // ---- 5. high-priority post-pass ----
  if (rank == 0)
    alloc_highpass(p, b, n, n_prot, want, P, rank_src, tok_slot, tok_score, tok_flags, tok_acc, reinterpret_cast<int32_t*>(vb), sh);
  cluster_sync<CS>();

  // ---- 6. results in storage order ----
  for (int i = ct; i < n; i += NT) {
    const int s = (int)tok_slot[i];
    const int bits = c.bits[tok_acc[i]];
    p.new_bits[t1 + s] = (uint8_t)bits;
    if (tok_flags[i] & 8) p.rank_streak[t1 + s] = 0;  // accepted or touched by the post-pass (cache.py:511-514)
    atomicAdd(&sh.bucket_hist[bits_bucket(bits)], 1);
    if (bucket_bits(slot_bucket(p.g, s)) != bits) atomicAdd(&sh.changed, 1);
  }
  __syncthreads();
  if (tid < kNumBuckets && sh.bucket_hist[tid]) atomicAdd(&p.new_counts[b * kNumBuckets + tid], sh.bucket_hist[tid]);
  if (tid == 0 && sh.changed) atomicAdd(&p.changed[b], sh.changed);
  cluster_sync<CS>();  // no CTA leaves while another may still read its shared memory
}

template <int CS>
static int launch_alloc(const AllocParams& p, int B, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(B * CS);
  cfg.blockDim = dim3(kAllocThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CS > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, alloc_kernel<CS>, p) == cudaSuccess ? SKV_OK : SKV_ERR_CUDA;
}

}  // namespace skv

using namespace skv;

namespace {

// lays the workspace out inside `base` (nullptr: size query); returns the bytes needed
size_t carve(AllocWs& w, void* base, long long NT) {
  size_t off = 0;
  auto take = [&](size_t bytes) -> void* {
    void* ptr = base ? static_cast<uint8_t*>(base) + off : nullptr;
    off += align_up(bytes, 256);
    return ptr;
  };
  w.k64a = (uint64_t*)take(3 * NT * 8);
  w.k64b = (uint64_t*)take(3 * NT * 8);
  w.v32a = (uint32_t*)take(3 * NT * 4);
  w.v32b = (uint32_t*)take(3 * NT * 4);
  w.tok_slot = (uint32_t*)take(NT * 4);
  w.rank_src = (uint32_t*)take(NT * 4);
  w.posof = (int32_t*)take(3 * NT * 4);
  w.tok_score = (double*)take(NT * 8);
  w.tok_flags = (uint8_t*)take(NT);
  w.tok_acc = (int32_t*)take(NT * 4);
  w.item_valid = (uint8_t*)take(3 * NT);
  w.info = (SeqInfo*)take(1024 * sizeof(SeqInfo));
  return off;
}

}  // namespace

extern "C" int64_t skv_alloc_workspace_bytes(const SkvStoreDesc* desc) {
  if (!desc || desc->num_seqs <= 0 || desc->slots <= 0) return SKV_ERR_INVALID;
  AllocWs w;
  return (int64_t)carve(w, nullptr, (long long)desc->num_seqs * desc->slots);
}

extern "C" int skv_alloc_bits(const SkvStoreDesc* desc, const SkvAllocConfig* cfg, const int32_t* counts,
                              const int32_t* slot_token, const double* scores, const double* recency,
                              double* rank_pct, int8_t* rank_streak, uint8_t* new_bits, int32_t* new_counts,
                              int32_t* changed, void* workspace, void* stream) {
  if (!desc || !cfg || !counts || !slot_token || !scores || !rank_pct || !rank_streak || !new_bits || !new_counts ||
      !changed || !workspace)
    return SKV_ERR_INVALID;
  if (cfg->num_bits < 1 || cfg->num_bits > 4 || cfg->num_protected < 0 || cfg->num_protected > SKV_ALLOC_MAX_PROTECTED)
    return SKV_ERR_INVALID;
  if (!cfg->use_packing) return SKV_ERR_UNSUPPORTED;  // the store is always packed
  if (desc->num_seqs > 1024) return SKV_ERR_UNSUPPORTED;
  for (int i = 0; i < cfg->num_bits; ++i) {
    if (bits_bucket(cfg->bits[i]) < 0) return SKV_ERR_INVALID;
    if (i > 0 && cfg->bits[i] <= cfg->bits[i - 1]) return SKV_ERR_INVALID;
  }
  const int B = desc->num_seqs, T = desc->slots;
  const long long NT = (long long)B * T;
  if (3 * NT >= (1ll << 31)) return SKV_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  AllocParams p;
  p.g = make_geom(*desc);
  p.T = T;
  p.c.num_heads = cfg->num_heads;
  p.c.head_dim = cfg->head_dim;
  p.c.nb = cfg->num_bits;
  for (int i = 0; i < 4; ++i) {
    p.c.bits[i] = i < cfg->num_bits ? cfg->bits[i] : 0;
    p.c.util[i] = i < cfg->num_bits ? cfg->util[i] : 0.0;
  }
  p.c.budget = cfg->memory_budget;
  p.c.floor_ = cfg->importance_floor > 0.0 ? cfg->importance_floor : 0.0;
  p.c.rank_thr = cfg->rank_threshold > 0.0 ? cfg->rank_threshold : 0.0;
  p.c.high_frac = cfg->high_fraction < 0.0 ? 0.0 : (cfg->high_fraction > 0.5 ? 0.5 : cfg->high_fraction);
  p.c.high_boost = cfg->high_boost < 1.0 ? 1.0 : cfg->high_boost;
  p.c.intervals = cfg->hysteresis_intervals < 1 ? 1 : cfg->hysteresis_intervals;
  p.c.min_high = cfg->min_high_tokens < 0 ? 0 : cfg->min_high_tokens;
  p.c.scale_bits = cfg->scale_bits == 16 ? 16 : 32;
  p.c.critical_window = cfg->critical_window;
  p.c.nprot = cfg->num_protected;
  for (int i = 0; i < SKV_ALLOC_MAX_PROTECTED; ++i) p.c.prot[i] = i < cfg->num_protected ? cfg->protected_ids[i] : -1;
  p.counts = counts;
  p.slot_token = slot_token;
  p.scores = scores;
  p.recency = recency;
  p.rank_pct = rank_pct;
  p.rank_streak = rank_streak;
  p.new_bits = new_bits;
  p.new_counts = new_counts;
  p.changed = changed;
  carve(p.w, workspace, NT);

  // CTAs per sequence: one per 4096 storage indices (about a thousand live tokens: a couple per thread) as long as all sequences'
  // clusters run at once.  A cluster lies in one GPC and a CTA fills an SM's registers, so 74 clusters of 2, 33 of 4, 15 of 8 and
  // 7 of 16 do: 16 x 8192 tokens take 403 us with clusters of 8, in two waves, and 290 with clusters of 4.  Beyond 8, the portable
  // size, one sequence of 131072 tokens takes 864 instead of 1548 us (1425 with the device-wide sorts before the clusters).
  int cs = 1;
  if (T > 4096 && B <= 74) cs = 2;
  if (T > 2 * 4096 && B <= 33) cs = 4;
  if (T > 4 * 4096 && B <= 15) cs = 8;
  if (T > 8 * 4096 && B <= 7) {
    if (cudaFuncSetAttribute(alloc_kernel<16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        launch_alloc<16>(p, B, st) == SKV_OK)
      return cudaGetLastError() == cudaSuccess ? SKV_OK : SKV_ERR_CUDA;
    cudaGetLastError();  // such clusters are not to be had here
  }
  const int rc = cs == 1 ? launch_alloc<1>(p, B, st) : cs == 2 ? launch_alloc<2>(p, B, st)
               : cs == 4 ? launch_alloc<4>(p, B, st) : launch_alloc<8>(p, B, st);
  if (rc != SKV_OK) return rc;
  return cudaGetLastError() == cudaSuccess ? SKV_OK : SKV_ERR_CUDA;
}
