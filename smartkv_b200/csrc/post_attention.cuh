// Block-level bodies of the three steps that follow the streaming attention kernel of a layer:
//   combine     fold the split-KV partials of a (sequence, KV head), add the current token in full
//               precision, normalise (smartkv/core/fused_cpu.py:115-137)
//   importance  per-key attention mass -> cumulative importance + per-layer EMA
//               (smartkv/core/cache.py:232-264, smartkv/core/importance.py:44-101)
//   append      quantise + pack the step's new token into the store (smartkv/core/cache.py:1187-1355)
// The importance step of a layer needs what that layer's combine step produced, but nothing stops
// it from running one launch later: post_attention.cu runs the combine and the append of layer l
// side by side with the importance step of the layer before it.  The stand-alone entry points run
// the same bodies from their own kernels.
#pragma once

#include "attn_sched.cuh"
#include "quant_row.cuh"

namespace skv {

constexpr int kPostThreads = 256;
constexpr int kCombineChunk = 256;
constexpr int kMaxQHeads = 128;

bool attn_first_of_run(const SkvStoreDesc* desc, int query_dtype);  // decode_attention.cu

__host__ __device__ inline int partial_stride(int group, int head_dim) { return group * (head_dim + 2); }

__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// ---- combine ----------------------------------------------------------------------------------------
struct CombineParams {
  StoreGeom g;
  const int* plan;
  const void* query;
  int q_is_half;
  int num_q_heads;
  int group;
  const float* partials;
  int per_run;  // partials a run has room for
  int num_ctas;
  const void* cur_k;
  const void* cur_v;
  int kv_is_half;
  const float* cur_mask;  // additive mask of the current token per sequence, natural-log units (may be null)
  float* out;
  float* lse_max;
  float* lse_sum;
  float* cur_prob;
  float scale_log2;
};

__host__ __device__ inline int combine_heads_per_block(int head_dim) { return kPostThreads / head_dim; }
__host__ __device__ inline int combine_units(const StoreGeom& g, int group) {
  const int hpb = combine_heads_per_block(g.head_dim);
  return g.num_seqs * g.num_kv_heads * ((group + hpb - 1) / hpb);
}

struct CombineShared {
  float red[kPostThreads / 32][2];
  float f[kPostThreads / 64][kCombineChunk];   // per head of the block
  float lf[kPostThreads / 64][kCombineChunk];
};

// The scaled logit of the current token for one query head: q . k * scale, reduced over the D threads
// of the head in a fixed shape (warp tree, then the warps of the head in order).
// `sub` = head slot inside the block, `d` = thread's element.
__device__ __forceinline__ float head_dot(float prod, int sub, int d, int D, float (*red)[2], int slot) {
  const float s = warp_sum(prod);
  const int warp_in_head = d >> 5, lane = d & 31, wph = D >> 5;
  if (lane == 0) red[sub * wph + warp_in_head][slot] = s;
  __syncthreads();
  float acc = 0.f;
  for (int w = 0; w < wph; ++w) acc += red[sub * wph + w][slot];
  return acc;
}

// One unit = up to kPostThreads / D query heads of one (sequence, KV head); blockDim.x == kPostThreads.
// FIRST: of a run's partials only the first is filled, and of a segment's last run the second (fp16 queries,
// attn_first_of_run); otherwise all of them.
template <bool FIRST>
__device__ __forceinline__ void combine_unit(const CombineParams& p, int unit, CombineShared& sh) {
  const StoreGeom& g = p.g;
  const int D = g.head_dim, G = p.group, Hkv = g.num_kv_heads;
  const int hpb = combine_heads_per_block(D), groups = (G + hpb - 1) / hpb;
  const int seg = unit / groups, hg = unit - seg * groups;
  const int b = seg / Hkv, h = seg - b * Hkv;
  const int tid = threadIdx.x, sub = tid / D, d = tid - sub * D;
  const int gq = hg * hpb + sub;
  const bool valid = gq < G;
  const int gqc = valid ? gq : G - 1;  // threads of a missing head go through the motions of the last one
  const PlanView pv = plan_view(const_cast<int*>(p.plan), p.num_ctas, g.num_seqs * Hkv);
  const int runs = pv.seg_count[seg];
  const int nsplit = runs == 0 ? 0 : FIRST ? runs + 1 : runs * p.per_run;
  const int r0 = runs > 0 ? pv.seg_begin[seg] * p.per_run : 0;
  const int pstride = partial_stride(G, D);
  // the k-th filled partial, in floats from the segment's first (its runs are at most one a CTA)
  const int step = (FIRST ? p.per_run : 1) * pstride, last = (runs - 1) * step + pstride;
  auto at = [&](int k) { return FIRST && k == runs ? last : k * step; };
  const float* base = p.partials + (long long)r0 * pstride + gqc * (D + 2);
  const bool has_cur = p.cur_k != nullptr && p.cur_v != nullptr;
  const long long hq = (long long)b * p.num_q_heads + h * G + gqc;
  const long long kv = ((long long)b * Hkv + h) * D + d;

  // kRowsAhead rows at a time, their loads in flight together and the first of them beside the headers: a loop over the rows
  // with a load each waits for every one (segments of 12 and of 40 partials: the last block ended 7.0 and 14.2 us after
  // the attention launch, now 4.3 and 8 us).  Where a run leaves one partial the lists are short and eight do: sixteen and
  // twenty-four cost more in code and registers than the round trips they save (8 x 770 keys, 22 layers: 276 us a step at eight,
  // 8 and 22 us more at sixteen and twenty-four).  Where it leaves seven (fp32 queries) or four (tensor memory) a segment
  // has up to a thousand and sixteen are needed (us for four layers, one KV head, eight / sixteen: 1 x 2048 keys fp32 337 / 221,
  // 1 x 131072 fp32 439 / 304, tensor memory 308 / 232; eight KV heads: 1 x 2048 107 / 90, 16 x 8192 278 / 278).
  constexpr int kRowsAhead = FIRST ? 8 : 16;
  float x[kRowsAhead];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int k = 0; k < kRowsAhead; ++k) x[k] = k0 + k < nsplit ? base[at(k0 + k) + 2 + d] : 0.f;
  };
  fetch(0);
  float prod = 0.f;
  if (has_cur) {
    const float q = p.q_is_half ? __half2float(static_cast<const __half*>(p.query)[hq * D + d])
                                : static_cast<const float*>(p.query)[hq * D + d];
    const float k = p.kv_is_half ? __half2float(static_cast<const __half*>(p.cur_k)[kv])
                                 : static_cast<const float*>(p.cur_k)[kv];
    prod = q * k;
  }
  // (max, sum) headers of this thread's share of the partials: one 8-byte load each, kept in registers
  // when the segment has at most kCombineChunk partials (the usual case), so that the chain of
  // dependent loads is plan -> headers -> rows and nothing more
  constexpr int kHdrRegs = kCombineChunk / 64;  // D >= 64
  const bool small = nsplit <= kCombineChunk;
  float2 hdr[kHdrRegs];
  float mloc = -INFINITY;
  if (small) {
#pragma unroll
    for (int j = 0; j < kHdrRegs; ++j) {
      const int k = d + j * D;
      hdr[j] = k < nsplit ? *reinterpret_cast<const float2*>(base + at(k)) : make_float2(-INFINITY, 0.f);
      mloc = fmaxf(mloc, hdr[j].x);
    }
  } else {
    for (int k = d; k < nsplit; k += D) mloc = fmaxf(mloc, base[at(k)]);
  }
  float s_cur = head_dot(prod, sub, d, D, sh.red, 0) * p.scale_log2;
  if (has_cur && p.cur_mask != nullptr) s_cur = fmaf(p.cur_mask[b], 1.4426950408889634f, s_cur);
  {
    const float m = warp_max(mloc);
    const int wph = D >> 5;
    if ((d & 31) == 0) sh.red[sub * wph + (d >> 5)][1] = m;
    __syncthreads();
    mloc = -INFINITY;
    for (int w = 0; w < wph; ++w) mloc = fmaxf(mloc, sh.red[sub * wph + w][1]);
  }
  float M = mloc;
  if (has_cur) M = fmaxf(M, s_cur);

  // fold the partials in a fixed order, kCombineChunk at a time; the weights of a chunk go through
  // shared memory so that the row loads do not depend on anything loaded in the same loop
  float acc = 0.f, L = 0.f;
  for (int c0 = 0; c0 < nsplit; c0 += kCombineChunk) {
    const int cn = (nsplit - c0) < kCombineChunk ? (nsplit - c0) : kCombineChunk;
    __syncthreads();
    if (small) {
#pragma unroll
      for (int j = 0; j < kHdrRegs; ++j) {
        const int k = d + j * D;
        if (k < cn) {
          const float f = hdr[j].x == -INFINITY ? 0.f : ex2f(hdr[j].x - M);
          sh.f[sub][k] = f;
          sh.lf[sub][k] = f == 0.f ? 0.f : hdr[j].y * f;
        }
      }
    } else {
      for (int k = d; k < cn; k += D) {
        const float* row = base + at(c0 + k);
        const float mw = row[0];
        const float f = mw == -INFINITY ? 0.f : ex2f(mw - M);
        sh.f[sub][k] = f;
        sh.lf[sub][k] = f == 0.f ? 0.f : row[1] * f;
      }
    }
    __syncthreads();
    for (int k0 = 0; k0 < cn; k0 += kRowsAhead) {
      if (c0 + k0 > 0) fetch(c0 + k0);  // the first rows are on their way since the headers
#pragma unroll
      for (int k = 0; k < kRowsAhead; ++k) {
        if (k0 + k < cn) {
          const float f = sh.f[sub][k0 + k];
          acc = f == 0.f ? acc : fmaf(x[k], f, acc);  // a partial without keys holds stale bytes: select, not multiply
          L += sh.lf[sub][k0 + k];
        }
      }
    }
  }
  float pc = 0.f;
  if (has_cur) {
    pc = ex2f(s_cur - M);
    const float v = p.kv_is_half ? __half2float(static_cast<const __half*>(p.cur_v)[kv])
                                 : static_cast<const float*>(p.cur_v)[kv];
    acc = fmaf(pc, v, acc);
    L += pc;
  }
  if (!valid) return;
  p.out[hq * D + d] = L > 0.f ? acc / L : 0.f;
  if (d == 0) {
    if (p.lse_max) p.lse_max[hq] = M;
    if (p.lse_sum) p.lse_sum[hq] = L;
    if (p.cur_prob) p.cur_prob[hq] = (has_cur && L > 0.f) ? pc / L : 0.f;
  }
}

// ---- importance ---------------------------------------------------------------------------------------
struct ImportanceParams {
  StoreGeom g;
  int layer;
  const int32_t* counts;
  int num_q_heads;
  const float* logits;
  const float* lse_max;
  const float* lse_sum;
  const float* cur_prob;
  const int32_t* cur_slot;
  float* head_state;
  int parity;
  double* cumulative;
  float* layer_ema;
  uint8_t* touched;
  float decay;
  float head_decay;
};

struct ImportanceShared {
  float w[kMaxQHeads];      // head weight / final sum
  float mx[kMaxQHeads];     // final max
  float cprob[kMaxQHeads];  // pc (unnormalised probability of the current token)
};

// Maps the j-th *live* chunk of sequence b (chunks of CHUNK storage indices that hold a cached
// key or the slot the current token will take) to its chunk index; -1 when j is past the last one.
// Buckets lie at increasing storage indices, so their chunk ranges are increasing; a chunk that several buckets share belongs to
// the first of them.  j == 0 always maps to a chunk (chunk 0 if nothing is live): that block publishes the
// head-importance EMA.
template <int CHUNK>
__device__ __forceinline__ int live_chunk(const StoreGeom& g, const int32_t* counts4, int j) {
  int prev_last = -1, seen = 0;
#pragma unroll
  for (int i = 0; i < kNumBuckets; ++i) {
    const int cnt = counts4[i] + 1;  // + the slot a token appended this step would take
    if (g.cap[i] == 0) continue;
    int first = g.bucket_base[i] / CHUNK;
    const int last = (g.bucket_base[i] + cnt - 1) / CHUNK;
    if (first <= prev_last) first = prev_last + 1;
    if (last >= first) {
      const int n = last - first + 1;
      if (j < seen + n) return first + (j - seen);
      seen += n;
      prev_last = last;
    }
  }
  return (j == 0 && seen == 0) ? 0 : -1;
}

// Bucket counts and the current token's slot of one sequence.
struct ImportanceSeq {
  int cnt[kNumBuckets];
  int cur_slot;
  bool has_cur;
};

__device__ __forceinline__ ImportanceSeq importance_seq(const ImportanceParams& p, int b) {
  ImportanceSeq q;
#pragma unroll
  for (int i = 0; i < kNumBuckets; ++i) q.cnt[i] = p.counts[b * kNumBuckets + i];
  q.cur_slot = (p.cur_prob != nullptr && p.cur_slot != nullptr) ? p.cur_slot[b] : -1;
  q.has_cur = q.cur_slot >= 0;
  return q;
}

// How an importance block works: KPT consecutive storage indices a thread, HEADS rows of logits in flight, and whether the
// arrays are aligned for loads of four elements (they are the caller's).
template <int KPT_, int HEADS_, bool VEC_>
struct ImpShape {
  static constexpr int KPT = KPT_, HEADS = HEADS_, CHUNK = KPT * kPostThreads;
  static constexpr bool VEC = VEC_;
  static_assert(KPT == 1 || KPT == 4, "one or four indices a thread");
};
template <class S>
__device__ __forceinline__ void load_k(const float* p, float (&x)[S::KPT]) {
  if constexpr (S::VEC && S::KPT == 4) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
  } else {
#pragma unroll
    for (int i = 0; i < S::KPT; ++i) x[i] = p[i];
  }
}
template <class S>
__device__ __forceinline__ void load_k(const double* p, double (&x)[S::KPT]) {
  if constexpr (S::VEC && S::KPT == 4) {
    const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
    x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
  } else {
#pragma unroll
    for (int i = 0; i < S::KPT; ++i) x[i] = p[i];
  }
}
template <class S>
__device__ __forceinline__ void load_k(const uint8_t* p, uint8_t (&x)[S::KPT]) {
  if constexpr (S::VEC && S::KPT == 4) {
    const uchar4 v = *reinterpret_cast<const uchar4*>(p);
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
  } else {
#pragma unroll
    for (int i = 0; i < S::KPT; ++i) x[i] = p[i];
  }
}

// One chunk of sequence b; blockDim.x == kPostThreads.  `publish` marks the one block per sequence that writes the new
// head-importance EMA.
//
// Bound: round trips to memory, three one after the other (counts; state, (max, sum) and the first logits; the other logits)
// for few bytes a thread.  So every load that needs no weight is issued before the weights are worked out, and a launch of more
// than a wave of single indices takes four consecutive ones a thread with 16-byte loads.  64 x 16384 keys, 8 heads: from
// the end of the attention launch to the last block's 29 us -> 19.
template <class S>
__device__ __forceinline__ void importance_block(const ImportanceParams& p, int chunk, int b, bool publish, ImportanceShared& sh) {
  constexpr int KPT = S::KPT, HEADS = S::HEADS;
  const StoreGeom& g = p.g;
  const int tid = threadIdx.x, Hq = p.num_q_heads;
  const ImportanceSeq q = importance_seq(p, b);
  int total_keys = q.has_cur ? 1 : 0;
#pragma unroll
  for (int i = 0; i < kNumBuckets; ++i) total_keys += q.cnt[i];

  // The thread's storage indices s .. s + KPT - 1 lie in one bucket (capacities are multiples of 128): those before `live` hold
  // cached keys, `cur` is the one the current token will lie at.
  const int s = chunk * S::CHUNK + KPT * tid;
  int live = 0;
#pragma unroll
  for (int i = 0; i < kNumBuckets; ++i)
    if (s >= g.bucket_base[i] && s < g.bucket_base[i] + g.cap[i]) live = q.cnt[i] - (s - g.bucket_base[i]);
  const int cur = q.has_cur ? q.cur_slot - s : -1;
  const bool with_cur = cur >= 0 && cur < KPT && cur >= live;
  const bool active = live > 0 || with_cur;
  // most storage indices of a sequence are unused capacity: a block without a live key leaves at once
  // (the publishing block of every sequence stays)
  if (!__syncthreads_or(active || publish)) return;

  // final (max, sum) of every query head and the probability of the current token, as the combine
  // step of this layer left them; the state the thread updates; the first logits
  float lse_l = 0.f, lse_m = 0.f, pcur = 0.f, hs = 0.f;
  const float* hs_old = p.head_state + ((long long)b * 2 + p.parity) * Hq;
  float* hs_new = p.head_state + ((long long)b * 2 + (p.parity ^ 1)) * Hq;
  if (tid < Hq) {
    lse_l = p.lse_sum[(long long)b * Hq + tid];
    lse_m = p.lse_max[(long long)b * Hq + tid];
    pcur = q.has_cur ? p.cur_prob[(long long)b * Hq + tid] : 0.f;
    hs = hs_old[tid];
  }
  const long long ci = (long long)b * g.slots + s;
  const long long li = ((long long)p.layer * g.num_seqs + b) * g.slots + s;
  double cum[KPT];
  float ema[KPT], mass[KPT];
  uint8_t seen[KPT];
#pragma unroll
  for (int i = 0; i < KPT; ++i) mass[i] = 0.f;
  if (active) {
    load_k<S>(p.cumulative + ci, cum);
    load_k<S>(p.layer_ema + li, ema);
    load_k<S>(p.touched + li, seen);
  }
  const float* lg = p.logits + (long long)b * Hq * g.slots + s;
  float x[HEADS][KPT];
  auto fetch = [&](int h0) {
#pragma unroll
    for (int h = 0; h < HEADS; ++h)
      if (h0 + h < Hq) load_k<S>(lg + (long long)(h0 + h) * g.slots, x[h]);
  };
  if (live > 0) fetch(0);

  // head-importance EMA (cache.py:242-248).  Every softmax row sums to one, so the
  // mean over keys of a head's probabilities is 1 / (number of keys).
  const float head_mean = total_keys > 0 ? 1.0f / (float)total_keys : 0.f;
  float hn = 0.f;
  if (tid < Hq) {
    hn = hs * p.head_decay + head_mean * (1.0f - p.head_decay);
    sh.mx[tid] = hn;  // staged, replaced below
    if (publish) hs_new[tid] = hn;
  }
  __syncthreads();
  float my_w = 0.f;
  if (tid < Hq) {
    float acc = 0.f;
#pragma unroll 8
    for (int h = 0; h < Hq; ++h) acc += sh.mx[h];  // same order in every thread: one mean per block
    my_w = hn / (acc / (float)Hq + 1e-6f);
  }
  __syncthreads();
  if (tid < Hq) {
    sh.w[tid] = lse_l > 0.f ? my_w / lse_l : 0.f;
    sh.mx[tid] = lse_m;
    sh.cprob[tid] = pcur * lse_l;
  }
  __syncthreads();
  if (!active) return;

  if (live > 0) {  // per key the sum over the heads runs in head order
    for (int h0 = 0; h0 < Hq; h0 += HEADS) {
      if (h0 > 0) fetch(h0);
#pragma unroll
      for (int h = 0; h < HEADS; ++h) {
        if (h0 + h < Hq) {
          const float wv = sh.w[h0 + h], mv = sh.mx[h0 + h];
#pragma unroll
          for (int i = 0; i < KPT; ++i) mass[i] += wv * ex2f(x[h][i] - mv);
        }
      }
    }
  }
  if (with_cur) {
    // the newest token: it is stored at this storage index when the step's append commits
    float m = 0.f;
#pragma unroll 8
    for (int h = 0; h < Hq; ++h) m += sh.w[h] * sh.cprob[h];
#pragma unroll
    for (int i = 0; i < KPT; ++i)
      if (i == cur) mass[i] = m;
  }
#pragma unroll
  for (int i = 0; i < KPT; ++i) {
    cum[i] += (double)mass[i];
    ema[i] = seen[i] ? p.decay * ema[i] + (1.0f - p.decay) * mass[i] : mass[i];
  }
  if constexpr (S::VEC && KPT == 4) {
    if (live >= 4) {
      *reinterpret_cast<double2*>(p.cumulative + ci) = make_double2(cum[0], cum[1]);
      *reinterpret_cast<double2*>(p.cumulative + ci + 2) = make_double2(cum[2], cum[3]);
      *reinterpret_cast<float4*>(p.layer_ema + li) = make_float4(ema[0], ema[1], ema[2], ema[3]);
      if (!(seen[0] && seen[1] && seen[2] && seen[3])) *reinterpret_cast<uchar4*>(p.touched + li) = make_uchar4(1, 1, 1, 1);
      return;
    }
  }
#pragma unroll
  for (int i = 0; i < KPT; ++i) {
    if (i < live || (with_cur && i == cur)) {
      p.cumulative[ci + i] = cum[i];
      p.layer_ema[li + i] = ema[i];
      if (!seen[i]) p.touched[li + i] = 1;
    }
  }
}

inline bool importance_aligned(const ImportanceParams& p) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p.logits) | reinterpret_cast<uintptr_t>(p.cumulative) |
                      reinterpret_cast<uintptr_t>(p.layer_ema);
  return a % 16 == 0 && reinterpret_cast<uintptr_t>(p.touched) % 4 == 0;
}
// Single indices with all of 32 heads in flight where their blocks fit one wave of four an SM; else four indices a thread with
// eight heads in flight (80 registers, three blocks an SM).  Steps, us: 8 x 770 keys, 32 heads, 22 layers: single 276, four
// 317; 16 x 8192, 32 heads: four 1603, two with sixteen heads 1617; 64 x 16384, 8 heads: four 1253, two 1402.  Between them (four
// layers; a form with sixteen heads in flight had been kept for these), single / four with sixteen / four with eight:
// 4 x 32768, 32 heads 210 / 214 / 214; 2 x 65536, 64 heads 243 / 251 / 252; 2 x 100000, 16 heads (two layers) 106 / 102 / 101.
using ImpOne = ImpShape<1, 32, false>;
template <bool VEC>
using ImpFour = ImpShape<4, 8, VEC>;

// ---- append ---------------------------------------------------------------------------------------------
struct AppendParams {
  StoreGeom g;
  uint8_t* store;
  int layer;
  const void* k;
  const void* v;
  int dtype;
  int rows;
  const int32_t* dst_seq;
  const int32_t* dst_bucket;
  const int32_t* dst_pos;
  int32_t* err;
};

// One warp quantises and packs one row (one of K / V of one KV head of one new token).
template <int EPL>
__device__ __forceinline__ void append_row(const AppendParams& p, long long warp, int lane) {
  const StoreGeom& g = p.g;
  const int which = (int)(warp & 1);  // 0 = K, 1 = V
  const long long rh = warp >> 1;
  int h, r;
  if (rh >> 31) {  // 64-bit division is a long subroutine: only where the row count needs it
    h = (int)(rh % g.num_kv_heads);
    r = (int)(rh / g.num_kv_heads);
  } else {
    r = (int)rh / g.num_kv_heads;
    h = (int)rh - r * g.num_kv_heads;
  }
  // the row's values do not depend on where it goes: both loads are in flight together
  RowVals<EPL> x = load_row<EPL>(which ? p.v : p.k, p.dtype, rh, lane);
  const int seq = p.dst_seq[r], bucket = p.dst_bucket[r], pos = p.dst_pos[r];
  if (seq < 0 || seq >= g.num_seqs || bucket < 0 || bucket >= kNumBuckets || pos < 0 || pos >= g.cap[bucket]) {
    if (lane == 0 && p.err) atomicExch(p.err, 2);
    return;
  }
  const int bits = bucket_bits(bucket);
  int code[EPL];
  const float scale = quantize_row<EPL>(x, bits, code);
  uint8_t* arena = arena_ptr(g, p.store, p.layer, seq);
  const long long row_index = (long long)h * g.cap[bucket] + pos;
  uint8_t* dst = arena + (which ? g.v_off[bucket] : g.k_off[bucket]) + row_index * g.row_bytes[bucket];
  pack_store_row<EPL>(code, bits, dst, lane);
  if (lane == 0) {
    float* sc = reinterpret_cast<float*>(arena + g.sc_off[bucket]);
    sc[2 * row_index + which] = scale;
    if (which) note_v_scale(g, arena, scale);
  }
}

}  // namespace skv
