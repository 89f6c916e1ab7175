// The per-token state of a store from the side of token ids: where the tokens of a prompt lie, and what a prompt pass adds to
// their importance.  The state is kept in storage order, so both walk the live storage indices and look the token up, one
// index per thread; as index expressions over token ids the same took about 45 small launches per layer
// (8 generations of 512 + 16 tokens, 22 layers: 31.2 ms with those, 24.2 ms with these).
#include "common.cuh"

namespace skv {

constexpr int kTokenThreads = 256;

// the token at storage index s of sequence b (-1: none), and the index's bucket and position
__device__ __forceinline__ int live_token(const StoreGeom& g, const int32_t* counts, const int32_t* slot_token, int b, int s,
                                          int& bucket, int& pos) {
  bucket = 0;
#pragma unroll
  for (int i = 1; i < kNumBuckets; ++i)
    if (s >= g.bucket_base[i]) bucket = i;
  pos = s - g.bucket_base[bucket];
  return pos < counts[b * kNumBuckets + bucket] ? slot_token[(long long)b * g.slots + s] : -1;
}

// destinations of tokens first .. first + n - 1, as the append takes them; grid (ceil(slots / 256), num_seqs)
__global__ void __launch_bounds__(kTokenThreads)
    token_places_kernel(StoreGeom g, const int32_t* counts, const int32_t* slot_token, const int64_t* first, int n, int32_t* dst_seq,
                        int32_t* dst_bucket, int32_t* dst_pos, int32_t* storage) {
  const int b = blockIdx.y, s = blockIdx.x * kTokenThreads + threadIdx.x;
  if (s >= g.slots) return;
  int bucket, pos;
  const int id = live_token(g, counts, slot_token, b, s, bucket, pos);
  const long long i = (long long)id - (first ? *first : 0);
  if (id < 0 || i < 0 || i >= n) return;
  const long long at = (long long)b * n + i;
  dst_seq[at] = b;
  dst_bucket[at] = bucket;
  dst_pos[at] = pos;
  storage[at] = s;
}

template <typename Mass>
struct PromptParams {
  StoreGeom g;
  int layer;
  const int32_t* counts;
  const int32_t* slot_token;
  const Mass* mass;  // [num_seqs][n]
  int n, assign;
  float decay, fresh;
  double* cumulative;
  float* layer_ema;
  uint8_t* touched;
};
template <typename Mass>
__global__ void __launch_bounds__(kTokenThreads) prompt_importance_kernel(const PromptParams<Mass> p) {
  const int b = blockIdx.y, s = blockIdx.x * kTokenThreads + threadIdx.x;
  if (s >= p.g.slots) return;
  int bucket, pos;
  const int id = live_token(p.g, p.counts, p.slot_token, b, s, bucket, pos);
  if (id < 0 || id >= p.n) return;
  const Mass mass = p.mass[(long long)b * p.n + id];
  const float m = (float)mass;  // the layer's average is fp32 whatever the mass comes in
  const long long ci = (long long)b * p.g.slots + s;
  p.cumulative[ci] = p.assign ? (double)mass : p.cumulative[ci] + (double)mass;
  const long long li = ((long long)p.layer * p.g.num_seqs + b) * p.g.slots + s;
  if (p.touched[li]) {
    p.layer_ema[li] = __fadd_rn(__fmul_rn(p.decay, p.layer_ema[li]), __fmul_rn(p.fresh, m));
  } else {
    p.layer_ema[li] = m;
    p.touched[li] = 1;
  }
}

template <typename Mass>
static int prompt_importance(const SkvStoreDesc* desc, int layer, const int32_t* counts, const int32_t* slot_token,
                             const Mass* key_mass, int n, int assign, double decay, double* cumulative, float* layer_ema,
                             uint8_t* touched, void* stream) {
  if (!desc || !counts || !slot_token || !key_mass || n <= 0 || !cumulative || !layer_ema || !touched) return SKV_ERR_INVALID;
  if (layer < 0 || layer >= desc->num_layers) return SKV_ERR_INVALID;
  if (desc->num_seqs > 65535) return SKV_ERR_UNSUPPORTED;
  PromptParams<Mass> p = {make_geom(*desc), layer, counts, slot_token, key_mass, n, assign, (float)decay, (float)(1.0 - decay),
                          cumulative, layer_ema, touched};
  const dim3 grid((desc->slots + kTokenThreads - 1) / kTokenThreads, desc->num_seqs);
  prompt_importance_kernel<<<grid, kTokenThreads, 0, static_cast<cudaStream_t>(stream)>>>(p);
  return cudaGetLastError() == cudaSuccess ? SKV_OK : SKV_ERR_CUDA;
}

}  // namespace skv

using namespace skv;

extern "C" int skv_token_places(const SkvStoreDesc* desc, const int32_t* counts, const int32_t* slot_token,
                                const int64_t* first_token, int n, int32_t* dst_seq, int32_t* dst_bucket, int32_t* dst_pos,
                                int32_t* storage, void* stream) {
  if (!desc || !counts || !slot_token || n <= 0 || !dst_seq || !dst_bucket || !dst_pos || !storage) return SKV_ERR_INVALID;
  if (desc->num_seqs > 65535) return SKV_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // a token that is not there keeps a destination no kernel writes to
  const size_t bytes = (size_t)desc->num_seqs * n * sizeof(int32_t);
  if (cudaMemsetAsync(dst_seq, 0xff, bytes, st) != cudaSuccess || cudaMemsetAsync(storage, 0xff, bytes, st) != cudaSuccess)
    return SKV_ERR_CUDA;
  const dim3 grid((desc->slots + kTokenThreads - 1) / kTokenThreads, desc->num_seqs);
  token_places_kernel<<<grid, kTokenThreads, 0, st>>>(make_geom(*desc), counts, slot_token, first_token, n, dst_seq, dst_bucket,
                                                      dst_pos, storage);
  return cudaGetLastError() == cudaSuccess ? SKV_OK : SKV_ERR_CUDA;
}

extern "C" int skv_prompt_importance(const SkvStoreDesc* desc, int layer, const int32_t* counts, const int32_t* slot_token,
                                     const float* key_mass, int n, int assign, double decay, double* cumulative,
                                     float* layer_ema, uint8_t* touched, void* stream) {
  return prompt_importance(desc, layer, counts, slot_token, key_mass, n, assign, decay, cumulative, layer_ema, touched, stream);
}

extern "C" int skv_prompt_importance_f64(const SkvStoreDesc* desc, int layer, const int32_t* counts, const int32_t* slot_token,
                                         const double* key_mass, int n, int assign, double decay, double* cumulative,
                                         float* layer_ema, uint8_t* touched, void* stream) {
  return prompt_importance(desc, layer, counts, slot_token, key_mass, n, assign, decay, cumulative, layer_ema, touched, stream);
}
