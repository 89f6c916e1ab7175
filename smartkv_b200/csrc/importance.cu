// Fused importance update for the decode path.
//
// Replaces, for one (layer, decode step), the reference's
//   SmartKVCache.update_attention head weighting   (smartkv/core/cache.py:232-253)
//   ImportanceTracker.update_attention             (smartkv/core/importance.py:44-101)
// which copy the whole probability tensor to the host and loop over tokens in
// Python.  Here the probabilities are never materialised: the attention kernel
// left scaled logits per (query head, key) in storage order, the combine left the
// final max and sum per query head, and this kernel rebuilds
//   p = exp2(logit - max) / sum
// sums it over the query heads with the head weights and folds the per-key mass
// into the cumulative importance (fp64, what the allocator reads) and the
// per-layer EMA (decay 0.9 by default), both kept in storage order.
#include "post_attention.cuh"

namespace skv {

// grid = (ceil(slots / IMP::CHUNK), num_seqs)
template <class IMP>
__global__ void __launch_bounds__(kPostThreads) importance_update_kernel(const ImportanceParams p) {
  __shared__ ImportanceShared sh;
  importance_block<IMP>(p, blockIdx.x, blockIdx.y, blockIdx.x == 0, sh);
}

template <class IMP>
static void launch_importance(const ImportanceParams& p, cudaStream_t st) {
  const dim3 grid((p.g.slots + IMP::CHUNK - 1) / IMP::CHUNK, p.g.num_seqs);
  importance_update_kernel<IMP><<<grid, kPostThreads, 0, st>>>(p);
}

}  // namespace skv

using namespace skv;

extern "C" int skv_importance_update(const SkvStoreDesc* desc, int layer, const int32_t* counts, int num_q_heads,
                                     const float* logits, const float* lse_max, const float* lse_sum,
                                     const float* cur_prob, const int32_t* cur_slot, float* head_state, int parity,
                                     double* cumulative, float* layer_ema, uint8_t* touched, float decay,
                                     float head_decay, void* stream) {
  if (!desc || !counts || !logits || !lse_max || !lse_sum || !head_state || !cumulative || !layer_ema || !touched)
    return SKV_ERR_INVALID;
  if (layer < 0 || layer >= desc->num_layers || num_q_heads <= 0 || num_q_heads > kMaxQHeads) return SKV_ERR_INVALID;
  if (parity != 0 && parity != 1) return SKV_ERR_INVALID;
  ImportanceParams p = {};
  p.g = make_geom(*desc);
  p.layer = layer;
  p.counts = counts;
  p.num_q_heads = num_q_heads;
  p.logits = logits;
  p.lse_max = lse_max;
  p.lse_sum = lse_sum;
  p.cur_prob = cur_prob;
  p.cur_slot = cur_slot;
  p.head_state = head_state;
  p.parity = parity;
  p.cumulative = cumulative;
  p.layer_ema = layer_ema;
  p.touched = touched;
  p.decay = decay;
  p.head_decay = head_decay;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // as the launch after the attention chooses (post_attention.cuh), on a B200's 148 SMs; how many chunks are live and how many
  // SMs the attention has is not known here
  if ((long long)desc->slots * desc->num_seqs <= 4LL * 148 * ImpOne::CHUNK) launch_importance<ImpOne>(p, st);
  else if (importance_aligned(p)) launch_importance<ImpFour<true>>(p, st);
  else launch_importance<ImpFour<false>>(p, st);
  return cudaGetLastError() == cudaSuccess ? SKV_OK : SKV_ERR_CUDA;
}
