// One decode layer-step of the hybrid-cache path in one call.
//
// What the reference does between the projections and o_proj of a decode layer with
// hidden-cached requests (additional_designs/model_executor/models/aptserve_opt.py:99-134
// with additional_designs/attention/backends/aptserve_flash_attn.py:331-387, 449-475):
// write the new token's layer-input row for hidden-cached requests (hidden_to_cache), write
// the new token's K/V rows for K/V-cached requests (mixed_kv_to_cache / reshape_and_cache_flash),
// then attend.  Here that is one host call that enqueues its launches on the caller's
// stream: the new-token rows, addressed straight from the private
// block tables, the sequence lengths and the cache-type mask (no int64 index tensors), with the plan
// (a launch of its own when the rows are re-projected), K/V streaming, the hidden path (five launches per 256 requests when the
// cached rows are attended directly, three in fp32, one when they are re-projected), combine.

#include "step_plan.cuh"

using namespace aps;

namespace {

// Which form of the hidden path a step takes, from what the host knows: the hidden rows are attended
// directly (hidden_attention.cu) unless the whole batch, at the longest its block tables allow, is
// one wave of tile pairs of the re-projection kernel.  One wave costs E / 64 slabs of 520 cycles: 1 us for a
// 256-wide layer, 22 us for an OPT-13B layer, 40 us at E = 9216, in one launch against five; both forms
// read W_k and W_v once (16 us for an OPT-13B layer).  At the next size up, two waves, one request of 611 tokens of an
// OPT-13B layer takes 97 us a call re-projected (65 us of it the two waves) and 67 attended directly, and every
// further wave adds to the re-projection only.
bool folded_shape(int batch, int max_blocks, int block_size, int heads, int head_size, int hidden, int dtype) {
  if (!folded_supported(dtype, heads, head_size, hidden)) return false;
  const int64_t pairs = ((int64_t)batch * max_blocks * block_size + 255) / 256;
  const int64_t items = pairs * (((int64_t)heads * head_size + 127) / 128);
  return items > sm_count() / 2 || (heads * head_size) % 128 != 0;
}

bool use_folded(const HybridCall& c) {
  const AttnShape& s = c.shape;
  return folded_takes(c) && folded_shape(s.batch, s.max_blocks_per_seq, s.block_size, s.heads, s.head_size, c.hidden_size, s.dtype) &&
         c.workspace_bytes >= folded_workspace_bytes(s.batch, s.max_blocks_per_seq, s.block_size, s.heads, s.head_size,
                                                     c.hidden_size, s.dtype);
}

}  // namespace

extern "C" int aps_decode_layer_step(void* out, const void* query, const void* hidden_states,
                                     const void* new_key, const void* new_value, void* key_cache,
                                     void* value_cache, void* hidden_cache, const void* w_k,
                                     const void* b_k, const void* w_v, const void* b_v,
                                     const int32_t* block_tables, const int32_t* seq_lens,
                                     const int32_t* cache_type, int batch, int max_blocks_per_seq,
                                     int num_heads, int head_size, int hidden_size, int block_size,
                                     int64_t query_stride, int64_t out_stride, int64_t hidden_states_stride,
                                     int64_t new_key_stride, int64_t new_value_stride, int64_t block_stride,
                                     int64_t hidden_row_stride, int64_t num_hidden_rows, int64_t w_stride,
                                     float scale, void* workspace, size_t workspace_bytes, int dtype,
                                     void* stream) {
  HybridCall c{};
  c.shape = AttnShape{batch, max_blocks_per_seq, num_heads, head_size, block_size,
                      query_stride, out_stride, block_stride, scale, dtype};
  c.out = out; c.query = query; c.key_cache = key_cache; c.value_cache = value_cache;
  c.hidden_cache = hidden_cache; c.w_k = w_k; c.b_k = b_k; c.w_v = w_v; c.b_v = b_v;
  c.block_tables = block_tables; c.seq_lens = seq_lens; c.cache_type = cache_type;
  c.hidden_size = hidden_size; c.hidden_row_stride = hidden_row_stride;
  c.num_hidden_rows = num_hidden_rows; c.w_stride = w_stride;
  c.workspace = workspace; c.workspace_bytes = workspace_bytes;
  int st = check_hybrid_call("decode_layer_step", c);
  if (st != APS_OK || batch == 0) return st;
  APS_REQUIRE(hidden_size > 0 && hidden_states_stride >= hidden_size, APS_ERR_SHAPE,
              "decode_layer_step: bad hidden_states stride");
  const int64_t row = (int64_t)num_heads * head_size;
  APS_REQUIRE(new_key == nullptr || (new_key_stride >= row && new_value_stride >= row), APS_ERR_SHAPE,
              "decode_layer_step: new_key / new_value strides smaller than a row");
  APS_REQUIRE(hidden_states == nullptr || hidden_row_stride >= hidden_size, APS_ERR_SHAPE,
              "decode_layer_step: hidden cache rows shorter than the hidden size");
  cudaStream_t cs = (cudaStream_t)stream;
  NewTokenWrite nw{hidden_states, new_key, new_value, key_cache, value_cache, hidden_cache,
                   block_tables, seq_lens, cache_type, batch, max_blocks_per_seq, block_size,
                   num_heads, head_size, hidden_size, hidden_states_stride, new_key_stride,
                   new_value_stride, block_stride, hidden_row_stride, dtype};
  if (use_folded(c)) return enqueue_folded_attention(c, nw, cs);
  if (folded32_supported(c)) return enqueue_folded32_attention(c, nw, cs);
  if ((st = launch_step_plan(nullptr, nw, cs)) != APS_OK) return st;
  return enqueue_hybrid_attention(c, cs);
}

extern "C" size_t aps_decode_layer_step_workspace_bytes(int batch, int max_blocks_per_seq, int block_size,
                                                        int num_heads, int head_size, int hidden_size, int dtype) {
  const size_t base = aps_attention_workspace_bytes(batch, max_blocks_per_seq, block_size, num_heads, head_size);
  if (base != 0 && folded32_shape(dtype, num_heads, head_size, hidden_size))
    return folded32_workspace_bytes(batch, max_blocks_per_seq, block_size, num_heads, head_size, hidden_size);
  if (base == 0 || !folded_shape(batch, max_blocks_per_seq, block_size, num_heads, head_size, hidden_size, dtype)) return base;
  return folded_workspace_bytes(batch, max_blocks_per_seq, block_size, num_heads, head_size, hidden_size, dtype);
}
