// Device-side construction of the decode batch's index tensors.
//
// The reference builds them on the host: for every hidden-cached request a Python loop
// over all of its positions appends two slot ids (additional_designs/worker/
// aptserve_model_runner.py:527-539), the boolean masks are turned into index tensors
// (:613-648) and everything is shipped to the device (and broadcast to the
// tensor-parallel workers) every step -- about 2 x 8 bytes per cached hidden token.
// Here the host ships the two block tables, the sequence lengths and the cache types
// (a few bytes per 16 tokens) and small kernels expand them in place.  Tables that the host has padded:
//   layout_kernel   one CTA: prefix sums over the requests -> where each request starts
//                   in the expanded token space, among the hidden tokens, and its ordinal
//                   among the K/V-cached / hidden-cached requests;
//   fill_kernel     one CTA per request: writes the request's entries of all eight tensors.
// Tables as the engine has them, rows of any length one behind the other:
//   expand_lists_kernel   pads them and does what the two do, in one launch.
// Integer work only; results are bit-identical to the host construction.
//
// The caller sizes the outputs from its own view of the batch (num_tot_tokens,
// num_hidden_tokens) and may pass NULL for an output that is empty in that view.  The kernels
// trust neither: the four totals are recomputed from the device-side seq_lens and
// cache_type, and unless they equal the caller's claim no entry of the eight tensors is written
// (expand_lists_kernel pads the tables all the same).  fill_kernel bounds every store by its tensor's capacity besides;
// in expand_lists_kernel the totals are what bounds them, and where each row of the lists begins is the caller's word.

#include "aps_common.cuh"

namespace aps {
namespace {

constexpr int kScanThreads = 1024;

struct MetaLayout {       // per request, in the caller's scratch; entry [B] of each = the total
  int* exp_off;           // [B + 1] start in the expanded token space
  int* hid_off;           // [B + 1] start among the hidden tokens
  int* kv_ord;            // [B + 1] ordinal among the K/V-cached requests
  int* hid_ord;           // [B + 1] ordinal among the hidden-cached requests
};

__global__ void __launch_bounds__(kScanThreads)
layout_kernel(MetaLayout L, const int32_t* __restrict__ seq_lens, const int32_t* __restrict__ cache_type,
              int batch, int max_tokens, int64_t* __restrict__ counts) {
  __shared__ int s[4][kScanThreads];
  const int tid = threadIdx.x;
  const int per = (batch + kScanThreads - 1) / kScanThreads;
  const int r0 = min(batch, tid * per), r1 = min(batch, r0 + per);
  int v[4] = {0, 0, 0, 0};   // expanded tokens, hidden tokens, K/V requests, hidden requests
  for (int r = r0; r < r1; ++r) {
    const int len = max(1, min(seq_lens[r], max_tokens));
    if (cache_type[r] != 0) { v[0] += len; v[1] += len; v[3] += 1; }
    else { v[0] += 1; v[2] += 1; }
  }
  for (int k = 0; k < 4; ++k) s[k][tid] = v[k];
  __syncthreads();
  for (int off = 1; off < kScanThreads; off <<= 1) {
    int a[4] = {0, 0, 0, 0};
    if (tid >= off) for (int k = 0; k < 4; ++k) a[k] = s[k][tid - off];
    __syncthreads();
    for (int k = 0; k < 4; ++k) s[k][tid] += a[k];
    __syncthreads();
  }
  int o[4];
  for (int k = 0; k < 4; ++k) o[k] = s[k][tid] - v[k];
  for (int r = r0; r < r1; ++r) {
    const int len = max(1, min(seq_lens[r], max_tokens));
    L.exp_off[r] = o[0]; L.hid_off[r] = o[1]; L.kv_ord[r] = o[2]; L.hid_ord[r] = o[3];
    if (cache_type[r] != 0) { o[0] += len; o[1] += len; o[3] += 1; }
    else { o[0] += 1; o[2] += 1; }
  }
  if (tid == kScanThreads - 1) {
    L.exp_off[batch] = s[0][tid]; L.hid_off[batch] = s[1][tid];
    L.kv_ord[batch] = s[2][tid]; L.hid_ord[batch] = s[3][tid];
    if (counts != nullptr) { counts[0] = s[0][tid]; counts[1] = s[1][tid]; counts[2] = s[2][tid]; counts[3] = s[3][tid]; }
  }
}

struct MetaOut {
  int64_t* slot_mapping; int64_t* slot_mapping_shared; int64_t* hidden_cache_use_tot;
  int64_t* kv_cache_use_tot; int64_t* hidden_holder_upd; int64_t* hidden_holder_pull;
  int64_t* hidden_cache_store_tot; int64_t* hidden_cache_use_input;
  int64_t cap_tot, cap_hidden;   // capacities of the [N_tot] and [N_h] tensors (the caller's claim)
  int64_t cap_kv_req, cap_hid_req;   // capacities of the per-request lists [n_kv] and [n_h]
};

__global__ void __launch_bounds__(256)
fill_kernel(MetaLayout L, MetaOut O, const int32_t* __restrict__ block_tables,
            const int32_t* __restrict__ block_tables_shared, const int32_t* __restrict__ seq_lens,
            const int32_t* __restrict__ cache_type, int batch, int max_blocks, int block_size) {
  // the device-side totals must be what the caller sized (and NULL-ed) the outputs for
  if (L.exp_off[batch] != O.cap_tot || L.hid_off[batch] != O.cap_hidden ||
      L.kv_ord[batch] != O.cap_kv_req || L.hid_ord[batch] != O.cap_hid_req)
    return;
  for (int r = blockIdx.x; r < batch; r += gridDim.x) {
    const int len = max(1, min(seq_lens[r], max_blocks * block_size));
    const int64_t e0 = L.exp_off[r];
    const int32_t* priv = block_tables + (int64_t)r * max_blocks;
    if (cache_type[r] != 0) {
      const int64_t h0 = L.hid_off[r];
      const int32_t* shar = block_tables_shared + (int64_t)r * max_blocks;
      for (int j = threadIdx.x; j < len; j += blockDim.x) {
        const int b = j / block_size, o = j % block_size;
        if (e0 + j < O.cap_tot) O.slot_mapping[e0 + j] = (int64_t)priv[b] * block_size + o;
        if (h0 + j < O.cap_hidden) {
          O.slot_mapping_shared[h0 + j] = (int64_t)shar[b] * block_size + o;
          O.hidden_cache_use_tot[h0 + j] = e0 + j;
        }
        // every earlier request holds exactly one "current token" entry, and so far none of this one
        if (j < len - 1 && e0 + j - r >= 0 && e0 + j - r < O.cap_tot - batch) O.hidden_holder_pull[e0 + j - r] = e0 + j;
      }
      if (threadIdx.x == 0) {
        O.hidden_holder_upd[r] = e0 + len - 1;
        const int ord = L.hid_ord[r];
        if (ord < O.cap_hid_req) {
          O.hidden_cache_store_tot[ord] = e0 + len - 1;
          O.hidden_cache_use_input[ord] = r;
        }
      }
    } else if (threadIdx.x == 0) {
      const int j = len - 1;
      if (e0 < O.cap_tot) O.slot_mapping[e0] = (int64_t)priv[j / block_size] * block_size + j % block_size;
      if (L.kv_ord[r] < O.cap_kv_req) O.kv_cache_use_tot[L.kv_ord[r]] = e0;
      O.hidden_holder_upd[r] = e0;
    }
  }
}

// The same from tables that nobody has padded, in one launch: a CTA sums up the requests before its own by itself (256 requests:
// 1 - 2 KB a CTA) instead of reading what a layout kernel has left (256 OPT-13B requests, the whole call: 157 us with the two
// launches and sections padded to 128 bytes, 129 so; 163 with tables padded on the host), and pads the request's tables besides: the
// private one, the shared one (zero for K/V-cached requests) and the one that the type selects.
struct MetaLists { const int32_t* own; const int32_t* own_at; const int32_t* shared; const int32_t* shared_at; int32_t* tables; };

__global__ void __launch_bounds__(256)
expand_lists_kernel(const MetaLists T, MetaOut O, const int32_t* __restrict__ seq_lens, const int32_t* __restrict__ cache_type, int batch,
                    int max_blocks, int block_size) {
  __shared__ int s_sum[8][4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t plane = (int64_t)batch * max_blocks;
  // This CTA's requests, one behind the other: what comes before the first is summed up once.  Summed up for each, 20 000 requests
  // took 945 us and 50 000 3 166, more than with tables padded on the host (807, 1 630); so 763 and 1 544.
  const int each = (batch + gridDim.x - 1) / gridDim.x, first = blockIdx.x * each, last = min(batch, first + each);
  if (first >= last) return;
  // hidden requests and their tokens before the first, and in all
  int v[4] = {0, 0, 0, 0};
  for (int i = threadIdx.x; i < batch; i += 256) {
    const int len = cache_type[i] != 0 ? max(1, min(seq_lens[i], max_blocks * block_size)) : 0;
    if (i < first) { v[0] += len > 0; v[1] += len; }
    v[2] += len > 0; v[3] += len;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if (lane == 0) s_sum[warp][k] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = 0;
    for (int w = 0; w < 8; ++w) v[k] += s_sum[w][k];
  }
  // the device-side totals must be what the caller sized (and NULL-ed) the outputs for
  const bool agree = v[3] + (int64_t)(batch - v[2]) == O.cap_tot && v[3] == O.cap_hidden && batch - v[2] == O.cap_kv_req && v[2] == O.cap_hid_req;
  int hid_ord = v[0];
  int64_t h0 = v[1];
  for (int r = first; r < last; ++r) {
    const bool hid = cache_type[r] != 0;
    const int32_t *priv = T.own + T.own_at[r], *shar = T.shared + T.shared_at[r];
    const int n_priv = min(T.own_at[r + 1] - T.own_at[r], max_blocks), n_shar = min(T.shared_at[r + 1] - T.shared_at[r], max_blocks);
    int32_t* tables = T.tables + (int64_t)r * max_blocks;
    for (int b = threadIdx.x; b < max_blocks; b += 256) {
      const int32_t p = b < n_priv ? priv[b] : 0, s = hid && b < n_shar ? shar[b] : 0;
      tables[b] = p; tables[plane + b] = s; tables[2 * plane + b] = hid ? s : p;
    }
    if (!agree) continue;
    const int len = max(1, min(seq_lens[r], max_blocks * block_size)), kv_ord = r - hid_ord;
    const int64_t e0 = h0 + kv_ord;
    if (hid) {
      for (int j = threadIdx.x; j < len; j += 256) {
        const int b = j / block_size, o = j % block_size;
        O.slot_mapping[e0 + j] = (int64_t)(b < n_priv ? priv[b] : 0) * block_size + o;
        O.slot_mapping_shared[h0 + j] = (int64_t)(b < n_shar ? shar[b] : 0) * block_size + o;
        O.hidden_cache_use_tot[h0 + j] = e0 + j;
        // every earlier request holds exactly one "current token" entry, and so far none of this one
        if (j < len - 1) O.hidden_holder_pull[e0 + j - r] = e0 + j;
      }
      if (threadIdx.x == 0) {
        O.hidden_holder_upd[r] = e0 + len - 1;
        O.hidden_cache_store_tot[hid_ord] = e0 + len - 1;
        O.hidden_cache_use_input[hid_ord] = r;
      }
      ++hid_ord;
      h0 += len;
    } else if (threadIdx.x == 0) {
      const int j = len - 1, b = j / block_size;
      O.slot_mapping[e0] = (int64_t)(b < n_priv ? priv[b] : 0) * block_size + j % block_size;
      O.kv_cache_use_tot[kv_ord] = e0;
      O.hidden_holder_upd[r] = e0;
    }
  }
}

// Private block tables and the cache-type mask from the reference's decode metadata (what the fused
// layer-step needs and the reference does not ship): request r is hidden-cached if hidden_rows lists
// it; its private blocks are then read off its run of slot_mapping, which ends at holder_upd[r], one
// slot per block; a K/V-cached request keeps its row of block_tables.
// One CTA per request, one launch: the same thing as tensor operations is 24 launches of 2 us with 12 us of
// host work between them: an attention layer of 24 OPT-13B requests takes 319 us a call with this kernel, 570 with
// those.  What is left is
// one dependent chain of loads (hidden_rows, holder_upd, slot_mapping), about 4 us.  Every CTA scans
// hidden_rows itself: at most 8 bytes per request and CTA, from L2.
// An index outside its tensor is never followed, and no block is made up for it: a request whose run of slot_mapping leaves
// the tensor or holds a negative slot gets kCacheTypeNone and a table of -1 (no cache write, no attention, a zero
// output row), every request does if hidden_rows names one that does not exist (the request it was meant for would
// pass for a K/V-cached one), and g_metadata_status is set.
__device__ int g_metadata_status = 0;
constexpr int kDeriveThreads = 128;

__global__ void __launch_bounds__(kDeriveThreads)
derive_tables_kernel(int32_t* __restrict__ tables, int32_t* __restrict__ cache_type,
                     const int32_t* __restrict__ block_tables, const int64_t* __restrict__ slot_mapping,
                     int64_t num_slots, const int64_t* __restrict__ holder_upd,
                     const int64_t* __restrict__ hidden_rows, int64_t num_hidden, const int32_t* __restrict__ seq_lens,
                     int batch, int max_blocks, int64_t table_stride, int block_size) {
  const int r = blockIdx.x;
  bool mine = false, lost = false;
  for (int64_t i = threadIdx.x; i < num_hidden; i += kDeriveThreads) {
    int64_t row = hidden_rows[i];
    if (row < 0) row += batch;   // an index counts from the end when it is negative, as in the tensor form
    lost |= row < 0 || row >= batch;
    mine |= row == r;
  }
  const bool hidden = __syncthreads_or(mine) != 0;
  bool bad = lost;
  const int64_t len = seq_lens[r], start = hidden ? holder_upd[r] - (len - 1) : 0;
  for (int j = threadIdx.x; j < max_blocks; j += kDeriveThreads) {
    int32_t id = 0;
    if (!hidden) {
      id = block_tables[r * table_stride + j];
    } else if ((int64_t)j * block_size < len) {
      int64_t pos = start + (int64_t)j * block_size;
      if (pos < 0) pos += num_slots;
      const int64_t slot = pos >= 0 && pos < num_slots ? slot_mapping[pos] : -1;
      bad |= slot < 0;
      id = (int32_t)(slot / block_size);
    }
    tables[(int64_t)r * max_blocks + j] = id;
  }
  bad = __syncthreads_or(bad) != 0;
  if (bad)
    for (int j = threadIdx.x; j < max_blocks; j += kDeriveThreads) tables[(int64_t)r * max_blocks + j] = -1;
  if (threadIdx.x == 0) {
    cache_type[r] = bad ? kCacheTypeNone : hidden ? 1 : 0;
    if (bad) g_metadata_status = kStatusBadIndex;
  }
}

}  // namespace

int read_metadata_status(int* host_status, cudaStream_t stream) {
  void* addr = nullptr;
  APS_CUDA(cudaGetSymbolAddress(&addr, g_metadata_status));
  APS_CUDA(cudaMemcpyAsync(host_status, addr, sizeof(int), cudaMemcpyDeviceToHost, stream));
  APS_CUDA(cudaStreamSynchronize(stream));
  if (*host_status != 0) APS_CUDA(cudaMemsetAsync(addr, 0, sizeof(int), stream));   // reported once
  return APS_OK;
}

}  // namespace aps

using namespace aps;

extern "C" int aps_derive_private_tables(int32_t* tables, int32_t* cache_type, const int32_t* block_tables,
                                         const int64_t* slot_mapping, int64_t num_slots,
                                         const int64_t* hidden_holder_upd, const int64_t* hidden_cache_use_input,
                                         int64_t num_hidden, const int32_t* seq_lens, int batch,
                                         int max_blocks_per_seq, int64_t block_tables_stride, int block_size,
                                         void* stream) {
  APS_REQUIRE(batch >= 0 && max_blocks_per_seq >= 0 && num_slots >= 0 && num_hidden >= 0 && block_size > 0 &&
                  block_tables_stride >= max_blocks_per_seq,
              APS_ERR_SHAPE, "derive_private_tables: bad sizes");
  if (batch == 0) return APS_OK;
  APS_REQUIRE(cache_type && seq_lens && hidden_holder_upd && (num_slots == 0 || slot_mapping) &&
                  (num_hidden == 0 || hidden_cache_use_input) && (max_blocks_per_seq == 0 || (tables && block_tables)),
              APS_ERR_NULL_POINTER, "derive_private_tables: null pointer");
  derive_tables_kernel<<<batch, kDeriveThreads, 0, (cudaStream_t)stream>>>(
      tables, cache_type, block_tables, slot_mapping, num_slots, hidden_holder_upd, hidden_cache_use_input, num_hidden,
      seq_lens, batch, max_blocks_per_seq, block_tables_stride, block_size);
  return launch_status("derive_tables_kernel");
}

extern "C" size_t aps_decode_metadata_scratch_bytes(int batch) {
  return batch <= 0 ? 0 : (size_t)(4 * (batch + 1)) * sizeof(int);
}

extern "C" int aps_expand_decode_metadata(const int32_t* block_tables, const int32_t* block_tables_shared,
                                          const int32_t* seq_lens, const int32_t* cache_type, int batch,
                                          int max_blocks_per_seq, int block_size, int64_t* slot_mapping,
                                          int64_t* slot_mapping_shared, int64_t* hidden_cache_use_tot,
                                          int64_t* kv_cache_use_tot, int64_t* hidden_holder_upd,
                                          int64_t* hidden_holder_pull, int64_t* hidden_cache_store_tot,
                                          int64_t* hidden_cache_use_input, int64_t num_tot_tokens,
                                          int64_t num_hidden_tokens, int64_t* counts, void* scratch,
                                          size_t scratch_bytes, void* stream) {
  APS_REQUIRE(batch >= 0 && max_blocks_per_seq > 0 && block_size > 0 && num_tot_tokens >= batch &&
                  num_hidden_tokens >= 0 && num_hidden_tokens <= num_tot_tokens &&
                  num_tot_tokens - num_hidden_tokens <= batch,
              APS_ERR_SHAPE, "expand_decode_metadata: bad sizes (N_tot = %lld, N_h = %lld, batch = %d)",
              (long long)num_tot_tokens, (long long)num_hidden_tokens, batch);
  if (batch == 0) return APS_OK;
  // outputs whose length is zero for this batch may be NULL (an empty tensor has no storage)
  APS_REQUIRE(block_tables && seq_lens && cache_type && slot_mapping && hidden_holder_upd,
              APS_ERR_NULL_POINTER, "expand_decode_metadata: null pointer");
  // every hidden request holds at least one token, so N_h == 0 means there is none
  APS_REQUIRE(num_hidden_tokens == 0 || (block_tables_shared && slot_mapping_shared &&
                                         hidden_cache_use_tot && hidden_cache_store_tot &&
                                         hidden_cache_use_input),
              APS_ERR_NULL_POINTER, "expand_decode_metadata: null pointer (hidden-request outputs)");
  APS_REQUIRE(num_tot_tokens == num_hidden_tokens || kv_cache_use_tot != nullptr, APS_ERR_NULL_POINTER,
              "expand_decode_metadata: null pointer (kv_cache_use_tot)");
  APS_REQUIRE(num_tot_tokens == batch || hidden_holder_pull != nullptr, APS_ERR_NULL_POINTER,
              "expand_decode_metadata: null pointer (hidden_holder_pull)");
  APS_REQUIRE(scratch != nullptr && aligned_to(scratch, 4) &&
                  scratch_bytes >= aps_decode_metadata_scratch_bytes(batch),
              APS_ERR_WORKSPACE, "expand_decode_metadata: scratch must hold %zu bytes",
              aps_decode_metadata_scratch_bytes(batch));
  int* sc = static_cast<int*>(scratch);
  MetaLayout L{sc, sc + (batch + 1), sc + 2 * (batch + 1), sc + 3 * (batch + 1)};
  MetaOut O{slot_mapping, slot_mapping_shared, hidden_cache_use_tot, kv_cache_use_tot,
            hidden_holder_upd, hidden_holder_pull, hidden_cache_store_tot, hidden_cache_use_input,
            num_tot_tokens, num_hidden_tokens, num_tot_tokens - num_hidden_tokens,
            batch - (num_tot_tokens - num_hidden_tokens)};
  cudaStream_t cs = (cudaStream_t)stream;
  layout_kernel<<<1, kScanThreads, 0, cs>>>(L, seq_lens, cache_type, batch,
                                            max_blocks_per_seq * block_size, counts);
  int st = launch_status("layout_kernel");
  if (st != APS_OK) return st;
  const int grid = batch < sm_count() * 8 ? batch : sm_count() * 8;
  fill_kernel<<<grid, 256, 0, cs>>>(L, O, block_tables, block_tables_shared, seq_lens, cache_type,
                                    batch, max_blocks_per_seq, block_size);
  return launch_status("fill_kernel");
}

// One launch; nothing is padded on the host and the tables that the other calls take are left on the device.
extern "C" int aps_expand_decode_lists(const int32_t* entries, const int32_t* starts, const int32_t* shared_entries,
                                       const int32_t* shared_starts, const int32_t* seq_lens, const int32_t* cache_type, int batch,
                                       int max_blocks_per_seq, int block_size, int32_t* tables, int64_t* slot_mapping,
                                       int64_t* slot_mapping_shared, int64_t* hidden_cache_use_tot, int64_t* kv_cache_use_tot,
                                       int64_t* hidden_holder_upd, int64_t* hidden_holder_pull, int64_t* hidden_cache_store_tot,
                                       int64_t* hidden_cache_use_input, int64_t num_tot_tokens, int64_t num_hidden_tokens,
                                       void* stream) {
  APS_REQUIRE(batch >= 0 && max_blocks_per_seq > 0 && block_size > 0 && num_tot_tokens >= batch && num_hidden_tokens >= 0 &&
                  num_hidden_tokens <= num_tot_tokens && num_tot_tokens - num_hidden_tokens <= batch,
              APS_ERR_SHAPE, "expand_decode_lists: bad sizes (N_tot = %lld, N_h = %lld, batch = %d)", (long long)num_tot_tokens,
              (long long)num_hidden_tokens, batch);
  if (batch == 0) return APS_OK;
  APS_REQUIRE(entries && starts && shared_entries && shared_starts && seq_lens && cache_type && tables && slot_mapping && hidden_holder_upd &&
                  (num_hidden_tokens == 0 ||
                   (slot_mapping_shared && hidden_cache_use_tot && hidden_cache_store_tot && hidden_cache_use_input)) &&
                  (num_tot_tokens == num_hidden_tokens || kv_cache_use_tot) && (num_tot_tokens == batch || hidden_holder_pull),
              APS_ERR_NULL_POINTER, "expand_decode_lists: null pointer");
  const MetaOut O{slot_mapping, slot_mapping_shared, hidden_cache_use_tot, kv_cache_use_tot,
                  hidden_holder_upd, hidden_holder_pull, hidden_cache_store_tot, hidden_cache_use_input,
                  num_tot_tokens, num_hidden_tokens, num_tot_tokens - num_hidden_tokens,
                  batch - (num_tot_tokens - num_hidden_tokens)};
  const int grid = batch < sm_count() * 8 ? batch : sm_count() * 8;
  const MetaLists T{entries, starts, shared_entries, shared_starts, tables};
  expand_lists_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(T, O, seq_lens, cache_type, batch, max_blocks_per_seq, block_size);
  return launch_status("expand_lists_kernel");
}
