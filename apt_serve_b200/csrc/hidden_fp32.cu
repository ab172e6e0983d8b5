// Hidden-path decode attention in fp32 with the K / V projections moved to the query and to the output: the
// CUDA-core counterpart of hidden_attention.cu (same algebra, same place in the reference: paths under
// additional_designs/, model_executor/models/aptserve_opt.py:111-124 and
// attention/backends/aptserve_flash_attn.py:356-387, :462-473), all of it in fp32.
//
//   fold32_kernel     qt[r][h] = scale log2(e) W_k,h^T q[r][h]
//   attend32_kernel   per chunk of a request's tokens: s = x_t . qt, p = 2^(s - max), z = sum p x_t
//   unfold32_kernel   y[r][h] = W_v,h z[r][h], the chunks merged on the way in
// and the combine kernel adds the ranges of E and b_v.
//
// What bounds it: a batch of eight is a chain of small launches, each one or two rounds of loads deep; a large batch
// reads the cached rows once from memory and twice more per four heads from L1 / L2, which is what it then runs at.
// The re-projecting kernel (hidden_simt.cu) does D times the arithmetic for a long request.  A step of an OPT-125M
// layer in fp32, half of the requests hidden-cached, on one B200, that kernel -> this path: 8 requests of about 230 tokens
// 340 -> 38 us (the host side of six launches; the device needs 32), 64 of 700 2.74 -> 0.16 ms, 200 of 1200, three quarters of
// them hidden-cached, 20.2 -> 0.74 ms.  Its distance from 64 bits is a quarter of the re-projection's.
//
// Requests are taken in groups, so that the scratch (z: one row of E per request, chunk and head) stays bounded.

#include "step_plan.cuh"

#include <cfloat>

namespace aps {
namespace {

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kFoldReqs = 8;                    // requests per CTA of the fold
constexpr int kHeads = 4;                       // heads per CTA of the attention
constexpr int kMinChunk = 32, kMaxChunk = 256;  // tokens per CTA of the attention
constexpr size_t kScratch = size_t(256) << 20;  // aimed at for the partial weighted sums

struct Params {
  const GroupPlan* plan;   // every group of the step's plan
  const float* query; const float* x; const float* w_k; const float* w_v; const int32_t* block_tables;
  float* qt;               // [request of the group][head][E]
  float* ml;               // [request][chunk][head][2]
  float* z;                // [request][chunk][head][E], not normalised
  float* out_part;         // [range of E][hidden request][H * D]
  int first, count;        // the group: ordinals of hidden requests
  int heads, hidden, block_size, max_blocks, chunk, chunks, n_hidden_cap;
  int64_t query_stride, x_stride, w_stride;
  float scale_log2;
};

// Request and length of hidden request `i` of the launch's group; length 0 past the last one.
__device__ __forceinline__ int2 request_of(const Params& p, int i) {
  const int o = p.first + i;
  const GroupPlan* g = p.plan + o / kGroup;
  const int s = o % kGroup;
  return i < p.count && s < g->n ? make_int2(g->req[s], g->len[s]) : make_int2(-1, 0);
}
__device__ __forceinline__ float4 fma4(float a, const float4& x, const float4& c) {
  return make_float4(fmaf(a, x.x, c.x), fmaf(a, x.y, c.y), fmaf(a, x.z, c.z), fmaf(a, x.w, c.w));
}
__device__ __forceinline__ float dot4(const float4& a, const float4& b, float c) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, c))));
}
// Sums N values over the 32 lanes, N a power of two up to 32: lane l returns the sum of value l * N / 32.
template <int N>
__device__ __forceinline__ float transpose_sum(float (&v)[N], int lane) {
  int o = 16;
#pragma unroll
  for (int n = N / 2; n >= 1; n >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float keep = up ? v[i + n] : v[i], send = up ? v[i] : v[i + n];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  float s = v[0];
#pragma unroll
  for (; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// One CTA per (128 columns of E, head, kFoldReqs requests); warp w takes rows w, w + 8, ... of W_k,h (its loads are
// independent: one round trip), the warps' sums are added through shared memory.  It
// takes its requests from the plan, which is complete when the K/V kernel lets it start; behind that one it does not wait
// for it before it begins but before it exits (wait_last).
template <int D>
__global__ void __launch_bounds__(kThreads)
fold32_kernel(const Params p, const int wait_last) {
  __shared__ __align__(16) float s_q[kFoldReqs][D];
  __shared__ __align__(16) float s_red[kWarps][kFoldReqs][128];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, head = blockIdx.y, r0 = blockIdx.z * kFoldReqs;
  if (!wait_last) chain_wait();
  chain_next();
  if (request_of(p, r0).x < 0) { chain_wait(); return; }
  const int e = blockIdx.x * 128 + lane * 4;
  const bool in = e < p.hidden;
  float4 w[D / kWarps];
#pragma unroll
  for (int k = 0; k < D / kWarps; ++k)
    w[k] = in ? *reinterpret_cast<const float4*>(p.w_k + (int64_t)(head * D + warp + k * kWarps) * p.w_stride + e) : make_float4(0.f, 0.f, 0.f, 0.f);
  for (int i = threadIdx.x; i < kFoldReqs * D; i += kThreads) {
    const int2 rq = request_of(p, r0 + i / D);
    s_q[i / D][i % D] = rq.x >= 0 ? p.query[rq.x * p.query_stride + head * D + i % D] * p.scale_log2 : 0.f;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kFoldReqs; ++r) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < D / kWarps; ++k) a = fma4(s_q[r][warp + k * kWarps], w[k], a);
    *reinterpret_cast<float4*>(&s_red[warp][r][lane * 4]) = a;
  }
  __syncthreads();
  const int r = warp;   // one request per warp: kFoldReqs == kWarps
  static_assert(kFoldReqs == kWarps, "one request per warp in the reduction");
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int k = 0; k < kWarps; ++k) sum = fma4(1.f, *reinterpret_cast<const float4*>(&s_red[k][r][lane * 4]), sum);
  if (in && request_of(p, r0 + r).x >= 0)
    *reinterpret_cast<float4*>(p.qt + ((int64_t)(r0 + r) * p.heads + head) * p.hidden + e) = sum;
  chain_wait();
}

// One CTA per (chunk of tokens, request, kHeads heads).  Scores: a warp takes four tokens at a time, its lanes the
// columns; eight 16-byte loads feed 64 fmas.  Weighted sums: a thread takes four columns and walks the tokens, the
// weights of the four heads being one broadcast load.  The rows come from memory once and from L1 the second
// time (a chunk of 64 rows of 768 columns is 192 KB).
__global__ void __launch_bounds__(kThreads)
attend32_kernel(const Params p) {
  __shared__ __align__(16) float s_p[kMaxChunk][kHeads];
  __shared__ int64_t s_row[kMaxChunk];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  chain_wait();
  chain_next();
  const int i = blockIdx.y, c = blockIdx.x, h0 = blockIdx.z * kHeads;
  const int2 rq = request_of(p, i);
  const int tok0 = c * p.chunk, n = min(p.chunk, rq.y - tok0);
  if (n <= 0) return;
  const int32_t* bt = p.block_tables + (int64_t)rq.x * p.max_blocks;
  for (int t = threadIdx.x; t < n; t += kThreads) {
    const int tok = tok0 + t;
    s_row[t] = ((int64_t)bt[tok / p.block_size] * p.block_size + tok % p.block_size) * p.x_stride;
  }
  __syncthreads();
  const float* qt[kHeads];
#pragma unroll
  for (int h = 0; h < kHeads; ++h) qt[h] = p.qt + ((int64_t)i * p.heads + min(h0 + h, p.heads - 1)) * p.hidden;
  for (int t0 = warp * 4; t0 < n; t0 += kWarps * 4) {
    const float* x[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) x[t] = p.x + s_row[min(t0 + t, n - 1)];
    float acc[4 * kHeads];
#pragma unroll
    for (int k = 0; k < 4 * kHeads; ++k) acc[k] = 0.f;
#pragma unroll 2
    for (int e = lane * 4; e < p.hidden; e += 128) {
      float4 xv[4], qv[kHeads];
#pragma unroll
      for (int t = 0; t < 4; ++t) xv[t] = *reinterpret_cast<const float4*>(x[t] + e);
#pragma unroll
      for (int h = 0; h < kHeads; ++h) qv[h] = *reinterpret_cast<const float4*>(qt[h] + e);
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int h = 0; h < kHeads; ++h) acc[t * kHeads + h] = dot4(xv[t], qv[h], acc[t * kHeads + h]);
    }
    const float s = transpose_sum<4 * kHeads>(acc, lane);
    const int t = t0 + (lane >> 3);
    if ((lane & 1) == 0 && t < n) s_p[t][(lane >> 1) & 3] = s;
  }
  __syncthreads();
  if (warp < kHeads) {
    // not -infinity: where all scores are, the chunk has no weights and no NaN, the other chunks have them
    float m = -FLT_MAX, l = 0.f;
    for (int t = lane; t < n; t += 32) m = fmaxf(m, s_p[t][warp]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    for (int t = lane; t < n; t += 32) {
      const float w = exp2f(s_p[t][warp] - m);
      s_p[t][warp] = w;
      l += w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (lane == 0 && h0 + warp < p.heads)
      *reinterpret_cast<float2*>(p.ml + (((int64_t)i * p.chunks + c) * p.heads + h0 + warp) * 2) = make_float2(m, l);
  }
  __syncthreads();
  for (int e = threadIdx.x * 4; e < p.hidden; e += kThreads * 4) {
    float4 a[kHeads];
#pragma unroll
    for (int h = 0; h < kHeads; ++h) a[h] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int t = 0; t < n; ++t) {
      const float4 xv = *reinterpret_cast<const float4*>(p.x + s_row[t] + e);
      const float4 w = *reinterpret_cast<const float4*>(&s_p[t][0]);
      a[0] = fma4(w.x, xv, a[0]); a[1] = fma4(w.y, xv, a[1]); a[2] = fma4(w.z, xv, a[2]); a[3] = fma4(w.w, xv, a[3]);
    }
#pragma unroll
    for (int h = 0; h < kHeads; ++h)
      if (h0 + h < p.heads) *reinterpret_cast<float4*>(p.z + (((int64_t)i * p.chunks + c) * p.heads + h0 + h) * p.hidden + e) = a[h];
  }
}

// One CTA per (head, range of E, R requests).  128 columns at a time: the chunks' weighted sums are merged into shared
// memory (their weights come first, once per CTA), then warp w multiplies rows w, w + 8, ... of W_v,h with all
// R requests.
template <int D>
__global__ void __launch_bounds__(kThreads)
unfold32_kernel(const Params p) {
  constexpr int R = D == 128 ? 4 : 8, kRows = D / kWarps, kStep = 256;
  constexpr int kWeights = 512;                   // chunk weights kept; those of longer requests are formed again
  __shared__ __align__(16) float s_z[R][kStep];
  __shared__ float s_w[R][kWeights / R], s_max[R], s_inv[R];
  __shared__ int s_chunks[R];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, head = blockIdx.x, r0 = blockIdx.z * R;
  chain_wait();
  chain_next();
  if (request_of(p, r0).x < 0) return;
  for (int r = warp; r < R; r += kWarps) {
    const int n = (request_of(p, r0 + r).y + p.chunk - 1) / p.chunk;
    const float* ml = p.ml + ((int64_t)(r0 + r) * p.chunks * p.heads + head) * 2;
    float m = -INFINITY, l = 0.f;
    for (int c = lane; c < n; c += 32) m = fmaxf(m, ml[(int64_t)c * p.heads * 2]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    for (int c = lane; c < n; c += 32) {
      const float w = exp2f(ml[(int64_t)c * p.heads * 2] - m);
      if (c < kWeights / R) s_w[r][c] = w;
      l = fmaf(w, ml[(int64_t)c * p.heads * 2 + 1], l);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    // no weight in any chunk (all scores -infinity): NaN, as 0 / 0 is
    if (lane == 0) { s_max[r] = m; s_inv[r] = n == 0 ? 0.f : l > 0.f || l != l ? 1.f / l : __int_as_float(0x7fc00000); s_chunks[r] = n; }
  }
  const int steps = (p.hidden + kStep - 1) / kStep;
  const int sa = steps * blockIdx.y / gridDim.y, sb = steps * (blockIdx.y + 1) / gridDim.y;
  float acc[kRows * R];
#pragma unroll
  for (int k = 0; k < kRows * R; ++k) acc[k] = 0.f;
  for (int s = sa; s < sb; ++s) {
    const int e0 = s * kStep;
    __syncthreads();   // the weights are there; the last step's sums have been read
    for (int k = threadIdx.x; k < R * (kStep / 4); k += kThreads) {
      const int r = k / (kStep / 4), e = e0 + k % (kStep / 4) * 4, n = s_chunks[r];
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
      if (e < p.hidden) {
        const float* src = p.z + ((int64_t)(r0 + r) * p.chunks * p.heads + head) * p.hidden + e;
        const float* ml = p.ml + ((int64_t)(r0 + r) * p.chunks * p.heads + head) * 2;
#pragma unroll 4
        for (int c = 0; c < n; ++c) {
          const float w = c < kWeights / R ? s_w[r][c] : exp2f(ml[(int64_t)c * p.heads * 2] - s_max[r]);
          a = fma4(w, *reinterpret_cast<const float4*>(src + (int64_t)c * p.heads * p.hidden), a);
        }
      }
      const float inv = s_inv[r];
      *reinterpret_cast<float4*>(&s_z[r][e - e0]) = make_float4(a.x * inv, a.y * inv, a.z * inv, a.w * inv);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kStep; j += 128) {
      const int e = e0 + j + lane * 4;
      if (e >= p.hidden) break;
      float4 z[R];
#pragma unroll
      for (int r = 0; r < R; ++r) z[r] = *reinterpret_cast<const float4*>(&s_z[r][j + lane * 4]);
#pragma unroll
      for (int k = 0; k < kRows; ++k) {
        const float4 w = *reinterpret_cast<const float4*>(p.w_v + (int64_t)(head * D + warp + k * kWarps) * p.w_stride + e);
#pragma unroll
        for (int r = 0; r < R; ++r) acc[k * R + r] = dot4(w, z[r], acc[k * R + r]);
      }
    }
  }
  const int width = p.heads * D;
  float* out = p.out_part + ((int64_t)blockIdx.y * p.n_hidden_cap + p.first + r0) * width + head * D;
#pragma unroll
  for (int k = 0; k < kRows * R; k += 32) {
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = acc[k + j];
    const float y = transpose_sum<32>(v, lane);
    const int row = (k + lane) / R, r = (k + lane) % R;
    if (request_of(p, r0 + r).x >= 0) out[(int64_t)r * width + warp + row * kWarps] = y;
  }
}

struct Layout {
  int n_groups, n_hidden_cap, count, chunk, chunks, splits;
  size_t off_groups, off_slot, off_list, off_qt, off_ml, off_z, off_part, total;
};

// Tokens per chunk: the fewest (most CTAs) for which all of a plan group's partial sums fit the scratch aimed at; with
// the most tokens per chunk the group itself gets smaller.
Layout layout_of(int batch, int max_blocks, int block_size, int heads, int head_size, int hidden) {
  Layout l;
  const int64_t max_tokens = (int64_t)max_blocks * block_size;
  const size_t row = (size_t)heads * hidden * sizeof(float);
  l.n_groups = (batch + kGroup - 1) / kGroup;
  l.n_hidden_cap = l.n_groups == 1 ? batch : l.n_groups * kGroup;
  l.count = batch < kGroup ? batch : kGroup;
  l.chunk = kMinChunk;
  auto per_request = [&] { return (size_t)((max_tokens + l.chunk - 1) / l.chunk) * row; };
  // chunks of 32 tokens only where those of 64 make no more than two CTAs per SM, counting every request as hidden-cached and as
  // long as its table (the host knows no more): a CTA's time is its tokens' round trips, but every chunk's partial sums are
  // read again (four OPT-125M requests 13.2 -> 8.4 us)
  if ((int64_t)l.count * ((max_tokens + 63) / 64) * ((heads + kHeads - 1) / kHeads) > 2 * sm_count()) l.chunk = 64;
  while (l.chunk < kMaxChunk && (size_t)l.count * per_request() > kScratch) l.chunk *= 2;
  l.chunks = (int)((max_tokens + l.chunk - 1) / l.chunk);
  while (l.count > 1 && (size_t)l.count * per_request() > kScratch) l.count = (l.count + 1) / 2;
  l.splits = sm_count() / heads;   // one wave of unfold CTAs for one group of R requests
  const int steps = (hidden + 255) / 256;
  l.splits = l.splits < 1 ? 1 : l.splits > steps ? steps : l.splits;
  size_t o = 0;
  auto take = [&](size_t bytes) { const size_t at = o; o = align_up(o + bytes, 256); return at; };
  l.off_groups = take((size_t)l.n_groups * sizeof(GroupPlan));
  l.off_slot = take((size_t)batch * sizeof(int));
  l.off_list = take((size_t)batch * sizeof(int2));
  l.off_qt = take((size_t)l.count * row);
  l.off_ml = take((size_t)l.count * l.chunks * heads * 2 * sizeof(float));
  l.off_z = take((size_t)l.count * l.chunks * row);
  l.off_part = take((size_t)l.splits * l.n_hidden_cap * heads * head_size * sizeof(float));
  l.total = o;
  return l;
}

template <int D>
int launch_group(const Params& p, int splits, bool behind_kv, cudaStream_t stream) {
  constexpr int R = D == 128 ? 4 : 8;
  int st;
  if ((st = launch_chained("fold32_kernel", fold32_kernel<D>, dim3((p.hidden + 127) / 128, p.heads, (p.count + kFoldReqs - 1) / kFoldReqs),
                           kThreads, 0, stream, p, behind_kv ? 1 : 0)) != APS_OK) return st;
  if ((st = launch_chained("attend32_kernel", attend32_kernel, dim3(p.chunks, p.count, (p.heads + kHeads - 1) / kHeads), kThreads, 0,
                           stream, p)) != APS_OK) return st;
  return launch_chained("unfold32_kernel", unfold32_kernel<D>, dim3(p.heads, splits, (p.count + R - 1) / R), kThreads, 0, stream, p);
}

}  // namespace

// Rows of W and of the cache are read 16 bytes at a time: sizes and strides in multiples of four elements, aligned
// bases.  Anything else stays with the re-projecting kernel, as does a caller whose scratch has only that one's size.
bool folded32_shape(int dtype, int heads, int head_size, int hidden) {
  return dtype == APS_F32 && (head_size == 32 || head_size == 64 || head_size == 128) && hidden > 0 && hidden % 4 == 0 &&
         heads > 0 && heads <= 65535;   // heads are a grid dimension
}

bool folded32_supported(const HybridCall& c) {
  const AttnShape& s = c.shape;
  return folded32_shape(s.dtype, s.heads, s.head_size, c.hidden_size) && c.hidden_row_stride % 4 == 0 && c.w_stride % 4 == 0 &&
         c.hidden_cache && c.w_k && c.w_v && c.num_hidden_rows > 0 && c.hidden_row_stride >= c.hidden_size &&
         c.w_stride >= c.hidden_size && aligned_to(c.hidden_cache, 16) && aligned_to(c.w_k, 16) && aligned_to(c.w_v, 16) &&
         c.workspace_bytes >= folded32_workspace_bytes(s.batch, s.max_blocks_per_seq, s.block_size, s.heads, s.head_size, c.hidden_size);
}

size_t folded32_workspace_bytes(int batch, int max_blocks_per_seq, int block_size, int heads, int head_size, int hidden) {
  return align_up(workspace_layout(batch, max_blocks_per_seq, block_size, heads, head_size).total, 256) +
         layout_of(batch, max_blocks_per_seq, block_size, heads, head_size, hidden).total;
}

int enqueue_folded32_attention(const HybridCall& c, const NewTokenWrite& nw, cudaStream_t cs) {
  const AttnShape& s = c.shape;
  const WorkspaceLayout w = workspace_layout(s.batch, s.max_blocks_per_seq, s.block_size, s.heads, s.head_size);
  const WorkspacePtrs ws = workspace_ptrs(c.workspace, w);
  const Layout l = layout_of(s.batch, s.max_blocks_per_seq, s.block_size, s.heads, s.head_size, c.hidden_size);
  char* b = static_cast<char*>(c.workspace) + align_up(w.total, 256);
  GroupPlan* groups = reinterpret_cast<GroupPlan*>(b + l.off_groups);
  const bool have_kv = c.key_cache != nullptr && c.value_cache != nullptr;
  int st;

  PlanArgs pa{};
  pa.plan = ws.plan; pa.part_offset = ws.part_offset; pa.kv_chunks = ws.kv_chunks;
  pa.hid_slot = reinterpret_cast<int*>(b + l.off_slot); pa.hid_list = reinterpret_cast<int2*>(b + l.off_list);
  pa.groups = groups; pa.seq_lens = c.seq_lens; pa.cache_type = c.cache_type; pa.batch = s.batch;
  pa.max_tokens = s.max_blocks_per_seq * s.block_size; pa.kv_present = have_kv ? 1 : 0; pa.n_groups = l.n_groups;
  pa.steps = 1; pa.grid_scores = 1; pa.max_slice = 1; pa.item_target = 1;
  if ((st = launch_step_plan(&pa, nw, cs)) != APS_OK) return st;
  ScopedProfile prof(1, cs);   // with the K/V kernel's events inside, as in hidden_attention.cu
  if (have_kv &&
      (st = launch_kv_attention(ws, c.query, c.key_cache, c.value_cache, c.block_tables, c.seq_lens, s, cs)) != APS_OK) return st;

  Params p{};
  p.plan = groups; p.query = static_cast<const float*>(c.query); p.x = static_cast<const float*>(c.hidden_cache);
  p.w_k = static_cast<const float*>(c.w_k); p.w_v = static_cast<const float*>(c.w_v); p.block_tables = c.block_tables;
  p.qt = reinterpret_cast<float*>(b + l.off_qt); p.ml = reinterpret_cast<float*>(b + l.off_ml);
  p.z = reinterpret_cast<float*>(b + l.off_z); p.out_part = reinterpret_cast<float*>(b + l.off_part);
  p.heads = s.heads; p.hidden = c.hidden_size; p.block_size = s.block_size; p.max_blocks = s.max_blocks_per_seq;
  p.chunk = l.chunk; p.chunks = l.chunks; p.n_hidden_cap = l.n_hidden_cap;
  p.query_stride = s.query_stride; p.x_stride = c.hidden_row_stride; p.w_stride = c.w_stride;
  p.scale_log2 = s.scale * 1.4426950408889634f;
  for (int first = 0; first < s.batch; first += l.count) {
    p.first = first;
    p.count = s.batch - first < l.count ? s.batch - first : l.count;
    const bool behind_kv = have_kv && first == 0;
    switch (s.head_size) {
      case 128: st = launch_group<128>(p, l.splits, behind_kv, cs); break;
      case 64: st = launch_group<64>(p, l.splits, behind_kv, cs); break;
      default: st = launch_group<32>(p, l.splits, behind_kv, cs); break;
    }
    if (st != APS_OK) return st;
  }
  const HiddenOutputs ho{pa.hid_slot, p.out_part, c.b_v, c.seq_lens, l.splits, p.n_hidden_cap};
  return launch_combine(ws, c.out, &ho, s, cs);
}

}  // namespace aps
