// Hidden-path decode attention with the K / V projections moved to the query and to the output.
//
// What it replaces in the reference (paths under additional_designs/):
//   model_executor/models/aptserve_opt.py:111-124   gather of every cached hidden row and the
//       kv_only projection of all of them (model_executor/layers/aptserve_linear.py:123-130);
//   attention/backends/aptserve_flash_attn.py:356-387, :462-473   scatter of the projected K / V and
//       the paged attention over them.
//
// For a hidden-cached request with cached rows x_t and head h,
//     q . (W_k,h x_t + b_k) = (W_k,h^T q) . x_t + const        (the constant leaves the softmax)
//     sum_t p_t (W_v,h x_t + b_v) = W_v,h (sum_t p_t x_t) + b_v
// so the rows are attended as they are, with K = V = X and a head dimension of E.  Re-projecting T
// rows costs 4 T E H D operations; this form costs 4 E H (D + T): D times less for long contexts.
// What is left is bound by memory: the rows are read twice (scores, weighted sums), W_k once per 128 requests and W_v once
// per D requests (128, 64 or 32) of a group.
// Measured on one B200: a step of 256 requests of an OPT-13B layer, half of them hidden-cached (94.7k rows),
// 0.78 - 0.83 ms (the SM clock under the power cap) against 8.1 - 9.7 with the re-projecting kernel; one rank of eight of an
// OPT-66B layer, 128 requests, 0.41 - 0.43 ms against 1.6 - 2.0; 24 hidden-cached requests of about 1800 tokens 0.18 ms against 2.5.
//
//   step_plan_kernel the plan, and the new tokens' cache rows
//   fold_kernel      qt[r][h] = W_k,h^T q[r][h]                       tcgen05, M = 128 columns of E
//   scores_kernel    s[t][h] = x_t . qt[r][h]                         tcgen05, M = 128 tokens
//   softmax_kernel   p[t][h] = 2^(scale s - max)                      four warps per (request, two heads)
//   sum_kernel       z[r][h] = sum_t p[t][h] x_t / sum_t p[t][h]      tcgen05, M = 128 columns of E
//   unfold_kernel    y[r][h] = W_v,h z[r][h]                          tcgen05, M = 128 rows of W_v
// and the combine kernel adds b_v.
//
// Precision.  x, W and q are used as they are stored.  The three intermediates that meet a tensor-core
// operand (qt, p, z) are fp32 values carried as a sum of 16-bit TERMS (value = hi + rest, rest again
// rounded): two for fp16 (22 bits), three for bf16 (24 bits), each multiplied separately into fp32
// accumulators.  fp16 has a narrow exponent:
//   - q is normalised by a power of two before it is folded (|q| < 2) and the folded query is kept at 1 / 2D of its
//     value (both undone in the softmax): |qt| <= sum_d |q_d W_d| < 2 D 65504 always fits;
//   - p is kept at 2^15 times its value (undone by the normalisation), so that what its second term loses below
//     2^-24 is 2^-39 of the largest weight;
//   - the rests of qt and z are kept at 2^11 times their value and multiplied into accumulators of their own, which
//     the epilogues add with 2^-11.  Kept as they are they are subnormal as soon as the value is below 0.1: the weighted
//     sums then had an absolute error of 2^-26, 3.6 units of the output's last place for cached rows of N(0, 0.01) and
//     W_v of N(0, 1).  Now the value's error is 2^-23 of it or 2^-36, whichever is more.
//
// Requests are taken in groups of at most kGroup, so that most of the scratch (qt and z: kGroup x H x E terms, scores and
// weights) does not grow with the batch beyond one group (the projected outputs, splits x H x D per request, do); inside a
// group they are sorted by length, longest first.  The host does not know how many requests are hidden-cached and
// enqueues the five kernels for every group there could be; one that finds nothing to do takes 1 us.
//
// Every mbarrier wait is bounded by a clock budget; a wait that runs out records a code in the plan's
// status word, tells the other warps through shared memory, and the CTA drains and returns.

#include "attention_common.cuh"
#include "sm100.cuh"
#include "step_plan.cuh"
#include "tensor_maps.cuh"

#include <initializer_list>
#include <type_traits>

namespace aps {
namespace {

constexpr int kTile = 256;                // tokens per scores tile: two M128 accumulators share a qt slab
constexpr int kSubs = kTile / 16;         // 16-row boxes of the hidden cache per tile
constexpr int kTileCost = 4;              // fixed cost of a tile in boxes (its qt slab), for the work split
constexpr int kMinPiece = 2 * (kSubs + kTileCost);   // least work of a CTA of the scores kernel: two full steps
constexpr int kMaxSlice = 4;              // 128-column blocks of E per work item of the sum kernel
constexpr int kSumRounds = 2;             // work items per SM below which it takes narrower slices
constexpr float kProbShift = 15.f;        // p is kept at 2^15 times its value (fp16 range)
constexpr size_t kRingBytes = 200 * 1024; // shared memory of the operand rings

template <typename T> constexpr int kTerms = std::is_same<T, __nv_bfloat16>::value ? 3 : 2;
template <typename T> constexpr uint32_t kFmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;

// The scores work is a line of X box-steps, cut into pieces that are handed out in order: `levels` sizes, each
// half of the one before (the last two alike), `per_level` pieces of each.  Large pieces first keep the
// number of cut tiles down, small ones last let the CTAs end together: one equal piece per CTA left the SMs
// idle for a fifth of the kernel (they do not get equal shares of the memory bandwidth).  In units of the
// smallest size there are per_level << (levels - 1) of them; piece c starts at unit_of_piece(c), position
// X * unit / units.
__device__ inline int unit_of_piece(int c, int levels, int per_level) {
  const int l = c / per_level, k = c - l * per_level;
  const int size = l >= levels - 2 ? 1 : 1 << (levels - 2 - l);
  return l >= levels ? per_level << (levels - 1) : per_level * ((1 << (levels - 1)) - (1 << (levels - 1 - l))) + k * size;
}

struct Params {
  GroupPlan* plan;
  const void* query; const int32_t* block_tables; const int32_t* cache_type;
  void* qt;              // [request][term][head][E]
  float* qscale;         // [request][head] scale * log2(e) / (power of two q was multiplied with)
  float* scores;         // [tile + piece][head][kTile] partial scores over a range of E
  int2* tile_pieces;     // [tile] the first and the last piece with a part of it
  void* probs;           // [16-token block][K half][term][heads padded][8 tokens]; some blocks' first term last (SumColumns)
  float* inv_sum;        // [request][head]
  void* z;               // [term][head][request capacity][E]
  float* out_part;       // [split][hidden request][H * D]
  int* status;
  int batch, heads, np, head_size, hidden, slabs;   // np: heads padded to a multiple of 16; slabs: E / 64
  int block_size, max_blocks, n_cap;         // n_cap: requests a group can hold here
  int group_first;                           // ordinal of the group's first hidden request
  int n_hidden_cap, splits, grid_scores;
  uint32_t unfold_ring;                      // bytes of the unfold kernel's ring
  int sum_threads, sum_copiers;              // of the sum kernel
  int w_box_rows;                            // rows of a W_v box: 128, fewer when W_v has fewer
  int64_t query_stride;
  float scale_log2;
};

// SCALED: fp16's second term at kRestUp times its value, for products that have accumulators of their own.
constexpr float kRestUp = 2048.f;
template <typename T> constexpr float kRestDown = kTerms<T> == 2 ? 1.f / kRestUp : 1.f;
template <typename T, bool SCALED>
__device__ __forceinline__ void split_terms(float v, T (&t)[kTerms<T>]) {
#pragma unroll
  for (int i = 0; i < kTerms<T>; ++i) {
    t[i] = Elem<T>::from_float(v);
    v -= Elem<T>::to_float(t[i]);
    if (SCALED && kTerms<T> == 2) v *= kRestUp;
  }
}
// The value whose terms' products are v, the smaller ones added first.
template <int NT, int N>
__device__ __forceinline__ float add_terms(const uint32_t (&v)[NT][N], int j) {
  if constexpr (NT == 2) return fmaf(__uint_as_float(v[1][j]), 1.f / kRestUp, __uint_as_float(v[0][j]));
  float x = __uint_as_float(v[NT - 1][j]);
#pragma unroll
  for (int i = NT - 2; i >= 0; --i) x += __uint_as_float(v[i][j]);
  return x;
}
// The folded query is kept at this fraction of its value.
template <typename T, int D> constexpr float kFoldDown = kTerms<T> == 2 ? 0.5f / D : 1.f;
template <typename T>
__device__ __forceinline__ uint32_t pack_pair(T a, T b) {
  return (uint32_t)reinterpret_cast<const unsigned short&>(a) | ((uint32_t)reinterpret_cast<const unsigned short&>(b) << 16);
}
// Two columns a, b of an accumulator whose rows are the lanes: lane pairs exchange values so that
// an even lane returns (row, row + 1) of column a and an odd lane (row - 1, row) of column b.
__device__ __forceinline__ float2 pair_rows(float a, float b, int lane) {
  const bool odd = (lane & 1) != 0;
  const float got = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
  return odd ? make_float2(got, b) : make_float2(a, got);
}

// Copies still in flight get a bounded time to land before the CTA's shared memory is released.
__device__ __forceinline__ void drain() {
  const long long t0 = clock64();
  while (clock64() - t0 < 2000000LL) { }
}

// ---- plan and new-token writes --------------------------------------------------------
// The first kernel of a layer-step.  CTA 0 plans: K/V-cached requests: the chunk list of the K/V kernel and the partial
// slots.  Hidden-cached requests: the groups.  Runs of requests per thread, warp-shuffle scans.  The other CTAs write the
// step's new rows, addressed straight from the block tables: a warp per 2 KB of a row, three round trips (length and
// type, block, row).  One launch instead of two one after the other, and the fold
// beside it: a step of one OPT-13B request 70 -> 60 us, of 48 OPT-1.3B requests 118 -> 108, of 8 in fp32 52 -> 45.

struct StepWrite {
  const char* hidden; const char* key; const char* value; char* key_cache; char* value_cache; char* hidden_cache;
  const int32_t* block_tables; const int32_t* seq_lens; const int32_t* cache_type;
  int batch, max_blocks, block_size, chunks;   // chunks: per row, of the longer kind
  uint32_t kv_row_bytes, hidden_row_bytes;
  int64_t hidden_stride_b, key_stride_b, value_stride_b, block_stride_b, slot_stride_b;
};

// Row 2 r is the K row (K/V-cached request) or the layer-input row (hidden-cached request) of request r, row 2 r + 1 its
// V row (K/V-cached requests only).  The token's position is seq_lens[r] - 1.
__device__ __forceinline__ void write_new_rows(const StepWrite& w, int64_t job, int lane) {
  const int64_t row = job / w.chunks, r = row >> 1;
  if (r >= w.batch) return;
  const uint32_t at = (uint32_t)(job - row * w.chunks) * kWriteChunk;
  const bool second = (row & 1) != 0;
  const int pos = min(w.seq_lens[r], w.max_blocks * w.block_size) - 1, type = w.cache_type[r];
  if (pos < 0 || type == kCacheTypeNone) return;
  const bool hid = type != 0;
  const uint32_t bytes = hid ? w.hidden_row_bytes : w.kv_row_bytes;
  const char* base = hid ? w.hidden : second ? w.value : w.key;
  if (base == nullptr || (hid && second) || at >= bytes) return;
  const int64_t blk = w.block_tables[r * w.max_blocks + pos / w.block_size];
  const char* src = base + r * (hid ? w.hidden_stride_b : second ? w.value_stride_b : w.key_stride_b);
  char* dst = hid ? w.hidden_cache + (blk * w.block_size + pos % w.block_size) * w.slot_stride_b
                  : (second ? w.value_cache : w.key_cache) + blk * w.block_stride_b + (int64_t)(pos % w.block_size) * bytes;
  move_chunk(dst, src, at, bytes, lane);
}

__global__ void __launch_bounds__(kPlanThreads)
step_plan_kernel(const PlanArgs a, const StepWrite w, const int plan_ctas) {
  __shared__ int2 warp_sums[32];
  __shared__ int s_missing;
  __shared__ int s_req[kGroup], s_len[kGroup], s_toff[kGroup + 1], s_woff[kGroup + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_missing = 0;
  chain_wait();
  chain_next();
  if ((int)blockIdx.x >= plan_ctas) {
    write_new_rows(w, (int64_t)((int)blockIdx.x - plan_ctas) * (kPlanThreads / 32) + warp, lane);
    return;
  }
  __syncthreads();
  const int per = (a.batch + kPlanThreads - 1) / kPlanThreads;
  const int r0 = min(a.batch, tid * per), r1 = min(a.batch, r0 + per);
  auto chunks_of = [&](int s) { return a.kv_present ? (s + kChunkTokens - 1) / kChunkTokens : 0; };
  int2 mine = make_int2(0, 0);
  for (int r = r0; r < r1; ++r) {
    const int s = max(0, min(a.seq_lens[r], a.max_tokens)), type = a.cache_type[r];
    if (type == kCacheTypeNone) continue;
    if (type != 0) ++mine.y;
    else { mine.x += chunks_of(s); if (!a.kv_present) s_missing = 1; }
  }
  int2 total;
  const int2 inc = block_scan(mine, warp_sums, tid, total);
  int o_kv = inc.x - mine.x, o_hid = inc.y - mine.y;
  for (int r = r0; r < r1; ++r) {
    const int s = max(0, min(a.seq_lens[r], a.max_tokens)), type = a.cache_type[r];
    a.part_offset[r] = o_kv;
    if (type != 0 && type != kCacheTypeNone) {
      a.hid_list[o_hid++] = make_int2(r, s);
    } else {
      a.hid_slot[r] = -1;
      const int c = type != 0 ? 0 : chunks_of(s);
      for (int j = 0; j < c; ++j) a.kv_chunks[o_kv + j] = make_int2(r, j);
      o_kv += c;
    }
  }
  if (tid == 0) {
    a.part_offset[a.batch] = total.x;
    a.plan[kPlanNumKvChunks] = total.x;
    a.plan[kPlanKvCounter] = 0;
    a.plan[kPlanStatus] = s_missing ? kStatusNoKvCache : kStatusOk;
  }
  if (tid >= kPlanStatsWord && tid < kPlanStatsWord + 18) a.plan[tid] = 0;
  for (int g = 0; g < a.n_groups; ++g) {
    __syncthreads();   // hid_list is complete; the shared arrays are free
    GroupPlan* gp = a.groups + g;
    const int n = max(0, min(kGroup, total.y - g * kGroup));
    if (n == 0) {
      if (tid == 0) gp->n = 0;
      continue;
    }
    // sort by length, longest first: rank = requests that come before (four threads per request)
    const int i = tid >> 2, part = tid & 3;
    int2 rec = make_int2(0, -1);
    if (i < n) rec = a.hid_list[g * kGroup + i];
    if (part == 0) s_len[i] = rec.y;
    __syncthreads();
    int rank = 0;
    for (int j = part; j < n; j += 4) {
      const int l = s_len[j];
      rank += l > rec.y || (l == rec.y && j < i);
    }
    rank += __shfl_xor_sync(0xffffffffu, rank, 1);
    rank += __shfl_xor_sync(0xffffffffu, rank, 2);
    __syncthreads();
    if (i < n && part == 0) {
      s_req[rank] = rec.x; s_len[rank] = rec.y;
      gp->req[rank] = rec.x; gp->len[rank] = rec.y; gp->ord[rank] = i;
      a.hid_slot[rec.x] = g * kGroup + rank;
    }
    __syncthreads();
    if (warp == 0) {   // prefix sums over the sorted requests, eight per lane
      int t8 = 0, b8 = 0, w8 = 0;
      for (int k = 0; k < kGroup / 32; ++k) {
        const int s = lane * (kGroup / 32) + k;
        if (s >= n) break;
        const int blocks = (s_len[s] + 15) / 16, tiles = (blocks + kSubs - 1) / kSubs;
        t8 += tiles; b8 += blocks; w8 += blocks + tiles * kTileCost;
      }
      int ti = t8, bi = b8, wi = w8;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, ti, o), y = __shfl_up_sync(0xffffffffu, bi, o),
                  z = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= o) { ti += x; bi += y; wi += z; }
      }
      int to = ti - t8, bo = bi - b8, wo = wi - w8;
      for (int k = 0; k < kGroup / 32; ++k) {
        const int s = lane * (kGroup / 32) + k;
        if (s > n) break;
        s_toff[s] = to; s_woff[s] = wo;
        gp->tile_off[s] = to; gp->blk_off[s] = bo;
        if (s == n) break;
        const int blocks = (s_len[s] + 15) / 16, tiles = (blocks + kSubs - 1) / kSubs;
        to += tiles; bo += blocks; wo += blocks + tiles * kTileCost;
      }
      if (lane == 31 && n == kGroup) {
        s_toff[n] = to; s_woff[n] = wo;
        gp->tile_off[n] = to; gp->blk_off[n] = bo;
      }
    }
    __syncthreads();
    const int n_tiles = s_toff[n], weight = s_woff[n];
    if (tid == 0) {
      // sum kernel: the widest slice of E that still gives item_target items.  Wide slices leave a DRAM page after
      // up to 1 KB of a row, not 256 bytes, and read the weights less often (a slice of one block reads as many bytes of
      // weights as of rows); more items even out requests of different lengths.  On one B200, slices of 1 / 2 / 3 / 4
      // blocks: 24 requests of 1800 OPT-13B tokens 95 / 76 / 79 / 87 us, 128 of 740 - / - / 197 / 186; before the
      // narrow slices had stages of four cache blocks 52 of 950 OPT-66B tp 8 - / 255 / 177 / 167, 34 of 500 OPT-1.3B
      // 36 / 54 / - / 53.
      int slice = a.max_slice;
      while (slice > 1 && n * ((a.steps + slice - 1) / slice) < a.item_target) --slice;
      gp->n = n; gp->slice = slice; gp->turns = (a.turns >> (4 * slice)) & 15;
    }
    // cut the scores work.  No piece is smaller than kMinPiece (more than a full step), so that none is empty
    // and the partial sums of a tile stay few.
    const int64_t work = (int64_t)weight * a.steps;
    const int per_level = (int)max((int64_t)1, min((int64_t)a.grid_scores, work / kMinPiece));
    int levels = 1;
    while (levels < kMaxLevels && work / ((int64_t)per_level << levels) >= kMinPiece) ++levels;
    if (tid == 0) { gp->levels = levels; gp->per_level = per_level; gp->next_piece = 0; gp->next_item = 0; }
    for (int c = tid; c <= levels * per_level; c += kPlanThreads) {
      int t = n_tiles, step = 0;
      if (c < levels * per_level && weight > 0) {
        const int64_t pos = work * unit_of_piece(c, levels, per_level) / ((int64_t)per_level << (levels - 1));
        int lo = 0, hi = n;   // last request whose cost offset is <= pos
        while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if ((int64_t)s_woff[mid] * a.steps <= pos) lo = mid; else hi = mid; }
        const int64_t rem = pos - (int64_t)s_woff[lo] * a.steps;
        const int blocks = (s_len[lo] + 15) / 16, tiles = (blocks + kSubs - 1) / kSubs;
        const int k = min((int)(rem / ((int64_t)(kSubs + kTileCost) * a.steps)), tiles - 1);
        const int w = min(kSubs, blocks - k * kSubs) + kTileCost;
        t = s_toff[lo] + k;
        step = (int)((rem - (int64_t)k * (kSubs + kTileCost) * a.steps) / w);
      }
      gp->bound_tile[c] = t; gp->bound_step[c] = step;
    }
  }
}

// ---- fold ---------------------------------------------------------------------------
// D[column of E][request] = sum_d W_k,h[d][column] q[request][d], exact 16-bit operands, fp32 accumulators.
// One CTA per (range of E, head, 128 requests): q is gathered once by all threads into a K-major B operand
// and stays; W_k,h streams past it in tiles of 128 columns (two boxes of 64 columns x D rows, an MN-major
// A operand) through a two-stage ring, the accumulators are double-buffered.  Two CTAs per SM.
// It takes the group's requests in batch order; the first group's are found in cache_type by itself, so that it needs neither
// the plan nor the new rows: that fold runs beside the step's first kernel (wait_last; what was enqueued before that
// one is complete, since it waits before it lets this one start) and waits before it exits.
// Warps: 0 copies, 1 MMA issue, 2-9 epilogue, two per quarter of the accumulators' lanes, which take 16 requests in turns:
// with one the kernel waited for its chain of tensor-memory loads, shuffles and stores (issue slots a third full, no unit
// near its limit): 40 -> 30 us for 128
// OPT-13B requests, 50 -> 35 in bf16, 23 -> 17 for 64.
constexpr int kFoldThreads = 320;
constexpr int kFoldReqs = 128;
constexpr int kFoldStages = 2;

struct FoldAux {
  uint64_t full[kFoldStages], empty[kFoldStages], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

template <int D> constexpr size_t fold_smem() {
  return 1024 + (size_t)kFoldStages * 2 * D * 128 + (size_t)((D + 63) / 64) * kFoldReqs * 128;
}

// Gathers q[request][head] of m requests, reqs, of ordinals from r0 on (zero rows up to np) into shared memory: slabs of
// 64 elements, rows of 128 bytes, 128-byte swizzle.  All warps of the CTA.
template <typename T, int D>
__device__ __forceinline__ void stage_queries(const Params& p, const int* reqs, uint32_t q_at, int r0, int m, int np, int head, bool keep_scale) {
  constexpr int kWarps = kFoldThreads / 32, U = 4, EPL = D / 32;   // U requests at a time, EPL elements per lane
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* query = static_cast<const T*>(p.query);
  for (int r = warp; r < np; r += kWarps * U) {
    T v[U][EPL];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int rr = r + u * kWarps;
      const bool in = rr < m;
      const T* src = query + (in ? (int64_t)reqs[rr] * p.query_stride + head * D + lane * EPL : 0);
#pragma unroll
      for (int e = 0; e < EPL; ++e) v[u][e] = in ? src[e] : Elem<T>::from_float(0.f);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int rr = r + u * kWarps;
      if (rr >= np) break;
      float f[EPL], mx = 0.f;
#pragma unroll
      for (int e = 0; e < EPL; ++e) { f[e] = Elem<T>::to_float(v[u][e]); mx = fmaxf(mx, fabsf(f[e])); }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      // power of two that brings max |q| into [1, 2); zero, infinite and NaN rows stay as they are
      int k = 0;
      if (mx > 0.f && mx < INFINITY) k = max(-100, min(100, (int)((__float_as_uint(mx) >> 23) & 0xff) - 127));
      const float up = __uint_as_float((uint32_t)(127 - k) << 23), down = __uint_as_float((uint32_t)(127 + k) << 23);
      unsigned short w[EPL];
#pragma unroll
      for (int e = 0; e < EPL; ++e) { const T t = Elem<T>::from_float(f[e] * up); w[e] = reinterpret_cast<const unsigned short&>(t); }
      const int el = lane * EPL, slab = el / 64, piece = (el % 64) / 8, in_piece = el % 8;
      const uint32_t dst = q_at + slab * (kFoldReqs * 128) + rr * 128 + ((piece ^ (rr & 7)) << 4) + in_piece * 2;
      if constexpr (EPL == 4) asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst), "r"((uint32_t)w[0] | ((uint32_t)w[1] << 16)), "r"((uint32_t)w[2] | ((uint32_t)w[3] << 16)) : "memory");
      else if constexpr (EPL == 2) asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst), "r"((uint32_t)w[0] | ((uint32_t)w[1] << 16)) : "memory");
      else asm volatile("st.shared.b16 [%0], %1;" ::"r"(dst), "h"(w[0]) : "memory");
      if (keep_scale && lane == 0 && rr < m) p.qscale[(int64_t)(r0 + rr) * p.heads + head] = p.scale_log2 * (down * (1.f / kFoldDown<T, D>));
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // read by the tensor cores next
}

// The batch rows of hidden-cached requests first ... first + kFoldReqs - 1 (counted over the batch); returns how many there
// are of them.  All warps of the CTA; a warp counts 32 rows at a time.
__device__ __forceinline__ int find_requests(const int32_t* cache_type, int batch, int first, int* reqs, int* counts) {
  constexpr int kWarps = kFoldThreads / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int before = 0;
  for (int b = 0; b < batch && before < first + kFoldReqs; b += kFoldThreads) {
    const int r = b + threadIdx.x, type = r < batch ? cache_type[r] : 0;
    const bool hid = type != 0 && type != kCacheTypeNone;
    const uint32_t mask = __ballot_sync(0xffffffffu, hid);
    __syncthreads();   // the last round's counts have been read
    if (lane == 0) counts[warp] = __popc(mask);
    __syncthreads();
    int at = before + __popc(mask & ((1u << lane) - 1)) - first;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) {
      at += k < warp ? counts[k] : 0;
      before += counts[k];
    }
    if (hid && at >= 0 && at < kFoldReqs) reqs[at] = r;
  }
  __syncthreads();
  return max(0, min(kFoldReqs, before - first));
}

// The same from the plan, where it is complete: the first group's fold runs beside the planning, the others behind it.  Counting
// in these too, an empty group's fold took 9 us instead of 4 (700 OPT-1.3B requests without hidden-cached ones, three groups).
__device__ __forceinline__ int planned_requests(const GroupPlan* gp, int first, int* reqs) {
  static_assert(kFoldThreads >= kGroup, "a thread per request of the group");
  const int n = gp->n;
  if ((int)threadIdx.x < n) {
    const int at = gp->ord[threadIdx.x] - first;
    if (at >= 0 && at < kFoldReqs) reqs[at] = gp->req[threadIdx.x];
  }
  __syncthreads();
  return max(0, min(kFoldReqs, n - first));
}

template <typename T, int D>
__global__ void __launch_bounds__(kFoldThreads, 2)
fold_kernel(const __grid_constant__ CUtensorMap map_w, const Params p, const int wait_last) {
  constexpr int NT = kTerms<T>;
  constexpr uint32_t kBox = D * 128, kStage = 2 * kBox;   // 64 columns of E x D rows; two of them
  extern __shared__ uint8_t smem_raw[];
  const uint32_t ring = (smem_u32(smem_raw) + 1023) & ~1023u, q_at = ring + kFoldStages * kStage;
  __shared__ FoldAux aux;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  if (!wait_last) chain_wait();
  __shared__ int s_reqs[kFoldReqs], s_counts[kFoldThreads / 32];
  const int r0 = blockIdx.z * kFoldReqs, head = blockIdx.y;
  const int m = wait_last ? find_requests(p.cache_type, p.batch, r0, s_reqs, s_counts) : planned_requests(p.plan, r0, s_reqs),
            np = (m + 15) & ~15;
  if (m == 0) { chain_wait(); return; }
  const int blocks = p.hidden / 128;
  const int ta = blocks * blockIdx.x / gridDim.x, tb = blocks * (blockIdx.x + 1) / gridDim.x;
  volatile int* abort_flag = &aux.abort_flag;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kFoldStages; ++s) { mbar_init(&aux.full[s], 1); mbar_init(&aux.empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&aux.acc_full[b], 1); mbar_init(&aux.acc_empty[b], kFoldThreads / 32 - 2); }
    aux.abort_flag = 0;
    mbar_init_fence();
    for (int i = 0; i < kFoldStages && ta + i < tb; ++i) {   // the first tiles are on their way while q is staged
      const uint32_t bar = smem_u32(&aux.full[i]), dst = ring + i * kStage;
      mbar_expect_tx_addr(bar, kStage);
      tma_load_2d_cta(dst, &map_w, bar, (ta + i) * 128, head * D);
      tma_load_2d_cta(dst + kBox, &map_w, bar, (ta + i) * 128 + 64, head * D);
    }
  }
  if (warp == 1) tmem_alloc(&aux.tmem_base, 2 * kFoldReqs);
  stage_queries<T, D>(p, s_reqs, q_at, r0, m, np, head, blockIdx.x == 0);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_next();
  const uint32_t tmem = aux.tmem_base;
  bool ok = true;
  if (warp == 0) {
    for (int t = ta + kFoldStages; t < tb; ++t) {
      const int i = t - ta, s = i % kFoldStages;
      if (!mbar_wait_warp(smem_u32(&aux.empty[s]), (uint32_t)(i / kFoldStages - 1) & 1u, abort_flag, p.status, 1, lane)) { ok = false; break; }
      if (lane == 0) {
        const uint32_t bar = smem_u32(&aux.full[s]), dst = ring + s * kStage;
        mbar_expect_tx_addr(bar, kStage);
        tma_load_2d_cta(dst, &map_w, bar, t * 128, head * D);
        tma_load_2d_cta(dst + kBox, &map_w, bar, t * 128 + 64, head * D);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    const uint32_t idesc = mma_idesc(kFmt<T>, 128, (uint32_t)np, true);
    for (int t = ta; t < tb; ++t) {
      const int i = t - ta, s = i % kFoldStages, buf = i & 1;
      if (!mbar_wait_warp(smem_u32(&aux.acc_empty[buf]), ((uint32_t)(i >> 1) & 1u) ^ 1u, abort_flag, p.status, 2, lane)) { ok = false; break; }
      if (!mbar_wait_warp(smem_u32(&aux.full[s]), (uint32_t)(i / kFoldStages) & 1u, abort_flag, p.status, 3, lane)) { ok = false; break; }
      tc_fence_after();
      if (elect_one()) {
        const uint32_t a_lo = desc_lo(ring + s * kStage, kBox);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          tc_mma_cta(tmem + buf * kFoldReqs, a_lo + ks * 128, desc_hi(1024, true),
                     desc_lo(q_at + (ks / 4) * (kFoldReqs * 128) + (ks % 4) * 32, 16), desc_hi(1024, true), idesc, ks != 0);
        tc_commit_cta(smem_u32(&aux.empty[s]));
        tc_commit_cta(smem_u32(&aux.acc_full[buf]));
      }
      __syncwarp();
    }
  } else {
    // lanes are columns of E, accumulator columns are requests
    const int quarter = warp & 3, turn = (warp - 2) >> 2;
    const int64_t req_stride = (int64_t)NT * p.heads * p.hidden, term_stride = (int64_t)p.heads * p.hidden;
    T* qt = static_cast<T*>(p.qt) + (r0 + turn * 16 + (lane & 1)) * req_stride + (int64_t)head * p.hidden + quarter * 32 + (lane & ~1);
    for (int t = ta; t < tb; ++t) {
      const int i = t - ta, buf = i & 1;
      if (!mbar_wait_warp(smem_u32(&aux.acc_full[buf]), (uint32_t)(i >> 1) & 1u, abort_flag, p.status, 4, lane)) { ok = false; break; }
      tc_fence_after();
      T* dst = qt + t * 128;
      for (int c = turn * 16; c < np; c += 32) {
        uint32_t v[16];
        tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + buf * kFoldReqs + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const float2 f = pair_rows(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), lane);
          if (c + j + (lane & 1) < m) {
            T x[NT], y[NT];
            split_terms<T, true>(f.x * kFoldDown<T, D>, x);
            split_terms<T, true>(f.y * kFoldDown<T, D>, y);
#pragma unroll
            for (int k = 0; k < NT; ++k) *reinterpret_cast<uint32_t*>(dst + k * term_stride) = pack_pair<T>(x[k], y[k]);
          }
          dst += 2 * req_stride;
        }
        dst += 16 * req_stride;   // the other warp's
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_addr(smem_u32(&aux.acc_empty[buf]));
    }
  }
  if (!ok) drain();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_free(tmem, 2 * kFoldReqs); }
  chain_wait();
}

// ---- scores -------------------------------------------------------------------------
// D[token][head] = sum_e x[token][e] qt[head][e] for tiles of 256 tokens of one request (two M128
// accumulators that share a qt step).  The work is a line of (tile, 128 columns of E) steps, cut into
// contiguous pieces (see unit_of_piece): a tile that straddles a cut leaves one partial sum per piece (slot =
// tile + piece), added by the softmax kernel, so that one long request uses the whole chip and a large
// batch has no partly filled last wave.  94.7k rows of an OPT-13B layer (0.97 GB): 190 us; one equal piece per
// CTA took 26 us longer.
// A box is (64 columns, 8 rows, 2): 256 contiguous bytes of a cached row, so that a DRAM page is left after
// 256 bytes and not 128, and 8-row groups that lie 2 KB apart, as the K-major operand needs them.  X and qt
// have a ring each: a unit of X is 128 tokens x 128 columns (32 KB), a unit of qt serves both halves of a
// tile.  Behind the K/V kernel it does not wait for that one (wait_last): plan and folded queries were complete when the K/V
// kernel let it start, and its CTAs fill the SMs which that one leaves; it waits before it exits.  L2: qt (105 MB for 128 OPT-13B requests) is read once per tile and was fetched from memory almost every time,
// because the rows, which are read once by this kernel, pushed it out (1.25 GB of DRAM traffic for 0.97 GB of rows).  The
// rows are the first to go (evict_first), qt stays (evict_last): 205 -> 190 us for 128 OPT-13B requests, 172 -> 155 for 52
// OPT-66B tp 8 requests, 69 -> 63 for 24 of 1800 OPT-13B tokens, 313 -> 283 for 100 OPT-66B tp 2.  Warps: 0 qt boxes, 1 MMA issue, 2-5 epilogue, 6-7 boxes of X (eight lanes each).
constexpr int kScoresThreads = 256;
constexpr int kMaxStages = 12;
constexpr int kMaxQUnits = 3;
constexpr uint32_t kUnitBytes = 128 * 256;
constexpr size_t kScoresRing = 216 * 1024;

struct RingAux {
  uint64_t full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2], q_full[kMaxQUnits], q_empty[kMaxQUnits];
  uint32_t tmem_base;
  int abort_flag;
};

constexpr int kItemSlots = 4;
// Work items passed from the copying warp that takes them to the other warps of the CTA.
struct ItemRing { uint64_t full[kItemSlots], empty[kItemSlots]; int item[kItemSlots]; };

struct Ring {
  uint32_t stage = 0, phase = 0;
  __device__ __forceinline__ void step(int stages) { if (++stage == (uint32_t)stages) { stage = 0; phase ^= 1u; } }
};

__host__ __device__ inline uint32_t scores_q_bytes(int terms, int np) { return (uint32_t)terms * np * 256; }
// The terms of qt as further columns of the B operand (N = terms x np, an accumulator per term, added in the epilogue)
// where N and the accumulators allow: the tensor cores read every X row from shared memory once per instruction, 4 KB
// or 32 cycles of its bandwidth against 12 - 24 of arithmetic, so an instruction per term costs two or three
// times that.
__host__ __device__ inline bool stacked_terms(int terms, int np) { return terms * np <= 256; }
// Heads too many for that: an instruction per term, into accumulators of its own for fp16 (its second term has a
// scale of its own) and, if those of a tile's two halves do not fit the tensor memory, the halves one after the
// other, with a second copy of qt.
// qt units in the ring: a step of a short tile takes less time than a unit's round trip, so three of them where that
// leaves three units of X (two and two, one otherwise).  Two -> three: scores of 128 OPT-13B requests of 740 tokens
// 213 -> 207 us, of 64 of 340 71 -> 67, of 52 OPT-66B tp 8 requests 182 -> 170; with four and fewer units of X the
// bf16 layers lose it again.
__host__ __device__ inline int scores_q_units(int terms, int np) {
  for (int n = kMaxQUnits; n > 1; --n)
    if (n * scores_q_bytes(terms, np) + n * kUnitBytes <= kScoresRing) return n;
  return 1;
}

template <typename T>
__global__ void __launch_bounds__(kScoresThreads, 1)
scores_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_q, const Params p, const int wait_last) {
  constexpr int NT = kTerms<T>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t x_ring = (smem_u32(smem_raw) + 1023) & ~1023u;
  __shared__ RingAux aux;
  __shared__ int s_toff[kGroup + 1], s_len[kGroup], s_req[kGroup], s_ord[kGroup];
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  __shared__ ItemRing items;
  if (!wait_last) chain_wait();
  GroupPlan* gp = p.plan;
  const int n = gp->n, n_pieces = gp->levels * gp->per_level;
  if (n == 0 || (int)blockIdx.x >= n_pieces) { chain_wait(); return; }
  for (int i = threadIdx.x; i <= n; i += kScoresThreads) {
    s_toff[i] = gp->tile_off[i];
    if (i < n) { s_len[i] = gp->len[i]; s_req[i] = gp->req[i]; s_ord[i] = gp->ord[i]; }
  }
  const int np = p.np, steps = p.hidden / 128;
  const uint32_t q_bytes = scores_q_bytes(NT, np);
  const int nq = scores_q_units(NT, np), nx = min(kMaxStages, (int)((kScoresRing - nq * q_bytes) / kUnitBytes));
  const uint32_t q_ring = x_ring + nx * kUnitBytes;
  const bool stacked = stacked_terms(NT, np), own_acc = NT == 2 || stacked;   // own_acc: an accumulator per term
  const int n_acc = own_acc ? NT * np : np, n_rep = stacked ? 1 : NT, m_step = 2 * n_acc <= 512 ? 2 : 1;
  const int n_buf = 2 * m_step * n_acc <= 512 ? 2 : 1;
  uint32_t tmem_cols = 32;
  while (tmem_cols < (uint32_t)(n_buf * m_step * n_acc)) tmem_cols <<= 1;
  if (threadIdx.x == 0) {
    for (int s = 0; s < nx; ++s) { mbar_init(&aux.full[s], 2); mbar_init(&aux.empty[s], 1); }
    for (int b = 0; b < kMaxQUnits; ++b) { mbar_init(&aux.q_full[b], 1); mbar_init(&aux.q_empty[b], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&aux.acc_full[b], 1); mbar_init(&aux.acc_empty[b], 4); }
    for (int i = 0; i < kItemSlots; ++i) { mbar_init(&items.full[i], 1); mbar_init(&items.empty[i], kScoresThreads / 32 - 1); }
    aux.abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(&aux.tmem_base, tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_next();
  const uint32_t tmem = aux.tmem_base;
  volatile int* abort_flag = &aux.abort_flag;
  const uint32_t full0 = smem_u32(&aux.full[0]), empty0 = smem_u32(&aux.empty[0]);
  const uint32_t q_full0 = smem_u32(&aux.q_full[0]), q_empty0 = smem_u32(&aux.q_empty[0]);
  const uint64_t once = l2_policy_evict_first(), again = l2_policy_evict_last();
  bool ok = true;
  Ring xr, qr, ir;
  uint32_t n_local = 0;
  int next = blockIdx.x;   // the first piece needs no counter
  while (ok) {
    int piece;
    if (warp == 0) {
      piece = next;
      if (!mbar_wait_warp(smem_u32(&items.empty[ir.stage]), ir.phase ^ 1u, abort_flag, p.status, 1, lane)) { ok = false; break; }
      if (lane == 0) {
        items.item[ir.stage] = piece;
        mbar_arrive_addr(smem_u32(&items.full[ir.stage]));
      }
    } else {
      if (!mbar_wait_warp(smem_u32(&items.full[ir.stage]), ir.phase, abort_flag, p.status, 6, lane)) { ok = false; break; }
      piece = items.item[ir.stage];
      __syncwarp();
      if (lane == 0) mbar_arrive_addr(smem_u32(&items.empty[ir.stage]));
    }
    ir.step(kItemSlots);
    if (piece >= n_pieces) break;
    if (warp == 0) {
      if (lane == 0) next = (int)gridDim.x + atomicAdd(&gp->next_piece, 1);
      next = __shfl_sync(0xffffffffu, next, 0);
    }
    const int t0 = gp->bound_tile[piece], t1 = gp->bound_tile[piece + 1];
    const int b0 = gp->bound_step[piece], b1 = gp->bound_step[piece + 1];
    int slot = 0;   // request of tile t0
    {
      int lo = 0, hi = n;
      while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (s_toff[mid] <= t0) lo = mid; else hi = mid; }
      slot = lo;
    }
    for (int t = t0; t <= t1 && ok; ++t) {
      const int sa = t == t0 ? b0 : 0, sb = t == t1 ? b1 : steps;
      if (sa >= sb) continue;
      while (t >= s_toff[slot + 1]) ++slot;
      const int tok0 = (t - s_toff[slot]) * kTile;
      const int n_sub = min(kSubs, (s_len[slot] - tok0 + 15) >> 4);
      const int n_m = n_sub > 8 ? 2 : 1;
      // box g of a unit: rows 8 g ... of its 128 tokens; warp 6 the first eight, warp 7 the others
      const int g = (warp - 6) * 8 + lane;
      int row[2] = {0, 0};
      bool has[2] = {false, false};
      int boxes[2] = {0, 0};
      if (warp >= 6) {
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const int sub = m * 8 + (g >> 1);
          has[m] = lane < 8 && sub < n_sub;
          boxes[m] = max(0, min(8, 2 * (n_sub - m * 8) - (warp - 6) * 8));
          if (has[m]) {
            const int tok = tok0 + sub * 16;
            row[m] = p.block_tables[(int64_t)s_req[slot] * p.max_blocks + tok / p.block_size] * p.block_size + tok % p.block_size + (g & 1) * 8;
          }
        }
      }
      for (int m0 = 0; m0 < n_m && ok; m0 += m_step) {   // halves m0 ... m1 - 1 of the tile, one set of accumulators
        const int m1 = min(n_m, m0 + m_step);
        const uint32_t buf = n_local % n_buf, use = n_local / n_buf;
        ++n_local;
        if (warp == 0) {
          for (int s = sa; s < sb; ++s) {
            if (!mbar_wait_warp(q_empty0 + qr.stage * 8, qr.phase ^ 1u, abort_flag, p.status, 1, lane)) { ok = false; break; }
            const uint32_t bar = q_full0 + qr.stage * 8;
            if (lane == 0) mbar_expect_tx_addr(bar, (uint32_t)(NT * 2 * p.heads * 128));
            __syncwarp();
            if (lane < 2 * NT)   // lane = (term, half of the columns); the terms of a half lie one behind the other
              tma_load_2d_hint(q_ring + qr.stage * q_bytes + ((lane & 1) * NT + (lane >> 1)) * np * 128, &map_q, bar, s * 128 + (lane & 1) * 64, (s_ord[slot] * NT + (lane >> 1)) * p.heads, again);
            __syncwarp();
            qr.step(nq);
          }
        } else if (warp >= 6) {
          for (int s = sa; s < sb && ok; ++s) {
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              if (m < m0 || m >= m1) continue;
              if (!mbar_wait_warp(empty0 + xr.stage * 8, xr.phase ^ 1u, abort_flag, p.status, 1, lane)) { ok = false; break; }
              const uint32_t bar = full0 + xr.stage * 8;
              if (lane == 0) mbar_expect_tx_addr(bar, (uint32_t)boxes[m] * 2048);
              __syncwarp();
              if (has[m]) tma_load_3d_hint(x_ring + xr.stage * kUnitBytes + g * 2048, &map_x, bar, 0, row[m], s * 2, once);
              __syncwarp();
              xr.step(nx);
            }
          }
        } else if (warp == 1) {
          if (!mbar_wait_warp(smem_u32(&aux.acc_empty[buf]), (use & 1u) ^ 1u, abort_flag, p.status, 2, lane)) { ok = false; break; }
          tc_fence_after();
          const uint32_t idesc = mma_idesc(kFmt<T>, 128, (uint32_t)(stacked ? NT * np : np), false);
          const uint32_t rep_acc = own_acc ? (uint32_t)np : 0u;
          for (int s = sa; s < sb && ok; ++s) {
            if (!mbar_wait_warp(q_full0 + qr.stage * 8, qr.phase, abort_flag, p.status, 3, lane)) { ok = false; break; }
            for (int m = m0; m < m1; ++m) {
              if (!mbar_wait_warp(full0 + xr.stage * 8, xr.phase, abort_flag, p.status, 3, lane)) { ok = false; break; }
              tc_fence_after();
              if (elect_one()) {
                const uint32_t a_lo = desc_lo(x_ring + xr.stage * kUnitBytes, 16), b_lo = desc_lo(q_ring + qr.stage * q_bytes, 16);
                const uint32_t d = tmem + (buf * m_step + m - m0) * n_acc;
                uint32_t acc = s != sa;
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                  for (int k = 0; k < 4; ++k) {
                    for (int i = 0; i < n_rep; ++i) {
                      tc_mma_cta(d + i * rep_acc, a_lo + j * 64 + k * 2, desc_hi(2048, true), b_lo + (j * NT + i) * (np * 8) + k * 2, desc_hi(1024, true), idesc, acc);
                      if (rep_acc == 0) acc = 1u;
                    }
                    acc = 1u;
                  }
                tc_commit_cta(empty0 + xr.stage * 8);
                if (m == m1 - 1) tc_commit_cta(q_empty0 + qr.stage * 8);
              }
              __syncwarp();
              xr.step(nx);
            }
            qr.step(nq);
          }
          if (ok && elect_one()) tc_commit_cta(smem_u32(&aux.acc_full[buf]));
          __syncwarp();
        } else {
          const int quarter = warp & 3;
          if (!mbar_wait_warp(smem_u32(&aux.acc_full[buf]), use & 1u, abort_flag, p.status, 4, lane)) { ok = false; break; }
          tc_fence_after();
          float* dst = p.scores + (int64_t)(t + piece) * p.heads * kTile;
          if (quarter == 0 && lane == 0) {
            if (sa == 0) p.tile_pieces[t].x = piece;
            if (sb == steps) p.tile_pieces[t].y = piece;
          }
          for (int m = m0; m < m1; ++m)
            for (int h0 = 0; h0 < np; h0 += 16) {
              const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + (buf * m_step + m - m0) * n_acc + h0;
              uint32_t v[NT][16];
              tmem_ld16(at, v[0]);
              if (own_acc) {
#pragma unroll
                for (int i = 1; i < NT; ++i) tmem_ld16(at + i * np, v[i]);
              }
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (h0 + j < p.heads)
                  dst[(int64_t)(h0 + j) * kTile + m * 128 + quarter * 32 + lane] = own_acc ? add_terms(v, j) : __uint_as_float(v[0][j]);
            }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_addr(smem_u32(&aux.acc_empty[buf]));
        }
      }
    }
  }
  if (!ok) drain();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_free(tmem, tmem_cols); }
  chain_wait();
}

// ---- columns of the weighted sums ---------------------------------------------------
// Where an item's accumulators lie in its half of the tensor memory.  The cache blocks take turns among n_hi accumulators for the
// first terms; the rests have theirs.  STACKED: several terms of a block are columns of one instruction's B operand, so that X is read from
// shared memory once for them (an M128 K16 instruction takes (4096 + 32 N) / 128 cycles: two for the 48 padded heads of an
// OPT-13B layer 88, one 56).  A column block then has [first 0 | rests | first 1 | first 2 | first 3]: blocks of turn 0 write
// the first two, blocks of turn 1 the next two with the weights' terms in the order (rests, first); turns 2 and 3 take an
// instruction for the first term and one for the rests.  Not stacked: an instruction per term, all rests in one accumulator.
// Stacked where as many first accumulators fit as without and slices of two column blocks remain (a slice of one reads the
// weights twice as often): sums in bf16 of 128 OPT-13B requests 216 us not stacked, 249 in stacked slices of one.
struct SumColumns {
  bool stacked;
  uint32_t n_hi, col, set, rest;   // columns from a column block, a first accumulator (not stacked), the first terms to the next / the rests'
  int rests;                       // accumulators of the rests
  __host__ __device__ static uint32_t turns(int np, int slice) { return 5 * slice * np <= 256 ? 4 : 3 * slice * np <= 256 ? 2 : 1; }
  __host__ __device__ static bool fits(int terms, int np, int slice) {
    return stacked_terms(terms, np) && (terms - 1 + turns(np, slice)) * slice * np <= 256;
  }
  __host__ __device__ static bool stack(int terms, int np) { return fits(terms, np, 1) && (fits(terms, np, 2) || 4 * np > 256); }
  __host__ __device__ SumColumns(int terms, int np, int slice) {
    n_hi = turns(np, slice);
    stacked = stack(terms, np) && fits(terms, np, slice);
    if (stacked) {
      col = (terms - 1 + n_hi) * np; set = 0; rest = np; rests = terms - 1;
    } else {
      col = np; set = slice * np; rests = 2 * slice * np <= 256 ? 1 : 0; rest = rests ? n_hi * set : 0;
    }
  }
  // stacked: the k-th accumulator of a column block that has `used` first ones: those, then the rests'
  __device__ __forceinline__ uint32_t at(int k, int used, int terms, int np) const {
    return k >= used ? rest + (k - used) * np : k == 0 ? 0u : (uint32_t)((terms - 1 + k) * np);
  }
  // The weights of the request's block b have the first term last where b & turn_mask() is 1.
  __host__ __device__ int turn_mask() const { return stacked ? (int)n_hi - 1 : 0; }
};

// ---- softmax ------------------------------------------------------------------------
// One CTA per (request, two heads) at a time, one warp per tile.  A lane takes eight consecutive tokens of the
// tile for both heads: it adds the tile's partial sums, and after the maxima are known writes the eight weights of each
// term and head as one 16-byte piece of the sum kernel's B operand, the two heads' pieces together as one 32-byte sector.
// The scores of kHold tiles per warp stay in registers (2048 tokens); those of longer requests are added up twice.
// What bounds it is the chain of round trips of a unit (plan, pieces, scores, two reductions): two heads share it
// and the address arithmetic, and which pieces have a part of a tile is left there by the scores kernel (finding it from the
// cut's formula took two 64-bit divisions per tile).  A batch of no more than two (request, head) per SM takes single
// heads (one OPT-13B request 7.7 -> 6.1).  26.5 -> 17.3 us for 128 OPT-13B requests, 31.5 -> 22.5 in bf16, 14.0 -> 11.6 for 24 of 1800 tokens.
constexpr int kSoftmaxWarps = 4;
constexpr int kHold = 2;

template <typename T, int PER>
__device__ __forceinline__ void softmax_units(const Params& p, float (*s_max)[kSoftmaxWarps], float (*s_sum)[kSoftmaxWarps]) {
  constexpr int NT = kTerms<T>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const GroupPlan* gp = p.plan;
  const int units_of = (p.heads + PER - 1) / PER, n_units = gp->n * units_of, n_pieces = gp->levels * gp->per_level;
  T* probs = static_cast<T*>(p.probs);
  for (int unit = blockIdx.x; unit < n_units; unit += gridDim.x) {
    const int slot = unit / units_of, h = (unit - slot * units_of) * PER;
    const bool two = PER == 2 && h + 1 < p.heads;
    const int len = gp->len[slot];
    const int tile0 = gp->tile_off[slot], n_tiles = gp->tile_off[slot + 1] - tile0;
    const float* scales = p.qscale + (int64_t)gp->ord[slot] * p.heads + h;
    const float scale[2] = {scales[0], two ? scales[1] : 0.f};
    const int n_blk = (len + 15) / 16, blk0 = gp->blk_off[slot];
    // scores of this lane's eight tokens of tile k
    auto load = [&](int k, float (&s)[PER][8]) {
      const int2 c = clamp_pieces(p.tile_pieces[tile0 + k], n_pieces);   // the first and the last piece with a part of the tile
#pragma unroll
      for (int i = 0; i < PER; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) s[i][e] = 0.f;
      const float4* src = reinterpret_cast<const float4*>(p.scores + ((int64_t)(tile0 + k + c.x) * p.heads + h) * kTile + lane * 8);
#pragma unroll (4 / PER)
      for (int j = c.x; j <= c.y; ++j) {
        float4 x[PER], y[PER];
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const bool in = i == 0 || two;
          x[i] = in ? src[i * (kTile / 4)] : make_float4(0.f, 0.f, 0.f, 0.f);
          y[i] = in ? src[i * (kTile / 4) + 1] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        src += p.heads * (kTile / 4);
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          s[i][0] += x[i].x; s[i][1] += x[i].y; s[i][2] += x[i].z; s[i][3] += x[i].w;
          s[i][4] += y[i].x; s[i][5] += y[i].y; s[i][6] += y[i].z; s[i][7] += y[i].w;
        }
      }
      const int tok = k * kTile + lane * 8;
#pragma unroll
      for (int i = 0; i < PER; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) s[i][e] = tok + e < len ? s[i][e] * scale[i] : -INFINITY;
    };
    float held[kHold][PER][8], mx[2] = {-INFINITY, -INFINITY};
    auto take_max = [&](const float (&s)[PER][8]) {
#pragma unroll
      for (int i = 0; i < PER; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) mx[i] = fmaxf(mx[i], s[i][e]);
    };
#pragma unroll
    for (int j = 0; j < kHold; ++j) {
      const int k = warp + j * kSoftmaxWarps;
      if (k < n_tiles) { load(k, held[j]); take_max(held[j]); }
    }
    for (int k = warp + kHold * kSoftmaxWarps; k < n_tiles; k += kSoftmaxWarps) {
      float s[PER][8];
      load(k, s);
      take_max(s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], o));
      mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], o));
    }
    if (lane < 2) s_max[lane][warp] = lane == 0 ? mx[0] : mx[1];
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kSoftmaxWarps; ++w) { mx[0] = fmaxf(mx[0], s_max[0][w]); mx[1] = fmaxf(mx[1], s_max[1][w]); }
    float sum[2] = {0.f, 0.f};
    auto store = [&](int k, const float (&s)[PER][8]) {
      T terms[PER][8][NT];
#pragma unroll
      for (int i = 0; i < PER; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float w = exp2f(s[i][e] - mx[i] + kProbShift);
          sum[i] += w;
          split_terms<T, false>(w, terms[i][e]);
        }
      const int blk = k * kSubs + (lane >> 1);
      if (blk < n_blk) {
        // A tile begins with a block of turn 0.  The mask lies beside what was read of the plan first (in the L1), and is read here
        // for want of registers.
        int turns;
        asm volatile("ld.global.ca.s32 %0, [%1];" : "=r"(turns) : "l"(&gp->turns));
        const bool turned = (lane >> 1 & turns) == 1;
        T* at = probs + ((int64_t)((blk0 + blk) * 2 + (lane & 1)) * NT * p.np + h) * 8;   // 32-byte aligned: np and h are even
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          uint32_t v[2][4] = {};
#pragma unroll
          for (int i = 0; i < PER; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) v[i][e] = pack_pair<T>(terms[i][2 * e][t], terms[i][2 * e + 1][t]);
          T* dst = at + (t == 0 ? (turned ? NT - 1 : 0) : turned ? t - 1 : t) * p.np * 8;
          if (two)
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(v[0][0]), "r"(v[0][1]), "r"(v[0][2]),
                         "r"(v[0][3]), "r"(v[1][0]), "r"(v[1][1]), "r"(v[1][2]), "r"(v[1][3]) : "memory");
          else
            *reinterpret_cast<uint4*>(dst) = make_uint4(v[0][0], v[0][1], v[0][2], v[0][3]);
        }
      }
    };
#pragma unroll
    for (int j = 0; j < kHold; ++j) {
      const int k = warp + j * kSoftmaxWarps;
      if (k < n_tiles) store(k, held[j]);
    }
    for (int k = warp + kHold * kSoftmaxWarps; k < n_tiles; k += kSoftmaxWarps) {
      float s[PER][8];
      load(k, s);
      store(k, s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], o);
      sum[1] += __shfl_xor_sync(0xffffffffu, sum[1], o);
    }
    if (lane < 2) s_sum[lane][warp] = lane == 0 ? sum[0] : sum[1];
    __syncthreads();
    if (threadIdx.x < (two ? 2 : 1)) {
      float total = 0.f;
#pragma unroll
      for (int w = 0; w < kSoftmaxWarps; ++w) total += s_sum[threadIdx.x][w];
      p.inv_sum[(int64_t)slot * p.heads + h + threadIdx.x] = 1.f / total;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kSoftmaxWarps * 32, kTerms<T> == 2 ? 6 : 5)
softmax_kernel(const Params p) {
  __shared__ float s_max[2][kSoftmaxWarps], s_sum[2][kSoftmaxWarps];
  chain_wait();
  chain_next();
  if (p.plan->n * p.heads <= 2 * p.grid_scores) softmax_units<T, 1>(p, s_max, s_sum);
  else softmax_units<T, 2>(p, s_max, s_sum);
}

// ---- weighted sums ------------------------------------------------------------------
// D[column of E][head] = sum_t x_t[column] p[t][head]: work item = (request, slice of up to kMaxSlice x 128
// columns), the item's accumulators together in half of the tensor memory, so that the epilogue of one item
// overlaps the next one's main loop.  Items in order of their length, longest first, handed out by a counter:
// the copying warp takes the next one when it has requested all of its item and passes it to the other warps.
// A stage holds two cache blocks of 16 tokens, four for slices of one or two column blocks (a stage costs 0.35 us of
// waits and commits whatever its size: sums of 34 OPT-1.3B requests 36 -> 29 us, of 8 long OPT-13B requests 54 -> 41, of
// one 12.9 -> 11.0): per cache block and 128 columns one box of (64 columns, 16 rows, 2) =
// an MN-major A operand, and the block's weights (one bulk copy, already in the layout of an unswizzled
// K-major B operand).  The rows of a CTA's first stages are requested while the softmax kernel is still running: what a
// kernel may read before chain_wait() is what was complete when the one before it called chain_next(), here all up
// to the scores.  Warps: 0 takes the items and copies, 1 MMA issue, 2-9 (2-5) epilogue, the one behind them copies: the two take
// turns at the stages, since one warp spends as long on a stage's wait and boxes as the stage takes to arrive (128 OPT-13B
// requests 187 -> 183 us, 24 long ones 69 -> 67.5).  Two producers that take turns need at least as many stages: a stage is then
// never two rounds behind the one that waits for it.  The columns of the accumulators and how many terms an instruction takes: SumColumns.
// With both: 128 OPT-13B requests of 740 tokens 187 -> 172 us, 24 of 1800 69 -> 63, 8 of 1500 41 -> 34, 52 OPT-66B tp 8 requests 171 -> 146,
// 34 OPT-1.3B 31 -> 25, 100 OPT-66B tp 2 280 -> 252, 128 OPT-13B in bf16 216 -> 212.
// The tensor cores drop what falls below the accumulator's last place at every instruction, so a sum's error grows with
// the number of instructions that went into one accumulator (terms x cache blocks).  Where few heads leave the
// tensor memory for it, the rests have accumulators of their own and the cache blocks' first terms take turns among two
// or four, added in fp32; slices are narrow enough for the rests'.  Error before the output's rounding, 2048 tokens
// among 150 requests, all terms in one -> this (the re-projection's for comparison): OPT-13B fp16 8.5e-6 -> 4.3e-6
// (6.2e-6), bf16 1.15e-5 -> 3.8e-6 (6.1e-6), OPT-1.3B bf16 7.3e-6 -> 2.8e-6 (3.1e-6); OPT-66B tp 8 bf16, three requests,
// 7.3e-6 -> 2.7e-6 (1.1e-5).  It costs 2 - 3 % of a step of 256 OPT-13B requests (slices of two blocks instead of four), 2 %
// of 128 OPT-66B tp 8 requests, 1 % of 48 OPT-1.3B requests; 24 long OPT-13B requests gain 1 %.
// Two epilogue warps per quarter of the accumulators' lanes take turns at an item's groups of 16 heads and 128 columns, from six
// groups on: with one, an item of a short request (300 tokens) takes as long to be split into terms and written as to be read.
// 64 OPT-13B requests of 340 tokens 77 -> 65 us, 128 of 740 198 -> 191, in bf16 228 -> 217; with fewer groups the second warp
// costs more than it takes over (52 OPT-66B tp 8 requests, four groups, 170 -> 175; 8 long OPT-13B requests, three, 40 -> 43).
constexpr int kSumThreads = 352;
// Given to the kernel as a value: compiled in, the loops over the stages come out longer and short requests wait for them
// (32 OPT-66B tp 8 requests of 60 tokens 22.5 -> 26 us).
constexpr int kSumCopiers = 2;
// Where no item of the batch can have six, the kernel is launched without the second ones: their registers keep its CTAs from
// starting beside the softmax's.
__host__ __device__ inline int sum_epilogue_warps(int slice, int np) { return slice * np >= 96 ? 8 : 4; }

__host__ __device__ inline uint32_t probs_block_bytes(int terms, int np) { return (uint32_t)terms * np * 32; }
__host__ __device__ inline int sum_stage_blocks(int terms, int np, int slice) {
  return slice <= 2 && 3 * 4 * (slice * 4096 + probs_block_bytes(terms, np)) <= kRingBytes ? 4 : 2;   // three stages at least
}
__host__ __device__ inline uint32_t sum_stage_bytes(int terms, int np, int slice) {
  const uint32_t blocks = sum_stage_blocks(terms, np, slice);
  return blocks * slice * 4096 + ((blocks * probs_block_bytes(terms, np) + 1023) & ~1023u);
}

template <typename T, bool STACKED>
__global__ void __launch_bounds__(kSumThreads, 1)
sum_kernel(const __grid_constant__ CUtensorMap map_x, const Params p) {
  constexpr int NT = kTerms<T>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t ring = (smem_u32(smem_raw) + 1023) & ~1023u;
  __shared__ RingAux aux;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  __shared__ ItemRing items;
  GroupPlan* gp = p.plan;
  const int n = gp->n;
  if (n == 0) { chain_wait(); return; }
  const int np = p.np, e_blocks = p.hidden / 128, slice = gp->slice;
  const int n_slices = (e_blocks + slice - 1) / slice, n_items = n * n_slices;
  if ((int)blockIdx.x >= n_items) { chain_wait(); return; }
  const uint32_t pblk = probs_block_bytes(NT, np), per_stage = sum_stage_blocks(NT, np, slice), x_bytes = per_stage * slice * 4096,
                 stage_bytes = sum_stage_bytes(NT, np, slice);
  const int stages = min(kMaxStages, (int)(kRingBytes / stage_bytes));
  const SumColumns cols(NT, np, slice);
  const int n_epilogue = sum_epilogue_warps(slice, np);   // the others only wait
  const int n_copiers = p.sum_copiers;
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { mbar_init(&aux.full[s], 1); mbar_init(&aux.empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&aux.acc_full[b], 1); mbar_init(&aux.acc_empty[b], n_epilogue); }
    for (int i = 0; i < kItemSlots; ++i) { mbar_init(&items.full[i], 1); mbar_init(&items.empty[i], n_copiers + n_epilogue); }
    aux.abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(&aux.tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_next();
  const uint32_t tmem = aux.tmem_base;
  volatile int* abort_flag = &aux.abort_flag;
  const uint32_t full0 = smem_u32(&aux.full[0]), empty0 = smem_u32(&aux.empty[0]);
  bool ok = true;
  Ring rg;
  uint32_t n_local = 0;
  Ring ir;
  int next = blockIdx.x;   // the first item needs no counter
  const uint64_t once = l2_policy_evict_first();
  int ahead = 0;           // stages of the first item whose rows are requested before the wait
  const int copier = warp == 0 ? 0 : n_copiers == 2 && warp == 2 + n_epilogue ? 1 : -1;   // the two take turns at the stages
  uint32_t n_stage = 0;    // of all items so far
  bool waited = copier < 0;
  if (waited) chain_wait();
  while (ok && warp < 1 + n_copiers + n_epilogue) {
    int item;
    if (warp == 0) {
      item = next;
      if (!mbar_wait_warp(smem_u32(&items.empty[ir.stage]), ir.phase ^ 1u, abort_flag, p.status, 1, lane)) { ok = false; break; }
      if (lane == 0) {
        items.item[ir.stage] = item;
        mbar_arrive_addr(smem_u32(&items.full[ir.stage]));
      }
    } else {
      if (!mbar_wait_warp(smem_u32(&items.full[ir.stage]), ir.phase, abort_flag, p.status, 6, lane)) { ok = false; break; }
      item = items.item[ir.stage];
      __syncwarp();
      if (lane == 0) mbar_arrive_addr(smem_u32(&items.empty[ir.stage]));
    }
    ir.step(kItemSlots);
    if (item >= n_items) break;
    if (warp == 0) {
      if (lane == 0) next = (int)gridDim.x + atomicAdd(&gp->next_item, 1);
      next = __shfl_sync(0xffffffffu, next, 0);
    }
    const int slot = item / n_slices, first = (item % n_slices) * slice;
    const int len = gp->len[slot];
    if (len <= 0) {
      if (!waited) { chain_wait(); waited = true; }
      continue;
    }
    const int n_col = min(slice, e_blocks - first);   // 128-column blocks of this item
    const int n_blk = (len + 15) >> 4;
    const uint32_t buf = n_local & 1u, use = n_local >> 1;
    ++n_local;
    if (copier >= 0) {
      const int32_t* bt = p.block_tables + (int64_t)gp->req[slot] * p.max_blocks;
      const char* probs = static_cast<const char*>(p.probs) + (int64_t)gp->blk_off[slot] * pblk;
      int rows = 0;
      auto request_rows = [&](int b, uint32_t stage, bool mine) {   // the stage's byte count, then the rows of the blocks from b on
        if ((b & 31) == 0) {   // first cache rows of the next 32 blocks
          const int tok = (b + lane) * 16;
          rows = b + lane < n_blk ? bt[tok / p.block_size] * p.block_size + tok % p.block_size : 0;
        }
        if (!mine) return;
        const int nb = min((int)per_stage, n_blk - b);
        const uint32_t bar = full0 + stage * 8, dst = ring + stage * stage_bytes;
        if (lane == 0) mbar_expect_tx_addr(bar, (uint32_t)nb * (n_col * 4096 + pblk));
        __syncwarp();
        const int k = lane / n_col, col = lane - k * n_col;
        const int row = __shfl_sync(0xffffffffu, rows, ((b & 31) + k) & 31);
        if (lane < nb * n_col) tma_load_3d_hint(dst + (k * slice + col) * 4096, &map_x, bar, 0, row, (first + col) * 2, once);
      };
      if (!waited) {
        ahead = min(min(stages, 32 / (int)per_stage), (n_blk + (int)per_stage - 1) / (int)per_stage);   // `rows` holds 32 blocks
#pragma unroll 1
        for (int i = 0; i < ahead; ++i) request_rows(i * (int)per_stage, i, (i & (n_copiers - 1)) == copier);
        chain_wait();
        waited = true;
      }
#pragma unroll 1
      for (int b = 0; b < n_blk; b += (int)per_stage) {
        const int nb = min((int)per_stage, n_blk - b);
        const bool mine = (int)(n_stage++ & (uint32_t)(n_copiers - 1)) == copier;
        if (ahead > 0) {
          --ahead;
        } else {
          if (mine && !mbar_wait_warp(empty0 + rg.stage * 8, rg.phase ^ 1u, abort_flag, p.status, 1, lane)) { ok = false; break; }
          request_rows(b, rg.stage, mine);
        }
        const uint32_t bar = full0 + rg.stage * 8, dst = ring + rg.stage * stage_bytes;
        if (mine && lane == 31) bulk_load(dst + x_bytes, probs + (int64_t)b * pblk, nb * pblk, bar);   // blocks lie one behind the other
        __syncwarp();
        rg.step(stages);
      }
    } else if (warp == 1) {
      if (!mbar_wait_warp(smem_u32(&aux.acc_empty[buf]), (use & 1u) ^ 1u, abort_flag, p.status, 2, lane)) { ok = false; break; }
      tc_fence_after();
      const uint32_t idesc = mma_idesc(kFmt<T>, 128, (uint32_t)np, true), idesc_rests = mma_idesc(kFmt<T>, 128, (uint32_t)((NT - 1) * np), true),
                     idesc_all = mma_idesc(kFmt<T>, 128, (uint32_t)(STACKED ? NT * np : np), true);
      const uint32_t mask = cols.n_hi - 1, d0 = tmem + buf * 256;
      for (int b = 0; b < n_blk; b += (int)per_stage) {
        const int nb = min((int)per_stage, n_blk - b);
        if (!mbar_wait_warp(full0 + rg.stage * 8, rg.phase, abort_flag, p.status, 3, lane)) { ok = false; break; }
        const uint32_t x_at = ring + rg.stage * stage_bytes, p_at = x_at + x_bytes;
        const int valid = len - (b + nb - 1) * 16;   // tokens of the stage's last block
        if (valid < 16) {
          // rows past the sequence length hold whatever the cache block holds; their weights are zero,
          // but zero times NaN is not
          const uint32_t at = x_at + (nb - 1) * slice * 4096 + ((lane >> 3) & 1) * 2048 + (lane & 7) * 16;
          for (int col = 0; col < n_col; ++col)
            for (int r = valid + (lane >> 4); r < 16; r += 2)
              asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(at + col * 4096 + r * 128), "r"(0u) : "memory");
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
        }
        tc_fence_after();
        if (elect_one()) {
          const uint32_t x_lo = desc_lo(x_at, 2048), p_lo = desc_lo(p_at, (uint32_t)(NT * np * 16)), x_step = slice * 256, p_step = pblk >> 4;
          auto mma = [&](uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t what, uint32_t acc) {
            tc_mma_cta(d, a_lo, desc_hi(1024, true), b_lo, desc_hi(128, false), what, acc);
          };
          if constexpr (!STACKED) {
            for (int k = 0; k < nb; ++k) {
              const uint32_t turn = (uint32_t)(b + k) & mask, later = (uint32_t)(b + k) > mask;   // later: the turn's accumulator holds a sum
              for (int col = 0; col < n_col; ++col)
#pragma unroll
                for (int i = 0; i < NT; ++i)
                  mma(d0 + (i == 0 ? turn * cols.set : cols.rest) + col * np, x_lo + k * x_step + col * 256, p_lo + k * p_step + i * np, idesc,
                      i == 0 ? later : i > 1 || cols.rests == 0 || b + k > 0);
            }
          } else if (mask == 0) {
            for (int k = 0; k < nb; ++k)
#pragma unroll
              for (int col = 0; col < kMaxSlice; ++col) {
                if (col >= n_col) break;
                mma(d0 + col * cols.col, x_lo + k * x_step + col * 256, p_lo + k * p_step, idesc_all, b + k > 0);
              }
          } else if ((b & mask) != 0) {   // stages of two blocks, turns 2 and 3
            for (int k = 0; k < nb; ++k)
              for (int col = 0; col < n_col; ++col) {
                mma(d0 + (NT + 1 + k) * np + col * cols.col, x_lo + k * x_step + col * 256, p_lo + k * p_step, idesc, b > 2);
                mma(d0 + np + col * cols.col, x_lo + k * x_step + col * 256, p_lo + k * p_step + np, idesc_rests, 1u);
              }
          } else {
            // from turn 0 on, in straight line: with a loop that looks at every block's turn the issuing thread was what the kernel waited for
            const uint32_t d_hi = d0 + (NT - 1) * np, later = b > 0;
            for (int col = 0; col < n_col; ++col) {
              const uint32_t at = col * cols.col, x = x_lo + col * 256;
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                if (k >= nb) break;
                const uint32_t xk = x + k * x_step, pk = p_lo + k * p_step;
                if (k == 0 || (k == 2 && mask == 1)) {
                  mma(d0 + at, xk, pk, idesc_all, k == 2 ? 1u : later);
                } else if (k == 1 || (k == 3 && mask == 1)) {
                  if (k == 3 || later) {
                    mma(d0 + np + at, xk, pk, idesc_all, 1u);
                  } else {
                    mma(d0 + np + at, xk, pk, idesc_rests, 1u);
                    mma(d_hi + np + at, xk, pk + (NT - 1) * np, idesc, 0u);
                  }
                } else {
                  mma(d_hi + k * np + at, xk, pk, idesc, later);
                  mma(d0 + np + at, xk, pk + np, idesc_rests, 1u);
                }
              }
            }
          }
          tc_commit_cta(empty0 + rg.stage * 8);
        }
        __syncwarp();
        rg.step(stages);
      }
      if (ok && elect_one()) tc_commit_cta(smem_u32(&aux.acc_full[buf]));
      __syncwarp();
    } else {
      const int quarter = warp & 3, turn = (warp - 2) >> 2;
      const float* inv = p.inv_sum + (int64_t)slot * p.heads;
      T* z = static_cast<T*>(p.z);
      if (!mbar_wait_warp(smem_u32(&aux.acc_full[buf]), use & 1u, abort_flag, p.status, 4, lane)) { ok = false; break; }
      tc_fence_after();
      const int used = (int)min(cols.n_hi, (uint32_t)n_blk), n_in = used + cols.rests;
      // accumulators of a column block: four first terms' and the rests'; that many read together (142 - 144 registers; one after the other,
      // in 128, short requests' items wait for it: 16 OPT-13B requests of 60 tokens 16.5 -> 19 us).  Not stacked, where one set of rests
      // is all there is, four accumulators at even distances and no table of them: bf16, 91 OPT-13B requests of 71 tokens 71.5 -> 67.8,
      // 60 of 200 61.4 -> 59, 128 of 400 73.7 -> 71.9
      constexpr int kMost = NT + 3, kAtOnce = 6 - NT;
      uint32_t off[kMost];
#pragma unroll
      for (int k = 1; STACKED && k < kMost; ++k) off[k] = cols.at(k, used, NT, np);
      const int h_steps = np / 16;
      for (int it = turn; it < n_col * h_steps; it += n_epilogue / 4) {
        const int col = it / h_steps, h0 = (it - col * h_steps) * 16;
        const int e = (first + col) * 128 + quarter * 32 + lane;
        uint32_t v[16];
        const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + buf * 256 + col * cols.col + h0;
        tmem_ld16(at, v);
        if constexpr (STACKED) {
#pragma unroll
          for (int k0 = 1; k0 < kMost; k0 += kAtOnce) {
            if (k0 > 1 && k0 >= n_in) break;
            uint32_t more[kAtOnce][16];
#pragma unroll
            for (int k = k0; k < k0 + kAtOnce && k < kMost; ++k)
              if (k < n_in) tmem_ld16(at + off[k], more[k - k0]);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              float x = __uint_as_float(v[j]);
#pragma unroll
              for (int k = k0; k < k0 + kAtOnce && k < kMost; ++k)
                if (k < n_in) x += __uint_as_float(more[k - k0][j]);
              v[j] = __float_as_uint(x);
            }
          }
        } else {
          uint32_t more[3][16], rest[16];
#pragma unroll
          for (int i = 0; i < 3; ++i)
            if (i + 1 < used) tmem_ld16(at + (i + 1) * cols.set, more[i]);
          if (cols.rests != 0) tmem_ld16(at + cols.rest, rest);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            float x = __uint_as_float(v[j]);
#pragma unroll
            for (int i = 0; i < 3; ++i)
              if (i + 1 < used) x += __uint_as_float(more[i][j]);
            if (cols.rests != 0) x += __uint_as_float(rest[j]);
            v[j] = __float_as_uint(x);
          }
        }
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          float2 f = pair_rows(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), lane);
          const int h = h0 + j + (lane & 1);
          if (h < p.heads) {
            const float w = inv[h];
            T a[NT], b[NT];
            split_terms<T, true>(f.x * w, a);
            split_terms<T, true>(f.y * w, b);
#pragma unroll
            for (int t = 0; t < NT; ++t)
              *reinterpret_cast<uint32_t*>(z + (((int64_t)t * p.heads + h) * p.n_cap + slot) * p.hidden + (e & ~1)) = pack_pair<T>(a[t], b[t]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_addr(smem_u32(&aux.acc_empty[buf]));
    }
  }
  if (!ok) drain();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_free(tmem, 512); }
}

// ---- unfold -------------------------------------------------------------------------
// D[row of W_v][request] = sum_e W_v[row][e] z[request][head of the row][e]: one CTA per (128 rows of W_v,
// range of E, 128 / HT requests), HT = 128 / D heads per 128 rows.  Rows of every head are multiplied with
// every one of the HT heads' z and the epilogue keeps the matching quarter (half): for D = 128 nothing
// is wasted.  The first term and the rests have accumulators of their own (see SumColumns); where few enough requests leave
// the columns, all terms and heads are columns of one instruction (one OPT-13B request 11.1 -> 10.2 us with the rows below, 16 OPT-125M
// in bf16 5.2 -> 4.3).  Partial sums over the
// ranges of E are added by the combine kernel.
constexpr int kUnfoldThreads = 192;

// A stage: 64 columns of 128 rows of W_v and of z in boxes of 16 requests, so that few requests leave room for more
// stages.
__host__ __device__ inline uint32_t unfold_stage_bytes(int z_boxes) { return 16384u + (uint32_t)z_boxes * 2048u; }

template <typename T, int D>
__global__ void __launch_bounds__(kUnfoldThreads, 1)
unfold_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_z, const Params p) {
  constexpr int NT = kTerms<T>, HT = 128 / D, NC = 128 / HT;   // NC: requests per CTA
  constexpr uint32_t kRestAcc = 128, kCols = 256;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t ring = (smem_u32(smem_raw) + 1023) & ~1023u;
  __shared__ RingAux aux;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int n = p.plan->n, r0 = blockIdx.z * NC;
  if (r0 >= n) { chain_wait(); return; }
  const int m = min(NC, n - r0), boxes = (m + 15) / 16;
  const uint32_t z_head = boxes * 2048;   // bytes of one (term, head) slab
  const bool stacked = NT * HT * boxes * 16 <= 256;   // their rows lie one behind the other: all as columns of one instruction
  const int head0 = blockIdx.x * HT, n_heads = min(HT, p.heads - head0);
  const int sa = (int)((int64_t)p.slabs * blockIdx.y / gridDim.y), sb = (int)((int64_t)p.slabs * (blockIdx.y + 1) / gridDim.y);
  const uint32_t stage_bytes = unfold_stage_bytes(NT * HT * boxes);
  const int stages = min(kMaxStages, (int)(p.unfold_ring / stage_bytes));
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { mbar_init(&aux.full[s], 1); mbar_init(&aux.empty[s], 1); }
    mbar_init(&aux.acc_full[0], 1);
    aux.abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(&aux.tmem_base, kCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_next();
  const uint32_t tmem = aux.tmem_base;
  volatile int* abort_flag = &aux.abort_flag;
  const uint32_t full0 = smem_u32(&aux.full[0]), empty0 = smem_u32(&aux.empty[0]);
  bool ok = true;
  Ring rg;
  if (warp == 0) {
    const int n_boxes = NT * n_heads * boxes;
    auto request_w = [&](int s, uint32_t stage) {
      const uint32_t bar = full0 + stage * 8;
      if (lane == 0) {
        mbar_expect_tx_addr(bar, (uint32_t)p.w_box_rows * 128 + (uint32_t)n_boxes * 2048);
        tma_load_2d_cta(ring + stage * stage_bytes, &map_w, bar, s * 64, head0 * D);
      }
      __syncwarp();
    };
    // the first stages' rows of W_v are requested while the sum kernel is still running, z once it is complete
    int ahead = min(stages, sb - sa);
    for (int i = 0; i < ahead; ++i) request_w(sa + i, i);
    // and the other rows of the range as far as L2, where the sum kernel's items leave SMs idle (one OPT-13B request 11.1 -> 10.7 us; with more
    // items the rows that it still waits for come later: its 576 for 32 OPT-66B tp 8 requests of 60 tokens 22.7 -> 25.9)
    const int slice = p.plan->slice;
    if (n * ((p.slabs / 2 + slice - 1) / slice) <= p.grid_scores)
      for (int s = sa + ahead + lane; s < sb; s += 32) tma_prefetch_2d(&map_w, s * 64, head0 * D);
    __syncwarp();
    chain_wait();
    for (int s = sa; s < sb; ++s) {
      if (ahead > 0) {
        --ahead;
      } else {
        if (!mbar_wait_warp(empty0 + rg.stage * 8, rg.phase ^ 1u, abort_flag, p.status, 1, lane)) { ok = false; break; }
        request_w(s, rg.stage);
      }
      const uint32_t bar = full0 + rg.stage * 8, dst = ring + rg.stage * stage_bytes;
      for (int i = lane; i < n_boxes; i += 32) {   // i = (term, head, box of 16 requests)
        const int b = i % boxes, hh = (i / boxes) % n_heads, t = i / (boxes * n_heads);
        tma_load_2d_cta(dst + 16384 + (t * HT + hh) * z_head + b * 2048, &map_z, bar, s * 64,
                        (t * p.heads + head0 + hh) * p.n_cap + r0 + b * 16);
      }
      __syncwarp();
      rg.step(stages);
    }
  } else if (warp == 1) {
    const uint32_t idesc = mma_idesc(kFmt<T>, 128, (uint32_t)(stacked ? NT * HT * boxes * 16 : boxes * 16), false);
    uint32_t acc = 0;
    for (int s = sa; s < sb; ++s) {
      if (!mbar_wait_warp(full0 + rg.stage * 8, rg.phase, abort_flag, p.status, 3, lane)) { ok = false; break; }
      tc_fence_after();
      if (elect_one()) {
        const uint32_t a_lo = desc_lo(ring + rg.stage * stage_bytes, 16), b_lo = a_lo + (16384 >> 4);
        if (stacked) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            tc_mma_cta(tmem, a_lo + k * 2, desc_hi(1024, true), b_lo + k * 2, desc_hi(1024, true), idesc, k > 0 ? 1u : acc);
        } else for (int hh = 0; hh < n_heads; ++hh) {
          uint32_t first = acc;
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int t = 0; t < NT; ++t) {
              tc_mma_cta(tmem + (t == 0 ? 0 : kRestAcc) + hh * NC, a_lo + k * 2, desc_hi(1024, true), b_lo + (t * HT + hh) * (z_head >> 4) + k * 2,
                         desc_hi(1024, true), idesc, first);
              if (t > 0) first = 1u;
            }
        }
        tc_commit_cta(empty0 + rg.stage * 8);
      }
      __syncwarp();
      acc = 1u;
      rg.step(stages);
    }
    if (ok && elect_one()) tc_commit_cta(smem_u32(&aux.acc_full[0]));
    __syncwarp();
  } else {
    const int quarter = warp & 3;
    ok = mbar_wait_warp(smem_u32(&aux.acc_full[0]), 0, abort_flag, p.status, 4, lane);
    if (ok) {
      tc_fence_after();
      const int row = quarter * 32 + lane, hh = row / D;
      if (hh < n_heads) {   // uniform in a warp: D is 32, 64 or 128
        const int width = p.heads * D;
        float* dst = p.out_part + ((int64_t)blockIdx.y * p.n_hidden_cap + p.group_first + r0) * width + head0 * D + row;
        for (int c = 0; c < m; c += 16) {
          uint32_t v[16], rest[16], last[16];
          const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + (stacked ? hh * boxes * 16 : hh * NC) + c;
          tmem_ld16(at, v);
          tmem_ld16(at + (stacked ? HT * boxes * 16 : (int)kRestAcc), rest);
          if (NT == 3 && stacked) tmem_ld16(at + 2 * HT * boxes * 16, last);
          tmem_ld_wait();
          if (NT == 3 && stacked) {
#pragma unroll
            for (int j = 0; j < 16; ++j) rest[j] = __float_as_uint(__uint_as_float(rest[j]) + __uint_as_float(last[j]));
          }
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c + j < m) dst[(int64_t)(c + j) * width] = fmaf(__uint_as_float(rest[j]), kRestDown<T>, __uint_as_float(v[j]));
        }
      }
    }
  }
  if (!ok) drain();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_free(tmem, kCols); }
}

// ---- scratch and host side --------------------------------------------------------------
int terms_of(int dtype) { return dtype == APS_BF16 ? 3 : 2; }

struct Layout {
  int np, n_cap, n_groups, n_hidden_cap, splits, max_slice;
  uint32_t unfold_ring;
  size_t off_groups, off_slot, off_list, off_qscale, off_inv, off_scores, off_pieces, off_probs, off_qz, off_part, total;
};

Layout layout_of(int batch, int max_blocks, int block_size, int heads, int head_size, int hidden, int dtype) {
  Layout l;
  const int nt = terms_of(dtype);
  l.np = (heads + 15) / 16 * 16;
  l.n_cap = ((batch < kGroup ? batch : kGroup) + 15) / 16 * 16;
  l.n_groups = (batch + kGroup - 1) / kGroup;
  l.n_hidden_cap = l.n_groups == 1 ? l.n_cap : l.n_groups * kGroup;
  // One wave of unfold CTAs; at least four slabs each.  A CTA spends 0.4 us on a slab whatever its requests, so few
  // requests take two CTAs per SM (half the ring each, three stages at least) and ranges half as long: one OPT-13B
  // request 14.2 -> 11.4 us, 24 requests 15.6 -> 12.3, 64 requests 20.8 -> 17.1.
  const int w_tiles = (heads * head_size + 127) / 128, slabs = hidden / 64, ht = 128 / head_size;
  const int z_boxes = nt * ht * (((batch < head_size ? batch : head_size) + 15) / 16);   // 128 / ht requests per CTA
  const bool two = 3 * unfold_stage_bytes(z_boxes) <= kRingBytes / 2;
  l.unfold_ring = (uint32_t)(two ? kRingBytes / 2 : kRingBytes);
  int splits = (two ? 2 : 1) * sm_count() / w_tiles;
  if (splits > slabs / 4) splits = slabs / 4;
  l.splits = splits < 1 ? 1 : splits;
  int ms = 256 / l.np;
  if (ms > kMaxSlice) ms = kMaxSlice;
  while (ms > 1 && 2 * ms * l.np > 256) --ms;   // room for the rests' accumulators
  if (SumColumns::stack(nt, l.np))
    for (int s = 2; s <= ms; ++s)
      if (!SumColumns::fits(nt, l.np, s)) ms = s - 1;
  while (ms > 1 && 3 * sum_stage_bytes(nt, l.np, ms) > kRingBytes) --ms;   // at least three stages
  l.max_slice = ms;
  const int64_t max_tokens = (int64_t)max_blocks * block_size;
  const int64_t reqs = batch < kGroup ? batch : kGroup, blks = reqs * ((max_tokens + 15) / 16);
  const int64_t all_tiles = reqs * ((max_tokens + kTile - 1) / kTile);
  int64_t tiles = all_tiles;
  const int64_t pieces = (blks + tiles * kTileCost) * (hidden / 128) / kMinPiece;   // none is smaller than kMinPiece
  tiles += pieces < 1 ? 1 : pieces < kMaxPieces ? pieces : kMaxPieces;
  size_t o = 0;
  auto take = [&](size_t bytes) { const size_t at = o; o = align_up(o + bytes, 256); return at; };
  l.off_pieces = take((size_t)all_tiles * sizeof(int2));
  l.off_groups = take((size_t)l.n_groups * sizeof(GroupPlan));
  l.off_slot = take((size_t)batch * sizeof(int));
  l.off_list = take((size_t)batch * sizeof(int2));
  l.off_qscale = take((size_t)l.n_cap * heads * sizeof(float));
  l.off_inv = take((size_t)l.n_cap * heads * sizeof(float));
  l.off_scores = take((size_t)tiles * heads * kTile * sizeof(float));
  l.off_probs = take((size_t)blks * probs_block_bytes(nt, l.np));
  // qt is dead once the scores are there, z is written after them: one buffer
  l.off_qz = take((size_t)l.n_cap * nt * heads * hidden * 2);
  l.off_part = take((size_t)l.splits * l.n_hidden_cap * heads * head_size * sizeof(float));
  l.total = o;
  return l;
}

int map_2d(CUtensorMap* map, const void* base, int dtype, uint64_t cols, uint64_t rows, uint64_t row_stride,
           uint32_t box_rows, const char* what) {
  TensorMapSpec spec{};
  spec.base = base; spec.dtype = dtype; spec.rank = 2;
  spec.dims[0] = cols; spec.dims[1] = rows;
  spec.strides_bytes[0] = row_stride * 2;
  spec.box[0] = 64; spec.box[1] = box_rows;
  return cached_tensor_map(map, spec, what);
}

// Dynamic shared memory above 48 KB has to be allowed once per kernel and device.
template <typename K>
int allow_smem(K kernel, size_t bytes, bool* done) {
  int dev = 0;
  APS_CUDA(cudaGetDevice(&dev));
  APS_REQUIRE(dev >= 0 && dev < 64, APS_ERR_CUDA, "device index %d out of range", dev);
  if (!done[dev]) {
    APS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    done[dev] = true;
  }
  return APS_OK;
}

struct Maps { CUtensorMap x_scores, x_sum, q, wk, wv, z; };

template <typename T, int D>
int launch_group(const Maps& m, Params p, int n_cap, int w_tiles, const HybridCall* kv, const WorkspacePtrs& ws, cudaStream_t stream) {
  const size_t ring = 1024 + kRingBytes;
  const int first = p.group_first == 0 ? 1 : 0;
  int st;
  {
    static bool done[64] = {false};
    constexpr size_t smem = fold_smem<D>();
    auto k = fold_kernel<T, D>;
    if ((st = allow_smem(k, smem, done)) != APS_OK) return st;
    const int blocks = p.hidden / 128, chunks = (n_cap + kFoldReqs - 1) / kFoldReqs;
    int splits = 2 * sm_count() / p.heads;   // one wave at two CTAs per SM when one chunk of requests is in use
    splits = splits < 1 ? 1 : splits > blocks ? blocks : splits;
    if ((st = launch_chained("fold_kernel", k, dim3(splits, p.heads, chunks), kFoldThreads, smem, stream, m.wk, p,
                             first)) != APS_OK) return st;
  }
  // Behind the fold whatever the batch.  Before it, K/V-only steps of more than 700 requests would be 0.5 - 1.3 % faster (their empty
  // fold holds the K/V kernel back: 1100 OPT-1.3B requests 291 -> 287 us, 1500 374 -> 370), but the host does not know the
  // types, and steps with hidden-cached requests would lose what the fold beside the plan gives (400, 30 % of them
  // hidden-cached, 243 -> 249, 700 half 462 -> 471, 1500 half 717 -> 735, all 1061 -> 1091).
  if (kv != nullptr && (st = launch_kv_attention(ws, kv->query, kv->key_cache, kv->value_cache, kv->block_tables, kv->seq_lens,
                                                 kv->shape, stream)) != APS_OK) return st;
  {
    static bool done[64] = {false};
    auto k = scores_kernel<T>;
    if ((st = allow_smem(k, 1024 + kScoresRing, done)) != APS_OK) return st;
    if ((st = launch_chained("scores_kernel", k, p.grid_scores, kScoresThreads, 1024 + kScoresRing, stream, m.x_scores,
                             m.q, p, kv != nullptr ? 1 : 0)) != APS_OK) return st;
  }
  const int units = n_cap * p.heads, resident = sm_count() * 12;
  if ((st = launch_chained("softmax_kernel", softmax_kernel<T>, units < resident ? units : resident, kSoftmaxWarps * 32, 0,
                           stream, p)) != APS_OK) return st;
  {
    static bool done[64] = {false}, done_apart[64] = {false};
    auto k = sum_kernel<T, true>;
    if (!SumColumns::stack(kTerms<T>, p.np)) k = sum_kernel<T, false>;
    if ((st = allow_smem(sum_kernel<T, true>, ring, done)) != APS_OK || (st = allow_smem(sum_kernel<T, false>, ring, done_apart)) != APS_OK)
      return st;
    if ((st = launch_chained("sum_kernel", k, sm_count(), p.sum_threads, ring, stream, m.x_sum, p)) != APS_OK) return st;
  }
  {
    static bool done[64] = {false};
    auto k = unfold_kernel<T, D>;
    if ((st = allow_smem(k, ring, done)) != APS_OK) return st;
    constexpr int kReqs = 128 / (128 / D);
    if ((st = launch_chained("unfold_kernel", k, dim3(w_tiles, p.splits, (n_cap + kReqs - 1) / kReqs), kUnfoldThreads,
                             1024 + p.unfold_ring, stream, m.wv, m.z, p)) != APS_OK) return st;
  }
  return APS_OK;
}

}  // namespace
}  // namespace aps

extern "C" int aps_selftest_tile_pieces(int first, int last, int num_pieces, int* pieces_out) {
  APS_REQUIRE(num_pieces > 0 && num_pieces <= aps::kMaxPieces, APS_ERR_SHAPE, "selftest_tile_pieces: no such number of pieces");
  APS_REQUIRE(pieces_out != nullptr, APS_ERR_NULL_POINTER, "selftest_tile_pieces: null pointer");
  const int2 c = aps::clamp_pieces(make_int2(first, last), num_pieces);
  pieces_out[0] = c.x;
  pieces_out[1] = c.y;
  return APS_OK;
}

namespace aps {

// plan may be NULL: the new-token writes alone.
int launch_step_plan(const PlanArgs* plan, const NewTokenWrite& n, cudaStream_t stream) {
  const int64_t es = dtype_size(n.dtype), row = (int64_t)n.heads * n.head_size;
  const bool kv = n.key != nullptr, hid = n.hidden != nullptr;
  if (plan == nullptr && !kv && !hid) return APS_OK;
  APS_REQUIRE(!kv || (n.value && n.key_cache && n.value_cache), APS_ERR_NULL_POINTER,
              "decode_layer_step: new_key given without new_value / K/V cache");
  APS_REQUIRE(!hid || n.hidden_cache, APS_ERR_NULL_POINTER, "decode_layer_step: hidden_states given without hidden cache");
  auto fits = [](std::initializer_list<const void*> p, std::initializer_list<int64_t> bytes) {
    for (const void* x : p) if (!aligned_to(x, 16)) return false;
    for (int64_t x : bytes) if (x % 16 != 0) return false;
    return true;
  };
  APS_REQUIRE((!kv || fits({n.key, n.value, n.key_cache, n.value_cache}, {row * es, n.key_stride * es, n.value_stride * es, n.block_stride * es})) &&
                  (!hid || fits({n.hidden, n.hidden_cache}, {n.hidden_size * es, n.hidden_stride * es, n.slot_stride * es})),
              APS_ERR_MISALIGNED,
              "decode_layer_step: step inputs and caches must be 16-byte aligned with 16-byte rows and strides");
  StepWrite w{};
  w.hidden = (const char*)n.hidden; w.key = (const char*)n.key; w.value = (const char*)n.value;
  w.key_cache = (char*)n.key_cache; w.value_cache = (char*)n.value_cache; w.hidden_cache = (char*)n.hidden_cache;
  w.block_tables = n.block_tables; w.seq_lens = n.seq_lens; w.cache_type = n.cache_type;
  w.batch = n.batch; w.max_blocks = n.max_blocks_per_seq; w.block_size = n.block_size;
  w.kv_row_bytes = (uint32_t)(row * es); w.hidden_row_bytes = (uint32_t)(n.hidden_size * es);
  w.hidden_stride_b = n.hidden_stride * es; w.key_stride_b = n.key_stride * es; w.value_stride_b = n.value_stride * es;
  w.block_stride_b = n.block_stride * es; w.slot_stride_b = n.slot_stride * es;
  const uint32_t widest = !kv ? w.hidden_row_bytes : !hid ? w.kv_row_bytes : w.kv_row_bytes > w.hidden_row_bytes ? w.kv_row_bytes : w.hidden_row_bytes;
  w.chunks = (int)((widest + kWriteChunk - 1) / kWriteChunk);
  const int64_t jobs = kv || hid ? 2 * (int64_t)n.batch * w.chunks : 0, ctas = (jobs + kPlanThreads / 32 - 1) / (kPlanThreads / 32);
  const int plan_ctas = plan != nullptr ? 1 : 0;
  APS_REQUIRE(ctas + plan_ctas < (int64_t(1) << 31), APS_ERR_SHAPE, "decode_layer_step: batch too large");
  return launch_chained("step_plan_kernel", step_plan_kernel, dim3((unsigned)(ctas + plan_ctas)), kPlanThreads, 0, stream,
                        plan != nullptr ? *plan : PlanArgs{}, w, plan_ctas);
}

bool folded_supported(int dtype, int heads, int head_size, int hidden) {
  return (dtype == APS_F16 || dtype == APS_BF16) && (head_size == 128 || head_size == 64 || head_size == 32) &&
         heads > 0 && heads <= 256 && hidden > 0 && hidden % 128 == 0 &&
         scores_q_bytes(terms_of(dtype), (heads + 15) / 16 * 16) + 2 * kUnitBytes <= kScoresRing;
}

size_t folded_workspace_bytes(int batch, int max_blocks_per_seq, int block_size, int heads, int head_size,
                              int hidden, int dtype) {
  return align_up(workspace_layout(batch, max_blocks_per_seq, block_size, heads, head_size).total, 256) +
         layout_of(batch, max_blocks_per_seq, block_size, heads, head_size, hidden, dtype).total;
}

// Tensor maps: 16-byte aligned bases and row strides.  The CUDA-core re-projection, which serves the head counts that do not
// fill a tile, takes any others, so they are left to it and not refused.
bool folded_takes(const HybridCall& c) {
  return c.hidden_cache && c.w_k && c.w_v && c.num_hidden_rows > 0 && c.hidden_row_stride >= c.hidden_size &&
         c.w_stride >= c.hidden_size && c.hidden_row_stride % 8 == 0 && c.w_stride % 8 == 0 && aligned_to(c.hidden_cache, 16) &&
         aligned_to(c.w_k, 16) && aligned_to(c.w_v, 16) && sm_count() <= kMaxGrid;   // kMaxGrid: bounds the plan keeps
}

int enqueue_folded_attention(const HybridCall& c, const NewTokenWrite& nw, cudaStream_t cs) {
  const AttnShape& s = c.shape;
  const WorkspaceLayout w = workspace_layout(s.batch, s.max_blocks_per_seq, s.block_size, s.heads, s.head_size);
  const WorkspacePtrs ws = workspace_ptrs(c.workspace, w);
  const Layout l = layout_of(s.batch, s.max_blocks_per_seq, s.block_size, s.heads, s.head_size, c.hidden_size, s.dtype);
  char* b = static_cast<char*>(c.workspace) + align_up(w.total, 256);
  GroupPlan* groups = reinterpret_cast<GroupPlan*>(b + l.off_groups);
  const bool have_kv = c.key_cache != nullptr && c.value_cache != nullptr;
  const int nt = terms_of(s.dtype), e_blocks = c.hidden_size / 128;
  int st;

  PlanArgs pa{};
  pa.plan = ws.plan; pa.part_offset = ws.part_offset; pa.kv_chunks = ws.kv_chunks;
  pa.hid_slot = reinterpret_cast<int*>(b + l.off_slot); pa.hid_list = reinterpret_cast<int2*>(b + l.off_list);
  pa.groups = groups; pa.seq_lens = c.seq_lens; pa.cache_type = c.cache_type; pa.batch = s.batch;
  pa.max_tokens = s.max_blocks_per_seq * s.block_size; pa.kv_present = have_kv ? 1 : 0; pa.n_groups = l.n_groups;
  pa.steps = e_blocks; pa.grid_scores = sm_count();
  pa.max_slice = l.max_slice < e_blocks ? l.max_slice : e_blocks; pa.item_target = kSumRounds * sm_count();
  for (int i = 1; i <= kMaxSlice; ++i) pa.turns |= SumColumns(nt, l.np, i).turn_mask() << (4 * i);
  if ((st = launch_step_plan(&pa, nw, cs)) != APS_OK) return st;

  Maps m;
  const uint64_t hd = (uint64_t)s.heads * s.head_size;
  void* qz = b + l.off_qz;
  {
    // cached rows as [64 columns][rows][E / 64], boxes of (64, 8 or 16 rows, 2)
    TensorMapSpec spec{};
    spec.base = c.hidden_cache; spec.dtype = s.dtype; spec.rank = 3;
    spec.dims[0] = 64; spec.dims[1] = c.num_hidden_rows; spec.dims[2] = c.hidden_size / 64;
    spec.strides_bytes[0] = c.hidden_row_stride * 2; spec.strides_bytes[1] = 128;
    spec.box[0] = 64; spec.box[1] = 16; spec.box[2] = 2;
    if ((st = cached_tensor_map(&m.x_sum, spec, "hidden cache")) != APS_OK) return st;
    spec.box[1] = 8;
    if ((st = cached_tensor_map(&m.x_scores, spec, "hidden cache")) != APS_OK) return st;
  }
  if ((st = map_2d(&m.q, qz, s.dtype, c.hidden_size, (uint64_t)l.n_cap * nt * s.heads, c.hidden_size, s.heads, "folded queries")) != APS_OK) return st;
  if ((st = map_2d(&m.wk, c.w_k, s.dtype, c.hidden_size, hd, c.w_stride, s.head_size, "W_k")) != APS_OK) return st;
  if ((st = map_2d(&m.wv, c.w_v, s.dtype, c.hidden_size, hd, c.w_stride, hd < 128 ? (uint32_t)hd : 128, "W_v")) != APS_OK) return st;
  if ((st = map_2d(&m.z, qz, s.dtype, c.hidden_size, (uint64_t)nt * s.heads * l.n_cap, c.hidden_size, 16, "weighted sums")) != APS_OK) return st;

  Params p{};
  p.query = c.query; p.block_tables = c.block_tables; p.cache_type = c.cache_type; p.batch = s.batch;
  p.qt = qz; p.z = qz;
  p.qscale = reinterpret_cast<float*>(b + l.off_qscale); p.inv_sum = reinterpret_cast<float*>(b + l.off_inv);
  p.scores = reinterpret_cast<float*>(b + l.off_scores); p.probs = b + l.off_probs;
  p.tile_pieces = reinterpret_cast<int2*>(b + l.off_pieces);
  p.out_part = reinterpret_cast<float*>(b + l.off_part);
  p.status = ws.plan + kPlanStatus;
  p.heads = s.heads; p.np = l.np; p.head_size = s.head_size; p.hidden = c.hidden_size; p.slabs = c.hidden_size / 64;
  p.block_size = s.block_size; p.max_blocks = s.max_blocks_per_seq; p.n_cap = l.n_cap;
  p.n_hidden_cap = l.n_hidden_cap; p.splits = l.splits; p.unfold_ring = l.unfold_ring; p.grid_scores = pa.grid_scores;
  p.sum_copiers = kSumCopiers; p.sum_threads = 32 + 32 * (kSumCopiers + sum_epilogue_warps(pa.max_slice, l.np));
  p.query_stride = s.query_stride; p.scale_log2 = s.scale * 1.4426950408889634f;
  p.w_box_rows = hd < 128 ? (int)hd : 128;
  const int w_tiles = (int)((hd + 127) / 128);
  ScopedProfile prof(1, cs);
  for (int g = 0; g < l.n_groups; ++g) {
    p.plan = groups + g;
    p.group_first = g * kGroup;
    const bool bf16 = s.dtype == APS_BF16;
    const HybridCall* kv = have_kv && g == 0 ? &c : nullptr;   // the K/V kernel runs between the first fold and its scores
    switch (s.head_size) {
      case 128: st = bf16 ? launch_group<__nv_bfloat16, 128>(m, p, l.n_cap, w_tiles, kv, ws, cs) : launch_group<__half, 128>(m, p, l.n_cap, w_tiles, kv, ws, cs); break;
      case 64: st = bf16 ? launch_group<__nv_bfloat16, 64>(m, p, l.n_cap, w_tiles, kv, ws, cs) : launch_group<__half, 64>(m, p, l.n_cap, w_tiles, kv, ws, cs); break;
      default: st = bf16 ? launch_group<__nv_bfloat16, 32>(m, p, l.n_cap, w_tiles, kv, ws, cs) : launch_group<__half, 32>(m, p, l.n_cap, w_tiles, kv, ws, cs); break;
    }
    if (st != APS_OK) return st;
  }
  const HiddenOutputs ho{pa.hid_slot, p.out_part, c.b_v, c.seq_lens, l.splits, p.n_hidden_cap};
  return launch_combine(ws, c.out, &ho, s, cs);
}

}  // namespace aps
