// Causal self-attention of packed prompts (prefill), fp16 / bf16, head sizes 64 and 128.
//
// Replaces the third-party flash_attn_varlen_func call of the reference
// (additional_designs/attention/backends/aptserve_flash_attn.py:414-426) on the layouts its model produces: q, k, v as
// column ranges of one projection ([T, H D] with any row stride), prompts one behind the other, their bounds on the device.
//
// One CTA per (128 query rows, head, prompt), two CTAs per SM, key tiles of 64 rows up to the diagonal:
//   S = Q K^T      tcgen05, M = 128 queries, N = 64 keys, both operands K-major in shared memory, S in one of two buffers
//   P = 2^(S - m)  a thread per query row takes its row of S from tensor memory and writes the weights in the inputs' type over it
//   O += P V       tcgen05, A = P from tensor memory, B = V MN-major as it lies in the projection
// S of the next tile is computed while the weights of this one are formed, so that the softmax warps, whose turn is the longest
// (64 exponentials per row and tile, 16 per cycle and SM), find the next tile's scores ready.  O stays in tensor
// memory.  The running maximum is only moved (and O rescaled, by the rows' own threads, after the last tile's P V) when it
// has grown by more than 2^8; weights are kept at 2^7 times their value, at most 2^15 in all (fp16 range).
// A weight goes into P V as two 16-bit terms, itself rounded and the rounded rest, so that what is left of the error is the
// rounding of the output: with one term, a library's and this kernel's alike, the weights' rounding added a fifth to it
// (40 heads of 128, six prompts, fp16: 2.46e-4 -> 2.00e-4; bf16 2.00e-3 -> 1.61e-3; at most half a unit of the last place).
// It costs a fifth of the time (61 -> 73 us).
// Measured on one B200, the library call (flash_attn 2.8) -> this kernel: six OPT-13B prompts of 226 - 972 tokens 120 -> 73 us,
// eight of 677 - 2048 565 -> 312 (580 TFLOP/s of causal attention, the second terms not counted), eight OPT-1.3B prompts 85 -> 52.
// With one buffer of S and tiles of 128 keys, where scores, weights and P V are one chain, 93 and 429 us.
//
// Warps: 0 copies, 1 MMA issue, 2-5 softmax (a warp's tensor-memory lanes are given by its number modulo four).
// Every mbarrier wait is bounded by a clock budget; one that runs out leaves the CTA's rows as NaN and a status that
// aps_cache_ops_status reports.

#include "attention_common.cuh"   // read_prefill_status
#include "sm100.cuh"
#include "tensor_maps.cuh"

#include <type_traits>

namespace aps {
namespace {

constexpr int kThreads = 192, kRows = 128, kKeys = 64;
constexpr float kSlack = 8.f;   // log2 of how much the maximum may have grown before O is rescaled
constexpr float kUp = 7.f;      // log2 of what the weights are kept at

__device__ int g_prefill_status = 0;   // a wait has run out since this was read last; the calls have no scratch to hold it

struct Args {
  const int32_t* bounds; void* out;
  int64_t total, out_stride;
  float scale_log2;
};

struct Aux {
  uint64_t q_full, k_full[2], v_full[2], k_empty[2], v_empty[2], s_full[2], p_full[2];   // tile j: entry j & 1, phase j >> 1
  uint32_t tmem_base;
  int abort_flag;
};

// D (+)= A B with A in tensor memory (two elements of K per column).
__device__ __forceinline__ void tc_mma_tmem_a(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "mov.b64 db, {%2, %3};\n\tsetp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
template <typename T> __device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// The two values as they have been packed.
template <typename T> __device__ __forceinline__ float2 unpack2(uint32_t w);
template <> __device__ __forceinline__ float2 unpack2<__half>(uint32_t w) { return __half22float2(*reinterpret_cast<const __half2*>(&w)); }
template <> __device__ __forceinline__ float2 unpack2<__nv_bfloat16>(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

template <int D> constexpr size_t prefill_smem() { return 1024 + (size_t)(kRows + 4 * kKeys) * D * 2; }

template <typename T, int D>
__global__ void __launch_bounds__(kThreads, 2)
prefill_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
               const __grid_constant__ CUtensorMap map_v, const Args a) {
  constexpr int kSlabs = D / 64;                       // boxes of 64 columns
  constexpr uint32_t kQSlab = kRows * 128, kSlab = kKeys * 128, kQBytes = kSlabs * kQSlab, kTileBytes = kSlabs * kSlab;
  constexpr uint32_t kFmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
  constexpr uint32_t kCols = 256, kO = 128;            // tensor memory: two buffers of S (and P over it), then O
  extern __shared__ uint8_t smem_raw[];
  const uint32_t q_at = (smem_u32(smem_raw) + 1023) & ~1023u, k_at = q_at + kQBytes, v_at = k_at + 2 * kTileBytes;
  __shared__ Aux aux;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int head = blockIdx.y, start = a.bounds[blockIdx.z], len = a.bounds[blockIdx.z + 1] - start;
  const int row0 = (int)(gridDim.x - 1 - blockIdx.x) * kRows;    // the rows with the most keys first
  if (row0 >= len) return;
  if (threadIdx.x == 0) {
    mbar_init(&aux.q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&aux.k_full[i], 1); mbar_init(&aux.v_full[i], 1); mbar_init(&aux.k_empty[i], 1); mbar_init(&aux.v_empty[i], 1);
      mbar_init(&aux.s_full[i], 1); mbar_init(&aux.p_full[i], 4);
    }
    aux.abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 1) tmem_alloc(&aux.tmem_base, kCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = aux.tmem_base;
  volatile int* abort_flag = &aux.abort_flag;
  const int n_tiles = (min(len, row0 + kRows) + kKeys - 1) / kKeys;
  auto wait = [&](uint64_t* bars, int tile, int code) {
    return mbar_wait_warp(smem_u32(&bars[tile & 1]), (uint32_t)(tile >> 1) & 1u, abort_flag, &g_prefill_status, code, lane);
  };
  bool ok = true;
  if (warp == 0) {
    auto load = [&](uint64_t* bar, const CUtensorMap* map, uint32_t dst, uint32_t slab, int row) {
      if (lane == 0) mbar_expect_tx_addr(smem_u32(bar), kSlabs * slab);
      __syncwarp();
      if (lane < kSlabs) tma_load_2d_cta(dst + lane * slab, map, smem_u32(bar), head * D + lane * 64, row);
      __syncwarp();
    };
    load(&aux.q_full, &map_q, q_at, kQSlab, start + row0);
    for (int j = 0; j < n_tiles; ++j) {
      const int i = j & 1;
      if (j > 1 && !wait(aux.k_empty, j - 2, 1)) { ok = false; break; }
      load(&aux.k_full[i], &map_k, k_at + i * kTileBytes, kSlab, start + j * kKeys);
      if (j > 1 && !wait(aux.v_empty, j - 2, 2)) { ok = false; break; }
      load(&aux.v_full[i], &map_v, v_at + i * kTileBytes, kSlab, start + j * kKeys);
    }
  } else if (warp == 1) {
    constexpr uint32_t s_idesc = mma_idesc(kFmt, 128, kKeys, false);
    constexpr uint32_t o_idesc = mma_idesc(kFmt, 128, D, false) | (1u << 16);   // B is MN-major
    auto scores = [&](int j) {   // S of tile j
      const int i = j & 1;
      // the buffer still holds the weights of tile j - 2
      if (!wait(aux.k_full, j, 3) || (j > 1 && !wait(aux.v_empty, j - 2, 4))) return false;
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          tc_mma_cta(tmem + i * kKeys, desc_lo(q_at + k / 4 * kQSlab + k % 4 * 32, 16), desc_hi(1024, true),
                     desc_lo(k_at + i * kTileBytes + k / 4 * kSlab + k % 4 * 32, 16), desc_hi(1024, true), s_idesc, k != 0);
        tc_commit_cta(smem_u32(&aux.k_empty[i]));
        tc_commit_cta(smem_u32(&aux.s_full[i]));
      }
      __syncwarp();
      return true;
    };
    ok = mbar_wait_warp(smem_u32(&aux.q_full), 0, abort_flag, &g_prefill_status, 3, lane) && scores(0);
    for (int j = 0; j < n_tiles && ok; ++j) {
      const int i = j & 1;
      if ((j + 1 < n_tiles && !scores(j + 1)) || !wait(aux.v_full, j, 3) || !wait(aux.p_full, j, 4)) { ok = false; break; }
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < kKeys / 16; ++k)
#pragma unroll
          for (int t = 0; t < 2; ++t)   // the weights' terms
            tc_mma_tmem_a(tmem + kO, tmem + i * kKeys + t * (kKeys / 2) + k * 8, desc_lo(v_at + i * kTileBytes + k * 2048, kSlab),
                          desc_hi(1024, true), o_idesc, j > 0 || k + t != 0);
        tc_commit_cta(smem_u32(&aux.v_empty[i]));
      }
      __syncwarp();
    }
  } else {
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16), o_at = lanes + kO;
    float m = -INFINITY, l = 0.f;   // maximum the weights refer to (of the raw scores), their sum
    for (int j = 0; j < n_tiles; ++j) {
      const uint32_t s_at = lanes + (j & 1) * kKeys;
      const int seen = row0 + row - j * kKeys;   // the last key of the tile that the row attends to
      const bool diagonal = j * kKeys + kKeys - 1 > row0;
      if (!wait(aux.s_full, j, 5)) { ok = false; break; }
      tc_fence_after();
      uint32_t v[kKeys];
      tmem_ld32(s_at, v);
      tmem_ld32(s_at + 32, v + 32);
      tmem_ld_wait();
      if (diagonal) {
#pragma unroll
        for (int i = 0; i < kKeys; ++i)
          if (i > seen) v[i] = 0xff800000u;   // -infinity
      }
      float tops[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < kKeys; ++i) tops[i & 3] = fmaxf(tops[i & 3], __uint_as_float(v[i]));
      const float top = fmaxf(fmaxf(tops[0], tops[1]), fmaxf(tops[2], tops[3]));
      if (j == 0) {
        m = top;
      } else {
        const bool move = top > m && !((top - m) * a.scale_log2 <= kSlack);
        if (__any_sync(0xffffffffu, move)) {
          if (!wait(aux.v_empty, j - 1, 6)) { ok = false; break; }   // O is as the last tile left it
          tc_fence_after();
          const float new_m = move ? top : m, down = move && m != -INFINITY ? ex2((m - new_m) * a.scale_log2) : 1.f;
          l *= down;
          m = new_m;
#pragma unroll
          for (int c = 0; c < D; c += 16) {
            uint32_t o[16];
            tmem_ld16(o_at + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * down);
            tmem_st16(o_at + c, o);
          }
        }
      }
      const float shift = (m == -INFINITY ? 0.f : m * a.scale_log2) - kUp;
      float sums[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t rest[kKeys / 2];
#pragma unroll
      for (int i = 0; i < kKeys; i += 2) {
        const float x = ex2(fmaf(__uint_as_float(v[i]), a.scale_log2, -shift)), y = ex2(fmaf(__uint_as_float(v[i + 1]), a.scale_log2, -shift));
        sums[i / 2 & 3] += x + y;
        v[i / 2] = pack2<T>(x, y);
        const float2 r = unpack2<T>(v[i / 2]);
        rest[i / 2] = pack2<T>(x - r.x, y - r.y);
      }
      l += (sums[0] + sums[1]) + (sums[2] + sums[3]);
      tmem_st16(s_at, v);
      tmem_st16(s_at + 16, v + 16);
      tmem_st16(s_at + 32, rest);
      tmem_st16(s_at + 48, rest + 16);
      tmem_st_wait();
      tc_fence_before();
      // rows past the prompt are the next one's: their weights are zero, but zero times infinity is not
      const int valid = len - j * kKeys;
      if (valid < kKeys) {
        if (!wait(aux.v_full, j, 6)) { ok = false; break; }
        for (int i = row; i < (kKeys - valid) * kSlabs * 8; i += 128) {
          const int r = valid + i / (kSlabs * 8), rem = i % (kSlabs * 8);
          asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(v_at + (j & 1) * kTileBytes + (rem >> 3) * kSlab + r * 128 + (rem & 7) * 16), "r"(0u) : "memory");
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      __syncwarp();
      if (lane == 0) mbar_arrive_addr(smem_u32(&aux.p_full[j & 1]));
    }
    ok = ok && wait(aux.v_empty, n_tiles - 1, 7);
    tc_fence_after();
    const int64_t at = (int64_t)start + row0 + row;
    const bool mine = row0 + row < len && at >= 0 && at < a.total;
    const float inv = l > 0.f || l != l ? 1.f / l : 0.f;
    T* dst = static_cast<T*>(a.out) + at * a.out_stride + (int64_t)head * D;
#pragma unroll
    for (int c = 0; c < D; c += 16) {
      uint32_t v[16], w[8];
      tmem_ld16(o_at + c, v);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; i += 2) {
        const float bad = __int_as_float(0x7fc00000);
        w[i / 2] = pack2<T>(ok ? __uint_as_float(v[i]) * inv : bad, ok ? __uint_as_float(v[i + 1]) * inv : bad);
      }
      if (mine) {
        *reinterpret_cast<uint4*>(dst + c) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(dst + c + 8) = make_uint4(w[4], w[5], w[6], w[7]);
      }
    }
  }
  if (!ok) {   // copies still in flight get a bounded time to land
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) { }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_free(tmem, kCols); }
}

// A wait on a barrier that nothing arrives on, as the kernel's waits.
__global__ void prefill_wait_selftest_kernel(long long budget) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x != 0) return;
  abort_flag = 0;
  mbar_init(&bar, 1);
  mbar_init_fence();
  mbar_wait_addr(smem_u32(&bar), 0, &abort_flag, &g_prefill_status, 1, budget);
}

template <typename T, int D>
int launch(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const Args& a, int blocks, int heads, int prompts,
           cudaStream_t stream) {
  static bool done[64] = {false};
  auto kernel = prefill_kernel<T, D>;
  int dev = 0;
  APS_CUDA(cudaGetDevice(&dev));
  APS_REQUIRE(dev >= 0 && dev < 64, APS_ERR_CUDA, "device index %d out of range", dev);
  if (!done[dev]) {
    APS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prefill_smem<D>()));
    done[dev] = true;
  }
  kernel<<<dim3(blocks, heads, prompts), kThreads, prefill_smem<D>(), stream>>>(q, k, v, a);
  return launch_status("prefill_kernel");
}

}  // namespace

int read_prefill_status(int* host_status, cudaStream_t stream) {
  void* addr = nullptr;
  APS_CUDA(cudaGetSymbolAddress(&addr, g_prefill_status));
  APS_CUDA(cudaMemcpyAsync(host_status, addr, sizeof(int), cudaMemcpyDeviceToHost, stream));
  APS_CUDA(cudaStreamSynchronize(stream));
  if (*host_status != 0) {
    *host_status = 3;
    APS_CUDA(cudaMemsetAsync(addr, 0, sizeof(int), stream));   // reported once
  }
  return APS_OK;
}

}  // namespace aps

using namespace aps;

extern "C" int aps_selftest_prefill_wait(long long budget_cycles, void* stream) {
  APS_REQUIRE(budget_cycles > 0 && budget_cycles <= 100000000LL, APS_ERR_SHAPE,
              "selftest_prefill_wait: the budget must be between 1 and 1e8 clock cycles");
  prefill_wait_selftest_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(budget_cycles);
  return launch_status("prefill_wait_selftest_kernel");
}

extern "C" int aps_prefill_attention(void* out, const void* query, const void* key, const void* value, const int32_t* bounds,
                                     int num_prompts, int max_prompt_len, int64_t num_tokens, int num_heads, int head_size,
                                     int64_t query_stride, int64_t key_stride, int64_t value_stride, int64_t out_stride,
                                     float scale, int dtype, void* stream) {
  APS_REQUIRE(dtype == APS_F16 || dtype == APS_BF16, APS_ERR_DTYPE, "prefill_attention: unsupported dtype %d", dtype);
  APS_REQUIRE(head_size == 64 || head_size == 128, APS_ERR_UNSUPPORTED, "prefill_attention: head size %d is not supported", head_size);
  APS_REQUIRE(num_prompts >= 0 && num_prompts <= 65535 && max_prompt_len >= 0 && num_tokens >= 0 && num_heads > 0 && num_heads <= 65535 &&
                  num_tokens < (int64_t(1) << 31) - kRows,
              APS_ERR_SHAPE, "prefill_attention: bad sizes");
  if (num_prompts == 0 || max_prompt_len == 0 || num_tokens == 0) return APS_OK;
  APS_REQUIRE(out && query && key && value && bounds, APS_ERR_NULL_POINTER, "prefill_attention: null pointer");
  // the running maximum is that of the raw scores, and a masked score stays -infinity only times a positive number
  APS_REQUIRE(scale >= 1.17549435e-38f && scale < 1.70141183e38f, APS_ERR_UNSUPPORTED,
              "prefill_attention: the scale must be positive and below 2^127 (got %g)", (double)scale);
  const int64_t row = (int64_t)num_heads * head_size;
  APS_REQUIRE(query_stride >= row && key_stride >= row && value_stride >= row && out_stride >= row, APS_ERR_SHAPE,
              "prefill_attention: strides smaller than a row");
  APS_REQUIRE(aligned_to(query, 16) && aligned_to(key, 16) && aligned_to(value, 16) && aligned_to(out, 16) && query_stride % 8 == 0 &&
                  key_stride % 8 == 0 && value_stride % 8 == 0 && out_stride % 8 == 0,
              APS_ERR_MISALIGNED, "prefill_attention: tensors must be 16-byte aligned with 16-byte strides");
  TensorMapSpec spec{};
  spec.dtype = dtype; spec.rank = 2;
  spec.dims[0] = (uint64_t)row; spec.dims[1] = (uint64_t)num_tokens;
  spec.box[0] = 64; spec.box[1] = kRows;
  CUtensorMap q, k, v;
  int st;
  spec.base = query; spec.strides_bytes[0] = (uint64_t)query_stride * 2;
  if ((st = cached_tensor_map(&q, spec, "prompt queries")) != APS_OK) return st;
  spec.box[1] = kKeys;
  spec.base = key; spec.strides_bytes[0] = (uint64_t)key_stride * 2;
  if ((st = cached_tensor_map(&k, spec, "prompt keys")) != APS_OK) return st;
  spec.base = value; spec.strides_bytes[0] = (uint64_t)value_stride * 2;
  if ((st = cached_tensor_map(&v, spec, "prompt values")) != APS_OK) return st;
  const Args a{bounds, out, num_tokens, out_stride, scale * 1.4426950408889634f};
  const int blocks = (max_prompt_len + kRows - 1) / kRows;
  cudaStream_t cs = (cudaStream_t)stream;
  if (dtype == APS_BF16)
    return head_size == 128 ? launch<__nv_bfloat16, 128>(q, k, v, a, blocks, num_heads, num_prompts, cs)
                            : launch<__nv_bfloat16, 64>(q, k, v, a, blocks, num_heads, num_prompts, cs);
  return head_size == 128 ? launch<__half, 128>(q, k, v, a, blocks, num_heads, num_prompts, cs)
                          : launch<__half, 64>(q, k, v, a, blocks, num_heads, num_prompts, cs);
}
