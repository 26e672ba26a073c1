// The element-wise part of one batched Llama decode step around the sparse
// attention layer-step: residual add + RMSNorm, rotary embedding fused with the
// KV-cache append, SiLU(gate) * up, and the greedy arg-max over the vocabulary.
//
// In the reference these run as the Hugging Face model's own PyTorch ops inside
// the captured decode step (condition_block_triton_impl/core.py:190-316): about
// forty small kernels per layer.  Here each group is one launch.  Every kernel
// reproduces the bf16 rounding points of the PyTorch expression it replaces
// (transformers/models/llama/modeling_llama.py: LlamaRMSNorm.forward,
// apply_rotary_pos_emb, LlamaMLP.forward), so the fused step and the module-by-module
// step agree to the last bit except for the order of the fp32 sum of squares.
//
// All tensors are bf16, rows are contiguous.
#include "gemm_parts.cuh"

namespace ia {
namespace {

__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// 8 bf16 values <-> 8 floats through one 16-byte access
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 w = *reinterpret_cast<const uint4*>(p);
  v[0] = bf16lo(w.x); v[1] = bf16hi(w.x); v[2] = bf16lo(w.y); v[3] = bf16hi(w.y);
  v[4] = bf16lo(w.z); v[5] = bf16hi(w.z); v[6] = bf16lo(w.w); v[7] = bf16hi(w.w);
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&v)[8]) {
  uint4 w;
  w.x = pack2(v[0], v[1]); w.y = pack2(v[2], v[3]); w.z = pack2(v[4], v[5]); w.w = pack2(v[6], v[7]);
  *reinterpret_cast<uint4*>(p) = w;
}

// ---- residual add + RMSNorm ------------------------------------------------------
// x = residual (+ delta, rounded to bf16 and written back); out = weight * bf16(x * rsqrt(mean(x^2) + eps)).
// One CTA per row; kChunks * 8 * blockDim >= hidden, the row stays in registers.
constexpr int kNormThreads = 256;
template <int kChunks>
__global__ void __launch_bounds__(kNormThreads)
llama_add_rmsnorm_kernel(__nv_bfloat16* __restrict__ residual, const __nv_bfloat16* __restrict__ delta,
                         const __nv_bfloat16* __restrict__ weight, __nv_bfloat16* __restrict__ out, int hidden,
                         float eps) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int64_t row = (int64_t)blockIdx.x * hidden;
  float x[kChunks][8];
  float sq = 0.f;
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    const int i = (c * kNormThreads + threadIdx.x) * 8;
    if (i < hidden) {
      load8(residual + row + i, x[c]);
      if (delta != nullptr) {
        float d[8];
        load8(delta + row + i, d);
#pragma unroll
        for (int j = 0; j < 8; ++j) x[c][j] = round_bf16(x[c][j] + d[j]);
        store8(residual + row + i, x[c]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) sq = fmaf(x[c][j], x[c][j], sq);
    }
  }
  __shared__ float part[kNormThreads / 32];
  __shared__ float scale_s;
  sq = warp_sum(sq);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sq;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < kNormThreads / 32 ? part[threadIdx.x] : 0.f;
    v = warp_sum(v);
    if (threadIdx.x == 0) scale_s = rsqrtf(v / (float)hidden + eps);
  }
  __syncthreads();
  const float scale = scale_s;
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    const int i = (c * kNormThreads + threadIdx.x) * 8;
    if (i < hidden) {
      float w[8], y[8];
      load8(weight + i, w);
#pragma unroll
      for (int j = 0; j < 8; ++j) y[j] = w[j] * round_bf16(x[c][j] * scale);
      store8(out + row + i, y);
    }
  }
}

// ---- rotary embedding + cache append ---------------------------------------------
// qkv row of a sequence: [Hq * D | Hkv * D | Hkv * D].  One CTA per (sequence, head of
// the fused row), D / 2 threads; thread d owns the pair (d, d + D/2):
//   out[d]       = bf16( bf16(x[d] * cos[d])             + bf16(-x[d + D/2] * sin[d]) )
//   out[d + D/2] = bf16( bf16(x[d + D/2] * cos[d + D/2]) + bf16( x[d]       * sin[d + D/2]) )
// q goes to q_out [B, Hq, D]; k (rotated) and v (as is) go to the cache row of position
// seq_lens[b] - 1.  A position outside [0, max_pos) or the cache leaves the row untouched.
__global__ void llama_rope_append_kernel(const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ cos_t,
                                         const __nv_bfloat16* __restrict__ sin_t, int max_pos,
                                         const int32_t* __restrict__ seq_lens, __nv_bfloat16* __restrict__ k_cache,
                                         __nv_bfloat16* __restrict__ v_cache, int64_t seq_stride, int64_t head_stride,
                                         int cache_len, __nv_bfloat16* __restrict__ q_out, int n_q_heads,
                                         int n_kv_heads, int D) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int b = blockIdx.x, head = blockIdx.y, d = threadIdx.x, half = D >> 1;
  const int pos = seq_lens[b] - 1;
  if (pos < 0 || pos >= max_pos || pos >= cache_len) return;
  const int row_elems = (n_q_heads + 2 * n_kv_heads) * D;
  const __nv_bfloat16* src = qkv + (int64_t)b * row_elems + (int64_t)head * D;
  if (head >= n_q_heads + n_kv_heads) {  // value head: plain copy
    const int h = head - n_q_heads - n_kv_heads;
    __nv_bfloat16* dst = v_cache + b * seq_stride + h * head_stride + (int64_t)pos * D;
    dst[d] = src[d];
    dst[d + half] = src[d + half];
    return;
  }
  const float x1 = __bfloat162float(src[d]), x2 = __bfloat162float(src[d + half]);
  const __nv_bfloat16* c = cos_t + (int64_t)pos * D;
  const __nv_bfloat16* s = sin_t + (int64_t)pos * D;
  const float lo = round_bf16(x1 * __bfloat162float(c[d])) + round_bf16(-x2 * __bfloat162float(s[d]));
  const float hi = round_bf16(x2 * __bfloat162float(c[d + half])) + round_bf16(x1 * __bfloat162float(s[d + half]));
  __nv_bfloat16* dst = head < n_q_heads
                           ? q_out + ((int64_t)b * n_q_heads + head) * D
                           : k_cache + b * seq_stride + (head - n_q_heads) * head_stride + (int64_t)pos * D;
  dst[d] = __float2bfloat16_rn(lo);
  dst[d + half] = __float2bfloat16_rn(hi);
}

// ---- SiLU(gate) * up ----------------------------------------------------------------
// gate_up row: [I gate | I up]; out = bf16( bf16(g / (1 + exp(-g))) * u )
__global__ void llama_silu_mul_kernel(const __nv_bfloat16* __restrict__ gate_up, __nv_bfloat16* __restrict__ out,
                                      int n_rows, int inter) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int per_row = inter >> 3;
  const int64_t unit = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (unit >= (int64_t)n_rows * per_row) return;
  const int64_t r = unit / per_row;
  const int i = (int)(unit - r * per_row) * 8;
  float g[8], u[8], y[8];
  load8(gate_up + r * 2 * inter + i, g);
  load8(gate_up + r * 2 * inter + inter + i, u);
#pragma unroll
  for (int j = 0; j < 8; ++j) y[j] = round_bf16(g[j] / (1.f + expf(-g[j]))) * u[j];
  store8(out + r * inter + i, y);
}

// ---- arg-max over the vocabulary --------------------------------------------------
// One CTA per row; the lowest index among equal maxima wins.  NaN never wins.
constexpr int kArgmaxThreads = 1024;
__global__ void __launch_bounds__(kArgmaxThreads)
llama_argmax_kernel(const __nv_bfloat16* __restrict__ logits, int64_t row_stride, int vocab,
                    int64_t* __restrict__ out) {
  grid_launch_dependents();
  grid_dependency_wait();
  const __nv_bfloat16* row = logits + (int64_t)blockIdx.x * row_stride;
  float best = -INFINITY;
  int best_i = 0x7fffffff;
  const int vec_end = ((reinterpret_cast<uintptr_t>(row) & 15u) == 0) ? (vocab & ~7) : 0;
  for (int i = threadIdx.x * 8; i < vec_end; i += kArgmaxThreads * 8) {
    float v[8];
    load8(row + i, v);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (v[j] > best) { best = v[j]; best_i = i + j; }  // ascending i: the first maximum stays
  }
  for (int i = vec_end + threadIdx.x; i < vocab; i += kArgmaxThreads) {
    const float v = __bfloat162float(row[i]);
    if (v > best || (v == best && i < best_i)) { best = v; best_i = i; }
  }
  __shared__ float best_s[kArgmaxThreads / 32];
  __shared__ int idx_s[kArgmaxThreads / 32];
  auto merge = [](float& a, int& ai, float b, int bi) {
    if (b > a || (b == a && bi < ai)) { a = b; ai = bi; }
  };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    merge(best, best_i, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, best_i, o));
  if ((threadIdx.x & 31) == 0) { best_s[threadIdx.x >> 5] = best; idx_s[threadIdx.x >> 5] = best_i; }
  __syncthreads();
  if (threadIdx.x < 32) {
    best = best_s[threadIdx.x];
    best_i = idx_s[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      merge(best, best_i, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, best_i, o));
    if (threadIdx.x == 0) out[blockIdx.x] = best_i == 0x7fffffff ? 0 : best_i;
  }
}

// ---- the same kernels on a projection's partial sums (gemm_parts.cuh) ---------------------------------
// Latency bound: a few hundred KB out of L2 and one row reduction.  The sums of a column's slots replace the load of
// the finished projection (up to eight slots in flight at once); everything after that, rounding points included, is
// the kernel above.
constexpr int kPartNormThreads = 512;
template <int kChunks>
__global__ void __launch_bounds__(kPartNormThreads)
llama_add_rmsnorm_parts_kernel(__nv_bfloat16* __restrict__ residual, const PartsView parts,
                               const __nv_bfloat16* __restrict__ weight, __nv_bfloat16* __restrict__ out, int hidden,
                               float eps) {
  grid_launch_dependents();
  float w[kChunks][8];  // weights do not depend on the kernel before
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    const int i = (c * kPartNormThreads + threadIdx.x) * 8;
    if (i < hidden) load8(weight + i, w[c]);
  }
  grid_dependency_wait();
  const int64_t row = (int64_t)blockIdx.x * hidden;
  float x[kChunks][8];
  float sq = 0.f;
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    const int i = (c * kPartNormThreads + threadIdx.x) * 8;
    if (i < hidden) {
      load8(residual + row + i, x[c]);
      int count;
      const float* tile = parts.tile((uint32_t)i / kPartCols, count);
      float d[8];
      sum_parts<8, 8>(tile, count, blockIdx.x, i % kPartCols, d);
#pragma unroll
      for (int j = 0; j < 8; ++j) x[c][j] = round_bf16(x[c][j] + d[j]);
      store8(residual + row + i, x[c]);
#pragma unroll
      for (int j = 0; j < 8; ++j) sq = fmaf(x[c][j], x[c][j], sq);
    }
  }
  __shared__ float part[kPartNormThreads / 32];
  sq = warp_sum(sq);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sq;
  __syncthreads();
  float v = (threadIdx.x & 31) < kPartNormThreads / 32 ? part[threadIdx.x & 31] : 0.f;
  const float scale = rsqrtf(warp_sum(v) / (float)hidden + eps);  // every warp for itself: the same order, one barrier
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
    const int i = (c * kPartNormThreads + threadIdx.x) * 8;
    if (i < hidden) {
      float y[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) y[j] = w[c][j] * round_bf16(x[c][j] * scale);
      store8(out + row + i, y);
    }
  }
}

__device__ __forceinline__ void load4(const __nv_bfloat16* p, float (&v)[4]) {
  const uint2 w = *reinterpret_cast<const uint2*>(p);
  v[0] = bf16lo(w.x); v[1] = bf16hi(w.x); v[2] = bf16lo(w.y); v[3] = bf16hi(w.y);
}
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float (&v)[4]) {
  uint2 w;
  w.x = pack2(v[0], v[1]); w.y = pack2(v[2], v[3]);
  *reinterpret_cast<uint2*>(p) = w;
}

// One thread per four coordinates of both halves of a head: unit = (sequence, head, d / 4)
__global__ void __launch_bounds__(128)
llama_rope_append_parts_kernel(const PartsView parts, const __nv_bfloat16* __restrict__ cos_t,
                               const __nv_bfloat16* __restrict__ sin_t, int max_pos,
                               const int32_t* __restrict__ seq_lens, __nv_bfloat16* __restrict__ k_cache,
                               __nv_bfloat16* __restrict__ v_cache, int64_t seq_stride, int64_t head_stride,
                               int cache_len, __nv_bfloat16* __restrict__ q_out, int batch, int n_q_heads,
                               int n_kv_heads, int D) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int half = D >> 1, per_head = D >> 3, n_heads = n_q_heads + 2 * n_kv_heads;
  const int unit = blockIdx.x * 128 + threadIdx.x;
  if (unit >= batch * n_heads * per_head) return;
  const int d = (unit % per_head) * 4, head = unit / per_head % n_heads, b = unit / (per_head * n_heads);
  const int pos = seq_lens[b] - 1;
  if (pos < 0 || pos >= max_pos || pos >= cache_len) return;
  float x1[4], x2[4];
  {
    const int c1 = head * D + d, c2 = c1 + half;
    int n1, n2;
    const float* t1 = parts.tile((uint32_t)c1 / kPartCols, n1);
    const float* t2 = parts.tile((uint32_t)c2 / kPartCols, n2);
    sum_parts<4, 8>(t1, n1, b, c1 % kPartCols, x1);
    sum_parts<4, 8>(t2, n2, b, c2 % kPartCols, x2);
  }
  if (head >= n_q_heads + n_kv_heads) {  // value head: plain copy
    __nv_bfloat16* dst = v_cache + b * seq_stride + (head - n_q_heads - n_kv_heads) * head_stride + (int64_t)pos * D;
    store4(dst + d, x1);
    store4(dst + d + half, x2);
    return;
  }
  float c1[4], c2[4], s1[4], s2[4], lo[4], hi[4];
  load4(cos_t + (int64_t)pos * D + d, c1);
  load4(cos_t + (int64_t)pos * D + d + half, c2);
  load4(sin_t + (int64_t)pos * D + d, s1);
  load4(sin_t + (int64_t)pos * D + d + half, s2);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    lo[j] = round_bf16(x1[j] * c1[j]) + round_bf16(-x2[j] * s1[j]);
    hi[j] = round_bf16(x2[j] * c2[j]) + round_bf16(x1[j] * s2[j]);
  }
  __nv_bfloat16* dst = head < n_q_heads
                           ? q_out + ((int64_t)b * n_q_heads + head) * D
                           : k_cache + b * seq_stride + (head - n_q_heads) * head_stride + (int64_t)pos * D;
  store4(dst + d, lo);
  store4(dst + d + half, hi);
}

__global__ void __launch_bounds__(256)
llama_silu_mul_parts_kernel(const PartsView parts, __nv_bfloat16* __restrict__ out, int n_rows, int inter) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int per_row = inter >> 3;
  const int64_t unit = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (unit >= (int64_t)n_rows * per_row) return;
  const int r = (int)(unit / per_row);
  const int i = (int)(unit - (int64_t)r * per_row) * 8;
  float g[8], u[8], y[8];
  int ng, nu;
  const float* tg = parts.tile((uint32_t)i / kPartCols, ng);
  const float* tu = parts.tile((uint32_t)(inter + i) / kPartCols, nu);
  sum_parts<8, 4>(tg, ng, r, i % kPartCols, g);
  sum_parts<8, 4>(tu, nu, r, (inter + i) % kPartCols, u);
#pragma unroll
  for (int j = 0; j < 8; ++j) y[j] = round_bf16(g[j] / (1.f + expf(-g[j]))) * u[j];
  store8(out + (int64_t)r * inter + i, y);
}

// Completes the logits whose tiles several CTAs summed, then the arg-max.  A row is shared by a cluster of CTAs,
// each with a run of whole tiles, and merged through rank 0's shared memory: a few rows alone would leave
// most SMs idle (one CTA of 1024 threads per row takes 6.4 us at 128256 columns, this form ends 3 us after the product).
constexpr int kArgmaxPartsThreads = 512, kArgmaxCluster = 8;
__global__ void __cluster_dims__(kArgmaxCluster, 1, 1) __launch_bounds__(kArgmaxPartsThreads)
llama_argmax_parts_kernel(const PartsView parts, __nv_bfloat16* __restrict__ logits, int vocab,
                          int64_t* __restrict__ out) {
  cluster_arrive_started();
  grid_launch_dependents();
  grid_dependency_wait();
  __shared__ float best_s[kArgmaxPartsThreads / 32];
  __shared__ int idx_s[kArgmaxPartsThreads / 32];
  __shared__ float rank_best[kArgmaxCluster];
  __shared__ int rank_idx[kArgmaxCluster];
  const int rank = blockIdx.x % kArgmaxCluster, row_i = blockIdx.x / kArgmaxCluster;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __nv_bfloat16* row = logits + (int64_t)row_i * vocab;
  const int n_tiles = (vocab + kPartCols - 1) / kPartCols;
  const int t_lo = (int)((int64_t)n_tiles * rank / kArgmaxCluster), t_hi = (int)((int64_t)n_tiles * (rank + 1) / kArgmaxCluster);
  // A tile is split where a CTA's range starts inside it.  The boundaries T c / P are walked by the warps; the first
  // boundary inside a tile stands for it.
  const bool pairs = (vocab & 3) == 0;  // rows start on 8-byte boundaries
  const uint32_t c_lo = max(parts.owner((uint32_t)t_lo * parts.k_chunks), 1u) ;
  const uint32_t c_hi = t_hi > t_lo ? parts.owner((uint32_t)t_hi * parts.k_chunks - 1u) : 0u;
  for (uint32_t c = c_lo + warp; c <= c_hi; c += kArgmaxPartsThreads / 32) {
    const uint32_t x = (uint32_t)((uint64_t)parts.total * c / parts.ctas);  // CTA c's first chunk
    const uint32_t t = x / parts.k_chunks;
    if (x % parts.k_chunks == 0 || (int)t < t_lo || (int)t >= t_hi || parts.owner(t * parts.k_chunks) != c - 1) continue;
    int count;
    const float* tile = parts.tile(t, count);
    float v[4];
    sum_parts<4, 4>(tile, count, row_i, lane * 4, v);
    const int n = (int)t * kPartCols + lane * 4;
    if (pairs && n + 3 < vocab) {
      store4(row + n, v);
    } else {
      for (int j = 0; j < 4; ++j)
        if (n + j < vocab) row[n + j] = __float2bfloat16_rn(v[j]);
    }
  }
  __syncthreads();  // this CTA's columns are complete

  const int lo = t_lo * kPartCols, hi = min(t_hi * kPartCols, vocab);
  float best = -INFINITY;
  int best_i = 0x7fffffff;
  const int vec_end = (reinterpret_cast<uintptr_t>(row + lo) & 15u) == 0 ? lo + ((hi - lo) & ~7) : lo;
  for (int i = lo + threadIdx.x * 8; i < vec_end; i += kArgmaxPartsThreads * 8) {
    float v[8];
    load8(row + i, v);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (v[j] > best) { best = v[j]; best_i = i + j; }  // ascending i: the first maximum stays
  }
  for (int i = vec_end + threadIdx.x; i < hi; i += kArgmaxPartsThreads) {
    const float v = __bfloat162float(row[i]);
    if (v > best || (v == best && i < best_i)) { best = v; best_i = i; }
  }
  auto merge = [](float& a, int& ai, float b, int bi) {
    if (b > a || (b == a && bi < ai)) { a = b; ai = bi; }
  };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    merge(best, best_i, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, best_i, o));
  if (lane == 0) { best_s[warp] = best; idx_s[warp] = best_i; }
  __syncthreads();
  cluster_wait_started();  // rank 0 runs: its shared memory may be written (a rank without tiles is here at once)
  if (warp == 0) {
    best = lane < kArgmaxPartsThreads / 32 ? best_s[lane] : -INFINITY;
    best_i = lane < kArgmaxPartsThreads / 32 ? idx_s[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      merge(best, best_i, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, best_i, o));
    if (lane == 0) {
      uint32_t dst_b, dst_i;
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(dst_b) : "r"((uint32_t)__cvta_generic_to_shared(rank_best + rank)));
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(dst_i) : "r"((uint32_t)__cvta_generic_to_shared(rank_idx + rank)));
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst_b), "f"(best) : "memory");
      asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(dst_i), "r"(best_i) : "memory");
    }
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (rank == 0 && threadIdx.x == 0) {
    best = -INFINITY;
    best_i = 0x7fffffff;
    for (int r = 0; r < kArgmaxCluster; ++r) merge(best, best_i, rank_best[r], rank_idx[r]);
    out[row_i] = best_i == 0x7fffffff ? 0 : best_i;
  }
}

template <typename Kern, typename... Args>
int launch(const char* what, Kern kern, dim3 grid, dim3 block, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  int n = 0;
  if (overlapped_launch_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = (unsigned)n;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  if (e != cudaSuccess) return fail(IA_ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(e));
  return check_launch(what);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace
}  // namespace ia

using namespace ia;

extern "C" {

int ia_llama_add_rmsnorm(void* residual, const void* delta, const void* weight, void* out, int n_rows, int hidden,
                         float eps, ia_stream_t stream) {
  if (!residual || !weight || !out) return fail(IA_ERR_BAD_ARG, "add_rmsnorm: null pointer");
  if (n_rows < 0 || hidden <= 0 || hidden % 8 != 0)
    return fail(IA_ERR_BAD_ARG, "add_rmsnorm: %d rows of %d (a multiple of 8)", n_rows, hidden);
  if (!aligned16(residual) || !aligned16(weight) || !aligned16(out) || (delta && !aligned16(delta)))
    return fail(IA_ERR_BAD_ARG, "add_rmsnorm: pointers must be 16-byte aligned");
  if (n_rows == 0) return IA_OK;
  auto* r = static_cast<__nv_bfloat16*>(residual);
  auto* d = static_cast<const __nv_bfloat16*>(delta);
  auto* w = static_cast<const __nv_bfloat16*>(weight);
  auto* o = static_cast<__nv_bfloat16*>(out);
  const int chunks = (hidden + kNormThreads * 8 - 1) / (kNormThreads * 8);
  const dim3 grid((unsigned)n_rows), block(kNormThreads);
  cudaStream_t st = (cudaStream_t)stream;
  switch (chunks) {
    case 1: return launch("llama_add_rmsnorm_kernel", llama_add_rmsnorm_kernel<1>, grid, block, st, r, d, w, o, hidden, eps);
    case 2: return launch("llama_add_rmsnorm_kernel", llama_add_rmsnorm_kernel<2>, grid, block, st, r, d, w, o, hidden, eps);
    case 3:
    case 4: return launch("llama_add_rmsnorm_kernel", llama_add_rmsnorm_kernel<4>, grid, block, st, r, d, w, o, hidden, eps);
    case 5: case 6: case 7:
    case 8: return launch("llama_add_rmsnorm_kernel", llama_add_rmsnorm_kernel<8>, grid, block, st, r, d, w, o, hidden, eps);
    default: return fail(IA_ERR_UNSUPPORTED, "add_rmsnorm: hidden size %d above %d", hidden, kNormThreads * 64);
  }
}

int ia_llama_rope_append(const void* qkv, const void* cos_table, const void* sin_table, int max_pos,
                         const int32_t* seq_lens, void* k_cache, void* v_cache, int64_t cache_seq_stride,
                         int64_t cache_head_stride, int cache_len, void* q_out, int batch, int n_q_heads,
                         int n_kv_heads, int head_dim, ia_stream_t stream) {
  if (!qkv || !cos_table || !sin_table || !seq_lens || !k_cache || !v_cache || !q_out)
    return fail(IA_ERR_BAD_ARG, "rope_append: null pointer");
  if (batch < 0 || n_q_heads <= 0 || n_kv_heads <= 0 || max_pos <= 0 || cache_len <= 0)
    return fail(IA_ERR_BAD_ARG, "rope_append: batch %d, heads %d/%d, %d positions, cache of %d", batch, n_q_heads,
                n_kv_heads, max_pos, cache_len);
  if (head_dim <= 0 || head_dim % 2 != 0 || head_dim > 2048)
    return fail(IA_ERR_UNSUPPORTED, "rope_append: head_dim %d (even, at most 2048)", head_dim);
  if (cache_head_stride < (int64_t)cache_len * head_dim)
    return fail(IA_ERR_BAD_ARG, "rope_append: head stride %lld below %d rows of %d", (long long)cache_head_stride,
                cache_len, head_dim);
  if (batch == 0) return IA_OK;
  const dim3 grid((unsigned)batch, (unsigned)(n_q_heads + 2 * n_kv_heads)), block((unsigned)(head_dim / 2));
  return launch("llama_rope_append_kernel", llama_rope_append_kernel, grid, block, (cudaStream_t)stream,
                static_cast<const __nv_bfloat16*>(qkv), static_cast<const __nv_bfloat16*>(cos_table),
                static_cast<const __nv_bfloat16*>(sin_table), max_pos, seq_lens, static_cast<__nv_bfloat16*>(k_cache),
                static_cast<__nv_bfloat16*>(v_cache), cache_seq_stride, cache_head_stride, cache_len,
                static_cast<__nv_bfloat16*>(q_out), n_q_heads, n_kv_heads, head_dim);
}

int ia_llama_silu_mul(const void* gate_up, void* out, int n_rows, int intermediate, ia_stream_t stream) {
  if (!gate_up || !out) return fail(IA_ERR_BAD_ARG, "silu_mul: null pointer");
  if (n_rows < 0 || intermediate <= 0 || intermediate % 8 != 0)
    return fail(IA_ERR_BAD_ARG, "silu_mul: %d rows of %d (a multiple of 8)", n_rows, intermediate);
  if (!aligned16(gate_up) || !aligned16(out)) return fail(IA_ERR_BAD_ARG, "silu_mul: pointers must be 16-byte aligned");
  if (n_rows == 0) return IA_OK;
  const int64_t units = (int64_t)n_rows * (intermediate / 8);
  const dim3 grid((unsigned)ceil_div64(units, 256)), block(256);
  return launch("llama_silu_mul_kernel", llama_silu_mul_kernel, grid, block, (cudaStream_t)stream,
                static_cast<const __nv_bfloat16*>(gate_up), static_cast<__nv_bfloat16*>(out), n_rows, intermediate);
}

int ia_llama_argmax(const void* logits, int64_t row_stride, int n_rows, int vocab, int64_t* out, ia_stream_t stream) {
  if (!logits || !out) return fail(IA_ERR_BAD_ARG, "argmax: null pointer");
  if (n_rows < 0 || vocab <= 0 || row_stride < vocab)
    return fail(IA_ERR_BAD_ARG, "argmax: %d rows of %d, row stride %lld", n_rows, vocab, (long long)row_stride);
  if (n_rows == 0) return IA_OK;
  // rows that start off a 16-byte boundary take the scalar loop
  const dim3 grid((unsigned)n_rows), block(kArgmaxThreads);
  return launch("llama_argmax_kernel", llama_argmax_kernel, grid, block, (cudaStream_t)stream,
                static_cast<const __nv_bfloat16*>(logits), row_stride, vocab, out);
}

static int parts_view(const void* parts, int n, int k, PartsView* out) {
  if (!parts || !aligned16(parts)) return fail(IA_ERR_BAD_ARG, "parts: null or not 16-byte aligned");
  if (n <= 0 || k <= 0) return fail(IA_ERR_BAD_ARG, "parts: n %d, k %d", n, k);
  const GemmSplit s = gemm_split(n, k);
  if (s.total == 0) return fail(IA_ERR_UNSUPPORTED, "parts: %d x %d is too large", n, k);
  *out = PartsView{static_cast<const float*>(parts), (uint32_t)s.k_chunks, (uint32_t)s.total, (uint32_t)s.ctas};
  return IA_OK;
}

int ia_llama_add_rmsnorm_parts(void* residual, const void* parts, int k, const void* weight, void* out, int n_rows,
                               int hidden, float eps, ia_stream_t stream) {
  if (!residual || !weight || !out) return fail(IA_ERR_BAD_ARG, "add_rmsnorm_parts: null pointer");
  if (n_rows < 0 || n_rows > kPartRows || hidden <= 0 || hidden % 8 != 0)
    return fail(IA_ERR_BAD_ARG, "add_rmsnorm_parts: %d rows of %d (a multiple of 8)", n_rows, hidden);
  if (!aligned16(residual) || !aligned16(weight) || !aligned16(out))
    return fail(IA_ERR_BAD_ARG, "add_rmsnorm_parts: pointers must be 16-byte aligned");
  PartsView v;
  if (int s = parts_view(parts, hidden, k, &v)) return s;
  if (n_rows == 0) return IA_OK;
  auto* r = static_cast<__nv_bfloat16*>(residual);
  auto* w = static_cast<const __nv_bfloat16*>(weight);
  auto* o = static_cast<__nv_bfloat16*>(out);
  const char* what = "llama_add_rmsnorm_parts_kernel";
  const dim3 grid((unsigned)n_rows), block(kPartNormThreads);
  cudaStream_t st = (cudaStream_t)stream;
  switch ((hidden + kPartNormThreads * 8 - 1) / (kPartNormThreads * 8)) {
    case 1: return launch(what, llama_add_rmsnorm_parts_kernel<1>, grid, block, st, r, v, w, o, hidden, eps);
    case 2: return launch(what, llama_add_rmsnorm_parts_kernel<2>, grid, block, st, r, v, w, o, hidden, eps);
    case 3:
    case 4: return launch(what, llama_add_rmsnorm_parts_kernel<4>, grid, block, st, r, v, w, o, hidden, eps);
    default: return fail(IA_ERR_UNSUPPORTED, "add_rmsnorm_parts: hidden size %d above %d", hidden, kPartNormThreads * 32);
  }
}

int ia_llama_rope_append_parts(const void* parts, int k, const void* cos_table, const void* sin_table, int max_pos,
                               const int32_t* seq_lens, void* k_cache, void* v_cache, int64_t cache_seq_stride,
                               int64_t cache_head_stride, int cache_len, void* q_out, int batch, int n_q_heads,
                               int n_kv_heads, int head_dim, ia_stream_t stream) {
  if (!cos_table || !sin_table || !seq_lens || !k_cache || !v_cache || !q_out)
    return fail(IA_ERR_BAD_ARG, "rope_append_parts: null pointer");
  if (batch < 0 || batch > kPartRows || n_q_heads <= 0 || n_kv_heads <= 0 || max_pos <= 0 || cache_len <= 0)
    return fail(IA_ERR_BAD_ARG, "rope_append_parts: batch %d, heads %d/%d, %d positions, cache of %d", batch, n_q_heads,
                n_kv_heads, max_pos, cache_len);
  if (head_dim <= 0 || head_dim % 8 != 0 || head_dim > 2048)
    return fail(IA_ERR_UNSUPPORTED, "rope_append_parts: head_dim %d (a multiple of 8, at most 2048)", head_dim);
  if (cache_head_stride < (int64_t)cache_len * head_dim || cache_head_stride % 4 != 0 || cache_seq_stride % 4 != 0)
    return fail(IA_ERR_BAD_ARG, "rope_append_parts: cache strides %lld, %lld for %d rows of %d", (long long)cache_seq_stride,
                (long long)cache_head_stride, cache_len, head_dim);
  if ((reinterpret_cast<uintptr_t>(cos_table) | reinterpret_cast<uintptr_t>(sin_table) |
       reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) | reinterpret_cast<uintptr_t>(q_out)) & 7u)
    return fail(IA_ERR_BAD_ARG, "rope_append_parts: pointers must be 8-byte aligned");
  const int64_t n = (int64_t)(n_q_heads + 2 * n_kv_heads) * head_dim;
  if (n > 0x7fffffff) return fail(IA_ERR_UNSUPPORTED, "rope_append_parts: %lld columns", (long long)n);
  PartsView v;
  if (int s = parts_view(parts, (int)n, k, &v)) return s;
  if (batch == 0) return IA_OK;
  const dim3 grid((unsigned)ceil_div64((int64_t)batch * (n / 8), 128)), block(128);
  return launch("llama_rope_append_parts_kernel", llama_rope_append_parts_kernel, grid, block, (cudaStream_t)stream, v,
                static_cast<const __nv_bfloat16*>(cos_table), static_cast<const __nv_bfloat16*>(sin_table), max_pos,
                seq_lens, static_cast<__nv_bfloat16*>(k_cache), static_cast<__nv_bfloat16*>(v_cache), cache_seq_stride,
                cache_head_stride, cache_len, static_cast<__nv_bfloat16*>(q_out), batch, n_q_heads, n_kv_heads, head_dim);
}

int ia_llama_silu_mul_parts(const void* parts, int k, void* out, int n_rows, int intermediate, ia_stream_t stream) {
  if (!out || !aligned16(out)) return fail(IA_ERR_BAD_ARG, "silu_mul_parts: null or misaligned out");
  if (n_rows < 0 || n_rows > kPartRows || intermediate <= 0 || intermediate % 8 != 0 || intermediate > 0x3fffffff)
    return fail(IA_ERR_BAD_ARG, "silu_mul_parts: %d rows of %d (a multiple of 8)", n_rows, intermediate);
  PartsView v;
  if (int s = parts_view(parts, 2 * intermediate, k, &v)) return s;
  if (n_rows == 0) return IA_OK;
  const dim3 grid((unsigned)ceil_div64((int64_t)n_rows * (intermediate / 8), 256)), block(256);
  return launch("llama_silu_mul_parts_kernel", llama_silu_mul_parts_kernel, grid, block, (cudaStream_t)stream, v,
                static_cast<__nv_bfloat16*>(out), n_rows, intermediate);
}

int ia_llama_argmax_parts(const void* parts, int k, void* logits, int n_rows, int vocab, int64_t* out,
                          ia_stream_t stream) {
  if (!logits || !out || (reinterpret_cast<uintptr_t>(logits) & 7u)) return fail(IA_ERR_BAD_ARG, "argmax_parts: null or misaligned pointer");
  if (n_rows < 0 || n_rows > kPartRows || vocab <= 0) return fail(IA_ERR_BAD_ARG, "argmax_parts: %d rows of %d", n_rows, vocab);
  PartsView v;
  if (int s = parts_view(parts, vocab, k, &v)) return s;
  if (n_rows == 0) return IA_OK;
  const dim3 grid((unsigned)(n_rows * kArgmaxCluster)), block(kArgmaxPartsThreads);
  return launch("llama_argmax_parts_kernel", llama_argmax_parts_kernel, grid, block, (cudaStream_t)stream, v,
                static_cast<__nv_bfloat16*>(logits), vocab, out);
}

}  // extern "C"
