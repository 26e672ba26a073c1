// Everything the reference's _build_prompt_blocks returns for one sequence over a contiguous cache, in one pass
// (llama/script/analysis/condition_block_gen/methods/condition_block_triton_impl/core.py:449-500): the block
// summaries in their storage type and, where asked for, as fp32 copies; the zero-padded blocked copies of K and V;
// the token index, the valid mask and the per-block counts; the largest value norm of a head; and the identity
// block table and lengths by which the decode kernels address the cache.
#include "ia_common.cuh"

namespace ia {
namespace {

constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;
constexpr int kAuxPerCta = 2048;  // entries of the index arrays one of the trailing CTAs writes

// 16 bytes <-> floats
__device__ __forceinline__ void unpack16(const uint4& w, float (&v)[8]) {
  v[0] = bf16lo(w.x); v[1] = bf16hi(w.x); v[2] = bf16lo(w.y); v[3] = bf16hi(w.y);
  v[4] = bf16lo(w.z); v[5] = bf16hi(w.z); v[6] = bf16lo(w.w); v[7] = bf16hi(w.w);
}
__device__ __forceinline__ void unpack16(const uint4& w, float (&v)[4]) {
  v[0] = __uint_as_float(w.x); v[1] = __uint_as_float(w.y); v[2] = __uint_as_float(w.z); v[3] = __uint_as_float(w.w);
}

template <typename T>
struct PromptParams {
  const T* k;
  const T* v;
  ia_summaries s;
  ia_prompt_extras x;
  int64_t head_stride;
  int n_heads, n_blocks, block_size, length, flags;
};

// One CTA per (kv head, block), four warps that take a quarter of the block's tokens each.  What bounds it: HBM for
// long prompts (each K / V byte read once, the copies written once; the four-warp CTAs keep sixteen 16-byte loads
// per lane in flight), the launch for short ones.  A token row is read by D sizeof(T) / 16 lanes with 16 bytes each,
// so one warp load covers 2 tokens (head_dim 128 bf16) and a lane owns eight coordinates; the paged kernels'
// 8-byte lanes need twice the instructions, and their persistent 14-warp CTAs cover a 4099-token prompt
// (520 blocks) with 38 of the 148 SMs.  8 heads, 4099 tokens, head_dim 128 bf16: 6.7 us for all outputs, where the
// paged kernel took 13.2 us for the summaries alone and 23 small launches made the rest; the whole call 206 - 219 ->
// 77 us, most of it now the host's allocation of the output tensors.
template <typename T, int D>
__global__ void __launch_bounds__(kThreads) condition_block_prompt_blocks_kernel(const __grid_constant__ PromptParams<T> p) {
  constexpr int VEC = 16 / (int)sizeof(T);  // coordinates per lane
  constexpr int LPR = D / VEC;              // lanes per token row
  constexpr int TPL = 32 / LPR;             // token rows per warp load
  constexpr int ROUND = 8;                  // warp loads of K (and of V) in flight
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_units = p.n_heads * p.n_blocks;
  if ((int)blockIdx.x >= n_units) {
    // ---- the arrays that depend on the length alone ---------------------------------------------
    const int lo = ((int)blockIdx.x - n_units) * kAuxPerCta;
    const int n_tok = p.n_blocks * p.block_size;
    for (int i = lo + tid; i < lo + kAuxPerCta; i += kThreads) {
      if (i < n_tok) {
        p.x.token_idx[i] = i;
        p.x.valid_token[i] = i < p.length;
      }
      if (i < p.n_blocks) p.x.counts[i] = min(p.block_size, p.length - i * p.block_size);
      if (i < p.x.table_entries) p.x.table[i] = i;
      if (i == 0) {
        *p.x.prefix_len = p.length;
        *p.x.seq_len = p.length;
      }
    }
    return;
  }
  const int head = (int)blockIdx.x / p.n_blocks, blk = (int)blockIdx.x - head * p.n_blocks;
  const int64_t unit = blockIdx.x;  // [head][block]
  const int first = blk * p.block_size;
  const int count = min(p.block_size, p.length - first);  // at least 1
  const int sub = lane / LPR, col = (lane % LPR) * VEC;
  const int per_warp = p.block_size / kWarps;  // block_size is a multiple of 16
  const int t0 = warp * per_warp, t1 = t0 + per_warp;
  const T* kp = p.k + (int64_t)head * p.head_stride + (int64_t)first * D + col;
  const T* vp = p.v + (int64_t)head * p.head_stride + (int64_t)first * D + col;
  T* kd = p.x.k_block == nullptr ? nullptr : static_cast<T*>(p.x.k_block) + unit * p.block_size * D + col;
  T* vd = p.x.v_block == nullptr ? nullptr : static_cast<T*>(p.x.v_block) + unit * p.block_size * D + col;

  float ksum[VEC], vsum[VEC], kmax[VEC], kmin[VEC], vn2max = 0.f;
#pragma unroll
  for (int i = 0; i < VEC; ++i) { ksum[i] = 0.f; vsum[i] = 0.f; kmax[i] = -INFINITY; kmin[i] = INFINITY; }
  for (int base = t0; base < t1; base += ROUND * TPL) {
    uint4 kw[ROUND], vw[ROUND];
#pragma unroll
    for (int r = 0; r < ROUND; ++r) {
      const int t = base + r * TPL + sub;
      const bool live = t < t1 && t < count;
      kw[r] = live ? __ldg(reinterpret_cast<const uint4*>(kp + (int64_t)t * D)) : make_uint4(0u, 0u, 0u, 0u);
      vw[r] = live ? __ldg(reinterpret_cast<const uint4*>(vp + (int64_t)t * D)) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int r = 0; r < ROUND; ++r) {
      const int t = base + r * TPL + sub;
      if (kd != nullptr && t < t1) {  // rows past the prompt's end are zero, as in the reference
        *reinterpret_cast<uint4*>(kd + (int64_t)t * D) = kw[r];
        *reinterpret_cast<uint4*>(vd + (int64_t)t * D) = vw[r];
      }
      float kv[VEC], vv[VEC];
      unpack16(kw[r], kv);
      unpack16(vw[r], vv);
      const bool live = t < t1 && t < count;
      float sq = 0.f;
#pragma unroll
      for (int i = 0; i < VEC; ++i) sq = fmaf(vv[i], vv[i], sq);
      if (live) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          ksum[i] += kv[i];
          vsum[i] += vv[i];
          kmax[i] = fmaxf(kmax[i], kv[i]);
          kmin[i] = fminf(kmin[i], kv[i]);
        }
      }
#pragma unroll
      for (int o = 1; o < LPR; o <<= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      vn2max = fmaxf(vn2max, sq);  // a dead row adds 0
    }
  }
  // the token rows a warp holds side by side, then the four warps: pairwise, so the fp32 sums round less often on
  // the way than one sum in token order
#pragma unroll
  for (int o = LPR; o < 32; o <<= 1) {
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      ksum[i] += __shfl_xor_sync(0xffffffffu, ksum[i], o);
      vsum[i] += __shfl_xor_sync(0xffffffffu, vsum[i], o);
      kmax[i] = fmaxf(kmax[i], __shfl_xor_sync(0xffffffffu, kmax[i], o));
      kmin[i] = fminf(kmin[i], __shfl_xor_sync(0xffffffffu, kmin[i], o));
    }
    vn2max = fmaxf(vn2max, __shfl_xor_sync(0xffffffffu, vn2max, o));
  }
  __shared__ float part[4][kWarps][D];  // ksum, vsum, kmax, kmin
  __shared__ float norm[kWarps];
  if (sub == 0) {
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      part[0][warp][col + i] = ksum[i];
      part[1][warp][col + i] = vsum[i];
      part[2][warp][col + i] = kmax[i];
      part[3][warp][col + i] = kmin[i];
    }
  }
  if (lane == 0) norm[warp] = vn2max;
  __syncthreads();
  static_assert(D <= kThreads && kWarps == 4, "one thread per coordinate, four partial sums");
  if (tid < D) {
    const float denom = (float)count;
    const float kb = ((part[0][0][tid] + part[0][1][tid]) + (part[0][2][tid] + part[0][3][tid])) / denom;
    const float vb = ((part[1][0][tid] + part[1][1][tid]) + (part[1][2][tid] + part[1][3][tid])) / denom;
    const float hi = fmaxf(fmaxf(part[2][0][tid], part[2][1][tid]), fmaxf(part[2][2][tid], part[2][3][tid]));
    const float lo = fminf(fminf(part[3][0][tid], part[3][1][tid]), fminf(part[3][2][tid], part[3][3][tid]));
    const int64_t at = unit * D + tid;
    const float kb1[1] = {kb}, vb1[1] = {vb}, hi1[1] = {hi}, lo1[1] = {lo};
    if (p.flags & IA_GEOM_KBAR_BF16) store_vec<1>(reinterpret_cast<__nv_bfloat16*>(p.s.k_bar) + at, kb1);
    else p.s.k_bar[at] = kb;
    T* vbar = static_cast<T*>(p.s.v_bar);
    store_vec<1>(vbar + at, vb1);
    if (p.flags & IA_GEOM_PACKED_BOUNDS) {
      store_vec<1>(static_cast<T*>(p.s.k_max) + 2 * at, hi1);
      store_vec<1>(static_cast<T*>(p.s.k_max) + 2 * at + 1, lo1);
    } else {
      store_vec<1>(static_cast<T*>(p.s.k_max) + at, hi1);
      store_vec<1>(static_cast<T*>(p.s.k_min) + at, lo1);
    }
    // fp32 copies hold the stored (rounded) values
    if (p.x.v_bar_f32 != nullptr) p.x.v_bar_f32[at] = to_f32(vbar[at]);
    if (p.x.k_max_f32 != nullptr) p.x.k_max_f32[at] = hi;  // bounds are copies of K values: exact in either type
    if (p.x.k_min_f32 != nullptr) p.x.k_min_f32[at] = lo;
  }
  if (tid == 0) {
    const float n = sqrtf(fmaxf(fmaxf(norm[0], norm[1]), fmaxf(norm[2], norm[3])));
    p.s.v_norm_max[unit] = n;
    atomicMax(reinterpret_cast<int*>(p.x.v_norm_all) + head, __float_as_int(n));  // n >= 0: ordered like its bits
  }
}

template <typename T, int D>
int launch(const void* k, const void* v, int length, const ia_geom& g, const ia_summaries& s, const ia_prompt_extras& x,
           cudaStream_t stream) {
  PromptParams<T> p{};
  p.k = static_cast<const T*>(k);
  p.v = static_cast<const T*>(v);
  p.s = s;
  p.x = x;
  p.head_stride = g.pool_head_stride;
  p.n_heads = g.n_kv_heads;
  p.block_size = g.block_size;
  p.length = length;
  p.n_blocks = (length + g.block_size - 1) / g.block_size;
  p.flags = g.reserved;
  const int64_t entries = max((int64_t)p.n_blocks * g.block_size, (int64_t)max(x.table_entries, 1));
  const int64_t grid = (int64_t)p.n_heads * p.n_blocks + (entries + kAuxPerCta - 1) / kAuxPerCta;
  if (grid > 0x7fffffff) return fail(IA_ERR_UNSUPPORTED, "prompt_blocks: grid too large");
  const cudaError_t e = cudaMemsetAsync(x.v_norm_all, 0, (size_t)g.n_kv_heads * 4, stream);
  if (e != cudaSuccess) return fail(IA_ERR_LAUNCH, "prompt_blocks: cudaMemsetAsync: %s", cudaGetErrorString(e));
  condition_block_prompt_blocks_kernel<T, D><<<(unsigned)grid, kThreads, 0, stream>>>(p);
  return check_launch("condition_block_prompt_blocks_kernel");
}

}  // namespace

int launch_prompt_blocks(const void* k, const void* v, int length, const ia_geom& g, const ia_summaries& s,
                         const ia_prompt_extras& x, cudaStream_t stream) {
  if (g.dtype == IA_BF16) {
    if (g.head_dim == 128) return launch<__nv_bfloat16, 128>(k, v, length, g, s, x, stream);
    if (g.head_dim == 64) return launch<__nv_bfloat16, 64>(k, v, length, g, s, x, stream);
  } else if (g.dtype == IA_F32) {
    if (g.head_dim == 128) return launch<float, 128>(k, v, length, g, s, x, stream);
    if (g.head_dim == 64) return launch<float, 64>(k, v, length, g, s, x, stream);
  }
  return fail(IA_ERR_UNSUPPORTED, "prompt_blocks: head_dim %d / dtype %d not built", g.head_dim, g.dtype);
}

}  // namespace ia
