// Paged sparse / hybrid decode attention - portable fp32-FMA kernel.
//
// Attention half of the reference's fused finalize kernel
// (llama/script/analysis/condition_block_gen/methods/condition_block_triton_impl/page_attention.py:173-309):
// a joint online softmax over the tokens of the selected blocks, the
// representatives (z, v_bar) of the unselected blocks (hybrid mode) and the
// generated suffix, for the G query rows that share one kv head.  This
// translation unit holds the all-fp32 CUDA-core version: it serves fp32 KV
// pools (1e-5 parity against the fp32 reference) and any geometry the
// tensor-core kernel is not built for.  One warp walks whole pages.
#include "decode_items.cuh"

namespace ia {

int launch_sparse_decode_mma(const DecodeParams& p, const ia_geom& g, bool flat, cudaStream_t stream);  // bf16 tensor-core path

namespace {

constexpr int kWarps = 4;

// A warp takes a page (or a tile of 16 representatives) at a time, and what bounds it is latency: these calls are
// small (fp32 pools: 8 KB of K and V per page and kv head at head_dim 64), a few pages per warp.  So everything a
// page needs is in flight at once - two lanes per token read the K row for the logits, all lanes the V rows - and
// each step serves the 16 tokens together: one exchange joins a token's two half dots, the maximum takes four
// exchanges per query row, and the weights reach the lanes of the V product through shared memory.  One token after
// the other (a warp reduction and an exponential chain each) took 0.3 us per token.  Two fp32 sequences of 1024
// tokens, 4 pairs x 16 pages, head_dim 64: 19.7 -> 8.1 us, the step 28.7 -> 15.4 us (it also
// overlaps the selection kernel's end now, by programmatic launch).
template <typename T, int D, int G>
__global__ void __launch_bounds__(kWarps * 32)
condition_block_finalize_attention_fma_kernel(const __grid_constant__ DecodeParams p) {
  constexpr int VEC = D / 32;                      // V coordinates per lane
  constexpr int PIECE = 16 / (int)sizeof(T);       // elements of a 16-byte piece of a K row
  constexpr int PIECES = D / (2 * PIECE);          // pieces per lane: the two lanes of a token alternate
  constexpr int kTok = kRepTile;                   // tokens of a page = blocks of a representative tile
  __shared__ Item items_s[kItemChunk];
  __shared__ int scratch[2];
  __shared__ float merge_m[kWarps][G], merge_l[kWarps][G];
  __shared__ __align__(16) float merge_o[kWarps][G][D];
  // the query rows and the warps' weights lie where the warps' outputs are merged at the end
  float(&q_s)[G][D] = merge_o[0];
  float(&w_s)[kWarps][kTok][G] = reinterpret_cast<float(&)[kWarps][kTok][G]>(merge_o[1]);
  static_assert(kWarps * kTok <= (kWarps - 1) * D, "the weights fit behind the query rows");
  extern __shared__ uint32_t sel_bits[];  // hybrid: one bit per block

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int split = blockIdx.x % p.n_splits;
  const int pair = blockIdx.x / p.n_splits;
  const int head = pair % p.n_kv_heads, seq = pair / p.n_kv_heads;
  const int rows = p.n_kv_heads * G;
  grid_dependency_wait();  // the selection kernel wrote the index list, the counts and z
  grid_launch_dependents();

  ExchangeView xv{};
  if (p.px.n_ranks > 0) xv = exchange_view(p);
  const T* qp = static_cast<const T*>(p.q) + ((int64_t)seq * rows + head * G) * D;
  for (int i = threadIdx.x; i < G * D; i += kWarps * 32) q_s[i / D][i % D] = to_f32(qp[i]);
  const ItemRange r = item_range(p, seq, head, split, scratch);
  if (p.rep_mode == IA_REP_HYBRID) {
    const int words = (p.max_blocks + 31) / 32;
    for (int i = threadIdx.x; i < words; i += blockDim.x) sel_bits[i] = 0u;
    __syncthreads();
    const int count = min(p.sel_count[pair], p.max_sel);
    const int32_t* idx = p.sel_idx + (int64_t)pair * p.max_sel;
    for (int i = threadIdx.x; i < count; i += blockDim.x) {
      const int b = idx[i];
      if (b >= 0 && b < p.max_blocks) atomicOr(&sel_bits[b >> 5], 1u << (b & 31));
    }
    __syncthreads();
  }

  float acc[G][VEC], m[G], l[G];  // m: the warp's running maximum; l: this lane's share of the sum (even lanes)
#pragma unroll
  for (int g = 0; g < G; ++g) {
    m[g] = -INFINITY;
    l[g] = 0.f;
#pragma unroll
    for (int i = 0; i < VEC; ++i) acc[g][i] = 0.f;
  }
  const float root = sqrtf((float)D);
  const int tok = lane >> 1, half = lane & 1;
  const T* kp = static_cast<const T*>(p.k_pool) + (int64_t)head * p.head_stride + tok * D + half * PIECE;
  const T* vp = static_cast<const T*>(p.v_pool) + (int64_t)head * p.head_stride + lane * VEC;
  const T* vbar = static_cast<const T*>(p.v_bar) + ((int64_t)pair * p.max_blocks) * D + lane * VEC;
  const float* zrow = p.z + ((int64_t)seq * rows + head * G) * p.max_blocks;

  for (int chunk = r.begin; chunk < r.end; chunk += kItemChunk) {
    const int chunk_end = min(chunk + kItemChunk, r.end);
    __syncthreads();  // previous chunk fully consumed
    resolve_items(p, r, seq, head, chunk, chunk_end, items_s);
    for (int i = chunk + warp; i < chunk_end; i += kWarps) {
      const Item it = items_s[i - chunk];
      const bool page = it.kind == ITEM_PAGE;
      bool live = tok >= it.lo && tok < it.hi;  // dead rows are not read: they may hold anything
      if (!page && live) {
        const int b = it.first + tok;
        live = ((sel_bits[b >> 5] >> (b & 31)) & 1u) == 0u;  // selected: its tokens are attended exactly
      }
      const uint32_t live_tok = __ballot_sync(0xffffffffu, live);  // bit 2 t: token t
      const int64_t base = page ? (int64_t)it.first * p.page_stride : 0;
      const T* vrow = page ? vp + base : vbar + (int64_t)it.first * D;
      float v[kTok][VEC];
#pragma unroll
      for (int t = 0; t < kTok; ++t) {
        if ((live_tok >> (2 * t)) & 1u) {
          load_vec<VEC>(vrow + t * D, v[t]);
        } else {
#pragma unroll
          for (int j = 0; j < VEC; ++j) v[t][j] = 0.f;
        }
      }
      float logit[G];
      if (page) {
        uint4 kw[PIECES];
#pragma unroll
        for (int c = 0; c < PIECES; ++c)
          kw[c] = live ? *reinterpret_cast<const uint4*>(kp + base + c * 2 * PIECE) : make_uint4(0u, 0u, 0u, 0u);
        // eight short sums per row, joined pairwise: no product goes through more additions than in a reduction
        // tree over the warp, so the logits are as exact
#pragma unroll
        for (int g = 0; g < G; ++g) {
          float part[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int c = 0; c < PIECES; ++c) {
            float kv[PIECE];
            if constexpr (sizeof(T) == 4) {
              kv[0] = __uint_as_float(kw[c].x); kv[1] = __uint_as_float(kw[c].y);
              kv[2] = __uint_as_float(kw[c].z); kv[3] = __uint_as_float(kw[c].w);
            } else {
              kv[0] = bf16lo(kw[c].x); kv[1] = bf16hi(kw[c].x); kv[2] = bf16lo(kw[c].y); kv[3] = bf16hi(kw[c].y);
              kv[4] = bf16lo(kw[c].z); kv[5] = bf16hi(kw[c].z); kv[6] = bf16lo(kw[c].w); kv[7] = bf16hi(kw[c].w);
            }
            const int d0 = (2 * c + half) * PIECE;
#pragma unroll
            for (int j = 0; j < PIECE; j += 4) {
              const float4 qv = *reinterpret_cast<const float4*>(&q_s[g][d0 + j]);
              const int u = sizeof(T) == 4 ? 4 * (c & 1) : j;
              part[u] = fmaf(qv.x, kv[j], part[u]);
              part[u + 1] = fmaf(qv.y, kv[j + 1], part[u + 1]);
              part[u + 2] = fmaf(qv.z, kv[j + 2], part[u + 2]);
              part[u + 3] = fmaf(qv.w, kv[j + 3], part[u + 3]);
            }
          }
          float s = ((part[0] + part[4]) + (part[1] + part[5])) + ((part[2] + part[6]) + (part[3] + part[7]));
          s += __shfl_xor_sync(0xffffffffu, s, 1);
          logit[g] = live ? s / root : -INFINITY;
        }
      } else {
#pragma unroll
        for (int g = 0; g < G; ++g) logit[g] = live ? zrow[(int64_t)g * p.max_blocks + it.first + tok] : -INFINITY;
      }
      float a[G];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float top = logit[g];
#pragma unroll
        for (int x = 2; x < 32; x <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
        top = fmaxf(m[g], top);
        const float ref = top == -INFINITY ? 0.f : top;  // nothing live yet: every weight is 0
        a[g] = expf(m[g] - ref);
        const float w = expf(logit[g] - ref);
        m[g] = top;
        l[g] = l[g] * a[g] + w;
        if (half == 0) w_s[warp][tok][g] = w;
      }
      __syncwarp();
#pragma unroll
      for (int g = 0; g < G; ++g) {
#pragma unroll
        for (int j = 0; j < VEC; ++j) acc[g][j] *= a[g];
      }
#pragma unroll
      for (int t = 0; t < kTok; ++t) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
          const float w = w_s[warp][t][g];
#pragma unroll
          for (int j = 0; j < VEC; ++j) acc[g][j] = fmaf(w, v[t][j], acc[g][j]);
        }
      }
      __syncwarp();  // the weights may be overwritten
    }
  }
#pragma unroll
  for (int g = 0; g < G; ++g) {
    l[g] = half == 0 ? l[g] : 0.f;  // both lanes of a token counted it
    l[g] = warp_sum(l[g]);
  }
  __syncthreads();  // every warp is done with the query rows

  // ---- merge the four warps, emit (o, lse) ------------------------------------
#pragma unroll
  for (int g = 0; g < G; ++g) {
    if (lane == 0) { merge_m[warp][g] = m[g]; merge_l[warp][g] = l[g]; }
#pragma unroll
    for (int i = 0; i < VEC; ++i) merge_o[warp][g][lane * VEC + i] = acc[g][i];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < G * D; e += blockDim.x) {
    const int g = e / D, d = e - g * D;
    float top = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) top = fmaxf(top, merge_m[w][g]);
    float num = 0.f, den = 0.f;
    if (top > -INFINITY) {
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const float a = expf(merge_m[w][g] - top);
        num = fmaf(a, merge_o[w][g][d], num);
        den = fmaf(a, merge_l[w][g], den);
      }
    }
    const int64_t orow = ((int64_t)seq * rows + head * G + g) * p.n_splits + split;
    const float ov = den > 0.f ? num / den : 0.f;
    const float lv = den > 0.f ? top + logf(den) : -INFINITY;
    if (p.px.n_ranks > 0) {
      exchange_store(p, xv, orow * D + d, ov);
      if (d == 0) exchange_store(p, xv, p.px.lse_offset + orow, lv);
    } else {
      p.o_partial[orow * D + d] = ov;
      if (d == 0) p.lse_partial[orow] = lv;
    }
  }
  if (p.px.n_ranks > 0) {
    exchange_publish(p, xv);
    return;
  }
  finish_pair<D>(p, seq, head, G, scratch);
}

template <typename T, int D, int G>
int launch_fma(const DecodeParams& p, const ia_geom& g, cudaStream_t stream) {
  const int64_t grid = (int64_t)g.batch * g.n_kv_heads * p.n_splits;
  if (grid <= 0) return IA_OK;
  const size_t dyn = p.rep_mode == IA_REP_HYBRID ? (size_t)((g.max_blocks + 31) / 32) * 4 : 0;
  const cudaError_t e = launch_overlapped(condition_block_finalize_attention_fma_kernel<T, D, G>, (unsigned)grid,
                                          kWarps * 32, dyn, stream, p);
  if (e != cudaSuccess)
    return fail(IA_ERR_LAUNCH, "condition_block_finalize_attention_fma_kernel: %s", cudaGetErrorString(e));
  return check_launch("condition_block_finalize_attention_fma_kernel");
}

template <typename T, int D>
int launch_fma_group(const DecodeParams& p, const ia_geom& g, cudaStream_t stream) {
  switch (g.group_size) {
    case 1: return launch_fma<T, D, 1>(p, g, stream);
    case 2: return launch_fma<T, D, 2>(p, g, stream);
    case 4: return launch_fma<T, D, 4>(p, g, stream);
    case 8: return launch_fma<T, D, 8>(p, g, stream);
    default: return fail(IA_ERR_UNSUPPORTED, "sparse_decode (fma): group_size %d not built (1, 2, 4, 8)", g.group_size);
  }
}

}  // namespace

int launch_sparse_decode(const void* q, const void* k_pool, const void* v_pool,
                         const int32_t* block_table, const int32_t* prefix_lens,
                         const int32_t* seq_lens, const int32_t* sel_idx, const int32_t* sel_count,
                         int max_sel, const ia_summaries* summaries, const float* z, const ia_geom& g,
                         int rep_mode, int n_splits, int block_lo, int block_hi, int with_suffix,
                         float* o_partial, float* lse_partial, const FusedFinalize* fused, cudaStream_t stream,
                         const ia_peer_exchange* exchange) {
  DecodeParams p{};
  if (exchange != nullptr) p.px = *exchange;
  if (fused != nullptr) {
    p.final_out = fused->out;
    p.split_counters = fused->split_counters;
    p.final_dtype = fused->out_dtype;
    p.flat_o = fused->flat_o;
    p.flat_lse = fused->flat_lse;
  }
  p.n_pool_pages = g.n_pool_pages;
  p.status = device_status_address();
  p.n_pairs = g.batch * g.n_kv_heads;
#ifdef IA_DECODE_TRACE
  p.trace = getenv("IA_TRACE_PTR") ? reinterpret_cast<float*>(strtoull(getenv("IA_TRACE_PTR"), nullptr, 16)) : nullptr;
#endif
  p.q = q; p.k_pool = k_pool; p.v_pool = v_pool; p.block_table = block_table;
  p.prefix_lens = prefix_lens; p.seq_lens = seq_lens; p.suffix_lens = (g.reserved & IA_GEOM_SUFFIX_LENS) != 0; p.sel_idx = sel_idx; p.sel_count = sel_count;
  p.v_bar = summaries ? summaries->v_bar : nullptr;
  p.z = z;
  p.o_partial = o_partial; p.lse_partial = lse_partial;
  p.page_stride = g.pool_page_stride; p.head_stride = g.pool_head_stride;
  p.n_kv_heads = g.n_kv_heads; p.group_size = g.group_size; p.page_size = g.page_size;
  p.block_size = g.block_size; p.max_pages = g.max_pages; p.max_blocks = g.max_blocks; p.max_sel = max_sel;
  p.rep_mode = rep_mode; p.n_splits = n_splits; p.block_lo = block_lo; p.block_hi = block_hi;
  p.with_suffix = with_suffix;

  const char* force = getenv("INTERATTN_B200_DECODE_KERNEL");  // "fma" pins the portable kernel (profiling aid)
  const bool want_fma = force != nullptr && force[0] == 'f';
  if (g.dtype == IA_BF16 && g.page_size == 16 && g.group_size <= 16 && !want_fma &&
      (g.head_dim == 128 || g.head_dim == 64)) {
    const bool flat = p.flat_o != nullptr &&
                      decode_flat_grid_applies(g, fused != nullptr, block_lo <= 0 && block_hi >= g.max_blocks,
                                               exchange != nullptr);
    return launch_sparse_decode_mma(p, g, flat, stream);
  }
  if (g.dtype == IA_BF16) {
    if (g.head_dim == 128) return launch_fma_group<__nv_bfloat16, 128>(p, g, stream);
    if (g.head_dim == 64) return launch_fma_group<__nv_bfloat16, 64>(p, g, stream);
  } else if (g.dtype == IA_F32) {
    if (g.head_dim == 128) return launch_fma_group<float, 128>(p, g, stream);
    if (g.head_dim == 64) return launch_fma_group<float, 64>(p, g, stream);
  }
  return fail(IA_ERR_UNSUPPORTED, "sparse_decode: head_dim %d / dtype %d not built", g.head_dim, g.dtype);
}

}  // namespace ia
