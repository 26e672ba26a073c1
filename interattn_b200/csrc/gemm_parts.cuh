// How the row-major GEMM of the decode step (skinny_gemm.cu) cuts its work, and how the kernels that read the
// projection add up the partial sums it leaves (llama_step.cu).
#pragma once

#include "ia_common.cuh"

namespace ia {

constexpr int kPartRows = 16, kPartCols = 128;  // a slot: [16 token rows][128 output columns] fp32
constexpr int kPartChunk = 64;                  // columns of K per chunk

// Chunks of (128 rows of W) x (64 columns of K), K fastest; CTA c of P streams [T c / P, T (c + 1) / P).
struct GemmSplit { int k_chunks, total, ctas; };
// total = 0: too large for the 32-bit walk
inline GemmSplit gemm_split(int n, int k) {
  if (n <= 0 || k <= 0) return GemmSplit{0, 0, 0};
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
    sms = 148;
  const int64_t k_chunks = ((int64_t)k + kPartChunk - 1) / kPartChunk;
  const int64_t total = ((int64_t)n + kPartCols - 1) / kPartCols * k_chunks;
  if ((total + 1) * (sms + 1) > 0x7fffffff) return GemmSplit{0, 0, 0};
  return GemmSplit{(int)k_chunks, (int)total, (int)(total < sms ? total : sms)};
}

// The partial sums of a projection as its consumer sees them.
struct PartsView {
  const float* slots;
  uint32_t k_chunks, total, ctas;
  // CTA that streamed chunk x
  __device__ __forceinline__ uint32_t owner(uint32_t x) const { return ((x + 1) * ctas + total - 1) / total - 1; }
  // the slots of a tile of 128 columns: `count` of them, kPartRows * kPartCols floats apart, from the returned one
  __device__ __forceinline__ const float* tile(uint32_t t, int& count) const {
    const uint32_t first = owner(t * k_chunks), last = owner(t * k_chunks + k_chunks - 1);
    count = (int)(last - first) + 1;
    return slots + (int64_t)(first + t) * (kPartRows * kPartCols);
  }
};

// N consecutive columns (4 or 8, inside a tile, `at` a multiple of N) of one token row: the slots added in CTA order,
// rounded to bf16 as a finished projection is.  Up to kBatch slots are in flight together.
template <int N, int kBatch>
__device__ __forceinline__ void sum_parts(const float* tile, int count, int row, int at, float (&v)[N]) {
  const float* src = tile + row * kPartCols + at;
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = 0.f;
  for (int c0 = 0; c0 < count; c0 += kBatch) {
    float4 w[kBatch][N / 4];
#pragma unroll
    for (int c = 0; c < kBatch; ++c)
#pragma unroll
      for (int i = 0; i < N / 4; ++i)
        w[c][i] = c0 + c < count
                      ? __ldcg(reinterpret_cast<const float4*>(src + (int64_t)(c0 + c) * (kPartRows * kPartCols)) + i)
                      : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < kBatch; ++c)
#pragma unroll
      for (int i = 0; i < N / 4; ++i) {
        if (c0 + c < count) {
          v[4 * i] += w[c][i].x; v[4 * i + 1] += w[c][i].y; v[4 * i + 2] += w[c][i].z; v[4 * i + 3] += w[c][i].w;
        }
      }
  }
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = __bfloat162float(__float2bfloat16_rn(v[i]));
}

}  // namespace ia
