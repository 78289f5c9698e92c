// Paged grouped-query attention for any mixture of prompt portions and decode tokens:
// the general kernel of the 32-bit path, and the reference shape for the faster ones.
//
// For query token t of request s at absolute position p, head h (kv head g = h / group):
//   score_j = (q . k_j) * scale  for j in [lo, p],  lo = window > 0 ? max(0, p - window + 1) : 0
//   out = softmax(score) . v                         (src/operators.cpp:102-146)
// Causality comes from attending only to positions <= p, exactly as the reference attends
// to the first position+1 cache entries (src/model.cpp:159-169).  Keys and values are read
// through the request's block table from pages laid out
// [page][2 (k, v)][kv head][slot][head_dim].
//
// One warp owns one (token, head) pair and walks the keys in ascending order, 32 at a
// time, with a running maximum and sum in 32-bit.  The order of operations for a row
// depends only on the row's own position, never on the batch, so the 32-bit path gives
// bit-identical rows however the tokens were cut into steps.
//
// 32-bit rows of head size 64 or 128 without a window run on a second kernel with the same order of operations: a CTA owns one
// kv head and a run of rows, so that the query heads of the group and the neighbouring rows share every key and value,
// which the CTA copies to shared memory 32 keys at a time while it works on the 32 before.
#include "common.cuh"
#include "mma_utils.cuh"
#include "shared_memory_limit.cuh"

namespace tlie {

constexpr int kMaxHeadDim = 256;
constexpr int kWarpsPerBlock = 4;

template <typename T>
__global__ void paged_attention_generic_kernel(const T* __restrict__ q, int q_row_stride, const T* __restrict__ pages,
                                               const int* __restrict__ positions, const int* __restrict__ token_seq,
                                               const int* __restrict__ block_table, int table_stride,
                                               T* __restrict__ out, int tokens, int q_heads, int kv_heads,
                                               int head_dim, int page_size, int window, float scale) {
  __shared__ float q_smem[kWarpsPerBlock][kMaxHeadDim];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const long long pair = (long long)blockIdx.x * kWarpsPerBlock + warp;
  if (pair >= (long long)tokens * q_heads) return;
  const int t = (int)(pair / q_heads);
  const int h = (int)(pair - (long long)t * q_heads);
  const int g = h / (q_heads / kv_heads);
  const int pos = positions[t];
  const int* table = block_table + (size_t)token_seq[t] * table_stride;

  const T* q_row = q + (size_t)t * q_row_stride + (size_t)h * head_dim;
  for (int d = lane; d < head_dim; d += 32) q_smem[warp][d] = to_float(q_row[d]);
  __syncwarp();

  const size_t plane = (size_t)kv_heads * page_size * head_dim;
  const size_t head_offset = (size_t)g * page_size * head_dim;
  const int dims_per_lane = (head_dim + 31) / 32;

  float acc[kMaxHeadDim / 32];
#pragma unroll
  for (int i = 0; i < kMaxHeadDim / 32; ++i) acc[i] = 0.0f;
  float running_max = -INFINITY;
  float running_sum = 0.0f;

  const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  for (int base = lo; base <= pos; base += 32) {
    const int key = base + lane;
    const bool valid = key <= pos;
    float score = -INFINITY;
    if (valid) {
      const int page = table[key / page_size];
      const T* k_row = pages + (size_t)page * 2 * plane + head_offset + (size_t)(key % page_size) * head_dim;
      float dot = 0.0f;
      for (int d = 0; d < head_dim; ++d) dot += q_smem[warp][d] * to_float(k_row[d]);
      score = dot * scale;
    }
    const float chunk_max = warp_max(score);
    const float new_max = fmaxf(running_max, chunk_max);
    const float rescale = expf(running_max - new_max);  // exp(-inf) = 0 on the first chunk
    const float p = valid ? expf(score - new_max) : 0.0f;
    running_sum = running_sum * rescale + warp_sum(p);
    running_max = new_max;
#pragma unroll
    for (int i = 0; i < kMaxHeadDim / 32; ++i) acc[i] *= rescale;
    const int count = min(32, pos - base + 1);
    for (int j = 0; j < count; ++j) {
      const float pj = __shfl_sync(0xffffffffu, p, j);
      const int kj = base + j;
      const int page = table[kj / page_size];
      const T* v_row = pages + (size_t)page * 2 * plane + plane + head_offset + (size_t)(kj % page_size) * head_dim;
#pragma unroll
      for (int i = 0; i < kMaxHeadDim / 32; ++i) {
        const int d = lane + 32 * i;
        if (i < dims_per_lane && d < head_dim) acc[i] += pj * to_float(v_row[d]);
      }
    }
  }
  T* o_row = out + (size_t)t * q_heads * head_dim + (size_t)h * head_dim;
  const float inv = 1.0f / running_sum;
#pragma unroll
  for (int i = 0; i < kMaxHeadDim / 32; ++i) {
    const int d = lane + 32 * i;
    if (i < dims_per_lane && d < head_dim) o_row[d] = from_float<T>(acc[i] * inv);
  }
}


// --- the 32-bit kernel over shared keys and values ------------------------------------------------------
constexpr int kSharedWarps = 8;
constexpr int kSharedKeys = 32;
constexpr int kSharedStages = 3;

template <int HEAD_DIM, int SLOTS>
struct SharedAttention {
  static constexpr int kStride = HEAD_DIM + 4;   // eight rows' 16-byte reads fall into different banks
  static constexpr int kPlane = kSharedKeys * kStride;
  static constexpr int kSmem = (kSharedStages * 2 * kPlane + kSharedWarps * SLOTS * HEAD_DIM) * (int)sizeof(float);
};

// A warp owns SLOTS (row, head) pairs: pair slot * 8 + warp of the CTA's `rows_per_tile` rows x group heads.  Rounding is spelled out
// (no contraction left to the compiler), so that every build of the kernel gives a row the same bits.
template <int HEAD_DIM, int SLOTS>
__global__ void __launch_bounds__(kSharedWarps * 32) paged_attention_shared_f32_kernel(
    const float* __restrict__ q, int q_row_stride, const float* __restrict__ pages, const int* __restrict__ positions, const int* __restrict__ token_seq,
    const int* __restrict__ block_table, int table_stride, float* __restrict__ out, int tokens, int q_heads, int kv_heads, int page_size, float scale,
    int rows_per_tile) {
  using Shape = SharedAttention<HEAD_DIM, SLOTS>;
  extern __shared__ __align__(16) float smem[];
  float* qs = smem + kSharedStages * 2 * Shape::kPlane;   // [slot * 8 + warp][HEAD_DIM]
  constexpr int kQuads = HEAD_DIM / 4, kDims = HEAD_DIM / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = q_heads / kv_heads;
  const int g = blockIdx.y;
  const int t0 = blockIdx.x * rows_per_tile, t1 = min(tokens, t0 + rows_per_tile);
  const size_t plane = (size_t)kv_heads * page_size * HEAD_DIM;
  const float* head_pages = pages + (size_t)g * page_size * HEAD_DIM;
  const int page_shift = (page_size & (page_size - 1)) == 0 ? 31 - __clz(page_size) : -1;   // pages of a power of two: no division

  int row[SLOTS], head[SLOTS], pos[SLOTS];
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    const int pair = s * kSharedWarps + warp;
    row[s] = t0 + pair / group;
    head[s] = g * group + pair % group;
    const bool live = row[s] < t1;
    pos[s] = live ? positions[row[s]] : -1;
    float* mine = qs + pair * HEAD_DIM;
    for (int d = lane; d < HEAD_DIM; d += 32) mine[d] = live ? q[(size_t)row[s] * q_row_stride + (size_t)head[s] * HEAD_DIM + d] : 0.0f;
  }

  // the rows of one request at a time (a tile may reach into the next request's rows)
  for (int first = t0; first < t1;) {
    const int entry = token_seq[first];
    int last = first, longest = positions[first];
    while (last + 1 < t1 && token_seq[last + 1] == entry) longest = max(longest, positions[++last]);
    const int* table = block_table + (size_t)entry * table_stride;
    const int chunks = longest / kSharedKeys + 1;
    // A thread's pieces of a chunk lie in pages that it has looked up a chunk before: the table's answer is a trip to L2, and a copy that waited for it held every warp up in every
    // chunk (four requests of 250 keys, 32 heads of 64 over 4: 17.3 us a launch).
    constexpr int kPieces = kSharedKeys * kQuads / (kSharedWarps * 32);
    int page[kPieces];
    auto key_of = [&](int chunk, int i) { return chunk * kSharedKeys + ((int)threadIdx.x + i * kSharedWarps * 32) / kQuads; };
    auto look_up = [&](int chunk) {
#pragma unroll
      for (int i = 0; i < kPieces; ++i) {
        const int at = key_of(chunk, i);
        page[i] = at <= longest ? table[page_shift >= 0 ? at >> page_shift : at / page_size] : 0;
      }
    };
    auto copy = [&](int chunk) {   // whose pages have been looked up; then the next one's are
      float* stage = smem + (chunk % kSharedStages) * 2 * Shape::kPlane;
#pragma unroll
      for (int i = 0; i < kPieces; ++i) {
        const int at = key_of(chunk, i), key = at - chunk * kSharedKeys, d = ((int)threadIdx.x + i * kSharedWarps * 32) % kQuads * 4;
        const bool seen = at <= longest;   // keys past the last one are zeros: nobody wrote them
        const int in_page = page_shift >= 0 ? at & (page_size - 1) : at % page_size;
        const float* source = seen ? head_pages + (size_t)page[i] * 2 * plane + (size_t)in_page * HEAD_DIM + d : pages;
        cp_async_16(stage + key * Shape::kStride + d, source, seen);
        cp_async_16(stage + Shape::kPlane + key * Shape::kStride + d, seen ? source + plane : pages, seen);
      }
      look_up(chunk + 1);
    };
    __syncthreads();   // everyone is done with the last request's stages
    look_up(0);
    for (int c = 0; c < kSharedStages - 1; ++c) {
      if (c < chunks) copy(c);
      cp_async_commit();
    }
    bool active[SLOTS];
    bool any = false;
    float running_max[SLOTS], running_sum[SLOTS], acc[SLOTS][kDims];
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      active[s] = row[s] >= first && row[s] <= last;
      any = any || active[s];
      running_max[s] = -INFINITY;
      running_sum[s] = 0.0f;
#pragma unroll
      for (int i = 0; i < kDims; ++i) acc[s][i] = 0.0f;
    }
    for (int c = 0; c < chunks; ++c) {
      cp_async_wait<kSharedStages - 2>();
      __syncthreads();
      if (c + kSharedStages - 1 < chunks) copy(c + kSharedStages - 1);
      cp_async_commit();
      if (!any) continue;
      const float* ks = smem + (c % kSharedStages) * 2 * Shape::kPlane + lane * Shape::kStride;
      const float* vs = smem + (c % kSharedStages) * 2 * Shape::kPlane + Shape::kPlane + lane;
      float dot[SLOTS];
#pragma unroll
      for (int s = 0; s < SLOTS; ++s) dot[s] = 0.0f;
#pragma unroll 8
      for (int i = 0; i < kQuads; ++i) {
        const float4 k = *reinterpret_cast<const float4*>(ks + 4 * i);
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) {
          const float4 v = *reinterpret_cast<const float4*>(qs + (s * kSharedWarps + warp) * HEAD_DIM + 4 * i);
          dot[s] = fmaf(v.w, k.w, fmaf(v.z, k.z, fmaf(v.y, k.y, fmaf(v.x, k.x, dot[s]))));
        }
      }
      const int base = c * kSharedKeys;
      float p[SLOTS];
      int count = kSharedKeys;   // keys of this chunk that all of the warp's rows see
#pragma unroll
      for (int s = 0; s < SLOTS; ++s) {
        const bool seen = active[s] && base + lane <= pos[s];
        const float score = seen ? __fmul_rn(dot[s], scale) : -INFINITY;
        const float new_max = fmaxf(running_max[s], warp_max(score));
        const float rescale = (active[s] && base <= pos[s]) ? expf(__fsub_rn(running_max[s], new_max)) : 1.0f;
        p[s] = seen ? expf(__fsub_rn(score, new_max)) : 0.0f;
        running_sum[s] = fmaf(running_sum[s], rescale, warp_sum(p[s]));
        running_max[s] = new_max;
#pragma unroll
        for (int i = 0; i < kDims; ++i) acc[s][i] = __fmul_rn(acc[s][i], rescale);
        count = min(count, active[s] ? pos[s] - base + 1 : 0);
      }
      if (count == kSharedKeys) {
#pragma unroll 8
        for (int j = 0; j < kSharedKeys; ++j) {
          float v[kDims];
#pragma unroll
          for (int i = 0; i < kDims; ++i) v[i] = vs[j * Shape::kStride + 32 * i];
#pragma unroll
          for (int s = 0; s < SLOTS; ++s) {
            const float pj = __shfl_sync(0xffffffffu, p[s], j);
#pragma unroll
            for (int i = 0; i < kDims; ++i) acc[s][i] = fmaf(pj, v[i], acc[s][i]);
          }
        }
      } else {   // a row takes only the values it sees: what lies past it may be anything, and 0 times that is not always 0
#pragma unroll
        for (int s = 0; s < SLOTS; ++s) {
          const int mine = active[s] ? min(kSharedKeys, pos[s] - base + 1) : 0;   // the same for the whole warp
          for (int j = 0; j < mine; ++j) {
            const float pj = __shfl_sync(0xffffffffu, p[s], j);
#pragma unroll
            for (int i = 0; i < kDims; ++i) acc[s][i] = fmaf(pj, vs[j * Shape::kStride + 32 * i], acc[s][i]);
          }
        }
      }
    }
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      if (!active[s]) continue;
      const float inv = 1.0f / running_sum[s];
#pragma unroll
      for (int i = 0; i < kDims; ++i)
        out[(size_t)row[s] * q_heads * HEAD_DIM + (size_t)head[s] * HEAD_DIM + lane + 32 * i] = acc[s][i] * inv;
    }
    first = last + 1;
  }
}

template <int HEAD_DIM, int SLOTS>
static int launch_shared(const float* q, int q_row_stride, const float* pages, const int* positions, const int* token_seq, const int* block_table,
                         int table_stride, float* out, int tokens, int q_heads, int kv_heads, int page_size, float scale, int rows_per_tile, cudaStream_t stream) {
  constexpr int smem = SharedAttention<HEAD_DIM, SLOTS>::kSmem;
  static std::atomic<unsigned long long> devices{0};
  const cudaError_t allowed = allow_shared_memory(paged_attention_shared_f32_kernel<HEAD_DIM, SLOTS>, smem, devices);
  if (allowed != cudaSuccess) return (int)allowed;
  paged_attention_shared_f32_kernel<HEAD_DIM, SLOTS><<<dim3((tokens + rows_per_tile - 1) / rows_per_tile, kv_heads), kSharedWarps * 32, smem, stream>>>(
      q, q_row_stride, pages, positions, token_seq, block_table, table_stride, out, tokens, q_heads, kv_heads, page_size, scale, rows_per_tile);
  return (int)cudaGetLastError();
}

}  // namespace tlie

using namespace tlie;

TLIE_EXPORT int tlie_paged_attention_generic(int dtype, const void* q, int q_row_stride, const void* pages,
                                             const int* positions, const int* token_seq, const int* block_table,
                                             int table_stride, void* out, int tokens, int q_heads, int kv_heads,
                                             int head_dim, int page_size, int window, float scale,
                                             cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (head_dim > kMaxHeadDim || head_dim <= 0 || kv_heads <= 0 || q_heads % kv_heads != 0)
    return (int)cudaErrorInvalidValue;
  const long long pairs = (long long)tokens * q_heads;
  const int blocks = (int)((pairs + kWarpsPerBlock - 1) / kWarpsPerBlock);
  if (dtype == TLIE_F32)
    paged_attention_generic_kernel<float><<<blocks, kWarpsPerBlock * 32, 0, stream>>>(
        (const float*)q, q_row_stride, (const float*)pages, positions, token_seq, block_table, table_stride,
        (float*)out, tokens, q_heads, kv_heads, head_dim, page_size, window, scale);
  else
    paged_attention_generic_kernel<__nv_bfloat16><<<blocks, kWarpsPerBlock * 32, 0, stream>>>(
        (const __nv_bfloat16*)q, q_row_stride, (const __nv_bfloat16*)pages, positions, token_seq, block_table,
        table_stride, (__nv_bfloat16*)out, tokens, q_heads, kv_heads, head_dim, page_size, window, scale);
  return (int)cudaGetLastError();
}

// The same for 32-bit rows of head size 64 or 128 without a window, 16-byte aligned pages, at most 32 query heads per kv head.  rows_per_tile: rows of a CTA
// (times the group at most 32).  A CTA works on the requests of its rows one after the other: who calls keeps a tile to few of them.
TLIE_EXPORT int tlie_paged_attention_shared_f32(const float* q, int q_row_stride, const float* pages, const int* positions, const int* token_seq,
                                                const int* block_table, int table_stride, float* out, int tokens, int q_heads, int kv_heads, int head_dim,
                                                int page_size, float scale, int rows_per_tile, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if ((head_dim != 64 && head_dim != 128) || kv_heads <= 0 || kv_heads > 65535 || q_heads % kv_heads != 0 || rows_per_tile < 1 ||
      (long long)rows_per_tile * (q_heads / kv_heads) > 4 * kSharedWarps || (reinterpret_cast<uintptr_t>(pages) & 15) != 0)
    return (int)cudaErrorInvalidValue;
  if (rows_per_tile * (q_heads / kv_heads) <= kSharedWarps)   // a pair per warp
    return head_dim == 64 ? launch_shared<64, 1>(q, q_row_stride, pages, positions, token_seq, block_table, table_stride, out, tokens, q_heads, kv_heads, page_size, scale, rows_per_tile, stream)
                          : launch_shared<128, 1>(q, q_row_stride, pages, positions, token_seq, block_table, table_stride, out, tokens, q_heads, kv_heads, page_size, scale, rows_per_tile, stream);
  return head_dim == 64 ? launch_shared<64, 4>(q, q_row_stride, pages, positions, token_seq, block_table, table_stride, out, tokens, q_heads, kv_heads, page_size, scale, rows_per_tile, stream)
                        : launch_shared<128, 4>(q, q_row_stride, pages, positions, token_seq, block_table, table_stride, out, tokens, q_heads, kv_heads, page_size, scale, rows_per_tile, stream);
}
