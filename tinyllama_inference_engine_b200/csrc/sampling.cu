// Token selection on the device: greedy argmax and temperature / top-p sampling.
//
// Greedy: the largest logit, the lowest id on ties (src/operators.cpp:166-175,
// tests/unit_tests.cpp:198-202).
// Temperature / top-p (app/server.cpp:237-277): p_i = exp((l_i - max) / T); keep the
// smallest set of most probable tokens whose share of the total reaches top_p (the token
// that crosses the line included); draw a point uniformly in the kept mass and return the
// token it falls on.  The reference sorts and walks the sorted list with a per-request
// mt19937; here the kept set is found by bisecting on the probability threshold (no sort),
// the walk is in token-id order, and the uniform number comes from a counter-based hash
// of (seed, draw index), so a request's draws do not depend on what else is in the batch.
// All arithmetic is 32-bit; one block owns one row, or a cluster of blocks a long one (see sample_kernel).
#include <cooperative_groups.h>

#include "common.cuh"

namespace tlie {

constexpr int kSampleThreads = 1024;

// A thread's share of a row's maximum and the lowest index that holds it (0x7fffffff: no value in its share can be compared).  Rows that allow it are read 16 bytes at a
// time, kInFlight loads in flight per thread: one block reads a whole row, so its time is the latency of its loads in turn.
template <int kInFlight = 4>
__device__ __forceinline__ void row_max_and_arg(const float* __restrict__ row, int vocab, float& best, int& arg) {
  auto take = [&](float v, int i) {
    if (v > best || (v == best && i < arg)) {
      best = v;
      arg = i;
    }
  };
  // what fills up the last loads: no value is taken from it, while -INFINITY would be the maximum of a row without any comparable value, at an index past the row
  const float nan = __int_as_float(0x7fffffff);
  if ((vocab & 3) == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
    const float4* row4 = reinterpret_cast<const float4*>(row);
    const int quads = vocab >> 2;
    const float4 nothing = make_float4(nan, nan, nan, nan);
    for (int q0 = threadIdx.x; q0 < quads; q0 += kInFlight * blockDim.x) {
      float4 v[kInFlight];
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) {
        const int q = q0 + u * blockDim.x;
        v[u] = q < quads ? row4[q] : nothing;
      }
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) {
        const int i = (q0 + u * blockDim.x) * 4;
        take(v[u].x, i);
        take(v[u].y, i + 1);
        take(v[u].z, i + 2);
        take(v[u].w, i + 3);
      }
    }
  } else {
    for (int i0 = threadIdx.x; i0 < vocab; i0 += kInFlight * blockDim.x) {
      float v[kInFlight];
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) v[u] = i0 + u * blockDim.x < vocab ? row[i0 + u * blockDim.x] : nan;
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) take(v[u], i0 + u * blockDim.x);
    }
  }
}

// The lowest index of a row's maximum, by one block; token 0 for a row without any comparable value.
// `temperature` (optional): rows above 0 are somebody else's; the kernel behind this one may then start early.
__global__ void __launch_bounds__(kSampleThreads) argmax_kernel(const float* __restrict__ logits, int vocab, const float* __restrict__ temperature,
                                                                int* __restrict__ out) {
  __shared__ float best_value[32];
  __shared__ int best_index[32];
  if (temperature != nullptr) {
    grid_launch_dependents();
    if (temperature[blockIdx.x] > 0.0f) return;
  }
  const float* row = logits + (size_t)blockIdx.x * vocab;
  float value = -INFINITY;
  int index = 0x7fffffff;
  row_max_and_arg(row, vocab, value, index);
  for (int offset = 16; offset > 0; offset >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, value, offset);
    const int oi = __shfl_xor_sync(0xffffffffu, index, offset);
    if (ov > value || (ov == value && oi < index)) {
      value = ov;
      index = oi;
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    best_value[warp] = value;
    best_index[warp] = index;
  }
  __syncthreads();
  if (warp == 0) {
    const int warps = (blockDim.x + 31) >> 5;
    value = lane < warps ? best_value[lane] : -INFINITY;
    index = lane < warps ? best_index[lane] : 0x7fffffff;
    for (int offset = 16; offset > 0; offset >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, value, offset);
      const int oi = __shfl_xor_sync(0xffffffffu, index, offset);
      if (ov > value || (ov == value && oi < index)) {
        value = ov;
        index = oi;
      }
    }
    if (lane == 0) out[blockIdx.x] = index == 0x7fffffff ? 0 : index;
  }
}

// splitmix64 finaliser over (seed, counter): the uniform number of draw `counter` of a request.
__host__ __device__ inline float uniform_from(unsigned long long seed, unsigned long long counter) {
  unsigned long long z = seed * 0x9E3779B97F4A7C15ull + (counter + 1ull) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z = z ^ (z >> 31);
  return (float)(z >> 40) * (1.0f / 16777216.0f);  // 24 bits -> [0, 1)
}

// Rows too long for sample_kernel, and rows so short that most of its registers would hold nothing: one block per row that works every probability out again in each pass.  temperature <= 0 means greedy for that row.
__global__ void __launch_bounds__(kSampleThreads)
    sample_simple_kernel(const float* __restrict__ logits, int vocab, const float* __restrict__ temperature,
                  const float* __restrict__ top_p, const long long* __restrict__ seeds,
                  const long long* __restrict__ counters, int* __restrict__ out) {
  __shared__ float scratch[32];
  __shared__ float prefix[kSampleThreads];
  __shared__ int chosen;
  const float* row = logits + (size_t)blockIdx.x * vocab;
  const float temp = temperature[blockIdx.x];

  float local_max = -INFINITY;
  int local_arg = 0x7fffffff;
  row_max_and_arg(row, vocab, local_max, local_arg);
  const float row_max = block_max(local_max, scratch);
  if (!(temp > 0.0f)) {
    // greedy: lowest id among the maxima
    __shared__ int arg_smem;
    if (threadIdx.x == 0) arg_smem = 0x7fffffff;
    __syncthreads();
    if (local_max == row_max) atomicMin(&arg_smem, local_arg);
    __syncthreads();
    // a row without any comparable value (all NaN) leaves no maximum: token 0, as argmax_kernel answers
    if (threadIdx.x == 0) out[blockIdx.x] = (arg_smem < 0 || arg_smem >= vocab) ? 0 : arg_smem;
    return;
  }
  const float inv_temp = 1.0f / temp;
  // contiguous slice of the row per thread, so that the walk is in token-id order
  const int per_thread = (vocab + blockDim.x - 1) / blockDim.x;
  const int begin = min(vocab, (int)threadIdx.x * per_thread);
  const int end = min(vocab, begin + per_thread);

  float sum = 0.0f;
  for (int i = begin; i < end; ++i) sum += expf((row[i] - row_max) * inv_temp);
  const float total = block_sum(sum, scratch);

  // Largest threshold tau with mass{p >= tau} >= top_p * total, by bisection on the bit
  // pattern of positive floats (monotone in value).  The kept set is {p >= tau}.
  float tau = 0.0f;
  const float want = top_p[blockIdx.x] * total;
  if (top_p[blockIdx.x] < 1.0f) {
    unsigned lo = 0u;                    // mass{p >= 0} = total >= want
    unsigned hi = __float_as_uint(1.0f) + 1u;  // p <= 1, so mass{p >= hi} = 0 < want
    while (hi - lo > 1u) {
      const unsigned mid = lo + (hi - lo) / 2u;
      const float threshold = __uint_as_float(mid);
      float mass = 0.0f;
      for (int i = begin; i < end; ++i) {
        const float p = expf((row[i] - row_max) * inv_temp);
        if (p >= threshold) mass += p;
      }
      mass = block_sum(mass, scratch);
      if (mass >= want) lo = mid; else hi = mid;
    }
    tau = __uint_as_float(lo);
  }
  float kept = 0.0f;
  for (int i = begin; i < end; ++i) {
    const float p = expf((row[i] - row_max) * inv_temp);
    if (p >= tau) kept += p;
  }
  prefix[threadIdx.x] = kept;
  __syncthreads();
  if (threadIdx.x == 0) {
    float running = 0.0f;
    for (int i = 0; i < blockDim.x; ++i) {  // exclusive scan in thread order
      const float v = prefix[i];
      prefix[i] = running;
      running += v;
    }
    scratch[0] = running;
    chosen = -1;
  }
  __syncthreads();
  const float kept_total = scratch[0];
  const float target = uniform_from((unsigned long long)seeds[blockIdx.x], (unsigned long long)counters[blockIdx.x]) * kept_total;
  // the slice whose [start, start + kept) holds the target walks its tokens
  const float start = prefix[threadIdx.x];
  if (kept > 0.0f && target >= start && target < start + kept) {
    float cursor = start;
    int pick = -1;
    for (int i = begin; i < end; ++i) {
      const float p = expf((row[i] - row_max) * inv_temp);
      if (p >= tau) {
        cursor += p;
        pick = i;
        if (target < cursor) break;
      }
    }
    atomicMax(&chosen, pick);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int pick = chosen;
    if (pick < 0) {  // rounding put the target past the last kept token: take the last kept one
      for (int i = vocab - 1; i >= 0 && pick < 0; --i)
        if (expf((row[i] - row_max) * inv_temp) >= tau) pick = i;
    }
    // non-finite logits can leave nothing kept at all; the answer must still be a token of the vocabulary
    out[blockIdx.x] = (pick < 0 || pick >= vocab) ? 0 : pick;
  }
}

// A cluster of CTAS blocks per row (one block up to 32,768 tokens, up to four), temperature <= 0 means greedy for that row.
//
// The bisection asks some thirty times how much probability lies above a threshold.  Bound by those questions' chain of sums, not by bytes: the row's
// probabilities stay in registers, 32 * CTAS per thread, so a question is that many comparisons and one sum over the block (and over the cluster through
// distributed shared memory).  Read and exponentiated again for every question by one block, 64 rows of 32,000 took 550 us and 4 rows of
// 128,256 took 800.
// Every sum keeps the simple kernel's order: 1,024 runs of consecutive tokens, one per thread of the cluster, added run by run, then 32 runs at a time, then
// those.  A token far down the tail has a probability near the rounding of the sums before it, so in another order one draw in a hundred that falls
// into a flat tail would be another token.
struct SampleShared {
  float exchange[2][32];                    // the warps' partial results of the whole cluster, double buffered: one barrier per exchange
  int arg_exchange[2][32];
  __align__(16) float prefix[kSampleThreads];
  float kept_total;
  int chosen, last_kept;                    // the first block's are the row's
};

// One row.  `parity`: which half of the exchange buffers comes next (from row to row).
template <int CTAS>
__device__ __forceinline__ void sample_row(SampleShared& shared, int& parity, int row_index, const float* __restrict__ logits, int vocab,
                                           const float* __restrict__ temperature, const float* __restrict__ top_p, const long long* __restrict__ seeds,
                                           const long long* __restrict__ counters, int* __restrict__ out) {
  namespace cg = cooperative_groups;
  constexpr int kThreads = kSampleThreads / CTAS, kWarps = kThreads / 32, kHeld = 32 * CTAS;
  auto& exchange = shared.exchange;
  auto& arg_exchange = shared.arg_exchange;
  auto& prefix = shared.prefix;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = CTAS > 1 ? (int)cluster.block_rank() : 0;
  const float* row = logits + (size_t)row_index * vocab;
  const float temp = temperature[row_index];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int run = rank * kThreads + (int)threadIdx.x;    // which of the 1,024 runs is this thread's
  auto sync_all = [&] {
    if (CTAS > 1) cluster.sync();
    else __syncthreads();
  };
  // this thread's view of all 32 warps' values, lane w holds warp w's
  auto all_warps = [&](float mine) {
    if (lane < CTAS) *(CTAS > 1 ? cluster.map_shared_rank(&exchange[parity][rank * kWarps + warp], lane) : &exchange[parity][warp]) = mine;
    sync_all();
    const float value = exchange[parity][lane];
    parity ^= 1;
    return value;
  };

  if (!(temp > 0.0f)) {
    // greedy: lowest id among the maxima.  Each block takes a quarter (or all) of the row in whole lines.
    const int each = ((vocab + CTAS - 1) / CTAS + 3) & ~3;
    const int first_id = min(vocab, rank * each), end_id = min(vocab, first_id + each);
    float value = -INFINITY;
    int index = 0x7fffffff;
    row_max_and_arg<4 * CTAS>(row + first_id, end_id - first_id, value, index);   // as many in flight per row as one block of all the threads has
    if (index != 0x7fffffff) index += first_id;
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, value, offset);
      const int oi = __shfl_xor_sync(0xffffffffu, index, offset);
      if (ov > value || (ov == value && oi < index)) {
        value = ov;
        index = oi;
      }
    }
    if (lane < CTAS) *(CTAS > 1 ? cluster.map_shared_rank(&arg_exchange[parity][rank * kWarps + warp], lane) : &arg_exchange[parity][warp]) = index;
    value = all_warps(value);
    index = arg_exchange[parity ^ 1][lane];
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, value, offset);
      const int oi = __shfl_xor_sync(0xffffffffu, index, offset);
      if (ov > value || (ov == value && oi < index)) {
        value = ov;
        index = oi;
      }
    }
    // a row without any comparable value (all NaN) leaves no maximum: token 0, as argmax_kernel answers
    if (rank == 0 && threadIdx.x == 0) out[row_index] = (index < 0 || index >= vocab) ? 0 : index;
    return;
  }

  const int per_run = (vocab + kSampleThreads - 1) / kSampleThreads;   // at most kHeld
  const int begin = min(vocab, run * per_run), count = min(vocab, begin + per_run) - begin;
  float p[kHeld];   // logits first, then probabilities
  float local_max = -INFINITY;
  if ((per_run & 3) == 0 && (vocab & 3) == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
#pragma unroll
    for (int i = 0; i < kHeld; i += 4) {
      const float4 v = i < count ? *reinterpret_cast<const float4*>(row + begin + i) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
      p[i] = v.x, p[i + 1] = v.y, p[i + 2] = v.z, p[i + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < kHeld; ++i) p[i] = i < count ? row[begin + i] : -INFINITY;
  }
#pragma unroll
  for (int i = 0; i < kHeld; ++i)
    if (i < count && p[i] > local_max) local_max = p[i];
  const float row_max = warp_max(all_warps(warp_max(local_max)));
  const float inv_temp = 1.0f / temp;
  float sum = 0.0f;
#pragma unroll
  for (int i = 0; i < kHeld; ++i)
    if (i < count) {
      p[i] = expf((p[i] - row_max) * inv_temp);
      sum += p[i];
    } else {
      p[i] = -1.0f;   // no token: never kept
    }
  const float total = warp_sum(all_warps(warp_sum(sum)));

  // Largest threshold tau with mass{p >= tau} >= top_p * total, by bisection on the bit
  // pattern of positive floats (monotone in value).  The kept set is {p >= tau}.
  float tau = 0.0f;
  if (top_p[row_index] < 1.0f) {
    const float want = top_p[row_index] * total;
    unsigned lo = 0u;                    // mass{p >= 0} = total >= want
    unsigned hi = __float_as_uint(1.0f) + 1u;  // p <= 1, so mass{p >= hi} = 0 < want
    while (hi - lo > 1u) {
      const unsigned mid = lo + (hi - lo) / 2u;
      const float threshold = __uint_as_float(mid);
      float mass = 0.0f;
#pragma unroll
      for (int i = 0; i < kHeld; ++i)
        if (p[i] >= threshold) mass += p[i];
      if (warp_sum(all_warps(warp_sum(mass))) >= want) lo = mid; else hi = mid;
    }
    tau = __uint_as_float(lo);
  }
  float kept = 0.0f;
  int last = -1;
#pragma unroll
  for (int i = 0; i < kHeld; ++i)
    if (p[i] >= tau) {
      kept += p[i];
      last = begin + i;
    }
  if (threadIdx.x == 0) shared.chosen = shared.last_kept = -1;
#pragma unroll
  for (int c = 0; c < CTAS; ++c) *(CTAS > 1 ? cluster.map_shared_rank(&prefix[run], c) : &prefix[run]) = kept;
  sync_all();
  if (threadIdx.x == 0) {   // exclusive scan in run order, in every block
    float running = 0.0f;
#pragma unroll 8
    for (int i = 0; i < kSampleThreads; i += 4) {
      const float4 v = *reinterpret_cast<const float4*>(prefix + i);
      float4 start;
      start.x = running;
      running += v.x;
      start.y = running;
      running += v.y;
      start.z = running;
      running += v.z;
      start.w = running;
      running += v.w;
      *reinterpret_cast<float4*>(prefix + i) = start;
    }
    shared.kept_total = running;
  }
  __syncthreads();
  const float target = uniform_from((unsigned long long)seeds[row_index], (unsigned long long)counters[row_index]) * shared.kept_total;
  // the run whose [start, start + kept) holds the target walks its tokens
  const float start = prefix[run];
  int* row_chosen = CTAS > 1 ? cluster.map_shared_rank(&shared.chosen, 0) : &shared.chosen;
  int* row_last = CTAS > 1 ? cluster.map_shared_rank(&shared.last_kept, 0) : &shared.last_kept;
  if (kept > 0.0f && target >= start && target < start + kept) {
    float cursor = start;
    int pick = -1;
    bool reached = false;
#pragma unroll
    for (int i = 0; i < kHeld; ++i)
      if (!reached && p[i] >= tau) {
        cursor += p[i];
        pick = begin + i;
        reached = target < cursor;
      }
    atomicMax(row_chosen, pick);
  }
  last = __reduce_max_sync(0xffffffffu, last);
  if (lane == 0) atomicMax(row_last, last);
  sync_all();
  if (rank == 0 && threadIdx.x == 0) {
    // rounding can put the target past the last kept token: take the last kept one; non-finite logits can leave nothing kept at all: the answer must
    // still be a token of the vocabulary
    const int pick = shared.chosen < 0 ? shared.last_kept : shared.chosen;
    out[row_index] = (pick < 0 || pick >= vocab) ? 0 : pick;
  }
}

// A cluster takes rows until there are none: its registers let one block run per SM, and of more clusters than the SMs hold each would start anew, ask for its
// row's temperature and wait.  What a row leaves in shared memory has been read when its cluster passes the next row's first barrier, and is written again behind that.
// sampled_only: the greedy rows are argmax_kernel's.
template <int CTAS>
__global__ void __launch_bounds__(kSampleThreads / CTAS)
    sample_kernel(const float* __restrict__ logits, int rows, int vocab, const float* __restrict__ temperature, const float* __restrict__ top_p,
                  const long long* __restrict__ seeds, const long long* __restrict__ counters, int* __restrict__ out, int sampled_only) {
  __shared__ SampleShared shared;
  int parity = 0;
  if (CTAS == 1) {
    sample_row<1>(shared, parity, blockIdx.x, logits, vocab, temperature, top_p, seeds, counters, out);
    return;
  }
  grid_dependency_wait();
  cooperative_groups::this_cluster().sync();   // a block's shared memory may be written once the block runs
  const int clusters = gridDim.x / CTAS, lane = threadIdx.x & 31;
  for (int first = blockIdx.x / CTAS; first < rows; first += 32 * clusters) {
    const int mine = first + lane * clusters;
    unsigned todo = __ballot_sync(0xffffffffu, mine < rows && (!sampled_only || temperature[mine] > 0.0f));
    for (; todo != 0u; todo &= todo - 1u)
      sample_row<CTAS>(shared, parity, first + (__ffs(todo) - 1) * clusters, logits, vocab, temperature, top_p, seeds, counters, out);
  }
}

// With more rows than clusters run at once, greedy ones go to argmax_kernel in front: a cluster's barriers cost as much as its part of such a row (us, all rows greedy, by the simple
// kernel, by a cluster each, so: 64 rows of 128,256 10.1, 10.9, 9.0; 256 rows 24.8, 66, 23.9; 100 rows of 50,304 5.6, about 7, 6.6; none greedy, 256 rows of 128,256: 1,405, 390, 370).
template <int CTAS>
static int launch_sample(const float* logits, int rows, int vocab, const float* temperature, const float* top_p, const long long* seeds, const long long* counters,
                         int* out, cudaStream_t stream) {
  cudaLaunchConfig_t config = {};
  config.blockDim = dim3(kSampleThreads / CTAS);
  config.stream = stream;
  if (CTAS == 1) {
    config.gridDim = dim3(rows);
    return (int)cudaLaunchKernelEx(&config, sample_kernel<CTAS>, logits, rows, vocab, temperature, top_p, seeds, counters, out, 0);
  }
  cudaLaunchAttribute attribute[2];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = CTAS;
  attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
  attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute;
  config.numAttrs = 1;
  config.gridDim = dim3(CTAS);   // (asked for a cluster's needs)
  static const int resident = [&config] {
    int clusters = 0;
    return cudaOccupancyMaxActiveClusters(&clusters, sample_kernel<CTAS>, &config) == cudaSuccess && clusters > 0 ? clusters : 1;
  }();
  const int sampled_only = rows > resident;
  if (sampled_only) {
    argmax_kernel<<<rows, kSampleThreads, 0, stream>>>(logits, vocab, temperature, out);
    config.numAttrs = 2;
  }
  config.gridDim = dim3((sampled_only ? resident : rows) * CTAS);
  return (int)cudaLaunchKernelEx(&config, sample_kernel<CTAS>, logits, rows, vocab, temperature, top_p, seeds, counters, out, sampled_only);
}

}  // namespace tlie

using namespace tlie;

TLIE_EXPORT int tlie_argmax(const float* logits, int rows, int vocab, int* out, cudaStream_t stream) {
  if (rows <= 0) return 0;
  argmax_kernel<<<rows, kSampleThreads, 0, stream>>>(logits, vocab, nullptr, out);
  return (int)cudaGetLastError();
}

// By the simple kernel, whatever the rows' length: the order of sums that the other kernels keep.
TLIE_EXPORT int tlie_sample_simple(const float* logits, int rows, int vocab, const float* temperature, const float* top_p,
                                   const long long* seeds, const long long* counters, int* out, cudaStream_t stream) {
  if (rows <= 0) return 0;
  sample_simple_kernel<<<rows, kSampleThreads, 0, stream>>>(logits, vocab, temperature, top_p, seeds, counters, out);
  return (int)cudaGetLastError();
}

TLIE_EXPORT int tlie_sample(const float* logits, int rows, int vocab, const float* temperature, const float* top_p,
                            const long long* seeds, const long long* counters, int* out, cudaStream_t stream) {
  if (rows <= 0) return 0;
  constexpr int kHeld = 32 * kSampleThreads;   // what a block's registers hold
  constexpr int kShort = 3 * kSampleThreads;   // (1,000 tokens: 25 us, 30 by the kernel with 32 places per thread; 3,000: 30 and 30.4; 4,096: 32 and 30)
  if (vocab <= kShort) return tlie_sample_simple(logits, rows, vocab, temperature, top_p, seeds, counters, out, stream);
  if (vocab <= kHeld) return launch_sample<1>(logits, rows, vocab, temperature, top_p, seeds, counters, out, stream);
  if (vocab <= 2 * kHeld) return launch_sample<2>(logits, rows, vocab, temperature, top_p, seeds, counters, out, stream);
  if (vocab <= 4 * kHeld) return launch_sample<4>(logits, rows, vocab, temperature, top_p, seeds, counters, out, stream);
  return tlie_sample_simple(logits, rows, vocab, temperature, top_p, seeds, counters, out, stream);
}

TLIE_EXPORT float tlie_uniform_from(long long seed, long long counter) {
  return uniform_from((unsigned long long)seed, (unsigned long long)counter);
}

// After a decode step: the sampled tokens become the next step's inputs and every request
// moves one position on.  Lets a run of decode steps stay on the device.
// `mailbox` (optional): pinned host memory of count + 2 words, written by this kernel over the bus: the sampled tokens, the device
// error word, and last (after a system-wide fence) the number of the step, which the host polls instead of asking the stream.
// One block: the block barrier orders every token's store before the number's.
__global__ void decode_advance_kernel(int* __restrict__ token_ids, const int* __restrict__ sampled,
                                      int* __restrict__ positions, int* __restrict__ seq_lens,
                                      int* __restrict__ first_positions, long long* __restrict__ counters, int count,
                                      volatile int* mailbox, const int* __restrict__ error_word, int* __restrict__ steps_done) {
  for (int i = threadIdx.x; i < count; i += blockDim.x) {
    const int token = sampled[i];
    token_ids[i] = token;
    positions[i] += 1;
    seq_lens[i] += 1;
    first_positions[i] += 1;
    counters[i] += 1;
    if (mailbox != nullptr) mailbox[i] = token;
  }
  if (mailbox == nullptr) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    mailbox[count] = error_word != nullptr ? *error_word : 0;
    const int number = *steps_done + 1;
    *steps_done = number;
    __threadfence_system();
    mailbox[count + 1] = number;
  }
}

// mailbox: null, or pinned host memory of count + 2 int32 (then steps_done: a device int32 that counts the steps; error_word may be null).
TLIE_EXPORT int tlie_decode_advance(int* token_ids, const int* sampled, int* positions, int* seq_lens,
                                    int* first_positions, long long* counters, int count, int* mailbox, const int* error_word,
                                    int* steps_done, cudaStream_t stream) {
  if (count <= 0) return 0;
  if (mailbox != nullptr && steps_done == nullptr) return (int)cudaErrorInvalidValue;
  decode_advance_kernel<<<1, count <= 128 ? 128 : 256, 0, stream>>>(token_ids, sampled, positions, seq_lens, first_positions, counters, count, mailbox,
                                                                    error_word, steps_done);
  return (int)cudaGetLastError();
}
