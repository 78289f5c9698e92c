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

// A thread's share of a row's maximum and the lowest index that holds it.  Rows that allow it are read 16 bytes at a
// time, four loads in flight per thread: one block reads a whole row, so its time is the latency of its loads in turn.
__device__ __forceinline__ void row_max_and_arg(const float* __restrict__ row, int vocab, float& best, int& arg) {
  auto take = [&](float v, int i) {
    if (v > best || (v == best && i < arg)) {
      best = v;
      arg = i;
    }
  };
  if ((vocab & 3) == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
    const float4* row4 = reinterpret_cast<const float4*>(row);
    const int quads = vocab >> 2;
    constexpr int kInFlight = 4;
    for (int q0 = threadIdx.x; q0 < quads; q0 += kInFlight * blockDim.x) {
      float4 v[kInFlight];
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) {
        const int q = q0 + u * blockDim.x;
        v[u] = q < quads ? row4[q] : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
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
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) take(row[i], i);
  }
}

__global__ void __launch_bounds__(kSampleThreads) argmax_kernel(const float* __restrict__ logits, int vocab,
                                                                int* __restrict__ out) {
  __shared__ float best_value[32];
  __shared__ int best_index[32];
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

// Rows too long for sample_kernel: one block per row that works every probability out again in each pass.  temperature <= 0 means greedy for that row.
__global__ void __launch_bounds__(kSampleThreads)
    sample_long_kernel(const float* __restrict__ logits, int vocab, const float* __restrict__ temperature,
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

// A cluster of CTAS blocks per row (one block up to 32,768 tokens, up to eight), temperature <= 0 means greedy for that row.
//
// The bisection asks some thirty times how much probability lies above a threshold.  Bound by those questions' chain of sums, not by bytes: the row's
// probabilities stay in registers, 32 per thread, so a question is 32 comparisons and one sum over the block (and over the cluster through
// distributed shared memory).  Read and exponentiated again for every question by one block, 64 rows of 32,000 took 550 us and 4 rows of
// 128,256 took 800.
// A block owns a run of token ids; its thread t holds the quads t, t + 1024, ... of the run, so that loads are whole lines; token-id order is
// block, then round of quads, then thread.
template <int CTAS>
__global__ void __launch_bounds__(kSampleThreads)
    sample_kernel(const float* __restrict__ logits, int vocab, const float* __restrict__ temperature, const float* __restrict__ top_p,
                  const long long* __restrict__ seeds, const long long* __restrict__ counters, int* __restrict__ out) {
  namespace cg = cooperative_groups;
  constexpr int kRounds = 8, kWarps = kSampleThreads / 32;
  __shared__ float scratch[32];
  __shared__ float exchange[2][8];          // the blocks' partial results, double buffered: one cluster barrier per exchange
  __shared__ int exchanged_index[8];
  __shared__ float rounds[kRounds][kWarps];
  __shared__ int found;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = CTAS > 1 ? (int)cluster.block_rank() : 0;
  const int row_index = blockIdx.x / CTAS;
  const float* row = logits + (size_t)row_index * vocab;
  const float temp = temperature[row_index];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int quads = (vocab + 3) / 4, quads_each = (quads + CTAS - 1) / CTAS;
  const int first_id = min(vocab, rank * quads_each * 4), end_id = min(vocab, (rank + 1) * quads_each * 4);   // this block's token ids

  if (CTAS > 1) cluster.sync();   // a block's shared memory may be written once the block runs
  int parity = 0;
  // every block's value in every block, in block order
  auto all_values = [&](float mine, float (&values)[CTAS]) {
    if (CTAS == 1) {
      values[0] = mine;
      return;
    }
    if (threadIdx.x < CTAS) *cluster.map_shared_rank(&exchange[parity][rank], threadIdx.x) = mine;
    cluster.sync();
#pragma unroll
    for (int c = 0; c < CTAS; ++c) values[c] = exchange[parity][c];
    parity ^= 1;
  };
  auto sum_of_all = [&](float v) {
    float values[CTAS];
    all_values(block_sum(v, scratch), values);
    float sum = values[0];
#pragma unroll
    for (int c = 1; c < CTAS; ++c) sum += values[c];
    return sum;
  };

  if (!(temp > 0.0f)) {
    // greedy: lowest id among the maxima
    float local_max = -INFINITY;
    int local_arg = 0x7fffffff;
    row_max_and_arg(row + first_id, end_id - first_id, local_max, local_arg);
    const float block_best = block_max(local_max, scratch);
    if (threadIdx.x == 0) found = 0x7fffffff;
    __syncthreads();
    if (local_max == block_best && local_arg != 0x7fffffff) atomicMin(&found, first_id + local_arg);
    __syncthreads();
    int best_id = found;
    if (CTAS > 1) {
      if (threadIdx.x < CTAS) *cluster.map_shared_rank(&exchanged_index[rank], threadIdx.x) = best_id;
      float values[CTAS];
      all_values(block_best, values);
      float best = -INFINITY;
      best_id = 0x7fffffff;
#pragma unroll
      for (int c = 0; c < CTAS; ++c)
        if (exchanged_index[c] != 0x7fffffff && (values[c] > best || best_id == 0x7fffffff)) {   // blocks are in id order: a tie stays with the first
          best = values[c];
          best_id = exchanged_index[c];
        }
    }
    // a row without any comparable value (all NaN) leaves no maximum: token 0, as argmax_kernel answers
    if (rank == 0 && threadIdx.x == 0) out[row_index] = (best_id < 0 || best_id >= vocab) ? 0 : best_id;
    return;
  }

  float p[kRounds][4];   // logits first, then probabilities; -inf (so 0) past the end
  const bool whole = (vocab & 3) == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  float local_max = -INFINITY;
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int id = first_id + (r * kSampleThreads + (int)threadIdx.x) * 4;
    if (whole) {
      const float4 v = id < end_id ? *reinterpret_cast<const float4*>(row + id) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
      p[r][0] = v.x, p[r][1] = v.y, p[r][2] = v.z, p[r][3] = v.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) p[r][i] = id + i < end_id ? row[id + i] : -INFINITY;
    }
  }
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
#pragma unroll
    for (int i = 0; i < 4; ++i) local_max = fmaxf(local_max, p[r][i]);
  float row_max;
  {
    float values[CTAS];
    all_values(block_max(local_max, scratch), values);
    row_max = values[0];
#pragma unroll
    for (int c = 1; c < CTAS; ++c) row_max = fmaxf(row_max, values[c]);
  }
  const float inv_temp = 1.0f / temp;
  float sum = 0.0f;
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int id = first_id + (r * kSampleThreads + (int)threadIdx.x) * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      p[r][i] = id + i < end_id ? expf((p[r][i] - row_max) * inv_temp) : -1.0f;   // -1: no token, never kept
      sum += id + i < end_id ? p[r][i] : 0.0f;
    }
  }
  const float total = sum_of_all(sum);

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
      float mass[2] = {0.0f, 0.0f};
#pragma unroll
      for (int r = 0; r < kRounds; ++r)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (p[r][i] >= threshold) mass[i & 1] += p[r][i];
      if (sum_of_all(mass[0] + mass[1]) >= want) lo = mid; else hi = mid;
    }
    tau = __uint_as_float(lo);
  }

  // what is kept, per round and warp, then per block
  float kept[kRounds];
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    kept[r] = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (p[r][i] >= tau) kept[r] += p[r][i];
    const float of_warp = warp_sum(kept[r]);
    if (lane == 0) rounds[r][warp] = of_warp;
  }
  if (threadIdx.x == 0) found = -1;
  __syncthreads();
  float of_round[kRounds], of_block = 0.0f;
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    of_round[r] = warp_sum(rounds[r][lane]);
    of_block += of_round[r];
  }
  float blocks[CTAS];
  all_values(of_block, blocks);
  float kept_total = blocks[0];
#pragma unroll
  for (int c = 1; c < CTAS; ++c) kept_total += blocks[c];
  const float target = uniform_from((unsigned long long)seeds[row_index], (unsigned long long)counters[row_index]) * kept_total;

  // The last block, round and thread with something kept that starts at or before the target holds it (whatever rounding does to the starts), and of its
  // quad the first token that reaches past the target, or the last kept one.
  int block_of = -1;
  float start = 0.0f, running = 0.0f;
#pragma unroll
  for (int c = 0; c < CTAS; ++c) {
    if (blocks[c] > 0.0f && running <= target) {
      block_of = c;
      start = running;
    }
    running += blocks[c];
  }
  if (block_of == rank) {   // the same for the whole block
    int round_of = -1;
    running = start;
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      if (of_round[r] > 0.0f && running <= target) {
        round_of = r;
        start = running;
      }
      running += of_round[r];
    }
    if (round_of >= 0) {
      float mine = 0.0f, quad[4];
#pragma unroll
      for (int r = 0; r < kRounds; ++r)
        if (r == round_of) {
          mine = kept[r];
#pragma unroll
          for (int i = 0; i < 4; ++i) quad[i] = p[r][i];
        }
      float inclusive = mine;   // over the warp's lanes, then the warps before it
#pragma unroll
      for (int offset = 1; offset < 32; offset <<= 1) {
        const float before = __shfl_up_sync(0xffffffffu, inclusive, offset);
        if (lane >= offset) inclusive += before;
      }
      float cursor = start + warp_sum(lane < warp ? rounds[round_of][lane] : 0.0f) + (inclusive - mine);
      const bool here = mine > 0.0f && cursor <= target;
      if (here) atomicMax(&found, (int)threadIdx.x);
      __syncthreads();
      const int holder = found;
      __syncthreads();
      // rounding can put the first kept thread's start past the target: then it is that one
      if (holder < 0 && threadIdx.x == 0) found = kSampleThreads;
      __syncthreads();
      if (holder < 0 && mine > 0.0f) atomicMin(&found, (int)threadIdx.x);
      __syncthreads();
      if (found == (int)threadIdx.x) {
        int pick = -1;
        const int id = first_id + (round_of * kSampleThreads + (int)threadIdx.x) * 4;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (quad[i] >= tau && !(pick >= 0 && target < cursor)) {
            cursor += quad[i];
            pick = id + i;
          }
        out[row_index] = (pick < 0 || pick >= vocab) ? 0 : pick;
      }
      if (found >= kSampleThreads && threadIdx.x == 0) out[row_index] = 0;
    } else if (threadIdx.x == 0) {
      out[row_index] = 0;
    }
  } else if (block_of < 0 && rank == 0) {
    // non-finite logits: nothing kept, or no comparable target: the last kept token of the row, and at any rate one of the vocabulary
    int last = 0;
    for (int i = threadIdx.x; i < vocab; i += kSampleThreads)
      if (expf((row[i] - row_max) * inv_temp) >= tau) last = max(last, i);
    atomicMax(&found, last);
    __syncthreads();
    if (threadIdx.x == 0) out[row_index] = max(found, 0);
  }
  // no block leaves while another may still write its part of an exchange: the last exchange ended in a barrier that follows all writes
}

template <int CTAS>
static int launch_sample(const float* logits, int rows, int vocab, const float* temperature, const float* top_p, const long long* seeds, const long long* counters,
                         int* out, cudaStream_t stream) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(rows * CTAS);
  config.blockDim = dim3(kSampleThreads);
  config.stream = stream;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = CTAS;
  attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
  config.attrs = attribute;
  config.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&config, sample_kernel<CTAS>, logits, vocab, temperature, top_p, seeds, counters, out);
}

}  // namespace tlie

using namespace tlie;

TLIE_EXPORT int tlie_argmax(const float* logits, int rows, int vocab, int* out, cudaStream_t stream) {
  if (rows <= 0) return 0;
  argmax_kernel<<<rows, kSampleThreads, 0, stream>>>(logits, vocab, out);
  return (int)cudaGetLastError();
}

TLIE_EXPORT int tlie_sample(const float* logits, int rows, int vocab, const float* temperature, const float* top_p,
                            const long long* seeds, const long long* counters, int* out, cudaStream_t stream) {
  if (rows <= 0) return 0;
  // a block holds 32 probabilities per thread
  constexpr int kHeld = 32 * kSampleThreads;
  if (vocab <= kHeld) return launch_sample<1>(logits, rows, vocab, temperature, top_p, seeds, counters, out, stream);
  if (vocab <= 2 * kHeld) return launch_sample<2>(logits, rows, vocab, temperature, top_p, seeds, counters, out, stream);
  if (vocab <= 4 * kHeld) return launch_sample<4>(logits, rows, vocab, temperature, top_p, seeds, counters, out, stream);
  if (vocab <= 8 * kHeld) return launch_sample<8>(logits, rows, vocab, temperature, top_p, seeds, counters, out, stream);
  sample_long_kernel<<<rows, kSampleThreads, 0, stream>>>(logits, vocab, temperature, top_p, seeds, counters, out);
  return (int)cudaGetLastError();
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
