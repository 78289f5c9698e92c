// 32-bit matrix product for the float32 path: out[M, N] = x[M, K] . w[N, K]^T (rows of x ``lda`` elements apart), on the tensor cores, each number in three bfloat16 parts.
//
// The reference's 32-bit model computes each output as one dot product over K in index order (src/model.cpp:53-78).  The FP32 pipes are bound by what shared memory
// delivers to them (45 of 72 TFLOP/s at 2,048 rows) and a sum over k in order by the chain of its multiply-adds.  Here every number is cut into three bfloat16 parts,
// v = high + middle + low, each the rounded rest of the ones before it: 24 bits, nothing lost where v is not tiny (see the end).  The product of two such numbers is the sum of nine products of parts;
// the three that are below 2^-24 of it are left out, the other six are tensor-core products with 32-bit sums.
//
// The order of a sum is a definition, the same for every output whatever M, N, the kernel and the tile:
//   * chunks of 64 k; a chunk's sum starts from zero and takes, 16 k at a time, first the five small kinds of products (low high, high low, middle middle,
//     middle high, high middle; all 64 k of them), then the large one (high high).  The tensor core cuts off what lies below the last bit of the largest number it adds, so what is
//     small is summed while the sum is small, and only four additions of a chunk are taken at full size;
//   * the chunks' sums are added in order, in 32-bit, rounded to nearest.
// A tcgen05.mma and an mma.sync m16n8k16 of the same 16 k give the same bits, and the place of a k among the 16 does not matter; so both kernels below keep to the definition:
//   * up to 16 rows (decoding), and more where that is cheaper (see `cheapest`): bound by the weights' bytes; warps of a CTA take chunks of 16 rows of w in turn, each lane the fragments it
//     needs (mma.sync);
//   * more rows: tiles of 128 rows of x by 64 or 96 rows of w on tcgen05, operands cut on their way into shared memory.  A chunk of 64 k takes 2,550 clocks at 96 rows of w, its 24 products
//     1,150 of them.  Every number goes through shared memory raw (112 KB a chunk in and out), in parts (84 KB) and as operands (168 KB); ncu has the tensor pipe busy 37 % of the time, shared
//     memory's wavefronts of loads, stores and copies 52 %, issue slots 39 %;
//   * sums of up to six terms: multiply-adds in order, a thread an output.
// Against 64-bit sums the error is a sixth to a seventh of what multiply-adds in order give (2-norms over normal numbers: K = 2,048 1.3e-7, 8.1e-7; K = 5,632 1.9e-7, 1.34e-6).
// Back to back in a graph, weights from HBM, the register kernels before -> these, in us:
//   rows      2,560 x 2,048    2,048 x 2,048    11,264 x 2,048    2,048 x 5,632    32,000 x 2,048
//      1      10.9 ->  8.7     10.0 ->  6.3      23.3 ->  21.7     25.9 -> 12.4      49 ->  48
//      4      13.8 ->  9.1     10.4 ->  6.5      25.9 ->  21.8     31.6 -> 12.6      57 ->  48
//     16      32.4 -> 12.6     17.7 ->  7.7      64.9 ->  27.3     43.8 -> 16.2     155 ->  71
//     24      51.6 -> 16.8     51.3 -> 12.2       129 ->  50       139 ->  28       244 -> 135
//    150       130 ->  54       116 ->  44        252 -> 100       321 -> 110       538 -> 241
//    760       233 ->  88       236 ->  47        902 -> 236       627 -> 124
//  2,048       673 -> 143       461 -> 137      2,224 -> 671     1,234 -> 355
// What the parts cannot hold is worked out again as one sum of multiply-adds over k in order.  Parts of an infinity, and of numbers that round to one, are not finite: nor is such an output.
// Parts of numbers below 2^-102 (their last bits), and products of parts where the operands' product is below 2^-98, leave the range of normal numbers; what a term loses then is at
// most 2^-124 of the largest operand, or 2^-123.  So an output is also worked out again where its rows of x and w hold such numbers (other than zeros) and it is below
// K * 2^-98 * max(1, largest operand), 2^25 times what it may have lost.  Both are properties of the output and its two rows, whatever kernel and tile it is in.
#include "mma_utils.cuh"
#include "shared_memory_limit.cuh"
#define TLIE_WITHOUT_TENSOR_MAPS
#include "tcgen05_utils.cuh"

namespace tlie {

constexpr int kChunkK = 64;

// a and b less a part of each, two subtractions in one instruction (exact: the part is the number's own leading bits, rounded).
__device__ __forceinline__ void take_off(float& a, float& b, uint32_t part) {
  unsigned long long both, parts, minus;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(both) : "f"(a), "f"(b));
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(parts) : "r"(part << 16), "r"(part & 0xffff0000u));
  asm("mov.b64 %0, {%1, %1};\n" : "=l"(minus) : "f"(-1.0f));
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(both) : "l"(parts), "l"(minus), "l"(both));
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(both));
}
// Two neighbours cut into parts (the first in the lower half of every word).
__device__ __forceinline__ void cut_pair(float a, float b, uint32_t& high, uint32_t& middle, uint32_t& low) {
  high = pack_bf16(a, b);
  take_off(a, b, high);
  middle = pack_bf16(a, b);
  take_off(a, b, middle);
  low = pack_bf16(a, b);
}

// Four neighbours of a row of K; zeros past its end.  The kernel before may still write them when this one starts: ordinary loads, in their place behind the dependency wait, which makes what it
// wrote visible to them (not to the read-only path, which is for what nobody writes while the kernel runs, and which the compiler takes for pointers that it knows to be read only).
// Through L1, since a CTA's tiles read the same x: 16 rows, 11,264 x 2,048 27.4 us, 30.4 past it.
template <bool ALIGNED>
__device__ __forceinline__ float4 load_four(const float* row, int k, int K) {
  float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (ALIGNED) {
    if (k < K) asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(row + k));
  } else {
    if (k < K) asm volatile("ld.global.f32 %0, [%1];\n" : "=f"(v.x) : "l"(row + k));
    if (k + 1 < K) asm volatile("ld.global.f32 %0, [%1];\n" : "=f"(v.y) : "l"(row + k + 1));
    if (k + 2 < K) asm volatile("ld.global.f32 %0, [%1];\n" : "=f"(v.z) : "l"(row + k + 2));
    if (k + 3 < K) asm volatile("ld.global.f32 %0, [%1];\n" : "=f"(v.w) : "l"(row + k + 3));
  }
  return v;
}

// Asynchronous copies into shared memory; nothing is read and zeros arrive where `valid` is not set.  Unlike those of mma_utils.cuh they hold the compiler to their place among plain reads and
// writes of shared memory: a thread reads what it copied itself, without a barrier between.
__device__ __forceinline__ void copy_16(void* to, const void* from, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(to)), "l"(from), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_4(void* to, const void* from, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(smem_u32(to)), "l"(from), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ void copies_sent() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait_for_copies() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// --- what the parts cannot hold (see above) -----------------------------------------------------------
constexpr float kLargest = 3.402823466e38f;
// What a sum of K terms has to reach if nothing that may have left the range of normal numbers is to matter to it; most: the largest magnitude among its operands.
__device__ __forceinline__ float safe_from(float most, int K) { return (float)K * 3.1554436e-30f * fmaxf(1.0f, most); }   // 2^-98

// A CTA has to tell at little cost whether one of its outputs may need it: it keeps sums of squares of what it cuts, a packed multiply-add a pair (2 to 5 % of a product; smallest magnitudes
// took 10 to 15, largest ones 7 to 15).  While they are below 2^100, no operand is above 2^50 and every output from safe_from(2^50) on stands.
__device__ __forceinline__ void keep_squares(unsigned long long& squares, float a, float b) {
  unsigned long long both;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(both) : "f"(a), "f"(b));
  asm("fma.rn.f32x2 %0, %1, %1, %0;\n" : "+l"(squares) : "l"(both));
}
__device__ __forceinline__ bool squares_are_large(unsigned long long squares) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(squares));
  return !(a < 1.2676506e30f && b < 1.2676506e30f);   // (NaN among them)
}
__device__ __forceinline__ bool stands(float v, int K) { return fabsf(v) >= safe_from(1.1258999e15f, K) && fabsf(v) <= kLargest; }

struct RowRange {
  uint32_t least;   // bits of the smallest magnitude but zero, times two, less one (2^32 - 1: all zeros)
  uint32_t most;    // bits of the largest magnitude
};
// Of a row of K, by a warp.
template <bool ALIGNED>
__device__ __forceinline__ RowRange row_range(const float* row, int K) {
  uint32_t least = 0xffffffffu, most = 0;
#pragma unroll 8
  for (int k = (threadIdx.x & 31) * 4; k < K; k += 128) {
    const float4 v = load_four<ALIGNED>(row, k, K);
    const uint32_t a = __float_as_uint(v.x) * 2, b = __float_as_uint(v.y) * 2, c = __float_as_uint(v.z) * 2, d = __float_as_uint(v.w) * 2;
    least = min(min(least, min(a - 1, b - 1)), min(c - 1, d - 1));
    most = max(max(most, max(a, b)), max(c, d));
  }
  return {__reduce_min_sync(0xffffffffu, least), __reduce_max_sync(0xffffffffu, most) / 2};
}
// Of an output and the ranges of its two rows.
__device__ __forceinline__ bool work_out_again(float v, RowRange x, RowRange w, int K) {
  if (!(fabsf(v) <= kLargest)) return true;
  if (x.most == 0 || w.most == 0 || !(fabsf(v) < safe_from(fmaxf(__uint_as_float(x.most), __uint_as_float(w.most)), K))) return false;
  const int a = (int)((x.least + 1) >> 24), b = (int)((w.least + 1) >> 24);   // exponents, 127 too large
  return a < 127 - 102 || b < 127 - 102 || a + b < 2 * 127 - 98;
}

template <int BARRIER, int THREADS>
__device__ __forceinline__ void barrier_of() { asm volatile("bar.sync %0, %1;\n" ::"n"(BARRIER), "n"(THREADS) : "memory"); }

// A tile of a product, as what is rarely needed finds it in shared memory.  (With the kernel's own parameters used there, registers held them through the loops: 760 rows, 2,048 x 2,048
// 46.4 -> 48.9 us.)
struct Tile {
  const float *x, *w;
  float* out;
  long long lda;
  int M, N, K, m0, n0;
};

// Sums in order of TM x TN outputs a thread, of a tile of TM * ROWS rows of x and TN * 16 rows of w that THREADS threads bring to shared memory STEP columns at a time, a step ahead: rows
// thread / 16 + ROWS i, columns thread % 16 + 16 j.  Threads that do not want theirs only copy.
template <int TM, int TN, int ROWS, int STEP, int THREADS, int BARRIER, bool ALIGNED>
__device__ __forceinline__ void sums_in_order(float (&sum)[TM][TN], const Tile& t, int thread, bool wanted, float* stages) {
  constexpr int kRows = TM * ROWS + TN * 16, kStride = STEP + 4, kWide = ALIGNED ? 4 : 1;
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) sum[i][j] = 0.0f;
  auto copy = [&](int step) {
    float* stage = stages + (step & 1) * kRows * kStride;
    for (int at = thread; at < kRows * STEP / kWide; at += THREADS) {   // columns past K are zeros
      const int r = at / (STEP / kWide), within = at % (STEP / kWide) * kWide, k = step * STEP + within;
      const float* row = r < TM * ROWS ? t.x + min(t.m0 + r, t.M - 1) * t.lda : t.w + (long long)min(t.n0 + r - TM * ROWS, t.N - 1) * t.K;
      if (ALIGNED) {
        copy_16(stage + r * kStride + within, k < t.K ? row + k : row, k < t.K);
      } else {
        copy_4(stage + r * kStride + within, k < t.K ? row + k : row, k < t.K);
      }
    }
    copies_sent();
  };
  const int steps = (t.K + STEP - 1) / STEP;
  copy(0);
  for (int step = 0; step < steps; ++step) {
    wait_for_copies<0>();
    __syncwarp();
    barrier_of<BARRIER, THREADS>();   // this step's columns are here for every thread, and everyone is done with the other stage
    if (step + 1 < steps) copy(step + 1);
    const float* xs = stages + ((step & 1) * kRows + thread / 16) * kStride;
    const float* ws = stages + ((step & 1) * kRows + TM * ROWS + thread % 16) * kStride;
    if (!wanted) continue;
#pragma unroll 4
    for (int k = 0; k < STEP; k += 2) {
      float2 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float2*>(xs + i * ROWS * kStride + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float2 b = *reinterpret_cast<const float2*>(ws + j * 16 * kStride + k);
#pragma unroll
        for (int i = 0; i < TM; ++i) sum[i][j] = fmaf(a[i].y, b.y, fmaf(a[i].x, b.x, sum[i][j]));
      }
    }
  }
}

// Outputs of a tile that are not sure to stand, decided and stored by THREADS threads from FIRST on, which have a barrier of their own.  values: [BM][BN + 1], as they were summed; behind
// them room for the rows' ranges and two stages of sums_in_order.  They come from warps of 32 rows and COLUMNS columns; bit row / 32 + 4 (column / COLUMNS) of `unsure` stands for theirs (the
// other warps have stored theirs).  large: an operand may be above 2^50.
// Rows of x and of w that have open outputs are looked at, those of the lesser side first: a row that holds a NaN, or nothing but zeros, settles its outputs.  What has to be worked out
// again is worked out by the whole tile together, operands through shared memory.  760 rows, 2,048 x 2,048, 46 us without: one NaN in x 108, in w 110, an infinity in x 300, in every row 550
// (a thread for each such output: 3,700 and 24,000; register kernels with all sums in order 232).
template <int BM, int BN, int COLUMNS, int STEP, int FIRST, int THREADS, int BARRIER, bool ALIGNED>
__device__ __noinline__ void store_unsure(const Tile* tile, float* values, uint32_t unsure, bool large) {
  constexpr int kRows = BM < THREADS / 16 ? BM : THREADS / 16, TM = BM / kRows, TN = BN / 16;
  static_assert(BM % kRows == 0 && BN % 16 == 0 && TM * TN <= 64, "a bit per output of a thread");
  const Tile t = *tile;
  RowRange* ranges = reinterpret_cast<RowRange*>(values + BM * (BN + 1));      // rows of x, rows of w
  uint32_t* open = reinterpret_cast<uint32_t*>(ranges + BM + BN);              // [2][BM + BN]: whether a row has open outputs, to begin with and once one side is settled
  uint32_t* counts = open + 2 * (BM + BN);                                     // of x's rows and w's rows that have; of threads that have in the end
  float* stage = reinterpret_cast<float*>(((uintptr_t)(counts + 3) + 15) & ~(uintptr_t)15);
  const int thread = (int)threadIdx.x - FIRST, row0 = thread / 16, column0 = thread % 16;
  auto barrier = [] {
    __syncwarp();
    barrier_of<BARRIER, THREADS>();
  };
  unsigned long long mine = 0;   // this thread's open outputs
  // What `settle` does with every open output: it gives back whether the output stays open, or stores it.
  auto each = [&](auto settle) {
    unsigned long long left = mine;
    while (left != 0) {
      const int at = __ffsll((long long)left) - 1;
      left &= left - 1;
      const int row = row0 + at / TN * kRows, column = column0 + at % TN * 16;
      float v = values[row * (BN + 1) + column];
      if (settle(row, column, v)) continue;
      mine &= ~(1ull << at);
      t.out[(size_t)(t.m0 + row) * t.N + t.n0 + column] = v;
    }
  };
  auto look = [&](bool of_w, const uint32_t* flags) {
    for (int r = (of_w ? BM : 0) + thread / 32; r < (of_w ? BM + BN : BM); r += THREADS / 32) {
      if (flags[r] == 0) continue;
      const RowRange found = row_range<ALIGNED>(of_w ? t.w + (long long)(t.n0 + r - BM) * t.K : t.x + (t.m0 + r) * t.lda, t.K);
      if ((thread & 31) == 0) ranges[r] = found;
    }
  };
  for (int i = thread; i < 2 * (BM + BN) + 3; i += THREADS) open[i] = 0;
  barrier();
  if (thread < kRows * 16) {
#pragma unroll 1
    for (int at = 0; at < TM * TN; ++at) {
      const int row = row0 + at / TN * kRows, column = column0 + at % TN * 16;
      if (t.m0 + row < t.M && t.n0 + column < t.N && (unsure >> (row / 32 + 4 * (column / COLUMNS)) & 1)) mine |= 1ull << at;
    }
  }
  each([&](int row, int column, float v) {
    if (!large && stands(v, t.K)) return false;
    if (atomicExch(&open[row], 1u) == 0) atomicAdd(&counts[0], 1u);
    if (atomicExch(&open[BM + column], 1u) == 0) atomicAdd(&counts[1], 1u);
    return true;
  });
  barrier();
  const bool w_first = counts[1] < counts[0];
  look(w_first, open);
  barrier();
  each([&](int row, int column, float& v) {
    const RowRange range = ranges[w_first ? BM + column : row];
    if (range.most > 0x7f800000u) v = __uint_as_float(0x7fffffffu);
    if (range.most > 0x7f800000u || (range.most == 0 && fabsf(v) <= kLargest)) return false;
    open[BM + BN + (w_first ? row : BM + column)] = 1;
    return true;
  });
  barrier();
  look(!w_first, open + BM + BN);
  barrier();
  each([&](int row, int column, float& v) {
    if (ranges[w_first ? row : BM + column].most > 0x7f800000u) {
      v = __uint_as_float(0x7fffffffu);
      return false;
    }
    return work_out_again(v, ranges[row], ranges[BM + column], t.K);
  });
  if (mine != 0) counts[2] = 1;
  barrier();
  if (counts[2] != 0) {
    float sum[TM][TN];
    sums_in_order<TM, TN, kRows, STEP, THREADS, BARRIER, ALIGNED>(sum, t, thread, mine != 0, stage);
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j)
        if (mine >> (i * TN + j) & 1) t.out[(size_t)(t.m0 + row0 + i * kRows) * t.N + t.n0 + column0 + j * 16] = sum[i][j];
  }
  barrier();
}

// --- few rows ----------------------------------------------------------------------------------------
constexpr int kFewRows = 16;        // rows of w of a CTA
constexpr int kFewAhead = 2;        // chunks of w on their way to a warp
constexpr int kFewRound = 96;       // chunks whose sums are in shared memory at a time

// NT: blocks of 8 rows of x.  A lane (g = lane / 4, t = lane % 4) holds rows g and g + 8 of w and row g of every block of x, k 4 t ... 4 t + 3 of every 16.
// A lane copies what it will read itself (w of two chunks ahead, whichever tile they belong to), so a warp's ring needs no barrier.  WARPS: with one block sixteen where a CTA has its SM to
// itself and eight where two share one, 128 KB an SM on their way from HBM (with the next chunk on its way to registers it was half of that: 11,264 x 2,048 24.5 us, 2,048 x 5,632 13); with
// two blocks eight, 64 KB: registers hold no more.
// A CTA walks row tiles blockIdx.x, + gridDim.x, ...  SHORT: a row has so few chunks that the warps take those of `together` tiles at a time (one tile after the other,
// one to four warps of eight worked: K = 64, 16 rows x 11,264 5.6 -> 4.2 us, 128 x 2,048 8.2 -> 4.7, 600 x 256 6.4 -> 4.1).
template <int NT, int WARPS, bool ALIGNED, bool SHORT>
__global__ void __launch_bounds__(WARPS * 32, NT == 1 && WARPS == 8 ? 2 : 1) gemm_few_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out,
                                                                                                int M, int N, int K, long long lda) {
  extern __shared__ __align__(16) float ring[];   // [warp][kFewAhead][8][lane] float4, then the sums
  float* sums = ring + WARPS * kFewAhead * kFewRows * kChunkK;   // [chunk of the round][NT][rows of x][rows of w]: 8 x 16 each
  constexpr int kOutputs = 8 * kFewRows * NT;
  static_assert(kOutputs <= WARPS * 32, "a thread adds up one output");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int tiles = (N + kFewRows - 1) / kFewRows, chunks = (K + kChunkK - 1) / kChunkK;
  const int m0 = blockIdx.y * 8 * NT;
  const float* x_rows[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) x_rows[j] = x + (long long)min(m0 + 8 * j + g, M - 1) * lda;
  // While the kernel before this one runs, L2 fetches the CTA's first chunks of weights.  Nothing is read: w may be what that kernel writes.
  for (int c = warp; c < chunks && c < 4 * WARPS; c += WARPS) {
    const int k = c * kChunkK + (lane & 1) * 32;
    if (k < K) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(w + (long long)min((int)blockIdx.x * kFewRows + (lane >> 1), N - 1) * K + k));
  }
  grid_launch_dependents();
  grid_dependency_wait();
  float4* const mine = reinterpret_cast<float4*>(ring) + warp * kFewAhead * 8 * 32 + lane;
  const int together = SHORT ? WARPS / chunks : 1, stride = together * (int)gridDim.x;
  const int own_chunk = SHORT ? warp % chunks : warp;                       // a warp's first chunk of a tile
  const int own_tile = SHORT ? warp / chunks * (int)gridDim.x : 0;          // and of which tile, from the CTA's first
  const bool works = SHORT ? warp / chunks < together : warp < chunks;
  int ask_tile = works ? (int)blockIdx.x + own_tile : tiles, ask_chunk = own_chunk;
  auto ask = [&](int slot) {   // w of the next chunk in this warp's order; a group each (an empty one behind the last keeps the count)
    if (ask_tile < tiles) {
      const int n = ask_tile * kFewRows + g;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float* row = w + (long long)min(n + 8 * r, N - 1) * K;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int k = ask_chunk * kChunkK + 16 * s + 4 * t;
          float4* place = mine + (slot * 8 + r * 4 + s) * 32;
          if (ALIGNED) {
            copy_16(place, k < K ? row + k : row, k < K);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) copy_4(reinterpret_cast<float*>(place) + e, k + e < K ? row + k + e : row, k + e < K);
          }
        }
      }
      ask_chunk += WARPS;
      if (ask_chunk >= chunks) ask_chunk = own_chunk, ask_tile += stride;
    }
    copies_sent();
  };
  float4 xv[NT][4];
  auto load_x = [&](int chunk) {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int s = 0; s < 4; ++s) xv[j][s] = load_four<ALIGNED>(x_rows[j], chunk * kChunkK + 16 * s + 4 * t, K);
  };
#pragma unroll
  for (int s = 0; s < kFewAhead; ++s) ask(s);
  if (works) load_x(own_chunk);
  int slot = 0;
  unsigned long long squares = 0;
  for (int first_tile = blockIdx.x; first_tile < tiles; first_tile += stride) {
    float total = 0.0f;
    bool unsure = false;
    for (int first = 0; first < chunks; first += kFewRound) {
      const int here = min(kFewRound, chunks - first);
      const int end = SHORT ? (works && first_tile + own_tile < tiles ? warp + 1 : 0) : first + here;   // (SHORT: one chunk a warp, its sums in the warp's place)
      for (int c = first + warp; c < end; c += WARPS) {
        float acc[NT][4];
        uint32_t wh[4][4], xh[NT][4][2];
        wait_for_copies<kFewAhead - 1>();
        float4 wv[2][4];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int s = 0; s < 4; ++s) wv[r][s] = mine[(slot * 8 + r * 4 + s) * 32];
        ask(slot);
        slot = slot + 1 == kFewAhead ? 0 : slot + 1;
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          uint32_t wm[4], wl[4], xm[NT][2], xl[NT][2];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            keep_squares(squares, wv[r][s].x, wv[r][s].y);
            keep_squares(squares, wv[r][s].z, wv[r][s].w);
            cut_pair(wv[r][s].x, wv[r][s].y, wh[s][r], wm[r], wl[r]);
            cut_pair(wv[r][s].z, wv[r][s].w, wh[s][r + 2], wm[r + 2], wl[r + 2]);
          }
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            keep_squares(squares, xv[j][s].x, xv[j][s].y);
            keep_squares(squares, xv[j][s].z, xv[j][s].w);
            cut_pair(xv[j][s].x, xv[j][s].y, xh[j][s][0], xm[j][0], xl[j][0]);
            cut_pair(xv[j][s].z, xv[j][s].w, xh[j][s][1], xm[j][1], xl[j][1]);
          }
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            mma_bf16(acc[j], wh[s], xl[j][0], xl[j][1]);
            mma_bf16(acc[j], wl, xh[j][s][0], xh[j][s][1]);
            mma_bf16(acc[j], wm, xm[j][0], xm[j][1]);
            mma_bf16(acc[j], wh[s], xm[j][0], xm[j][1]);
            mma_bf16(acc[j], wm, xh[j][s][0], xh[j][s][1]);
          }
        }
        if (!SHORT) load_x(c + WARPS < chunks ? c + WARPS : own_chunk);   // of the next chunk, or of the next tile's first one
#pragma unroll
        for (int s = 0; s < 4; ++s)
#pragma unroll
          for (int j = 0; j < NT; ++j) mma_bf16(acc[j], wh[s], xh[j][s][0], xh[j][s][1]);
        float* to = sums + (c - first) * kOutputs;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          float* block = to + j * 8 * kFewRows;
          block[(2 * t) * kFewRows + g] = acc[j][0];
          block[(2 * t + 1) * kFewRows + g] = acc[j][1];
          block[(2 * t) * kFewRows + g + 8] = acc[j][2];
          block[(2 * t + 1) * kFewRows + g + 8] = acc[j][3];
        }
      }
      __syncthreads();
      if (SHORT) break;
      if (threadIdx.x < kOutputs) {
#pragma unroll 8
        for (int c = 0; c < here; ++c) total += sums[c * kOutputs + threadIdx.x];
      }
      unsure = __syncthreads_or(squares_are_large(squares) || (threadIdx.x < kOutputs && !stands(total, K)));   // (of the last round, all of K)
    }
    for (int part = 0; part < together && first_tile + part * (int)gridDim.x < tiles; ++part) {
      const int tile = first_tile + part * (int)gridDim.x, n0 = tile * kFewRows;
      if (SHORT) {
        total = 0.0f;
        if (threadIdx.x < kOutputs)
          for (int c = 0; c < chunks; ++c) total += sums[(part * chunks + c) * kOutputs + threadIdx.x];
        unsure = __syncthreads_or(squares_are_large(squares) || (threadIdx.x < kOutputs && !stands(total, K)));
      }
      const int m = m0 + threadIdx.x / kFewRows, n = n0 + threadIdx.x % kFewRows;
      if (!unsure) {
        if (threadIdx.x < kOutputs && m < M && n < N) out[(size_t)m * N + n] = total;
        continue;
      }
      wait_for_copies<0>();   // the ring is put to another use; what was on its way is asked for again
      const bool large = __syncthreads_or(squares_are_large(squares));
      Tile* here = reinterpret_cast<Tile*>(ring);
      float* values = ring + sizeof(Tile) / sizeof(float);
      if (threadIdx.x == 0) *here = {x, w, out, lda, M, N, K, m0, n0};
      if (threadIdx.x < kOutputs) values[threadIdx.x / kFewRows * (kFewRows + 1) + threadIdx.x % kFewRows] = total;
      __syncthreads();
      store_unsure<8 * NT, kFewRows, kFewRows, 128, 0, WARPS * 32, 0, ALIGNED>(here, values, 1, large);
      ask_tile = works ? first_tile + own_tile + stride : tiles;
      ask_chunk = own_chunk;
      slot = 0;
#pragma unroll 1
      for (int s = 0; s < kFewAhead; ++s) ask(s);
    }
  }
  wait_for_copies<0>();
}

// With 4-byte copies, which go through L1, a kernel starts only once the one before it is done.
template <bool ALIGNED, typename Kernel, typename... Args>
static int launch_product(Kernel* kernel, dim3 grid, int threads, int smem, cudaStream_t stream, Args... args) {
  if (ALIGNED) return (int)launch_pdl(kernel, grid, dim3(threads), smem, stream, args...);
  kernel<<<grid, threads, smem, stream>>>(args...);
  return (int)cudaGetLastError();
}

// CTAs of a block of rows, and tiles that a CTA's eight warps take at a time.
static long long few_across(long long places, long long blocks, long long tiles) {
  const long long across = places / blocks > 1 ? places / blocks : 1;
  return tiles < across ? tiles : across;
}
static int few_together(int K, long long tiles, long long across) {
  const int chunks = (K + kChunkK - 1) / kChunkK;
  return 2 * chunks <= 8 && tiles > across ? 8 / chunks : 1;
}

template <int NT, int WARPS, bool ALIGNED, bool SHORT = false>
static int launch_few(const float* x, const float* w, float* out, int M, int N, int K, long long lda, cudaStream_t stream) {
  const int chunks = (K + kChunkK - 1) / kChunkK, tiles = (N + kFewRows - 1) / kFewRows;
  const int places = (NT == 1 && WARPS == 8 ? 2 : 1) * device_sm_count(), blocks = (M + 8 * NT - 1) / (8 * NT);
  const int across = (int)few_across(places, blocks, tiles);
  if (!SHORT && WARPS == 8 && few_together(K, tiles, across) > 1) return launch_few<NT, WARPS, ALIGNED, WARPS == 8>(x, w, out, M, N, K, lda, stream);
  constexpr int ring = WARPS * kFewAhead * kFewRows * kChunkK * (int)sizeof(float), chunk_sums = 8 * kFewRows * NT * (int)sizeof(float);
  const int smem = ring + (SHORT ? WARPS : chunks < kFewRound ? chunks : kFewRound) * chunk_sums;
  static std::atomic<unsigned long long> devices{0};
  const cudaError_t allowed = allow_shared_memory(gemm_few_f32_kernel<NT, WARPS, ALIGNED, SHORT>, ring + (SHORT ? WARPS : kFewRound) * chunk_sums, devices);
  if (allowed != cudaSuccess) return (int)allowed;
  return launch_product<ALIGNED>(gemm_few_f32_kernel<NT, WARPS, ALIGNED, SHORT>, dim3(across, blocks), WARPS * 32, smem, stream, x, w, out, M, N, K, lda);
}

// --- more rows ---------------------------------------------------------------------------------------
// Warps 0-7 cut and store the operands of a chunk (a ring of two stages), warp 8 issues its 24 products, warps 9-16 add the chunk's sum to the ones before it in
// registers while the next chunk's products run into the other half of tensor memory.
constexpr int kCutWarps = 8, kAddWarps = 8;
constexpr int kManyThreads = (kCutWarps + 1 + kAddWarps) * 32;
constexpr int kManyStages = 2;

template <int BN>
struct ManyShape {
  static constexpr int kPlaneX = kBM * 128, kPlaneW = BN * 128;           // 64 k of one part
  static constexpr int kStage = 3 * (kPlaneX + kPlaneW);                  // [x high, middle, low | w high, middle, low]
  static constexpr int kFours = (kBM + BN) * (kChunkK / 4) / (kCutWarps * 32);   // float4 of a thread and chunk
  static constexpr int kBatch = kFours % 7 == 0 ? 7 : 4;
  static constexpr int kArrivals = kFours * kCutWarps * 32 * 16;          // where they arrive: a place for each
  static constexpr int kSmem = kManyStages * kStage + kArrivals + 1024 + 256;
  static_assert(kSmem <= 227 * 1024, "shared memory of one CTA");
  static constexpr int kColumns = BN / 2;                                 // columns of an adding warp
  static_assert(kColumns == 32 || kColumns == 48, "what an adding warp reads at once");
};

__device__ __forceinline__ uint32_t elect_one() {
  uint32_t chosen;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "elect.sync _|p, 0xffffffff;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(chosen));
  return chosen;
}
// The issuing warp walks its loop as a whole and one thread of it, always the same, executes what is issued: descriptors stay in uniform registers.
__device__ __forceinline__ void umma_bf16_if(uint32_t issue, uint32_t tmem_d, uint32_t a_low, uint32_t b_low, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      ".reg .b64 da, db;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "setp.ne.b32 q, %6, 0;\n"
      "mov.b64 da, {%1, %5};\n"
      "mov.b64 db, {%2, %5};\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(a_low), "r"(b_low), "r"(idesc), "r"(accumulate), "r"(kUmmaDescHigh), "r"(issue)
      : "memory");
}
__device__ __forceinline__ void umma_commit_if(uint32_t issue, uint32_t bar) {
  asm volatile(
      "{\n"
      ".reg .pred q;\n"
      "setp.ne.b32 q, %1, 0;\n"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
      "}\n" ::"r"(bar), "r"(issue)
      : "memory");
}

template <int BN, bool ALIGNED>
__global__ void __launch_bounds__(kManyThreads, 1) gemm_many_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out, int M, int N, int K,
                                                                       long long lda, int* __restrict__ error_flag) {
  using Shape = ManyShape<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* arrivals = ring + kManyStages * Shape::kStage;   // [float4 of a thread][thread]
  uint64_t* full = reinterpret_cast<uint64_t*>(arrivals + Shape::kArrivals);
  uint64_t* empty = full + kManyStages;
  uint64_t* summed = empty + kManyStages;   // [2]: a chunk's products are done
  uint64_t* taken = summed + 2;             // [2]: its sum has been read
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(taken + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  uint32_t* unsure = tmem_holder + 2;       // a bit per adding warp whose outputs are not stored yet
  uint32_t* large = tmem_holder + 3;        // not 0: an operand may be above 2^50
  Tile* this_tile = reinterpret_cast<Tile*>(tmem_holder + 4);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int m_blocks = (M + kBM - 1) / kBM;
  const int m0 = ((int)blockIdx.x % m_blocks) * kBM, n0 = ((int)blockIdx.x / m_blocks) * BN;   // neighbours share their weights
  const int chunks = (K + kChunkK - 1) / kChunkK;
  constexpr int kTmemStride = BN <= 64 ? 64 : 128, kTmemCols = 2 * kTmemStride;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kManyStages; ++s) {
      mbar_init(&full[s], kCutWarps);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&summed[a], 1);
      mbar_init(&taken[a], kAddWarps);
    }
    *abort_flag = 0;
    *unsure = *large = 0;
    *this_tile = {x, w, out, lda, M, N, K, m0, n0};
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == kCutWarps) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_holder)), "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = *tmem_holder;
  grid_launch_dependents();
  grid_dependency_wait();

  if (warp < kCutWarps) {
    unsigned long long squares = 0;
    // A thread's float4 i: row (thread / 16) + 16 i of the tile (x rows, then w rows), k 4 (thread % 16) of the chunk.  Rows past M or N repeat the last one.
    const int first_row = threadIdx.x / 16, k_of = (threadIdx.x % 16) * 4;
    // Each is copied to a place of its own thread's and read there by that thread; as soon as it has been read, the same place is asked to take the next chunk's, which
    // travels while the others are cut.  (Held in registers instead, the loads of a chunk began when the cutting of the one before had ended, and a chunk took 4,400
    // clocks for 1,536 of products.)
    const bool whole = m0 + kBM <= M && n0 + BN <= N;
    const float* x_first = x + (long long)min(m0 + first_row, M - 1) * lda;
    const float* w_first = w + (long long)min(n0 + first_row, N - 1) * K;
    auto row_of = [&](int i) {
      if (whole) return i < kBM / 16 ? x_first + 16 * i * lda : w_first + (long long)(16 * (i - kBM / 16)) * K;
      return i < kBM / 16 ? x + (long long)min(m0 + first_row + 16 * i, M - 1) * lda : w + (long long)min(n0 + first_row + 16 * i - kBM, N - 1) * K;
    };
    float4* const places = reinterpret_cast<float4*>(arrivals) + threadIdx.x;
    auto ask = [&](int chunk, int i) {
      const int k = chunk * kChunkK + k_of;
      if (chunk < chunks) {
        const float* row = row_of(i);
        float4* place = places + i * (kCutWarps * 32);
        if (ALIGNED) {
          copy_16(place, k < K ? row + k : row, k < K);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) copy_4(reinterpret_cast<float*>(place) + e, k + e < K ? row + k + e : row, k + e < K);
        }
      }
    };
    // kBatch at a time, a group each (an empty one behind the last chunk keeps the count), so that the chains of one number's cuts run beside those of others
    constexpr int kBatch = Shape::kBatch, kBatches = Shape::kFours / kBatch;
    // 8-byte pieces of 16-byte chunks of 128-byte rows, the chunks moved by the swizzle: rows 16 apart have the same r % 8
    const uint32_t to = (uint32_t)first_row * 128 + ((((uint32_t)(k_of / 8)) ^ (first_row & 7)) << 4) + (k_of & 4) * 2;
#pragma unroll
    for (int g = 0; g < kBatches; ++g) {
#pragma unroll
      for (int i = 0; i < kBatch; ++i) ask(0, g * kBatch + i);
      copies_sent();
    }
    for (int c = 0; c < chunks; ++c) {
      const int s = c % kManyStages;
      if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], ((c / kManyStages) & 1) ^ 1, abort_flag))) break;
      uint8_t* stage = ring + s * Shape::kStage + to;
#pragma unroll
      for (int g = 0; g < kBatches; ++g) {
        wait_for_copies<kBatches - 1>();   // the oldest of the groups on their way is this one
        float4 v[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) v[i] = places[(g * kBatch + i) * (kCutWarps * 32)];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) ask(c + 1, g * kBatch + i);
        copies_sent();
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          constexpr int kXFours = kBM / 16;
          const int row = g * kBatch + i;
          const bool of_x = row < kXFours;
          uint2 high, middle, low;
          keep_squares(squares, v[i].x, v[i].y);
          keep_squares(squares, v[i].z, v[i].w);
          cut_pair(v[i].x, v[i].y, high.x, middle.x, low.x);
          cut_pair(v[i].z, v[i].w, high.y, middle.y, low.y);
          uint8_t* at = stage + (of_x ? row * 2048 : 3 * Shape::kPlaneX + (row - kXFours) * 2048);
          const int plane = of_x ? Shape::kPlaneX : Shape::kPlaneW;
          *reinterpret_cast<uint2*>(at) = high;
          *reinterpret_cast<uint2*>(at + plane) = middle;
          *reinterpret_cast<uint2*>(at + 2 * plane) = low;
        }
      }
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // these writes -> visible to the tensor core
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[s]);
    }
    wait_for_copies<0>();
    if (squares_are_large(squares)) atomicOr(large, 1u);
    __syncwarp();
    asm volatile("bar.arrive 1, %0;\n" ::"n"((kCutWarps + kAddWarps) * 32) : "memory");   // (of the word above, to the adding warps)
  } else if (warp == kCutWarps) {
    const uint32_t issue = elect_one();
    constexpr uint32_t idesc = umma_instr_desc(kBM, BN);
    constexpr uint32_t kX = Shape::kPlaneX >> 4, kW = Shape::kPlaneW >> 4;   // in descriptor units
    const uint32_t ring_low = umma_desc_low(smem_u32(ring));
    for (int c = 0; c < chunks; ++c) {
      const int s = c % kManyStages, b = c & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(&full[s], (c / kManyStages) & 1, abort_flag))) break;
      if (!__all_sync(0xffffffffu, mbar_wait(&taken[b], ((c / 2) & 1) ^ 1, abort_flag))) break;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t to = tmem + b * kTmemStride, xs = ring_low + s * (Shape::kStage >> 4), ws = xs + 3 * kX;
#pragma unroll
      for (int k = 0; k < 4; ++k) {   // 16 k: 32 bytes inside the swizzle span
        umma_bf16_if(issue, to, xs + 2 * kX + 2 * k, ws + 2 * k, idesc, k > 0 ? 1u : 0u);   // low of x, high of w
        umma_bf16_if(issue, to, xs + 2 * k, ws + 2 * kW + 2 * k, idesc, 1u);                // high, low
        umma_bf16_if(issue, to, xs + kX + 2 * k, ws + kW + 2 * k, idesc, 1u);               // middle, middle
        umma_bf16_if(issue, to, xs + kX + 2 * k, ws + 2 * k, idesc, 1u);                    // middle, high
        umma_bf16_if(issue, to, xs + 2 * k, ws + kW + 2 * k, idesc, 1u);                    // high, middle
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) umma_bf16_if(issue, to, xs + 2 * k, ws + 2 * k, idesc, 1u);
      umma_commit_if(issue, smem_u32(&empty[s]));
      umma_commit_if(issue, smem_u32(&summed[b]));
    }
  } else {
    const int sub = warp & 3, half = (warp - kCutWarps - 1) / 4;   // the quarter of the lanes that this warp may read; its half of the columns
    const uint32_t from = tmem + ((uint32_t)(sub * 32) << 16) + half * Shape::kColumns;
    float total[Shape::kColumns];
#pragma unroll
    for (int i = 0; i < Shape::kColumns; ++i) total[i] = 0.0f;
    bool ok = true;
    for (int c = 0; c < chunks; ++c) {
      const int b = c & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&summed[b], (c / 2) & 1, abort_flag));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      uint32_t v[32], rest[16];
      tmem_load_32(from + b * kTmemStride, v);
      if (Shape::kColumns > 32) tmem_load_16(from + b * kTmemStride + 32, rest);
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&taken[b]);
#pragma unroll
      for (int j = 0; j < 32; ++j) total[j] += __uint_as_float(v[j]);
      if (Shape::kColumns > 32) {
#pragma unroll
        for (int j = 32; j < Shape::kColumns; ++j) total[j] += __uint_as_float(rest[j - 32]);
      }
    }
    __syncwarp();
    asm volatile("bar.sync 1, %0;\n" ::"n"((kCutWarps + kAddWarps) * 32) : "memory");
    const int row = sub * 32 + lane, m = m0 + row, first = n0 + half * Shape::kColumns;
    bool sure = *reinterpret_cast<volatile uint32_t*>(large) == 0;
#pragma unroll
    for (int i = 0; i < Shape::kColumns; ++i) sure = sure && stands(total[i], K);
    if (!__all_sync(0xffffffffu, sure)) {
      float* values = reinterpret_cast<float*>(ring) + row * (BN + 1) + half * Shape::kColumns;   // every product is done with the stages
#pragma unroll
      for (int i = 0; i < Shape::kColumns; ++i) values[i] = total[i];
      if (lane == 0) atomicOr(unsure, 1u << (sub + 4 * half));
    } else if (ok && m < M) {
      float* dst = out + (size_t)m * N + first;
      const bool wide = N % 4 == 0 && ((uintptr_t)out & 15) == 0;
#pragma unroll
      for (int i = 0; i < Shape::kColumns; i += 4) {
        if (wide && first + i < N) {
          *reinterpret_cast<float4*>(dst + i) = make_float4(total[i], total[i + 1], total[i + 2], total[i + 3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (first + i + j < N) dst[i + j] = total[i + j];
        }
      }
    }
    __syncwarp();
    barrier_of<1, kAddWarps * 32>();
    if (*reinterpret_cast<volatile uint32_t*>(unsure) != 0 && *abort_flag == 0)
      store_unsure<kBM, BN, Shape::kColumns, 32, (kCutWarps + 1) * 32, kAddWarps * 32, 1, ALIGNED>(this_tile, reinterpret_cast<float*>(ring), *unsure, *large != 0);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  }
  close_and_report(abort_flag, error_flag);
  if (warp == kCutWarps) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kTmemCols));
}

template <int BN, bool ALIGNED>
static int launch_many(const float* x, const float* w, float* out, int M, int N, int K, long long lda, int* error_flag, cudaStream_t stream) {
  static std::atomic<unsigned long long> devices{0};
  const cudaError_t allowed = allow_shared_memory(gemm_many_f32_kernel<BN, ALIGNED>, ManyShape<BN>::kSmem, devices);
  if (allowed != cudaSuccess) return (int)allowed;
  const long long tiles = (long long)((M + kBM - 1) / kBM) * ((N + BN - 1) / BN);
  return launch_product<ALIGNED>(gemm_many_f32_kernel<BN, ALIGNED>, dim3((unsigned)tiles), kManyThreads, ManyShape<BN>::kSmem, stream, x, w, out, M, N, K, lda, error_flag);
}

// What a product of more than 16 rows takes, in us, by the schedule that each kernel has for it.  Fitted to 1,411 products of 17 to 4,096 rows, N from 1 to 11,264 and K from 64 to 5,632, weights
// in L2: the choice is 0.25 % slower than the best of the three in the geometric mean, and more than 10 % slower at 10 of them.
//   * blocks of 16 rows: CTAs walk tiles of 16 columns (or as many as fit their warps, see SHORT), 5 us each at K = 2,048;
//   * tiles of 128 x 96 and 128 x 64: waves of 46 and 39 us at K = 2,048, up to twice that where rows of a tile repeat the last one (2,048 columns of 24 / 64 / 128 rows: 47 / 40 / 38; 11,264
//     columns of 24 rows 79, of 128 46).
enum Kernels { FEW, TILES_OF_96, TILES_OF_64 };
static Kernels cheapest(int M, int N, int K) {
  auto up = [](long long a, long long b) { return (a + b - 1) / b; };
  const long long sms = device_sm_count(), blocks = up(M, 16), columns = up(N, kFewRows), across = few_across(sms, blocks, columns);
  const int together = few_together(K, columns, across);
  const long long steps = up(blocks * across, sms) * up(up(columns, across), together);
  const float few = 0.5f + (float)steps * (0.5f + 0.0022f * (float)K + (together > 1 ? 0.3f * (float)together : 0.0f));
  const long long m_blocks = up(M, kBM);
  const float share = (float)(m_blocks * kBM - M) / (float)(m_blocks * kBM), repeated = 1.0f + 1.1f * share * sqrtf(share);
  const float wide = (float)up(m_blocks * up(N, 96), sms) * (5.5f + 0.02f * (float)K) * repeated;
  const float narrow = (float)up(m_blocks * up(N, 64), sms) * (4.5f + 0.0168f * (float)K) * repeated;
  if (few <= fminf(wide, narrow) && blocks <= 65535) return FEW;   // (blocks are the grid's second dimension)
  return wide <= narrow ? TILES_OF_96 : TILES_OF_64;
}

template <bool ALIGNED>
static int launch_f32(const float* x, const float* w, float* out, int M, int N, int K, long long lda, int* error_flag, cudaStream_t stream) {
  if (M <= 8) {
    if ((N + kFewRows - 1) / kFewRows <= device_sm_count()) return launch_few<1, 16, ALIGNED>(x, w, out, M, N, K, lda, stream);
    return launch_few<1, 8, ALIGNED>(x, w, out, M, N, K, lda, stream);
  }
  if (M <= 16) return launch_few<2, 8, ALIGNED>(x, w, out, M, N, K, lda, stream);
  switch (cheapest(M, N, K)) {
    case FEW: return launch_few<2, 8, ALIGNED>(x, w, out, M, N, K, lda, stream);
    case TILES_OF_96: return launch_many<96, ALIGNED>(x, w, out, M, N, K, lda, error_flag, stream);
    default: return launch_many<64, ALIGNED>(x, w, out, M, N, K, lda, error_flag, stream);
  }
}

// --- short sums --------------------------------------------------------------------------------------
// Six terms and fewer, in order: the parts' products that are left out, and what the tensor core cuts off, are more than the roundings of so few multiply-adds (error against 64 bits, 2-norms,
// at 1 / 2 / 4 / 5 terms: 2.5, 3.1, 4.0, 4.3e-8; by parts 4.6e-8 at any of them.  From seven on the parts are ahead: 5.1 and 4.8, at 16 terms 7.4 and 4.8).  A thread an output: 32 columns, 8 rows.
constexpr int kShortK = 6;

__global__ void __launch_bounds__(256) gemm_short_f32_kernel(const float* x, const float* w, float* out, int M, int N, int K, long long lda) {
  const int across = (N + 31) / 32;
  const int m = (int)(blockIdx.x / across) * 8 + (int)threadIdx.x / 32, n = (int)(blockIdx.x % across) * 32 + (int)threadIdx.x % 32;
  if (m >= M || n >= N) return;
  float sum = 0.0f;
  for (int k = 0; k < K; ++k) sum = fmaf(x[m * lda + k], w[(long long)n * K + k], sum);
  out[(size_t)m * N + n] = sum;
}

}  // namespace tlie

using namespace tlie;

// error_flag (device int, may be null): bit 0 is set if a wait gave up.
TLIE_EXPORT int tlie_gemm_nt_f32_reporting(const float* x, const float* w, float* out, int M, int N, int K, long long lda, int* error_flag, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || lda < K) return (int)cudaErrorInvalidValue;
  if (K <= kShortK) {
    gemm_short_f32_kernel<<<(unsigned)((long long)((M + 7) / 8) * ((N + 31) / 32)), 256, 0, stream>>>(x, w, out, M, N, K, lda);
    return (int)cudaGetLastError();
  }
  if (K % 4 == 0 && lda % 4 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0)
    return launch_f32<true>(x, w, out, M, N, K, lda, error_flag, stream);
  return launch_f32<false>(x, w, out, M, N, K, lda, error_flag, stream);
}

TLIE_EXPORT int tlie_gemm_nt_f32(const float* x, const float* w, float* out, int M, int N, int K, long long lda, cudaStream_t stream) {
  return tlie_gemm_nt_f32_reporting(x, w, out, M, N, K, lda, nullptr, stream);
}
