// True 32-bit matrix product for the float32 path: out[M, N] = x[M, K] . w[N, K]^T (rows of x ``lda`` elements apart).
//
// The reference's 32-bit model computes each output as one dot product over K in index
// order (src/model.cpp:53-78).  These kernels keep that property on the GPU: every output
// element is accumulated by one thread with fused multiply-adds in ascending k, so its
// value depends on neither M nor N nor the kernel or tile it falls in, and no reduced-precision
// tensor-core mode can be involved.  Three kernels, the same bits:
//   * up to 16 rows (decoding): bound by the weights' bytes, or, for narrow products of long rows, by the chain of K dependent
//     multiply-adds; a CTA streams 16 weight rows through a ring in shared memory that all of its threads fill, a thread per output;
//   * more rows: register tiles of up to 8 x 8 outputs per thread, bound by the reads of shared memory that feed the FP32 pipes, operands in shared memory as they lie in
//     global memory (k innermost, so that 16-byte asynchronous copies fill them and one 16-byte read feeds four steps of k);
//   * operands that are not 16-byte aligned: a plain tile kernel.
#include "common.cuh"
#include "mma_utils.cuh"
#include "shared_memory_limit.cuh"

namespace tlie {

constexpr int kTile = 64;
constexpr int kTileK = 16;

__device__ __forceinline__ float4 read_four(unsigned addr) {   // k .. k + 3
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}

__global__ void __launch_bounds__(256) gemm_nt_f32_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                          float* __restrict__ out, int M, int N, int K, long long lda) {
  __shared__ float xs[kTileK][kTile + 1];
  __shared__ float ws[kTileK][kTile + 1];
  const int tx = threadIdx.x % 16;
  const int ty = threadIdx.x / 16;
  const int row0 = blockIdx.y * kTile;
  const int col0 = blockIdx.x * kTile;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

  for (int k0 = 0; k0 < K; k0 += kTileK) {
    for (int idx = threadIdx.x; idx < kTile * kTileK; idx += 256) {
      const int r = idx / kTileK;
      const int k = idx % kTileK;
      const int gk = k0 + k;
      const int gr = row0 + r;
      const int gc = col0 + r;
      xs[k][r] = (gr < M && gk < K) ? x[(size_t)gr * lda + gk] : 0.0f;
      ws[k][r] = (gc < N && gk < K) ? w[(size_t)gc * K + gk] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kTileK; ++k) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = xs[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = ws[k][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gr = row0 + ty * 4 + i;
    if (gr >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gc = col0 + tx * 4 + j;
      if (gc < N) out[(size_t)gr * N + gc] = acc[i][j];
    }
  }
}


// --- up to 16 rows -----------------------------------------------------------------------------------
constexpr int kStreamN = 16;         // weight rows of a CTA
constexpr int kStreamK = 128;        // columns of a ring stage
constexpr int kStreamStride = kStreamK + 4;   // shared-memory row stride: 8 rows' 16-byte reads fall into different banks
constexpr int kStreamAhead = 4;      // operands are in registers this many steps before they are used

// Back to back in a graph, weights from HBM, 4 rows, K = 2,048: 2,560 / 2,048 / 11,264 columns 13.2 / 11.1 / 25.8 us, 2,048 columns of K = 5,632: 30.4 us (the plain kernel
// 336 / 331 / 388 / 901); every read behind the dependency wait, which costs 1 to 2 us of that against weights copied in front of it.
// MP: rows of x, rounded up to a power of two.  One or two warps own the outputs, a thread one weight row and MM rows of x; the others only
// copy.  STAGES: what the CTA keeps in flight.  With at most one CTA per SM that has to cover the trip to HBM by itself.
template <int MP, int MM, int STAGES>
__global__ void __launch_bounds__(128) gemm_stream_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out, int M, int N,
                                                              int K, long long lda, int sms) {
  extern __shared__ __align__(16) float ring[];   // [stages][kStreamN + MP][kStreamStride]
  constexpr int kThreads = 128;
  constexpr int kStageFloats = (kStreamN + MP) * kStreamStride;
  constexpr int kQuads = kStreamK / 4;
  constexpr int kRows = MP / MM;
  static_assert(kRows == 1 || kRows == 2 || kRows == 4, "");
  struct Operands {
    float4 w[kStreamAhead], x[kStreamAhead][MM];
  };
  const int n0 = blockIdx.x * kStreamN;
  const int chunks = (K + kStreamK - 1) / kStreamK;
  // rows past N or M repeat the last one (their outputs are not stored); columns past K are zeros.  A warp copies whole rows of a stage.
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto copy_w = [&](int chunk) {
    float* stage = ring + (chunk % STAGES) * kStageFloats + lane * 4;
    const int k = chunk * kStreamK + lane * 4;
    const bool inside = k < K;
#pragma unroll
    for (int r = 0; r < kStreamN / 4; ++r)
      cp_async_16(stage + (warp + 4 * r) * kStreamStride, w + (long long)min(n0 + warp + 4 * r, N - 1) * K + (inside ? k : 0), inside);
  };
  auto copy_x = [&](int chunk) {
    float* stage = ring + (chunk % STAGES) * kStageFloats + kStreamN * kStreamStride + lane * 4;
    const int k = chunk * kStreamK + lane * 4;
    const bool inside = k < K;
    for (int r = warp; r < MP; r += 4) cp_async_16(stage + r * kStreamStride, x + (long long)min(r, M - 1) * lda + (inside ? k : 0), inside);
  };
  // While the kernel before this one runs, L2 fetches the first stages' weights.  Nothing is read: w may be what that kernel (or the one before it) writes.
  auto ask_for_w = [&](int chunk) {
    const int k = chunk * kStreamK + lane * 4;
#pragma unroll
    for (int r = 0; r < kStreamN / 4; ++r)
      if (k < K) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(w + (long long)min(n0 + warp + 4 * r, N - 1) * K + k));
  };
  for (int c = 0; c < STAGES - 1 && c < chunks; ++c) ask_for_w(c);
  grid_launch_dependents();
  grid_dependency_wait();
  for (int c = 0; c < STAGES - 1; ++c) {   // (empty groups keep the count)
    if (c < chunks) {
      copy_w(c);
      copy_x(c);
    }
    cp_async_commit();
  }
  // a warp is 8 outputs x 4 rows (16 x 1, 16 x 2); CTAs that share an SM compute in different warps, so on different schedulers
  constexpr int kWarpsNeeded = kRows == 4 ? 2 : 1;
  const int turn = (kThreads / 32 + warp - (int)((blockIdx.x / sms) * kWarpsNeeded & 3)) & 3;
  const bool computes = turn < kWarpsNeeded && (kRows > 1 || lane < 16);
  const int n = kRows == 4 ? turn * 8 + (lane & 7) : lane & 15;
  const int m = kRows == 4 ? lane >> 3 : (kRows == 2 ? lane >> 4 : 0);
  float acc[MM];
#pragma unroll
  for (int j = 0; j < MM; ++j) acc[j] = 0.0f;
  for (int c = 0; c < chunks; ++c) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();   // stage c is here for every thread, and everyone is done with the stage that is filled next
    if (c + STAGES - 1 < chunks) {
      copy_w(c + STAGES - 1);
      copy_x(c + STAGES - 1);
    }
    cp_async_commit();
    if (computes) {
      const unsigned stage = (unsigned)__cvta_generic_to_shared(ring + (c % STAGES) * kStageFloats);
      const unsigned ws = stage + n * kStreamStride * 4, xs = stage + (kStreamN + m) * kStreamStride * 4;
      // Two sets of operands in a rolled loop, one read while the other is used: what one pass of a loop reads for the next cannot be moved down to its use
      // (unrolled, the reads are, whatever their order in the source, and every step waited for shared memory).
      Operands even, odd;
      auto fetch = [&](Operands& to, int group) {
#pragma unroll
        for (int i = 0; i < kStreamAhead; ++i) {
          to.w[i] = read_four(ws + 16 * (group * kStreamAhead + i));
#pragma unroll
          for (int j = 0; j < MM; ++j) to.x[i][j] = read_four(xs + j * kRows * kStreamStride * 4 + 16 * (group * kStreamAhead + i));
        }
      };
      auto use = [&](const Operands& from) {
#pragma unroll
        for (int i = 0; i < kStreamAhead; ++i) {
#pragma unroll
          for (int j = 0; j < MM; ++j) acc[j] = fmaf(from.x[i][j].x, from.w[i].x, acc[j]);
#pragma unroll
          for (int j = 0; j < MM; ++j) acc[j] = fmaf(from.x[i][j].y, from.w[i].y, acc[j]);
#pragma unroll
          for (int j = 0; j < MM; ++j) acc[j] = fmaf(from.x[i][j].z, from.w[i].z, acc[j]);
#pragma unroll
          for (int j = 0; j < MM; ++j) acc[j] = fmaf(from.x[i][j].w, from.w[i].w, acc[j]);
        }
      };
      constexpr int kGroups = kQuads / kStreamAhead;
      fetch(even, 0);
#pragma unroll 1
      for (int group = 0; group < kGroups; group += 2) {
        fetch(odd, group + 1);
        use(even);
        fetch(even, group + 2 < kGroups ? group + 2 : 0);   // (the last pass reads something it has)
        use(odd);
      }
    }
  }
  if (!computes || n0 + n >= N) return;
#pragma unroll
  for (int j = 0; j < MM; ++j)
    if (m + j * kRows < M) out[(size_t)(m + j * kRows) * N + n0 + n] = acc[j];
}

template <int MP, int MM, int STAGES>
static int launch_stream_stages(const float* x, const float* w, float* out, int M, int N, int K, long long lda, cudaStream_t stream) {
  constexpr int smem = STAGES * (kStreamN + MP) * kStreamStride * (int)sizeof(float);
  static std::atomic<unsigned long long> devices{0};
  const cudaError_t allowed = allow_shared_memory(gemm_stream_f32_kernel<MP, MM, STAGES>, smem, devices);
  if (allowed != cudaSuccess) return (int)allowed;
  return (int)launch_pdl(gemm_stream_f32_kernel<MP, MM, STAGES>, dim3((N + kStreamN - 1) / kStreamN), dim3(128), smem, stream, x, w, out, M, N, K, lda, device_sm_count());
}

// MM rows per thread where a CTA has an SM (nearly) to itself and a sum's own chain is the time; MANY where there are more tiles than that and shared
// memory's bandwidth is (4 rows x 11,264 columns, K = 2,048: 27.4 us with one row per thread, 26 with two; x 32,000: 69 and 58; 8 rows x 11,264: 47 with two, 37 with four).
template <int MP, int MM, int MANY>
static int launch_stream(const float* x, const float* w, float* out, int M, int N, int K, long long lda, cudaStream_t stream) {
  if ((N + kStreamN - 1) / kStreamN <= 2 * device_sm_count()) return launch_stream_stages<MP, MM, 10>(x, w, out, M, N, K, lda, stream);
  return launch_stream_stages<MP, MANY, 4>(x, w, out, M, N, K, lda, stream);
}

// --- more rows ---------------------------------------------------------------------------------------
constexpr int kTileStages = 4;
constexpr int kWideK = 16;
constexpr int kWideStride = kWideK + 4;   // as above: 8 rows' 16-byte reads in one pass over the banks

// A warp is 4 x 8 lanes, a lane TM x TN outputs: rows lane / 8 + 4 i, columns lane % 8 + 8 j (the eight lanes of one pass over the banks read eight
// neighbouring weight rows, and one row of x).  Held back by what shared memory delivers, 16 values of four bytes per lane and k in the time of 64
// multiply-adds: 45 TFLOP/s at 2,048 rows with 8 x 8 outputs per lane, of 72 (the plain kernel: 22; 8 x 16 outputs in twice the registers: 44; the next step's
// operands read into a second set of registers: 43).
template <int TM, int TN, int WM, int WN>
__global__ void __launch_bounds__(WM * WN * 32) gemm_wide_f32_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                     float* __restrict__ out, int M, int N, int K, long long lda) {
  extern __shared__ __align__(16) float ring[];   // [stages][BM + BN][kWideStride]
  constexpr int LM = 4, LN = 8;
  constexpr int BM = TM * LM * WM, BN = TN * LN * WN;
  constexpr int kThreads = WM * WN * 32;
  constexpr int kStageFloats = (BM + BN) * kWideStride;
  constexpr int kCopies = (BM + BN) * (kWideK / 4) / kThreads;
  static_assert((BM + BN) * (kWideK / 4) % kThreads == 0, "every thread copies as much");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int m_blocks = (M + BM - 1) / BM;
  const int row0 = (blockIdx.x % m_blocks) * BM, col0 = (blockIdx.x / m_blocks) * BN;   // neighbours share their weights
  const float* source[kCopies];
#pragma unroll
  for (int i = 0; i < kCopies; ++i) {
    const int r = (threadIdx.x + i * kThreads) / (kWideK / 4);
    source[i] = r < BM ? x + (long long)min(row0 + r, M - 1) * lda : w + (long long)min(col0 + r - BM, N - 1) * K;
  }
  const int k_of = (threadIdx.x % (kWideK / 4)) * 4;
  auto copy = [&](int chunk) {
    const int k = chunk * kWideK + k_of;
    const bool inside = k < K;
    float* stage = ring + (chunk % kTileStages) * kStageFloats + k_of;
#pragma unroll
    for (int i = 0; i < kCopies; ++i)
      cp_async_16(stage + ((threadIdx.x + i * kThreads) / (kWideK / 4)) * kWideStride, source[i] + (inside ? k : 0), inside);
  };
  const int chunks = (K + kWideK - 1) / kWideK;
  grid_launch_dependents();
  grid_dependency_wait();
  for (int c = 0; c < kTileStages - 1; ++c) {
    if (c < chunks) copy(c);
    cp_async_commit();
  }
  const int m_of = (warp % WM) * TM * LM + (lane >> 3);
  const int n_of = (warp / WM) * TN * LN + (lane & 7);
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
  for (int c = 0; c < chunks; ++c) {
    cp_async_wait<kTileStages - 2>();
    __syncthreads();
    if (c + kTileStages - 1 < chunks) copy(c + kTileStages - 1);
    cp_async_commit();
    const float* xs = ring + (c % kTileStages) * kStageFloats + m_of * kWideStride;
    const float* ws = ring + (c % kTileStages) * kStageFloats + (BM + n_of) * kWideStride;
#pragma unroll
    for (int q = 0; q < kWideK / 4; ++q) {
      float4 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(xs + LM * i * kWideStride + 4 * q);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float4 b = *reinterpret_cast<const float4*>(ws + LN * j * kWideStride + 4 * q);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int row = row0 + m_of + LM * i;
    if (row >= M) break;
#pragma unroll
    for (int j = 0; j < TN; ++j)
      if (col0 + n_of + LN * j < N) out[(size_t)row * N + col0 + n_of + LN * j] = acc[i][j];
  }
}

static long long wide_tiles(int M, int N, int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); }

template <int TM, int TN, int WM, int WN>
static int launch_wide(const float* x, const float* w, float* out, int M, int N, int K, long long lda, cudaStream_t stream) {
  constexpr int BM = TM * 4 * WM, BN = TN * 8 * WN;
  constexpr int smem = kTileStages * (BM + BN) * kWideStride * (int)sizeof(float);
  static std::atomic<unsigned long long> devices{0};
  const cudaError_t allowed = allow_shared_memory(gemm_wide_f32_kernel<TM, TN, WM, WN>, smem, devices);
  if (allowed != cudaSuccess) return (int)allowed;
  return (int)launch_pdl(gemm_wide_f32_kernel<TM, TN, WM, WN>, dim3((unsigned)wide_tiles(M, N, BM, BN)), dim3(WM * WN * 32), smem, stream, x, w, out, M, N, K, lda);
}

// Which tile: the time of a product is that of the SM with the most tiles, about linear in their number.  Fitted to measurements at K = 2,048 alone: `each` grows with K and `once` does not, so at
// a larger K the rule weighs the first tile's wait too much, which matters where two tiles are close.
// In us (a first tile that has the SM to itself waits for its own loads, the 8 x 8 tiles most): 24 rows x 2,048 columns 119 / 87 / 57 for the three tiles,
// 150 x 11,264 257 / 200 / 210, 300 x 11,264 341 / 386 / 398, 760 x 11,264 853 / 934 / 927 (the plain kernel: 387, 523, 743, 1,717).
static int wide_choice(int M, int N) {
  const int sms = device_sm_count();
  const int bm[3] = {64, 32, 32}, bn[3] = {64, 128, 64};
  const float each[3] = {57.0f, 62.0f, 32.0f}, once[3] = {40.0f, 25.0f, 25.0f};
  int best = 0;
  float least = 0.0f;
  for (int i = 0; i < 3; ++i) {
    const float time = each[i] * (float)((wide_tiles(M, N, bm[i], bn[i]) + sms - 1) / sms) + once[i];
    if (i == 0 || time < least) {
      best = i;
      least = time;
    }
  }
  return best;
}

}  // namespace tlie

using namespace tlie;

TLIE_EXPORT int tlie_gemm_nt_f32(const float* x, const float* w, float* out, int M, int N, int K, long long lda,
                                 cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || lda < K) return (int)cudaErrorInvalidValue;
  if (K % 4 == 0 && lda % 4 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0) {
    if (M == 1) return launch_stream<1, 1, 1>(x, w, out, M, N, K, lda, stream);
    if (M == 2) return launch_stream<2, 1, 1>(x, w, out, M, N, K, lda, stream);
    if (M <= 4) return launch_stream<4, 1, 2>(x, w, out, M, N, K, lda, stream);
    if (M <= 8) return launch_stream<8, 2, 4>(x, w, out, M, N, K, lda, stream);
    if (M <= 16) return launch_stream<16, 4, 4>(x, w, out, M, N, K, lda, stream);
    switch (wide_choice(M, N)) {
      case 0: return launch_wide<8, 8, 2, 1>(x, w, out, M, N, K, lda, stream);    // 64 x 64
      case 1: return launch_wide<4, 8, 2, 2>(x, w, out, M, N, K, lda, stream);    // 32 x 128
      default: return launch_wide<4, 4, 2, 2>(x, w, out, M, N, K, lda, stream);   // 32 x 64
    }
  }
  dim3 grid((N + kTile - 1) / kTile, (M + kTile - 1) / kTile);
  gemm_nt_f32_kernel<<<grid, 256, 0, stream>>>(x, w, out, M, N, K, lda);
  return (int)cudaGetLastError();
}
