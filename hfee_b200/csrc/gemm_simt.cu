// out[M,N] (+)= A[M,K] . W[N,K]^T with float32 FFMA accumulation on the CUDA cores.
//
// This is the matrix product of the true 32-bit path (no tensor cores, no
// reduced-precision mode) and the fallback of the bfloat16 path for shapes the
// tensor-core kernels refuse.  Every output element is summed in one order, whatever M is and whichever of
// the kernels below runs, so a row's result does not depend on the batch: K is cut into segments of SEG, a segment is
// two chains of fused multiply-adds, over its even and over its odd k, and the segments' sums (even + odd) are added in their
// order.  One chain over all of K would take 4 clocks for each k (17 us at K = 8,192, whatever the number of warps); segments
// can run side by side, the sums of shorter chains are closer to the exact ones, and two neighbouring k lie as the pair that
// the packed multiply-add takes: single FFMA issue at half of the rate on this chip (a 64-row tile that did nothing else stopped at
// 29 TFLOP/s).
//
// Three kernels.  float32 operands whose rows start on 16-byte boundaries take `gemm_rows_kernel` (at most
// ROWS_MAX_M tokens) or `gemm_tiles_kernel` (more) unless their sums are short; bfloat16 operands, other alignments and short sums
// (`short_sums`) take `gemm_simt_kernel`.
// Reference: out[t*Rows+r] = Dot(W[r,:], x[t,:]), hostfog/hfee internal/ggml/ops.go:54-70.
#include <atomic>
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4, THREADS = 256;
constexpr unsigned EARLY_BLOCKS = 128;      // grids of no more than these let the kernel behind in at once
constexpr int SEG = 512;        // k of a segment; a multiple of every kernel's piece of K

template <typename T>
__device__ __forceinline__ float load_guarded(const T* p, long long ld, int r, int c, int rows, int cols) {
  return (r < rows && c < cols) ? to_f32<T>(p[(long long)r * ld + c]) : 0.f;
}

// TOut: float or bf16.  ACCUM (float out only): out += product (the residual add).  ONE: K is one segment, without the segments' sums
// (2,048 x 8,192 x 512 732 us with them, 676 without).  Three blocks an SM: with registers for two 700 x 2,048 x 512 in bfloat16 takes 102 us in
// place of 77, with four 99.
template <typename TIn, typename TOut, bool ACCUM, bool ONE>
__global__ void __launch_bounds__(THREADS, 3)
gemm_simt_kernel(const TIn* __restrict__ A, long long lda, const TIn* __restrict__ W, long long ldw,
                 TOut* __restrict__ C, long long ldc, int M, int N, int K) {
  pdl_wait();
  // blocks of a kernel behind that are let in while this one has one or two an SM settle unevenly: 2,048 x 512 x 512 79 us in a row of such
  const bool early = gridDim.x * gridDim.y <= EARLY_BLOCKS;
  if (early) pdl_launch_dependents();
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  int tid = threadIdx.x;
  int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  int tr = tid / (BN / TN), tc = tid % (BN / TN);   // 16 x 16 thread grid
  float acc[2][TM][TN], sum[TM][TN];    // of this segment (even and odd k), of the segments before it
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[0][i][j] = acc[1][i][j] = sum[i][j] = 0.f;
  auto add = [&]() {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) { sum[i][j] += acc[0][i][j] + acc[1][i][j]; acc[0][i][j] = acc[1][i][j] = 0.f; }
  };

  // each thread stages 4 consecutive k of one row of A and one row of W, asked for while the piece before is multiplied
  int lr = tid / (BK / 4), lk = (tid % (BK / 4)) * 4;   // 64 rows x 4 groups
  float next_a[4], next_w[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      next_a[j] = load_guarded(A, lda, m0 + lr, k0 + lk + j, M, K);
      next_w[j] = load_guarded(W, ldw, n0 + lr, k0 + lk + j, N, K);
    }
  };
  fetch(0);
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      As[lk + j][lr] = next_a[j];
      Ws[lk + j][lr] = next_w[j];
    }
    if (k0 + BK < K) fetch(k0 + BK);
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][tr * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = Ws[kk][tc * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[kk & 1][i][j] = fmaf(a[i], b[j], acc[kk & 1][i][j]);
    }
    __syncthreads();
    if (!ONE && (k0 + BK) % SEG == 0 && k0 + BK < K) add();
  }
  add();
  if (!early) pdl_launch_dependents();
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    int r = m0 + tr * TM + i;
    if (r >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      int c = n0 + tc * TN + j;
      if (c >= N) continue;
      long long o = (long long)r * ldc + c;
      if constexpr (ACCUM) C[o] = to_f32<TOut>(C[o]) + sum[i][j];
      else C[o] = from_f32<TOut>(sum[i][j]);
    }
  }
}

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Two float32 multiply-adds, of the low and of the high halves.
__device__ __forceinline__ void fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ float halves(unsigned long long v) { return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32)); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A decode step of the 32-bit path, bound by the bytes of W (each read once).  A CTA owns 16 rows of W; its warps take the
// segments of K in turn, each with its own ring of STAGES pieces [16 rows + tokens][KT] that 16-byte asynchronous copies fill,
// and lane l sums row l & 15 with TPL tokens (l >> 4, l >> 4 + 2, ..).  After every round of one segment a warp the sums meet in
// shared memory and warp 0 adds them in the segments' order.  Rows are KT + 4 floats apart, so that eight lanes' 16-byte reads
// fall into different banks.  W does not depend on the kernel in front: its first pieces are requested before the wait for it.
// 1B layer sizes at two tokens, a warp for each segment against one for all of K: o + down projection 23.6 against 73 us a layer
// (the chain of 8,192 additions alone is 17; the bytes 13), q/k/v + gate/up 39 against 53 us (25).
constexpr int ROWS_KT = 32, ROWS_STAGES = 4;

template <int TPL, int WARPS, typename TOut, bool ACCUM>
__global__ void __launch_bounds__(WARPS * 32)
gemm_rows_kernel(const float* __restrict__ A, long long lda, const float* __restrict__ W, long long ldw,
                 TOut* __restrict__ C, long long ldc, int M, int N, int K) {
  constexpr int KT = ROWS_KT, STAGES = ROWS_STAGES, LD = KT + 4, CHUNKS = KT / 4, STAGE = (16 + 2 * TPL) * LD, PIECES = SEG / KT;
  extern __shared__ __align__(16) float rows_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = lane & 15, g = lane >> 4;
  float* ring = rows_smem + warp * (STAGES * STAGE);
  float* parts = rows_smem + WARPS * (STAGES * STAGE);            // [2][WARPS][TPL][32]
  const int n0 = blockIdx.x * 16;
  const int rounds = (K + SEG * WARPS - 1) / (SEG * WARPS), steps = rounds * PIECES;

  auto first_k = [&](int step) { return ((step / PIECES) * WARPS + warp) * SEG + (step % PIECES) * KT; };
  auto load_w = [&](int step) {
    float* dst = ring + (step % STAGES) * STAGE;
    const int k0 = first_k(step);
#pragma unroll
    for (int i = 0; i < 16 * CHUNKS / 32; ++i) {
      const int c = lane + 32 * i, r = c / CHUNKS, k = (c % CHUNKS) * 4;
      if (k0 + k < K) cp_async16(dst + r * LD + k, W + (long long)min(n0 + r, N - 1) * ldw + k0 + k);
    }
  };
  auto load_a = [&](int step) {
    float* dst = ring + (step % STAGES) * STAGE + 16 * LD;
    const int k0 = first_k(step);
    for (int c = lane; c < M * CHUNKS; c += 32) {
      const int r = c / CHUNKS, k = (c % CHUNKS) * 4;
      if (k0 + k < K) cp_async16(dst + r * LD + k, A + (long long)r * lda + k0 + k);
    }
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) load_w(s);
  pdl_wait();
  pdl_launch_dependents();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    load_a(s);
    cp_async_commit();
  }

  unsigned long long acc[TPL];
  float sum[TPL];
#pragma unroll
  for (int t = 0; t < TPL; ++t) { acc[t] = 0; sum[t] = 0.f; }
  auto four = [&](const float* wr, const float* xr, int k) {
    const ulonglong2 w = *(const ulonglong2*)(wr + k);
    ulonglong2 x[TPL];
#pragma unroll
    for (int t = 0; t < TPL; ++t) x[t] = *(const ulonglong2*)(xr + 2 * t * LD + k);
#pragma unroll
    for (int t = 0; t < TPL; ++t) fma2(acc[t], x[t].x, w.x);
#pragma unroll
    for (int t = 0; t < TPL; ++t) fma2(acc[t], x[t].y, w.y);
  };
#pragma unroll 1
  for (int step = 0; step < steps; ++step) {
    cp_async_wait<STAGES - 2>();
    __syncwarp();                               // this piece is everybody's; the piece before it has been read by all
    if (step + STAGES - 1 < steps) {
      load_w(step + STAGES - 1);
      load_a(step + STAGES - 1);
    }
    cp_async_commit();
    const float* wr = ring + (step % STAGES) * STAGE + row * LD;
    const float* xr = ring + (step % STAGES) * STAGE + (16 + g) * LD;
    const int left = K - first_k(step);
    if (left >= KT) {
#pragma unroll
      for (int k = 0; k < KT; k += 4) four(wr, xr, k);
    } else {
      for (int k = 0; k < left; k += 4) four(wr, xr, k);
    }
    if (step % PIECES == PIECES - 1) {          // the round's segments are done; the buffer before last is free again by now
      const int round = step / PIECES;
      float* mine = parts + (round & 1) * (WARPS * TPL * 32);
#pragma unroll
      for (int t = 0; t < TPL; ++t) { mine[(warp * TPL + t) * 32 + lane] = halves(acc[t]); acc[t] = 0; }
      __syncthreads();
      if (warp == 0)
        for (int w = 0; w < WARPS && (round * WARPS + w) * SEG < K; ++w)
#pragma unroll
          for (int t = 0; t < TPL; ++t) sum[t] += mine[(w * TPL + t) * 32 + lane];
    }
  }
  const int n = n0 + row;
  if (warp != 0 || n >= N) return;
#pragma unroll
  for (int t = 0; t < TPL; ++t) {
    const int m = g + 2 * t;
    if (m >= M) continue;
    const long long o = (long long)m * ldc + n;
    if constexpr (ACCUM) C[o] = to_f32<TOut>(C[o]) + sum[t];
    else C[o] = from_f32<TOut>(sum[t]);
  }
}

// Prompts of the 32-bit path, bound by the FFMA rate (128 a clock and SM) and, right behind it, by shared memory, which gives a
// lane 4 bytes a clock: a thread with a x b outputs needs a + b floats for a b / 4 clocks of FFMA, so 8 x 8 is the smallest
// square that keeps up (4 x 4 stopped at 42 % of the rate).  A warp owns a whole tile of 32 x 64 outputs over one segment of K,
// with its own ring of pieces filled by 16-byte asynchronous copies, and the four warps of a CTA take the segments of the same
// tile in turn: short prompts have few tiles, and this way each fills an SM's four schedulers.  After every round the sums of
// the four meet in shared memory, a quarter of the outputs at a time, and are added in the segments' order; each warp keeps
// the running sums of its quarter.  The next pair of k is read while one is multiplied, and two CTAs share an SM, for which the
// launch asks for all of its shared memory: with the step's carve-out one CTA fits, and its four warps stop at 25 TFLOP/s.
// The four products of a 1B layer at 285 tokens: 954 us, with tiles of 32 x 64 and 4 x 4 a thread 1,220.  8 x 16 a thread spills.
// Rows and columns that are not there are not read (whatever lies in their place gives outputs that nobody stores): read again from the
// last row, all tiles' copies met in one line (33 tokens, N = 8,192, K = 1,024: 75 us, 64 tokens 62).
// A thread's rows lie 4 and its columns 8 apart, rows of a piece KT + 4 floats: no bank is hit
// twice.  M tiles run fastest over the grid, so that a W tile is read from L2 by its row tiles.
constexpr int TILE_M = 32, TILE_N = 64, TILE_KT = 16, TILE_STAGES = 3, TILE_WARPS = 4;
constexpr int TILE_LD = TILE_KT + 4, TILE_STAGE = (TILE_M + TILE_N) * TILE_LD;
constexpr int TILES_SMEM = (TILE_WARPS * TILE_STAGES * TILE_STAGE + TILE_WARPS * 16 * 32) * 4;

template <typename TOut, bool ACCUM>
__global__ void __launch_bounds__(TILE_WARPS * 32, 2)
gemm_tiles_kernel(const float* __restrict__ A, long long lda, const float* __restrict__ W, long long ldw,
                  TOut* __restrict__ C, long long ldc, int M, int N, int K, int m_tiles) {
  constexpr int KT = TILE_KT, STAGES = TILE_STAGES, LD = TILE_LD, STAGE = TILE_STAGE, CHUNKS = KT / 4, PIECES = SEG / KT, WARPS = TILE_WARPS;
  extern __shared__ __align__(16) float tiles_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tr = lane >> 3, tc = lane & 7;
  float* ring = tiles_smem + warp * (STAGES * STAGE);
  float* parts = tiles_smem + WARPS * (STAGES * STAGE);           // [WARPS][16][32]
  const int m0 = (blockIdx.x % m_tiles) * TILE_M, n0 = (blockIdx.x / m_tiles) * TILE_N;
  const int rounds = (K + SEG * WARPS - 1) / (SEG * WARPS), steps = rounds * PIECES;

  auto first_k = [&](int step) { return ((step / PIECES) * WARPS + warp) * SEG + (step % PIECES) * KT; };
  const int lr = lane / CHUNKS, lk = (lane % CHUNKS) * 4;          // 8 rows of a piece an instruction
  auto load_w = [&](int step) {
    float* dst = ring + (step % STAGES) * STAGE + (TILE_M + lr) * LD + lk;
    const int k = first_k(step) + lk;
    if (k < K)
#pragma unroll
      for (int i = 0; i < TILE_N / 8; ++i)
        if (n0 + lr + i * 8 < N) cp_async16(dst + i * 8 * LD, W + (long long)(n0 + lr + i * 8) * ldw + k);
  };
  auto load_a = [&](int step) {
    float* dst = ring + (step % STAGES) * STAGE + lr * LD + lk;
    const int k = first_k(step) + lk;
    if (k < K)
#pragma unroll
      for (int i = 0; i < TILE_M / 8; ++i)
        if (m0 + lr + i * 8 < M) cp_async16(dst + i * 8 * LD, A + (long long)(m0 + lr + i * 8) * lda + k);
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) load_w(s);
  pdl_wait();
  pdl_launch_dependents();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    load_a(s);
    cp_async_commit();
  }
  unsigned long long acc[8][8];
  float sum[16];                                // sum: this warp's quarter, acc's rows 2 warp and 2 warp + 1 of every lane
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0;
#pragma unroll
  for (int e = 0; e < 16; ++e) sum[e] = 0.f;
#pragma unroll 1
  for (int step = 0; step < steps; ++step) {
    cp_async_wait<STAGES - 2>();
    __syncwarp();
    if (step + STAGES - 1 < steps) {
      load_w(step + STAGES - 1);
      load_a(step + STAGES - 1);
    }
    cp_async_commit();
    const float* as = ring + (step % STAGES) * STAGE + tr * LD;
    const float* ws = ring + (step % STAGES) * STAGE + (TILE_M + tc) * LD;
    unsigned long long a[2][8], b[2][8];          // the pairs of k being multiplied and the next ones
    auto read = [&](int buf, int k) {
#pragma unroll
      for (int i = 0; i < 8; ++i) a[buf][i] = *(const unsigned long long*)(as + i * 4 * LD + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) b[buf][j] = *(const unsigned long long*)(ws + j * 8 * LD + k);
    };
    auto multiply = [&](int buf) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) fma2(acc[i][j], a[buf][i], b[buf][j]);
    };
    const int left = K - first_k(step);
    if (left >= KT) {
      read(0, 0);
#pragma unroll
      for (int k = 0; k < KT; k += 2) {
        if (k + 2 < KT) read((k / 2 + 1) & 1, k + 2);
        multiply((k / 2) & 1);
      }
    } else {
#pragma unroll 1
      for (int k = 0; k < left; k += 2) {
        read(0, k);
        multiply(0);
      }
    }
    if (step % PIECES == PIECES - 1) {          // the round's segments are done
      const int live = min(WARPS, (K - (step / PIECES) * WARPS * SEG + SEG - 1) / SEG);
#pragma unroll
      for (int q = 0; q < WARPS; ++q) {         // the outputs whose sums warp q keeps
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 16; ++e) parts[(warp * 16 + e) * 32 + lane] = halves(acc[2 * q + e / 8][e % 8]);
        __syncthreads();
        if (warp == q)
          for (int w = 0; w < live; ++w)
#pragma unroll
            for (int e = 0; e < 16; ++e) sum[e] += parts[(w * 16 + e) * 32 + lane];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0;
    }
  }
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const int m = m0 + tr + (2 * warp + e / 8) * 4, n = n0 + tc + (e % 8) * 8;
    if (m >= M || n >= N) continue;
    const long long o = (long long)m * ldc + n;
    if constexpr (ACCUM) C[o] = to_f32<TOut>(C[o]) + sum[e];
    else C[o] = from_f32<TOut>(sum[e]);
  }
}

constexpr int ROWS_MAX_M = 16;

// Which devices have been asked for a kernel's shared memory: the consent is each device's own.
struct OptIn {
  std::atomic<unsigned long long> asked{0};
  template <typename Kernel>
  bool room(Kernel kernel, int bytes) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return false;
    const unsigned long long bit = device < 64 ? 1ull << device : 0;
    if (asked.load(std::memory_order_relaxed) & bit) return true;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return false;
    asked.fetch_or(bit, std::memory_order_relaxed);
    return true;
  }
};

template <int TPL, int WARPS, typename TOut, bool ACCUM>
int launch_rows_of(const float* A, long long lda, const float* W, long long ldw, TOut* C, long long ldc, int M, int N, int K,
                   cudaStream_t stream) {
  constexpr int smem = WARPS * (ROWS_STAGES * (16 + 2 * TPL) * (ROWS_KT + 4) + 2 * TPL * 32) * 4;
  static OptIn opted;
  if (!opted.room(gemm_rows_kernel<TPL, WARPS, TOut, ACCUM>, smem)) return hfee_fail(HFEE_ERR_CUDA, "gemm_simt: no shared memory for its rings");
  hfee_launch(gemm_rows_kernel<TPL, WARPS, TOut, ACCUM>, dim3((N + 15) / 16), dim3(WARPS * 32), smem, stream, A, lda, W, ldw, C, ldc,
              M, N, K);
  return hfee_check_launch("gemm_simt rows");
}

// As many warps as there are segments, up to eight.
template <int TPL, typename TOut, bool ACCUM>
int launch_rows(const float* A, long long lda, const float* W, long long ldw, TOut* C, long long ldc, int M, int N, int K,
                cudaStream_t stream) {
  if (K <= SEG) return launch_rows_of<TPL, 1, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  if (K <= 4 * SEG) return launch_rows_of<TPL, 4, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  return launch_rows_of<TPL, 8, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
}

template <typename TOut, bool ACCUM>
int launch_f32(const float* A, long long lda, const float* W, long long ldw, TOut* C, long long ldc, int M, int N, int K,
               cudaStream_t stream) {
  // Up to ROWS_MAX_M tokens the bytes of W bound the product; TPL tokens a lane cost TPL FFMA per weight.
  if (M <= 2) return launch_rows<1, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  if (M <= 4) return launch_rows<2, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  if (M <= 8) return launch_rows<4, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  if (M <= ROWS_MAX_M) return launch_rows<8, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  static OptIn opted;
  if (!opted.room(gemm_tiles_kernel<TOut, ACCUM>, TILES_SMEM)) return hfee_fail(HFEE_ERR_CUDA, "gemm_simt: no shared memory for its tiles");
  const int m_tiles = (M + TILE_M - 1) / TILE_M;
  const long long tiles = (long long)m_tiles * ((N + TILE_N - 1) / TILE_N);
  HFEE_REQUIRE(tiles <= 0x7fffffff, "gemm_simt: M=%d N=%d are too large", M, N);
  hfee_launch_carved(100, gemm_tiles_kernel<TOut, ACCUM>, dim3((unsigned)tiles), dim3(TILE_WARPS * 32), TILES_SMEM, stream, A, lda, W, ldw, C, ldc, M, N, K,
              m_tiles);
  return hfee_check_launch("gemm_simt tiles");
}

// Products whose sums are too short for the two kernels above, which the general one takes (its blocks are 64 x 64; the order of the sums
// is the same).  us, the kernel above / the general one.  A decode step's ring of copies: 8 tokens, N = 512: K = 32 4.9 / 2.8, 64 5.1 / 4.4,
// 96 5.3 / 5.9.  The tiles give each of their four warps whole segments, so up to K = 512 three have nothing to do and up to 1,024 two: 2,048
// tokens, N = 2,048: K = 32 54 / 15, 256 145 / 89, 512 248 / 172, 640 259 / 234, 768 268 / 312, 1,024 325 / 375.  Where all tiles fit the chip
// side by side they take what one segment takes: 285 tokens, N = 512: K = 512 35 / 30, 640 35 / 42; and up to K = 512 they win only where
// the general kernel's blocks do not fit: 285 tokens, N = 2,048: K = 128 14.0 / 13.7, 256 21.5 / 25.6, 512 36 / 49.
bool short_sums(int M, int N, int K) {
  if (M <= ROWS_MAX_M) return K <= 64;
  if (K >= 3 * SEG / 2 || (M + BM - 1) / BM > 65535) return false;      // (rows of blocks a grid can have)
  const long long sms = hfee_sm_count();
  const long long tiles = (long long)((M + TILE_M - 1) / TILE_M) * ((N + TILE_N - 1) / TILE_N);
  const long long blocks = (long long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  return tiles > 2 * sms || K < SEG / 2 || (K <= SEG && blocks <= sms);
}

template <typename TIn>
int launch(const void* A, long long lda, const void* W, long long ldw, void* C, long long ldc, int out_dtype,
           int accumulate, int M, int N, int K, cudaStream_t stream) {
  if constexpr (sizeof(TIn) == 4) {
    const bool aligned = !short_sums(M, N, K) && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
    if (aligned && out_dtype == HFEE_F32)
      return accumulate ? launch_f32<float, true>((const float*)A, lda, (const float*)W, ldw, (float*)C, ldc, M, N, K, stream)
                        : launch_f32<float, false>((const float*)A, lda, (const float*)W, ldw, (float*)C, ldc, M, N, K, stream);
    if (aligned && out_dtype == HFEE_BF16 && !accumulate)
      return launch_f32<__nv_bfloat16, false>((const float*)A, lda, (const float*)W, ldw, (__nv_bfloat16*)C, ldc, M, N, K, stream);
  }
  const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  auto run = [&](auto kernel, auto* out) {
    hfee_launch(kernel, grid, dim3(THREADS), 0, stream, (const TIn*)A, lda, (const TIn*)W, ldw, out, ldc, M, N, K);
    return hfee_check_launch("gemm_simt");
  };
  const bool one = K <= SEG;
  if (out_dtype == HFEE_F32) {
    if (accumulate) return run(one ? gemm_simt_kernel<TIn, float, true, true> : gemm_simt_kernel<TIn, float, true, false>, (float*)C);
    return run(one ? gemm_simt_kernel<TIn, float, false, true> : gemm_simt_kernel<TIn, float, false, false>, (float*)C);
  }
  if (out_dtype != HFEE_BF16) return hfee_fail(HFEE_ERR_ARG, "gemm_simt: unknown output dtype %d", out_dtype);
  if (accumulate) return hfee_fail(HFEE_ERR_ARG, "gemm_simt: accumulate needs a float32 output");
  return run(one ? gemm_simt_kernel<TIn, __nv_bfloat16, false, true> : gemm_simt_kernel<TIn, __nv_bfloat16, false, false>, (__nv_bfloat16*)C);
}

}  // namespace

HFEE_API int hfee_gemm_simt(const void* A, long long lda, const void* W, long long ldw, int in_dtype, void* C,
                            long long ldc, int out_dtype, int accumulate, int M, int N, int K,
                            cudaStream_t stream) {
  if (M == 0 || N == 0) return HFEE_OK;
  HFEE_REQUIRE(M > 0 && N > 0 && K > 0 && lda >= K && ldw >= K && ldc >= N,
               "gemm_simt: bad sizes M=%d N=%d K=%d lda=%lld ldw=%lld ldc=%lld", M, N, K, lda, ldw, ldc);
  HFEE_REQUIRE((M + BM - 1) / BM <= 65535, "gemm_simt: M=%d is too large", M);
  if (in_dtype == HFEE_F32) return launch<float>(A, lda, W, ldw, C, ldc, out_dtype, accumulate, M, N, K, stream);
  if (in_dtype == HFEE_BF16) return launch<__nv_bfloat16>(A, lda, W, ldw, C, ldc, out_dtype, accumulate, M, N, K, stream);
  return hfee_fail(HFEE_ERR_ARG, "gemm_simt: unknown input dtype %d", in_dtype);
}
