// out[M,N] (+)= A[M,K] . W[N,K]^T with float32 FFMA accumulation on the CUDA cores.
//
// This is the matrix product of the true 32-bit path (no tensor cores, no
// reduced-precision mode) and the fallback of the bfloat16 path for shapes the
// tensor-core kernels refuse.  Every output element is the sum over k = 0..K-1 in
// that order, whatever M is and whichever of the kernels below runs, so a row's result does
// not depend on the batch.
//
// Three kernels.  float32 operands whose rows start on 16-byte boundaries take `gemm_rows_kernel` (at most
// ROWS_MAX_M tokens) or `gemm_tiles_kernel` (more); bfloat16 operands and other alignments take `gemm_simt_kernel`.
// Reference: out[t*Rows+r] = Dot(W[r,:], x[t,:]), hostfog/hfee internal/ggml/ops.go:54-70.
#include <type_traits>

#include "common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4, THREADS = 256;

template <typename T>
__device__ __forceinline__ float load_guarded(const T* p, long long ld, int r, int c, int rows, int cols) {
  return (r < rows && c < cols) ? to_f32<T>(p[(long long)r * ld + c]) : 0.f;
}

// TOut: float or bf16.  ACCUM (float out only): out += product (the residual add).
template <typename TIn, typename TOut, bool ACCUM>
__global__ void __launch_bounds__(THREADS)
gemm_simt_kernel(const TIn* __restrict__ A, long long lda, const TIn* __restrict__ W, long long ldw,
                 TOut* __restrict__ C, long long ldc, int M, int N, int K) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  int tid = threadIdx.x;
  int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  int tr = tid / (BN / TN), tc = tid % (BN / TN);   // 16 x 16 thread grid
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  // each thread stages 4 consecutive k of one row of A and one row of W
  int lr = tid / (BK / 4), lk = (tid % (BK / 4)) * 4;   // 64 rows x 4 groups
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      As[lk + j][lr] = load_guarded(A, lda, m0 + lr, k0 + lk + j, M, K);
      Ws[lk + j][lr] = load_guarded(W, ldw, n0 + lr, k0 + lk + j, N, K);
    }
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
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    int r = m0 + tr * TM + i;
    if (r >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      int c = n0 + tc * TN + j;
      if (c >= N) continue;
      long long o = (long long)r * ldc + c;
      if constexpr (ACCUM) C[o] = to_f32<TOut>(C[o]) + acc[i][j];
      else C[o] = from_f32<TOut>(acc[i][j]);
    }
  }
}

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A decode step of the 32-bit path.  Bound by the bytes of W (each read once) and, for long rows, by the chain of K
// dependent additions that one output is (4 clocks each: 17 us at K = 8,192): so an output is one lane's, and what is
// left to do is to keep the loads running.  One warp per CTA owns 16 rows of W (lane & 15) and two groups of TPL tokens
// (lane >> 4), and has its own ring of STAGES pieces [16 rows + tokens][KT], filled by 16-byte asynchronous copies; N =
// 2,048 then gives 128 SMs a warp each, N = 16,384 seven.  Rows are KT + 4 floats apart, so that eight lanes' 16-byte
// reads fall into different banks.  W does not depend on the kernel in front: its first pieces are requested before the
// wait for it.  Llama-3.2-1B layer sizes at two tokens: o + down projection 74 us a layer against 797 us with the general
// kernel's 64-row tiles.
template <int TPL, int KT, int STAGES, typename TOut, bool ACCUM>
__global__ void __launch_bounds__(32)
gemm_rows_kernel(const float* __restrict__ A, long long lda, const float* __restrict__ W, long long ldw,
                 TOut* __restrict__ C, long long ldc, int M, int N, int K) {
  constexpr int LD = KT + 4, CHUNKS = KT / 4, STAGE = (16 + 2 * TPL) * LD;
  extern __shared__ __align__(16) float ring[];
  const int lane = threadIdx.x, row = lane & 15, g = lane >> 4;
  const int n0 = blockIdx.x * 16, steps = (K + KT - 1) / KT;

  auto load_w = [&](int step) {
    float* dst = ring + (step % STAGES) * STAGE;
#pragma unroll
    for (int i = 0; i < 16 * CHUNKS / 32; ++i) {
      const int c = lane + 32 * i, r = c / CHUNKS, k = (c % CHUNKS) * 4;
      if (step * KT + k < K) cp_async16(dst + r * LD + k, W + (long long)min(n0 + r, N - 1) * ldw + step * KT + k);
    }
  };
#pragma unroll 1
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < steps) load_w(s);
    cp_async_commit();
  }
  pdl_wait();
  pdl_launch_dependents();
  for (int s = 0; s < min(STAGES - 1, steps); ++s)
    for (int c = lane; c < M * CHUNKS; c += 32) {
      const int r = c / CHUNKS, k = (c % CHUNKS) * 4;
      if (s * KT + k < K)
        *(float4*)(ring + s * STAGE + (16 + r) * LD + k) = *(const float4*)(A + (long long)r * lda + s * KT + k);
    }

  float acc[TPL];
#pragma unroll
  for (int t = 0; t < TPL; ++t) acc[t] = 0.f;
  auto four = [&](const float* wr, const float* xr, int k) {
    const float4 w = *(const float4*)(wr + k);
    float4 x[TPL];
#pragma unroll
    for (int t = 0; t < TPL; ++t) x[t] = *(const float4*)(xr + 2 * t * LD + k);
#pragma unroll
    for (int t = 0; t < TPL; ++t) acc[t] = fmaf(x[t].x, w.x, acc[t]);
#pragma unroll
    for (int t = 0; t < TPL; ++t) acc[t] = fmaf(x[t].y, w.y, acc[t]);
#pragma unroll
    for (int t = 0; t < TPL; ++t) acc[t] = fmaf(x[t].z, w.z, acc[t]);
#pragma unroll
    for (int t = 0; t < TPL; ++t) acc[t] = fmaf(x[t].w, w.w, acc[t]);
  };
#pragma unroll 1
  for (int step = 0; step < steps; ++step) {
    cp_async_wait<STAGES - 2>();
    __syncwarp();                               // this piece is everybody's; the piece before it has been read by all
    const int next = step + STAGES - 1;
    if (next < steps) {
      load_w(next);
      float* dst = ring + (next % STAGES) * STAGE + 16 * LD;
      for (int c = lane; c < M * CHUNKS; c += 32) {
        const int r = c / CHUNKS, k = (c % CHUNKS) * 4;
        if (next * KT + k < K) cp_async16(dst + r * LD + k, A + (long long)r * lda + next * KT + k);
      }
    }
    cp_async_commit();
    const float* wr = ring + (step % STAGES) * STAGE + row * LD;
    const float* xr = ring + (step % STAGES) * STAGE + (16 + g) * LD;
    const int left = K - step * KT;
    if (left >= KT) {
#pragma unroll
      for (int k = 0; k < KT; k += 4) four(wr, xr, k);
    } else {
      for (int k = 0; k < left; k += 4) four(wr, xr, k);
    }
  }
  const int n = n0 + row;
#pragma unroll
  for (int t = 0; t < TPL; ++t) {
    const int m = g + 2 * t;
    if (m >= M || n >= N) continue;
    const long long o = (long long)m * ldc + n;
    if constexpr (ACCUM) C[o] = to_f32<TOut>(C[o]) + acc[t];
    else C[o] = from_f32<TOut>(acc[t]);
  }
}

// Prompts of the 32-bit path, bound by the FFMA rate (128 a clock and SM).  A thread owns TM x TN outputs whose rows and
// columns lie RG and CG apart, so that a warp's 16-byte reads (four k at once) touch 4 and 8 neighbouring rows of the
// tiles, KT + 4 floats apart: no bank is hit twice, and 8 reads feed 64 FFMA.  Tiles come in by 16-byte asynchronous
// copies STAGES - 1 blocks ahead.  M tiles run fastest over the grid, so that a W tile is read from L2 by its row tiles.
// The four products of a 1B layer at 278 tokens: 1,220 us.
template <int BM_, int BN_, int TM_, int TN_, typename TOut, bool ACCUM>
__global__ void __launch_bounds__((BM_ / TM_) * (BN_ / TN_))
gemm_tiles_kernel(const float* __restrict__ A, long long lda, const float* __restrict__ W, long long ldw,
                  TOut* __restrict__ C, long long ldc, int M, int N, int K, int m_tiles) {
  constexpr int KT = 32, STAGES = 3, LD = KT + 4, CHUNKS = KT / 4, RG = BM_ / TM_, CG = BN_ / TN_, NT = RG * CG;
  constexpr int STAGE = (BM_ + BN_) * LD;
  static_assert(RG % 4 == 0 && CG % 8 == 0 && (BM_ * CHUNKS) % NT == 0 && (BN_ * CHUNKS) % NT == 0, "tile");
  extern __shared__ __align__(16) float ring[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tr = (warp / (CG / 8)) * 4 + (lane >> 3), tc = (warp % (CG / 8)) * 8 + (lane & 7);
  const int m0 = (blockIdx.x % m_tiles) * BM_, n0 = (blockIdx.x / m_tiles) * BN_;
  const int steps = (K + KT - 1) / KT;
  auto load_rows = [&](const float* src, long long ld, int first, int rows, int step, float* dst, auto count) {
#pragma unroll
    for (int i = 0; i < decltype(count)::value * CHUNKS / NT; ++i) {
      const int c = tid + NT * i, r = c / CHUNKS, k = (c % CHUNKS) * 4;
      if (step * KT + k < K) cp_async16(dst + r * LD + k, src + (long long)min(first + r, rows - 1) * ld + step * KT + k);
    }
  };
  auto load_w = [&](int s) { load_rows(W, ldw, n0, N, s, ring + (s % STAGES) * STAGE + BM_ * LD, std::integral_constant<int, BN_>{}); };
  auto load_a = [&](int s) { load_rows(A, lda, m0, M, s, ring + (s % STAGES) * STAGE, std::integral_constant<int, BM_>{}); };
  for (int s = 0; s < min(STAGES - 1, steps); ++s) load_w(s);
  pdl_wait();
  pdl_launch_dependents();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < steps) load_a(s);
    cp_async_commit();
  }
  float acc[TM_][TN_];
#pragma unroll
  for (int i = 0; i < TM_; ++i)
#pragma unroll
    for (int j = 0; j < TN_; ++j) acc[i][j] = 0.f;
#pragma unroll 1
  for (int step = 0; step < steps; ++step) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    if (step + STAGES - 1 < steps) {
      load_w(step + STAGES - 1);
      load_a(step + STAGES - 1);
    }
    cp_async_commit();
    const float* as = ring + (step % STAGES) * STAGE + tr * LD;
    const float* ws = ring + (step % STAGES) * STAGE + (BM_ + tc) * LD;
    const int count = min(KT, K - step * KT);
#pragma unroll 2
    for (int k = 0; k < count; k += 4) {
      float4 a[TM_], b[TN_];
#pragma unroll
      for (int i = 0; i < TM_; ++i) a[i] = *(const float4*)(as + i * RG * LD + k);
#pragma unroll
      for (int j = 0; j < TN_; ++j) b[j] = *(const float4*)(ws + j * CG * LD + k);
#pragma unroll
      for (int i = 0; i < TM_; ++i)
#pragma unroll
        for (int j = 0; j < TN_; ++j) acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM_; ++i)
#pragma unroll
        for (int j = 0; j < TN_; ++j) acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM_; ++i)
#pragma unroll
        for (int j = 0; j < TN_; ++j) acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM_; ++i)
#pragma unroll
        for (int j = 0; j < TN_; ++j) acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < TM_; ++i) {
    const int m = m0 + tr + i * RG;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN_; ++j) {
      const int n = n0 + tc + j * CG;
      if (n >= N) continue;
      const long long o = (long long)m * ldc + n;
      if constexpr (ACCUM) C[o] = to_f32<TOut>(C[o]) + acc[i][j];
      else C[o] = from_f32<TOut>(acc[i][j]);
    }
  }
}

constexpr int ROWS_MAX_M = 16;

template <int TPL, int KT, int STAGES, typename TOut, bool ACCUM>
int launch_rows(const float* A, long long lda, const float* W, long long ldw, TOut* C, long long ldc, int M, int N, int K,
                cudaStream_t stream) {
  constexpr int smem = STAGES * (16 + 2 * TPL) * (KT + 4) * 4;
  static_assert(smem <= 48 * 1024, "the ring fits without an opt-in");
  hfee_launch(gemm_rows_kernel<TPL, KT, STAGES, TOut, ACCUM>, dim3((N + 15) / 16), dim3(32), smem, stream, A, lda, W, ldw, C, ldc,
              M, N, K);
  return hfee_check_launch("gemm_simt rows");
}

template <int BM_, int BN_, int TM_, int TN_, typename TOut, bool ACCUM>
int launch_tiles(const float* A, long long lda, const float* W, long long ldw, TOut* C, long long ldc, int M, int N, int K,
                 cudaStream_t stream) {
  constexpr int smem = 3 * (BM_ + BN_) * 36 * 4;
  static const cudaError_t opted = cudaFuncSetAttribute(gemm_tiles_kernel<BM_, BN_, TM_, TN_, TOut, ACCUM>,
                                                        cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (opted != cudaSuccess) return hfee_fail(HFEE_ERR_CUDA, "gemm_simt: no shared memory for its tiles");
  const int m_tiles = (M + BM_ - 1) / BM_;
  const long long tiles = (long long)m_tiles * ((N + BN_ - 1) / BN_);
  HFEE_REQUIRE(tiles <= 0x7fffffff, "gemm_simt: M=%d N=%d are too large", M, N);
  hfee_launch(gemm_tiles_kernel<BM_, BN_, TM_, TN_, TOut, ACCUM>, dim3((unsigned)tiles), dim3((BM_ / TM_) * (BN_ / TN_)), smem, stream,
              A, lda, W, ldw, C, ldc, M, N, K, m_tiles);
  return hfee_check_launch("gemm_simt tiles");
}

template <typename TOut, bool ACCUM>
int launch_f32(const float* A, long long lda, const float* W, long long ldw, TOut* C, long long ldc, int M, int N, int K,
               cudaStream_t stream) {
  // Up to ROWS_MAX_M tokens the bytes of W bound the product; TPL tokens a lane cost TPL FFMA per weight.
  if (M <= 2) return launch_rows<1, 64, 8, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  if (M <= 4) return launch_rows<2, 64, 8, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  if (M <= 8) return launch_rows<4, 64, 7, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  if (M <= ROWS_MAX_M) return launch_rows<8, 32, 8, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  // The tile that needs the least time: rounds over the SMs x outputs x what an output costs with that tile (more reads of
  // shared memory per FFMA in the smaller ones).
  const int sms = hfee_sm_count() > 0 ? hfee_sm_count() : 1;
  auto cost = [&](int bm, int bn, double each) {
    const long long tiles = (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn);
    return (double)((tiles + sms - 1) / sms) * bm * bn * each;
  };
  const double small = cost(32, 64, 1.25), middle = cost(64, 128, 1.08), large = cost(128, 128, 1.0);
  if (small <= middle && small <= large) return launch_tiles<32, 64, 4, 4, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  if (middle <= large) return launch_tiles<64, 128, 8, 4, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
  return launch_tiles<128, 128, 8, 8, TOut, ACCUM>(A, lda, W, ldw, C, ldc, M, N, K, stream);
}

template <typename TIn>
int launch(const void* A, long long lda, const void* W, long long ldw, void* C, long long ldc, int out_dtype,
           int accumulate, int M, int N, int K, cudaStream_t stream) {
  if constexpr (sizeof(TIn) == 4) {
    const bool aligned = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
    if (aligned && out_dtype == HFEE_F32)
      return accumulate ? launch_f32<float, true>((const float*)A, lda, (const float*)W, ldw, (float*)C, ldc, M, N, K, stream)
                        : launch_f32<float, false>((const float*)A, lda, (const float*)W, ldw, (float*)C, ldc, M, N, K, stream);
    if (aligned && out_dtype == HFEE_BF16 && !accumulate)
      return launch_f32<__nv_bfloat16, false>((const float*)A, lda, (const float*)W, ldw, (__nv_bfloat16*)C, ldc, M, N, K, stream);
  }
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (out_dtype == HFEE_F32) {
    if (accumulate)
      hfee_launch(gemm_simt_kernel<TIn, float, true>, dim3(grid), dim3(THREADS), 0, stream, (const TIn*)A, lda, (const TIn*)W, ldw, (float*)C, ldc, M, N, K);
    else
      hfee_launch(gemm_simt_kernel<TIn, float, false>, dim3(grid), dim3(THREADS), 0, stream, (const TIn*)A, lda, (const TIn*)W, ldw, (float*)C, ldc, M, N, K);
  } else if (out_dtype == HFEE_BF16) {
    if (accumulate) return hfee_fail(HFEE_ERR_ARG, "gemm_simt: accumulate needs a float32 output");
    hfee_launch(gemm_simt_kernel<TIn, __nv_bfloat16, false>, dim3(grid), dim3(THREADS), 0, stream, (const TIn*)A, lda, (const TIn*)W, ldw, (__nv_bfloat16*)C, ldc, M, N, K);
  } else {
    return hfee_fail(HFEE_ERR_ARG, "gemm_simt: unknown output dtype %d", out_dtype);
  }
  return hfee_check_launch("gemm_simt");
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
