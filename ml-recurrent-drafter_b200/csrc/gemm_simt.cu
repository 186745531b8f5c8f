// C = epilogue(A * W^T) on CUDA cores with fp32 accumulation, for fp32 models (exact-fp32 parity
// with a CPU run is only possible without tensor cores) and as the cross-check of the tcgen05
// path.  Two kernels with 256 threads: 64x64 tiles, and 32x32 tiles where launch() finds them to finish first.  Both add
// an output's products in ascending order of K, so they give the same bits.
#include "rd_common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16;

template <typename OutT>
__device__ __forceinline__ void store_out(OutT* p, float v);
template <>
__device__ __forceinline__ void store_out<float>(float* p, float v) {
  *p = v;
}
template <>
__device__ __forceinline__ void store_out<__nv_bfloat16>(__nv_bfloat16* p, float v) {
  *p = __float2bfloat16_rn(v);
}

// The element-wise part for W consecutive output features of a token (W even), and the store.
template <int W, typename T, typename OutT, int EPI>
__device__ __forceinline__ void finish(const float* acc, int m, int n, int N, OutT* C, int64_t ldc, const T* bias, const OutT* R,
                                        int64_t ldr, float act0, float act1) {
  if (EPI == RD_EPI_SWIGLU || EPI == RD_EPI_CLAMPED_GLU) {
#pragma unroll
    for (int j = 0; j < W; j += 2)
      if (n + j + 1 < N)
        store_out<OutT>(C + (int64_t)m * ldc + ((n + j) >> 1), EPI == RD_EPI_SWIGLU ? rd::silu_exact(acc[j]) * acc[j + 1]
                                                                                   : rd::clamped_glu_exact(acc[j], acc[j + 1], act0, act1));
    return;
  }
#pragma unroll
  for (int j = 0; j < W; ++j) {
    if (n + j >= N) continue;
    float v = acc[j];
    if (EPI == RD_EPI_BIAS || EPI == RD_EPI_BIAS_SILU || EPI == RD_EPI_BIAS_SILU_RES) v += rd::Num<T>::to_f(bias[n + j]);
    if (EPI == RD_EPI_BIAS_SILU || EPI == RD_EPI_BIAS_SILU_RES) v = rd::silu_exact(v);
    if (EPI == RD_EPI_XIELU) v = rd::xielu_exact(v, act0, act1);
    if (EPI == RD_EPI_BIAS_SILU_RES || EPI == RD_EPI_RES) v += rd::Num<OutT>::to_f(R[(int64_t)m * ldr + n + j]);
    store_out<OutT>(C + (int64_t)m * ldc + n + j, v);
  }
}

template <typename T, typename OutT, int EPI>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const T* __restrict__ A, int64_t lda, const T* __restrict__ W,
                                                        int64_t ldw, OutT* C, int64_t ldc, const T* __restrict__ bias,
                                                        const OutT* R, int64_t ldr, int m_max,
                                                        const int32_t* __restrict__ m_dev, int N, int K, float act0,
                                                        float act1) {
  const int M = rd::live_rows(m_dev, m_max);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  if (m0 >= M) return;
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;  // 16 x 16 threads
  const int lr = tid >> 2, lk = (tid & 3) * 4;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int kk = k0 + lk + e;
      const int am = m0 + lr, wn = n0 + lr;
      As[lk + e][lr] = (am < M && kk < K) ? rd::Num<T>::to_f(A[(int64_t)am * lda + kk]) : 0.f;
      Ws[lk + e][lr] = (wn < N && kk < K) ? rd::Num<T>::to_f(W[(int64_t)wn * ldw + kk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
    finish<4, T, OutT, EPI>(acc[i], m, n0 + tx * 4, N, C, ldc, bias, R, ldr, act0, act1);
  }
}

// 4 consecutive elements of a row from k on, zeros outside [0, K) or for a row that does not exist
template <typename T>
__device__ __forceinline__ void load4(float* f, const T* row, bool exists, int k, int K, bool vec) {
  f[0] = f[1] = f[2] = f[3] = 0.f;
  if (!exists) return;
  if (vec && k + 4 <= K) {
    T e[4];
    if constexpr (sizeof(T) == 4)
      *reinterpret_cast<uint4*>(e) = *reinterpret_cast<const uint4*>(row + k);
    else
      *reinterpret_cast<uint2*>(e) = *reinterpret_cast<const uint2*>(row + k);
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = rd::Num<T>::to_f(e[i]);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (k + i < K) f[i] = rd::Num<T>::to_f(row[k + i]);
  }
}

// Few tokens or features: 32x32 tiles, 2x2 outputs per thread.  Such a launch is one chain of loads and barriers per step of K
// (16 steps of 16 at K = 256 took 16 us on 64x64 tiles), so a step takes 64 of K and the next step's operands are on their way
// meanwhile.  24 tokens, one B200: 256 x 256 weights 16 -> 7 us, 256 x 688 43 -> 18 us.
constexpr int SM = 32, SN = 32, SK = 64, kLd = 34;

template <typename T, typename OutT, int EPI>
__global__ void __launch_bounds__(256) gemm_simt_small_kernel(const T* A, int64_t lda, const T* W, int64_t ldw, OutT* C, int64_t ldc,
                                                              const T* bias, const OutT* R, int64_t ldr, int m_max,
                                                              const int32_t* m_dev, int N, int K, float act0, float act1, int vec_a,
                                                              int vec_w) {
  rd::pdl_launch_dependents();
  rd::pdl_wait();
  const int M = rd::live_rows(m_dev, m_max);
  const int m0 = blockIdx.y * SM, n0 = blockIdx.x * SN;
  if (m0 >= M) return;
  __shared__ __align__(16) float As[SK * kLd], Ws[SK * kLd];  // [k][row]
  const int tid = threadIdx.x;
  const int lr = tid & 31, lk = (tid >> 5) * 4;  // loads: a warp takes 4 of K of all 32 rows, then the 4 that lie 32 further on
  const int tx = tid & 15, ty = tid >> 4;
  const bool has_a = m0 + lr < M, has_w = n0 + lr < N;
  const T* arow = A + (int64_t)(has_a ? m0 + lr : 0) * lda;
  const T* wrow = W + (int64_t)(has_w ? n0 + lr : 0) * ldw;
  float a[2][4], w[2][4], acc[2][2] = {};
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    load4(a[i], arow, has_a, lk + 32 * i, K, vec_a != 0);
    load4(w[i], wrow, has_w, lk + 32 * i, K, vec_w != 0);
  }
  for (int k0 = 0; k0 < K; k0 += SK) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        As[(lk + 32 * i + e) * kLd + lr] = a[i][e];
        Ws[(lk + 32 * i + e) * kLd + lr] = w[i][e];
      }
    __syncthreads();
    if (k0 + SK < K) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        load4(a[i], arow, has_a, k0 + SK + lk + 32 * i, K, vec_a != 0);
        load4(w[i], wrow, has_w, k0 + SK + lk + 32 * i, K, vec_w != 0);
      }
    }
#pragma unroll 16
    for (int kk = 0; kk < SK; ++kk) {
      const float2 x = *reinterpret_cast<const float2*>(As + kk * kLd + ty * 2);
      const float2 y = *reinterpret_cast<const float2*>(Ws + kk * kLd + tx * 2);
      acc[0][0] = fmaf(x.x, y.x, acc[0][0]);
      acc[0][1] = fmaf(x.x, y.y, acc[0][1]);
      acc[1][0] = fmaf(x.y, y.x, acc[1][0]);
      acc[1][1] = fmaf(x.y, y.y, acc[1][1]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int m = m0 + ty * 2 + i;
    if (m < M) finish<2, T, OutT, EPI>(acc[i], m, n0 + tx * 2, N, C, ldc, bias, R, ldr, act0, act1);
  }
}

template <typename T, typename OutT>
int launch(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, const void* bias, const void* R,
           int64_t ldr, int m_max, const int32_t* m_dev, int N, int K, int epilogue, float act0, float act1, cudaStream_t s) {
  dim3 grid((N + BN - 1) / BN, (m_max + BM - 1) / BM);
  // Both kernels keep several blocks on an SM (48 registers, 256 threads: five), but what an SM's blocks take adds up: K = 2048, one
  // B200, us of a launch by itself with 1 / 2 / 3 / 4 small tiles per SM: 59 / 100 / 145 / 190, with 1 / 2 large ones 133 / 240 (123 / 223
  // where half of their rows are empty).  So small tiles as long as there are at most two of them for each large one that an SM would
  // have: 64 x 4736 100 and not 133, but 64 x 6144 133 and not 145, 512 x 2304 221 and not 371.  K = 256 and 688 lie the same way.
  // From two large tiles per SM on there are only these, although few rows would gain (20 x 18944: 223, small ones 180).
  constexpr int kSMs = 148;
  const auto per_sm = [](int64_t blocks) { return (blocks + kSMs - 1) / kSMs; };
  const dim3 small_grid((N + SN - 1) / SN, (m_max + SM - 1) / SM);
  const int64_t n_large = (int64_t)grid.x * grid.y, n_small = (int64_t)small_grid.x * small_grid.y;
  const bool small = n_large < 2 * kSMs && per_sm(n_small) <= 2 * per_sm(n_large);
  // Launched programmatically only while two such launches have an SM for each block: blocks that are placed beside those of the
  // launch before crowd on some SMs.  In a row, K = 2048: 64 blocks 53 us (ordinary launches 54), 128 blocks 107 (56), 288 blocks
  // 202 (97); K = 256: 64 blocks 8.1 (10.5), 256 blocks 25.5 (14.9).
  const bool chained = 2 * n_small <= kSMs;
  const auto row_vec = [](const void* p, int64_t ld) { return ((uintptr_t)p | (uintptr_t)(ld * sizeof(T))) % (4 * sizeof(T)) == 0; };
  const int vec_a = row_vec(A, lda), vec_w = row_vec(W, ldw);
#define RD_LAUNCH_EPI(E)                                                                                              \
  case E:                                                                                                             \
    if (small && chained) {                                                                                           \
      cudaError_t err = rd::launch_chained(gemm_simt_small_kernel<T, OutT, E>, small_grid, dim3(256), 0, s, 1, (const T*)A, lda, \
                                           (const T*)W, ldw, (OutT*)C, ldc, (const T*)bias, (const OutT*)R, ldr, m_max, m_dev, N, K, \
                                           act0, act1, vec_a, vec_w);                                                \
      RD_CHECK_CHAINED(err);                                                                                          \
    } else if (small) {                                                                                               \
      gemm_simt_small_kernel<T, OutT, E><<<small_grid, 256, 0, s>>>((const T*)A, lda, (const T*)W, ldw, (OutT*)C, ldc,  \
                                                                    (const T*)bias, (const OutT*)R, ldr, m_max, m_dev, N, K, act0, act1, \
                                                                    vec_a, vec_w);                                    \
    } else {                                                                                                          \
      gemm_simt_kernel<T, OutT, E><<<grid, 256, 0, s>>>((const T*)A, lda, (const T*)W, ldw, (OutT*)C, ldc, (const T*)bias, \
                                                        (const OutT*)R, ldr, m_max, m_dev, N, K, act0, act1);         \
    }                                                                                                                 \
    break;
  switch (epilogue) {
    RD_LAUNCH_EPI(RD_EPI_NONE)
    RD_LAUNCH_EPI(RD_EPI_BIAS)
    RD_LAUNCH_EPI(RD_EPI_BIAS_SILU)
    RD_LAUNCH_EPI(RD_EPI_BIAS_SILU_RES)
    RD_LAUNCH_EPI(RD_EPI_RES)
    RD_LAUNCH_EPI(RD_EPI_SWIGLU)
    RD_LAUNCH_EPI(RD_EPI_XIELU)
    RD_LAUNCH_EPI(RD_EPI_CLAMPED_GLU)
    default:
      return RD_ERR_ARG;
  }
#undef RD_LAUNCH_EPI
  RD_CHECK_LAUNCH();
  return RD_OK;
}

}  // namespace

static int gemm_checked(int dtype, int out_dtype, const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc,
                        const void* bias, const void* R, int64_t ldr, int m_max, const int32_t* m_dev, int N, int K,
                        int epilogue, float act0, float act1, void* stream) {
  RD_REQUIRE(A && W && C, RD_ERR_ARG);
  RD_REQUIRE(m_max >= 1 && N >= 1 && K >= 1 && lda >= K && ldw >= K, RD_ERR_SIZE);
  const bool need_bias = epilogue == RD_EPI_BIAS || epilogue == RD_EPI_BIAS_SILU || epilogue == RD_EPI_BIAS_SILU_RES;
  const bool need_res = epilogue == RD_EPI_BIAS_SILU_RES || epilogue == RD_EPI_RES;
  RD_REQUIRE(!need_bias || bias, RD_ERR_ARG);
  RD_REQUIRE(!need_res || R, RD_ERR_ARG);
  const bool glu = epilogue == RD_EPI_SWIGLU || epilogue == RD_EPI_CLAMPED_GLU;
  RD_REQUIRE(!glu || N % 2 == 0, RD_ERR_SIZE);
  RD_REQUIRE(ldc >= (glu ? N / 2 : N), RD_ERR_SIZE);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == RD_F32 && out_dtype == RD_F32)
    return launch<float, float>(A, lda, W, ldw, C, ldc, bias, R, ldr, m_max, m_dev, N, K, epilogue, act0, act1, s);
  if (dtype == RD_BF16 && out_dtype == RD_BF16)
    return launch<__nv_bfloat16, __nv_bfloat16>(A, lda, W, ldw, C, ldc, bias, R, ldr, m_max, m_dev, N, K, epilogue, act0, act1, s);
  if (dtype == RD_BF16 && out_dtype == RD_F32)
    return launch<__nv_bfloat16, float>(A, lda, W, ldw, C, ldc, bias, R, ldr, m_max, m_dev, N, K, epilogue, act0, act1, s);
  return RD_ERR_DTYPE;
}

extern "C" int rd_gemm(int dtype, int out_dtype, const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc,
                       const void* bias, const void* R, int64_t ldr, int m_max, const int32_t* m_dev, int N,
                       int K, int epilogue, void* stream) {
  // these have parameters: rd_gemm_xielu, rd_gemm_clamped_glu
  RD_REQUIRE(epilogue != RD_EPI_XIELU && epilogue != RD_EPI_CLAMPED_GLU, RD_ERR_ARG);
  return gemm_checked(dtype, out_dtype, A, lda, W, ldw, C, ldc, bias, R, ldr, m_max, m_dev, N, K, epilogue, 0.f, 0.f, stream);
}

extern "C" int rd_gemm_xielu(int dtype, const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, int m_max,
                             const int32_t* m_dev, int N, int K, float pos, float neg, void* stream) {
  return gemm_checked(dtype, dtype, A, lda, W, ldw, C, ldc, nullptr, nullptr, 0, m_max, m_dev, N, K, RD_EPI_XIELU, pos, neg,
                      stream);
}

extern "C" int rd_gemm_clamped_glu(int dtype, const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, int m_max,
                                   const int32_t* m_dev, int N, int K, float limit, float alpha, void* stream) {
  return gemm_checked(dtype, dtype, A, lda, W, ldw, C, ldc, nullptr, nullptr, 0, m_max, m_dev, N, K, RD_EPI_CLAMPED_GLU, limit, alpha,
                      stream);
}
