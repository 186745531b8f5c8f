// Shared device/host helpers for the ReDrafter B200 kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/redrafter_b200.h"

#define RD_LOG_0 (-50000.0f)

// Launch-time check: returns a negative code for an invalid argument found on the host.
#define RD_REQUIRE(cond, code) \
  do {                         \
    if (!(cond)) return (code); \
  } while (0)

// Returns RD_ERR_LAUNCH when the launch itself was rejected (bad configuration).
#define RD_CHECK_LAUNCH()                                   \
  do {                                                      \
    cudaError_t e__ = cudaPeekAtLastError();                \
    if (e__ != cudaSuccess) {                               \
      rd_set_last_cuda_error((int)e__);                     \
      return RD_ERR_LAUNCH;                                 \
    }                                                       \
  } while (0)

// The same for a cudaError_t already in hand (rd::launch_chained() returns one).
#define RD_CHECK_CHAINED(err)                               \
  do {                                                      \
    if ((err) != cudaSuccess) {                             \
      rd_set_last_cuda_error((int)(err));                   \
      return RD_ERR_LAUNCH;                                 \
    }                                                       \
  } while (0)

void rd_set_last_cuda_error(int e);
// 1 unless the environment variable RD_PDL is "0" (read once): launch the kernels of the decode
// chain with programmatic stream serialisation so that a kernel's launch and prologue overlap the
// tail of its predecessor.
int rd_pdl_enabled();
// CTA pairs that the tcgen05 GEMM launches at most; 0 when it runs without pairs.
int rd_gemm_pairs();

namespace rd {

template <typename T>
struct Num;
template <>
struct Num<float> {
  static __device__ __forceinline__ float to_f(float v) { return v; }
  static __device__ __forceinline__ float from_f(float v) { return v; }
};
template <>
struct Num<__nv_bfloat16> {
  static __device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 from_f(float v) { return __float2bfloat16_rn(v); }
};

// fast form for rounded (bf16) outputs: approximate exp and division, ~2 ulp
__device__ __forceinline__ float silu_f(float x) { return __fdividef(x, 1.0f + __expf(-x)); }
// expf with full fp32 accuracy (used where parity with a CPU fp32 path matters)
__device__ __forceinline__ float silu_exact(float x) { return x / (1.0f + expf(-x)); }

// xIELU: pos z^2 + z/2 above zero, neg (e^z - 1 - z) + z/2 elsewhere.  Each part vanishes on the other's side, so neither
// needs a branch.
__device__ __forceinline__ float xielu_exact(float z, float pos, float neg) {
  const float p = fmaxf(z, 0.f), m = fminf(z, 0.f);
  return fmaf(pos * p, p, neg * (expm1f(m) - m)) + 0.5f * z;
}
// form for rounded (bf16) outputs: e^z - 1 carries an absolute error of about 1e-7 near zero
__device__ __forceinline__ float xielu_f(float z, float pos, float neg) {
  const float p = fmaxf(z, 0.f), m = fminf(z, 0.f);
  return fmaf(pos * p, p, fmaf(neg, __expf(m) - 1.0f - m, 0.5f * z));
}

// Gated unit with cut inputs: g sigmoid(alpha g) (u + 1), g = min(gate, limit), u = up cut to [-limit, limit].
__device__ __forceinline__ float clamped_glu_exact(float gate, float up, float limit, float alpha) {
  const float g = fminf(gate, limit), u = fminf(fmaxf(up, -limit), limit);
  return g / (1.0f + expf(-alpha * g)) * (u + 1.0f);
}
// form for rounded (bf16) outputs
__device__ __forceinline__ float clamped_glu_f(float gate, float up, float limit, float alpha) {
  const float g = fminf(gate, limit), u = fminf(fmaxf(up, -limit), limit);
  return __fdividef(g, 1.0f + __expf(-alpha * g)) * (u + 1.0f);
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ int warp_sum_i(int v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Order-preserving map float -> uint32 (larger float <=> larger key).
__device__ __forceinline__ uint32_t float_key(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Effective row count: min(*m_dev, m_max) when a device-side count is given.
__device__ __forceinline__ int live_rows(const int* m_dev, int m_max) {
  if (m_dev == nullptr) return m_max;
  int m = *m_dev;
  return m < m_max ? (m < 0 ? 0 : m) : m_max;
}

// Into how many shares K of a projection with a residual is cut when few rows are live (RD_EPI_RES; 1 = never).  Up to
// kShareRows rows are one token chunk, and the weights' tiles of 256 rows alone occupy few CTA pairs (16 of 74 for 4096
// features); the shares fill one wave, each of at least 8 k-blocks of 64.  With more rows the token chunks fill the wave, and
// writing and reading the shares costs what the idle pairs would gain.  Launches for more than kShareCapacity rows hardly ever run
// with so few (a packed draft keeps about 2 rows in 5) and are left as they are: their norm would pay for the question.
// Projection and norm together, bf16, one B200: 4096 x 11008 weights, 1 row 42 -> 24 us, some 110 rows 44 -> 27 us; 4096 x 4096,
// 1 row 22 -> 15 us, some 110 rows 23 -> 19 us.
constexpr int kShareRows = 256;
constexpr int kShareCapacity = 1024;
constexpr int kMaxShares = 8;
inline int share_count(int m_max, int N, int K, int pairs) {
  if (m_max > kShareCapacity || N < 256) return 1;
  int s = pairs / ((N + 255) / 256);
  const int by_length = (K + 63) / 64 / 8;
  s = s < by_length ? s : by_length;
  s = s < kMaxShares ? s : kMaxShares;
  return s > 1 ? s : 1;
}
// The shares of such a projection: partial products [shares][rows][N] in fp32, rows = min(m_max, kShareRows), and what they are
// added to.
template <typename T>
struct Shares {
  const float* parts;
  const T* residual;  // [m, N]
  int count, rows;    // count 1: the projection's output is complete
};
// the projection and the norm after it come to the same answer from the live rows
__device__ __forceinline__ int live_shares(int count, int M) { return M <= kShareRows ? count : 1; }
// residual + sum of the shares of features [d, d + VEC) of row t, the shares in ascending order of K
template <int VEC, typename T>
__device__ __forceinline__ void add_shares(const Shares<T>& sh, int t, int N, int d, float* f) {
  static_assert(VEC == 1 || VEC * sizeof(T) == 16, "vector width");
  const float* p = sh.parts + (int64_t)t * N + d;
  float acc[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) acc[i] = 0.f;
#pragma unroll 4
  for (int s = 0; s < sh.count; ++s, p += (int64_t)sh.rows * N) {
    if constexpr (VEC == 1) {
      acc[0] += *p;
    } else {
#pragma unroll
      for (int i = 0; i < VEC; i += 4) {
        const float4 q = *reinterpret_cast<const float4*>(p + i);
        acc[i] += q.x, acc[i + 1] += q.y, acc[i + 2] += q.z, acc[i + 3] += q.w;
      }
    }
  }
  T r[VEC];
  if constexpr (VEC == 1)
    r[0] = sh.residual[(int64_t)t * N + d];
  else
    *reinterpret_cast<uint4*>(r) = *reinterpret_cast<const uint4*>(sh.residual + (int64_t)t * N + d);
#pragma unroll
  for (int i = 0; i < VEC; ++i) f[i] = acc[i] + Num<T>::to_f(r[i]);
}

// Programmatic dependent launch.  A kernel launched with rd::launch_chained() may begin before the
// previous kernel of the stream has finished: it must execute pdl_wait() before its first access to
// global memory (reads of the predecessor's results and writes to anything the predecessor may still
// read), and it lets its own successor start early with pdl_launch_dependents().  Both are no-ops
// in a kernel that was launched the ordinary way.  Data of an earlier kernel must not be read through a const
// __restrict__ pointer in straight-line code after the wait: the compiler may treat such loads as invariant and
// hoist them above it (a commit kernel read the previous step's acceptance that way once its launch overlapped).
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// True in one lane of a converged warp, the same one each time.  Code that issues tcgen05 instructions or bulk copies belongs under
// this and not under `lane == 0`: their operands live in uniform registers, and only here does the compiler know that a
// single thread runs.  Under `lane == 0` an MMA of the GEMM cost its issuer some 60 cycles and a k-block of 64 at
// least 0.29 us, however few its tokens; elected, 0.2 us (4096 x 11008 weights, 1 token: 56.7 -> 40.5 us; 22016 x 4096
// weights, 1000 tokens: 131 -> 125 us).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
  return p != 0;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_chained(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, int cluster_x,
                                  Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (cluster_x > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster_x;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (rd_pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

}  // namespace rd
