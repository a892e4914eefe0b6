// Shared device/host helpers for the SSD kernels (sm_100a only).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <utility>

#include "../../include/ssd_b200.h"

// floats per (batch, chunk, head) decay table written by the cumsum kernel for the tensor-core
// family: [cs*log2e | dt | column factors | per-step decays], 128 each
#define SSD_TAB_FLOATS 512

namespace ssd {

// Internal, fully-resolved geometry handed to every kernel by value.
struct Geo {
  int B, L, H, P, N, G, Q, nc, hpg;  // hpg = heads per group
  long long xsb, xsl, dtsb, dtsl, bsb, bsl, csb, csl, zsb, zsl, ysb, ysl;
  int dt_softplus;                     // step size = softplus(dt + dt_bias) instead of dt + dt_bias
  int any_y;                           // y / dy need not suit TMA: the caller takes care of them (see Plan in ssd_api.cu)
  int onetile;                         // tensor family: the one-tile-per-CTA kernels for every shape (SSD_ALGO_TENSOR_ONETILE)
  int hsplit = 1;                      // scan kernels: G and hpg describe parts of a group, `hsplit` to the group (see split_heads)
};

// The step-size pre-activation of a Mamba-2 layer, fused where dt is first read.  Above 20 softplus is the
// identity in fp32 (same cut-off as torch.nn.functional.softplus).
__device__ __forceinline__ float dt_activation(float raw, float bias, int softplus) {
  const float v = raw + bias;
  return (softplus && v <= 20.f) ? log1pf(expf(v)) : v;
}

// Workspace segments (offsets in bytes from the workspace base; 0-size segments unused).
struct WsLayout {
  size_t status;                                     // 256-byte status block (int32 code first)
  size_t cs, dtf, states, fin, cb;                   // forward
  size_t tab, prev_bf, hand;                         // forward, tensor-core family only (else empty)
  size_t ds_bf;                                      // backward, tensor-core family only
  size_t dstates, wsum, dyp, dcsp, ddtd, ddot, sdot, dapart, ddpart, dbpart, dini;  // backward extras (wsum: CUDA-core family only)
  size_t total_fwd, total_bwd;
};

// 16-byte asynchronous copies global -> shared, tracked per thread in groups (commit, then wait until at most N groups
// are outstanding).  With `valid` false nothing is read and the 16 bytes are written as zeros.
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(gsrc), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <typename T> __device__ __forceinline__ float ldf(const T* p);
template <> __device__ __forceinline__ float ldf<float>(const float* p) { return __ldg(p); }
template <> __device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(*p);
}
template <typename T> __device__ __forceinline__ void stf(T* p, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, float v) {
  *p = __float2bfloat16_rn(v);
}

// Packed pairs of fp32 (one 64-bit register): sm_100 executes fma / add on both halves in one instruction, with the same
// rounding as the scalar forms.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// The sums of R values over groups of LPR lanes, R values at a time: every exchange folds two values into one, so a tile row
// set costs R - 1 + log2(LPR / R) shuffles instead of R log2(LPR).  Lane `lir` ends up with the sum of value `u` (returned);
// all lanes whose lir agrees in its log2(R) top bits hold the same one.
template <int LPR, int R>
__device__ __forceinline__ float fold_rows(float (&v)[R], int lir, int& u) {
  u = 0;
  int o = LPR / 2;
#pragma unroll
  for (int n = R; n > 1; n >>= 1, o >>= 1) {
    const bool up = lir & o;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const float keep = up ? v[n / 2 + i] : v[i], give = up ? v[i] : v[n / 2 + i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
    u += up ? n / 2 : 0;
  }
  float t = v[0];
#pragma unroll
  for (; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

__device__ __forceinline__ float sigmoidf_(float z) { return 1.f / (1.f + __expf(-z)); }

// Thread-local error string shared by every translation unit of the library.
void set_error(const char* fmt, ...);
void clear_error();

// Bookkeeping after every kernel launch: counts it and, while a profile is open on this thread,
// records an event behind it on the launch stream.
void after_launch(const char* what, cudaStream_t s);

// Programmatic dependent launch.  Every kernel of the library that launch() starts may be scheduled as soon as the blocks of
// the one in front of it have ended and touches no global memory before that one's writes are visible (pdl_wait), so launch
// latency, barrier set-up and tensor-memory allocation run beside the predecessor's completion and flush: 5-8 us less on a
// backward of four short kernels (batch 4 x 1024 policy step 109 -> 94 us, mixer 64x1024 433 -> 393 us).  No kernel triggers
// its successor early: blocks that only wait take the places that free up first, and the successor then runs unevenly spread
// over the SMs (fp32 16x1000 step 914 us without the attribute, 949 with an early trigger, 881 like this).  All threads call
// pdl_wait: completion of a kernel then implies completion of all before it.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launch with that attribute; a large dynamic shared memory is asked for when a kernel first needs as much on a device.
template <auto Kernel, class... A>
static inline cudaError_t launch(dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  if (smem > 32 * 1024) {   // 48 KB without asking, static shared memory included
    static std::atomic<int> allowed[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev > 63 || allowed[dev].load(std::memory_order_relaxed) < (int)smem) {
      const cudaError_t e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      if (dev <= 63) allowed[dev].store((int)smem, std::memory_order_relaxed);
    }
  }
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, Kernel, std::forward<A>(args)...);
}

// SMs of the current device.
int sm_count();

// Uses the cudaStream_t named `s` in the enclosing scope.
#define SSD_CUDA_CHECK_LAUNCH(what)                                              \
  do {                                                                           \
    cudaError_t e__ = cudaGetLastError();                                        \
    if (e__ != cudaSuccess) {                                                    \
      ::ssd::set_error("%s: launch failed: %s", what, cudaGetErrorString(e__));  \
      return SSD_ERR_CUDA;                                                       \
    }                                                                            \
    ::ssd::after_launch(what, s);                                                \
  } while (0)

static inline int cdiv(int a, int b) { return (a + b - 1) / b; }

}  // namespace ssd
