// Shared helpers for the mLSTM sm_100a kernels: element-type conversion, math, launch checks.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/mlstm_b200.h"

namespace mlstm {

// ---- element types ---------------------------------------------------------------------
__device__ __forceinline__ float to_f32(float x) { return x; }
__device__ __forceinline__ float to_f32(__nv_bfloat16 x) { return __bfloat162float(x); }
__device__ __forceinline__ float to_f32(__half x) { return __half2float(x); }

template <typename T> __device__ __forceinline__ T from_f32(float x);
template <> __device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ __half from_f32<__half>(float x) { return __float2half_rn(x); }

// ---- math ---------------------------------------------------------------------------------
// log(sigmoid(x)) without overflow, full-precision transcendental functions.
__device__ __forceinline__ float logsigmoid_f(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + expf(-x)); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ---- host side --------------------------------------------------------------------------
void set_last_cuda_error(cudaError_t e, const char* where);

#define MLSTM_CUDA_CHECK(expr)                         \
  do {                                                 \
    cudaError_t _e = (expr);                           \
    if (_e != cudaSuccess) {                           \
      ::mlstm::set_last_cuda_error(_e, #expr);         \
      return MLSTM_ERR_CUDA;                           \
    }                                                  \
  } while (0)

// SMs of the current device (of a B200 where there is none: sizes are asked for on hosts without a GPU too)
constexpr int kB200Sms = 148;
int sm_count();

// every kernel launch of this library is counted (mlstm_b200_launch_count)
void note_launch();
#define MLSTM_LAUNCH_CHECK()                  \
  do {                                        \
    ::mlstm::note_launch();                   \
    MLSTM_CUDA_CHECK(cudaGetLastError());     \
  } while (0)

// Programmatic dependent launch: a kernel launched with launch_pdl may be scheduled once every CTA of the kernel before it
// in the stream has called pdl_launch_dependents() (or has ended), so that its launch latency and set-up overlap that
// kernel's tail; pdl_wait() then blocks until that kernel has completed and its writes are visible.  Every thread block
// calls pdl_wait() before it touches global memory.  What such a kernel reads may be written while it is already resident,
// so it takes its inputs as plain pointers (const __restrict__ lets the compiler read through the non-coherent path, which is
// for memory that nothing writes during the whole kernel) and streams through ld_stream, which stays behind pdl_wait().  Saves 1-2 us per launch boundary, which is what small calls are
// made of (a decode step of one sequence, back to back: 6.1 -> 3.7 us; the forward of 500 tokens 31.0 -> 28.5 us); overlap = false is a plain launch.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// evict-first loads of data that is read once
__device__ __forceinline__ uint4 ld_stream(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.cs.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_stream(const float4* p) {
  float4 v;
  asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint2 ld_stream(const uint2* p) {
  uint2 v;
  asm volatile("ld.global.cs.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}

// Larger launches start plainly: their own CTAs hide the gap, and CTAs of the next kernel that are resident early would take
// room on an SM from those of a second chain of launches.
inline unsigned pdl_max_ctas() { return 4u * (unsigned)sm_count(); }

// started (nullable): recorded once every CTA of the launch is running.
template <typename... KArgs, typename... Args>
int launch_ex(bool overlap, cudaEvent_t started, void (*kern)(KArgs...), unsigned grid, unsigned threads, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2] = {};
  if (overlap) {
    at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (started != nullptr) {
    at[cfg.numAttrs].id = cudaLaunchAttributeLaunchCompletionEvent;
    at[cfg.numAttrs++].val.launchCompletionEvent.event = started;
  }
  cfg.attrs = at;
  note_launch();
  MLSTM_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, KArgs(args)...));
  return MLSTM_OK;
}

template <typename... KArgs, typename... Args>
int launch_pdl(bool overlap, void (*kern)(KArgs...), unsigned grid, unsigned threads, size_t smem, cudaStream_t st, Args... args) {
  return launch_ex(overlap, nullptr, kern, grid, threads, smem, st, args...);
}

// Optional per-phase device timing (mlstm_b200_profile_*): when enabled, a pair of CUDA events
// brackets each phase on the launching stream.
enum Phase { PH_GATES = 0, PH_REC_FW, PH_PAR_FW, PH_REC_BW, PH_PAR_BW, PH_GATE_GRADS, PH_STEP, PH_COUNT };
struct PhaseScope {
  PhaseScope(int phase, cudaStream_t st);
  ~PhaseScope();
  int slot;
  cudaStream_t st;
  bool nvtx;
};

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }
inline bool is_pow2(int x) { return x > 0 && (x & (x - 1)) == 0; }
inline size_t dtype_size(int dtype) { return dtype == MLSTM_F32 ? 4 : 2; }

// Problem description passed to every launcher.
// The last chunk may be ragged (S not a multiple of L; tcgen05 path only): NC = ceil(S / L) and the library's own
// per-token vectors are laid out with SP = NC * L slots per (batch, head), the slots past S holding neutral values
// (input gate switched off, nothing decays), so that the contraction kernels need no per-token bounds checks on
// them.  User-visible per-token arrays (i, f, n_out, m_out, dI, dF) keep S entries per (batch, head).
struct ChunkwiseDims {
  int B, NH, S, DHQK, DHHV, L, NC;
  int variant;  // MLSTM_EXP / MLSTM_SIG / MLSTM_SIG_NONORM
  float eps;
  float qk_scale;
  int SP;       // NC * L
  int dtype;    // element type of q, k, v, h and the gradients (MLSTM_F32 / MLSTM_BF16 / MLSTM_F16)
};
inline ChunkwiseDims make_dims(int B, int NH, int S, int DHQK, int DHHV, int L, int variant, float eps, int dtype) {
  const int NC = (S + L - 1) / L;
  return ChunkwiseDims{B, NH, S, DHQK, DHHV, L, NC, variant, eps, 1.0f / sqrtf((float)DHQK), NC * L, dtype};
}

// Per-token / per-chunk gate vectors produced by the gate pre-pass (all f32, device memory).
// Per-token arrays have SP slots per (batch, head) (see ChunkwiseDims).
struct GateBuffers {
  float* vecB;     // (BNH, S)  in-chunk inclusive cumsum of logsigmoid(f)
  float* iota;     // (BNH, S)  i, or logsigmoid(i) for the sigmoid input gate
  float* m_tok;    // (BNH, S)  combined max state per token (0 for the sigmoid gate)
  float* abar;     // (BNH, S)  exp(a_j - m_{k+1})
  float* bbar;     // (BNH, S)  exp(b_i + m_k - m_i)
  float* gbar;     // (BNH, NC) exp(g_k + m_k - m_{k+1})
  float* inv_den;  // (BNH, S)  backward only: 1 / (n_out + eps) (1 when there is no normaliser)
  float* scratch;  // (BNH, 2*NC) per-chunk g and max_j a_j
};

}  // namespace mlstm
