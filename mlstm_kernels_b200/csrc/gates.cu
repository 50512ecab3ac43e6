// Gate pre-pass and gate-gradient kernels (scalar work per token; HBM traffic is negligible).
//
// Pre-pass: from the raw gate logits i, f produce every per-token and per-chunk scalar the
// contraction kernels need, including the serial max-state recursion over chunks, which is
// evaluated as a block-wide scan over (max,+) affine maps.
// Follows mlstm_kernels/torch/chunkwise/triton_xl_chunk/chunkwise_gates.py:15-65 (vecB, vecA),
// mlstm_kernels/triton/chunkwise/xl_chunk/fw_kernel_recurrent.py:150-176 (m recursion) and
// mlstm_kernels/torch/chunkwise/native/fw.py:178-195 (per-token max state).
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "launch.cuh"

namespace mlstm {

// One launch for the whole pre-pass: a cluster of up to eight CTAs per (batch, head), the chunks of a sequence split
// contiguously over its CTAs, one warp per chunk at a time.
//   1. per chunk:   b_j (inclusive sums of log f), a_j = sum_{t>j} log f_t + iota_j, g_k, max_j a_j
//   2. per cluster: m_{k+1} = max(g_k + m_k, amax_k) as a scan over the maps x -> max(x + G, A): threads compose their
//                   chunks, warps scan by shuffles, CTAs exchange their totals through distributed shared memory
//   3. per chunk:   m_i, abar_j, bbar_i, 1/(den+eps)
// The work is a few loads and transcendentals per token: launch and dependency latency are all there is to save.  As
// three launches with a serial 256-step combine in the middle it took 15.2 us (8 heads x 4 chunks), 26 us
// (128 heads x 64 chunks) and 27.6 us (8 heads x 1024 chunks).
struct GateScan {
  const float* m_initial;
  float m_default;       // max state before the first chunk where m_initial is null
  float* m_states;       // (BNH, NC+1)
  float* m_last;         // (BNH) or null: copy of the last one
  float* g_sum;          // (BNH) or null: total log forget gate of the sequence (for chaining segments)
};

// NV: register-held token values per lane, NV * 32 >= L
template <typename T, int NV>
__global__ void __launch_bounds__(1024)
gates_kernel(const T* vecI, const T* vecF, const float* n_out, float* __restrict__ m_out, GateBuffers gb, GateScan sc, int S, int SP, int L, int NC, int variant, float eps) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ float s_wG[32], s_wA[32];    // totals of the warps
  __shared__ float s_total[2];            // total of the CTA, read by the rest of the cluster
  const int ncta = cluster.num_blocks(), rank = cluster.block_rank(), bh = blockIdx.x / ncta;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
  const int per = (NC + ncta - 1) / ncta, c0 = min(NC, rank * per), c1 = min(NC, c0 + per);   // chunks of this CTA
  const bool siging = variant != MLSTM_EXP;
  pdl_launch_dependents();
  pdl_wait();
  float* g_arr = gb.scratch + (size_t)bh * 2 * NC;
  float* amax_arr = g_arr + NC;
  // inputs have S tokens per (batch, head), the gate vectors SP = NC * L slots; slots past the sequence end are
  // filled with neutral values: log forget gate 0 (nothing decays), input gate -inf (contributes nothing)
  for (int k = c0 + warp; k < c1; k += nwarp) {
    const size_t base_in = (size_t)bh * S + (size_t)k * L;
    const size_t base = (size_t)bh * SP + (size_t)k * L;
    const int valid = min(L, S - k * L);
    float lf[NV], iota[NV];
#pragma unroll
    for (int u = 0; u < NV; ++u) {
      const int j = u * 32 + lane;
      lf[u] = 0.f; iota[u] = -INFINITY;
      if (j < valid) {
        lf[u] = to_f32(vecF[base_in + j]);
        iota[u] = to_f32(vecI[base_in + j]);
      }
    }
#pragma unroll
    for (int u = 0; u < NV; ++u) {
      if (u * 32 + lane < valid) {
        lf[u] = logsigmoid_f(lf[u]);
        if (siging) iota[u] = logsigmoid_f(iota[u]);
      }
    }
    float carry = 0.f;
#pragma unroll
    for (int u = 0; u < NV; ++u) {
      float x = lf[u];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      x += carry;
      if (u * 32 + lane < L) gb.vecB[base + u * 32 + lane] = x;
      carry = __shfl_sync(0xffffffffu, x, 31);
    }
    // a_j as a reverse scan that never includes position j
    float suffix = 0.f, amax = -INFINITY;
#pragma unroll
    for (int u = NV - 1; u >= 0; --u) {
      float x = lf[u];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float y = __shfl_down_sync(0xffffffffu, x, o);
        if (lane + o < 32) x += y;
      }
      float excl = __shfl_down_sync(0xffffffffu, x, 1);
      if (lane == 31) excl = 0.f;
      excl += suffix;
      suffix += __shfl_sync(0xffffffffu, x, 0);
      if (u * 32 + lane < L) {
        const float a = excl + iota[u];
        gb.iota[base + u * 32 + lane] = iota[u];
        gb.abar[base + u * 32 + lane] = a;  // finalised in step 3
        amax = fmaxf(amax, a);
      }
    }
    amax = warp_max(amax);
    if (lane == 0) { g_arr[k] = carry; amax_arr[k] = amax; }
  }
  __syncthreads();

  // composition of the maps of a thread's chunks, then exclusive scan over the threads of the CTA
  const int seg = (c1 - c0 + (int)blockDim.x - 1) / (int)blockDim.x;
  const int k0 = min(c1, c0 + tid * seg), k1 = min(c1, k0 + seg);
  float G = 0.f, A = -INFINITY;
  for (int k = k0; k < k1; ++k) { A = fmaxf(A + g_arr[k], amax_arr[k]); G += g_arr[k]; }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {   // earlier map first: (G1, A1) then (G2, A2) = (G1 + G2, max(A1 + G2, A2))
    const float g1 = __shfl_up_sync(0xffffffffu, G, o), a1 = __shfl_up_sync(0xffffffffu, A, o);
    if (lane >= o) { A = fmaxf(a1 + G, A); G += g1; }
  }
  if (lane == 31) { s_wG[warp] = G; s_wA[warp] = A; }
  float Gx = __shfl_up_sync(0xffffffffu, G, 1), Ax = __shfl_up_sync(0xffffffffu, A, 1);   // maps of the lanes before
  if (lane == 0) { Gx = 0.f; Ax = -INFINITY; }
  __syncthreads();
  if (tid == 0) {
    float g = 0.f, a = -INFINITY;
    for (int w = 0; w < nwarp; ++w) { a = fmaxf(a + s_wG[w], s_wA[w]); g += s_wG[w]; }
    s_total[0] = g; s_total[1] = a;
  }
  cluster.sync();
  float m = sc.m_initial ? sc.m_initial[bh] : sc.m_default, g_before = 0.f;
  for (int r = 0; r < rank; ++r) {     // the CTAs before this one
    const float* t = cluster.map_shared_rank(s_total, r);
    m = fmaxf(m + t[0], t[1]);
    g_before += t[0];
  }
  float* ms = sc.m_states + (size_t)bh * (NC + 1);
  if (tid == 0) {
    // the max state after this CTA's chunks, by the same arithmetic as in the next CTA (which stores the same bits)
    const float m_end = siging ? 0.f : fmaxf(m + s_total[0], s_total[1]);
    ms[c1] = m_end;
    if (rank == ncta - 1) {
      if (sc.m_last != nullptr) sc.m_last[bh] = m_end;
      if (sc.g_sum != nullptr) sc.g_sum[bh] = g_before + s_total[0];
    }
  }
  for (int w = 0; w < warp; ++w) m = fmaxf(m + s_wG[w], s_wA[w]);
  m = fmaxf(m + Gx, Ax);
  for (int k = k0; k < k1; ++k) {
    ms[k] = siging ? 0.f : m;
    m = fmaxf(g_arr[k] + m, amax_arr[k]);
  }
  __syncthreads();
  // the decay of a chunk from the stored max states at its two ends: every factor below uses the same values
  for (int k = k0; k < k1; ++k) gb.gbar[(size_t)bh * NC + k] = siging ? expf(g_arr[k]) : expf(g_arr[k] + ms[k] - ms[k + 1]);

  for (int k = c0 + warp; k < c1; k += nwarp) {
    const size_t base_in = (size_t)bh * S + (size_t)k * L;
    const size_t base = (size_t)bh * SP + (size_t)k * L;
    const int valid = min(L, S - k * L);
    const float m_prev = ms[k], m_next = ms[k + 1];
    float carry = -INFINITY;
#pragma unroll
    for (int u = 0; u < NV; ++u) {
      const int j = u * 32 + lane;
      float b = 0.f, x = -INFINITY;
      if (j < L) { b = gb.vecB[base + j]; x = gb.iota[base + j] - b; }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x = fmaxf(x, y);
      }
      x = fmaxf(x, carry);
      carry = __shfl_sync(0xffffffffu, x, 31);
      if (j < L) {
        float m_i, bbar, abar;
        const float a = gb.abar[base + j];
        if (siging) {
          m_i = 0.f; bbar = expf(b); abar = expf(a);
        } else {
          m_i = fmaxf(b + m_prev, b + x);
          bbar = expf(b + m_prev - m_i);
          abar = expf(a - m_next);
        }
        const bool pad = j >= valid;     // slot past the sequence end: finite max state, every factor zero
        gb.m_tok[base + j] = m_i;
        gb.bbar[base + j] = pad ? 0.f : bbar;
        gb.abar[base + j] = pad ? 0.f : abar;
        if (m_out != nullptr && !pad) m_out[base_in + j] = m_i;
        if (gb.inv_den) {
          gb.inv_den[base + j] = pad ? 0.f
                                 : ((variant == MLSTM_SIG_NONORM || n_out == nullptr) ? 1.f : 1.f / (n_out[base_in + j] + eps));
        }
      }
    }
  }
  cluster.sync();   // no CTA leaves while another may still read its total
}

// Per-token reductions for the gate gradients:
//   qdq_t = sum_d q dq,  kdk_t = sum_d k dk
// mlstm_kernels/torch/chunkwise/triton_xl_chunk/chunkwise_gates.py:68-95. One warp per token.
template <typename T>
__global__ void __launch_bounds__(256)
gate_grad_rows_kernel(const T* q, const T* k, const T* dq, const T* dk, float* __restrict__ acc, float* __restrict__ kdk,
                      size_t ntok, int DHQK) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t tok = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (tok >= ntok) return;
  const int lane = threadIdx.x & 31;
  const size_t base = tok * DHQK;
  float a = 0.f, b = 0.f;
  for (int d = lane; d < DHQK; d += 32) {
    a += to_f32(q[base + d]) * to_f32(dq[base + d]);
    b += to_f32(k[base + d]) * to_f32(dk[base + d]);
  }
  a = warp_sum(a); b = warp_sum(b);
  if (lane == 0) { acc[tok] = a; kdk[tok] = b; }
}

// deltaF_t = sigmoid(-f_t) * sum_{t' >= t over the whole sequence} (qdq_t' - kdk_t') ; deltaI_t = kdk_t (* sigmoid(-i_t)).
// qdq / kdk may arrive as `nparts` partial sums (one per 128-wide head-dim tile), `part_stride` floats apart;
// they are added in a fixed order, so the result does not depend on scheduling.
// One CTA per (batch, head); each thread owns a contiguous token range, block scan over the range sums.
//
// Anchors (tcgen05 path).  q.dq and k.dk nearly cancel, and what is left of their rounding errors (bf16 states and
// operands) adds up along the reverse sum like a random walk: its error grows with the square root of the sequence
// length.  At a chunk boundary the exact value of the sum is known in closed form: with C_k the state before chunk k
// and dC_k its gradient,  sum over all tokens t' >= k L of (q.dq - k.dk) = <C_k, dC_k> - <C_NC, dC_NC>
// (the per-chunk totals telescope: <C_k, dP_k> - <P_k, dC_{k+1}> = <C_k, dC_k> - <C_{k+1}, dC_{k+1}> for
// C_{k+1} = g C_k + P_k, dC_k = g dC_{k+1} + dP_k).  `anchors` holds those inner products for every
// `anchor_tokens`-th token position (state_dot_kernel); the running sum of a token is then taken from the next anchor
// instead of from the end of the sequence, which bounds the walk to one anchor interval (gate_grad_anchored_kernel).
// gate_grad_scan_kernel is the plain form (portable path: f32 states, no anchors).
// The gate gradients leave in the element type the caller asked for (f32, or that of the gate logits).
__device__ __forceinline__ void store_gate_grad(void* p, size_t idx, float x, int dtype) {
  if (dtype == MLSTM_F32) static_cast<float*>(p)[idx] = x;
  else if (dtype == MLSTM_BF16) static_cast<__nv_bfloat16*>(p)[idx] = __float2bfloat16_rn(x);
  else static_cast<__half*>(p)[idx] = __float2half_rn(x);
}

constexpr int kScanThreads = 1024;
template <typename T>
__global__ void __launch_bounds__(kScanThreads)
gate_grad_scan_kernel(const T* vecI, const T* vecF, const float* qdq, const float* kdk, void* __restrict__ dI, void* __restrict__ dF,
                      int out_dtype, int S, int SP, int variant, int nparts, size_t part_stride) {
  __shared__ float s_part[kScanThreads];
  pdl_launch_dependents();
  pdl_wait();
  const int bh = blockIdx.x, t = threadIdx.x;
  const size_t base = (size_t)bh * S;      // gate logits and outputs: S tokens per (batch, head)
  const size_t pbase = (size_t)bh * SP;    // row sums: SP slots per (batch, head)
  const int seg = (S + kScanThreads - 1) / kScanThreads;
  const int s0 = min(S, t * seg), s1 = min(S, (t + 1) * seg);
  auto parts = [&](const float* src, size_t idx) {
    float t = 0.f;
    for (int pp = 0; pp < nparts; ++pp) t += src[pp * part_stride + idx];
    return t;
  };
  float sum = 0.f;
  for (int s = s0; s < s1; ++s) sum += parts(qdq, pbase + s) - parts(kdk, pbase + s);
  s_part[t] = sum;
  __syncthreads();
  // suffix sums over threads (exclusive): sum of the ranges to the right
  for (int o = 1; o < kScanThreads; o <<= 1) {
    float y = (t + o < kScanThreads) ? s_part[t + o] : 0.f;
    __syncthreads();
    s_part[t] += y;
    __syncthreads();
  }
  float run = (t + 1 < kScanThreads) ? s_part[t + 1] : 0.f;
  for (int s = s1 - 1; s >= s0; --s) {
    float di = parts(kdk, pbase + s);
    run += parts(qdq, pbase + s) - di;
    store_gate_grad(dF, base + s, run * sigmoid_f(-to_f32(vecF[base + s])), out_dtype);
    if (variant != MLSTM_EXP) di *= sigmoid_f(-to_f32(vecI[base + s]));
    store_gate_grad(dI, base + s, di, out_dtype);
  }
}

// The anchored form.  Between two anchors the running sum needs nothing from outside the interval: for a token t
// with next anchor position p,  sum_{t' >= t} = sum_{t <= t' < p} (qdq - kdk)  +  anchors[p] - anchors[end]
// (the last interval ends at the end of the sequence, where both anchor terms vanish).  So every interval of
// `anchor_tokens` tokens is an independent CTA: grid (intervals, batch x heads), one token per thread, the suffix
// sum inside the interval by warp shuffles in a fixed order.
constexpr int kAnchorThreads = 512;
template <typename T>
__global__ void __launch_bounds__(kAnchorThreads)
gate_grad_anchored_kernel(const T* vecI, const T* vecF, const float* qdq, const float* kdk, void* __restrict__ dI,
                          void* __restrict__ dF, int out_dtype, int S, int SP, int variant, int nparts, size_t part_stride,
                          const float* anchors, int n_anchors) {
  __shared__ float s_warp[kAnchorThreads / 32];
  const int nint = (S + kAnchorThreads - 1) / kAnchorThreads;   // 1-D grid: intervals of one (batch, head) adjacent
  const int a = blockIdx.x % nint, bh = blockIdx.x / nint, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  pdl_launch_dependents();
  pdl_wait();
  const int s = a * kAnchorThreads + t;
  const bool live = s < S;
  float qd = 0.f, kd = 0.f;
  if (live) {
    const size_t idx = (size_t)bh * SP + s;
    for (int pp = 0; pp < nparts; ++pp) { qd += qdq[pp * part_stride + idx]; kd += kdk[pp * part_stride + idx]; }
  }
  // inclusive suffix sum over the interval: inside the warp, then over the warps to the right
  float x = qd - kd;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float y = __shfl_down_sync(0xffffffffu, x, o);
    if (lane + o < 32) x += y;
  }
  if (lane == 0) s_warp[warp] = x;
  __syncthreads();
  float right = 0.f;
  for (int w = kAnchorThreads / 32 - 1; w > warp; --w) right += s_warp[w];
  float total = x + right;
  if (a + 1 < n_anchors - 1) {   // the interval ends at an interior anchor
    const float* anc = anchors + (size_t)bh * n_anchors;
    total += anc[a + 1] - anc[n_anchors - 1];
  }
  if (live) {
    const size_t o = (size_t)bh * S + s;
    store_gate_grad(dF, o, total * sigmoid_f(-to_f32(vecF[o])), out_dtype);
    store_gate_grad(dI, o, (variant != MLSTM_EXP) ? kd * sigmoid_f(-to_f32(vecI[o])) : kd, out_dtype);
  }
}

// anchors[bh][a] = <C_k, dC_k> over the whole DHQK x DHHV state, k = min(a * every, NC), a = 1 .. n_anchors - 1
// (a = 0 is never read).  One CTA per (anchor, batch x head); the partial sums are added in a fixed order.
template <typename TS>
__global__ void __launch_bounds__(256)
state_dot_kernel(const TS* c_states, const TS* dc_states, float* __restrict__ anchors, int NC, int every, int n_anchors,
                 size_t state_elems) {
  __shared__ float s_w[8];
  const int bh = blockIdx.x / (n_anchors - 1), a = blockIdx.x % (n_anchors - 1) + 1;   // 1-D grid
  const int k = min(a * every, NC);
  pdl_launch_dependents();
  pdl_wait();
  const size_t off = ((size_t)bh * (NC + 1) + k) * state_elems;
  const uint4* pc = reinterpret_cast<const uint4*>(c_states + off);
  const uint4* pd = reinterpret_cast<const uint4*>(dc_states + off);
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (size_t idx = threadIdx.x; idx < state_elems / 8; idx += 256) {
    const uint4 x = ld_stream(pc + idx), y = ld_stream(pd + idx);
    const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, yw[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const TS* xa = reinterpret_cast<const TS*>(&xw[e]);
      const TS* ya = reinterpret_cast<const TS*>(&yw[e]);
      acc[e] = fmaf(to_f32(xa[0]), to_f32(ya[0]), acc[e]);
      acc[e] = fmaf(to_f32(xa[1]), to_f32(ya[1]), acc[e]);
    }
  }
  float v = warp_sum((acc[0] + acc[1]) + (acc[2] + acc[3]));
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.f;
    for (int w = 0; w < 8; ++w) tot += s_w[w];
    anchors[(size_t)bh * n_anchors + a] = tot;
  }
}

// ---- launchers ----------------------------------------------------------------------------------
template <typename T, int NV>
static int launch_gates_nv(const void* i, const void* f, const float* n_out, float* m_out, const GateBuffers& gb,
                           const GateScan& sc, const ChunkwiseDims& d, cudaStream_t st) {
  // enough CTAs per sequence that a warp has one chunk where possible (a cluster holds at most eight); larger CTAs once
  // that leaves a warp more than two
  int ncta = 1;
  while (ncta < 8 && ncta * 8 < d.NC && (long)d.B * d.NH * ncta < 2048) ncta *= 2;
  const int threads = ceil_div(d.NC, ncta) > 16 ? 1024 : 256;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(d.B * d.NH) * ncta);
  cfg.blockDim = dim3(threads);
  cfg.stream = st;
  cudaLaunchAttribute at[2] = {};
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ncta; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = cfg.gridDim.x <= pdl_max_ctas() ? 2 : 1;
  note_launch();
  MLSTM_CUDA_CHECK(cudaLaunchKernelEx(&cfg, gates_kernel<T, NV>, (const T*)i, (const T*)f, n_out, m_out, gb, sc, d.S, d.SP,
                                      d.L, d.NC, d.variant, d.eps));
  return MLSTM_OK;
}

int launch_gates(int dtype, const void* i, const void* f, const float* m_initial, const float* n_out, float* m_out,
                 const GateBuffers& gb, float* m_states, float* m_last, const ChunkwiseDims& d, cudaStream_t st,
                 float m_default, float* g_sum) {
  PhaseScope ps(PH_GATES, st);
  const GateScan sc{m_initial, m_default, m_states, m_last, g_sum};
#define GATES_CASE(DT, T) \
  case DT: return d.L <= 128 ? launch_gates_nv<T, 4>(i, f, n_out, m_out, gb, sc, d, st) \
                             : launch_gates_nv<T, 32>(i, f, n_out, m_out, gb, sc, d, st);
  switch (dtype) {
    GATES_CASE(MLSTM_F32, float)
    GATES_CASE(MLSTM_BF16, __nv_bfloat16)
    GATES_CASE(MLSTM_F16, __half)
  }
#undef GATES_CASE
  return MLSTM_ERR_DTYPE;
}

int gates_force_load() {
  cudaFuncAttributes a;
  MLSTM_CUDA_CHECK(cudaFuncGetAttributes(&a, (gates_kernel<float, 4>)));
  MLSTM_CUDA_CHECK(cudaFuncGetAttributes(&a, (gates_kernel<__nv_bfloat16, 4>)));
  MLSTM_CUDA_CHECK(cudaFuncGetAttributes(&a, (gates_kernel<__half, 4>)));
  MLSTM_CUDA_CHECK(cudaFuncGetAttributes(&a, (gates_kernel<float, 32>)));
  MLSTM_CUDA_CHECK(cudaFuncGetAttributes(&a, (gates_kernel<__nv_bfloat16, 32>)));
  MLSTM_CUDA_CHECK(cudaFuncGetAttributes(&a, (gates_kernel<__half, 32>)));
  return MLSTM_OK;
}

template <typename T>
int launch_gate_grad_rows_t(const void* q, const void* k, const void* dq, const void* dk, float* acc, float* kdk,
                            const ChunkwiseDims& d, cudaStream_t st) {
  const size_t ntok = (size_t)d.B * d.NH * d.S;
  const unsigned grid = (unsigned)((ntok + 7) / 8);
  return launch_pdl(grid <= pdl_max_ctas(), gate_grad_rows_kernel<T>, grid, 256, 0, st, (const T*)q, (const T*)k, (const T*)dq, (const T*)dk,
                    acc, kdk, ntok, d.DHQK);
}



int launch_gate_grads(int dtype, int gate_dtype, const void* q, const void* k, const void* dq, const void* dk,
                      const void* i, const void* f, float* acc, float* kdk, void* dI, void* dF, int out_dtype,
                      const ChunkwiseDims& d, cudaStream_t st) {
  PhaseScope ps(PH_GATE_GRADS, st);
  int rc = MLSTM_ERR_DTYPE;
  switch (dtype) {
    case MLSTM_F32: rc = launch_gate_grad_rows_t<float>(q, k, dq, dk, acc, kdk, d, st); break;
    case MLSTM_BF16: rc = launch_gate_grad_rows_t<__nv_bfloat16>(q, k, dq, dk, acc, kdk, d, st); break;
    case MLSTM_F16: rc = launch_gate_grad_rows_t<__half>(q, k, dq, dk, acc, kdk, d, st); break;
  }
  if (rc != MLSTM_OK) return rc;
  return launch_gate_grad_scan(gate_dtype, i, f, acc, kdk, 1, dI, dF, out_dtype, d, st, nullptr, 0, 1);
}

// Joins the state a sequence segment produced from the EMPTY state (C = 0, n = 0, m = -inf) onto the state that
// enters the segment:  m_out = max(G + m_in, m_loc),  X_out = exp(G + m_in - m_out) X_in + exp(m_loc - m_out) X_loc
// for X in {C, n}; G = total log forget gate of the segment.  Same recursion as the per-chunk update
// (mlstm_kernels/triton/chunkwise/xl_chunk/fw_kernel_recurrent.py:175-196) applied to a whole segment.
__global__ void __launch_bounds__(256)
state_combine_kernel(const float* __restrict__ c_in, const float* __restrict__ n_in, const float* __restrict__ m_in,
                     const float* __restrict__ c_loc, const float* __restrict__ n_loc, const float* __restrict__ m_loc,
                     const float* __restrict__ g_total, float* __restrict__ c_out, float* __restrict__ n_out,
                     float* __restrict__ m_out, int DHQK, int DHHV, int variant, int nblk) {
  const int bh = blockIdx.x / nblk, blk = blockIdx.x % nblk;   // 1-D grid: nblk CTAs per (batch, head)
  float a, b, mo = 0.f;
  if (variant == MLSTM_EXP) {
    const float mi = m_in ? m_in[bh] : 0.f, ml = m_loc[bh], G = g_total[bh];
    mo = fmaxf(G + mi, ml);
    a = expf(G + mi - mo);
    b = expf(ml - mo);
  } else {
    a = expf(g_total[bh]);
    b = 1.f;
  }
  const size_t nC = (size_t)DHQK * DHHV;
  for (size_t e = (size_t)blk * blockDim.x + threadIdx.x; e < nC; e += (size_t)nblk * blockDim.x) {
    const size_t idx = (size_t)bh * nC + e;
    c_out[idx] = a * (c_in ? c_in[idx] : 0.f) + b * c_loc[idx];
    if (e < (size_t)DHQK && n_out != nullptr) {
      const size_t ni = (size_t)bh * DHQK + e;
      n_out[ni] = a * (n_in ? n_in[ni] : 0.f) + b * n_loc[ni];
    }
  }
  if (blk == 0 && threadIdx.x == 0 && m_out != nullptr) m_out[bh] = mo;
}

int launch_state_combine(const float* c_in, const float* n_in, const float* m_in, const float* c_loc,
                         const float* n_loc, const float* m_loc, const float* g_total, float* c_out, float* n_out,
                         float* m_out, int BNH, int DHQK, int DHHV, int variant, cudaStream_t st) {
  const size_t nC = (size_t)DHQK * DHHV;
  const int nblk = (int)std::min<size_t>((nC + 255) / 256, 64);
  state_combine_kernel<<<(unsigned)nblk * (unsigned)BNH, 256, 0, st>>>(c_in, n_in, m_in, c_loc, n_loc, m_loc, g_total,
                                                                      c_out, n_out, m_out, DHQK, DHHV, variant, nblk);
  MLSTM_LAUNCH_CHECK();
  return MLSTM_OK;
}

// inv_den_t = 1 / (n_out_t + eps), or 1 where the variant has no normaliser; 0 in the slots past the sequence end
// (n_out has S entries per (batch, head), inv_den SP slots)
__global__ void __launch_bounds__(256)
inv_den_kernel(const float* __restrict__ n_out, float* __restrict__ inv_den, size_t nslots, int S, int SP, int variant,
               float eps) {
  const size_t t = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (t >= nslots) return;
  const size_t bh = t / SP;
  const int s = (int)(t - bh * SP);
  float v = 0.f;
  if (s < S) v = (variant == MLSTM_SIG_NONORM || n_out == nullptr) ? 1.f : 1.f / (n_out[bh * S + s] + eps);
  inv_den[t] = v;
}

int launch_inv_den(const float* n_out, float* inv_den, const ChunkwiseDims& d, cudaStream_t st) {
  PhaseScope ps(PH_GATES, st);
  const size_t nslots = (size_t)d.B * d.NH * d.SP;
  inv_den_kernel<<<(unsigned)((nslots + 255) / 256), 256, 0, st>>>(n_out, inv_den, nslots, d.S, d.SP, d.variant, d.eps);
  MLSTM_LAUNCH_CHECK();
  return MLSTM_OK;
}

// Scan-only entry: the row sums were already produced (in f32, before rounding) by the backward kernels.
// With `anchors` (see above) the sum restarts from an exact value every `anchor_tokens` tokens and the intervals run
// as independent CTAs; without, one CTA per (batch, head) scans the whole sequence.
template <typename T>
static int gate_grad_scan_t(const void* i, const void* f, const float* qdq, const float* kdk, int nparts, void* dI,
                            void* dF, int out_dtype, const ChunkwiseDims& d, cudaStream_t st, const float* anchors, int n_anchors,
                            int anchor_tokens) {
  const size_t stride = (size_t)d.B * d.NH * d.SP;
  if (anchors != nullptr && anchor_tokens == kAnchorThreads) {
    const unsigned grid = (unsigned)ceil_div(d.S, kAnchorThreads) * (unsigned)(d.B * d.NH);
    return launch_pdl(grid <= pdl_max_ctas(), gate_grad_anchored_kernel<T>, grid, kAnchorThreads, 0, st, (const T*)i, (const T*)f, qdq,
                      kdk, dI, dF, out_dtype, d.S, d.SP, d.variant, nparts, stride, anchors, n_anchors);
  }
  const unsigned grid = (unsigned)(d.B * d.NH);
  return launch_pdl(grid <= pdl_max_ctas(), gate_grad_scan_kernel<T>, grid, kScanThreads, 0, st, (const T*)i, (const T*)f, qdq, kdk, dI, dF,
                    out_dtype, d.S, d.SP, d.variant, nparts, stride);
}

int launch_gate_grad_scan(int dtype, const void* i, const void* f, const float* qdq, const float* kdk, int nparts,
                          void* dI, void* dF, int out_dtype, const ChunkwiseDims& d, cudaStream_t st, const float* anchors,
                          int n_anchors, int anchor_tokens) {
  switch (dtype) {
    case MLSTM_F32: return gate_grad_scan_t<float>(i, f, qdq, kdk, nparts, dI, dF, out_dtype, d, st, anchors, n_anchors, anchor_tokens);
    case MLSTM_BF16: return gate_grad_scan_t<__nv_bfloat16>(i, f, qdq, kdk, nparts, dI, dF, out_dtype, d, st, anchors, n_anchors, anchor_tokens);
    case MLSTM_F16: return gate_grad_scan_t<__half>(i, f, qdq, kdk, nparts, dI, dF, out_dtype, d, st, anchors, n_anchors, anchor_tokens);
  }
  return MLSTM_ERR_DTYPE;
}

// <C_k, dC_k> at every `every`-th chunk boundary and at the end (16-bit states of the tcgen05 path).
int launch_state_dot(const void* c_states, const void* dc_states, float* anchors, int every, int n_anchors,
                     const ChunkwiseDims& d, cudaStream_t st) {
  if (n_anchors < 2) return MLSTM_OK;
  const unsigned grid = (unsigned)(n_anchors - 1) * (unsigned)(d.B * d.NH);
  const size_t elems = (size_t)d.DHQK * d.DHHV;
  if (d.dtype == MLSTM_F16)
    return launch_pdl(grid <= pdl_max_ctas(), state_dot_kernel<__half>, grid, 256, 0, st, (const __half*)c_states,
                      (const __half*)dc_states, anchors, d.NC, every, n_anchors, elems);
  return launch_pdl(grid <= pdl_max_ctas(), state_dot_kernel<__nv_bfloat16>, grid, 256, 0, st, (const __nv_bfloat16*)c_states,
                    (const __nv_bfloat16*)dc_states, anchors, d.NC, every, n_anchors, elems);
}

}  // namespace mlstm
