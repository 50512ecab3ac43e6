// Recurrent decode step (HBM-bound): streams the f32 state C once in and once out with 128-bit
// accesses, keeps everything else on chip.
//
//   m' = max(logsigmoid(f) + m, i);  fbar = exp(logsigmoid(f) + m - m');  ibar = exp(i - m')
//   C' = fbar C + ibar k v^T;  n' = fbar n + ibar k;  h = (s q) C' / (max(|s q . n'|, exp(-m')) + eps)
// mlstm_kernels/triton/recurrent/fw_step_fused.py:19-195, mlstm_kernels/torch/recurrent/native_step.py:8-101.
//
// One CTA owns all DHQK rows of a TV-wide column slice of one (batch, head): the q.C' reduction is
// local to the CTA; q.n' is recomputed per CTA (DHQK values, negligible).
#include "common.cuh"
#include "f32x2.cuh"
#include "launch.cuh"

namespace mlstm {

constexpr int STEP_THREADS = 256;

template <typename TS> struct Vec4;
template <> struct Vec4<float> {
  static __device__ __forceinline__ float4 load(const float* p) { return ld_stream(reinterpret_cast<const float4*>(p)); }
  static __device__ __forceinline__ void store(float* p, float4 v) { __stcs(reinterpret_cast<float4*>(p), v); }
};
template <> struct Vec4<__nv_bfloat16> {
  static __device__ __forceinline__ float4 load(const __nv_bfloat16* p) {
    uint2 raw = ld_stream(reinterpret_cast<const uint2*>(p));
    __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&raw.x), b = *reinterpret_cast<__nv_bfloat162*>(&raw.y);
    return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, float4 v) {
    __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    uint2 raw;
    raw.x = *reinterpret_cast<uint32_t*>(&a);
    raw.y = *reinterpret_cast<uint32_t*>(&b);
    __stcs(reinterpret_cast<uint2*>(p), raw);
  }
};

// The gate pre-activations keep their own element type (f32 gates next to bf16 q, k, v is the usual set-up) and are
// widened to f32 before any arithmetic, as the reference does (fw_step_fused.py:88-94).
__device__ __forceinline__ float load_gate(const void* p, size_t idx, int gate_dtype) {
  if (gate_dtype == MLSTM_F32) return static_cast<const float*>(p)[idx];
  if (gate_dtype == MLSTM_BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[idx]);
  return __half2float(static_cast<const __half*>(p)[idx]);
}

// Bound by HBM where the state does not fit L2 (B = 256: 329 us, the copy bandwidth): four CTAs per SM, rows in batches of
// eight loads then eight stores.  Bound by latency at small batch: while 64-wide column slices would leave SMs without a
// CTA the slices are 32 wide (TV), twice the CTAs with half the rows per thread, and the first eight rows are requested
// before anything waits for the gates, q, k or n (one sequence of 8 heads 256/512: 4.5 -> 3.6 us).  In the wide form the
// early request costs registers, an SM then holds three CTAs, and B = 256 takes 5 % longer (forcing four CTAs by a
// register bound: 1.5 %).
template <typename T, typename TS, int TV, bool PDL>
__global__ void __launch_bounds__(STEP_THREADS)
step_kernel(const T* q, const T* k, const T* v, const void* gi, const void* gf, int gate_dtype, const TS* c, const TS* n,
            const TS* m, T* __restrict__ h, TS* c_new, TS* __restrict__ n_new, TS* __restrict__ m_new, int DHQK, int DHHV,
            float eps) {
  constexpr int CG = TV / 4, RG = STEP_THREADS / CG, NW = STEP_THREADS / 32, UNR = 8;
  constexpr bool EARLY = TV == 32;
  extern __shared__ float sm[];
  float* s_q = sm;                 // [DHQK] scaled q
  float* s_k = s_q + DHQK;         // [DHQK] ibar k
  float* s_red = s_k + DHQK;       // [NW][TV] partial h
  __shared__ float s_warp[NW];
  __shared__ float s_den;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // 1-D grid (no 65535 limit on batch x heads): the column tiles of one (batch, head) next to each other
  const int ntile = (DHHV + TV - 1) / TV;
  const int bh = blockIdx.x / ntile, tile = blockIdx.x % ntile, e0 = tile * TV;
  const int cgi = tid % CG, rg = tid / CG;
  const int e = e0 + cgi * 4;
  const bool live = e < DHHV;

  if (PDL) {
    pdl_launch_dependents();
    pdl_wait();
  }
  float4 first[EARLY ? UNR : 1];
  if (EARLY && live) {
#pragma unroll
    for (int u = 0; u < UNR; ++u)
      if (rg + u * RG < DHQK) first[EARLY ? u : 0] = Vec4<TS>::load(c + ((size_t)bh * DHQK + rg + u * RG) * DHHV + e);
  }

  const float lf = logsigmoid_f(load_gate(gf, bh, gate_dtype));
  const float iv = load_gate(gi, bh, gate_dtype);
  const float m_old = to_f32(m[bh]);
  const float m_n = fmaxf(lf + m_old, iv);
  const float fbar = expf(lf + m_old - m_n);
  const float ibar = expf(iv - m_n);
  const float scale = rsqrtf((float)DHQK);

  // q, k into shared memory; q.n' partial
  float qn = 0.f;
  for (int d = tid; d < DHQK; d += STEP_THREADS) {
    const float qs = to_f32(q[(size_t)bh * DHQK + d]) * scale;
    const float ik = ibar * to_f32(k[(size_t)bh * DHQK + d]);
    const float nn = fmaf(fbar, to_f32(n[(size_t)bh * DHQK + d]), ik);
    s_q[d] = qs;
    s_k[d] = ik;
    qn = fmaf(qs, nn, qn);
    if (tile == 0) n_new[(size_t)bh * DHQK + d] = from_f32<TS>(nn);
  }
  qn = warp_sum(qn);
  if (lane == 0) s_warp[warp] = qn;
  __syncthreads();
  if (tid == 0) {
    float t = 0.f;
    for (int w = 0; w < NW; ++w) t += s_warp[w];
    s_den = fmaxf(fabsf(t), expf(-m_n)) + eps;
    if (tile == 0) m_new[bh] = from_f32<TS>(m_n);
  }

  float4 hv = make_float4(0.f, 0.f, 0.f, 0.f), vv = hv;
  auto step_row = [&](int d, const float4& x, TS* cn) {
    const float kk = s_k[d], qq = s_q[d];
    float4 o;
    o.x = fmaf(fbar, x.x, kk * vv.x);
    o.y = fmaf(fbar, x.y, kk * vv.y);
    o.z = fmaf(fbar, x.z, kk * vv.z);
    o.w = fmaf(fbar, x.w, kk * vv.w);
    Vec4<TS>::store(cn + (size_t)d * DHHV, o);
    hv.x = fmaf(qq, o.x, hv.x); hv.y = fmaf(qq, o.y, hv.y);
    hv.z = fmaf(qq, o.z, hv.z); hv.w = fmaf(qq, o.w, hv.w);
  };
  if (live)
    vv = make_float4(to_f32(v[(size_t)bh * DHHV + e]), to_f32(v[(size_t)bh * DHHV + e + 1]),
                     to_f32(v[(size_t)bh * DHHV + e + 2]), to_f32(v[(size_t)bh * DHHV + e + 3]));
  if (live) {
    const TS* cp = c + (size_t)bh * DHQK * DHHV + e;
    TS* cn = c_new + (size_t)bh * DHQK * DHHV + e;
    int d = rg;
    if (EARLY) {
#pragma unroll
      for (int u = 0; u < UNR; ++u, d += RG)
        if (d < DHQK) step_row(d, first[EARLY ? u : 0], cn);
    }
    for (; d + (UNR - 1) * RG < DHQK; d += UNR * RG) {
      float4 cv[UNR];
#pragma unroll
      for (int u = 0; u < UNR; ++u)
        cv[u] = Vec4<TS>::load(cp + (size_t)(d + u * RG) * DHHV);
#pragma unroll
      for (int u = 0; u < UNR; ++u) step_row(d + u * RG, cv[u], cn);
    }
    for (; d < DHQK; d += RG) step_row(d, Vec4<TS>::load(cp + (size_t)d * DHHV), cn);
  }
  // reduce the column partials over the row groups: first inside the warp (lanes CG apart), then over the warps
#pragma unroll
  for (int o = CG; o < 32; o <<= 1) {
    hv.x += __shfl_xor_sync(0xffffffffu, hv.x, o);
    hv.y += __shfl_xor_sync(0xffffffffu, hv.y, o);
    hv.z += __shfl_xor_sync(0xffffffffu, hv.z, o);
    hv.w += __shfl_xor_sync(0xffffffffu, hv.w, o);
  }
  if (lane < CG) {
    float* dst = s_red + warp * TV + cgi * 4;
    dst[0] = hv.x; dst[1] = hv.y; dst[2] = hv.z; dst[3] = hv.w;
  }
  __syncthreads();
  if (tid < TV && e0 + tid < DHHV) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) t += s_red[w * TV + tid];
    h[(size_t)bh * DHHV + e0 + tid] = from_f32<T>(t / s_den);
  }
}

// T tokens in one launch, the state resident in registers: a CTA owns all DHQK rows of a TV-wide column slice, a thread
// ROWS rows of four columns.  Tokens go through in blocks of SEQ_TB.  What a block needs besides C - gates and their
// max-state recursion, scaled q and k, v, q.n' - is prepared for the whole block at once (one exposed load latency and
// three barriers per block), the token loop itself runs on registers and broadcast shared-memory reads without a
// barrier, and the partial h of the block's tokens are summed over the warps together.  Bound by latency and the issue
// slots: a block's loads, preparation, token loop and reduction follow one another.  What the parts gave, as time per call
// (bf16, 8 heads 256/512 unless stated):
//   token by token with five barriers and a load latency each: 56.5 us for 4 sequences x 13 tokens; in blocks 22.7, and
//   39.1 for 1 x 64, 604 for 16 x 64 with 16 heads.
//   All loads of a block before its first store to shared memory, packed multiply-adds (half the issue slots, the same
//   roundings), the next launch started while this one drains: 20.0 / 41.1 / 558.
//   No test of the row within the token loop where DHQK fills the rows (it kept a row's read of q and k behind the
//   multiply-adds of the row before), two tokens unrolled: 1 x 64 41.1 -> 26.8.  For head dims of q and k above 128 that fill them in
//   part, as many rows as there are, and a test of the last one or two only: 16 x 64, 16 heads 192/384 448 -> 350, 248/496 645 -> 527.
//   At most eight rows per thread up to DHQK = 256 and sixteen up to 512, by narrower slices (see the launch): 19.0 / 26.8 /
//   490; 8 x 16 tokens, DHQK 512: 151 -> 83.
// Two CTAs per SM hide a good part of the chain: bounded by one, the compiler takes more than 128 registers for the eight-row form
// too (490 -> 775).  Above DHQK = 256 the rows alone are up to 64 registers, and 128 leave 64 bytes of spills: a launch that has an
// SM for every CTA takes all registers instead (2 x 48 tokens, 8 heads 264/256: 67.6 -> 34.8; 512/256 65.6 -> 36.9).
constexpr int SEQ_TB = 8;

// FULL: rows that every thread has (DHQK >= FULL * RG); CTAS: per SM
template <typename T, int ROWS, int FULL, int TV, int CTAS>
__global__ void __launch_bounds__(STEP_THREADS, CTAS)
step_sequence_kernel(const T* q, const T* k, const T* v, const void* gi, const void* gf, int gate_dtype, const float* c,
                     const float* n, const float* m, T* __restrict__ h, float* __restrict__ c_new, float* __restrict__ n_new,
                     float* __restrict__ m_new, int Tn, int DHQK, int DHHV, float eps) {
  constexpr int CG = TV / 4, RG = STEP_THREADS / CG, NW = STEP_THREADS / 32;
  constexpr int NV = SEQ_TB * TV / STEP_THREADS;               // elements of v per thread and block
  constexpr int ND = ROWS * RG > STEP_THREADS ? 2 : 1;         // rows per thread of the q, k, n work
  extern __shared__ __align__(16) float sm[];
  float* s_v = sm;                                             // [SEQ_TB][TV]
  float* s_red = s_v + SEQ_TB * TV;                            // [SEQ_TB][NW][TV] partial h
  float2* s_kq = reinterpret_cast<float2*>(s_red + SEQ_TB * NW * TV);   // [SEQ_TB][DHQK] (ibar k, scaled q)
  __shared__ float s_qn[SEQ_TB][NW], s_floor[SEQ_TB];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // 1-D grid (no 65535 limit on batch x heads): the column tiles of one (batch, head) next to each other
  const int ntile = (DHHV + TV - 1) / TV;
  const int bh = blockIdx.x / ntile, tile = blockIdx.x % ntile, e0 = tile * TV;
  const int cgi = tid % CG, rg = tid / CG;
  const int e = e0 + cgi * 4;
  const float scale = rsqrtf((float)DHQK);

  pdl_launch_dependents();
  pdl_wait();
  uint64_t C[ROWS][2];   // four columns of a row, in pairs
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const int d = rg + r * RG;
    const float4 x = (c && d < DHQK && e < DHHV) ? ld_stream(reinterpret_cast<const float4*>(c + ((size_t)bh * DHQK + d) * DHHV + e))
                                                 : make_float4(0.f, 0.f, 0.f, 0.f);
    C[r][0] = f2(x.x, x.y); C[r][1] = f2(x.z, x.w);
  }
  float nv[ND];
#pragma unroll
  for (int u = 0; u < ND; ++u) {
    const int d = tid + u * STEP_THREADS;
    nv[u] = (n && d < DHQK) ? n[(size_t)bh * DHQK + d] : 0.f;
  }
  float m_run = m ? m[bh] : 0.f;

  for (int t0 = 0; t0 < Tn; t0 += SEQ_TB) {
    const int nt = min(SEQ_TB, Tn - t0);
    const size_t tok0 = (size_t)bh * Tn + t0;
    // raw operands of the block first, before anything is stored: all loads of a thread in flight together
    T qr[ND][SEQ_TB], kr[ND][SEQ_TB];
#pragma unroll
    for (int u = 0; u < ND; ++u)
#pragma unroll
      for (int t = 0; t < SEQ_TB; ++t) {
        const int d = tid + u * STEP_THREADS;
        if (d < DHQK && t < nt) {
          qr[u][t] = q[(tok0 + t) * DHQK + d];
          kr[u][t] = k[(tok0 + t) * DHQK + d];
        }
      }
    float vr[NV];
#pragma unroll
    for (int u = 0; u < NV; ++u) {
      const int t = (tid + u * STEP_THREADS) / TV, col = e0 + tid % TV;
      vr[u] = (t < nt && col < DHHV) ? to_f32(v[(tok0 + t) * DHHV + col]) : 0.f;
    }
    // gates: lane t holds token t of the block (every warp for itself); the recursion hands m from lane to lane
    float lf = 0.f, iv = 0.f;
    if (lane < nt) {
      lf = load_gate(gf, tok0 + lane, gate_dtype);
      iv = load_gate(gi, tok0 + lane, gate_dtype);
      lf = logsigmoid_f(lf);
    }
#pragma unroll
    for (int u = 0; u < NV; ++u) s_v[tid + u * STEP_THREADS] = vr[u];
    float m_prev = 0.f, m_tok = 0.f;
    for (int t = 0; t < nt; ++t) {
      const float m_n = fmaxf(__shfl_sync(0xffffffffu, lf, t) + m_run, __shfl_sync(0xffffffffu, iv, t));
      if (lane == t) { m_prev = m_run; m_tok = m_n; }
      m_run = m_n;
    }
    const float fbar_l = expf(lf + m_prev - m_tok), ibar_l = expf(iv - m_tok);
    if (warp == 0 && lane < nt) s_floor[lane] = expf(-m_tok);
    float qn[SEQ_TB];
#pragma unroll
    for (int t = 0; t < SEQ_TB; ++t) {
      const float fbar = __shfl_sync(0xffffffffu, fbar_l, t), ibar = __shfl_sync(0xffffffffu, ibar_l, t);
      qn[t] = 0.f;
#pragma unroll
      for (int u = 0; u < ND; ++u) {
        const int d = tid + u * STEP_THREADS;
        if (d < DHQK && t < nt) {
          const float qs = to_f32(qr[u][t]) * scale;
          const float ik = ibar * to_f32(kr[u][t]);
          nv[u] = fmaf(fbar, nv[u], ik);
          s_kq[t * DHQK + d] = make_float2(ik, qs);
          qn[t] = fmaf(qs, nv[u], qn[t]);
        }
      }
    }
    // the eight sums over the warp together: each step halves the tokens a lane still carries (9 shuffles, not 40)
    static_assert(SEQ_TB == 8, "three halving steps");
#pragma unroll
    for (int half = 4; half >= 1; half >>= 1) {
      const bool up = (lane & (half * 4)) != 0;
#pragma unroll
      for (int t = 0; t < half; ++t) {
        const float mine = up ? qn[t + half] : qn[t], theirs = up ? qn[t] : qn[t + half];
        qn[t] = mine + __shfl_xor_sync(0xffffffffu, theirs, half * 4);
      }
    }
    qn[0] += __shfl_xor_sync(0xffffffffu, qn[0], 2);
    qn[0] += __shfl_xor_sync(0xffffffffu, qn[0], 1);
    if ((lane & 3) == 0) s_qn[lane >> 2][warp] = qn[0];   // bits 4, 3, 2 of the lane spell the token
    __syncthreads();
    const auto token = [&](int t, auto full) {
      const float fbar = __shfl_sync(0xffffffffu, fbar_l, t);
      const ulonglong2 vv = *reinterpret_cast<const ulonglong2*>(s_v + t * TV + cgi * 4);
      const uint64_t ff = f2(fbar, fbar);
      uint64_t h2[2] = {0ull, 0ull};
      const float2* kq = s_kq + t * DHQK + rg;
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        if (r < FULL || decltype(full)::value || rg + r * RG < DHQK) {
          const float2 x = kq[r * RG];
          const uint64_t k2 = f2(x.x, x.x), q2 = f2(x.y, x.y);
          C[r][0] = fma2(ff, C[r][0], mul2(k2, vv.x));
          C[r][1] = fma2(ff, C[r][1], mul2(k2, vv.y));
          h2[0] = fma2(q2, C[r][0], h2[0]);
          h2[1] = fma2(q2, C[r][1], h2[1]);
        }
      }
      float4 hv;
      unf2(h2[0], hv.x, hv.y);
      unf2(h2[1], hv.z, hv.w);
      // over the row groups of the warp (lanes CG apart)
#pragma unroll
      for (int o = CG; o < 32; o <<= 1) {
        hv.x += __shfl_xor_sync(0xffffffffu, hv.x, o);
        hv.y += __shfl_xor_sync(0xffffffffu, hv.y, o);
        hv.z += __shfl_xor_sync(0xffffffffu, hv.z, o);
        hv.w += __shfl_xor_sync(0xffffffffu, hv.w, o);
      }
      if (lane < CG) *reinterpret_cast<float4*>(s_red + (t * NW + warp) * TV + cgi * 4) = hv;
    };
    if (FULL == ROWS || ROWS * RG == DHQK) {
#pragma unroll 2
      for (int t = 0; t < nt; ++t) token(t, std::true_type());
    } else {
#pragma unroll 1
      for (int t = 0; t < nt; ++t) token(t, std::false_type());
    }
    __syncthreads();
    for (int idx = tid; idx < nt * TV; idx += STEP_THREADS) {
      const int t = idx / TV, col = idx % TV;
      if (e0 + col < DHHV) {
        float a = 0.f, qn = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) { a += s_red[(t * NW + w) * TV + col]; qn += s_qn[t][w]; }
        h[(tok0 + t) * DHHV + e0 + col] = from_f32<T>(a / (fmaxf(fabsf(qn), s_floor[t]) + eps));
      }
    }
    __syncthreads();   // the block's buffers are free
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const int d = rg + r * RG;
    float4 x;
    unf2(C[r][0], x.x, x.y);
    unf2(C[r][1], x.z, x.w);
    if (d < DHQK && e < DHHV) __stcs(reinterpret_cast<float4*>(c_new + ((size_t)bh * DHQK + d) * DHHV + e), x);
  }
  if (tile == 0) {
#pragma unroll
    for (int u = 0; u < ND; ++u) {
      const int d = tid + u * STEP_THREADS;
      if (d < DHQK) n_new[(size_t)bh * DHQK + d] = nv[u];
    }
    if (tid == 0) m_new[bh] = m_run;
  }
}

// ---- launchers ----------------------------------------------------------------------------------------
template <typename T, typename TS, int TV, bool PDL>
static int step_tv(const void* q, const void* k, const void* v, const void* i, const void* f, int gate_dtype, const void* c,
                   const void* n, const void* m, void* h, void* c_new, void* n_new, void* m_new, int B, int NH, int DHQK,
                   int DHHV, float eps, cudaStream_t st) {
  const unsigned grid = (unsigned)ceil_div(DHHV, TV) * (unsigned)(B * NH);
  const size_t smem = sizeof(float) * (2 * (size_t)DHQK + (STEP_THREADS / 32) * TV);
  auto kern = step_kernel<T, TS, TV, PDL>;
  if (smem > 48 * 1024) MLSTM_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  return launch_pdl(PDL, kern, grid, STEP_THREADS, smem, st, (const T*)q, (const T*)k, (const T*)v, i, f, gate_dtype,
                    (const TS*)c, (const TS*)n, (const TS*)m, (T*)h, (TS*)c_new, (TS*)n_new, (TS*)m_new, DHQK, DHHV, eps);
}

template <typename T, typename TS>
int step_t(const void* q, const void* k, const void* v, const void* i, const void* f, int gate_dtype, const void* c,
           const void* n, const void* m, void* h, void* c_new, void* n_new, void* m_new, int B, int NH, int DHQK,
           int DHHV, float eps, cudaStream_t st) {
  PhaseScope ps(PH_STEP, st);
#define STEP_RUN(TV, PDL) step_tv<T, TS, TV, PDL>(q, k, v, i, f, gate_dtype, c, n, m, h, c_new, n_new, m_new, B, NH, DHQK, DHHV, eps, st)
  // launches of more than one wave (four CTAs per SM) start plainly: they gain nothing from overlapping their start with
  // the last step's end
  const long ctas = (long)ceil_div(DHHV, 64) * B * NH;
  if (ctas < sm_count()) return STEP_RUN(32, true);
  if (ctas <= 4L * sm_count()) return STEP_RUN(64, true);
  return STEP_RUN(64, false);
#undef STEP_RUN
}

int launch_step(const void* q, const void* k, const void* v, const void* i, const void* f, const void* c,
                const void* n, const void* m, void* h, void* c_new, void* n_new, void* m_new, int B, int NH, int DHQK,
                int DHHV, int dtype, int gate_dtype, int state_dtype, float eps, cudaStream_t st) {
#define STEP_CASE(DT, T, SDT, TS) \
  if (dtype == DT && state_dtype == SDT) return step_t<T, TS>(q, k, v, i, f, gate_dtype, c, n, m, h, c_new, n_new, m_new, B, NH, DHQK, DHHV, eps, st);
  STEP_CASE(MLSTM_F32, float, MLSTM_F32, float)
  STEP_CASE(MLSTM_BF16, __nv_bfloat16, MLSTM_F32, float)
  STEP_CASE(MLSTM_F16, __half, MLSTM_F32, float)
  STEP_CASE(MLSTM_F32, float, MLSTM_BF16, __nv_bfloat16)
  STEP_CASE(MLSTM_BF16, __nv_bfloat16, MLSTM_BF16, __nv_bfloat16)
  STEP_CASE(MLSTM_F16, __half, MLSTM_BF16, __nv_bfloat16)
#undef STEP_CASE
  return MLSTM_ERR_DTYPE;
}

template <typename T, int ROWS, int FULL, int TV, int CTAS>
int step_seq_t(const void* q, const void* k, const void* v, const void* i, const void* f, int gate_dtype, const float* c,
               const float* n, const float* m, void* h, float* c_new, float* n_new, float* m_new, int B, int NH, int Tn,
               int DHQK, int DHHV, float eps, cudaStream_t st) {
  const unsigned grid = (unsigned)ceil_div(DHHV, TV) * (unsigned)(B * NH);
  const size_t smem = sizeof(float) * SEQ_TB * (TV + (STEP_THREADS / 32) * TV + 2 * (size_t)DHQK);
  // Started while the launch before drains, CTAs go where there is room at that moment.  A grid that leaves SMs free ends up two
  // to an SM, which a launch of many tokens pays for (1 x 64 tokens, 128 CTAs: 26.8 us, 36.3 overlapped; 1 x 24: 12.4, 15.1)
  // and one of two blocks does not (1 x 13: 8.9 us, 7.6 overlapped).  Up to half the SMs both launches find SMs of their own,
  // and a grid above their number shares them in any case.
  const unsigned sms = (unsigned)sm_count();
  const bool overlap = grid <= pdl_max_ctas() && (2 * grid <= sms || grid > sms || Tn <= 2 * SEQ_TB);
  auto kern = step_sequence_kernel<T, ROWS, FULL, TV, CTAS>;
  if (smem > 48 * 1024) MLSTM_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  return launch_pdl(overlap, kern, grid, STEP_THREADS, smem, st, (const T*)q, (const T*)k, (const T*)v, i, f, gate_dtype, c, n, m,
                    (T*)h, c_new, n_new, m_new, Tn, DHQK, DHHV, eps);
}

template <typename T>
int step_seq_rows(const void* q, const void* k, const void* v, const void* i, const void* f, int gate_dtype,
                  const float* c, const float* n, const float* m, void* h, float* c_new, float* n_new, float* m_new,
                  int B, int NH, int Tn, int DHQK, int DHHV, float eps, cudaStream_t st) {
  // 32-column slices while 64-column ones would leave SMs without a CTA, and for DHQK above 128: half the rows per thread,
  // for q, k and n prepared once more.  With sixteen rows in 64 columns instead of eight in 32 the registers run short (8 x 64
  // tokens, 8 heads 256/512: 157 us, 125 in 32 columns); with eight in 64 they do not, and the second preparation costs more
  // (16 x 8 tokens, 8 heads 128/256: 13.1 us, 18.6 in 32).
  const bool narrow = DHQK > 128 || (long)ceil_div(DHHV, 64) * B * NH < sm_count();
  // The form with the fewest rows that hold DHQK (up to 128 there is one for each width); at DHQK = 256 the eight-row form that also
  // takes fewer is the faster one by 0.8 % (16 x 64 tokens, 16 heads: 499.5 and 503.5 us).
#define SEQ_CASE(R, F, TV, CTAS) \
  if (ceil_div(DHQK, STEP_THREADS / (TV / 4)) <= R) \
    return step_seq_t<T, R, F, TV, CTAS>(q, k, v, i, f, gate_dtype, c, n, m, h, c_new, n_new, m_new, B, NH, Tn, DHQK, DHHV, eps, st);
  if (narrow) {
    SEQ_CASE(4, 0, 32, 2) SEQ_CASE(5, 4, 32, 2) SEQ_CASE(6, 5, 32, 2) SEQ_CASE(7, 6, 32, 2)
    if (DHQK == 256) { SEQ_CASE(8, 0, 32, 2) }
    SEQ_CASE(8, 7, 32, 2)
    if ((long)ceil_div(DHHV, 32) * B * NH <= sm_count()) { SEQ_CASE(12, 8, 32, 1) SEQ_CASE(14, 12, 32, 1) SEQ_CASE(16, 14, 32, 1) }
    if (DHQK == 512) { SEQ_CASE(16, 16, 32, 2) }
    SEQ_CASE(12, 8, 32, 2) SEQ_CASE(14, 12, 32, 2) SEQ_CASE(16, 14, 32, 2)
  }
  SEQ_CASE(4, 0, 64, 2) SEQ_CASE(8, 0, 64, 2)
#undef SEQ_CASE
  return MLSTM_ERR_SHAPE;
}

int launch_step_sequence(const void* q, const void* k, const void* v, const void* i, const void* f, const float* c,
                         const float* n, const float* m, void* h, float* c_new, float* n_new, float* m_new, int B,
                         int NH, int T, int DHQK, int DHHV, int dtype, int gate_dtype, float eps, cudaStream_t st) {
  switch (dtype) {
    case MLSTM_F32: return step_seq_rows<float>(q, k, v, i, f, gate_dtype, c, n, m, h, c_new, n_new, m_new, B, NH, T, DHQK, DHHV, eps, st);
    case MLSTM_BF16: return step_seq_rows<__nv_bfloat16>(q, k, v, i, f, gate_dtype, c, n, m, h, c_new, n_new, m_new, B, NH, T, DHQK, DHHV, eps, st);
    case MLSTM_F16: return step_seq_rows<__half>(q, k, v, i, f, gate_dtype, c, n, m, h, c_new, n_new, m_new, B, NH, T, DHQK, DHHV, eps, st);
  }
  return MLSTM_ERR_DTYPE;
}

}  // namespace mlstm
