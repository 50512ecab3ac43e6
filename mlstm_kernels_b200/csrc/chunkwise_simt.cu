// Portable CUDA-core implementation of the chunkwise mLSTM kernels (any chunk size >= 16, any head
// dimension, f32 / bf16 / f16 inputs, exact f32 arithmetic).  It covers the shapes the tcgen05 path
// does not (small chunks, odd head dims, f32 inputs) and is the on-device cross-check for it.
//
//   part_kernel, rec_scan_kernel, rec_final_kernel : inter-chunk recurrence, forward (C_k, n_k) and backward (deltaC_k);
//                 part_kernel also computes the gated score blocks that the output tiles of a chunk share
//                 mlstm_kernels/triton/chunkwise/xl_chunk/fw_kernel_recurrent.py:14-230,
//                 bw_kernel_recurrent.py:15-181
//   par_fw_kernel, par_bw_kernel  : intra-chunk gated products + inter-chunk contribution for H; deltaV, deltaK, deltaQ
//                 fw_kernel_parallel.py:14-289, bw_kernel_parallel_dV.py, _dK.py, _dQ.py
#include "common.cuh"
#include "f32x2.cuh"
#include "launch.cuh"

namespace mlstm {

constexpr int TILE = 64;   // output tile edge per CTA
constexpr int KSL = 32;    // contraction slice staged in shared memory
constexpr int NTHR = 256;  // 16 x 16 threads, 4 x 4 outputs each

// ---- 64 x 64 tile product: 256 threads, double-buffered slices of 32 along the contraction --------------------
// Slices lie in shared memory contraction-major ([k][64]), so that a thread reads its 4 rows and 4 columns of one k as
// two 16-byte words for 16 multiply-adds, issued as 8 packed fma.rn.f32x2 (same rounding as two fmaf).  16-byte
// groups are XOR-swizzled by bits 2..4 of k: rows written transposed (contraction contiguous in memory) and rows
// written straight both land without bank conflicts.  The next slice is fetched into registers while the current one
// is multiplied.  Bound by the shared-memory port in large launches (84 % of its wavefronts: a warp's two reads return
// 1 KB for 8 packed multiply-adds) and by load and barrier latency in small ones, where two warps per scheduler and CTA
// measured faster than one with 8 x 4 outputs per thread.  Measured 30-34 TFLOP/s at B=4 NH=4 S=2048 128/256; unbuffered
// slices, scalar reads and a serial recurrence ran at 4.
__device__ __forceinline__ int swz(int k, int x) { return k * TILE + (((x >> 2) ^ ((k >> 2) & 7)) << 2) + (x & 3); }

__device__ __forceinline__ int row_group(int tid) { return tid >> 4; }
__device__ __forceinline__ int col_group(int tid) { return tid & 15; }
// sum over the 16 column groups of a row group
__device__ __forceinline__ float sum_columns(float x) {
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

struct Acc {   // rows 4 ty + {0..3} in pairs, columns 4 tx + {0..3}
  uint64_t v[2][4];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) v[a][b] = 0ull;
  }
  __device__ __forceinline__ void get(float (&x)[4][4]) const {
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        unf2(v[a][b], x[2 * a][b], x[2 * a + 1][b]);
      }
  }
};

// acc += A B over the 32 contraction steps of one staged slice pair.  Rolled over groups of four steps that share a
// swizzle: unrolled further, the kernels' several copies of this loop outgrew the instruction cache.
__device__ __forceinline__ void mma_slice(Acc& acc, const float* A, const float* B, int ty, int tx) {
#pragma unroll 2
  for (int kq = 0; kq < KSL / 4; ++kq) {
    const float* pa = A + kq * 4 * TILE + ((ty ^ kq) << 2);
    const float* pb = B + kq * 4 * TILE + ((tx ^ kq) << 2);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(pa + k * TILE);
      const float4 b = *reinterpret_cast<const float4*>(pb + k * TILE);
      const uint64_t av[2] = {a.x, a.y};
      const uint64_t bv[4] = {f2(b.x, b.x), f2(b.y, b.y), f2(b.z, b.z), f2(b.w, b.w)};
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n) acc.v[m][n] = fma2(av[m], bv[n], acc.v[m][n]);
    }
  }
}

// four consecutive elements of a row, zero outside [0, cols); `vec`: rows start on 4-element boundaries
__device__ __forceinline__ float4 load4(const float* p, int c, int cols, bool vec) {
  if (vec) return c < cols ? *reinterpret_cast<const float4*>(p + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  return make_float4(c < cols ? p[c] : 0.f, c + 1 < cols ? p[c + 1] : 0.f, c + 2 < cols ? p[c + 2] : 0.f,
                     c + 3 < cols ? p[c + 3] : 0.f);
}
template <typename T>
__device__ __forceinline__ void store4(T* p, int c, int cols, bool vec, float4 v) {
  if (vec && sizeof(T) == 4) {
    if (c < cols) *reinterpret_cast<float4*>(p + c) = v;
    return;
  }
  if (c < cols) p[c] = from_f32<T>(v.x);
  if (c + 1 < cols) p[c + 1] = from_f32<T>(v.y);
  if (c + 2 < cols) p[c + 2] = from_f32<T>(v.z);
  if (c + 3 < cols) p[c + 3] = from_f32<T>(v.w);
}

// A matrix operand in global memory: rows x cols, `scale` (or null) multiplies whole rows.
template <typename T>
struct Mat {
  const T* p;
  const float* scale;
  int rows, cols, ld;
};

// One slice of an operand in flight: 2048 elements, two groups of four per thread.  The loads' results are not touched
// before put() (no conversion, no scaling: either would wait for the load), so they travel under the current slice's
// multiply-adds.  VEC: rows start on four-element boundaries.
//   TR = true   tile rows x0.. are matrix rows, the contraction k0.. runs along the columns (transposed into shared memory)
//   TR = false  the contraction k0.. runs over matrix rows, the tile columns x0.. along the columns
template <typename T, bool TR, bool VEC>
struct Slice {
  struct __align__(4 * sizeof(T)) Raw { T e[4]; };
  Raw v[2];
  float sc[2];
  __device__ __forceinline__ void fetch(const Mat<T>& m, int x0, int k0, int tid) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = TR ? x0 + (tid >> 3) + 32 * u : k0 + (tid >> 4) + 16 * u;
      const int c = TR ? k0 + 4 * (tid & 7) : x0 + 4 * (tid & 15);
      const T* p = m.p + (size_t)r * m.ld + c;
      if (VEC) {
        v[u] = Raw{};
        if (r < m.rows && c < m.cols) v[u] = *reinterpret_cast<const Raw*>(p);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          v[u].e[e] = from_f32<T>(0.f);
          if (r < m.rows && c + e < m.cols) v[u].e[e] = p[e];
        }
      }
      sc[u] = 1.f;
      if (m.scale && r < m.rows) sc[u] = m.scale[r];
    }
  }
  __device__ __forceinline__ void put(float* s, int tid) const {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = to_f32(v[u].e[e]) * sc[u];
      if (TR) {
        const int r = (tid >> 3) + 32 * u, k = 4 * (tid & 7);
#pragma unroll
        for (int e = 0; e < 4; ++e) s[swz(k + e, r)] = x[e];
      } else {
        *reinterpret_cast<float4*>(s + swz((tid >> 4) + 16 * u, 4 * (tid & 15))) = make_float4(x[0], x[1], x[2], x[3]);
      }
    }
  }
};

constexpr int SLICE = KSL * TILE;   // floats of one staged slice

// acc += A B over the contraction [0, K); buf: 4 slices (two of A, two of B).  After the last slice every thread has
// passed a barrier that follows its last read of the older buffer pair only: callers synchronise before reusing buf.
// each(slice of A, k0) runs once per slice while it lies in shared memory.
template <bool VEC, bool TRA, bool TRB, typename TA, typename TB, typename F>
__device__ __forceinline__ void tile_product(Acc& acc, const Mat<TA>& A, int a0, const Mat<TB>& B, int b0, int K, float* buf,
                                             int tid, F each) {
  const int ty = row_group(tid), tx = col_group(tid);
  Slice<TA, TRA, VEC> sa;
  Slice<TB, TRB, VEC> sb;
  sa.fetch(A, a0, 0, tid);
  sb.fetch(B, b0, 0, tid);
  int cur = 0;
  for (int k0 = 0; k0 < K; k0 += KSL) {
    float* As = buf + cur * SLICE;
    float* Bs = buf + (2 + cur) * SLICE;
    sa.put(As, tid);
    sb.put(Bs, tid);
    __syncthreads();
    if (k0 + KSL < K) {
      sa.fetch(A, a0, k0 + KSL, tid);
      sb.fetch(B, b0, k0 + KSL, tid);
    }
    each(As, k0);
    mma_slice(acc, As, Bs, ty, tx);
    cur ^= 1;
  }
}
struct NoEach { __device__ __forceinline__ void operator()(const float*, int) const {} };

// =====================================================================================================
// Inter-chunk recurrence.  state <- gbar * state + lmul * (left * lscale)^T (right * rscale)
//   forward : left = K, lscale = abar, right = V;  also n <- gbar n + sum_j abar_j k_j
//   backward: left = Q, lscale = bbar, lmul = qk_scale, right = deltaH, rscale = 1/(den+eps); chunks reversed
// Where the per-chunk states are wanted, the chunks' contributions are independent CTAs that leave them in the state
// buffer itself (part_kernel), and an element-wise scan over the chunks turns them into states in place
// (rec_scan_kernel, one thread per four elements): a CTA that walks a whole sequence took 9.6 us per chunk of 64 tokens
// while most SMs idled.  Without a state buffer (segment summaries) rec_final_kernel walks the chunks of its tile.
// =====================================================================================================
template <typename T>
struct RecArgs {
  const T *left, *right;
  const float *lscale, *rscale, *gbar;
  float lmul;
  const float *c_init, *n_init;
  float *c_states, *n_states, *c_final, *n_final;
  int S, L, NC, DHQK, DHHV;
};

// P = (left * lscale)^T (right * rscale) of chunk ck for the tile (d0, e0); ns: column sums of the scaled left rows
template <typename T, bool VEC>
__device__ __forceinline__ void chunk_part(const RecArgs<T>& p, int bh, int ck, int d0, int e0, bool do_n, float* buf, Acc& acc,
                                           float (&ns)[4]) {
  const int tid = threadIdx.x, ty = row_group(tid), tx = col_group(tid);
  const size_t tok0 = (size_t)bh * p.S + (size_t)ck * p.L;
  const Mat<T> A{p.left + tok0 * p.DHQK, p.lscale + tok0, p.L, p.DHQK, p.DHQK};
  const Mat<T> B{p.right + tok0 * p.DHHV, p.rscale ? p.rscale + tok0 : nullptr, p.L, p.DHHV, p.DHHV};
  acc.zero();
#pragma unroll
  for (int a = 0; a < 4; ++a) ns[a] = 0.f;
  tile_product<VEC, false, false>(acc, A, d0, B, e0, p.L, buf, tid, [&](const float* As, int) {
    if (!do_n) return;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int a = 0; a < 4; ++a) ns[a] += As[swz(2 * tx + u, 4 * ty + a)];
  });
  if (do_n) {
#pragma unroll
    for (int a = 0; a < 4; ++a) ns[a] = sum_columns(ns[a]);
  }
}

// One tile of one chunk's contribution to the state, of the forward's recurrence or (bwd) the gradient's.
template <typename T, bool VEC>
__device__ __forceinline__ void rec_part_tile(const RecArgs<T>& p, const bool bwd, const unsigned block, float* buf) {
  // the tiles of one chunk next to each other (they share its operands through L2)
  const int n_et = (p.DHHV + TILE - 1) / TILE, n_dt = (p.DHQK + TILE - 1) / TILE;
  const int et = block % n_et, dt = (block / n_et) % n_dt, bc = block / (n_et * n_dt);
  const int bh = bc / p.NC, ck = bc % p.NC, e0 = et * TILE, d0 = dt * TILE;
  const bool do_n = !bwd && et == 0 && p.n_states != nullptr;
  const int ty = row_group(threadIdx.x), tx = col_group(threadIdx.x);
  Acc acc;
  float ns[4], x[4][4];
  chunk_part<T, VEC>(p, bh, ck, d0, e0, do_n, buf, acc, ns);
  acc.get(x);
  const size_t slot = (size_t)bh * (p.NC + 1) + (bwd ? ck : ck + 1);
  float* out = p.c_states + slot * p.DHQK * p.DHHV;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int d = d0 + 4 * ty + a;
    if (d < p.DHQK)
      store4(out + (size_t)d * p.DHHV, e0 + 4 * tx, p.DHHV, VEC,
             make_float4(x[a][0] * p.lmul, x[a][1] * p.lmul, x[a][2] * p.lmul, x[a][3] * p.lmul));
    if (do_n && tx == 0 && d < p.DHQK) p.n_states[slot * p.DHQK + d] = ns[a];
  }
}

// ---- gated score blocks ------------------------------------------------------------------------------
// block[i][j] = qk_scale * (a_i . b_j) * D(i,j) for j <= i, else 0: 64 x 64 tokens of one chunk.
template <typename T>
struct ScoreArgs {
  const T *a, *b;          // rows i and j
  const float* a_scale;    // per token or null
  float* out;              // [chunk][pair of 64-token blocks, (0,0), (1,0), (1,1), ..][64][64]
  int D;                   // contraction
};
struct ScoreGate {
  const float *vecB, *iota, *m_tok;
  int S, L, NC;
  float qk_scale;
};
__host__ __device__ constexpr int score_pairs(int L) { const int nb = (L + TILE - 1) / TILE; return nb * (nb + 1) / 2; }
__device__ __forceinline__ int score_pair(int rb, int cb) { return rb * (rb + 1) / 2 + cb; }

__device__ __forceinline__ float gate_score(float s, float qk_scale, float b_i, float b_j, float iota_j, float m_i) {
  return qk_scale * s * expf((b_i - b_j) + iota_j - m_i);
}

template <typename T, bool VEC>
__device__ __forceinline__ void score_tile(const ScoreArgs<T>& p, const ScoreGate& g, const unsigned block, float* buf) {
  const int np = score_pairs(g.L), pair = block % np, bc = block / np, bh = bc / g.NC, ck = bc % g.NC;
  int rb = 0;
  while (score_pair(rb + 1, 0) <= pair) ++rb;
  const int r0 = rb * TILE, c0 = (pair - score_pair(rb, 0)) * TILE;
  const int tid = threadIdx.x, ty = row_group(tid), tx = col_group(tid);
  const size_t tok0 = (size_t)bh * g.S + (size_t)ck * g.L;
  const Mat<T> A{p.a + tok0 * p.D, p.a_scale ? p.a_scale + tok0 : nullptr, g.L, p.D, p.D}, B{p.b + tok0 * p.D, nullptr, g.L, p.D, p.D};
  Acc pr;
  pr.zero();
  tile_product<VEC, true, true>(pr, A, r0, B, c0, p.D, buf, tid, NoEach());
  float s[4][4], b_j[4], iota_j[4];
  pr.get(s);
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const int c = c0 + 4 * tx + b;
    b_j[b] = c < g.L ? g.vecB[tok0 + c] : 0.f;
    iota_j[b] = c < g.L ? g.iota[tok0 + c] : 0.f;
  }
  float* out = p.out + (size_t)block * TILE * TILE;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = r0 + 4 * ty + a;
    const float b_i = r < g.L ? g.vecB[tok0 + r] : 0.f, m_i = r < g.L ? g.m_tok[tok0 + r] : 0.f;
    float v[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int c = c0 + 4 * tx + b;
      v[b] = r < g.L && c <= r ? gate_score(s[a][b], g.qk_scale, b_i, b_j[b], iota_j[b], m_i) : 0.f;
    }
    *reinterpret_cast<float4*>(out + (4 * ty + a) * TILE + 4 * tx) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

// None of these kernels lets the next launch in before its CTAs end (there is no pdl_launch_dependents()): three of them fit an SM, more
// in the scan, and the CTAs of a launch that does not fill the GPU, placed while another one still has most SMs, come to lie
// three to an SM (2 x 4 x 512 tokens, 64/128, forward and backward in us, with it at the start and without: chunk 128 141 and 101,
// chunk 64 87 and 69; 4 x 4 x 512, 104/104, chunk 256, raw calls 397 and 351; 1 x 4 x 64, 64/64 52.1 and 50.1).

// The products that need nothing but inputs and gate vectors, in one launch: the score blocks (the longer ones, first) and the
// chunks' contributions of one recurrence or two.  Alone each of them is a launch of one wave or less, bound by load and
// barrier latency; the score blocks ran in every output tile of their chunk, a quarter of the forward's multiply-adds and 43 % of
// the backward's (B=2 NH=4 S=512 128/256, chunk 64, forward and backward phases in us: recurrences 42 and 21, now, with the
// scores, 25 and 37; intra-chunk 35 and 81, now 23 and 50; the call 180 -> 136, same bits).
template <typename T>
struct PartArgs {
  ScoreArgs<T> sc[2];
  RecArgs<T> rec[2];
  ScoreGate gate;
  unsigned end[4];         // CTAs up to and with: sc[0], sc[1], rec[0], rec[1]
  bool bwd[2];             // rec[i] is the state gradient's
};

// SCORES: there are score blocks.  Without them 64 registers do, and a fourth CTA to an SM (0: the compiler's choice, 80): 4 heads, 2048
// tokens, 128/256, chunk 32, recurrence 52 us at 80, 41 at 64.
template <typename T, bool VEC, bool SCORES>
__global__ void __launch_bounds__(NTHR, SCORES ? 0 : 4) part_kernel(const __grid_constant__ PartArgs<T> p) {
  __shared__ __align__(16) float buf[4 * SLICE];
  pdl_wait();
  const unsigned x = blockIdx.x;
  if (SCORES && x < p.end[1]) {
    const int i = x >= p.end[0];
    score_tile<T, VEC>(p.sc[i], p.gate, i ? x - p.end[0] : x, buf);
  } else {
    const int i = x >= p.end[2];
    rec_part_tile<T, VEC>(p.rec[i], p.bwd[i], x - p.end[1 + i], buf);
  }
}

template <int V> struct Vec;
template <> struct Vec<1> { float v[1]; __device__ void load(const float* p) { v[0] = *p; } __device__ void store(float* p) const { *p = v[0]; } };
template <> struct Vec<4> {
  float v[4];
  __device__ void load(const float* p) { const float4 f = *reinterpret_cast<const float4*>(p); v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w; }
  __device__ void store(float* p) const { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
};

// Element-wise: states[k+1] = gbar_k states[k] + states[k+1] in place (BWD: right to left).  Bound by memory (each
// element read and written once); four loads in flight ahead of the dependent multiply-adds.
template <int V, bool BWD>
__device__ __forceinline__ void scan_elements(float* states, const float* init, float* fin, const float* gbar, size_t E, size_t e, int NC) {
  Vec<V> c;
#pragma unroll
  for (int i = 0; i < V; ++i) c.v[i] = 0.f;
  if (init) c.load(init + e);
  c.store(states + (size_t)(BWD ? NC : 0) * E + e);
  constexpr int AHEAD = 4;
  for (int s0 = 0; s0 < NC; s0 += AHEAD) {
    Vec<V> part[AHEAD];
    float g[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      if (s0 + u < NC) {
        const int ck = BWD ? NC - 1 - (s0 + u) : s0 + u;
        part[u].load(states + (size_t)(BWD ? ck : ck + 1) * E + e);
        g[u] = gbar[ck];
      }
    }
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      if (s0 + u < NC) {
        const int ck = BWD ? NC - 1 - (s0 + u) : s0 + u;
#pragma unroll
        for (int i = 0; i < V; ++i) c.v[i] = fmaf(g[u], c.v[i], part[u].v[i]);
        c.store(states + (size_t)(BWD ? ck : ck + 1) * E + e);
      }
    }
  }
  if (fin) c.store(fin + e);
}

struct ScanArgs {
  float* c_states;
  const float* c_init;
  float *c_final, *n_states;
  const float* n_init;
  float* n_final;
  int nblk;                // CTAs per (batch, head)
};
template <int V, bool BWD>
__device__ __forceinline__ void scan_tile(const ScanArgs& a, const float* gbar, int NC, int DHQK, int DHHV, const unsigned block) {
  const int bh = block / a.nblk;
  const size_t E = (size_t)DHQK * DHHV, t = (size_t)(block % a.nblk) * 128 + threadIdx.x;
  const float* g = gbar + (size_t)bh * NC;
  if (t * V < E) {
    scan_elements<V, BWD>(a.c_states + (size_t)bh * (NC + 1) * E, a.c_init ? a.c_init + bh * E : nullptr,
                          a.c_final ? a.c_final + bh * E : nullptr, g, E, t * V, NC);
  } else if (!BWD && a.n_states != nullptr && t - (E + V - 1) / V < (size_t)DHQK) {   // threads past the tiles: n
    scan_elements<1, BWD>(a.n_states + (size_t)bh * (NC + 1) * DHQK, a.n_init ? a.n_init + (size_t)bh * DHQK : nullptr,
                          a.n_final ? a.n_final + (size_t)bh * DHQK : nullptr, g, DHQK, t - (E + V - 1) / V, NC);
  }
}
// the first n_fw CTAs scan the forward's states, the others the gradient's; FW, BW: whether there are any of them (one kind takes 40
// registers, both in one kernel 56)
template <int V, bool FW, bool BW>
__global__ void __launch_bounds__(128)
rec_scan_kernel(const ScanArgs fw, const ScanArgs bw, const unsigned n_fw, const float* gbar, int NC, int DHQK, int DHHV) {
  pdl_wait();
  if (FW && (!BW || blockIdx.x < n_fw)) scan_tile<V, false>(fw, gbar, NC, DHQK, DHHV, blockIdx.x);
  else scan_tile<V, true>(bw, gbar, NC, DHQK, DHHV, FW ? blockIdx.x - n_fw : blockIdx.x);
}

// Final state only, one CTA per tile walking the chunks.
template <typename T, bool BWD, bool VEC>
__global__ void __launch_bounds__(NTHR) rec_final_kernel(RecArgs<T> p) {
  __shared__ __align__(16) float buf[4 * SLICE];
  const int n_et = (p.DHHV + TILE - 1) / TILE, n_dt = (p.DHQK + TILE - 1) / TILE;
  const int et = blockIdx.x % n_et, dt = (blockIdx.x / n_et) % n_dt, bh = blockIdx.x / (n_et * n_dt);
  const int e0 = et * TILE, d0 = dt * TILE, ty = row_group(threadIdx.x), tx = col_group(threadIdx.x);
  const bool do_n = !BWD && et == 0 && p.n_final != nullptr;
  float C[4][4], n[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int d = d0 + 4 * ty + a;
    const float4 c = (p.c_init && d < p.DHQK) ? load4(p.c_init + ((size_t)bh * p.DHQK + d) * p.DHHV, e0 + 4 * tx, p.DHHV, VEC)
                                             : make_float4(0.f, 0.f, 0.f, 0.f);
    C[a][0] = c.x; C[a][1] = c.y; C[a][2] = c.z; C[a][3] = c.w;
    n[a] = (do_n && p.n_init && d < p.DHQK) ? p.n_init[(size_t)bh * p.DHQK + d] : 0.f;
  }
  for (int s = 0; s < p.NC; ++s) {
    const int ck = BWD ? p.NC - 1 - s : s;
    Acc acc;
    float ns[4], x[4][4];
    chunk_part<T, VEC>(p, bh, ck, d0, e0, do_n, buf, acc, ns);
    acc.get(x);
    const float g = p.gbar[(size_t)bh * p.NC + ck];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      n[a] = fmaf(g, n[a], ns[a]);
#pragma unroll
      for (int b = 0; b < 4; ++b) C[a][b] = fmaf(g, C[a][b], x[a][b] * p.lmul);
    }
    __syncthreads();   // the slices are free for the next chunk
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int d = d0 + 4 * ty + a;
    if (d >= p.DHQK) continue;
    if (p.c_final) store4(p.c_final + ((size_t)bh * p.DHQK + d) * p.DHHV, e0 + 4 * tx, p.DHHV, VEC, make_float4(C[a][0], C[a][1], C[a][2], C[a][3]));
    if (do_n && tx == 0) p.n_final[(size_t)bh * p.DHQK + d] = n[a];
  }
}

// =====================================================================================================
// Intra-chunk kernel, four modes.  For the output tile rows r (tokens of one chunk) and columns o:
//   out[r,o] = sum_c P[r,c] X[c,o] + rowscale_r * sum_a U[r,a] Bm[a,o]
//   P[r,c]   = qk_scale * (U[r] . W[c]) * D(i,j),  D(i,j) = exp((b_i - b_j) + iota_j - m_i) for j <= i
//   mode  U        W        (i,j)   X        rowscale        Bm
//   H     Q        K        (r,c)   V        qk_scale*bbar   C_k[a][o]
//   DV    K        Q        (c,r)   dHbar    abar            dC_{k+1}[a][o]
//   DK    V        dHbar    (c,r)   Q        abar            dC_{k+1}[o][a]
//   DQ    dHbar    V        (r,c)   K        qk_scale*bbar   C_k[o][a]
// dHbar = deltaH / (den + eps).  1-D grid (output tiles x 64-row blocks of the chunk x B*NH*NC); the backward's three modes share a launch
// (their CTAs fill each other's last wave and find a chunk's operands in L2).
// The contraction runs on CUDA cores in exact f32: 64 x 64 tiles of the product above, at B=2 NH=4 S=512 128/256 a few
// hundred CTAs of a few million multiply-adds each.
// =====================================================================================================
enum { PAR_H = 0, PAR_DV = 1, PAR_DK = 2, PAR_DQ = 3 };

template <typename T>
struct ParArgs {
  const T *q, *k, *v, *dh;
  const float *vecB, *iota, *m_tok, *abar, *bbar, *inv_den;
  const float* c_states;   // slot k used by H and DQ
  const float* dc_states;  // slot k+1 used by DV and DK
  const float* n_states;
  const float *qk_blocks, *vh_blocks;   // gated score blocks (score_tile) of Q K^T and dHbar V^T, or null: computed by every output tile anew
  T *out_h, *out_dv, *out_dk, *out_dq;
  float* n_out;            // H only, may be null
  float* inv_den_out;      // H only, may be null
  int S, L, NC, DHQK, DHHV, variant;
  float eps, qk_scale;
};

// FW: mode PAR_H only; otherwise `mode` is one of the gradients, uniform over the CTA - one body for the three (three
// inlined copies stalled on instruction fetch as often as they issued).
template <typename T, bool FW, bool VEC>
__device__ __forceinline__ void par_tile(const ParArgs<T>& p, const int mode, int ot, int bc, int rb, float* smem) {
  const bool LOWER = FW || mode == PAR_DQ;
  const bool QK = FW || mode == PAR_DV;   // score over DHQK, output over DHHV (else the other way)
  const int L = p.L;
  float* buf = smem;                  // [4][32][64] slices
  float* Ps = buf + 4 * SLICE;        // [64 c][64 r] gated score block
  float* s_b = Ps + TILE * TILE;      // [L] each
  float* s_iota = s_b + L;
  float* s_m = s_iota + L;
  float* s_n = s_m + L;               // PAR_H: [DHQK, rounded up to whole slices] n_k

  const int tid = threadIdx.x, ty = row_group(tid), tx = col_group(tid);
  const int o0 = ot * TILE, r0 = rb * TILE, bh = bc / p.NC, ck = bc % p.NC;
  const size_t tok0 = (size_t)bh * p.S + (size_t)ck * L;
  const int DI = QK ? p.DHQK : p.DHHV;   // contraction of the score and of the inter-chunk term
  const int DO = QK ? p.DHHV : p.DHQK;   // output width
  const Mat<T> mq{p.q + tok0 * p.DHQK, nullptr, L, p.DHQK, p.DHQK}, mk{p.k + tok0 * p.DHQK, nullptr, L, p.DHQK, p.DHQK};
  const Mat<T> mv{p.v + tok0 * p.DHHV, nullptr, L, p.DHHV, p.DHHV};
  const Mat<T> mh{p.dh + tok0 * p.DHHV, p.inv_den + tok0, L, p.DHHV, p.DHHV};
  const Mat<T> U = FW ? mq : mode == PAR_DV ? mk : mode == PAR_DK ? mv : mh;
  const Mat<T> W = FW ? mk : mode == PAR_DV ? mq : mode == PAR_DK ? mh : mv;
  const Mat<T> X = FW ? mv : mode == PAR_DV ? mh : mode == PAR_DK ? mq : mk;
  const size_t state_elems = (size_t)p.DHQK * p.DHHV, slab = (size_t)bh * (p.NC + 1) + ck;
  const Mat<float> St{LOWER ? p.c_states + slab * state_elems : p.dc_states + (slab + 1) * state_elems, nullptr, p.DHQK,
                      p.DHHV, p.DHHV};

  for (int j = tid; j < L; j += NTHR) {
    s_b[j] = p.vecB[tok0 + j];
    s_iota[j] = p.iota[tok0 + j];
    s_m[j] = p.m_tok[tok0 + j];
  }
  // inter-chunk term first: scaled by row, it is what the intra-chunk products are added onto
  Acc acc;
  acc.zero();
  float qn[4], rowsum[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) { qn[a] = 0.f; rowsum[a] = 0.f; }
  const float* nsrc = (FW && p.n_states) ? p.n_states + slab * p.DHQK : nullptr;
  if (FW && nsrc != nullptr)
    for (int k = tid; k < (DI + KSL - 1) / KSL * KSL; k += NTHR) s_n[k] = k < DI ? nsrc[k] : 0.f;   // (a barrier follows in the product)
  auto dot_n = [&](const float* As, int k0) {
    if (!FW || nsrc == nullptr) return;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int k = 2 * tx + u;
      const float n = s_n[k0 + k];
#pragma unroll
      for (int a = 0; a < 4; ++a) qn[a] = fmaf(As[swz(k, 4 * ty + a)], n, qn[a]);
    }
  };
  if (QK) tile_product<VEC, true, false>(acc, U, r0, St, o0, DI, buf, tid, dot_n);
  else tile_product<VEC, true, true>(acc, U, r0, St, o0, DI, buf, tid, NoEach());
  float rs[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = r0 + 4 * ty + a;
    rs[a] = r < L ? (LOWER ? p.qk_scale * p.bbar[tok0 + r] : p.abar[tok0 + r]) : 0.f;
  }
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      float lo, hi;
      unf2(acc.v[a][b], lo, hi);
      acc.v[a][b] = f2(lo * rs[2 * a], hi * rs[2 * a + 1]);
    }

  const float* blocks = QK ? p.qk_blocks : p.vh_blocks;
  const int nblk = (L + TILE - 1) / TILE;
  const int cb_lo = LOWER ? 0 : rb, cb_hi = LOWER ? rb : nblk - 1;
  for (int cb = cb_lo; cb <= cb_hi; ++cb) {
    const int c0 = cb * TILE;
    __syncthreads();   // the slices and the gated block of the previous round have been read
    Slice<T, false, VEC> x0, x1;
    if (blocks != nullptr) {
      const Mat<float> P{blocks + ((size_t)bc * score_pairs(L) + (LOWER ? score_pair(rb, cb) : score_pair(cb, rb))) * TILE * TILE, nullptr,
                         TILE, TILE, TILE};
      x0.fetch(X, o0, c0, tid);
      x1.fetch(X, o0, c0 + KSL, tid);
      if (LOWER) {   // [i][j] -> [c = j][r = i]
        Slice<float, true, true> p0, p1;
        p0.fetch(P, 0, 0, tid);
        p1.fetch(P, 0, KSL, tid);
        p0.put(Ps, tid);
        p1.put(Ps + SLICE, tid);
      } else {       // [i][j] = [c][r]
        Slice<float, false, true> p0, p1;
        p0.fetch(P, 0, 0, tid);
        p1.fetch(P, 0, KSL, tid);
        p0.put(Ps, tid);
        p1.put(Ps + SLICE, tid);
      }
      x0.put(buf, tid);
      x1.put(buf + SLICE, tid);
      __syncthreads();
      if (FW) {
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const float4 v = *reinterpret_cast<const float4*>(Ps + swz(4 * tx + b, 4 * ty));
          rowsum[0] += v.x; rowsum[1] += v.y; rowsum[2] += v.z; rowsum[3] += v.w;
        }
      }
#pragma unroll 1
      for (int u = 0; u < 2; ++u) mma_slice(acc, Ps + u * SLICE, buf + u * SLICE, ty, tx);
      continue;
    }
    Acc pr;
    pr.zero();
    tile_product<VEC, true, true>(pr, U, r0, W, c0, DI, buf, tid, NoEach());
    float s[4][4];
    pr.get(s);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int r = r0 + 4 * ty + a, c = c0 + 4 * tx + b;
        const bool valid = (r < L) && (c < L) && (LOWER ? (c <= r) : (c >= r));
        float val = 0.f;
        if (valid) {
          const int ii = LOWER ? r : c, jj = LOWER ? c : r;
          val = gate_score(s[a][b], p.qk_scale, s_b[ii], s_b[jj], s_iota[jj], s_m[ii]);
        }
        s[a][b] = val;
        if (FW) rowsum[a] += val;
      }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      *reinterpret_cast<float4*>(Ps + swz(4 * tx + b, 4 * ty)) = make_float4(s[0][b], s[1][b], s[2][b], s[3][b]);
    }
    x0.fetch(X, o0, c0, tid);
    x1.fetch(X, o0, c0 + KSL, tid);
    __syncthreads();   // every thread has left the score product: its slices are free
    x0.put(buf, tid);
    x1.put(buf + SLICE, tid);
    __syncthreads();
#pragma unroll 1
    for (int u = 0; u < 2; ++u) mma_slice(acc, Ps + u * SLICE, buf + u * SLICE, ty, tx);
  }

  float out[4][4];
  acc.get(out);
  T* dst = FW ? p.out_h : mode == PAR_DV ? p.out_dv : mode == PAR_DK ? p.out_dk : p.out_dq;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = r0 + 4 * ty + a;
    if (FW) {
      rowsum[a] = sum_columns(rowsum[a]);
      qn[a] = sum_columns(qn[a]);
    }
    if (r >= L) continue;
    const size_t t = tok0 + r;
    if (FW) {
      const float nn = rowsum[a] + rs[a] * qn[a];
      float den = 1.f;
      if (p.variant == MLSTM_EXP) den = fmaxf(fabsf(nn), expf(-s_m[r]));
      else if (p.variant == MLSTM_SIG) den = fmaxf(fabsf(nn), 1.f);
      const bool norm = p.variant != MLSTM_SIG_NONORM;
      if (ot == 0 && tx == 0) {
        if (p.n_out) p.n_out[t] = den;
        if (p.inv_den_out) p.inv_den_out[t] = norm ? 1.f / (den + p.eps) : 1.f;
      }
      if (norm) {
#pragma unroll
        for (int b = 0; b < 4; ++b) out[a][b] = out[a][b] / (den + p.eps);
      }
    }
    store4(dst + t * DO, o0 + 4 * tx, DO, VEC, make_float4(out[a][0], out[a][1], out[a][2], out[a][3]));
  }
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(NTHR, 3) par_fw_kernel(ParArgs<T> p) {
  extern __shared__ __align__(16) float smem[];
  pdl_wait();
  const int n_ot = (p.DHHV + TILE - 1) / TILE, n_rb = (p.L + TILE - 1) / TILE, y = blockIdx.x / n_ot;
  par_tile<T, true, VEC>(p, PAR_H, blockIdx.x % n_ot, y / n_rb, y % n_rb, smem);
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(NTHR, 3) par_bw_kernel(ParArgs<T> p) {
  extern __shared__ __align__(16) float smem[];
  pdl_wait();
  const int n_v = (p.DHHV + TILE - 1) / TILE, n_k = (p.DHQK + TILE - 1) / TILE;
  const int n = n_v + 2 * n_k, n_rb = (p.L + TILE - 1) / TILE, x = blockIdx.x % n, y = blockIdx.x / n;
  // the modes with the longer contraction first
  const int mode = x < n_k ? PAR_DK : x < 2 * n_k ? PAR_DQ : PAR_DV;
  par_tile<T, false, VEC>(p, mode, x < n_k ? x : x < 2 * n_k ? x - n_k : x - 2 * n_k, y / n_rb, y % n_rb, smem);
}

static size_t par_smem_bytes(int L, int DHQK) {
  return sizeof(float) * ((size_t)4 * SLICE + TILE * TILE + 3 * L + ceil_div(DHQK, KSL) * KSL);
}

// ---- launchers ----------------------------------------------------------------------------------------
static bool vec_dims(const ChunkwiseDims& d) { return d.DHQK % 4 == 0 && d.DHHV % 4 == 0; }

// The chunks' contributions of one or two recurrences and the score blocks wanted, then the scans over the chunks.
template <typename T>
static int parts_t(PartArgs<T> a, int n_rec, const ChunkwiseDims& d, cudaStream_t st) {
  PhaseScope ps(a.bwd[n_rec - 1] ? PH_REC_BW : PH_REC_FW, st);
  const unsigned bnc = (unsigned)(d.B * d.NH) * (unsigned)d.NC;
  const unsigned tiles = (unsigned)ceil_div(d.DHHV, TILE) * ceil_div(d.DHQK, TILE) * bnc, pairs = (unsigned)score_pairs(d.L) * bnc;
  a.end[0] = a.sc[0].out ? pairs : 0;
  a.end[1] = a.end[0] + (a.sc[1].out ? pairs : 0);
  a.end[2] = a.end[1] + tiles;
  a.end[3] = a.end[2] + (n_rec > 1 ? tiles : 0);
  const bool vec = vec_dims(d);
  auto part = a.end[1] > 0 ? (vec ? part_kernel<T, true, true> : part_kernel<T, false, true>) : (vec ? part_kernel<T, true, false> : part_kernel<T, false, false>);
  if (int rc = launch_pdl(a.end[3] <= pdl_max_ctas(), part, a.end[3], NTHR, 0, st, a)) return rc;
  const size_t E = (size_t)d.DHQK * d.DHHV;
  const int V = E % 4 == 0 ? 4 : 1;
  ScanArgs scan[2] = {};   // forward, backward
  unsigned n[2] = {0, 0};
  const float* gbar = a.rec[0].gbar;
  for (int i = 0; i < n_rec; ++i) {
    const RecArgs<T>& r = a.rec[i];
    const int nblk = (int)((E / V + (!a.bwd[i] && r.n_states ? d.DHQK : 0) + 127) / 128);
    scan[a.bwd[i]] = ScanArgs{r.c_states, r.c_init, r.c_final, r.n_states, r.n_init, r.n_final, nblk};
    n[a.bwd[i]] = (unsigned)nblk * (unsigned)(d.B * d.NH);
  }
  const unsigned grid = n[0] + n[1];
  auto kern = n[1] == 0   ? (V == 4 ? rec_scan_kernel<4, true, false> : rec_scan_kernel<1, true, false>)
              : n[0] == 0 ? (V == 4 ? rec_scan_kernel<4, false, true> : rec_scan_kernel<1, false, true>)
                          : (V == 4 ? rec_scan_kernel<4, true, true> : rec_scan_kernel<1, true, true>);
  return launch_pdl(grid <= pdl_max_ctas(), kern, grid, 128, 0, st, scan[0], scan[1], n[0], gbar, d.NC, d.DHQK, d.DHHV);
}

template <typename T, bool BWD>
static int rec_final_t(const RecArgs<T>& a, const ChunkwiseDims& d, cudaStream_t st) {
  PhaseScope ps(BWD ? PH_REC_BW : PH_REC_FW, st);
  const unsigned tiles = (unsigned)ceil_div(d.DHHV, TILE) * ceil_div(d.DHQK, TILE) * (unsigned)(d.B * d.NH);
  if (vec_dims(d)) rec_final_kernel<T, BWD, true><<<tiles, NTHR, 0, st>>>(a);
  else rec_final_kernel<T, BWD, false><<<tiles, NTHR, 0, st>>>(a);
  MLSTM_LAUNCH_CHECK();
  return MLSTM_OK;
}

template <typename T>
static int par_t(ParArgs<T>& a, bool backward, const ChunkwiseDims& d, cudaStream_t st) {
  PhaseScope ps(backward ? PH_PAR_BW : PH_PAR_FW, st);
  const size_t smem = par_smem_bytes(d.L, d.DHQK);
  const int n_v = ceil_div(d.DHHV, TILE), n_k = ceil_div(d.DHQK, TILE);
  const unsigned grid = (unsigned)(backward ? n_v + 2 * n_k : n_v) * (unsigned)(d.B * d.NH * d.NC) * (unsigned)ceil_div(d.L, TILE);
  auto kern = vec_dims(d) ? (backward ? par_bw_kernel<T, true> : par_fw_kernel<T, true>)
                          : (backward ? par_bw_kernel<T, false> : par_fw_kernel<T, false>);
  MLSTM_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  return launch_pdl(grid <= pdl_max_ctas(), kern, grid, NTHR, smem, st, a);
}

template <typename T>
static ParArgs<T> par_args(const void* q, const void* k, const void* v, const GateBuffers& gb, const void* c_states,
                           const ChunkwiseDims& d) {
  ParArgs<T> a{};
  a.q = (const T*)q; a.k = (const T*)k; a.v = (const T*)v; a.dh = (const T*)v;
  a.vecB = gb.vecB; a.iota = gb.iota; a.m_tok = gb.m_tok; a.abar = gb.abar; a.bbar = gb.bbar; a.inv_den = gb.inv_den;
  a.c_states = (const float*)c_states;
  a.S = d.S; a.L = d.L; a.NC = d.NC; a.DHQK = d.DHQK; a.DHHV = d.DHHV; a.variant = d.variant;
  a.eps = d.eps; a.qk_scale = d.qk_scale;
  return a;
}

#define MLSTM_DISPATCH(dtype, ...)                                          \
  switch (dtype) {                                                          \
    case MLSTM_F32: { using T = float; __VA_ARGS__ }                        \
    case MLSTM_BF16: { using T = __nv_bfloat16; __VA_ARGS__ }               \
    case MLSTM_F16: { using T = __half; __VA_ARGS__ }                       \
  }                                                                         \
  return MLSTM_ERR_DTYPE;

// Scratch for the score blocks of a forward (one product) or a backward (two); 0 where they are not used.  A chunk of 64 or 128
// tokens has one or three blocks of 16 KB, used by every output tile of it.  Shorter chunks would mostly store padding.  Longer
// ones and small head dims would need more room than what the call has for states anyway: one set of blocks beside the
// forward's states, two beside the backward's states and state gradients.
size_t simt_score_bytes(const ChunkwiseDims& d, bool backward) {
  if ((d.L != TILE && d.L != 2 * TILE) || d.DHQK * d.DHHV < score_pairs(d.L) * TILE * TILE) return 0;
  return (size_t)(backward ? 2 : 1) * d.B * d.NH * d.NC * score_pairs(d.L) * TILE * TILE * sizeof(float);
}

static ScoreGate score_gate(const GateBuffers& gb, const ChunkwiseDims& d) {
  return ScoreGate{gb.vecB, gb.iota, gb.m_tok, d.S, d.L, d.NC, d.qk_scale};
}

int simt_recurrent_fw(int dtype, const void* q, const void* k, const void* v, const GateBuffers& gb, const float* c_initial,
                      const float* n_initial, void* c_states, float* n_states, float* c_last, float* n_last, float* scores,
                      const ChunkwiseDims& d, cudaStream_t st) {
  MLSTM_DISPATCH(dtype, {
    const RecArgs<T> r{(const T*)k, (const T*)v, gb.abar, nullptr, gb.gbar, 1.f, c_initial, n_initial,
                       (float*)c_states, n_states, c_last, n_last, d.S, d.L, d.NC, d.DHQK, d.DHHV};
    if (c_states == nullptr) return rec_final_t<T, false>(r, d, st);
    PartArgs<T> a{};
    a.rec[0] = r;
    a.gate = score_gate(gb, d);
    a.sc[0] = ScoreArgs<T>{(const T*)q, (const T*)k, nullptr, scores, d.DHQK};
    return parts_t<T>(a, 1, d, st);
  })
}
int simt_parallel_fw(int dtype, const void* q, const void* k, const void* v, const GateBuffers& gb, const void* c_states,
                     const float* n_states, void* h, float* n_out, const float* scores, const ChunkwiseDims& d, cudaStream_t st) {
  MLSTM_DISPATCH(dtype, {
    auto a = par_args<T>(q, k, v, gb, c_states, d);
    a.n_states = n_states; a.out_h = (T*)h; a.n_out = n_out; a.inv_den_out = gb.inv_den; a.qk_blocks = scores;
    return par_t<T>(a, false, d, st);
  })
}
int simt_recurrent_bw(int dtype, const void* q, const void* k, const void* v, const void* dh, const GateBuffers& gb, const float* dc_last,
                      void* dc_states, float* dc_initial, const float* c_initial, void* c_states, float* scores,
                      const ChunkwiseDims& d, cudaStream_t st) {
  MLSTM_DISPATCH(dtype, {
    const RecArgs<T> r{(const T*)q, (const T*)dh, gb.bbar, gb.inv_den, gb.gbar, d.qk_scale, dc_last, nullptr,
                       (float*)dc_states, nullptr, dc_initial, nullptr, d.S, d.L, d.NC, d.DHQK, d.DHHV};
    if (dc_states == nullptr) return rec_final_t<T, true>(r, d, st);
    PartArgs<T> a{};
    int n = 0;
    if (c_states != nullptr)   // the forward's states again
      a.rec[n++] = RecArgs<T>{(const T*)k, (const T*)v, gb.abar, nullptr, gb.gbar, 1.f, c_initial, nullptr, (float*)c_states, nullptr, nullptr, nullptr,
                              d.S, d.L, d.NC, d.DHQK, d.DHHV};
    a.bwd[n] = true;
    a.rec[n++] = r;
    a.gate = score_gate(gb, d);
    if (scores != nullptr) {
      a.sc[0] = ScoreArgs<T>{(const T*)dh, (const T*)v, gb.inv_den, scores + simt_score_bytes(d, false) / sizeof(float), d.DHHV};
      a.sc[1] = ScoreArgs<T>{(const T*)q, (const T*)k, nullptr, scores, d.DHQK};
    }
    return parts_t<T>(a, n, d, st);
  })
}
int simt_parallel_bw(int dtype, const void* q, const void* k, const void* v, const void* dh, const GateBuffers& gb,
                     const void* c_states, const void* dc_states, void* dq, void* dk, void* dv, const float* scores,
                     const ChunkwiseDims& d, cudaStream_t st) {
  MLSTM_DISPATCH(dtype, {
    auto a = par_args<T>(q, k, v, gb, c_states, d);
    a.dh = (const T*)dh; a.dc_states = (const float*)dc_states;
    a.out_dq = (T*)dq; a.out_dk = (T*)dk; a.out_dv = (T*)dv;
    if (scores != nullptr) { a.qk_blocks = scores; a.vh_blocks = scores + simt_score_bytes(d, false) / sizeof(float); }
    return par_t<T>(a, true, d, st);
  })
}

}  // namespace mlstm
