// tcgen05 / TMEM / TMA implementation of the chunkwise mLSTM kernels for B200 (sm_100a).
// bf16 or f16 operands, f32 accumulation in tensor memory, chunk size 128, head dims multiples of 8 (tiles of 128: a tile
// hanging over the edge of a head dim is zero-padded by TMA on the way in, masked or clipped on the way out).
//
//   rec_sm100<BWD>   inter-chunk recurrence (forward C_k, n_k; backward deltaC_k).  A CTA owns a 128 x 128 tile
//                    of the state for one (batch, head) and walks the chunks in order; per chunk one
//                    (gated left)^T x right contraction on the tensor cores into a double-buffered TMEM
//                    accumulator, decay + accumulate of the running state in registers, bf16 state store.
//                    mlstm_kernels/triton/chunkwise/xl_chunk/fw_kernel_recurrent.py:14-230, bw_kernel_recurrent.py:15-181
//   par_body         intra-chunk kernel of the forward (par_fw_sm100, par_fw_range_sm100).  Per (batch, head, chunk, 128-wide output tile):
//                    score = A B^T (TMEM) -> gate matrix applied by the CUDA cores, bf16 result written back to
//                    TMEM and used as the A operand of score x X; the inter-chunk term A x state is accumulated
//                    into the same TMEM tile first and row-scaled in place.  The L x L gate matrix never
//                    leaves the SM.
//                    fw_kernel_parallel.py:14-289
// Operands arrive by TMA (128-byte swizzle, no multicast) through mbarrier rings (half-chunk stages in the recurrence, three stages in the intra-chunk kernel); one warp produces,
// one thread issues the MMAs, the remaining warps do the element-wise work.  Every wait is bounded
// and a lane whose wait has run out keeps its warp company to the end of the role, without arriving anywhere: see warp_arrive.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "launch.cuh"
#include "segments.h"
#include "sm100.cuh"
#include "tensor_maps.cuh"

namespace mlstm {

using namespace sm100;

__device__ int g_sm100_status = 0;  // first error code raised by a bounded wait (0 = none)

constexpr int CL = 128;  // chunk length handled by these kernels

// =====================================================================================================
// Inter-chunk recurrence
// =====================================================================================================
struct RecParams {
  const float* lscale;  // per token: abar (fw) or bbar (bw)
  const float* rscale;  // per token: nullptr (fw) or 1/(den+eps) (bw)
  float lmul;           // 1 (fw) or qk_scale (bw)
  const float* gbar;    // (BNH, NC)
  const float* c_init;  // (BNH, DHQK, DHHV) f32 or nullptr
  const float* n_init;  // (BNH, DHQK) or nullptr
  void* c_states;           // (BNH, NC+1, DHQK, DHHV), 16-bit elements of the input type
  float* n_states;          // (BNH, NC+1, DHQK) or nullptr
  float* c_final;           // (BNH, DHQK, DHHV) f32 or nullptr
  float* n_final;
  int S, SP, NC, DHQK, DHHV;   // SP = NC * 128: slots per (batch, head) of the per-token scale vectors
  int bh0;                     // first (batch, head) unit of this launch (a launch may cover a sub-range of the units)
  int ck0, n_ck;               // forward: first chunk and number of chunks of this launch (backward: all of them)
};

constexpr int REC_THREADS = 640;                 // warp 0 TMA (left), 1 MMA, 2..9 gate the left tile, 10..17 own the state, 18 stores it and keeps n, 19 TMA (right)
constexpr int REC_HALF = 64;                     // tokens per ring stage: half a chunk
constexpr int REC_NPART_BYTES = 2 * 2 * 128 * 4; // column sums of the gated left tile, per half chunk, double-buffered
constexpr int REC_LBUF = 8;                      // gated left tiles in tensor memory, 32 columns each
constexpr int rec_right_bytes(int TN) { return TN * 128; }            // 64 tokens of the right operand (16 KB of the left one)
constexpr int rec_out_bytes(int TN) { return TN * 256; }              // 16-bit state tile staged for the TMA store (two of them)
// Depths of the two operand rings: a stage of the left operand goes back as soon as it has been gated, one of the right when
// the product that reads it is done.  The left ring's depth is even, so that a stage always goes to the same group of gating
// warps: a wait sees the parity of a phase only, and in an odd ring a group would come back to a stage two phases later, where
// the load before the other group's last one passes for its own.  With 64-column tiles the right operand is small: both travel as
// one stage, which saves the MMA thread a wait per half chunk (128 CTAs of 8 heads 256/512, 131072 tokens: 1096 us with two
// rings, 973 with one; with 128-column tiles, 8 x 8192 tokens, 16 heads 256/256: 373 and 390).
constexpr int rec_stages(int TN) { return TN == 128 ? 4 : 6; }
constexpr int rec_right_stages(int TN) { return TN == 128 ? 5 : 6; }
constexpr int rec_npart_offset(int TN) { return rec_stages(TN) * 16384 + rec_right_stages(TN) * rec_right_bytes(TN); }
constexpr int rec_smem_bytes(bool has_n, int TN) { return rec_npart_offset(TN) + (has_n ? REC_NPART_BYTES : 0) + 2 * rec_out_bytes(TN) + 1024; }

// A stage holds 64 tokens of one operand (boxes of 64 rows x 64 columns, 8 KB each: left columns d0.., d0+64.., right
// columns e0.., e0+64..).  A chunk is two stages of either; the product of a chunk is accumulated over both before the state
// warps fold it in.
// TN = columns of the state tile (128, or 64 for small problems: twice as many CTAs, so that a launch with few
// (batch, head) units still covers the GPU).
// F16: the 16-bit element type is IEEE half instead of bf16 (operands, gated tiles, stored states, outputs).
// HAS_N: the vector n is kept as well (forward, unless only the states are wanted again).
template <bool BWD, int TN, bool F16, bool HAS_N>
__device__ __forceinline__ void
rec_body(const CUtensorMap& mapL, const CUtensorMap& mapR, const CUtensorMap& mapS, const RecParams& p, const unsigned block) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int REC_STAGES = rec_stages(TN), RIGHT_STAGES = rec_right_stages(TN), RIGHT_BYTES = rec_right_bytes(TN), REC_OUT = rec_out_bytes(TN);
  uint8_t* smem_r = smem + REC_STAGES * 16384;
  constexpr int G_RING = 16;
  constexpr bool JOINT = TN == 64;   // one ring: a stage holds both operands and is free when its product is done
  static_assert(!JOINT || RIGHT_STAGES == REC_STAGES, "one ring");
  // (separate arrays: members of one shared struct cost 68 bytes of register spills in the 128-column forward)
  __shared__ uint64_t bar_full[REC_STAGES], bar_empty[REC_STAGES], bar_rfull[RIGHT_STAGES],
      bar_scaled[REC_LBUF], bar_done[REC_LBUF], bar_acc_free[2], bar_nsum[2],
      bar_nread[2], bar_out_full[2], bar_out_free[2];
  // Decay of the chunk.  The thread that writes it is at most STAGES / 2 + REC_LBUF / 2 + 3 <= 10 chunks ahead of its last reader: ring of 16.
  __shared__ float s_g[G_RING];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;   // set by the first wait of this CTA that runs out; every other wait polls it
  // per-row scale factors of the left tile, copied with the stage (backward: two factors per row)
  __shared__ __align__(16) float s_scale[REC_STAGES][REC_HALF], s_scale2[BWD ? REC_STAGES : 1][REC_HALF];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // 1-D grid (no 65535 limit on batch x heads), state tiles of one (batch, head) next to each other
  static_assert(TN == 128 || TN == 64, "state tile width");
  static_assert(REC_STAGES % 2 == 0, "the gating groups take the half chunks in turn: a stage must always meet the same group");
  constexpr int HC = TN / 2;   // columns each of the two state-warp groups owns
  // head dims need not be multiples of the tile: the last tile hangs over the edge, where loads read zeros (the
  // tensor maps know the true extents), plain accesses are masked and the state store is clipped
  const int n_et = (p.DHHV + TN - 1) / TN, n_dt = (p.DHQK + 127) / 128;
  const int et = block % n_et, dt = (block / n_et) % n_dt, bh = p.bh0 + block / (n_et * n_dt);
  const int e0 = et * TN, d0 = dt * 128;
  const int NC = p.NC, NS = p.n_ck, NH2 = 2 * NS;   // ring steps: two per chunk
  const int ck0 = BWD ? 0 : p.ck0;
  const bool do_n = HAS_N && et == 0 && (p.n_states != nullptr || p.n_final != nullptr);

  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < REC_STAGES; ++s) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 4); }   // (arrivals once per warp)
    for (int s = 0; s < RIGHT_STAGES; ++s) mbar_init(&bar_rfull[s], 1);
    for (int s = 0; s < REC_LBUF; ++s) { mbar_init(&bar_scaled[s], 4); mbar_init(&bar_done[s], 1); }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar_acc_free[s], 8); mbar_init(&bar_nsum[s], 8); mbar_init(&bar_nread[s], 1);
      mbar_init(&bar_out_full[s], 8); mbar_init(&bar_out_free[s], 1);
    }
    fence_barrier_init();
    tma_prefetch_desc(&mapL); tma_prefetch_desc(&mapR); tma_prefetch_desc(&mapS);
  }
  if (warp == 1) { tmem_alloc(&s_tmem, 512); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  // two accumulators of 128 columns, then the gated left tiles (64 tokens, 32 columns each)
  const uint32_t tmem = s_tmem, tL = tmem + 256;
  pdl_launch_dependents();
  pdl_wait();

  if (warp == 0) {
    // ---------------- TMA producer of the left operand ----------------
    // The per-row scale vectors travel with the stage (bulk copies on the same barrier).  Stage, phase and addresses are carried
    // along: the thread issues four copies per stage, and what it computes in between is in every stage's way.
    int issued = 0;   // by the issuing lane
    if (elect_one()) {
      int st = 0;
      uint32_t ph = 1;
      bool ok = true;
      int y = (BWD ? NC - 1 : ck0) * CL;                    // first token of the half chunk inside the sequence
      const float* gbar = p.gbar + (size_t)bh * NC + (BWD ? NC - 1 : ck0);
      float g = gbar[0];                                    // asked for a chunk ahead
      const float *ls = p.lscale + (size_t)bh * p.SP, *rs = BWD ? p.rscale + (size_t)bh * p.SP : nullptr;
      for (int h = 0; h < NH2; ++h) {
        if (JOINT) ok = ok && (h < REC_STAGES || mbar_wait(&bar_done[(h - REC_STAGES) & (REC_LBUF - 1)], ((h - REC_STAGES) / REC_LBUF) & 1, &s_abort, &g_sm100_status, 113));
        else ok = ok && mbar_wait(&bar_empty[st], ph, &s_abort, &g_sm100_status, 101);
        if ((h & 1) == 0) {   // (the arrival below releases it to the gating warps, theirs to the MMA thread, and its to the readers)
          const int s = h >> 1;
          s_g[s & (G_RING - 1)] = g;
          if (s + 1 < NS) g = gbar[BWD ? -(s + 1) : s + 1];
        }
        if (ok) {
          // token rows past the end of the sequence (ragged last chunk) arrive as zeros; their scale slots hold zeros
          uint8_t* sl = smem + st * 16384;
          mbar_expect_tx(&bar_full[st], 16384 + (JOINT ? RIGHT_BYTES : 0) + (BWD ? 2 : 1) * REC_HALF * 4);
          bulk_load(s_scale[st], ls + y, REC_HALF * 4, &bar_full[st]);
          if (BWD) bulk_load(s_scale2[st], rs + y, REC_HALF * 4, &bar_full[st]);
          tma_load_3d(sl, &mapL, &bar_full[st], d0, y, bh);
          tma_load_3d(sl + 8192, &mapL, &bar_full[st], d0 + 64, y, bh);
          if (JOINT) tma_load_3d(smem_r + st * RIGHT_BYTES, &mapR, &bar_full[st], e0, y, bh);
          issued = h + 1;
        }
        y += (BWD && (h & 1)) ? -CL - REC_HALF : REC_HALF;
        if (++st == REC_STAGES) { st = 0; ph ^= 1; }
      }
    }
    // the copies in flight land before the CTA retires, whichever role may have given up (the other lanes have issued none)
    for (int h = max(0, issued - REC_STAGES); h < issued; ++h)
      mbar_wait(&bar_full[h % REC_STAGES], (h / REC_STAGES) & 1, nullptr, nullptr, 0);
  } else if (warp == 19) {
    // ---------------- TMA producer of the right operand, where it has a ring of its own ----------------
    int issued = 0;
    if (!JOINT && elect_one()) {
      int st = 0;
      bool ok = true;
      int y = (BWD ? NC - 1 : ck0) * CL;
      for (int h = 0; h < NH2; ++h) {
        // the product of RIGHT_STAGES half chunks ago is done
        const int hb = h - RIGHT_STAGES;
        ok = ok && (hb < 0 || mbar_wait(&bar_done[hb & (REC_LBUF - 1)], (hb / REC_LBUF) & 1, &s_abort, &g_sm100_status, 110));
        if (ok) {
          uint8_t* sr = smem_r + st * RIGHT_BYTES;
          mbar_expect_tx(&bar_rfull[st], RIGHT_BYTES);
          tma_load_3d(sr, &mapR, &bar_rfull[st], e0, y, bh);
          tma_load_3d(sr + 8192, &mapR, &bar_rfull[st], e0 + 64, y, bh);
          issued = h + 1;
        }
        y += (BWD && (h & 1)) ? -CL - REC_HALF : REC_HALF;
        if (++st == RIGHT_STAGES) st = 0;
      }
    }
    for (int h = max(0, issued - RIGHT_STAGES); h < issued; ++h)
      mbar_wait(&bar_rfull[h % RIGHT_STAGES], (h / RIGHT_STAGES) & 1, nullptr, nullptr, 0);
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_16(F16, 128, TN, 0, 1);
      constexpr uint32_t desc_hi = umma_desc_hi(1024);
      const uint32_t desc0 = umma_desc_lo(smem_u32(smem_r), 8192);
      int st = 0;
      uint32_t ph = 0, desc = desc0;
      bool ok = true;
      for (int s = 0; s < NS && ok; ++s) {
        const int buf = s & 1;
        if (!(ok = mbar_wait(&bar_acc_free[buf], ((s >> 1) & 1) ^ 1, &s_abort, &g_sm100_status, 103))) break;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const int lb = (2 * s + hf) & (REC_LBUF - 1);
          ok = ok && (JOINT || mbar_wait(&bar_rfull[st], ph, &s_abort, &g_sm100_status, 111));
          ok = ok && mbar_wait(&bar_scaled[lb], ((2 * s + hf) / REC_LBUF) & 1, &s_abort, &g_sm100_status, 102);
          tc_fence_after_sync();
          if (!ok) break;
#pragma unroll
          for (int kk = 0; kk < REC_HALF / 16; ++kk)
            umma_ts(tmem + buf * 128, tL + lb * 32 + kk * 8, umma_desc(desc + kk * (2048 >> 4), desc_hi), idesc, (hf > 0 || kk > 0) ? 1u : 0u);
          umma_commit(&bar_done[lb]);
          desc += RIGHT_BYTES >> 4;
          if (++st == RIGHT_STAGES) { st = 0; ph ^= 1; desc = desc0; }
        }
      }
    }
  } else if (warp < 10) {
    // ---------------- gating warps: left tile, scaled and transposed, into tensor memory; column sums give n ----------------
    // Two groups of four warps take the half chunks in turn: a stage costs hundreds of cycles of dependent work and of waits and
    // hand-over, which one group would pay for every stage.  A warp reads its 32 columns (state rows d) of all 64 tokens with
    // transposing loads, so that a lane holds pairs of tokens of one d, and writes them where the MMA reads its A operand: the
    // shared-memory port, the busiest unit of this kernel, carries the left tile once instead of three times (read, rewritten in
    // place, read by the MMA; 288 -> 192 KB per chunk and 128 x 128 tile), and no writes have to be made visible to the tensor
    // core's proxy.  All reads go out before the first is used, and the stage is handed back then.  Measured (first rewriting in
    // place, then this): 8 x 8192 tokens, 16 heads 256/256, 402 -> 374 us (HBM at 0.82 of the copy rate), gradient 397 -> 362;
    // 8 heads 256/512, 131072 tokens 1135 -> 964 (narrow tiles: the chain of one half chunk after the other through gating,
    // product and fold); 4 x 4 x 1024, 96/192 18.8 -> 16.5.
    const int grp = (warp - 2) >> 2, quarter = warp & 3;
    // tile m = lane / 8 of a transposing load: columns 8 m of the warp's 32; row lane % 8, 16-byte pieces XOR-swizzled by the row
    const uint32_t src0 = smem_u32(smem) + (quarter >> 1) * 8192 + (lane & 7) * 128 + ((((quarter & 1) * 4 + (lane >> 3)) ^ (lane & 7)) << 4);
    const int tok2 = 2 * (lane & 3);               // first of the lane's two tokens in every eight
    // (a lane whose wait has run out goes on with its warp, and does not arrive: see warp_arrive)
    for (int h = grp; h < NH2; h += 2) {
      const int st = h % REC_STAGES, lb = h & (REC_LBUF - 1), s = h >> 1, nb = s & 1;
      bool ok = mbar_wait(&bar_full[st], (h / REC_STAGES) & 1, &s_abort, &g_sm100_status, 105);
      uint32_t x[REC_HALF / 8][4];
      float2 sc[REC_HALF / 8], sc2[BWD ? REC_HALF / 8 : 1];
#pragma unroll
      for (int tb = 0; tb < REC_HALF / 8; ++tb) ldmatrix_x4_trans(src0 + st * 16384 + tb * 1024, x[tb]);
#pragma unroll
      for (int tb = 0; tb < REC_HALF / 8; ++tb) {
        sc[tb] = *reinterpret_cast<const float2*>(&s_scale[st][8 * tb + tok2]);
        if (BWD) sc2[tb] = *reinterpret_cast<const float2*>(&s_scale2[st][8 * tb + tok2]);
      }
      if (!JOINT) warp_arrive(&bar_empty[st], ok);
      uint32_t w[2][16];
      uint64_t ns[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
      for (int tb = 0; tb < REC_HALF / 8; ++tb) {
        uint64_t ss = mul2(f2(sc[tb].x, sc[tb].y), f2(p.lmul, p.lmul));
        if (BWD) ss = mul2(ss, f2(sc2[tb].x, sc2[tb].y));
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const uint64_t y = mul2(unpack2<F16>(x[tb][m]), ss);
          if (HAS_N) ns[m] = add2(ns[m], y);
          w[m >> 1][2 * tb + (m & 1)] = pack2<F16>(y);
        }
      }
      // the product that read this buffer last is done (with one ring it was before the stage could be loaded)
      const bool free_ok = JOINT || h < REC_LBUF || mbar_wait(&bar_done[lb], ((h / REC_LBUF) - 1) & 1, &s_abort, &g_sm100_status, 112);
      tc_fence_after_sync();
      const uint32_t dst = tL + lb * 32 + ((uint32_t)(quarter * 32) << 16);
      tmem_st_16x128b_x8(dst, w[0]);
      tmem_st_16x128b_x8(dst + (16u << 16), w[1]);
      tmem_wait_st();
      tc_fence_before_sync();
      ok = ok && free_ok;
      warp_arrive(&bar_scaled[lb], ok);
      if (do_n) {   // column sums of this half chunk: the four lanes of a d hold the sums over their tokens
        float v[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          float lo, hi;
          unf2(ns[m], lo, hi);
          v[m] = lo + hi;
          v[m] += __shfl_xor_sync(0xffffffffu, v[m], 1);
          v[m] += __shfl_xor_sync(0xffffffffu, v[m], 2);
        }
        // the n warp has read the sums of chunk s - 2 out of this buffer
        const bool nok = s < 2 || mbar_wait(&bar_nread[nb], ((s >> 1) - 1) & 1, &s_abort, &g_sm100_status, 109);
        float* npart = reinterpret_cast<float*>(smem + rec_npart_offset(TN)) + (nb * 2 + grp) * 128;
        const int m = lane & 3;
        npart[quarter * 32 + m * 8 + (lane >> 2)] = m == 0 ? v[0] : (m == 1 ? v[1] : (m == 2 ? v[2] : v[3]));
        warp_arrive(&bar_nsum[nb], ok && nok);   // (complete when both halves of chunk s are in)
      }
    }
  } else if (warp == 18) {
    // ---------------- store and n warp ----------------
    // Per chunk boundary one TMA store per 64-column box of the staged state tile; then n_{s+1} = gbar n_s + column sums of the
    // gated left tile (no tensor cores needed), four columns per lane.
    const bool store = p.c_states != nullptr;
    uint8_t* stage_base = smem + rec_npart_offset(TN) + (HAS_N ? REC_NPART_BYTES : 0);
    float4 nv = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool d_in = do_n && d0 + 4 * lane < p.DHQK;   // the lane's four rows exist (DHQK is a multiple of 8)
    if (p.n_init && d_in) nv = *reinterpret_cast<const float4*>(p.n_init + (size_t)bh * p.DHQK + d0 + 4 * lane);
    if (p.n_states != nullptr && d_in)
      *reinterpret_cast<float4*>(p.n_states + ((size_t)bh * (NC + 1) + ck0) * p.DHQK + d0 + 4 * lane) = nv;
    bool ok = true;
    for (int n = 0; n <= NS; ++n) {
      if (store) {
        const int ob = n & 1;
        ok = ok && mbar_wait(&bar_out_full[ob], (n >> 1) & 1, &s_abort, &g_sm100_status, 108);
        if (lane == 0 && ok) {
          const int z = bh * (NC + 1) + (BWD ? NC - n : ck0 + n);
          tma_store_3d(&mapS, stage_base + ob * REC_OUT, e0, d0, z);
          if (TN == 128 && e0 + 64 < p.DHHV) tma_store_3d(&mapS, stage_base + ob * REC_OUT + 16384, e0 + 64, d0, z);
          tma_store_commit();
          asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");   // the previous tile has left its buffer
          if (n >= 1) mbar_arrive(&bar_out_free[ob ^ 1]);
        }
      }
      if (!do_n || n == NS) continue;
      const int nb = n & 1;
      ok = ok && mbar_wait(&bar_nsum[nb], (n >> 1) & 1, &s_abort, &g_sm100_status, 106);
      const float4* np4 = reinterpret_cast<const float4*>(smem + rec_npart_offset(TN)) + nb * 64 + lane;
      float4 cs = np4[0];
      const float4 c1 = np4[32];
      cs.x += c1.x; cs.y += c1.y; cs.z += c1.z; cs.w += c1.w;
      const float g = s_g[n & (G_RING - 1)];
      __syncwarp();
      if (lane == 0 && ok) mbar_arrive(&bar_nread[nb]);
      nv.x = fmaf(g, nv.x, cs.x); nv.y = fmaf(g, nv.y, cs.y); nv.z = fmaf(g, nv.z, cs.z); nv.w = fmaf(g, nv.w, cs.w);
      if (p.n_states != nullptr && d_in)
        *reinterpret_cast<float4*>(p.n_states + ((size_t)bh * (NC + 1) + ck0 + n + 1) * p.DHQK + d0 + 4 * lane) = nv;
    }
    if (ok && p.n_final && d_in) *reinterpret_cast<float4*>(p.n_final + (size_t)bh * p.DHQK + d0 + 4 * lane) = nv;
    if (store && lane == 0) tma_store_wait_all();   // all state tiles have been written before the CTA retires
  } else {
    // ---------------- state warps: fold each chunk's product into the running state, store it ----------------
    const int quarter = warp & 3, half = (warp - 10) >> 2;
    const int row = quarter * 32 + lane;           // state row (d)
    const int d = d0 + row, ecol = e0 + half * HC;
    float C[HC];
    if (p.c_init) {
      const float4* src = reinterpret_cast<const float4*>(p.c_init + ((size_t)bh * p.DHQK + d) * p.DHHV + ecol);
#pragma unroll
      for (int c = 0; c < HC / 4; ++c) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (d < p.DHQK && ecol + 4 * c < p.DHHV) v = src[c];
        C[4 * c] = v.x; C[4 * c + 1] = v.y; C[4 * c + 2] = v.z; C[4 * c + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int c = 0; c < HC; ++c) C[c] = 0.f;
    }
    // The bf16 state tile goes to shared memory in the 128-byte-swizzled box layout and leaves with one TMA store
    // per 64-column box (coalesced, asynchronous); two staging buffers, one store group in flight.
    uint8_t* stage_base = smem + rec_npart_offset(TN) + (HAS_N ? REC_NPART_BYTES : 0);
    // (the answer of a wait counts for the arrival after it only: a flag held over the loop costs the 128-column forms
    // register spills, and the waits after one that ran out end by the abort flag)
    auto store_c = [&](const int n_out) {   // n_out: tiles written before this one
      if (p.c_states == nullptr) return;
      const int ob = n_out & 1;
      const bool ok = n_out < 2 || mbar_wait<true>(&bar_out_free[ob], ((n_out >> 1) - 1) & 1, &s_abort, &g_sm100_status, 107);
      // TN = 128: each group fills its own 64-column box; TN = 64: the groups share one box (four 16-byte pieces each)
      uint8_t* rowp = stage_base + ob * REC_OUT + (TN == 128 ? half * 16384 : 0) + row * 128;
      const int piece0 = (TN == 128) ? 0 : half * 4;
#pragma unroll
      for (int c = 0; c < HC / 8; ++c) {
        uint4 v;
        v.x = Pair16<F16>::pack(C[8 * c], C[8 * c + 1]); v.y = Pair16<F16>::pack(C[8 * c + 2], C[8 * c + 3]);
        v.z = Pair16<F16>::pack(C[8 * c + 4], C[8 * c + 5]); v.w = Pair16<F16>::pack(C[8 * c + 6], C[8 * c + 7]);
        *reinterpret_cast<uint4*>(rowp + (((piece0 + c) ^ (row & 7)) << 4)) = v;
      }
      fence_proxy_async_smem();
      warp_arrive(&bar_out_full[ob], ok);   // the store warp ships the tile
    };
    store_c(0);   // the state before the first step (slot 0 forward, slot NC backward)
    for (int s = 0; s < NS; ++s) {
      const int buf = s & 1;
      const bool ok = mbar_wait<true>(&bar_done[(2 * s + 1) & (REC_LBUF - 1)], ((2 * s + 1) / REC_LBUF) & 1, &s_abort, &g_sm100_status, 104);
      tc_fence_after_sync();
      const float g = s_g[s & (G_RING - 1)];
      const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + buf * 128 + half * HC;
#pragma unroll
      for (int q4 = 0; q4 < HC / 16; ++q4) {
        uint32_t rr[16];
        tmem_ld16(ta + q4 * 16, rr);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 16; ++c) C[q4 * 16 + c] = fmaf(g, C[q4 * 16 + c], __uint_as_float(rr[c]));
      }
      tc_fence_before_sync();
      warp_arrive(&bar_acc_free[buf], ok);
      store_c(s + 1);
    }
    if (p.c_final) {
      float4* fd = reinterpret_cast<float4*>(p.c_final + ((size_t)bh * p.DHQK + d) * p.DHHV + ecol);
#pragma unroll
      for (int c = 0; c < HC / 4; ++c)
        if (d < p.DHQK && ecol + 4 * c < p.DHHV) fd[c] = make_float4(C[4 * c], C[4 * c + 1], C[4 * c + 2], C[4 * c + 3]);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

template <bool BWD, int TN, bool F16>
__global__ void __launch_bounds__(REC_THREADS, 1)
rec_sm100(const __grid_constant__ CUtensorMap mapL, const __grid_constant__ CUtensorMap mapR,
          const __grid_constant__ CUtensorMap mapS, const __grid_constant__ RecParams p) {
  rec_body<BWD, TN, F16, !BWD>(mapL, mapR, mapS, p, blockIdx.x);
}

// Both recurrences of a backward that finds no per-chunk states in one launch: the first n_fw CTAs run the forward's
// again (states only), the others the state gradient's.  They are independent, and a launch of few CTAs takes as long as one
// of them takes for its sequence: side by side they take half.
template <int TN, bool F16>
__global__ void __launch_bounds__(REC_THREADS, 1)
rec_pair_sm100(const __grid_constant__ CUtensorMap mL, const __grid_constant__ CUtensorMap mR,
               const __grid_constant__ CUtensorMap mS, const __grid_constant__ RecParams p,
               const __grid_constant__ CUtensorMap mLb, const __grid_constant__ CUtensorMap mRb,
               const __grid_constant__ CUtensorMap mSb, const __grid_constant__ RecParams pb, const unsigned n_fw) {
  if (blockIdx.x < n_fw) rec_body<false, TN, F16, false>(mL, mR, mS, p, blockIdx.x);
  else rec_body<true, TN, F16, false>(mLb, mRb, mSb, pb, blockIdx.x - n_fw);
}

// =====================================================================================================
// Intra-chunk kernel.  Output tile rows r = tokens of one chunk, 128 output columns.
//   H[r,:] = (sum_{c <= r} G[r,c] V[c,:] + s * bbar_r * (Q[r,:] . C_k)) / (den_r + eps)
//   G[r,c] = gate(r,c) * (Q[r,:] . K[c,:]),   gate = s * exp((b_r - b_c) + iota_c - m_r)
// grid (ceil(DHHV / 128 / PAR_MAXSUB), NC, B*NH), two CTAs per SM; 320 threads: warp 0 TMA, warp 1 MMA, warps 2..9
// element-wise (two warps per 32-row quarter of the tile, each owning two 32-column chunks).  One CTA produces up to
// PAR_MAXSUB neighbouring output tiles of its chunk, one after the other, from a single score tile.
// Time line of a CTA's first tile (measured with time stamps at the benchmark size, two CTAs sharing an SM): first
// slices land after ~1.8 us, score complete ~3.3 us, gating until ~5 us with the inter-chunk product arriving
// underneath (~5.5 us), second product ~6.4 us, epilogue and stores until ~8.8 us; every further tile takes ~5.5 us.
// Within a tile the kernel is bound by this chain of dependent steps (the same kernel with every operand resident in
// L2 runs at the same speed); the forward kernel as a whole runs at the HBM copy bandwidth.
// =====================================================================================================
struct ParParams {
  const float *vecB, *iota, *m_tok, *bbar;   // per token, f32
  const float* n_states;
  uint16_t* out_h;            // 16-bit elements of the input type
  float* n_out;               // denominator per token, or nullptr
  float* inv_den_out;         // 1 / (denominator + eps) per slot (0 past the sequence end), or nullptr
  int S, SP, NC, DHQK, DHHV, variant;   // SP = NC * 128: slots per (batch, head) of the per-token gate vectors
  float eps, qk_scale;
  int bh0;                    // first (batch, head) unit of this launch
  int ck0, n_ck;              // first chunk and number of chunks of this launch
  int maxsub;                 // most output tiles a CTA of this launch produces (par_maxsub)
};

constexpr int PAR_THREADS = 320;  // warp 0 TMA, warp 1 MMA, warps 2..9 element-wise
constexpr int PAR_STAGE = 32768;  // two 16 KB boxes: (A, B) slice pair, (A, state) slice pair, or a 128 x 128 tile
constexpr int PAR_NST = 3;        // ring depth
constexpr int PAR_MAXSUB = 4;     // output tiles one CTA produces at most
constexpr int PAR_SMEM = PAR_NST * PAR_STAGE + 1024;

// Shared-memory control block of one intra-chunk CTA (the operand ring lives in dynamic shared memory).
struct ParShared {
  uint64_t bar_full[PAR_NST], bar_empty[PAR_NST], bar_qdone[PAR_NST], bar_sfull, bar_afull, bar_gated, bar_hfull, bar_accfree, bar_done[2],
      bar_pair[4], bar_out;
  uint32_t tmem;
  int issued;                      // loads the producer has issued
  int abort;                       // set by the first wait of this CTA that runs out; every other wait polls it
  __align__(16) float s_colE[CL];  // per-column term of the gate exponent, base 2 (see par_body)
  __align__(16) float s_colF[CL];  // 2^(colE_c - colP of the column's 32-column block)
  float s_colP[4];                 // largest colE of each 32-column block
  float s_part[2][CL];           // per-row partial sums exchanged between the two warps of a row
  float s_qn[2][CL];
  float s_n[512];
};

// Gate factor of element (r, c), c <= r: 2^(rowE_r + colE_c), every positive factor folded into the exponent:
//   rowE = (b_r - m_r) log2e + log2(s),   colE = (iota_c - b_c) log2e
// A 32 x 32 block off the diagonal is gated without a transcendental per element: with colP = the largest colE of
// the block's columns, 2^(rowE_r + colE_c) = 2^(rowE_r + colP) * 2^(colE_c - colP); the column factors (one ex2 per
// column and CTA) lie in (0, 1], and the row factor (one ex2 per row and block) cannot overflow because every
// element of an off-diagonal block is a valid gate entry, bounded by s.  Where a column factor
// underflows the exact value is below 2^-100 as well.  The diagonal block keeps the exact per-element form (its
// masked columns may carry arbitrarily large colE).  The special-function unit (16 results per clock and SM) was
// the limit of the gating phase before: the warps of the busiest row quarter share one SM sub-partition.
// LOOP: the CTA runs the body again for another chunk afterwards: it keeps its tensor memory from the first run
// to the last, and leaves each run with no arrival on any barrier outstanding, so that the next one can set them up anew.
// Returns false after a run in which a wait ran out: its copies may still be on their way to barriers of that run.
template <bool F16, bool LOOP = false>
__device__ __forceinline__ bool
par_body(const CUtensorMap* mapA, const CUtensorMap* mapB, const CUtensorMap* mapX, const CUtensorMap* mapSt, const ParParams& p,
         ParShared& sh, const int o_tile0, const int nsub, const int ck, const int bh, const bool first_run = true,
         const bool last_run = true) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int o00 = o_tile0 * 128;   // first output column of the CTA's first tile
  const int DO = p.DHHV;                      // output width
  const int NC = p.NC, ND = (p.DHQK + 63) / 64;   // slices of 64 columns; a last partial slice is padded with zeros by TMA
  const int y0 = ck * CL;                         // first token of the chunk inside its sequence
  const int valid = min(CL, p.S - y0);            // tokens of the chunk that exist (ragged last chunk: < 128)
  const size_t out_row0 = (size_t)bh * p.S + y0;  // first row of the chunk in the (B*NH*S)-row token tensors
  const bool use_n = p.variant != MLSTM_SIG_NONORM && p.n_states != nullptr;

  if (tid == 0) {
    if (LOOP && !first_run) {
      for (int s = 0; s < PAR_NST; ++s) { mbar_inval(&sh.bar_full[s]); mbar_inval(&sh.bar_empty[s]); mbar_inval(&sh.bar_qdone[s]); }
      for (int s = 0; s < 4; ++s) mbar_inval(&sh.bar_pair[s]);
      mbar_inval(&sh.bar_sfull); mbar_inval(&sh.bar_afull); mbar_inval(&sh.bar_gated); mbar_inval(&sh.bar_hfull);
      mbar_inval(&sh.bar_out); mbar_inval(&sh.bar_accfree); mbar_inval(&sh.bar_done[0]); mbar_inval(&sh.bar_done[1]);
    }
    sh.abort = 0; sh.issued = 0;
    for (int s = 0; s < PAR_NST; ++s) {
      mbar_init(&sh.bar_full[s], 1); mbar_init(&sh.bar_empty[s], 1); mbar_init(&sh.bar_qdone[s], 8);
    }
    mbar_init(&sh.bar_sfull, 1); mbar_init(&sh.bar_afull, 1); mbar_init(&sh.bar_gated, 256); mbar_init(&sh.bar_hfull, 1);
    for (int s = 0; s < 4; ++s) mbar_init(&sh.bar_pair[s], 64);
    mbar_init(&sh.bar_out, 256); mbar_init(&sh.bar_accfree, 256); mbar_init(&sh.bar_done[0], 256); mbar_init(&sh.bar_done[1], 256);
    fence_barrier_init();
    tma_prefetch_desc(mapA); tma_prefetch_desc(mapB); tma_prefetch_desc(mapX); tma_prefetch_desc(mapSt);
  }
  if (warp == 1 && (!LOOP || first_run)) { tmem_alloc(&sh.tmem, 256); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = sh.tmem;
  const uint32_t tS = tmem, tAcc = tmem + 128;
  pdl_launch_dependents();
  pdl_wait();
  // Ring loads, in order: ND (A, B) slice pairs for the score product, ND (A, state) slice pairs for the inter-chunk
  // product (A comes from L2 the second time), the X tile.  The score is complete - and the element-wise
  // warps start gating - while the second group is still arriving.
  // A CTA produces `nsub` (1 .. PAR_MAXSUB) neighbouring 128-column output tiles of the same chunk.  The
  // score tile and its gated form are the same for all of them, so every tile after the first only needs its own
  // state slices and X tile: the gated tile stays in tensor memory, the accumulator is reused once the previous
  // tile's epilogue has read it.
  const int n0 = 2 * ND + 1;          // loads of the first tile
  const int n1 = ND + 1;              // loads of every further tile
  const int n_loads = n0 + (nsub - 1) * n1;
  enum { LK_SCORE = 0, LK_STATE = 1, LK_X = 2 };
  // kind of the load at position l of tile `sub` (no divisions: this runs on the load-issue path)
  auto load_kind = [&](int sub, int l, int& it) -> int {
    if (sub == 0 && l < ND) { it = l; return LK_SCORE; }
    const int ls = l - (sub == 0 ? ND : 0);
    if (ls < ND) { it = ls; return LK_STATE; }
    it = 0;
    return LK_X;
  };

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (elect_one()) {
      const int sz = bh * (NC + 1) + ck;   // slab of the state tensor (one DHQK x DHHV matrix per chunk boundary)
      int issued = 0;
      // Per stage: uses handed back by an MMA commit so far (phase counter of bar_empty) and score pairs read for
      // q . n so far (phase counter of bar_qdone).  Scalars picked by comparisons, not arrays: a dynamically indexed
      // array would live in local memory, and with nearly all of L1 configured as shared memory every access to it
      // is a round trip to L2 on the load-issue path.
      int rm0 = 0, rm1 = 0, rm2 = 0, rq0 = 0, rq1 = 0, rq2 = 0;
      int st = 0, sub = 0, l = 0;                        // stage, tile and position inside the tile of load `ld`
      int pk1 = 0, pk2 = 0, pk3 = 0, ps1 = 0, ps2 = 0, ps3 = 0;   // kind and tile of the last three loads
      for (int ld = 0; ld < n_loads; ++ld) {
        int it;
        const int kind = load_kind(sub, l, it);
        if (ld >= PAR_NST) {   // the stage's previous occupant (three loads back) must be gone
          const int pkind = pk3, psub = ps3;
          bool okw;
          if (pkind == LK_SCORE || pkind == LK_STATE) {
            const int rm = st == 0 ? rm0 : (st == 1 ? rm1 : rm2);
            okw = mbar_wait(&sh.bar_empty[st], (rm - 1) & 1, &sh.abort, &g_sm100_status, 201);
            // the element-wise warps read the A box of a score pair (q . n)
            if (okw && use_n && pkind == LK_SCORE) {
              const int rq = st == 0 ? rq0 : (st == 1 ? rq1 : rq2);
              okw = mbar_wait(&sh.bar_qdone[st], (rq - 1) & 1, &sh.abort, &g_sm100_status, 212);
            }
          } else {
            // The staging buffer of a tile (its X stage) is handed back when the tile has been stored.  Two barriers, for every other tile: with one operand slice (DHQK <= 64) a tile's loads are two
            // and the ring holds three, so that the next tile, too, can be done before this wait looks.
            okw = mbar_wait(&sh.bar_done[psub & 1], (psub >> 1) & 1, &sh.abort, &g_sm100_status, 215);
          }
          if (!okw) break;
        }
        const int o0 = o00 + 128 * sub;
        uint8_t* sb = smem + st * PAR_STAGE;
        mbar_expect_tx(&sh.bar_full[st], PAR_STAGE);
        if (kind == LK_SCORE) {
          tma_load_3d(sb, mapA, &sh.bar_full[st], 64 * it, y0, bh);
          tma_load_3d(sb + 16384, mapB, &sh.bar_full[st], 64 * it, y0, bh);
        } else if (kind == LK_STATE) {
          tma_load_3d(sb, mapA, &sh.bar_full[st], 64 * it, y0, bh);
          tma_load_3d(sb + 16384, mapSt, &sh.bar_full[st], o0, 64 * it, sz);
          tma_load_3d(sb + 16384 + 8192, mapSt, &sh.bar_full[st], o0 + 64, 64 * it, sz);
        } else {
          tma_load_3d(sb, mapX, &sh.bar_full[st], o0, y0, bh);
          tma_load_3d(sb + 16384, mapX, &sh.bar_full[st], o0 + 64, y0, bh);
        }
        if (kind == LK_SCORE || kind == LK_STATE) { rm0 += (st == 0); rm1 += (st == 1); rm2 += (st == 2); }
        if (kind == LK_SCORE) { rq0 += (st == 0); rq1 += (st == 1); rq2 += (st == 2); }
        issued = ld + 1;
        pk3 = pk2; pk2 = pk1; pk1 = kind; ps3 = ps2; ps2 = ps1; ps1 = sub;
        st = st == PAR_NST - 1 ? 0 : st + 1;
        if (++l == (sub == 0 ? n0 : n1)) { l = 0; ++sub; }
      }
      sh.issued = issued;
      if (LOOP && issued == n_loads) {   // the hand-backs of the last uses, which nobody else waits for
        if (rm0 > 0) mbar_wait(&sh.bar_empty[0], (rm0 - 1) & 1, &sh.abort, &g_sm100_status, 217);
        if (rm1 > 0) mbar_wait(&sh.bar_empty[1], (rm1 - 1) & 1, &sh.abort, &g_sm100_status, 217);
        if (rm2 > 0) mbar_wait(&sh.bar_empty[2], (rm2 - 1) & 1, &sh.abort, &g_sm100_status, 217);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_16(F16, 128, 128, 0, 0);
      constexpr uint32_t idesc_x = umma_idesc_16(F16, 128, 128, 0, 1), hi = umma_desc_hi(1024);
      constexpr uint32_t lbo8 = (8192u >> 4) << 16, lbo16 = (16384u >> 4) << 16;   // (unused with K-major operands)
      const uint32_t base = smem_u32(smem) >> 4;
      bool ok = true;
      for (int ld = 0; ld < ND; ++ld) {            // score: S = A . B^T
        const int st = ld % PAR_NST;
        if (!mbar_wait(&sh.bar_full[st], (ld / PAR_NST) & 1, &sh.abort, &g_sm100_status, 202)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t sa = base + st * (PAR_STAGE >> 4), sb = sa + (16384 >> 4);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_ss(tS, umma_desc(sa + kk * (32 >> 4), hi), umma_desc(sb + kk * (32 >> 4), hi), idesc_s, (ld > 0 || kk > 0) ? 1u : 0u);
        umma_commit(&sh.bar_empty[st]);
      }
      if (ok) umma_commit(&sh.bar_sfull);
      for (int sub = 0; sub < nsub && ok; ++sub) {
        const int lbase = sub == 0 ? ND : n0 + (sub - 1) * n1;   // first state pair of this tile
        // the accumulator tile is free once the previous tile's epilogue has read it
        if (sub > 0 && !mbar_wait(&sh.bar_accfree, (sub - 1) & 1, &sh.abort, &g_sm100_status, 216)) { ok = false; break; }
        if (sub > 0) tc_fence_after_sync();
        for (int it = 0; it < ND; ++it) {           // inter-chunk term: Acc = A . State
          const int ld = lbase + it, st = ld % PAR_NST;
          if (!mbar_wait(&sh.bar_full[st], (ld / PAR_NST) & 1, &sh.abort, &g_sm100_status, 213)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t sa = base + st * (PAR_STAGE >> 4), ss = (sa + (16384 >> 4)) | lbo8;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_ss(tAcc, umma_desc(sa + kk * (32 >> 4), hi), umma_desc(ss + kk * (2048 >> 4), hi), idesc_x, (it > 0 || kk > 0) ? 1u : 0u);
          umma_commit(&sh.bar_empty[st]);
        }
        if (!ok) break;
        umma_commit(&sh.bar_afull);
        const int ldx = lbase + ND, stx = ldx % PAR_NST;
        ok = mbar_wait(&sh.bar_full[stx], (ldx / PAR_NST) & 1, &sh.abort, &g_sm100_status, 203) &&
             mbar_wait(&sh.bar_gated, sub & 1, &sh.abort, &g_sm100_status, 204);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t sx = (base + stx * (PAR_STAGE >> 4)) | lbo16;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma_ts(tAcc, tS + kk * 8, umma_desc(sx + kk * (2048 >> 4), hi), idesc_x, 1u);
        umma_commit(&sh.bar_hfull);
      }
    }
  } else {
    // ---------------- element-wise warps: two warps per 32-row quarter, each owning two 32-column chunks ----
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;
    const size_t tok = (size_t)bh * p.SP + y0 + r;   // slot of this row in the per-token gate vectors
    const float b_r = p.vecB[tok], iota_r = p.iota[tok], m_r = p.m_tok[tok];
    constexpr float kLog2e = 1.4426950408889634f;
    const float rowE = (b_r - m_r) * kLog2e + __log2f(p.qk_scale);
    if (half == 0) {   // this thread's row in its role as a column of the gate matrix
      const float colE = (iota_r - b_r) * kLog2e;
      float colP = colE;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) colP = fmaxf(colP, __shfl_xor_sync(0xffffffffu, colP, o));
      if (!(colP > -3.0e38f)) colP = 0.f;   // a block whose columns are all switched off
      sh.s_colE[r] = colE;
      sh.s_colF[r] = ex2_approx(colE - colP);
      if (lane == 0) sh.s_colP[quarter] = colP;
    }
    const float rowscale = p.qk_scale * p.bbar[tok];
    if (use_n) {
      const float* nsrc = p.n_states + ((size_t)bh * (NC + 1) + ck) * p.DHQK;
      for (int dd = tid - 64; dd < ND * 64; dd += 256) sh.s_n[dd] = dd < p.DHQK ? nsrc[dd] : 0.f;   // zero padding
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");  // gate vectors and n visible to the element-wise warps

    // q . n_{k-1} for the denominator: each thread reads half of its row of every Q slice from the
    // TMA stage (the stage is released to the producer only after these reads)
    float qn = 0.f;
    if (use_n) {
      for (int it = 0; it < ND; ++it) {
        const int st = it % PAR_NST;
        if (!mbar_wait(&sh.bar_full[st], (it / PAR_NST) & 1, &sh.abort, &g_sm100_status, 207)) {
          for (; it < ND; ++it) __syncwarp();   // this lane has run out of patience: it meets the others without arriving
          break;
        }
        const uint8_t* rowp = smem + st * PAR_STAGE + r * 128;
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          const int lc = half * 4 + cc;                      // logical 16-byte chunk of the 64-column slice
          const uint4 v = *reinterpret_cast<const uint4*>(rowp + ((lc ^ (r & 7)) << 4));
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
          const float* nn = sh.s_n + it * 64 + lc * 8;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float lo, hi;
            Pair16<F16>::unpack(w[e], lo, hi);
            qn = fmaf(lo, nn[2 * e], qn);
            qn = fmaf(hi, nn[2 * e + 1], qn);
          }
        }
        fence_proxy_async_smem();   // generic-proxy reads ordered before the TMA refill of the stage
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.bar_qdone[st]);
      }
      sh.s_qn[half][r] = qn;
    }

    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    float rowsum = 0.f;
    mbar_wait(&sh.bar_sfull, 0, &sh.abort, &g_sm100_status, 205);
    tc_fence_after_sync();
    // Tensor memory is read 16 columns at a time, the next load in flight while the current one is processed.
    // gate the score tile; the bf16 result goes back to tensor memory as the A operand of the second product.
    // Both warps of a quarter first read their chunks, then (after a warp-pair sync) write: the bf16 words of
    // chunk cq land on columns [16 cq, 16 cq + 16), which the partner warp may still have to read.
    uint32_t pk[2][16];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int cq = half + 2 * u;
      const int c0 = cq * 32;
      const bool skip = cq > quarter;
      if (skip) {
#pragma unroll
        for (int c = 0; c < 16; ++c) pk[u][c] = 0u;
      } else {
        const bool diag = (cq == quarter);   // only the diagonal chunk needs the causal mask
        uint32_t va[16], vb[16];
        tmem_ld16(tS + lane_base + c0, va);
        tmem_wait_ld(va);
        tmem_ld16(tS + lane_base + c0 + 16, vb);
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          if (hh == 1) tmem_wait_ld(vb);
          const uint32_t (&v)[16] = hh ? vb : va;
          if (diag) {
            const float4* ce = reinterpret_cast<const float4*>(sh.s_colE + c0 + 16 * hh);
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) {
              const float4 e4 = ce[c4];
              const float ee[4] = {e4.x, e4.y, e4.z, e4.w};
              float g4[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int cl = 16 * hh + 4 * c4 + e;   // column inside the chunk; row inside the chunk is `lane`
                float val = __uint_as_float(v[4 * c4 + e]) * ex2_approx(rowE + ee[e]);
                if (cl > lane) val = 0.f;
                g4[e] = val;
                rowsum += val;
              }
              pk[u][8 * hh + 2 * c4] = Pair16<F16>::pack(g4[0], g4[1]);
              pk[u][8 * hh + 2 * c4 + 1] = Pair16<F16>::pack(g4[2], g4[3]);
            }
          } else {
            const float rf = ex2_approx(rowE + sh.s_colP[cq]);
            const float4* cf = reinterpret_cast<const float4*>(sh.s_colF + c0 + 16 * hh);
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) {
              const float4 f4 = cf[c4];
              const float g0 = __uint_as_float(v[4 * c4]) * (rf * f4.x), g1 = __uint_as_float(v[4 * c4 + 1]) * (rf * f4.y);
              const float g2 = __uint_as_float(v[4 * c4 + 2]) * (rf * f4.z), g3 = __uint_as_float(v[4 * c4 + 3]) * (rf * f4.w);
              rowsum += (g0 + g1) + (g2 + g3);
              pk[u][8 * hh + 2 * c4] = Pair16<F16>::pack(g0, g1);
              pk[u][8 * hh + 2 * c4 + 1] = Pair16<F16>::pack(g2, g3);
            }
          }
        }
      }
    }
    // pair sync (bounded): both warps of the quarter have finished reading the score tile
    tc_fence_before_sync();
    mbar_arrive(&sh.bar_pair[quarter]);
    mbar_wait(&sh.bar_pair[quarter], 0, &sh.abort, &g_sm100_status, 210);
    tc_fence_after_sync();
#pragma unroll
    for (int u = 0; u < 2; ++u) tmem_st16(tS + lane_base + (half + 2 * u) * 16, pk[u]);
    sh.s_part[half][r] = rowsum;
    tmem_wait_st();
    // From here to the end the warps go in step whatever their waits answer (see warp_arrive).  A hand-over to the other
    // roles takes place only if no wait has run out (the flag is read where it is needed: kept in a register over the epilogue
    // it costs the kernel 1-2 %); the element-wise warps' own barriers just count.
    // ---- per output tile: row-scale the inter-chunk product, second product, epilogue, store ----
    float inv = 1.f;
    for (int sub = 0; sub < nsub; ++sub) {
      const int o0 = o00 + 128 * sub;
      // the inter-chunk product of this tile has usually landed by now: row-scale it in place
      const bool acc_ok = mbar_wait(&sh.bar_afull, sub & 1, &sh.abort, &g_sm100_status, 214);
      tc_fence_after_sync();
#pragma unroll 1
      for (int cq = half; cq < 4; cq += 2) {
        uint32_t va[16], vb[16];
        const uint32_t ta = tAcc + lane_base + cq * 32;
        tmem_ld16(ta, va);
        tmem_wait_ld(va);
        tmem_ld16(ta + 16, vb);
#pragma unroll
        for (int c = 0; c < 16; ++c) va[c] = __float_as_uint(__uint_as_float(va[c]) * rowscale);
        tmem_wait_ld(vb);
        tmem_st16(ta, va);
#pragma unroll
        for (int c = 0; c < 16; ++c) vb[c] = __float_as_uint(__uint_as_float(vb[c]) * rowscale);
        tmem_st16(ta + 16, vb);
      }
      tmem_wait_st();
      tc_fence_before_sync();
      if (acc_ok) mbar_arrive(&sh.bar_gated);   // (first tile: the gated score tile is in place as well)
      mbar_wait(&sh.bar_hfull, sub & 1, &sh.abort, &g_sm100_status, 206);
      tc_fence_after_sync();
      if (sub == 0) {
        float den = 1.f;
        const float nn = (sh.s_part[0][r] + sh.s_part[1][r]) + rowscale * (use_n ? (sh.s_qn[0][r] + sh.s_qn[1][r]) : 0.f);
        if (p.variant == MLSTM_EXP) den = fmaxf(fabsf(nn), __expf(-m_r));
        else if (p.variant == MLSTM_SIG) den = fmaxf(fabsf(nn), 1.f);
        if (p.variant != MLSTM_SIG_NONORM) inv = 1.f / (den + p.eps);
        if (o_tile0 == 0 && half == 0) {
          if (p.n_out != nullptr && r < valid) p.n_out[out_row0 + r] = den;
          if (p.inv_den_out != nullptr) p.inv_den_out[tok] = r < valid ? inv : 0.f;
        }
      }
      const int ldx = (sub == 0 ? 2 * ND : n0 + (sub - 1) * n1 + ND);    // ring index of this tile's X load
      // The output tile is staged (bf16, two boxes of 128 rows x 128 bytes, 16-byte pieces XOR-swizzled by the row)
      // in the ring stage the X tile occupied (every MMA that read it has completed).  It is then written out by all element-wise
      // warps together, each warp instruction covering two full 256-byte rows of the tile.  Plain stores are posted, so the CTA
      // retires without waiting for them.
      uint8_t* ostage = smem + (ldx % PAR_NST) * PAR_STAGE;
#pragma unroll 1
      for (int cq = half; cq < 4; cq += 2) {
        uint32_t va[16], vb[16];
        const uint32_t ta = tAcc + lane_base + cq * 32;
        tmem_ld16(ta, va);
        tmem_wait_ld(va);
        tmem_ld16(ta + 16, vb);
        uint8_t* orow = ostage + (cq >> 1) * 16384 + r * 128;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c == 2) tmem_wait_ld(vb);
          const uint32_t (&v)[16] = (c < 2) ? va : vb;
          float x[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(v[8 * (c & 1) + e]) * inv;
          const int sw = (((cq & 1) * 4 + c) ^ (r & 7)) << 4;   // 16-byte chunk (cq*4 + c) of the row, swizzled
          uint4 o;
          o.x = Pair16<F16>::pack(x[0], x[1]); o.y = Pair16<F16>::pack(x[2], x[3]);
          o.z = Pair16<F16>::pack(x[4], x[5]); o.w = Pair16<F16>::pack(x[6], x[7]);
          *reinterpret_cast<uint4*>(orow + sw) = o;
        }
      }
      if (sub + 1 < nsub) {   // the accumulator tile may be overwritten by the next tile's inter-chunk product
        tc_fence_before_sync();
        if (!aborted(smem_u32(&sh.abort))) mbar_arrive(&sh.bar_accfree);
      }
      mbar_arrive(&sh.bar_out);
      mbar_wait(&sh.bar_out, sub & 1, &sh.abort, &g_sm100_status, 211);
      {
        uint8_t* gbase = reinterpret_cast<uint8_t*>(p.out_h + out_row0 * DO + o0);
        const int ew = warp - 2, j = lane & 15;          // 16-byte piece j of the 256-byte tile row
#pragma unroll
        for (int i2 = 0; i2 < 8; ++i2) {
          const int orow_i = 16 * i2 + 2 * ew + (lane >> 4);
          const uint4 o = *reinterpret_cast<const uint4*>(ostage + (j >> 3) * 16384 + orow_i * 128 + (((j & 7) ^ (orow_i & 7)) << 4));
          if (orow_i < valid && o0 + j * 8 < DO) *reinterpret_cast<uint4*>(gbase + (size_t)orow_i * DO * 2 + j * 16) = o;
        }
      }
      if (sub + 1 < nsub) {
        // The staging stage of this tile may be refilled.  The TMA engine writes shared memory through the async
        // proxy: without this fence its data can be overtaken by this thread's own earlier (generic-proxy) staging
        // writes to the same addresses.
        fence_proxy_async_smem();
        if (!aborted(smem_u32(&sh.abort))) mbar_arrive(&sh.bar_done[sub & 1]);
      }
    }
  }
  if (LOOP) fence_proxy_async_smem();   // staging writes above, the next run's copies after the barrier
  tc_fence_before_sync();
  __syncthreads();
  const bool go_on = sh.abort == 0;   // (the next run sets it to the 0 that it is)
  // Whichever role gave up: the copies in flight land before the CTA retires.  (On the abort flag alone: a producer that waited for
  // them on every way out, as in the recurrence, would poll while the other roles still work.)
  if (tid == 0 && !go_on)
    for (int ld = max(0, sh.issued - PAR_NST); ld < sh.issued; ++ld)
      mbar_wait(&sh.bar_full[ld % PAR_NST], (ld / PAR_NST) & 1, nullptr, nullptr, 0);
  if (warp == 1 && (!LOOP || last_run || !go_on)) tmem_dealloc(tmem, 256);
  return go_on;
}

template <bool F16>
__global__ void __launch_bounds__(PAR_THREADS, 2)
par_fw_sm100(const __grid_constant__ CUtensorMap mQ, const __grid_constant__ CUtensorMap mK,
             const __grid_constant__ CUtensorMap mV, const __grid_constant__ CUtensorMap mC,
             const __grid_constant__ ParParams p) {
  __shared__ ParShared sh;
  const int T = (p.DHHV + 127) / 128;                 // output tiles per chunk; a CTA takes up to maxsub of them
  // 1-D grid in the order (tile group, chunk, batch x head): no 65535 limit on chunks or batch x heads
  const int gx = (T + p.maxsub - 1) / p.maxsub;
  const int x = blockIdx.x % gx, ck = p.ck0 + (blockIdx.x / gx) % p.n_ck, bh = p.bh0 + blockIdx.x / (gx * p.n_ck);
  const int t0 = p.maxsub * x;
  par_body<F16>(&mQ, &mK, &mV, &mC, p, sh, t0, min(p.maxsub, T - t0), ck, bh);
}

// The same for a range of chunks, beside the recurrence of the following chunks: one CTA per resident place on the SMs that
// the recurrence leaves, each going through the work items with a stride.  A launch of one CTA per item would fill every SM
// between two segments, and the next recurrence, whose CTAs need a whole SM each, would wait for 25 us until they drain.
template <bool F16>
__global__ void __launch_bounds__(PAR_THREADS, 2)
par_fw_range_sm100(const __grid_constant__ CUtensorMap mQ, const __grid_constant__ CUtensorMap mK,
                   const __grid_constant__ CUtensorMap mV, const __grid_constant__ CUtensorMap mC,
                   const __grid_constant__ ParParams p, const unsigned n_items) {
  __shared__ ParShared sh;
  const int T = (p.DHHV + 127) / 128, gx = (T + p.maxsub - 1) / p.maxsub;
  for (unsigned w = blockIdx.x; w < n_items; w += gridDim.x) {
    const int x = w % gx, ck = p.ck0 + (w / gx) % p.n_ck, bh = p.bh0 + w / (gx * p.n_ck), t0 = p.maxsub * x;
    const bool last = w + gridDim.x >= n_items;
    if (!par_body<F16, true>(&mQ, &mK, &mV, &mC, p, sh, t0, min(p.maxsub, T - t0), ck, bh, w == blockIdx.x, last)) return;
  }
}

// =====================================================================================================
// Host side
// =====================================================================================================
bool sm100_supported(int S, int DHQK, int DHHV, int L, int dtype) {
  // any sequence length: a ragged last chunk is handled by zero-filled loads and masked stores
  // head dims: multiples of 8 (16-byte rows for TMA and the vector stores); tiles that hang over the edge of a head
  // dim are padded with zeros by TMA on the way in and masked or clipped on the way out
  return (dtype == MLSTM_BF16 || dtype == MLSTM_F16) && L == CL && S >= 1 && DHQK % 8 == 0 && DHHV % 8 == 0 &&
         DHQK >= 8 && DHHV >= 8 && DHQK <= 512 && DHHV <= 1024;
}

// The kernels address token rows and state rows with 32-bit TMA coordinates and use 1-D grids: both row counts and
// every grid must stay below 2^31.
bool sm100_sizes_ok(int B, int NH, int S, int DHQK, int DHHV) {
  const uint64_t lim = 0x7fffffffull;
  const uint64_t bnh = (uint64_t)B * NH, nc = ((uint64_t)S + CL - 1) / CL;
  const uint64_t tiles = (uint64_t)((DHHV + 127) / 128 + 2 * ((DHQK + 127) / 128));
  return bnh * S < lim && bnh * (nc + 1) * DHQK < lim && bnh * nc * tiles < lim &&
         bnh * (uint64_t)((DHHV + 63) / 64) * ((DHQK + 127) / 128) < lim;
}

// Tensor maps depend only on (base pointer, rows, columns, box): a training loop calls with the same buffers over
// and over, so the last few encodings are kept per thread instead of calling the driver 3-7 times per launch.
struct MapKey { const void* base; uint64_t rows, cols, slabs; uint32_t box_rows, box_cols; bool f16; };
// tensor [slabs x rows x cols]; f16: IEEE half, else bf16
static bool cached_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows,
                       uint32_t box_cols, uint64_t slabs, bool f16) {
  constexpr int N = 32;
  static thread_local MapKey keys[N];
  static thread_local CUtensorMap maps[N];
  static thread_local int used = 0, next = 0;
  for (int i = 0; i < used; ++i) {
    const MapKey& k = keys[i];
    if (k.base == base && k.rows == rows && k.cols == cols && k.slabs == slabs && k.box_rows == box_rows &&
        k.box_cols == box_cols && k.f16 == f16) {
      *m = maps[i];
      return true;
    }
  }
  auto encode = [&]() {
    return sm100_host::make_map_3d(m, base, slabs, rows, cols, box_rows, box_cols, f16);
  };
  if (!encode()) {
    // A thread whose first CUDA work this is (an autograd worker that found all its memory in the allocator's cache) has
    // no context bound yet, and the driver's encoder asks for one: cudaSetDevice binds the device's own.
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess || !encode()) return false;
  }
  keys[next] = MapKey{base, rows, cols, slabs, box_rows, box_cols, f16};
  maps[next] = *m;
  next = (next + 1) % N;
  if (used < N) ++used;
  return true;
}

bool tok_map(CUtensorMap* m, const void* base, const ChunkwiseDims& d, int cols, int box_rows) {
  return cached_map(m, base, (uint64_t)d.S, (uint64_t)cols, box_rows, 64, (uint64_t)d.B * d.NH, d.dtype == MLSTM_F16);
}
bool state_map(CUtensorMap* m, const void* base, const ChunkwiseDims& d, int box_rows) {
  return cached_map(m, base, (uint64_t)d.DHQK, (uint64_t)d.DHHV, box_rows, 64, (uint64_t)d.B * d.NH * (d.NC + 1),
                    d.dtype == MLSTM_F16);
}

template <bool BWD, int TN, bool F16>
static int launch_rec_tn(const CUtensorMap& mL, const CUtensorMap& mR, const CUtensorMap& mS, const RecParams& rp,
                         const ChunkwiseDims& d, int units, const UnitRange& ur, cudaStream_t st) {
  auto kern = rec_sm100<BWD, TN, F16>;
  static bool attr_done[64] = {};
  if (int rc = set_smem_once(kern, rec_smem_bytes(!BWD, TN), attr_done)) return rc;
  const unsigned grid = (unsigned)((d.DHHV + TN - 1) / TN) * (unsigned)((d.DHQK + 127) / 128) * (unsigned)units;
  return launch_ex(ur.overlap && grid <= pdl_max_ctas(), ur.started, kern, grid, REC_THREADS, rec_smem_bytes(!BWD, TN), st, mL, mR, mS, rp);
}

int sm100_forward_segments(const ChunkwiseDims& d) {
  return forward_segments(sm100_recurrence_ctas(d), d.NC, d.B * d.NH, d.DHQK, d.DHHV, sm_count());
}

long sm100_recurrence_ctas(const ChunkwiseDims& d) {
  return (long)((d.DHHV + 127) / 128) * ((d.DHQK + 127) / 128) * d.B * d.NH;
}

struct RecMaps { CUtensorMap l, r, s; };
static bool rec_maps(RecMaps* m, const void* left, const void* right, const void* states, const ChunkwiseDims& d) {
  // recurrence operands arrive in half-chunk boxes (64 tokens x 64 columns)
  return tok_map(&m->l, left, d, d.DHQK, REC_HALF) && tok_map(&m->r, right, d, d.DHHV, REC_HALF) &&
         // store map over the per-chunk states; when no states are wanted (segment summary) the map is never used
         state_map(&m->s, states ? states : left, d, 128);
}

// CTAs of the recurrence of one segment: at most half of the SMs, the others run the intra-chunk kernel
static long segment_ctas(const ChunkwiseDims& d) {
  const long c = sm100_recurrence_ctas(d);
  return 4 * c <= sm_count() ? 2 * c : c;
}

template <bool BWD>
static int launch_rec(const void* left, const void* right, RecParams rp, const ChunkwiseDims& d, UnitRange ur,
                      cudaStream_t st) {
  rp.bh0 = ur.first;
  rp.ck0 = ur.chunk0; rp.n_ck = ur.chunks < 0 ? d.NC - ur.chunk0 : ur.chunks;
  const int units = ur.count < 0 ? d.B * d.NH - ur.first : ur.count;
  if (units <= 0) return MLSTM_OK;
  RecMaps m;
  if (!rec_maps(&m, left, right, rp.c_states, d)) return MLSTM_ERR_CUDA;
  // One CTA per SM walks all chunks of its state tile.  With 128-column tiles a launch of few (batch, head) units
  // leaves SMs idle; 64-column tiles double the CTAs as long as they still fit one wave.
  const bool f16 = d.dtype == MLSTM_F16;
  const long ctas64 = 2 * sm100_recurrence_ctas(d);
  if (ur.chunks < 0 ? ctas64 <= sm_count() : segment_ctas(d) == ctas64)
    return f16 ? launch_rec_tn<BWD, 64, true>(m.l, m.r, m.s, rp, d, units, ur, st) : launch_rec_tn<BWD, 64, false>(m.l, m.r, m.s, rp, d, units, ur, st);
  return f16 ? launch_rec_tn<BWD, 128, true>(m.l, m.r, m.s, rp, d, units, ur, st) : launch_rec_tn<BWD, 128, false>(m.l, m.r, m.s, rp, d, units, ur, st);
}

template <int TN, bool F16>
static int launch_rec_pair(const RecMaps& m, const RecParams& rp, const RecMaps& mb, const RecParams& rpb, const ChunkwiseDims& d,
                           int units, bool overlap, cudaStream_t st) {
  auto kern = rec_pair_sm100<TN, F16>;
  static bool attr_done[64] = {};
  if (int rc = set_smem_once(kern, rec_smem_bytes(false, TN), attr_done)) return rc;
  const unsigned n = (unsigned)((d.DHHV + TN - 1) / TN) * (unsigned)((d.DHQK + 127) / 128) * (unsigned)units;
  return launch_pdl(overlap && 2 * n <= pdl_max_ctas(), kern, 2 * n, REC_THREADS, rec_smem_bytes(false, TN), st, m.l, m.r, m.s, rp, mb.l, mb.r,
                    mb.s, rpb, n);
}

int sm100_recurrent_fw(const void* k, const void* v, const GateBuffers& gb, const float* c_initial,
                       const float* n_initial, void* c_states, float* n_states, float* c_last, float* n_last,
                       const ChunkwiseDims& d, cudaStream_t st, UnitRange ur) {
  PhaseScope ps(PH_REC_FW, st);
  RecParams rp{gb.abar, nullptr, 1.f, gb.gbar, c_initial, n_initial, c_states,
               d.variant == MLSTM_SIG_NONORM ? nullptr : n_states, c_last, d.variant == MLSTM_SIG_NONORM ? nullptr : n_last, d.S, d.SP, d.NC, d.DHQK, d.DHHV, 0, 0, d.NC};
  return launch_rec<false>(k, v, rp, d, ur, st);
}

int sm100_recurrent_bw(const void* q, const void* dh, const GateBuffers& gb, const float* dc_last, void* dc_states,
                       float* dc_initial, const ChunkwiseDims& d, cudaStream_t st, UnitRange ur) {
  PhaseScope ps(PH_REC_BW, st);
  RecParams rp{gb.bbar, gb.inv_den, d.qk_scale, gb.gbar, dc_last, nullptr, dc_states, nullptr,
               dc_initial, nullptr, d.S, d.SP, d.NC, d.DHQK, d.DHHV, 0, 0, d.NC};
  return launch_rec<true>(q, dh, rp, d, ur, st);
}

int sm100_recurrent_pair(const void* k, const void* v, const float* c_initial, void* c_states, const void* q, const void* dh,
                         const float* dc_last, void* dc_states, float* dc_initial, const GateBuffers& gb,
                         const ChunkwiseDims& d, cudaStream_t st, UnitRange ur) {
  const int units = ur.count < 0 ? d.B * d.NH - ur.first : ur.count;
  if (units <= 0) return MLSTM_OK;
  PhaseScope ps(PH_REC_BW, st);
  const RecParams rp{gb.abar, nullptr, 1.f, gb.gbar, c_initial, nullptr, c_states, nullptr, nullptr, nullptr,
                     d.S, d.SP, d.NC, d.DHQK, d.DHHV, ur.first, 0, d.NC};
  const RecParams rpb{gb.bbar, gb.inv_den, d.qk_scale, gb.gbar, dc_last, nullptr, dc_states, nullptr, dc_initial, nullptr,
                      d.S, d.SP, d.NC, d.DHQK, d.DHHV, ur.first, 0, d.NC};
  RecMaps m, mb;
  if (!rec_maps(&m, k, v, c_states, d) || !rec_maps(&mb, q, dh, dc_states, d)) return MLSTM_ERR_CUDA;
  const bool f16 = d.dtype == MLSTM_F16;
  if (4 * sm100_recurrence_ctas(d) <= sm_count())   // (the rule of launch_rec, for twice the CTAs)
    return f16 ? launch_rec_pair<64, true>(m, rp, mb, rpb, d, units, ur.overlap, st) : launch_rec_pair<64, false>(m, rp, mb, rpb, d, units, ur.overlap, st);
  return f16 ? launch_rec_pair<128, true>(m, rp, mb, rpb, d, units, ur.overlap, st) : launch_rec_pair<128, false>(m, rp, mb, rpb, d, units, ur.overlap, st);
}

static ParParams base_params(const GateBuffers& gb, const ChunkwiseDims& d) {
  ParParams pp{};
  pp.vecB = gb.vecB; pp.iota = gb.iota; pp.m_tok = gb.m_tok; pp.bbar = gb.bbar;
  pp.S = d.S; pp.SP = d.SP; pp.NC = d.NC; pp.DHQK = d.DHQK; pp.DHHV = d.DHHV; pp.variant = d.variant; pp.eps = d.eps;
  pp.qk_scale = d.qk_scale;
  return pp;
}

// Output tiles per CTA.  Tiles of one chunk share the score tile and its gating, so a full launch gives a CTA up to
// PAR_MAXSUB of them; a launch whose CTAs would not fill the GPU (two fit on an SM) splits them over more CTAs instead,
// each computing the score for itself: one tile takes about 9 us, every further one 5.5 us, and the SMs are idle anyway
// (500 tokens, 8 heads 256/512: 32 CTAs of four tiles 18.5 us).
template <typename F>
static int par_maxsub(F ctas, int tiles) {
  int m = std::min(PAR_MAXSUB, tiles);
  while (m > 1 && ctas(m) < 2L * sm_count() && ctas((m + 1) / 2) <= 2L * sm_count()) m = (m + 1) / 2;
  return m;
}

int sm100_parallel_fw(const void* q, const void* k, const void* v, const GateBuffers& gb, const void* c_states,
                      const float* n_states, void* h, float* n_out, const ChunkwiseDims& d, cudaStream_t st,
                      UnitRange ur) {
  const int units = ur.count < 0 ? d.B * d.NH - ur.first : ur.count;
  if (units <= 0) return MLSTM_OK;
  PhaseScope ps(PH_PAR_FW, st);
  CUtensorMap mQ, mK, mV, mC;
  if (!tok_map(&mQ, q, d, d.DHQK) || !tok_map(&mK, k, d, d.DHQK) || !tok_map(&mV, v, d, d.DHHV) ||
      !state_map(&mC, c_states, d, 64))
    return MLSTM_ERR_CUDA;
  ParParams pp = base_params(gb, d);
  pp.n_states = n_states; pp.out_h = (uint16_t*)h; pp.n_out = n_out; pp.inv_den_out = gb.inv_den;
  pp.bh0 = ur.first; pp.ck0 = ur.chunk0; pp.n_ck = ur.chunks < 0 ? d.NC - ur.chunk0 : ur.chunks;
  const bool f16 = d.dtype == MLSTM_F16;
  const int T = (d.DHHV + 127) / 128;
  pp.maxsub = par_maxsub([&](int m) { return (long)ceil_div(T, m) * pp.n_ck * units; }, T);
  const unsigned grid = (unsigned)ceil_div(T, pp.maxsub) * (unsigned)pp.n_ck * (unsigned)units;
  if (ur.chunks >= 0 && ur.chunk0 + ur.chunks < d.NC) {   // another segment's recurrence runs beside this launch
    const unsigned places = 2u * (unsigned)(sm_count() - (int)segment_ctas(d));
    auto kern = f16 ? par_fw_range_sm100<true> : par_fw_range_sm100<false>;
    static bool range_attr[2][64] = {};
    if (int rc = set_smem_once(kern, PAR_SMEM, range_attr[f16])) return rc;
    return launch_pdl(false, kern, std::min(grid, places), PAR_THREADS, PAR_SMEM, st, mQ, mK, mV, mC, pp, grid);
  }
  auto kern = f16 ? par_fw_sm100<true> : par_fw_sm100<false>;
  static bool attr_done[2][64] = {};
  if (int rc = set_smem_once(kern, PAR_SMEM, attr_done[f16])) return rc;
  return launch_pdl(ur.overlap && grid <= pdl_max_ctas(), kern, grid, PAR_THREADS, PAR_SMEM, st, mQ, mK, mV, mC, pp);
}

// Self-test of the bounded wait: one thread waits, for at most `limit` polls, on an mbarrier that nothing arrives
// at.  No copy is in flight and no tensor memory is held, so giving up is all that happens: the wait records
// `code` in the status word and the kernel returns.
__global__ void wait_expiry_selftest_kernel(uint32_t limit, int code) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(&bar, 1);
    fence_barrier_init();
    mbar_wait(&bar, 0, &abort_flag, &g_sm100_status, code, limit);
  }
}

int sm100_wait_expiry_selftest(unsigned limit, int code, cudaStream_t st) {
  if (limit == 0 || limit > 1000000u || code <= 0) return MLSTM_ERR_UNSUPPORTED;   // a few milliseconds at most
  wait_expiry_selftest_kernel<<<1, 32, 0, st>>>(limit, code);
  MLSTM_LAUNCH_CHECK();
  return MLSTM_OK;
}

int sm100_force_load() {
  cudaFuncAttributes a;
  MLSTM_CUDA_CHECK(cudaFuncGetAttributes(&a, (rec_sm100<false, 128, false>)));
  MLSTM_CUDA_CHECK(cudaFuncGetAttributes(&a, (rec_sm100<false, 64, false>)));
  MLSTM_CUDA_CHECK(cudaFuncGetAttributes(&a, par_fw_sm100<false>));
  MLSTM_CUDA_CHECK(cudaFuncGetAttributes(&a, (rec_sm100<false, 128, true>)));
  MLSTM_CUDA_CHECK(cudaFuncGetAttributes(&a, (rec_sm100<false, 64, true>)));
  MLSTM_CUDA_CHECK(cudaFuncGetAttributes(&a, par_fw_sm100<true>));
  return MLSTM_OK;
}

// Reads (and optionally clears) the status word the bounded waits write on a timeout.  Synchronises the device.
int sm100_device_status(int reset, int* status) {
  MLSTM_CUDA_CHECK(cudaDeviceSynchronize());
  MLSTM_CUDA_CHECK(cudaMemcpyFromSymbol(status, g_sm100_status, sizeof(int)));
  if (reset) {
    const int zero = 0;
    MLSTM_CUDA_CHECK(cudaMemcpyToSymbol(g_sm100_status, &zero, sizeof(int)));
  }
  int bw = 0;
  const int rc = par_bw_status(reset, &bw);
  if (*status == 0) *status = bw;
  return rc;
}

}  // namespace mlstm
