// Intra-chunk backward of the chunkwise mLSTM for B200 (sm_100a): deltaV, deltaK, deltaQ of every chunk.
//   out[r,:] = sum_c G[r,c] X[c,:] + rowscale_r * (A[r,:] . State),   G[r,c] = gate(r,c) * (A[r,:] . B[c,:])
//   mode  A    B    contraction  gate   X    State operand                  rowscale            out
//   DV    K    Q    DHQK         upper  dH   dC_{k+1}   [DHQK x DHHV]       abar_r              dV
//   DK    V    dH   DHHV         upper  Q    dC_{k+1}^T (rows d, cols e)    abar_r              dK, row sums k . dk
//   DQ    dH   V    DHHV         lower  K    C_k^T      (rows d, cols e)    s*bbar_r/(den_r+e)  dQ, row sums q . dq
//   lower: c <= r, (i,j) = (r,c); upper: c >= r, (i,j) = (c,r); gate = s * exp((b_i - b_j) + iota_j - m_i) / (den_i+eps)
// bw_kernel_parallel_dV.py, bw_kernel_parallel_dK.py, bw_kernel_parallel_dQ.py of mlstm_kernels/triton/chunkwise/xl_chunk
//
// One CTA per SM goes through work items (chunk, mode, group of 128-column output tiles) with every ring and barrier running on
// from item to item, so that nothing has to drain in between:
//   warp 0        TMA producer of the operand ring (stages of 32 KB: an (A, B) or (A, State) pair of 64-column slices, or an X tile)
//   warp 1        MMA issuer
//   warp 2        loads the E tile (the tensor whose row sums with the output are wanted) into one of two buffers, from which
//                 the finished output tile leaves again
//   (warp 3 idle: a warp may touch the 32 rows of tensor memory that its number modulo four names)
//   warps 4-11    gate the score tile (two warps per 32-row quarter), scale the rows of the inter-chunk product
//   warps 12-19   read the finished accumulator, stage the output tile over the E tile
// Tensor memory: the score tile (128 columns), two gated tiles (16-bit pairs, 64 columns each), two accumulators (128 each).
// Order of the products:
//   score(item) | X(last tile of the item before) | inter(tile 0) | inter(tile 1) | X(tile 0) | ... | score(next item) | ...
// so that an item is gated while its inter-chunk products run, a tile is scaled while the next product runs, and the epilogue
// of a tile runs beside the next tile's products.
//
// What bounds it: HBM and the shared memory together.  Every operand byte is written to shared memory by TMA and read by the
// MMA, and E and the output pass through it too: 1.15 MB per item at 256/256, 9200 of the 11000 cycles that an item takes at 128 bytes
// per cycle, the rate that a 128 x 128 x 16 product of two shared operands asks for by itself.  Counters (2 x 8192 tokens, 16 heads
// 256/256, 260 us): 1.15 MB read and written per item (22 % of the banks' peak each way, which the counter puts at 256 bytes per
// cycle), tensor pipe busy 43 % of the cycles, 1.46 GB from and to HBM, 0.86 of the copy rate.
// (Before, one CTA per chunk and mode, two to an SM, each a chain of dependent steps: 8 x 8192 tokens, 16 heads
// 256/256 1302 us, now 1089; 16 x 2048, 128/256 431, now 342; 4 x 1024, 4 heads 96/192 22.9, now 20.9.)
// Measured and not taken: an accumulator of 256 columns (A read once for two tiles, 10 % less port traffic, but nothing left to
// overlap the epilogue with: 1260 and 440 us where this form then took 1130 and 351); the modes of one chunk in one CTA (the 148 chunks in flight no longer fit
// in L2: 1150 and 383); L2 prefetch of the next item's operands (1144-1230 and 396-408).

#include "common.cuh"
#include "launch.cuh"
#include "par_bw_items.h"
#include "sm100.cuh"
#include "tensor_maps.cuh"

namespace mlstm {

using namespace sm100;

__device__ int g_par_bw_status = 0;  // first error code raised by a bounded wait of this file's kernels (0 = none)

namespace {

constexpr int CL = 128;          // chunk length

struct BwMaps {
  CUtensorMap q, k, v, dh;           // 128 tokens x 64 columns
  CUtensorMap c_k, dc_mn, dc_k;      // states: C^T and dC^T slices 128 x 64, dC slices 64 x 64
  CUtensorMap dq, dk, dv;            // outputs
};

struct BwParams : BwItems {
  const float *vecB, *iota, *m_tok, *abar, *bbar, *inv_den;  // per token, f32
  float *rowdot_q, *rowdot_k;   // sum_d q dq (from DQ), sum_d k dk (from DK); one partial per output tile: [DHQK/128][tokens]
  size_t nslots;                // B * NH * SP
  int S, SP;                    // SP = NC * 128: slots per (batch, head) of the per-token gate vectors
  float qk_scale;
};

constexpr int NST = 5;                   // operand ring depth
constexpr int STAGE = 32768;
constexpr int TILE = 32768;              // E tile and output staging, two of them
constexpr int THREADS = 640;

struct BwShared {
  uint64_t full[NST], empty[NST], sfull, sread, gready[2], afull[2], accfree[2], scaled[2], hfull[2], ready[2], staged[2];
  uint32_t tmem;
  int issued;                 // ring loads the producer has issued
  int abort;                  // set by the first wait of this CTA that runs out; every other wait polls it
  alignas(16) float colE[CL]; // per-column term of the gate exponent, base 2
  alignas(16) float colF[CL]; // 2^(colE_c - colP of the column's 32-column block)
  float colP[4];              // largest colE of each 32-column block
  float dot[2][CL];           // row sums of the second 64 columns of a tile, for the warp that adds the two halves
};
constexpr int OFF_T = NST * STAGE, OFF_C = OFF_T + 2 * TILE, SMEM = OFF_C + 3072;
static_assert(sizeof(BwShared) <= 3072 && SMEM <= 232448, "shared memory of one CTA");

// gate vectors of a token; scale: its abar or bbar
struct RowGate { float b, iota, m, inv, scale; };

template <bool F16>
__global__ void __launch_bounds__(THREADS, 1)
par_bw_run_sm100(const __grid_constant__ BwMaps maps, const __grid_constant__ BwParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  BwShared& sh = *reinterpret_cast<BwShared*>(smem + OFF_C);
  uint8_t* tiles = smem + OFF_T;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if ((smem_u32(smem) & 1023u) != 0) {   // (the swizzle counts from 1024-byte boundaries; there is no static shared memory in front)
    if (tid == 0) atomicCAS(&g_par_bw_status, 0, 300);
    return;
  }

  if (tid == 0) {
    sh.abort = 0; sh.issued = 0;
    for (int s = 0; s < NST; ++s) { mbar_init(&sh.full[s], 1); mbar_init(&sh.empty[s], 1); }
    mbar_init(&sh.sfull, 1); mbar_init(&sh.sread, 8);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sh.gready[s], 8); mbar_init(&sh.afull[s], 1); mbar_init(&sh.accfree[s], 8); mbar_init(&sh.scaled[s], 8);
      mbar_init(&sh.hfull[s], 1); mbar_init(&sh.ready[s], 1); mbar_init(&sh.staged[s], 8);
    }
    fence_barrier_init();
    const CUtensorMap* m = &maps.q;
    for (int i = 0; i < (int)(sizeof(BwMaps) / sizeof(CUtensorMap)); ++i) tma_prefetch_desc(m + i);
  }
  if (warp == 1) { tmem_alloc(&sh.tmem, 512); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = sh.tmem;
  // No pdl_launch_dependents(): these CTAs take an SM each, registers and shared memory, for the whole launch, and CTAs of the next
  // launch that are let in before they end go, all of them, to the few SMs that have none, and stay there (8 heads, 1024 tokens,
  // forward and backward, with it at the start and without: 256/1024 263 and 141 us, 256/512 132 and 91; 3200 tokens 243 and 178;
  // with it behind the last product, 128/256, 1152 tokens 68.9 and 64.8).
  pdl_wait();

  BwRun it(p, blockIdx.x, gridDim.x);
  if (warp == 0) {
    // ---------------- TMA producer: same order as the MMA issuer ----------------
    if (elect_one()) {
      int st = 0, issued = 0;
      uint32_t ph = 1;
      bool ok = true;
      // two 64-column boxes, or one and two half ones, into the next stage
      auto acquire = [&]() -> uint8_t* {
        ok = ok && mbar_wait(&sh.empty[st], ph, &sh.abort, &g_par_bw_status, 301);
        if (ok) mbar_expect_tx(&sh.full[st], STAGE);
        return smem + st * STAGE;
      };
      auto advance = [&]() {
        ++issued;
        if (++st == NST) { st = 0; ph ^= 1; }
      };
      const CUtensorMap* px = nullptr;
      int po0 = 0, py0 = 0, pbh = 0;
      auto load_x = [&]() {   // X of the tile before
        uint8_t* sb = acquire();
        if (!ok) return;
        tma_load_3d(sb, px, &sh.full[st], po0, py0, pbh);
        tma_load_3d(sb + 16384, px, &sh.full[st], po0 + 64, py0, pbh);
        advance();
      };
      for (; it.left > 0 && ok; it.next(p)) {
        const int mode = it.mode(p), y0 = it.ck * CL, nd = it.slices(p), t0 = it.tile0(p), nsub = it.tiles(p);
        const CUtensorMap* a = mode == PM_DV ? &maps.k : (mode == PM_DK ? &maps.v : &maps.dh);
        const CUtensorMap* b = mode == PM_DV ? &maps.q : (mode == PM_DK ? &maps.dh : &maps.v);
        const CUtensorMap* x = mode == PM_DV ? &maps.dh : (mode == PM_DK ? &maps.q : &maps.k);
        const CUtensorMap* s = mode == PM_DV ? &maps.dc_mn : (mode == PM_DK ? &maps.dc_k : &maps.c_k);
        const int sz = it.bh * (p.NC + 1) + (mode == PM_DQ ? it.ck : it.ck + 1);
        for (int i = 0; i < nd; ++i) {
          uint8_t* sb = acquire();
          if (!ok) break;
          tma_load_3d(sb, a, &sh.full[st], 64 * i, y0, it.bh);
          tma_load_3d(sb + 16384, b, &sh.full[st], 64 * i, y0, it.bh);
          advance();
        }
        for (int sub = 0; sub < nsub && ok; ++sub) {
          if (sub == 0 && px != nullptr) load_x();
          const int o0 = 128 * (t0 + sub);
          for (int i = 0; i < nd; ++i) {
            uint8_t* sb = acquire();
            if (!ok) break;
            tma_load_3d(sb, a, &sh.full[st], 64 * i, y0, it.bh);
            if (mode == PM_DV) {
              tma_load_3d(sb + 16384, s, &sh.full[st], o0, 64 * i, sz);
              tma_load_3d(sb + 16384 + 8192, s, &sh.full[st], o0 + 64, 64 * i, sz);
            } else {
              tma_load_3d(sb + 16384, s, &sh.full[st], 64 * i, o0, sz);
            }
            advance();
          }
          if (sub > 0 && ok) load_x();
          px = x; po0 = o0; py0 = y0; pbh = it.bh;
        }
      }
      if (ok && px != nullptr) load_x();
      sh.issued = issued;
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      constexpr uint32_t idesc_kk = umma_idesc_16(F16, 128, 128, 0, 0), idesc_kn = umma_idesc_16(F16, 128, 128, 0, 1);
      constexpr uint32_t hi = umma_desc_hi(1024);
      const uint32_t tS = tmem, tG = tmem + 128, tA = tmem + 256;
      const uint32_t base = smem_u32(smem) >> 4;
      int st = 0;
      uint32_t ph = 0;
      bool ok = true;
      // low word of the descriptor of the next stage of the ring (its leading-dimension field still empty: unused with K-major operands)
      auto arrived = [&]() -> uint32_t {
        ok = ok && mbar_wait(&sh.full[st], ph, &sh.abort, &g_par_bw_status, 302);
        tc_fence_after_sync();
        return base + st * (STAGE >> 4);
      };
      constexpr uint32_t lbo8 = (8192u >> 4) << 16, lbo16 = (16384u >> 4) << 16;
      auto release = [&]() {
        umma_commit(&sh.empty[st]);
        if (++st == NST) { st = 0; ph ^= 1; }
      };
      int t = 0;   // tiles begun
      // second product of tile t - 1, of item n: the gated score tile times X, on top of the scaled inter-chunk product
      auto mul_x = [&](int n, bool first) {
        const int tp = t - 1;
        const uint32_t sx = arrived();
        if (first) ok = ok && mbar_wait(&sh.gready[n & 1], (n >> 1) & 1, &sh.abort, &g_par_bw_status, 303);
        if (!ok || !(ok = mbar_wait(&sh.scaled[tp & 1], (tp >> 1) & 1, &sh.abort, &g_par_bw_status, 304))) return;
        tc_fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma_ts(tA + (tp & 1) * 128, tG + (n & 1) * 64 + kk * 8, umma_desc((sx | lbo16) + kk * (2048 >> 4), hi), idesc_kn, 1u);
        release();
        umma_commit(&sh.hfull[tp & 1]);
      };
      int n = 0, before = 0;   // items begun; tiles of the item before
      for (; it.left > 0 && ok; it.next(p), ++n) {
        const int nd = it.slices(p), nsub = it.tiles(p);
        const bool mn = it.mode(p) == PM_DV;          // the state operand is N-contiguous in shared memory
        const uint32_t step = (mn ? 2048 : 32) >> 4, idesc = mn ? idesc_kn : idesc_kk;
        if (n > 0 && !(ok = mbar_wait(&sh.sread, (n - 1) & 1, &sh.abort, &g_par_bw_status, 305))) break;
        for (int i = 0; i < nd; ++i) {            // score: S = A . B^T
          const uint32_t sa = arrived(), sb = sa + (16384 >> 4);
          if (!ok) break;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_ss(tS, umma_desc(sa + kk * (32 >> 4), hi), umma_desc(sb + kk * (32 >> 4), hi), idesc_kk, (i > 0 || kk > 0) ? 1u : 0u);
          release();
        }
        if (!ok) break;
        umma_commit(&sh.sfull);
        for (int sub = 0; sub < nsub && ok; ++sub) {
          if (sub == 0 && t > 0) { mul_x(n - 1, before == 1); if (!ok) break; }
          // the accumulator is free once the epilogue has read the tile before the last
          if (t >= 2 && !(ok = mbar_wait(&sh.accfree[t & 1], ((t >> 1) - 1) & 1, &sh.abort, &g_par_bw_status, 306))) break;
          tc_fence_after_sync();
          const uint32_t acc = tA + (t & 1) * 128;
          for (int i = 0; i < nd; ++i) {           // inter-chunk term: Acc = A . State
            const uint32_t sa = arrived(), ss = (sa + (16384 >> 4)) | (mn ? lbo8 : 0u);
            if (!ok) break;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_ss(acc, umma_desc(sa + kk * (32 >> 4), hi), umma_desc(ss + kk * step, hi), idesc, (i > 0 || kk > 0) ? 1u : 0u);
            release();
          }
          if (!ok) break;
          umma_commit(&sh.afull[t & 1]);
          if (sub > 0) mul_x(n, sub == 1);
          ++t;
        }
        before = nsub;
      }
      if (ok && t > 0) mul_x(n - 1, before == 1);
    }
  } else if (warp == 2) {
    // ---------------- E tiles in, output tiles out ----------------
    if (elect_one()) {
      BwRun ahead = it;                     // two tiles ahead of the tile that is stored
      int asub = 0, loaded = 0;
      auto fill = [&]() {                   // make the buffer ready for the next tile, if there is one
        if (ahead.left <= 0) return;
        const int b = loaded & 1, mode = ahead.mode(p);
        if (mode == PM_DV) {
          mbar_arrive(&sh.ready[b]);
        } else {
          const CUtensorMap* e = mode == PM_DK ? &maps.k : &maps.q;
          const int o0 = 128 * (ahead.tile0(p) + asub), y0 = ahead.ck * CL;
          mbar_expect_tx(&sh.ready[b], TILE);
          tma_load_3d(tiles + b * TILE, e, &sh.ready[b], o0, y0, ahead.bh);
          tma_load_3d(tiles + b * TILE + 16384, e, &sh.ready[b], o0 + 64, y0, ahead.bh);
        }
        ++loaded;
        if (++asub == ahead.tiles(p)) { asub = 0; ahead.next(p); }
      };
      fill(); fill();
      int t = 0;
      bool ok = true;
      for (; it.left > 0 && ok; it.next(p)) {
        const int mode = it.mode(p), nsub = it.tiles(p), t0 = it.tile0(p), y0 = it.ck * CL;
        const CUtensorMap* out = mode == PM_DV ? &maps.dv : (mode == PM_DK ? &maps.dk : &maps.dq);
        const int DO = mode == PM_DV ? p.DHHV : p.DHQK;
        for (int sub = 0; sub < nsub; ++sub, ++t) {
          if (!(ok = mbar_wait(&sh.staged[t & 1], (t >> 1) & 1, &sh.abort, &g_par_bw_status, 307))) break;
          const uint8_t* src = tiles + (t & 1) * TILE;
          const int o0 = 128 * (t0 + sub);
          tma_store_3d(out, src, o0, y0, it.bh);                    // (clipped at the end of the sequence and of the head dim)
          if (o0 + 64 < DO) tma_store_3d(out, src + 16384, o0 + 64, y0, it.bh);
          tma_store_commit();
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the tile has left its buffer
          fill();
        }
      }
      // nothing of this thread's is in flight when the CTA retires
      for (int l = max(0, loaded - 2); l < loaded; ++l) mbar_wait(&sh.ready[l & 1], (l >> 1) & 1, nullptr, nullptr, 0);
      tma_store_wait_all();
    }
  } else if (warp >= 12) {
    // ---------------- output: accumulator -> 16-bit tile, row sums with E ----------------
    const int quarter = warp & 3, half = (warp - 12) >> 2;   // 32 rows, 64 columns
    const int r = quarter * 32 + lane;
    int t = 0, db = 0;
    for (; it.left > 0; it.next(p)) {
      const int mode = it.mode(p), nsub = it.tiles(p);
      const bool has_e = mode != PM_DV;
      float* rowdot = (mode == PM_DQ ? p.rowdot_q : p.rowdot_k) + (size_t)it.tile0(p) * p.nslots + (size_t)it.bh * p.SP + it.ck * CL + r;
      for (int sub = 0; sub < nsub; ++sub, ++t) {
        const bool rok = mbar_wait(&sh.ready[t & 1], (t >> 1) & 1, &sh.abort, &g_par_bw_status, 308);
        const bool hok = mbar_wait(&sh.hfull[t & 1], (t >> 1) & 1, &sh.abort, &g_par_bw_status, 309);
        tc_fence_after_sync();
        const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + 256 + (t & 1) * 128 + half * 64;
        uint8_t* orow = tiles + (t & 1) * TILE + half * 16384 + r * 128;
        float dot4[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t va[16], vb[16];
        auto put = [&](const uint32_t (&v)[16], int c0) {   // 16 columns: two 16-byte pieces, swizzled by the row
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int sw = ((c0 + c) ^ (r & 7)) << 4;
            if (has_e) {
              const uint4 ev = *reinterpret_cast<const uint4*>(orow + sw);
              const uint32_t w[4] = {ev.x, ev.y, ev.z, ev.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                float lo, hi;
                Pair16<F16>::unpack(w[e], lo, hi);
                dot4[e] = fmaf(lo, __uint_as_float(v[8 * c + 2 * e]), dot4[e]);
                dot4[e] = fmaf(hi, __uint_as_float(v[8 * c + 2 * e + 1]), dot4[e]);
              }
            }
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = Pair16<F16>::pack(__uint_as_float(v[8 * c + 2 * e]), __uint_as_float(v[8 * c + 2 * e + 1]));
            *reinterpret_cast<uint4*>(orow + sw) = make_uint4(o[0], o[1], o[2], o[3]);
          }
        };
        tmem_ld16(ta, va);
        tmem_wait_ld(va);
        tmem_ld16(ta + 16, vb);
        put(va, 0);
        tmem_wait_ld(vb);
        tmem_ld16(ta + 32, va);
        put(vb, 2);
        tmem_wait_ld(va);
        tmem_ld16(ta + 48, vb);
        put(va, 4);
        tmem_wait_ld(vb);
        tc_fence_before_sync();
        warp_arrive(&sh.accfree[t & 1], hok);
        put(vb, 6);
        fence_proxy_async_smem();
        warp_arrive(&sh.staged[t & 1], hok && rok);
        if (has_e) {   // (two buffers: a warp that is a tile ahead has met the other in between)
          const float dot = (dot4[0] + dot4[1]) + (dot4[2] + dot4[3]);
          if (half == 1) sh.dot[db][r] = dot;
          asm volatile("bar.sync %0, 64;" ::"r"(6 + quarter) : "memory");
          if (half == 0) rowdot[(size_t)sub * p.nslots] = dot + sh.dot[db][r];
          db ^= 1;
        }
      }
    }
  } else if (warp >= 4) {
    // ---------------- gating: score tile -> 16-bit A operand ----------------
    const int quarter = warp & 3, half = (warp - 4) >> 2;
    const int r = quarter * 32 + lane;
    constexpr float kLog2e = 1.4426950408889634f;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    auto load_gate = [&](const BwRun& i) -> RowGate {
      const size_t tok = (size_t)i.bh * p.SP + i.ck * CL + r;
      return RowGate{p.vecB[tok], p.iota[tok], p.m_tok[tok], p.inv_den[tok], i.mode(p) == PM_DQ ? p.bbar[tok] : p.abar[tok]};
    };
    RowGate g{};
    if (it.left > 0) g = load_gate(it);
    for (int n = 0, t = 0; it.left > 0; ++n) {
      const bool lower = it.mode(p) == PM_DQ;
      const int nsub = it.tiles(p);
      const float rowscale = lower ? p.qk_scale * g.scale * g.inv : g.scale;
      const float rowE = (lower ? (g.b - g.m) : (g.iota - g.b)) * kLog2e + __log2f(lower ? p.qk_scale * g.inv : p.qk_scale);
      float cE = 0.f, cF = 0.f, cP = 0.f;
      if (half == 0) {   // this thread's row in its role as a column of the gate matrix
        cE = lower ? (g.iota - g.b) * kLog2e : (g.b - g.m) * kLog2e + __log2f(g.inv);
        cP = cE;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cP = fmaxf(cP, __shfl_xor_sync(0xffffffffu, cP, o));
        if (!(cP > -3.0e38f)) cP = 0.f;   // a block whose columns are all switched off
        cF = ex2_approx(cE - cP);
      }
      // the next item's vectors are asked for as soon as this one's are used up: a trip to L2 less in every item's chain
      it.next(p);
      if (it.left > 0) g = load_gate(it);
      asm volatile("bar.sync 1, 256;" ::: "memory");   // every warp is through with the columns of the item before
      if (half == 0) {
        sh.colE[r] = cE;
        sh.colF[r] = cF;
        if (lane == 0) sh.colP[quarter] = cP;
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
      // (the products with the gated tile of two items ago are done: they were issued before this score)
      const bool sok = mbar_wait(&sh.sfull, n & 1, &sh.abort, &g_par_bw_status, 310);
      tc_fence_after_sync();
      const uint32_t tS = tmem + lane_base, tG = tmem + 128 + (n & 1) * 64 + lane_base;
#pragma unroll 1
      for (int cq = half; cq < 4; cq += 2) {
        uint32_t pk[16];
        if (lower ? (cq > quarter) : (cq < quarter)) {
#pragma unroll
          for (int c = 0; c < 16; ++c) pk[c] = 0u;
        } else {
          uint32_t va[16], vb[16];
          tmem_ld16(tS + cq * 32, va);
          tmem_ld16(tS + cq * 32 + 16, vb);
          const float rf = ex2_approx(rowE + sh.colP[cq]);
          tmem_wait_ld(va);
          tmem_wait_ld(vb);
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            const uint32_t (&v)[16] = hh ? vb : va;
            if (cq == quarter) {   // only the diagonal block needs the causal mask
              const float4* ce = reinterpret_cast<const float4*>(sh.colE + cq * 32 + 16 * hh);
#pragma unroll
              for (int c4 = 0; c4 < 4; ++c4) {
                const float4 e4 = ce[c4];
                const float ee[4] = {e4.x, e4.y, e4.z, e4.w};
                float g4[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const int cl = 16 * hh + 4 * c4 + e;   // column inside the block; row inside the block is `lane`
                  const float val = __uint_as_float(v[4 * c4 + e]) * ex2_approx(rowE + ee[e]);
                  g4[e] = (lower ? (cl > lane) : (cl < lane)) ? 0.f : val;
                }
                pk[8 * hh + 2 * c4] = Pair16<F16>::pack(g4[0], g4[1]);
                pk[8 * hh + 2 * c4 + 1] = Pair16<F16>::pack(g4[2], g4[3]);
              }
            } else {
              const float4* cf = reinterpret_cast<const float4*>(sh.colF + cq * 32 + 16 * hh);
#pragma unroll
              for (int c4 = 0; c4 < 4; ++c4) {
                const float4 f4 = cf[c4];
                pk[8 * hh + 2 * c4] = Pair16<F16>::pack(__uint_as_float(v[4 * c4]) * (rf * f4.x), __uint_as_float(v[4 * c4 + 1]) * (rf * f4.y));
                pk[8 * hh + 2 * c4 + 1] = Pair16<F16>::pack(__uint_as_float(v[4 * c4 + 2]) * (rf * f4.z), __uint_as_float(v[4 * c4 + 3]) * (rf * f4.w));
              }
            }
          }
        }
        tmem_st16(tG + cq * 16, pk);
      }
      tmem_wait_st();
      tc_fence_before_sync();
      warp_arrive(&sh.sread, sok);
      warp_arrive(&sh.gready[n & 1], sok);
      for (int sub = 0; sub < nsub; ++sub, ++t) {
        const bool aok = mbar_wait(&sh.afull[t & 1], (t >> 1) & 1, &sh.abort, &g_par_bw_status, 311);
        tc_fence_after_sync();
        const uint32_t ta = tmem + lane_base + 256 + (t & 1) * 128 + half * 64;
        uint32_t va[16], vb[16];
        auto scale = [&](uint32_t (&v)[16]) {
#pragma unroll
          for (int c = 0; c < 16; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) * rowscale);
        };
        tmem_ld16(ta, va);
        tmem_ld16(ta + 16, vb);
        tmem_wait_ld(va);
        tmem_wait_ld(vb);
        scale(va);
        tmem_st16(ta, va);
        tmem_ld16(ta + 32, va);
        scale(vb);
        tmem_st16(ta + 16, vb);
        tmem_ld16(ta + 48, vb);
        tmem_wait_ld(va);
        tmem_wait_ld(vb);
        scale(va);
        tmem_st16(ta + 32, va);
        scale(vb);
        tmem_st16(ta + 48, vb);
        tmem_wait_st();
        tc_fence_before_sync();
        warp_arrive(&sh.scaled[t & 1], aok);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && sh.abort != 0) {   // the ring's copies in flight land before the CTA retires
    for (int l = max(0, sh.issued - NST); l < sh.issued; ++l) mbar_wait(&sh.full[l % NST], (l / NST) & 1, nullptr, nullptr, 0);
  }
  if (warp == 1) tmem_dealloc(tmem, 512);
}

}  // namespace

int sm100_parallel_bw(const void* q, const void* k, const void* v, const void* dh, const GateBuffers& gb,
                      const void* c_states, const void* dc_states, void* dq, void* dk, void* dv, float* qdq_parts,
                      float* kdk_parts, const ChunkwiseDims& d, cudaStream_t st, UnitRange ur) {
  const int units = ur.count < 0 ? d.B * d.NH - ur.first : ur.count;
  if (units <= 0) return MLSTM_OK;
  PhaseScope ps(PH_PAR_BW, st);
  BwMaps m;
  if (!tok_map(&m.q, q, d, d.DHQK) || !tok_map(&m.k, k, d, d.DHQK) || !tok_map(&m.v, v, d, d.DHHV) || !tok_map(&m.dh, dh, d, d.DHHV) ||
      !state_map(&m.c_k, c_states, d, 128) || !state_map(&m.dc_mn, dc_states, d, 64) || !state_map(&m.dc_k, dc_states, d, 128) ||
      !tok_map(&m.dq, dq, d, d.DHQK) || !tok_map(&m.dk, dk, d, d.DHQK) || !tok_map(&m.dv, dv, d, d.DHHV))
    return MLSTM_ERR_CUDA;
  const BwItems w = bw_plan(units, ur.first, d.NC, d.DHQK, d.DHHV, sm_count());
  const BwParams p{w, gb.vecB, gb.iota, gb.m_tok, gb.abar, gb.bbar, gb.inv_den, qdq_parts, kdk_parts, (size_t)d.B * d.NH * d.SP,
                   d.S, d.SP, d.qk_scale};
  // A CTA takes up to 24 items: its start (2 us) is then 1-2 % of its time, and a launch beside another chain's recurrence, which
  // frees the SMs one by one, still spreads over them (8 x 8192 tokens, 16 heads 256/256, alone: 3, 6, 12, 24, 96 items per CTA
  // 1271, 1246, 1210, 1219, 1217 us in the first form of the kernel; 16 x 2048, 128/256: 435, 413, 393, 389, 379).
  const unsigned grid = bw_grid(w);
  const bool f16 = d.dtype == MLSTM_F16;
  static bool attr_done[2][64] = {};
  if (int rc = f16 ? set_smem_once(par_bw_run_sm100<true>, SMEM, attr_done[1]) : set_smem_once(par_bw_run_sm100<false>, SMEM, attr_done[0])) return rc;
  return launch_pdl(ur.overlap && grid <= pdl_max_ctas(), f16 ? par_bw_run_sm100<true> : par_bw_run_sm100<false>, grid, THREADS, SMEM, st, m, p);
}

int par_bw_status(int reset, int* status) {
  MLSTM_CUDA_CHECK(cudaMemcpyFromSymbol(status, g_par_bw_status, sizeof(int)));
  if (reset) {
    const int zero = 0;
    MLSTM_CUDA_CHECK(cudaMemcpyToSymbol(g_par_bw_status, &zero, sizeof(int)));
  }
  return MLSTM_OK;
}

}  // namespace mlstm
