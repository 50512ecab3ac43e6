// The chunkwise forward and backward as one struct per call: what the extern "C" entry points of
// include/mlstm_b200.h and the PyTorch host module (host.cpp) both fill in.
#pragma once
#include <stddef.h>

#include "../../include/mlstm_b200.h"

namespace mlstm {

struct CallDims {
  int B, NH, S, DHQK, DHHV, L, dtype, gate_dtype, variant, impl;
  float eps;
  void* stream;
};

struct FwCall {
  const void *q, *k, *v, *i, *f;
  const float *c_initial, *n_initial, *m_initial;   // each may be null
  void* h;
  float *n_out, *m_out;        // per-token denominator and max state, each may be null
  void* c_states;              // per-chunk states; n_states / m_states likewise
  float *n_states, *m_states;
  float *c_last, *n_last, *m_last;                  // each may be null
  float* inv_den;              // (B*NH, NC*L) 1 / (denominator + eps) for the backward, or null
  void* workspace;
  size_t workspace_bytes;
  bool allow_split;            // false: every launch stays on the caller's stream
  void* scores;                // scratch of score_scratch_bytes(), or null: slower without
};

struct BwCall {
  const void *q, *k, *v, *i, *f;
  const float* m_initial;
  const void* c_states;        // as the forward wrote them, or null with `recompute_into`
  void* recompute_into;        // scratch for the per-chunk states, recomputed from `recompute_c_initial`
  const float* recompute_c_initial;
  const float* n_out;          // null when `inv_den` is given
  const float* inv_den;        // as the forward wrote it, or null
  const void* fw_workspace;    // the forward's scratch buffer, intact, or null (gate pre-pass runs again)
  size_t fw_workspace_bytes;
  const void* dh;
  const float* dc_last;
  void *dq, *dk, *dv;
  void *di, *df;
  int grad_gate_dtype;         // element type of di, df
  float* dc_initial;
  void* workspace;
  size_t workspace_bytes;
  void* scores;                // as in FwCall
};

#if defined(__GNUC__)
#pragma GCC visibility push(default)
#endif
// scratch of a forward with allow_split = false (0: sizes it does not take)
size_t fw_bytes_one_stream(const CallDims& c);
// further scratch that a forward or backward call can use (0: none)
size_t score_scratch_bytes(const CallDims& c, bool backward);
int run_chunkwise_fw(const FwCall& a, const CallDims& c);
int run_chunkwise_bw(const BwCall& a, const CallDims& c);
#if defined(__GNUC__)
#pragma GCC visibility pop
#endif

}  // namespace mlstm
