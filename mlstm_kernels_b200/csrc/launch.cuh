// Host-side launcher prototypes shared between the translation units of libmlstm_b200.so.
#pragma once
#include "common.cuh"

namespace mlstm {

// gates.cu
// m_out (nullable): user-visible copy of the per-token max state, S entries per (batch, head); m_last (nullable): copy of
// the last entry of each m_states row
int launch_gates(int dtype, const void* i, const void* f, const float* m_initial, const float* n_out, float* m_out,
                 const GateBuffers& gb, float* m_states, float* m_last, const ChunkwiseDims& d, cudaStream_t st,
                 float m_default = 0.f, float* g_sum = nullptr);
int launch_inv_den(const float* n_out, float* inv_den, const ChunkwiseDims& d, cudaStream_t st);
int launch_state_combine(const float* c_in, const float* n_in, const float* m_in, const float* c_loc,
                         const float* n_loc, const float* m_loc, const float* g_total, float* c_out, float* n_out,
                         float* m_out, int BNH, int DHQK, int DHHV, int variant, cudaStream_t st);
int launch_gate_grads(int dtype, int gate_dtype, const void* q, const void* k, const void* dq, const void* dk, const void* i,
                      const void* f, float* acc, float* kdk, void* dI, void* dF, int out_dtype, const ChunkwiseDims& d,
                      cudaStream_t st);
int launch_gate_grad_scan(int dtype, const void* i, const void* f, const float* qdq, const float* kdk, int nparts,
                          void* dI, void* dF, int out_dtype, const ChunkwiseDims& d, cudaStream_t st, const float* anchors,
                          int n_anchors, int anchor_tokens);
int launch_state_dot(const void* c_states, const void* dc_states, float* anchors, int every, int n_anchors,
                     const ChunkwiseDims& d, cudaStream_t st);

// chunkwise_simt.cu : portable CUDA-core kernels, any shape, any element type
// scores (nullable): scratch of simt_score_bytes(), filled by the recurrence's launch and read by the intra-chunk kernel
size_t simt_score_bytes(const ChunkwiseDims& d, bool backward);
int simt_recurrent_fw(int dtype, const void* q, const void* k, const void* v, const GateBuffers& gb,
                      const float* c_initial, const float* n_initial, void* c_states, float* n_states,
                      float* c_last, float* n_last, float* scores, const ChunkwiseDims& d, cudaStream_t st);
int simt_parallel_fw(int dtype, const void* q, const void* k, const void* v, const GateBuffers& gb,
                     const void* c_states, const float* n_states, void* h, float* n_out, const float* scores, const ChunkwiseDims& d,
                     cudaStream_t st);
// c_states (nullable): where the forward's per-chunk states are written again, from c_initial
int simt_recurrent_bw(int dtype, const void* q, const void* k, const void* v, const void* dh, const GateBuffers& gb,
                      const float* dc_last, void* dc_states, float* dc_initial, const float* c_initial, void* c_states, float* scores,
                      const ChunkwiseDims& d, cudaStream_t st);
int simt_parallel_bw(int dtype, const void* q, const void* k, const void* v, const void* dh,
                     const GateBuffers& gb, const void* c_states, const void* dc_states, void* dq, void* dk, void* dv, const float* scores,
                     const ChunkwiseDims& d, cudaStream_t st);

// chunkwise_sm100.cu : tcgen05 + TMA kernels (bf16 / fp16, L = 128, head dims multiples of 8)
bool sm100_supported(int S, int DHQK, int DHHV, int L, int dtype);
bool sm100_sizes_ok(int B, int NH, int S, int DHQK, int DHHV);
// A launch may cover a sub-range of the B * NH independent (batch, head) units; all pointers stay those of the whole
// problem.  count < 0: every unit from `first` on.
// overlap: the launch may begin while the one before it in the stream drains (launch_pdl).
// The forward's launches may cover a range of chunks too (chunks < 0: every chunk from chunk0 on).
// started (forward recurrence, nullable): recorded once all of its CTAs are running.
struct UnitRange { int first = 0; int count = -1; bool overlap = true; int chunk0 = 0; int chunks = -1; cudaEvent_t started = nullptr; };
int sm100_recurrent_fw(const void* k, const void* v, const GateBuffers& gb, const float* c_initial,
                       const float* n_initial, void* c_states, float* n_states, float* c_last, float* n_last,
                       const ChunkwiseDims& d, cudaStream_t st, UnitRange ur = UnitRange());
int sm100_parallel_fw(const void* q, const void* k, const void* v, const GateBuffers& gb, const void* c_states,
                      const float* n_states, void* h, float* n_out, const ChunkwiseDims& d, cudaStream_t st,
                      UnitRange ur = UnitRange());
int sm100_recurrent_bw(const void* q, const void* dh, const GateBuffers& gb, const float* dc_last, void* dc_states,
                       float* dc_initial, const ChunkwiseDims& d, cudaStream_t st, UnitRange ur = UnitRange());
// the forward's recurrence again (states only) and the state gradient's, in one launch
int sm100_recurrent_pair(const void* k, const void* v, const float* c_initial, void* c_states, const void* q, const void* dh,
                         const float* dc_last, void* dc_states, float* dc_initial, const GateBuffers& gb,
                         const ChunkwiseDims& d, cudaStream_t st, UnitRange ur = UnitRange());
int sm100_parallel_bw(const void* q, const void* k, const void* v, const void* dh, const GateBuffers& gb,
                      const void* c_states, const void* dc_states, void* dq, void* dk, void* dv, float* qdq_parts,
                      float* kdk_parts, const ChunkwiseDims& d, cudaStream_t st, UnitRange ur = UnitRange());
// number of CTAs the recurrence launches for the whole problem with 128-column state tiles
long sm100_recurrence_ctas(const ChunkwiseDims& d);
// segments the forward cuts the sequence into (1: none); a function of the sizes alone
int sm100_forward_segments(const ChunkwiseDims& d);

int sm100_device_status(int reset, int* status);
int par_bw_status(int reset, int* status);   // (the part of it that chunkwise_bw_sm100.cu keeps)
int sm100_wait_expiry_selftest(unsigned limit, int code, cudaStream_t st);
// make the runtime load the forward kernels' code on the current device now (CUDA loads modules lazily, on first use)
int sm100_force_load();
int gates_force_load();

// step.cu
int launch_step(const void* q, const void* k, const void* v, const void* i, const void* f, const void* c,
                const void* n, const void* m, void* h, void* c_new, void* n_new, void* m_new, int B, int NH, int DHQK,
                int DHHV, int dtype, int gate_dtype, int state_dtype, float eps, cudaStream_t st);
int launch_step_sequence(const void* q, const void* k, const void* v, const void* i, const void* f, const float* c,
                         const float* n, const float* m, void* h, float* c_new, float* n_new, float* m_new, int B,
                         int NH, int T, int DHQK, int DHHV, int dtype, int gate_dtype, float eps, cudaStream_t st);

}  // namespace mlstm
