"""PyTorch-facing recurrent decode kernels backed by libmlstm_b200.so.

`mlstm_recurrent_step__b200` keeps the signature of mlstm_recurrent_step__triton
(mlstm_kernels/torch/recurrent/triton_step.py:130-158); `mlstm_recurrent_sequence__b200` that of the
sequence kernels (mlstm_kernels/torch/recurrent/native_sequence.py:125-170).

A decode step at small batch is a few microseconds of device time, so an eager call goes straight to the native host
module (csrc/host.cpp): tensors that already have the expected element type and layout are passed through untouched,
and the gate pre-activations keep their own element type (the kernel widens them to f32, as
mlstm_kernels/triton/recurrent/fw_step_fused.py:88-94 does).
"""

from __future__ import annotations

import torch

from . import _lib, _ops

_STATE_DTYPES = (torch.float32, torch.bfloat16)

# cheapest route to the current stream's handle
_raw_stream_c = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _raw_stream(device_index: int) -> int:
    if _raw_stream_c is not None:
        return _raw_stream_c(device_index)
    return torch.cuda.current_stream(device_index).cuda_stream


_STEP_FN = None


def _step_fn():
    global _STEP_FN
    if _STEP_FN is None:
        _STEP_FN = _lib.load().mlstm_b200_step
    return _STEP_FN


def mlstm_recurrent_step__b200_fw(
    matC_old: torch.Tensor,  # (B, NH, DHQK, DHHV)
    vecN_old: torch.Tensor,  # (B, NH, DHQK)
    scaM_old: torch.Tensor,  # (B, NH, 1)
    vecQ: torch.Tensor,  # (B, NH, DHQK)
    vecK: torch.Tensor,  # (B, NH, DHQK)
    vecV: torch.Tensor,  # (B, NH, DHHV)
    scaI: torch.Tensor,  # (B, NH, 1)
    scaF: torch.Tensor,  # (B, NH, 1)
    matC_new: torch.Tensor = None,
    vecN_new: torch.Tensor = None,
    scaM_new: torch.Tensor = None,
    eps: float = 1e-6,
    dtype_state: torch.dtype = torch.float32,
    vecH_out: torch.Tensor = None,  # optional caller-owned output (B, NH, DHHV) in q's dtype
    validate: bool = True,
    **kwargs,
):
    """One decode step.  `validate=False` is for decode loops that own all their buffers: every tensor (the new-state
    and `vecH_out` buffers included) must then be a contiguous CUDA tensor of the expected shape and element type on
    the current device; nothing is checked or converted.  (The call goes through ctypes: 6.3 us per step at batch 1, where
    the checked call, which is native, takes 4.2.)"""
    if not validate:
        B, NH, DHQK = vecQ.shape
        codes = _lib._DTYPE_CODE
        rc = _step_fn()(vecQ.data_ptr(), vecK.data_ptr(), vecV.data_ptr(), scaI.data_ptr(), scaF.data_ptr(),
                        matC_old.data_ptr(), vecN_old.data_ptr(), scaM_old.data_ptr(), vecH_out.data_ptr(),
                        matC_new.data_ptr(), vecN_new.data_ptr(), scaM_new.data_ptr(), B, NH, DHQK,
                        vecV.shape[-1], codes[vecQ.dtype], codes[scaI.dtype], codes[dtype_state], eps,
                        _raw_stream(vecQ.device.index))
        if rc != 0:
            _lib.check(rc, "mlstm_b200_step")
        return vecH_out, (matC_new, vecN_new, scaM_new)
    return _lib.host().step(matC_old, vecN_old, scaM_old, vecQ, vecK, vecV, scaI, scaF, matC_new, vecN_new, scaM_new,
                            eps, dtype_state, vecH_out)


def mlstm_recurrent_step__b200(
    q: torch.Tensor,  # (B, NH, DHQK)
    k: torch.Tensor,  # (B, NH, DHQK)
    v: torch.Tensor,  # (B, NH, DHHV)
    i: torch.Tensor,  # (B, NH, 1)
    f: torch.Tensor,  # (B, NH, 1)
    c: torch.Tensor,  # (B, NH, DHQK, DHHV)
    n: torch.Tensor,  # (B, NH, DHQK)
    m: torch.Tensor,  # (B, NH, 1)
    eps: float = 1e-6,
    dtype_state: torch.dtype = torch.float32,
    **kwargs,
) -> tuple[torch.Tensor, tuple[torch.Tensor, torch.Tensor, torch.Tensor]]:
    """One mLSTM decode step: returns h (B,NH,DHHV) and the new (C, n, m); the old states are untouched."""
    if torch.compiler.is_compiling():   # a tracer is watching: go through the custom operator
        if dtype_state not in _STATE_DTYPES:
            raise ValueError(f"Unsupported state dtype {dtype_state}.")
        h, c_new, n_new, m_new = _ops.step(q, k, v, i, f, c, n, m, eps, dtype_state is torch.bfloat16)
        return h, (c_new, n_new, m_new)
    if not kwargs:
        return _lib.host().step(c, n, m, q, k, v, i, f, None, None, None, eps, dtype_state, None)
    return mlstm_recurrent_step__b200_fw(matC_old=c, vecN_old=n, scaM_old=m, vecQ=q, vecK=k, vecV=v, scaI=i,
                                         scaF=f, eps=eps, dtype_state=dtype_state, **kwargs)


def mlstm_recurrent_sequence__b200(
    q: torch.Tensor,  # (B, NH, S, DHQK)
    k: torch.Tensor,
    v: torch.Tensor,  # (B, NH, S, DHHV)
    i: torch.Tensor,  # (B, NH, S)
    f: torch.Tensor,
    c_initial: torch.Tensor = None,
    n_initial: torch.Tensor = None,
    m_initial: torch.Tensor = None,
    return_last_states: bool = False,
    eps: float = 1e-6,
    dtype_state: torch.dtype = torch.float32,
    **kwargs,
):
    """S decode steps in ONE launch with the state held in registers (replaces the per-token Python loop)."""
    if torch.compiler.is_compiling():   # a tracer is watching: go through the custom operator
        h, c_new, n_new, m_new = _ops.step_sequence(q, k, v, i, f, c_initial, n_initial, m_initial, eps)
        if return_last_states:
            return h, (c_new.to(dtype_state), n_new.to(dtype_state), m_new.to(dtype_state))
        return h
    h, last = _lib.host().sequence(q, k, v, i, f, c_initial, n_initial, m_initial, eps,
                                   dtype_state if return_last_states else torch.float32)
    return (h, last) if return_last_states else h
