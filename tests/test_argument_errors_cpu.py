"""Malformed calls are refused with the same exceptions by the native host module (eager calls) and by the Python path (traced
and multi-GPU calls), before anything is launched: checked without a GPU, on fake CUDA tensors."""

import pytest
import torch
import torch.autograd.forward_ad as fwAD
from torch._subclasses.fake_tensor import FakeTensorMode

import mlstm_kernels_b200 as mk
from mlstm_kernels_b200 import _lib
from mlstm_kernels_b200.chunkwise import chunkwise_fw_raw

B, NH, S, DHQK, DHHV = 2, 3, 128, 32, 64


def operands(dtype=torch.bfloat16):
    e = lambda *s, dt=dtype: torch.empty(*s, dtype=dt, device="cuda")  # noqa: E731
    return dict(q=e(B, NH, S, DHQK), k=e(B, NH, S, DHQK), v=e(B, NH, S, DHHV), i=e(B, NH, S), f=e(B, NH, S),
                c_initial=e(B, NH, DHQK, DHHV, dt=torch.float32), n_initial=e(B, NH, DHQK, dt=torch.float32),
                m_initial=e(B, NH, 1, dt=torch.float32))


CASES = [
    ("k", (B, 1, S, DHQK), ValueError), ("v", (B, NH, S - 1, DHHV), ValueError), ("i", (B, NH, 5), ValueError),
    ("f", (B, NH, S, 1), ValueError),
    ("m_initial", (B, NH - 1, 1), RuntimeError), ("m_initial", (1,), RuntimeError), ("m_initial", (B, NH, 2), RuntimeError),
    ("c_initial", (B, NH, DHQK, DHHV - 1), ValueError), ("c_initial", (NH, DHQK, DHHV), ValueError),
    ("n_initial", (B, NH, DHQK - 1), ValueError),
]


@pytest.mark.parametrize("name,shape,error", CASES)
@pytest.mark.parametrize("path", ["eager", "python"])
def test_wrong_sizes_are_refused(path, name, shape, error):
    with FakeTensorMode():
        a = operands()
        a[name] = torch.empty(*shape, dtype=a[name].dtype, device="cuda")
        with pytest.raises(Exception) as e:
            if path == "eager":
                mk.mlstm_chunkwise__b200_xl_chunk(**a)
            else:
                chunkwise_fw_raw(**a, chunk_size=128, eps=1e-6, variant=_lib.EXP)
    assert e.type is error, e.value
    assert ("inconsistent shapes" if name in "kvif" else name) in str(e.value)


@pytest.mark.parametrize("name", ["c_initial", "n_initial", "m_initial"])
@pytest.mark.parametrize("path", ["eager", "python"])
def test_states_in_host_memory_are_refused(path, name):
    with FakeTensorMode():
        a = operands()
        a[name] = torch.empty(a[name].shape)
        with pytest.raises(RuntimeError, match="CUDA tensors only"):
            if path == "eager":
                mk.mlstm_chunkwise__b200_xl_chunk(**a)
            else:
                chunkwise_fw_raw(**a, chunk_size=128, eps=1e-6, variant=_lib.EXP)


@pytest.mark.parametrize("name", ["q", "f", "c_initial"])
def test_forward_mode_tangents_are_refused(name):
    with FakeTensorMode(), fwAD.dual_level():
        a = operands()
        a[name] = fwAD.make_dual(a[name], torch.empty_like(a[name]))
        with pytest.raises(NotImplementedError):
            mk.mlstm_chunkwise__b200_xl_chunk(**a)


@pytest.mark.parametrize("impl", ["cutlass", "\ud800", None, 1])
def test_unknown_implementation_is_a_key_error(impl):
    with FakeTensorMode(), pytest.raises(KeyError):
        mk.mlstm_chunkwise__b200_xl_chunk(**operands(), impl=impl)


def step_operands():
    e = lambda *s, dt=torch.bfloat16: torch.empty(*s, dtype=dt, device="cuda")  # noqa: E731
    f32 = torch.float32
    return dict(matC_old=e(B, NH, DHQK, DHHV, dt=f32), vecN_old=e(B, NH, DHQK, dt=f32), scaM_old=e(B, NH, 1, dt=f32),
                vecQ=e(B, NH, DHQK), vecK=e(B, NH, DHQK), vecV=e(B, NH, DHHV), scaI=e(B, NH, 1), scaF=e(B, NH, 1),
                matC_new=e(B, NH, DHQK, DHHV, dt=f32), vecN_new=e(B, NH, DHQK, dt=f32), scaM_new=e(B, NH, 1, dt=f32))


@pytest.mark.parametrize("name,shape,error", [
    ("vecK", (B, NH, DHQK - 1), AssertionError), ("vecV", (1, NH, DHHV), AssertionError),
    ("matC_old", (B, NH, DHQK, DHHV - 1), AssertionError), ("vecN_old", (NH, DHQK), AssertionError),
    ("scaM_old", (B, NH), AssertionError), ("scaI", (B, NH), AssertionError), ("scaF", (B, 1, 1), AssertionError),
    ("matC_new", (B, NH, DHQK, DHHV - 1), ValueError), ("vecN_new", (NH, DHQK), ValueError), ("scaM_new", (B, 1, 1), ValueError)])
def test_decode_step_refuses_wrong_sizes(name, shape, error):
    from mlstm_kernels_b200.recurrent import mlstm_recurrent_step__b200_fw
    with FakeTensorMode():
        a = step_operands()
        a[name] = torch.empty(*shape, dtype=a[name].dtype, device="cuda")
        with pytest.raises(Exception) as e:
            mlstm_recurrent_step__b200_fw(**a)
    assert e.type is error, e.value


@pytest.mark.parametrize("name", ["vecK", "vecV", "scaI", "scaF", "vecN_old", "scaM_old", "matC_new", "vecN_new", "scaM_new"])
def test_decode_step_refuses_host_memory(name):
    from mlstm_kernels_b200.recurrent import mlstm_recurrent_step__b200_fw
    with FakeTensorMode():
        a = step_operands()
        a[name] = torch.empty(a[name].shape, dtype=a[name].dtype)
        with pytest.raises(RuntimeError, match="CUDA tensors only"):
            mlstm_recurrent_step__b200_fw(**a)


@pytest.mark.parametrize("name,shape", [("k", (B, 1, S, DHQK)), ("v", (B, NH, S - 1, DHHV)), ("i", (B, NH, S - 1)), ("f", (B, 1, S)),
                                        ("c_initial", (B, NH, DHQK, DHHV - 1)), ("n_initial", (NH, DHQK)), ("m_initial", (B, 1, 1))])
def test_sequence_refuses_wrong_sizes_and_host_memory(name, shape):
    with FakeTensorMode():
        a = operands()
        a[name] = torch.empty(*shape, dtype=a[name].dtype, device="cuda")
        with pytest.raises(ValueError, match="inconsistent shapes|too small"):
            mk.mlstm_recurrent_sequence__b200(**a)
        a = operands()
        a[name] = torch.empty(a[name].shape, dtype=a[name].dtype)
        with pytest.raises(RuntimeError, match="CUDA tensors only"):
            mk.mlstm_recurrent_sequence__b200(**a)
