"""Malformed calls are refused with the same exceptions by the native host module (eager calls) and by the Python path (traced
and multi-GPU calls), before anything is launched: checked without a GPU, on fake CUDA tensors."""

import pytest
import torch
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
