"""Edges of the kernels' splits and of the launch rules, against the oracle."""

import math

import numpy as np
import pytest
import torch

import mlstm_kernels_b200 as mk
from inputs import max_rel_err
from oracle import mlstm_oracle as O
from util_gpu import case_inputs, npy, run_cuda_fwbw, run_oracle_fwbw

pytestmark = pytest.mark.gpu

KEYS = ("H", "C_last", "n_last", "m_last", "dQ", "dK", "dV", "dI", "dF")


def check(got, ref, tol):
    for k in KEYS:
        assert max_rel_err(got[k], ref[k]) < tol, k


@pytest.mark.parametrize("NC", [1, 2, 31, 32, 33, 63, 65, 129, 257, 513])
def test_gates_chunk_counts(NC):
    """The pre-pass gives every warp a run of chunks and every CTA of a cluster a share of them."""
    inp = case_inputs(100 + NC, 1, 2, 16 * NC, 16, 16)
    check(run_cuda_fwbw(inp, 16), run_oracle_fwbw(inp, 16), 2e-3)


@pytest.mark.parametrize("L", [256, 512, 1024])
def test_gates_long_chunks(L):
    """More tokens in a chunk than a warp handles at once."""
    inp = case_inputs(L, 1, 1, 3 * L, 16, 24)
    check(run_cuda_fwbw(inp, L), run_oracle_fwbw(inp, L), 2e-3)


@pytest.mark.parametrize("DHQK, DHHV", [(12, 20), (13, 18), (36, 68), (64, 132), (65, 67), (130, 260)])
def test_f32_head_dims(DHQK, DHHV):
    """16-byte and single-element accesses, partial tiles of the f32 kernels."""
    inp = case_inputs(DHQK, 1, 2, 256, DHQK, DHHV, init=True, dC_last=True)
    check(run_cuda_fwbw(inp, 64), run_oracle_fwbw(inp, 64), 2e-3)


@pytest.mark.parametrize("B, NH, S, DHQK, DHHV", [
    (1, 1, 130, 128, 520),     # few CTAs: one output tile each, the last 8 columns wide
    (1, 3, 384, 264, 392),     # 64-column state tiles, both recurrences of the backward in one launch
    (2, 19, 256, 128, 136),    # 76 state tiles: 128 columns in the backward's launch, 64 elsewhere
    (2, 40, 200, 256, 256),    # more state tiles than SMs
])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_tile_splits(B, NH, S, DHQK, DHHV, dtype):
    inp = case_inputs(S, B, NH, S, DHQK, DHHV)
    check(run_cuda_fwbw(inp, 128, dtype), run_oracle_fwbw(inp, math.gcd(S, 128), dtype), 2e-2)


@pytest.mark.parametrize("DHQK, DHHV", [(64, 512), (40, 384), (64, 1024)])
@pytest.mark.parametrize("siging", [False, True])
def test_one_operand_slice_and_several_output_tiles(DHQK, DHHV, siging):
    """A head dim of one 64-column slice in a launch that fills the GPU: a CTA takes three or four output tiles, with two
    loads each.  Two of the 32 units against the oracle; bounds as in the other 16-bit parity tests."""
    B, NH, S, units = 2, 16, 1344, (3, 30)
    inp = case_inputs(DHQK + DHHV, B, NH, S, DHQK, DHHV)
    got = run_cuda_fwbw(inp, 128, torch.bfloat16, siging=siging)
    one = {k: v.reshape(1, B * NH, *v.shape[2:])[:, list(units)] if v is not None and v.ndim >= 3 else v for k, v in inp.items()}
    ref = run_oracle_fwbw(one, 64, torch.bfloat16, siging=siging)
    for key in ("H", "dQ", "dK", "dV", "dI", "dF"):
        x = got[key].reshape(1, B * NH, *got[key].shape[2:])[:, list(units)]
        assert max_rel_err(x, ref[key]) < 2e-2, key


@pytest.mark.parametrize("B, NH, DHQK, DHHV", [(1, 1, 8, 8), (1, 3, 100, 36), (1, 5, 512, 28), (4, 9, 256, 68), (6, 16, 128, 100), (40, 9, 64, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_step_slices(B, NH, DHQK, DHHV, dtype):
    """Narrow column slices at small batch, wide ones beyond, widths that neither divides."""
    g = torch.Generator().manual_seed(B * NH + DHHV)
    r = lambda *s: torch.randn(*s, generator=g)
    q, k, v = r(B, NH, DHQK).to(dtype), r(B, NH, DHQK).to(dtype), r(B, NH, DHHV).to(dtype)
    i, f = r(B, NH, 1), r(B, NH, 1) + 2.0
    c, n, m = r(B, NH, DHQK, DHHV), r(B, NH, DHQK), r(B, NH, 1)
    cu = [t.cuda() for t in (q, k, v, i, f, c, n, m)]
    h, (c1, n1, m1) = mk.mlstm_recurrent_step__b200(*cu)
    d = [npy(t) for t in (q, k, v, i, f, c, n, m)]
    hr, (cr, nr, mr) = O.recurrent_step(*d)
    tol = 1e-4 if dtype is torch.float32 else 2e-2
    assert max_rel_err(npy(h), hr) < tol
    for a, b in ((c1, cr), (n1, nr), (m1, mr)):
        assert max_rel_err(npy(a), np.asarray(b).reshape(a.shape)) < 1e-4


def test_native_host_argument_errors():
    """The exception types are those of the Python wrappers (every malformed operand: test_argument_errors_cpu.py)."""
    q = torch.randn(1, 2, 64, 32, device="cuda")
    i = torch.randn(1, 2, 64, device="cuda")
    with pytest.raises(ValueError, match="inconsistent shapes"):
        mk.mlstm_chunkwise__b200_xl_chunk(q, q[:, :1], q, i, i)            # other number of heads in k
    with pytest.raises(ValueError, match="inconsistent shapes"):
        mk.mlstm_chunkwise__b200_xl_chunk(q, q, q, i[:, :, :5], i)         # fewer gates than tokens
    with pytest.raises(RuntimeError, match="m_initial"):                   # one max state for two heads
        mk.mlstm_chunkwise__b200_xl_chunk(q, q, q, i, i, m_initial=torch.zeros(1, 1, 1, device="cuda"))
    with pytest.raises(AssertionError, match="matC_old has wrong shape"):
        mk.mlstm_recurrent_step__b200(q[:, :, 0], q[:, :, 0], q[:, :, 0], i[:, :, :1], i[:, :, :1],
                                      torch.zeros(1, 2, 32, 31, device="cuda"), torch.zeros(1, 2, 32, device="cuda"),
                                      torch.zeros(1, 2, 1, device="cuda"))
