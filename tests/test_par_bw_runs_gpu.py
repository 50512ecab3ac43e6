"""Intra-chunk backward (csrc/chunkwise_bw_sm100.cu) where a CTA takes several work items and a launch several CTAs per SM,
against the oracle on units from the beginning, the middle and the end of the launch."""

import pytest
import torch

from inputs import max_rel_err
from util_gpu import case_inputs, run_cuda_fwbw, run_oracle_fwbw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B, NH, S, DHQK, DHHV", [
    (1, 149, 40, 8, 24),         # one ragged chunk per unit: an item's step crosses units, and is more than a unit long
    (2, 40, 300, 64, 128),       # five items per CTA, one tile each
    (3, 16, 500, 96, 320),       # one tile of two modes, three of the other, two of them partial
    (2, 11, 1030, 264, 136),     # nine chunks, the last of six tokens; a tile of eight columns
    (1, 4, 37900, 16, 16),       # more items than the CTAs of one wave take
    (1, 16, 300, 128, 256),      # whole items in one round
    (1, 8, 600, 256, 512),       # the same, with four tiles
    (1, 8, 1000, 256, 512),      # split items in two rounds, with a stride of its own
    (2, 8, 1700, 256, 1024),     # two tile groups of one mode, every CTA in turn through all kinds of items
])
@pytest.mark.parametrize("dtype, tol", [(torch.bfloat16, 2e-2), (torch.float16, 2e-2)])
@pytest.mark.parametrize("siging", [False, True])
def test_runs_of_items(B, NH, S, DHQK, DHHV, dtype, tol, siging):
    """Bounds as in the other 16-bit parity tests."""
    units = (0, B * NH // 2, B * NH - 1)
    inp = case_inputs(S + DHHV, B, NH, S, DHQK, DHHV)
    got = run_cuda_fwbw(inp, 128, dtype, siging=siging)
    one = {k: v.reshape(1, B * NH, *v.shape[2:])[:, list(units)] if v is not None and v.ndim >= 3 else v for k, v in inp.items()}
    ref = run_oracle_fwbw(one, next(c for c in (100, 20, 10, 2) if S % c == 0), dtype, siging=siging)
    for key in ("dQ", "dK", "dV", "dI", "dF"):
        x = got[key].reshape(1, B * NH, *got[key].shape[2:])[:, list(units)]
        assert max_rel_err(x, ref[key]) < tol, key
