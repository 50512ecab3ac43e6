"""Portable kernels with the score blocks of a chunk computed once (what the PyTorch functions do where it pays) and with every
output tile computing them anew (calls without that scratch): the same bits."""

import pytest
import torch

from mlstm_kernels_b200 import _lib
from mlstm_kernels_b200.chunkwise import (chunkwise_bw_raw, chunkwise_fw_raw, mlstm_chunkwise__b200_xl_chunk,
                                          mlstm_siging_chunkwise__b200_xl_chunk)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("DHQK, DHHV", [(64, 64), (128, 256), (96, 128), (65, 190), (130, 100)])   # smallest, partial tiles, single elements
@pytest.mark.parametrize("L", [64, 128])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("variant, recompute", [(_lib.EXP, True), (_lib.SIG, False), (_lib.SIG_NONORM, True)])
def test_score_blocks_equal_scores_per_tile(DHQK, DHHV, L, dtype, variant, recompute):
    B, NH, S = 2, 3, 3 * L
    g = torch.Generator(device="cuda").manual_seed(DHQK + L)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k, v, dh = (rnd(B, NH, S, d).to(dtype) for d in (DHQK, DHQK, DHHV, DHHV))
    i, f = rnd(B, NH, S), rnd(B, NH, S) + 3.0
    kw = dict(chunk_size=L, impl="simt", eps=1e-6)
    fw = chunkwise_fw_raw(q, k, v, i, f, variant=variant, **kw)
    bw = chunkwise_bw_raw(q, k, v, i, f, None, fw["C_states"], fw["n_out"], dh, variant=variant, **kw)
    x = [t.clone().requires_grad_(True) for t in (q, k, v, i, f)]
    if variant == _lib.EXP:
        h = mlstm_chunkwise__b200_xl_chunk(*x, recompute_states_in_bw=recompute, **kw)
    else:
        h = mlstm_siging_chunkwise__b200_xl_chunk(*x, normalize=variant == _lib.SIG, recompute_states_in_bw=recompute, **kw)
    assert torch.equal(h, fw["H"])
    grads = torch.autograd.grad(h, x, dh)
    for a, b in zip(grads[:3], bw[:3]):
        assert torch.equal(a, b)


# from the smallest of the rule (a chunk's blocks are no larger than its state); every gradient, the gates' among them
@pytest.mark.parametrize("DHQK, DHHV, L", [(64, 64, 64), (65, 190, 64), (64, 192, 128), (96, 128, 128), (130, 100, 128)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("recompute", [True, False])
def test_score_blocks_equal_scores_per_tile_in_every_gradient(DHQK, DHHV, L, dtype, recompute):
    assert DHQK * DHHV >= {64: 1, 128: 3}[L] * 64 * 64
    B, NH, S = 2, 3, 3 * L
    g = torch.Generator(device="cuda").manual_seed(DHQK + L)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x = [rnd(B, NH, S, d).to(dtype) for d in (DHQK, DHQK, DHHV)] + [rnd(B, NH, S), 3 + rnd(B, NH, S)]
    dh = rnd(B, NH, S, DHHV).to(dtype)
    kw = dict(chunk_size=L, impl="simt", eps=1e-6)
    fw = chunkwise_fw_raw(*x, variant=_lib.EXP, **kw)
    bw = chunkwise_bw_raw(*x, None, fw["C_states"], fw["n_out"], dh, variant=_lib.EXP, **kw)
    x = [t.requires_grad_(True) for t in x]
    h = mlstm_chunkwise__b200_xl_chunk(*x, recompute_states_in_bw=recompute, **kw)
    for a, b in zip((h, *torch.autograd.grad(h, x, dh)), (fw["H"], *bw[:5])):
        assert torch.equal(a, b)


def test_a_call_that_memory_is_too_short_for_does_without_the_score_blocks():
    """The allocator is kept (on the host) to less than the call takes with its score blocks, and to more than it needs."""
    B, NH, S, DHQK, DHHV, L = 1, 8, 16384, 64, 64, 64
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x = [rnd(B, NH, S, d).requires_grad_(True) for d in (DHQK, DHQK, DHHV)] + [rnd(B, NH, S).requires_grad_(True) for _ in "if"]
    dh = rnd(B, NH, S, DHHV)

    def call():
        torch.cuda.empty_cache()
        h = mlstm_chunkwise__b200_xl_chunk(*x, chunk_size=L, impl="simt")
        torch.cuda.empty_cache()
        return (h.detach(), *torch.autograd.grad(h, x, dh))

    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    want = call()
    most = torch.cuda.max_memory_reserved()
    blocks = 2 * B * NH * S // L * 64 * 64 * 4     # of the backward, where the call takes most
    want = [t.cpu() for t in want]
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((most - blocks // 2) / total)
        got = call()
        assert torch.cuda.max_memory_reserved() <= most
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for a, b in zip(got, want):
        assert torch.equal(a.cpu(), b)
