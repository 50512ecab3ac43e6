"""The forward of a long sequence with few (batch, head) units, cut into segments: same bits as in one piece."""

import pytest
import torch

from mlstm_kernels_b200 import _lib
from mlstm_kernels_b200.chunkwise import mlstm_chunkwise__b200_xl_chunk, mlstm_siging_chunkwise__b200_xl_chunk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B, NH, S, DHQK, DHHV, dtype, gate", [
    (1, 8, 65536, 256, 512, torch.bfloat16, "exp"),      # half of the SMs, wide state tiles
    (1, 8, 90000, 256, 512, torch.float16, "exp"),       # ragged last chunk, segments of unequal length
    (2, 4, 33333, 136, 200, torch.bfloat16, "exp"),      # narrow state tiles, over the edge of both head dims
    (1, 8, 40961, 256, 256, torch.bfloat16, "sig"),      # one token in the last chunk
])
@pytest.mark.parametrize("initial", [False, True])
def test_segments_equal_one_piece(B, NH, S, DHQK, DHHV, dtype, gate, initial):
    g = torch.Generator(device="cuda").manual_seed(S)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k, v = (rnd(B, NH, S, d).to(dtype) for d in (DHQK, DHQK, DHHV))
    i, f = rnd(B, NH, S), rnd(B, NH, S) + 4.0
    kw = dict(c_initial=rnd(B, NH, DHQK, DHHV), n_initial=rnd(B, NH, DHQK)) if initial else {}
    if gate == "exp" and initial:
        kw["m_initial"] = rnd(B, NH, 1)
    fn = mlstm_chunkwise__b200_xl_chunk if gate == "exp" else mlstm_siging_chunkwise__b200_xl_chunk
    lib = _lib.load()
    run = lambda: fn(q, k, v, i, f, return_last_states=True, chunk_size=128, **kw)
    before = lib.mlstm_b200_set_unit_split(0)
    try:
        h0, last0 = run()
        lib.mlstm_b200_set_unit_split(1)
        h1, last1 = run()
    finally:
        lib.mlstm_b200_set_unit_split(before)
    assert torch.equal(h0, h1)
    for a, b in zip(last0, last1):
        assert (a is None and b is None) or torch.equal(a, b)


def test_segments_under_capture():
    q, k, v = (torch.randn(1, 4, 32768, d, device="cuda").bfloat16() for d in (256, 256, 512))
    i, f = torch.randn(1, 4, 32768, device="cuda"), torch.randn(1, 4, 32768, device="cuda") + 4.0
    run = lambda: mlstm_chunkwise__b200_xl_chunk(q, k, v, i, f, return_last_states=True, chunk_size=128)
    h0, last0 = run()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        h1, last1 = run()
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(h0, h1) and all(torch.equal(a, b) for a, b in zip(last0, last1))


def test_allocation_free_forward_keeps_one_stream():
    """Sizes that the regular entry point cuts into segments: the static one still takes them, with its fixed scratch."""
    B, NH, S, DHQK, DHHV = 1, 4, 88000, 256, 512
    q, k, v = (torch.randn(B, NH, S, d, device="cuda").bfloat16() for d in (DHQK, DHQK, DHHV))
    i, f = torch.randn(B, NH, S, device="cuda"), torch.randn(B, NH, S, device="cuda") + 4.0
    NC = -(-S // 128)
    h = torch.empty_like(v)
    n_out, m_out = torch.empty(B, NH, S, device="cuda"), torch.empty(B, NH, S, device="cuda")
    cs = torch.empty(B, NH, NC + 1, DHQK, DHHV, device="cuda", dtype=torch.bfloat16)
    ns, ms = torch.empty(B, NH, NC + 1, DHQK, device="cuda"), torch.empty(B, NH, NC + 1, device="cuda")
    p = lambda t: t.data_ptr()
    rc = _lib.load().mlstm_b200_chunkwise_fw_static(p(q), p(k), p(v), p(i), p(f), None, None, None, p(h), p(n_out), p(m_out),
                                                    p(cs), p(ns), p(ms), None, None, None, B, NH, S, DHQK, DHHV, 128,
                                                    _lib.BF16, _lib.F32, _lib.EXP, 0, 1e-6,
                                                    torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert torch.equal(h, mlstm_chunkwise__b200_xl_chunk(q, k, v, i, f, chunk_size=128))
