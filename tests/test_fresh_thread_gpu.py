"""The backward as the first CUDA work of its thread: no allocation reaches the driver, so nothing has bound a context."""

import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import torch
import mlstm_kernels_b200 as mk
pool = [torch.empty(1 << 28, device="cuda", dtype=torch.uint8) for _ in range(4)]
pool += [torch.empty(1 << 19, device="cuda", dtype=torch.uint8) for _ in range(64)]
del pool                                    # everything below comes out of the allocator's cache
q, k, v = (torch.randn(2, 4, 512, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(3))
i, f = (torch.randn(2, 4, 512, device="cuda", requires_grad=True) for _ in range(2))
for recompute in (True, False):
    h = mk.mlstm_chunkwise__b200_xl_chunk(q, k, v, i, f, recompute_states_in_bw=recompute)
    g = torch.autograd.grad(h, (q, k, v, i, f), torch.ones_like(h))
    torch.cuda.synchronize()
    assert all(torch.isfinite(x).all() for x in g)
"""


def test_backward_on_a_fresh_thread():
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, timeout=240)
    assert r.returncode == 0, r.stderr[-2000:]
