"""float32 attention: what the tensor-core kernels of csrc/sdpa_f32_sm100.cu must keep of the CUDA-core kernels that
served these calls before them."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

FIRST_CALLS = """
import torch
from limn_b200._lib import check, lib

L = lib()
torch.manual_seed(0)
bh, t, d = 3, 200, 64
q, k, v, do = (torch.randn(bh, t, d, device="cuda") for _ in range(4))
out, dq, dk, dv = (torch.zeros_like(q) for _ in range(4))
lse, delta = (torch.zeros(bh, t, device="cuda") for _ in range(2))
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, capture_error_mode="global"):
    tail = (0, bh, t, t, d, d, 1, d**-0.5, torch.cuda.current_stream().cuda_stream)
    p = [x.data_ptr() for x in (q, k, v, out, do, lse, dq, delta, dk, dv)]
    check(L.limn_b200_sdpa_fwd(p[0], p[1], p[2], None, p[3], p[5], *tail), "sdpa")
    check(L.limn_b200_sdpa_bwd_q_fused(p[0], p[1], p[2], p[3], p[4], p[5], None, p[6], p[7], *tail), "sdpa_bwd_q_fused")
    check(L.limn_b200_sdpa_bwd_kv(p[0], p[1], p[2], p[4], p[5], p[7], None, p[8], p[9], *tail), "sdpa_bwd_kv")
graph.replay()
torch.cuda.synchronize()
args = [x.double().requires_grad_() for x in (q, k, v)]
s = (args[0] @ args[1].mT * d**-0.5).masked_fill(~torch.ones(t, t, dtype=torch.bool, device="cuda").tril(), -float("inf"))
want = s.softmax(-1) @ args[2]
want.backward(do.double())
for got, ref in zip((out, dq, dk, dv), (want.detach(), *(a.grad for a in args))):
    assert ((got - ref).norm() / ref.norm()).item() < 1e-5
"""


def test_the_first_float32_call_on_a_device_may_be_under_stream_capture():
    """Nothing is allocated and nothing waited for by a float32 forward and backward, the first call of a process included."""
    done = subprocess.run([sys.executable, "-c", FIRST_CALLS], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
