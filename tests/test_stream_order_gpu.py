"""Calls directly behind one another on a stream, without a wait of the host in between: a kernel may be scheduled while the one
before it still runs, and must not read what that one has yet to write."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import BF16

pytestmark = pytest.mark.gpu

# problems, keys, width: a decode with a cluster of 8 CTAs a problem, of 2, and with one CTA each
DECODE = [(8, 2000, 64), (100, 900, 128), (320, 500, 64)]
NAMES = {"bfloat16": BF16, "float16": np.dtype(np.float16), "float32": np.dtype(np.float32)}


@pytest.mark.parametrize("name", list(NAMES))
@pytest.mark.parametrize("shape", DECODE, ids=[f"{s[0]} x {s[1]} x {s[2]}" for s in DECODE])
def test_a_decode_step_between_the_kernel_that_writes_its_cache_and_the_one_that_reads_its_result(shape, name):
    """A forward whose O is the decode step's K and V; the decode step; a forward that has the decode step's O for keys and values.
    Each in turn with a wait of the host after it, then all at once, five times over buffers that were filled with something else."""
    from limn_b200 import runtime
    from limn_b200._lib import DTYPE_CODES, check, lib

    L = lib()
    runtime.set_device(0)
    bh, t, width = shape
    dtype, code = NAMES[name], DTYPE_CODES[name]
    rng = np.random.default_rng(sum(shape))
    rows = {"q": t, "k": t, "v": t, "one": 1, "last": 40}
    at = {key: runtime.upload(rng.standard_normal((bh, n, width)).astype(np.float32).astype(dtype)) for key, n in rows.items()}
    size = bh * width * dtype.itemsize
    cache, step, end = runtime.empty(size * t), runtime.empty(size), runtime.empty(size * 40)
    lse = [runtime.empty(bh * n * 4) for n in (t, 1, 40)]

    def forward(q, k, v, out, lse_out, t_q, t_k, causal):
        check(L.limn_b200_sdpa_fwd(q.ptr, k.ptr, v.ptr, None, out.ptr, lse_out.ptr, code, bh, t_q, t_k, width, width, causal, width**-0.5, None), "sdpa")

    def run(wait):
        forward(at["q"], at["k"], at["v"], cache, lse[0], t, t, 1)
        wait()
        forward(at["one"], cache, cache, step, lse[1], 1, t, 0)
        wait()
        forward(at["last"], step, step, end, lse[2], 40, 1, 0)
        runtime.synchronize()
        return [runtime.download(b, np.uint8, (b.nbytes,)) for b in (cache, step, end, *lse)]

    want = run(runtime.synchronize)
    assert np.isfinite(want[2].view(dtype).astype(np.float32)).all()
    for poison in (0xFF, 0x00, 0x3C, 0x7F, 0x42):
        for b in (cache, step, end, *lse):
            check(L.limn_b200_mem_set(b.ptr, poison, b.nbytes, None), "filling")
        for got, ref in zip(run(lambda: None), want, strict=True):
            np.testing.assert_array_equal(got, ref)
    assert runtime.device_status() == 0


@pytest.mark.parametrize("name", list(NAMES))
@pytest.mark.parametrize("shape", DECODE, ids=[f"{s[0]} x {s[1]} x {s[2]}" for s in DECODE])
def test_the_same_three_calls_as_a_graph(shape, name):
    """Captured once and replayed over buffers that were filled with something else: the edges between the calls hold there too."""
    import torch

    from limn_b200._lib import DTYPE_CODES, check, lib

    L = lib()
    bh, t, width = shape
    dtype = {"bfloat16": torch.bfloat16, "float16": torch.float16, "float32": torch.float32}[name]
    gen = torch.Generator(device="cuda").manual_seed(sum(shape))
    q, k, v, one, last = (torch.randn((bh, n, width), generator=gen, device="cuda").to(dtype) for n in (t, t, t, 1, 40))
    cache, step, end = torch.empty_like(q), torch.empty_like(one), torch.empty_like(last)
    lse = [torch.empty((bh, n), device="cuda") for n in (t, 1, 40)]

    def forward(q, k, v, out, lse_out, causal):
        stream = torch.cuda.current_stream().cuda_stream
        check(L.limn_b200_sdpa_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), None, out.data_ptr(), lse_out.data_ptr(), DTYPE_CODES[name], bh, q.shape[1],
                                   k.shape[1], width, width, causal, width**-0.5, stream), "sdpa")

    def run():
        forward(q, k, v, cache, lse[0], 1)
        forward(one, cache, cache, step, lse[1], 0)
        forward(last, step, step, end, lse[2], 0)

    results = (cache, step, end, *lse)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        run()
        stream.synchronize()
        want = [r.clone() for r in results]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            run()
            run()
        for value in (0.0, 3.5, float("nan")):
            for r in results:
                r.fill_(value)
            graph.replay()
            stream.synchronize()
            for got, ref in zip(results, want, strict=True):
                assert torch.equal(got, ref)
    graph.reset()
