"""The give-up path of the bounded waits, walked end to end without hanging or faulting anything.

Every wait in the tensor-core kernels (on a TMA copy, on the tensor pipe, on another warp) is bounded: when
its budget runs out the kernel records 0x5741rrbb in the device's status word and returns, and kernels that
start while the word is set stand down. limn_b200_wait_probe makes exactly that happen with a
one-warp kernel of its own that waits a few microseconds on a barrier nobody arrives at; the production
kernels are not touched. The test then checks what the rest of the library promises about that state."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
from conftest import BF16

pytestmark = pytest.mark.gpu


def _forward(L, check, runtime, q, k, v, shape, poison=0xFF):
    bh, t, d = shape
    out, lse = runtime.empty(bh * t * d * 2, poison=poison), runtime.empty(bh * t * 4, poison=poison)
    check(L.limn_b200_sdpa_fwd(q.ptr, k.ptr, v.ptr, None, out.ptr, lse.ptr, 2, bh, t, t, d, d, 1, d**-0.5, None), "sdpa")
    return out, lse


def test_a_wait_that_runs_out_is_reported_and_the_device_recovers():
    from limn_b200 import runtime
    from limn_b200._lib import DEVICE_TIMEOUT, check, last_error, lib

    L = lib()
    runtime.set_device(0)
    assert runtime.device_status() == 0
    shape = (40, 300, 128)  # 120 work items: enough CTAs to show that every one of them stands down
    rng = np.random.default_rng(31)
    q, k, v = (runtime.upload(rng.standard_normal(shape).astype(np.float32).astype(BF16)) for _ in range(3))
    out, lse = _forward(L, check, runtime, q, k, v, shape)
    good = runtime.download(out, np.uint16, shape), runtime.download(lse, np.uint32, shape[:2])

    # 1. the wait runs out: status code in the word, the probe's own flag says it gave up, the kernel returned
    gave_up = runtime.empty(4, poison=0)
    check(L.limn_b200_wait_probe(20000, gave_up.ptr, None), "wait probe")
    # 2. a production launch enqueued while the word is set writes nothing
    out2, lse2 = _forward(L, check, runtime, q, k, v, shape, poison=0xAB)
    runtime.synchronize()
    assert runtime.download(gave_up, np.uint32, (1,))[0] == 1
    assert (runtime.download(out2, np.uint8, (out2.nbytes,)) == 0xAB).all(), "a kernel ran although an earlier one had given up"
    assert (runtime.download(lse2, np.uint8, (lse2.nbytes,)) == 0xAB).all()
    # 3. the word is read as an error, once
    word = ctypes.c_uint(0)
    assert L.limn_b200_device_status(ctypes.byref(word)) == DEVICE_TIMEOUT
    assert word.value == 0x57417E57
    assert "gave up on a bounded wait" in last_error() and "57417e57" in last_error()
    assert L.limn_b200_device_status(ctypes.byref(word)) == 0 and word.value == 0
    # 4. and the next launches are right again: the aborted launch left its work counters at zero
    for _ in range(3):
        out3, lse3 = _forward(L, check, runtime, q, k, v, shape)
        np.testing.assert_array_equal(runtime.download(out3, np.uint16, shape), good[0])
        np.testing.assert_array_equal(runtime.download(lse3, np.uint32, shape[:2]), good[1])
    assert runtime.device_status() == 0


# bh, t_q, t_k, width, causal: more items than SMs, of one and two tiles, so that a producer draws from the work counter before it
# has to wait; one query tile against two key tiles (shared keys); long streams, which it has to wait in at its first item
STANDING_DOWN = [(300, 100, 100, 64, 0), (300, 100, 100, 128, 1), (200, 100, 200, 64, 0), (200, 60, 250, 128, 0), (20, 900, 900, 64, 1), (20, 900, 900, 128, 0)]


@pytest.mark.parametrize("shape", STANDING_DOWN, ids=[f"{s[0]} x {s[1]}x{s[2]} width {s[3]}{' causal' if s[4] else ''}" for s in STANDING_DOWN])
def test_every_kernel_stands_down_and_leaves_nothing_behind(shape):
    from limn_b200 import runtime
    from limn_b200._lib import DEVICE_TIMEOUT, check, lib

    L = lib()
    runtime.set_device(0)
    assert runtime.device_status() == 0
    bh, t_q, t_k, width, causal = shape
    rng = np.random.default_rng(sum(shape))
    q, k, v, do = (runtime.upload(rng.standard_normal((bh, t, width)).astype(np.float32).astype(BF16)) for t in (t_q, t_k, t_k, t_q))
    tail = (2, bh, t_q, t_k, width, width, causal, width**-0.5, None)
    rows, keys = bh * t_q, bh * t_k
    sizes = {"out": rows * width * 2, "lse": rows * 4, "delta": rows * 4, "dq": rows * width * 2, "fused_delta": rows * 4,
             "fused_dq": rows * width * 2, "dk": keys * width * 2, "dv": keys * width * 2}
    known = {}

    def launch(poison):
        """All four calls; the backward ones on the first launch's O, L and delta."""
        to = {name: runtime.empty(size, poison=poison) for name, size in sizes.items()}
        o = known or to
        check(L.limn_b200_sdpa_fwd(q.ptr, k.ptr, v.ptr, None, to["out"].ptr, to["lse"].ptr, *tail), "sdpa")
        if not known:
            check(L.limn_b200_sdpa_delta(o["out"].ptr, do.ptr, to["delta"].ptr, 2, rows, width, None), "row dot")
        check(L.limn_b200_sdpa_bwd_q(q.ptr, k.ptr, v.ptr, do.ptr, o["lse"].ptr, o["delta"].ptr, None, to["dq"].ptr, *tail), "dq")
        check(L.limn_b200_sdpa_bwd_q_fused(q.ptr, k.ptr, v.ptr, o["out"].ptr, do.ptr, o["lse"].ptr, None, to["fused_dq"].ptr, to["fused_delta"].ptr, *tail), "dq")
        check(L.limn_b200_sdpa_bwd_kv(q.ptr, k.ptr, v.ptr, do.ptr, o["lse"].ptr, o["delta"].ptr, None, to["dk"].ptr, to["dv"].ptr, *tail), "dk, dv")
        runtime.synchronize()
        return to

    def bytes_of(buffers):
        return {name: runtime.download(buffers[name], np.uint8, (size,)) for name, size in sizes.items() if name != "delta"}

    known.update(launch(0xFF))
    good = bytes_of(known)
    check(L.limn_b200_wait_probe(20000, None, None), "wait probe")
    for name, seen in bytes_of(launch(0xAB)).items():
        if name == "fused_delta" and t_k > 512:
            continue  # (long dense problems have a kernel of their own for it, which waits for nothing and runs regardless)
        assert (seen == 0xAB).all(), f"{name} was written although an earlier kernel had given up"
    word = ctypes.c_uint(0)
    assert L.limn_b200_device_status(ctypes.byref(word)) == DEVICE_TIMEOUT and word.value == 0x57417E57
    for _ in range(2):
        for name, seen in bytes_of(launch(0xAB)).items():
            np.testing.assert_array_equal(seen, good[name], err_msg=name)
    assert runtime.device_status() == 0


# dK and dV deferred (more items than SMs, and fewer); rows staged and exchanged; own rows of few
@pytest.mark.parametrize("shape", [(100, 600, 200, 64, 0), (20, 700, 100, 40, 0), (300, 250, 100, 64, 0), (160, 250, 130, 80, 0), (300, 40, 40, 128, 1)], ids=str)
def test_deferred_results_and_row_stores_stand_down(shape):
    test_every_kernel_stands_down_and_leaves_nothing_behind(shape)


# bh, t_q, t_k, hd, causal: in roles with one item to a block, several, and operands fetched ahead; two blocks to an SM; one-tile items; above head dim
# 64; rows that are not whole 16-byte pieces
FLOAT32_STANDING_DOWN = [(20, 300, 300, 64, 1), (100, 500, 500, 32, 0), (400, 129, 257, 64, 0), (200, 64, 200, 64, 0), (120, 64, 64, 64, 1), (148, 20, 30, 32, 0),
                         (160, 200, 200, 128, 1), (200, 150, 150, 30, 0)]


@pytest.mark.parametrize("shape", FLOAT32_STANDING_DOWN, ids=str)
def test_every_float32_kernel_stands_down_and_leaves_nothing_behind(shape):
    from limn_b200 import runtime
    from limn_b200._lib import DEVICE_TIMEOUT, check, lib

    L = lib()
    runtime.set_device(0)
    assert runtime.device_status() == 0
    bh, t_q, t_k, hd, causal = shape
    rng = np.random.default_rng(sum(shape))
    mask_host = (rng.random((bh, t_k)) > 0.1).astype(np.float32)
    mask_host[:, 0] = 1
    q, k, v, do, mask = (runtime.upload(x) for x in (*(rng.standard_normal((bh, t, hd)).astype(np.float32) for t in (t_q, t_k, t_k, t_q)), mask_host))
    tail = (0, bh, t_q, t_k, hd, hd, causal, hd**-0.5, None)
    rows, keys = 4 * bh * t_q, 4 * bh * t_k
    sizes = {"out": rows * hd, "lse": rows, "delta": rows, "dq": rows * hd, "dk": keys * hd, "dv": keys * hd}
    known = {}

    def launch(poison):
        """The three kernels and, the first time, the row dot, which waits for nothing; the backward ones on the first launch's L and delta."""
        to = {name: runtime.empty(size, poison=poison) for name, size in sizes.items()}
        given = known or to
        check(L.limn_b200_sdpa_fwd(q.ptr, k.ptr, v.ptr, mask.ptr, to["out"].ptr, to["lse"].ptr, *tail), "sdpa")
        if not known:
            check(L.limn_b200_sdpa_delta(to["out"].ptr, do.ptr, to["delta"].ptr, 0, bh * t_q, hd, None), "row dot")
        check(L.limn_b200_sdpa_bwd_q(q.ptr, k.ptr, v.ptr, do.ptr, given["lse"].ptr, given["delta"].ptr, mask.ptr, to["dq"].ptr, *tail), "dq")
        check(L.limn_b200_sdpa_bwd_kv(q.ptr, k.ptr, v.ptr, do.ptr, given["lse"].ptr, given["delta"].ptr, mask.ptr, to["dk"].ptr, to["dv"].ptr, *tail), "dk, dv")
        runtime.synchronize()
        return to

    def bytes_of(buffers):
        return {name: runtime.download(buffers[name], np.uint8, (size,)) for name, size in sizes.items() if name != "delta"}

    known.update(launch(0xFF))
    good = bytes_of(known)
    check(L.limn_b200_wait_probe(20000, None, None), "wait probe")
    for name, seen in bytes_of(launch(0xAB)).items():
        assert (seen == 0xAB).all(), f"{name} was written although an earlier kernel had given up"
    word = ctypes.c_uint(0)
    assert L.limn_b200_device_status(ctypes.byref(word)) == DEVICE_TIMEOUT and word.value == 0x57417E57
    for _ in range(2):
        for name, seen in bytes_of(launch(0xAB)).items():
            np.testing.assert_array_equal(seen, good[name], err_msg=name)
    assert runtime.device_status() == 0


def test_finish_raises_like_a_failed_kernel_of_the_reference():
    """limn_b200.install() wraps the device's finish(): after a batch in which one of our Runners ran, a set
    status word surfaces as RuntimeError("cuda: ..."), where limn raises for a failed kernel of its own."""
    import limn_b200
    from limn_b200 import registry, runtime
    from limn_b200._lib import check, lib

    class Device:
        def __init__(self):
            self.custom = {}
            self.synchronised = 0

        def finish(self):
            runtime.synchronize()
            self.synchronised += 1

    dev = limn_b200.install(Device())
    dev.finish()  # nothing of ours ran: no status read, nothing raised
    check(lib().limn_b200_wait_probe(5000, None, None), "wait probe")
    dev.finish()  # still nothing of ours in the batch: the word is not even looked at
    registry._note_launch()  # what every Runner does
    with pytest.raises(RuntimeError, match=r"cuda: waiting for the batch: a limn_b200 kernel gave up on a bounded wait \(status 0x57417e57\)"):
        dev.finish()
    dev.finish()
    assert dev.synchronised == 4 and runtime.device_status() == 0
