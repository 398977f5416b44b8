"""The layout entry points: operands held as (batch, t, heads, hd), read and written in place.

limn's frontend permutes such activations to (batch, heads, t, hd) and copies them dense before
every attention call (limn/tensor.py:561-562). The *_layout entry points reach the same rows
through the tensor maps' strides instead. The check is that they give, bit for bit, what the
dense entry points give on the permuted copies (every row is accumulated in the same order
either way), that the dense layout code is the dense entry point, and that one case also
matches the CPU oracle."""

from __future__ import annotations

import numpy as np
import pytest
from conftest import BF16, widen

from oracle import sdpa_oracle as oracle

pytestmark = pytest.mark.gpu

CASES = [
    # batch, heads, t_q, t_k, hd, causal, dtype
    (2, 3, 300, 300, 64, True, BF16),
    (1, 5, 257, 257, 128, True, BF16),
    (2, 2, 130, 390, 128, False, np.dtype(np.float16)),
    (3, 4, 128, 128, 64, False, BF16),
    (2, 3, 200, 200, 96, True, BF16),  # narrower heads run zero-padded in the 128 and the 64 kernel
    (2, 2, 150, 150, 40, False, np.dtype(np.float16)),
    (2, 3, 100, 300, 64, False, BF16),  # one query tile, key tiles shared by the two softmax groups
    (3, 2, 128, 400, 96, False, np.dtype(np.float16)),
]


def _run(layout: str, arrays, mask, batch, heads, t_q, t_k, hd, causal, dtype):
    """forward, delta, dQ, dK/dV through the layout entry points; arrays are in `layout` order."""
    from limn_b200 import runtime
    from limn_b200._lib import DTYPE_CODES, LAYOUT_CODES, check, lib

    L = lib()
    code = DTYPE_CODES["bfloat16" if dtype == BF16 else "float16"]
    q, k, v, do = (runtime.upload(a) for a in arrays)
    m = runtime.upload(mask) if mask is not None else None
    out, dq = runtime.empty(arrays[0].nbytes), runtime.empty(arrays[0].nbytes)
    dk, dv = runtime.empty(arrays[1].nbytes), runtime.empty(arrays[1].nbytes)
    lse, delta = runtime.empty(batch * heads * t_q * 4), runtime.empty(batch * heads * t_q * 4)
    tail = (LAYOUT_CODES[layout], code, batch, heads, t_q, t_k, hd, hd, int(causal), hd**-0.5, None)
    mp = m.ptr if m is not None else None
    check(L.limn_b200_sdpa_fwd_layout(q.ptr, k.ptr, v.ptr, mp, out.ptr, lse.ptr, *tail), "sdpa")
    check(L.limn_b200_sdpa_delta_layout(out.ptr, do.ptr, delta.ptr, LAYOUT_CODES[layout], code, batch, heads, t_q, hd, None), "row dot")
    check(L.limn_b200_sdpa_bwd_q_layout(q.ptr, k.ptr, v.ptr, do.ptr, lse.ptr, delta.ptr, mp, dq.ptr, *tail), "sdpa_bwd_q")
    check(L.limn_b200_sdpa_bwd_kv_layout(q.ptr, k.ptr, v.ptr, do.ptr, lse.ptr, delta.ptr, mp, dk.ptr, dv.ptr, *tail), "sdpa_bwd_kv")
    runtime.synchronize()
    assert runtime.device_status() == 0
    shape_q, shape_k = arrays[0].shape, arrays[1].shape
    return {
        "out": runtime.download(out, dtype, shape_q),
        "lse": runtime.download(lse, np.float32, (batch, heads, t_q)),
        "delta": runtime.download(delta, np.float32, (batch, heads, t_q)),
        "dq": runtime.download(dq, dtype, shape_q),
        "dk": runtime.download(dk, dtype, shape_k),
        "dv": runtime.download(dv, dtype, shape_k),
    }


def _inputs(seed, batch, heads, t_q, t_k, hd, dtype):
    rng = np.random.default_rng(seed)
    draw = lambda t: (rng.standard_normal((batch, heads, t, hd)).astype(np.float32) * 0.7).astype(dtype)
    q, k, v = draw(t_q), draw(t_k), draw(t_k)
    do = draw(t_q)
    return q, k, v, do


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"b{c[0]}h{c[1]}q{c[2]}k{c[3]}d{c[4]}{'c' if c[5] else 'f'}{c[6].name}")
def test_token_major_operands_give_the_dense_bits(case):
    batch, heads, t_q, t_k, hd, causal, dtype = case
    dense = _inputs(31, batch, heads, t_q, t_k, hd, dtype)
    token_major = tuple(np.ascontiguousarray(a.transpose(0, 2, 1, 3)) for a in dense)
    want = _run("bhtd", dense, None, *case)
    got = _run("bthd", token_major, None, *case)
    for name in ("out", "dq", "dk", "dv"):
        back = got[name].transpose(0, 2, 1, 3)
        np.testing.assert_array_equal(back.view(np.uint16), want[name].view(np.uint16), err_msg=name)
    for name in ("lse", "delta"):
        np.testing.assert_array_equal(got[name].view(np.uint32), want[name].view(np.uint32), err_msg=name)


def test_token_major_with_a_key_mask_matches_the_oracle():
    batch, heads, t, hd = 2, 3, 200, 64
    q, k, v, do = _inputs(32, batch, heads, t, t, hd, BF16)
    mask = np.ones((batch, heads, t), np.float32)
    mask[:, :, 150:] = 0
    mask[1, 2, 1::3] = 0
    mask = mask.astype(BF16)
    token_major = tuple(np.ascontiguousarray(a.transpose(0, 2, 1, 3)) for a in (q, k, v, do))
    got = _run("bthd", token_major, mask, batch, heads, t, t, hd, True, BF16)
    scale = hd**-0.5
    out, lse = oracle.sdpa_forward(q, k, v, mask, causal=True, scale=scale)
    delta = oracle.row_delta(do, out)
    dq = oracle.sdpa_backward_q(q, k, v, do, lse, delta, mask, causal=True, scale=scale)
    dk, dv = oracle.sdpa_backward_kv(q, k, v, do, lse, delta, mask, causal=True, scale=scale)
    for name, want in (("out", out), ("dq", dq), ("dk", dk), ("dv", dv)):
        err = np.abs(widen(got[name].transpose(0, 2, 1, 3)) - widen(want)).max()
        assert err <= 2e-2, f"{name}: {err}"
    assert np.abs(got["lse"] - lse[..., 0]).max() <= 1e-3
    assert (widen(got["dk"].transpose(0, 2, 1, 3))[:, :, 150:] == 0).all()


@pytest.mark.parametrize("hd,causal,t", [(64, True, 300), (128, False, 257), (80, True, 200)], ids=["d64 causal", "d128 full", "d80 causal"])
def test_slices_of_one_projection_buffer_give_the_dense_bits(hd, causal, t):
    """The strided entry points on what a transformer layer really holds: q, k, v as slices of one
    (batch, t, 3, heads, hd) projection output, dO and the results token-major, dK and dV written straight into a
    (batch, t, 2, heads, hd) buffer. Bit for bit what the dense entry points give on dense copies."""
    import ctypes

    from limn_b200 import runtime
    from limn_b200._lib import check, lib

    L = lib()
    batch, heads = 2, 3
    dense = _inputs(35, batch, heads, t, t, hd, BF16)
    want = _run("bhtd", dense, None, batch, heads, t, t, hd, causal, BF16)
    qkv = np.stack([a.transpose(0, 2, 1, 3) for a in dense[:3]], axis=2)  # (batch, t, 3, heads, hd)
    do = np.ascontiguousarray(dense[3].transpose(0, 2, 1, 3))               # (batch, t, heads, hd)
    qkv_dev, do_dev = runtime.upload(np.ascontiguousarray(qkv)), runtime.upload(do)
    row3, row2, row1 = 3 * heads * hd, 2 * heads * hd, heads * hd
    in_qkv = (t * row3, hd, row3)       # (batch, head, row) strides of a slice of the projection buffer
    token_major = (t * row1, hd, row1)
    in_kv_grad = (t * row2, hd, row2)
    q_ptr, k_ptr, v_ptr = (qkv_dev.ptr + i * row1 * 2 for i in range(3))
    out, dq = runtime.empty(do.nbytes), runtime.empty(do.nbytes)
    dkv = runtime.empty(2 * do.nbytes)
    lse, delta = runtime.empty(batch * heads * t * 4), runtime.empty(batch * heads * t * 4)
    arr = lambda *triples: (ctypes.c_longlong * (3 * len(triples)))(*[x for tr in triples for x in tr])
    tail = (2, batch, heads, t, t, hd, hd, int(causal), hd**-0.5, None)
    check(L.limn_b200_sdpa_fwd_strided(q_ptr, k_ptr, v_ptr, None, out.ptr, lse.ptr, arr(in_qkv, in_qkv, in_qkv, token_major), *tail), "sdpa")
    check(L.limn_b200_sdpa_bwd_q_fused_strided(q_ptr, k_ptr, v_ptr, out.ptr, do_dev.ptr, lse.ptr, None, dq.ptr, delta.ptr,
                                               arr(in_qkv, in_qkv, in_qkv, token_major, token_major, token_major), *tail), "dq")
    check(L.limn_b200_sdpa_bwd_kv_strided(q_ptr, k_ptr, v_ptr, do_dev.ptr, lse.ptr, delta.ptr, None, dkv.ptr, dkv.ptr + row1 * 2,
                                          arr(in_qkv, in_qkv, in_qkv, token_major, in_kv_grad, in_kv_grad), *tail), "dk, dv")
    runtime.synchronize()
    assert runtime.device_status() == 0
    got_out = runtime.download(out, BF16, (batch, t, heads, hd)).transpose(0, 2, 1, 3)
    got_dq = runtime.download(dq, BF16, (batch, t, heads, hd)).transpose(0, 2, 1, 3)
    got_dkv = runtime.download(dkv, BF16, (batch, t, 2, heads, hd))
    np.testing.assert_array_equal(got_out.view(np.uint16), want["out"].view(np.uint16))
    np.testing.assert_array_equal(runtime.download(lse, np.uint32, (batch, heads, t)), want["lse"].view(np.uint32))
    # the fused row dot sums in another order than the reduce kernel: gradients agree to a bfloat16 step
    for got, name in ((got_dq, "dq"), (got_dkv[:, :, 0].transpose(0, 2, 1, 3), "dk"), (got_dkv[:, :, 1].transpose(0, 2, 1, 3), "dv")):
        np.testing.assert_allclose(widen(got), widen(want[name]), rtol=2**-7, atol=2e-3, err_msg=name)
    # misuse is refused before anything is launched
    from limn_b200._lib import last_error

    bad = arr((t * row3, hd, row3 + 4), in_qkv, in_qkv, token_major)
    assert L.limn_b200_sdpa_fwd_strided(q_ptr, k_ptr, v_ptr, None, out.ptr, lse.ptr, bad, *tail) == 1 and "multiples of 8" in last_error()
    assert L.limn_b200_sdpa_fwd_strided(q_ptr, k_ptr, v_ptr, None, out.ptr, lse.ptr, None, *tail) == 1
    assert L.limn_b200_sdpa_fwd_strided(q_ptr, k_ptr, v_ptr, None, out.ptr, lse.ptr, arr(in_qkv, in_qkv, in_qkv, token_major),
                                        0, batch, heads, t, t, hd, hd, int(causal), hd**-0.5, None) == 2  # float32: not served strided


@pytest.mark.parametrize("t_q,t_k,hd", [(100, 300, 64), (128, 520, 128), (33, 129, 40)])
@pytest.mark.parametrize("masked", [False, True], ids=["", "masked"])
def test_cross_attention_out_of_a_key_value_projection_gives_the_dense_bits(t_q, t_k, hd, masked):
    """The strided forward where the two softmax groups share a problem's keys: q and O token-major, k and v slices of one
    (batch, t_k, 2, heads, hd) projection output."""
    import ctypes

    from limn_b200 import runtime
    from limn_b200._lib import check, lib

    L = lib()
    batch, heads = 3, 2
    q, k, v, do = _inputs(36, batch, heads, t_q, t_k, hd, BF16)
    mask = (np.arange(t_k) % 7 != 3).astype(np.float32).astype(BF16) * np.ones((batch, heads, 1), BF16) if masked else None
    want = _run("bhtd", (q, k, v, do), mask, batch, heads, t_q, t_k, hd, False, BF16)
    q_dev = runtime.upload(np.ascontiguousarray(q.transpose(0, 2, 1, 3)))
    kv_dev = runtime.upload(np.ascontiguousarray(np.stack([a.transpose(0, 2, 1, 3) for a in (k, v)], axis=2)))
    m_dev = runtime.upload(mask) if masked else None
    row1, row2 = heads * hd, 2 * heads * hd
    strides = (ctypes.c_longlong * 12)(*[t_q * row1, hd, row1], *[t_k * row2, hd, row2] * 2, *[t_q * row1, hd, row1])
    out, lse = runtime.empty(q.nbytes), runtime.empty(batch * heads * t_q * 4)
    check(L.limn_b200_sdpa_fwd_strided(q_dev.ptr, kv_dev.ptr, kv_dev.ptr + row1 * 2, m_dev.ptr if masked else None, out.ptr, lse.ptr, strides, 2, batch, heads,
                                       t_q, t_k, hd, hd, 0, hd**-0.5, None), "sdpa")
    assert runtime.device_status() == 0
    got = runtime.download(out, BF16, (batch, t_q, heads, hd)).transpose(0, 2, 1, 3)
    np.testing.assert_array_equal(got.view(np.uint16), want["out"].view(np.uint16))
    np.testing.assert_array_equal(runtime.download(lse, np.uint32, (batch, heads, t_q)), want["lse"].view(np.uint32))


@pytest.mark.parametrize("t_q,t_k,hd,causal", [(131, 131, 72, True), (100, 129, 120, False), (130, 70, 64, False), (33, 33, 8, True), (257, 250, 128, False), (96, 513, 40, False)])
def test_results_leave_what_lies_between_their_rows_alone(t_q, t_k, hd, causal):
    """Results whose rows, heads and batches have room between them: the epilogues exchange and stage pieces of neighbouring rows, and
    write the rows and columns there are, bit for bit, and nothing else."""
    import ctypes

    from limn_b200 import runtime
    from limn_b200._lib import check, lib

    L = lib()
    batch, heads = 2, 3
    dense = _inputs(41, batch, heads, t_q, t_k, hd, BF16)
    want = _run("bhtd", dense, None, batch, heads, t_q, t_k, hd, causal, BF16)
    q, k, v, do = (runtime.upload(a) for a in dense)

    def packed(t):
        return heads * t * hd, t * hd, hd

    def roomy(t):  # (batch, heads, t + 1, hd + 8)
        return heads * (t + 1) * (hd + 8), (t + 1) * (hd + 8), hd + 8

    def result(t):
        return runtime.empty(2 * batch * heads * (t + 1) * (hd + 8))

    out, dq, dk, dv = result(t_q), result(t_q), result(t_k), result(t_k)
    lse, delta = runtime.empty(batch * heads * t_q * 4), runtime.empty(batch * heads * t_q * 4)
    arr = lambda *triples: (ctypes.c_longlong * (3 * len(triples)))(*[x for tr in triples for x in tr])
    tail = (2, batch, heads, t_q, t_k, hd, hd, int(causal), hd**-0.5, None)
    a, b = packed(t_q), packed(t_k)
    check(L.limn_b200_sdpa_fwd_strided(q.ptr, k.ptr, v.ptr, None, out.ptr, lse.ptr, arr(a, b, b, roomy(t_q)), *tail), "sdpa")
    check(L.limn_b200_sdpa_bwd_q_fused_strided(q.ptr, k.ptr, v.ptr, out.ptr, do.ptr, lse.ptr, None, dq.ptr, delta.ptr, arr(a, b, b, roomy(t_q), a, roomy(t_q)), *tail), "dq")
    check(L.limn_b200_sdpa_bwd_kv_strided(q.ptr, k.ptr, v.ptr, do.ptr, lse.ptr, delta.ptr, None, dk.ptr, dv.ptr, arr(a, b, b, a, roomy(t_k), roomy(t_k)), *tail), "dk, dv")
    runtime.synchronize()
    assert runtime.device_status() == 0
    for buf, t, name in ((out, t_q, "out"), (dq, t_q, "dq"), (dk, t_k, "dk"), (dv, t_k, "dv")):
        got = runtime.download(buf, np.uint16, (batch, heads, t + 1, hd + 8))
        assert (got[:, :, t:] == 0xFFFF).all() and (got[..., hd:] == 0xFFFF).all(), name
        inner = np.ascontiguousarray(got[:, :, :t, :hd])
        if name == "out":
            np.testing.assert_array_equal(inner, want[name].view(np.uint16))
        else:  # the fused row dot sums in another order than the reduce kernel
            np.testing.assert_allclose(widen(inner.view(BF16)), widen(want[name]), rtol=2**-7, atol=2e-3, err_msg=name)


@pytest.mark.parametrize("t_q,t_k,hd", [(513, 200, 64), (700, 129, 40), (1100, 65, 64)])
def test_key_blocks_one_after_the_other_give_the_bits_of_one_alone(t_q, t_k, hd):
    """The dK/dV pass without masks from five query tiles on: a block's results are taken out while it is at its next item. More items
    than SMs, against launches of three problems."""
    batch, heads = 57, 3
    arrays = _inputs(43, batch, heads, t_q, t_k, hd, BF16)
    got = _run("bhtd", arrays, None, batch, heads, t_q, t_k, hd, False, BF16)
    for at in (0, 28, 49, 56):
        want = _run("bhtd", [x[at : at + 1] for x in arrays], None, 1, heads, t_q, t_k, hd, False, BF16)
        for name in ("dk", "dv", "dq", "out"):
            np.testing.assert_array_equal(got[name][at].view(np.uint16), want[name][0].view(np.uint16), err_msg=f"{name} of batch {at}")


@pytest.mark.parametrize("dtype", [BF16, np.dtype(np.float16)], ids=["bf16", "f16"])
@pytest.mark.parametrize("rows,all_rows,hd,causal", [(31, 127, 64, False), (79, 81, 64, False), (127, 128, 64, False), (200, 256, 64, False), (48, 49, 128, False), (32, 64, 128, True),
                                                     (127, 128, 128, False), (50, 70, 96, True), (77, 78, 80, False), (128, 130, 80, False), (40, 256, 48, False), (19, 255, 72, False)])
@pytest.mark.parametrize("batch", [1, 40])
def test_a_row_leaves_with_the_same_bits_in_every_way(rows, all_rows, hd, causal, dtype, batch):
    """Which way a kernel's rows leave depends on how many there are, of how many columns, and on how many problems: the first rows of a
    problem, on either side of those lines, are the rows of the shorter problem. A row of dK and dV does not see the other keys either,
    where it is given the row's own L and delta."""
    from limn_b200 import runtime
    from limn_b200._lib import DTYPE_CODES, check, lib

    L = lib()
    other, heads = (all_rows if causal else 100), 5
    bh, code = batch * heads, DTYPE_CODES["bfloat16" if dtype == BF16 else "float16"]
    q, k, v, do = (x.reshape(bh, -1, hd) for x in _inputs(45, batch, heads, all_rows, other, hd, dtype))
    up = lambda x: runtime.upload(np.ascontiguousarray(x))

    def forward_and_dq(n):
        t_k = n if causal else other
        ops = [up(x) for x in (q[:, :n], k[:, :t_k], v[:, :t_k], do[:, :n])]
        out, dq, lse, delta = (runtime.empty(size) for size in (2 * bh * n * hd, 2 * bh * n * hd, 4 * bh * n, 4 * bh * n))
        tail = (code, bh, n, t_k, hd, hd, int(causal), hd**-0.5, None)
        check(L.limn_b200_sdpa_fwd(ops[0].ptr, ops[1].ptr, ops[2].ptr, None, out.ptr, lse.ptr, *tail), "sdpa")
        check(L.limn_b200_sdpa_delta(out.ptr, ops[3].ptr, delta.ptr, code, bh * n, hd, None), "row dot")
        check(L.limn_b200_sdpa_bwd_q(ops[0].ptr, ops[1].ptr, ops[2].ptr, ops[3].ptr, lse.ptr, delta.ptr, None, dq.ptr, *tail), "dq")
        got = [runtime.download(out, np.uint16, (bh, n, hd)), runtime.download(dq, np.uint16, (bh, n, hd)), runtime.download(lse, np.uint32, (bh, n))]
        return got, lse, delta

    short, _, _ = forward_and_dq(rows)
    full, lse, delta = forward_and_dq(all_rows)
    for a, b, name in zip(short, full, ("out", "dq", "lse")):
        np.testing.assert_array_equal(a, b[:, :rows], err_msg=name)
    if causal:  # (its queries would be others)
        return

    def dkv(n):  # dK and dV of the first n rows of dO's problem taken as keys; the other side are the rows above
        ops = [up(x) for x in (q, do[:, :n], do[:, :n], q)]
        dk, dv = (runtime.empty(2 * bh * n * hd) for _ in range(2))
        check(L.limn_b200_sdpa_bwd_kv(ops[0].ptr, ops[1].ptr, ops[2].ptr, ops[3].ptr, lse.ptr, delta.ptr, None, dk.ptr, dv.ptr, code, bh, all_rows, n, hd, hd, 0, hd**-0.5, None), "dk, dv")
        return [runtime.download(x, np.uint16, (bh, n, hd)) for x in (dk, dv)]

    for a, b, name in zip(dkv(rows), dkv(all_rows), ("dk", "dv")):
        np.testing.assert_array_equal(a, b[:, :rows], err_msg=name)
    assert runtime.device_status() == 0


@pytest.mark.parametrize("dtype", [BF16, np.dtype(np.float16)], ids=["bf16", "f16"])
@pytest.mark.parametrize("t_q,hd", [(250, 64), (384, 56)])
def test_rows_staged_item_after_item_are_the_rows_of_one_item(t_q, hd, dtype):
    """A warp whose rows go by way of shared memory uses the same bytes for the next item's rows: more items than SMs, against one problem
    alone."""
    batch, heads = 80, 5
    arrays = _inputs(44, batch, heads, t_q, 100, hd, dtype)
    got = _run("bhtd", arrays, None, batch, heads, t_q, 100, hd, False, dtype)
    for at in (0, 41, 79):
        want = _run("bhtd", [x[at : at + 1, 4:] for x in arrays], None, 1, 1, t_q, 100, hd, False, dtype)
        for name in ("out", "dq"):
            np.testing.assert_array_equal(got[name][at, 4].view(np.uint16), want[name][0, 0].view(np.uint16), err_msg=f"{name} of batch {at}")


@pytest.mark.parametrize("t_q,t_k,hd", [(513, 200, 64), (1100, 65, 40)])
def test_key_blocks_one_after_the_other_in_half_precision(t_q, t_k, hd):
    """The deferred dK and dV as above, float16."""
    batch, heads, dtype = 57, 3, np.dtype(np.float16)
    arrays = _inputs(46, batch, heads, t_q, t_k, hd, dtype)
    got = _run("bhtd", arrays, None, batch, heads, t_q, t_k, hd, False, dtype)
    for at in (0, 28, 49, 56):
        want = _run("bhtd", [x[at : at + 1] for x in arrays], None, 1, heads, t_q, t_k, hd, False, dtype)
        for name in ("dk", "dv"):
            np.testing.assert_array_equal(got[name][at].view(np.uint16), want[name][0].view(np.uint16), err_msg=f"{name} of batch {at}")


def test_dense_layout_code_is_the_dense_entry_point():
    from limn_b200 import runtime
    from limn_b200._lib import check, lib

    L = lib()
    batch, heads, t, hd = 2, 2, 160, 64
    q, k, v, _ = _inputs(33, batch, heads, t, t, hd, BF16)
    bufs = [runtime.upload(a) for a in (q, k, v)]
    outs = []
    for which in range(2):
        out, lse = runtime.empty(q.nbytes), runtime.empty(batch * heads * t * 4)
        if which == 0:
            check(L.limn_b200_sdpa_fwd(*(b.ptr for b in bufs), None, out.ptr, lse.ptr, 2, batch * heads, t, t, hd, hd, 1, hd**-0.5, None), "sdpa")
        else:
            check(L.limn_b200_sdpa_fwd_layout(*(b.ptr for b in bufs), None, out.ptr, lse.ptr, 0, 2, batch, heads, t, t, hd, hd, 1, hd**-0.5, None), "sdpa")
        outs.append((runtime.download(out, BF16, q.shape), runtime.download(lse, np.float32, (batch * heads, t))))
    np.testing.assert_array_equal(outs[0][0].view(np.uint16), outs[1][0].view(np.uint16))
    np.testing.assert_array_equal(outs[0][1], outs[1][1])


def test_token_major_refuses_what_the_tensor_core_kernels_do_not_take():
    from limn_b200 import runtime
    from limn_b200._lib import last_error, lib

    L = lib()
    a = runtime.upload(np.zeros((1, 16, 2, 32), np.float32))
    out, lse = runtime.empty(a.nbytes), runtime.empty(2 * 16 * 4)
    code = L.limn_b200_sdpa_fwd_layout(a.ptr, a.ptr, a.ptr, None, out.ptr, lse.ptr, 1, 0, 1, 2, 16, 16, 32, 32, 0, 0.2, None)
    assert code == 2 and "contiguous" in last_error()
    assert L.limn_b200_last_launch_count() == 0
