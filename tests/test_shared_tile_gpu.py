"""The 16-bit forward for problems of at most 128 query rows, whose key tiles both softmax groups share (even ones to the first,
odd ones to the second), and scores that are infinite or NaN on either of the two ways exp2 is taken."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import BF16, parity
from oracle import sdpa_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    import limn_standin as host

    return host.Device()


def _check(dev, q, k, v, do, mask=None):
    """Forward and backward against the oracle, at the tolerances of the other kernel tests."""
    import limn_standin as host

    half = q.dtype == np.dtype(np.float16)
    scale = q.shape[-1] ** -0.5
    att = host.Attention(dev, q, k, v, causal=False, key_mask=mask)
    out, lse = att.forward()
    want_out, want_lse = oracle.sdpa_forward(q, k, v, mask, causal=False, scale=scale)
    parity(out, want_out, 2e-3 if half else 2e-2, "O")
    parity(lse, want_lse, 1e-3, "L")
    dq, dk, dv = att.backward(do)
    delta = oracle.row_delta(do, want_out)
    want = (oracle.sdpa_backward_q(q, k, v, do, want_lse, delta, mask, causal=False, scale=scale),
            *oracle.sdpa_backward_kv(q, k, v, do, want_lse, delta, mask, causal=False, scale=scale))
    for got, ref, what in zip((dq, dk, dv), want, ("dQ", "dK", "dV")):
        parity(got, ref, 4e-3 if half else 2e-2, what)


def _problem(seed, bh, t_q, t_k, hd, dtype=BF16):
    rng = np.random.default_rng(seed)
    return [rng.standard_normal((bh, t, hd)).astype(np.float32).astype(dtype) for t in (t_q, t_k, t_k, t_q)]


# bh, t_q, t_k, hd: two key tiles (the second of a single key), three, an even number, more problems than SMs, t_q at and beside 128
SHARED = [(2, 5, 129, 64), (3, 100, 300, 64), (2, 128, 512, 128), (2, 127, 257, 96), (200, 6, 260, 64), (3, 129, 300, 64), (2, 64, 128, 64), (160, 33, 385, 32)]


@pytest.mark.parametrize("case", SHARED, ids=[f"{c[0]} x {c[1]}x{c[2]} hd {c[3]}" for c in SHARED])
@pytest.mark.parametrize("dtype", [BF16, np.float16], ids=["bf16", "f16"])
def test_problems_of_one_query_tile(case, dtype, dev):
    _check(dev, *_problem(sum(case), *case, dtype))


def _rows_and_lse(dev, q, k, v, mask=None):
    import limn_standin as host

    out, lse = host.Attention(dev, q, k, v, causal=False, key_mask=mask).forward()
    return out.view(np.uint16), lse.view(np.uint32)


@pytest.mark.parametrize("t_k", [129, 256], ids=["129 keys", "256 keys"])
@pytest.mark.parametrize("t_q", [16, 128])
def test_two_key_tiles_at_width_128_are_not_shared(t_q, t_k, dev):
    """Sharing those costs more than it saves. Unshared rows are those of a problem of two query tiles, bit for bit."""
    q, k, v, _ = _problem(t_q + t_k, 3, 200, t_k, 128)
    out, lse = _rows_and_lse(dev, q, k, v)
    head_out, head_lse = _rows_and_lse(dev, np.ascontiguousarray(q[:, :t_q]), k, v)
    np.testing.assert_array_equal(head_out, out[:, :t_q])
    np.testing.assert_array_equal(head_lse, lse[:, :t_q])


# bh, t_q, t_k, hd: more problems than SMs, so that a CTA has shared items one after the other; odd and even numbers of key tiles
MANY = [(333, 60, 300, 64), (333, 20, 130, 64), (200, 100, 400, 128)]


@pytest.mark.parametrize("masked", [False, True], ids=["", "masked"])
@pytest.mark.parametrize("case", MANY, ids=[f"{c[0]} x {c[1]}x{c[2]} hd {c[3]}" for c in MANY])
def test_many_shared_problems(case, masked, dev):
    bh, t_q, t_k, hd = case
    operands = _problem(sum(case), *case)
    mask = None
    if masked:
        rng = np.random.default_rng(bh + t_k)
        mask = ((np.arange(t_k) < rng.integers(1, t_k + 1, (bh, 1))) & (rng.random((bh, t_k)) < 0.9)).astype(np.float32)
        mask[:, 0] = 1
        mask = mask.astype(BF16)
    _check(dev, *operands, mask)


@pytest.mark.parametrize("masked", [False, True], ids=["", "masked"])
@pytest.mark.parametrize("case", MANY, ids=[f"{c[0]} x {c[1]}x{c[2]} hd {c[3]}" for c in MANY])
def test_a_row_has_the_same_bits_however_many_problems_there_are(case, masked, dev):
    bh, t_q, t_k, hd = case
    q, k, v, _ = _problem(sum(case), *case)
    mask = (np.arange(t_k) < 1 + np.arange(bh)[:, None] * t_k // bh).astype(np.float32).astype(BF16) if masked else None
    out, lse = _rows_and_lse(dev, q, k, v, mask)
    for p in (0, 150, bh - 1):
        alone_out, alone_lse = _rows_and_lse(dev, *(np.ascontiguousarray(a[p : p + 1]) for a in (q, k, v)), None if mask is None else mask[p : p + 1])
        np.testing.assert_array_equal(alone_out[0], out[p])
        np.testing.assert_array_equal(alone_lse[0], lse[p])


@pytest.mark.parametrize("t_k,hd", [(300, 128), (1300, 128), (200, 64), (700, 64)])
def test_l_of_shared_rows_is_as_good_as_of_unshared_ones(t_k, hd, dev):
    """Against float64, as a root mean square over 16 000 rows: the same rows in problems of 100 query rows, which are shared, and of
    200, which are not. Under a mask, where all exponentials are as good as float32's. 1 % for the rows' chance (1 / sqrt(2 x 16000))."""
    rng = np.random.default_rng(t_k + hd)
    bh, t_q = 160, 100
    q, k, v = (rng.standard_normal((bh, t, hd)).astype(np.float32).astype(np.float16) for t in (2 * t_q, t_k, t_k))
    keep = np.arange(t_k) < rng.integers(t_k // 2, t_k + 1, (bh, 1))
    mask = keep.astype(np.float16)
    scores = np.where(keep[:, None], np.matmul(q[:, :t_q].astype(np.float64), k.astype(np.float64).transpose(0, 2, 1)) * hd**-0.5, -np.inf)
    top = scores.max(-1, keepdims=True)
    want = (top + np.log(np.exp(scores - top).sum(-1, keepdims=True)))[..., 0]

    def off(rows):
        lse = _rows_and_lse(dev, np.ascontiguousarray(q[:, :rows]), k, v, mask)[1].view(np.float32)
        return np.sqrt(np.mean((lse.reshape(bh, rows)[:, :t_q] - want) ** 2))

    shared, alone = off(t_q), off(2 * t_q)
    assert shared <= 1.01 * alone, f"{shared:.3e} against {alone:.3e}"


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("hidden", ["even tiles", "odd tiles", "all but one key"])
def test_a_group_whose_keys_are_all_hidden(hd, hidden, dev):
    t_k = 640
    q, k, v, do = _problem(hd, 2, 40, t_k, hd)
    tile = np.arange(t_k) // 128
    keep = {"even tiles": tile % 2 == 1, "odd tiles": tile % 2 == 0, "all but one key": np.arange(t_k) == 300}[hidden]
    mask = np.broadcast_to(keep, (2, t_k)).astype(np.float32).astype(BF16)
    _check(dev, q, k, v, do, mask)


# t_q, t_k, causal: both parts of a shared problem; a tile and a row more than sharing takes; two Q tiles; three key tiles; causal
# rows that see the first tile whole, in part and as all there is
ROWS = [(40, 256, False), (128, 256, False), (129, 256, False), (200, 384, False), (300, 300, True)]


@pytest.mark.parametrize("masked", [False, True], ids=["", "masked"])
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("first", [0, 128], ids=["first tile", "second tile"])
@pytest.mark.parametrize("rows", ROWS, ids=[f"{r[0]}x{r[1]}{' causal' if r[2] else ''}" for r in ROWS])
def test_a_tile_whose_scores_are_all_minus_infinity(rows, first, hd, masked, dev):
    """It counts nothing, whether it is the first a row meets, one of two parts of the row, or all the row has."""
    import limn_standin as host

    t_q, t_k, causal = rows
    q, k, v, _ = _problem(hd + first, 2, t_q, t_k, hd)
    q = np.abs(q.astype(np.float32)).astype(BF16)
    k[:, first : first + 128] = -np.inf
    mask = np.ones((2, t_k), np.float32).astype(BF16) if masked else None
    out, lse = host.Attention(dev, q, k, v, causal=causal, key_mask=mask).forward()
    want_out, want_lse = oracle.sdpa_forward(q, k, v, mask, causal=causal, scale=hd**-0.5)
    assert np.isfinite(want_lse[:, 128 if first == 0 and causal else 0 :]).all()
    parity(out, want_out, 2e-2, "O")
    parity(lse, want_lse, 1e-3, "L")


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("t_q", [40, 200])
@pytest.mark.parametrize("masked", [False, True], ids=["", "masked"])
def test_a_nan_key_makes_every_row_nan(hd, t_q, masked, dev):
    """Whichever of a tile's columns it falls on: some take exp2 as a polynomial, the others on the special-function unit."""
    import limn_standin as host

    t_k = 300
    q, k, v, do = _problem(hd + t_q, 16, t_q, t_k, hd)
    for p in range(16):
        k[p, 19 * p] = np.nan  # the 16 residues of a column index mod 16, over all three tiles (up to key 285)
    mask = np.ones((16, t_k), np.float32).astype(BF16) if masked else None
    att = host.Attention(dev, q, k, v, causal=False, key_mask=mask)
    out, lse = att.forward()
    assert np.isnan(out.astype(np.float32)).all()
    assert np.isnan(lse.astype(np.float32)).all()
    dq, _, _ = att.backward(do)
    assert np.isnan(dq.astype(np.float32)).all()
