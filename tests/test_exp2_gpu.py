"""The probabilities of the 16-bit dQ pass, some of which take exp2 as a polynomial and the others on the special-function unit:
as accurate as each other, and infinite where the row's L makes them so. What the pass computes is dS = P (dP - delta); with one
key whose dP is 1, delta 0 and K a unit vector, a row's dQ is that key's P rounded to 16 bits."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import BF16

pytestmark = pytest.mark.gpu

KEYS = [17 * p % 128 for p in range(16)]  # one key a problem: every residue mod 16, in both halves of the tile
HALVES = pytest.mark.parametrize("dtype", [BF16, np.dtype(np.float16)], ids=["bf16", "f16"])
WIDTHS = pytest.mark.parametrize("width", [64, 128])


def _dq(q, k, v, do, lse):
    """dQ of (16, t, width) operands with delta = 0 and scale 1/8, through the plain entry point."""
    from limn_b200 import runtime
    from limn_b200._lib import DTYPE_CODES, check, lib

    runtime.set_device(0)
    bh, t_q, width = q.shape
    bufs = [runtime.upload(np.ascontiguousarray(a)) for a in (q, k, v, do, lse, np.zeros_like(lse))]
    dq = runtime.empty(q.nbytes, poison=0xFF)
    code = DTYPE_CODES["bfloat16" if q.dtype == BF16 else "float16"]
    check(lib().limn_b200_sdpa_bwd_q(*(b.ptr for b in bufs), None, dq.ptr, code, bh, t_q, k.shape[1], width, width, 0, 0.125, None), "dq")
    assert runtime.device_status() == 0
    return runtime.download(dq, q.dtype, q.shape).astype(np.float64)


def _one_key_each(width, dtype, rows):
    """q, k, v, dO with dP = 1 at problem p's key KEYS[p] and 0 elsewhere, and that key's K a unit vector; q is 0."""
    q, do = np.zeros((16, rows, width), dtype), np.zeros((16, rows, width), dtype)
    k, v = np.zeros((16, 128, width), dtype), np.zeros((16, 128, width), dtype)
    do[:, :, 0] = 1
    for p, key in enumerate(KEYS):
        k[p, key, 0] = 1
        v[p, key, 0] = 1
    return q, k, v, do


@HALVES
@WIDTHS
def test_probabilities_are_as_good_as_float32_exp2(width, dtype):
    """Scores are 0, so every P is exp(-L). L is put a few 1e-7 to either side of where P is half way between two 16-bit values:
    which one comes out says where the pass sees P.

    The bound: -L log2(e) is rounded once, with a constant good to 2^-25 (together 1e-7 of |x| <= 1, 0.7e-7 of P), and exp2 is
    within 2^-22 = 2.4e-7 (the documented error of ex2.approx; the polynomial's is 1.7e-7): 3.1e-7. Twice that is let pass."""
    bound = 6.2e-7
    step = 2.0**-8 if dtype == BF16 else 2.0**-11  # between two values in [1/2, 1)
    lower = 0.5 + step * np.round(np.linspace(0, 0.5 / step - 1, 24)).astype(int)
    halfway = lower + step / 2
    exact = -np.log(halfway)[:, None] + np.linspace(-3.2e-6, 3.2e-6, 43)
    lse = exact.astype(np.float32).ravel()
    truth = np.exp(-lse.astype(np.float64))
    middle, below = np.repeat(halfway, 43), np.repeat(lower, 43)
    off = truth / middle - 1
    want = np.where(off > 0, below + step, below) * 0.125
    sure = np.abs(off) > bound
    assert sure.sum() > 700 and (off[sure] > 0).any() and (off[sure] < 0).any()
    got = _dq(*_one_key_each(width, dtype, lse.size), np.broadcast_to(lse, (16, lse.size)).copy())[:, :, 0]
    wrong = (got != want) & sure
    assert not wrong.any(), f"{wrong.sum()} of {16 * sure.sum()}: P is off by up to {np.abs(np.broadcast_to(off, got.shape)[wrong]).max():.1e}"
    assert (np.abs(got - middle * 0.125) <= step * 0.0626).all()  # (the unsure ones are one of the two values)


@HALVES
@WIDTHS
def test_a_probability_beyond_float32_is_not_finite(width, dtype):
    """An L far below the row's scores, which cannot be this row's: exp2 of 128.4 and more. The gradient must show it."""
    c = np.array([89, 89.5, 90, 92, 96, 104, 128, 136, 160, 176, 200, 256, 264, 354, 512, 1024, 5000, 8000], np.float64)
    assert c[0] * 8 * 0.125 * np.log2(np.e) > 128
    q, k, v, do = _one_key_each(width, dtype, c.size)
    q[:, :, 1] = c.astype(dtype)
    k[:, :, 1] = -8
    for p, key in enumerate(KEYS):
        k[p, key, 1] = 8  # (the other keys' P is 0)
    got = _dq(q, k, v, do, np.zeros((16, c.size), np.float32))
    assert not np.isfinite(got).any()


@HALVES
@WIDTHS
def test_a_probability_below_float32_is_zero(width, dtype):
    """Down to 2^-126 a P is a number, below it nothing: not a subnormal one, whatever it is multiplied by."""
    c = np.array([0, 1, 80, 89, 89.5, 90, 96, 128, 200, 256, 354, 1024, 8000], np.float64)
    q, k, v, do = _one_key_each(width, dtype, c.size)
    q[:, :, 1] = c.astype(dtype)
    k[:, :, 1] = -8  # x from 0 to -1.4 c
    for p, key in enumerate(KEYS):
        do[p, :, 0] = 2.0**14  # dP as large as float16 has it
    got = _dq(q, k, v, do, np.zeros((16, c.size), np.float32))
    q64 = q[0, :, 1].astype(np.float64)
    p64 = np.exp(-q64)
    gone = q64 * np.log2(np.e) > 126.5
    assert gone.sum() >= 6
    assert (got[:, gone] == 0).all()
    kept = q64 * np.log2(np.e) < 10
    assert np.allclose(got[:, kept, 0], (p64 * 2.0**14 * 0.125)[kept], rtol=2**-8)


@HALVES
@WIDTHS
def test_a_nan_score_or_l_makes_the_row_nan(width, dtype):
    q, k, v, do = _one_key_each(width, dtype, 4)
    lse = np.zeros((16, 4), np.float32)
    lse[:, 1] = np.nan
    q[:, 2, 2] = np.nan
    got = _dq(q, k, v, do, lse)
    assert np.isnan(got[:, 1]).all() and np.isnan(got[:, 2]).all()
    assert np.isfinite(got[:, [0, 3]]).all()
