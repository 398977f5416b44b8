"""float32 attention: what the tensor-core kernels of csrc/sdpa_f32_sm100.cu must keep of the CUDA-core kernels that
served these calls before them."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def dev():
    import limn_standin as host

    return host.Device()


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


def _problem(seed, bh, t_q, t_k, hd, hd_v):
    rng = np.random.default_rng(seed)
    return [rng.standard_normal((bh, t, w)).astype(np.float32) for t, w in ((t_q, hd), (t_k, hd), (t_k, hd_v), (t_q, hd_v))]


def _step(q, k, v, do, mask, causal, scale):
    """One training step's three calls; O, L, dQ, dK, dV."""
    from limn_b200 import runtime
    from limn_b200._lib import check, lib

    L = lib()
    (bh, t_q, hd), (t_k, hd_v) = q.shape, v.shape[1:]
    pq, pk, pv, pdo = (runtime.upload(a) for a in (q, k, v, do))
    pm = runtime.upload(mask) if mask is not None else None
    po, pl, pd, pdq, pdk, pdv = (runtime.empty(n) for n in (do.nbytes, 4 * bh * t_q, 4 * bh * t_q, q.nbytes, k.nbytes, v.nbytes))
    m = pm.ptr if pm is not None else None
    tail = (0, bh, t_q, t_k, hd, hd_v, int(causal), scale, None)
    check(L.limn_b200_sdpa_fwd(pq.ptr, pk.ptr, pv.ptr, m, po.ptr, pl.ptr, *tail), "sdpa")
    check(L.limn_b200_sdpa_bwd_q_fused(pq.ptr, pk.ptr, pv.ptr, po.ptr, pdo.ptr, pl.ptr, m, pdq.ptr, pd.ptr, *tail), "sdpa_bwd_q_fused")
    check(L.limn_b200_sdpa_bwd_kv(pq.ptr, pk.ptr, pv.ptr, pdo.ptr, pl.ptr, pd.ptr, m, pdk.ptr, pdv.ptr, *tail), "sdpa_bwd_kv")
    shapes = ((po, do.shape), (pl, (bh, t_q)), (pdq, q.shape), (pdk, k.shape), (pdv, v.shape))
    return [runtime.download(buf, np.float32, shape).astype(np.float64) for buf, shape in shapes]


def _step64(q, k, v, do, mask, causal, scale):
    q, k, v, do = (a.astype(np.float64) for a in (q, k, v, do))
    s = q @ k.transpose(0, 2, 1) * scale
    seen = np.ones(s.shape, bool)
    if causal:
        seen &= np.tril(np.ones(s.shape[1:], bool))
    if mask is not None:
        seen &= mask[:, None, :] != 0
    s = np.where(seen, s, -np.inf)
    top = s.max(-1, keepdims=True)
    p = np.exp(s - top)
    total = p.sum(-1, keepdims=True)
    p /= total
    out = p @ v
    ds = np.where(seen, p * (do @ v.transpose(0, 2, 1) - (do * out).sum(-1, keepdims=True)) * scale, 0)
    return [out, (top + np.log(total))[..., 0], ds @ k, ds.transpose(0, 2, 1) @ q, p.transpose(0, 2, 1) @ do]


def _compare(got, want, bound):
    for g, w, what in zip(got, want, ("O", "L", "dQ", "dK", "dV")):
        error = np.linalg.norm(g - w) / np.linalg.norm(w)
        assert error <= bound, f"{what}: {error:.2e} > {bound:.2e}"


BLOCKS = [(16, 40, 32, 32, False), (130, 130, 32, 24, True), (200, 200, 64, 64, True), (257, 300, 64, 33, False), (193, 193, 128, 128, True), (64, 129, 100, 128, False)]
BLOCK_IDS = [f"{a}x{b} hd {c}/{d} {'causal' if e else 'full'}" for a, b, c, d, e in BLOCKS]


@pytest.mark.parametrize("case", BLOCKS, ids=BLOCK_IDS)
def test_blocks_that_leave_the_tensor_cores_match_the_others(case):
    """An operand that has no bfloat16 pieces (here the largest float32, in hidden rows of V, where it counts for nothing)
    sends the blocks that meet it to the CUDA cores: every row of theirs, ragged ends and hidden keys included, against float64.
    The bound is that of the CUDA-core sums: sqrt(300) roundings of 2^-24, times 8."""
    t_q, t_k, hd, hd_v, causal = case
    q, k, v, do = _problem(t_q + hd, 3, t_q, t_k, hd, hd_v)
    mask = (np.random.default_rng(t_k).random((3, t_k)) > 0.2).astype(np.float32)
    mask[:, 0] = 1
    want = _step64(q, k, v, do, mask, causal, hd**-0.5)
    v[mask == 0] = np.finfo(np.float32).max
    got = _step(q, k, v, do, mask, causal, hd**-0.5)
    _compare(got, want, 8 * 300**0.5 * 2.0**-24)
    assert (got[3][mask == 0] == 0).all() and (got[4][mask == 0] == 0).all()


@pytest.mark.parametrize(("hd", "dtype"), [(32, np.float32), (64, np.float32), (128, np.float32), (192, np.float32), (36, np.float16)])
def test_a_row_whose_only_key_is_nan(hd, dtype, dev):
    """No running maximum sees a NaN score; the weight must."""
    import limn_standin as host

    q, k, v, _ = (a.astype(dtype) for a in _problem(hd, 2, 40, 40, hd, hd))
    k[0, 3, 1] = np.nan
    mask = np.ones((2, 40), dtype)
    mask[0, :3] = 0
    mask[0, 4:] = 0
    out, lse = host.Attention(dev, q, k, v, causal=True, key_mask=mask).forward()
    assert np.isnan(out[0].astype(np.float32)).all() and np.isnan(lse[0, 3:]).all() and np.isneginf(lse[0, :3]).all()
    assert np.isfinite(out[1].astype(np.float32)).all() and np.isfinite(lse[1]).all()


@pytest.mark.parametrize("hd", [32, 64, 100])
def test_a_query_whose_l_is_nan(hd):
    """dK and dV from operands that are finite and an L that is not: NaN for the keys that query sees (0 to 3), for the others what they are
    without it. A problem with no key at all (L is -inf throughout) beside it."""
    from limn_b200 import runtime
    from limn_b200._lib import check, lib

    q, k, v, do = _problem(47 + hd, 2, 150, 150, hd, hd)
    do[0, 3] = 0  # (query 3 adds nothing to any key when its weights are finite)
    mask = np.stack([np.ones(150, np.float32), np.zeros(150, np.float32)])
    want = _step64(q[:1], k[:1], v[:1], do[:1], None, True, hd**-0.5)
    lse, delta = (np.stack([x, np.full(150, fill)]).astype(np.float32) for x, fill in ((want[1][0], -np.inf), ((do[0] * want[0][0]).sum(-1), np.nan)))
    lse[0, 3] = np.nan
    ops = [runtime.upload(x) for x in (q, k, v, do, lse, delta, mask)]
    dk, dv = runtime.empty(k.nbytes), runtime.empty(v.nbytes)
    check(lib().limn_b200_sdpa_bwd_kv(*(x.ptr for x in ops), dk.ptr, dv.ptr, 0, 2, 150, 150, hd, hd, 1, hd**-0.5, None), "dk, dv")
    for got, w in ((runtime.download(dk, np.float32, k.shape), want[3]), (runtime.download(dv, np.float32, v.shape), want[4])):
        assert np.isnan(got[0, :4]).all() and (got[1] == 0).all()
        error = np.linalg.norm(got[0, 4:] - w[0, 4:]) / np.linalg.norm(w[0, 4:])
        assert error <= 8 * 150**0.5 * 2.0**-24, error


@pytest.mark.parametrize("hd", [32, 64, 128])
@pytest.mark.parametrize(("which", "power"), [("q", -118), ("v", -118), ("do", -118)])
def test_small_operands_keep_their_bits(which, power, hd):
    """Operands near the end of float32's range, whose third piece would lie below bfloat16's: the results keep the
    accuracy of float32 sums (the bound above; two pieces alone would leave 2^-17 of every operand)."""
    q, k, v, do = _problem(7 + hd, 2, 150, 150, hd, hd)
    scale = hd**-0.5
    small = np.float32(2.0**power)
    if which == "q":
        q, scale = q * small, scale * 2.0**60
        k = k * np.float32(2.0**58)
    elif which == "v":
        v = v * small
    else:
        do = do * small
    _compare(_step(q, k, v, do, None, True, scale), _step64(q, k, v, do, None, True, scale), 8 * 150**0.5 * 2.0**-24)


@pytest.mark.parametrize("hd", [32, 64, 128])
def test_small_gradients_keep_their_bits(hd):
    """dO is still large enough for its three pieces, dS (smaller by a probability and the scale) is not."""
    q, k, v, do = _problem(17 + hd, 2, 300, 300, hd, hd)
    do = (np.sign(do) * (1 + np.abs(do) % 1) * 2.0**-108).astype(np.float32)
    scale = hd**-0.5 / 256
    _compare(_step(q, k, v, do, None, False, scale), _step64(q, k, v, do, None, False, scale), 1.5e-6)


@pytest.mark.parametrize("hd", [24, 64, 100])
@pytest.mark.parametrize("scale", [-0.1, 0.0])
def test_scales_that_are_not_positive(scale, hd):
    """These stay on the tiled CUDA-core kernels at every width."""
    q, k, v, do = _problem(27 + hd, 2, 130, 130, hd, hd)
    got, want = _step(q, k, v, do, None, True, scale), _step64(q, k, v, do, None, True, scale)
    if scale == 0.0:
        assert (got[2] == 0).all() and (got[3] == 0).all()
        got[2], want[2], got[3], want[3] = got[0], want[0], got[0], want[0]
    _compare(got, want, 8 * 130**0.5 * 2.0**-24)


@pytest.mark.parametrize("hd", [8, 16, 24, 32, 72, 128])
def test_many_short_problems(hd):
    """Which kernels take a few hundred short problems depends on their number, sides and width: the edges of that rule, with
    and without masks, all against float64 (and so against one another)."""
    for bh, t_q, t_k, causal, masked in ((700, 16, 16, True, False), (700, 32, 33, False, True), (460, 64, 64, True, True), (700, 17, 64, False, False),
                                         (700, 64, 32, False, True), (160, 33, 16, False, False), (320, 64, 64, True, False), (600, 65, 64, False, False)):
        q, k, v, do = _problem(hd + t_q, bh, t_q, t_k, hd, hd)
        mask = None
        if masked:
            mask = (np.random.default_rng(t_k).random((bh, t_k)) > 0.2).astype(np.float32)
            mask[:, 0] = 1
        _compare(_step(q, k, v, do, mask, causal, hd**-0.5), _step64(q, k, v, do, mask, causal, hd**-0.5), 8 * 64**0.5 * 2.0**-24)


@pytest.mark.parametrize(("t", "hd", "hd_v", "which", "bound"), [(16, 24, 24, 4, 1.42e-7), (16, 24, 8, 2, 1.98e-7), (16, 24, 8, 3, 2.0e-7), (32, 16, 8, 3, 2.09e-7), (40, 12, 16, 3, 2.37e-7)])
def test_short_problems_stay_where_every_gradient_is_nearest(t, hd, hd_v, which, bound):
    """700 causal problems at head dims 24 and 16, where not every gradient of the tensor-core kernels is as near to float64 as the
    CUDA-core kernels': the bound lies half way between the two (the latter's are 1.39, 1.90, 1.96, 2.05 and 2.33e-7, and 0.2 % apart from seed to seed)."""
    q, k, v, do = _problem(t + hd, 700, t, t, hd, hd_v)
    got, want = (f(q, k, v, do, None, True, hd**-0.5)[which] for f in (_step, _step64))
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= bound


@pytest.mark.parametrize(("t_q", "t_k", "hd"), [(256, 256, 64), (256, 256, 48), (131, 200, 37)])
def test_truncated_scores_do_not_show_in_l(t_q, t_k, hd):
    """L against float64 over 32 problems: rounding it once leaves 2.6e-8; without the mean of what the scores' additions
    truncate put back it is 3.6e-8."""
    q, k, v, do = _problem(37 + hd, 32, t_q, t_k, hd, hd)
    causal = t_q == t_k
    got, want = (f(q, k, v, do, None, causal, hd**-0.5)[1] for f in (_step, _step64))
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 3.2e-8


@pytest.mark.parametrize(("bh", "t_q", "t_k", "hd", "hd_v", "causal"), [(4800, 70, 70, 32, 32, True), (4800, 66, 130, 64, 40, False), (300, 200, 200, 37, 33, True),
                                                                        (100, 257, 257, 64, 64, True), (37, 1000, 65, 24, 24, False), (320, 130, 130, 100, 128, True),
                                                                        (200, 129, 257, 128, 70, False), (4740, 33, 65, 80, 80, False)])
def test_a_problem_alone_and_among_many(bh, t_q, t_k, hd, hd_v, causal):
    """A block of the kernels that work in roles goes through several work items (one round, several, and more than a block may
    take): a problem has the same bits wherever it comes, also where the item before or after it leaves the tensor cores (hidden rows of V
    that do not split) and where the operands are not whole 16-byte pieces."""
    q, k, v, do = _problem(bh + t_q, bh, t_q, t_k, hd, hd_v)
    mask = np.ones((bh, t_k), np.float32)
    mask[:, -1] = 0
    v[[1, bh // 2, bh - 1], -1] = np.finfo(np.float32).max
    picks = sorted({0, 1, 2, 147 % bh, 148 % bh, 295 % bh, bh // 2 - 1, bh // 2, bh // 2 + 1, bh - 2, bh - 1})
    scale = hd**-0.5
    got = _step(q, k, v, do, mask, causal, scale)
    alone = _step(q[picks], k[picks], v[picks], do[picks], mask[picks], causal, scale)
    for g, a, what in zip(got, alone, ("O", "L", "dQ", "dK", "dV")):
        assert np.isfinite(g[:, :-1]).all(), what
        assert np.array_equal(g[picks], a), what


@pytest.mark.parametrize(("bh", "t_q", "t_k", "hd", "hd_v", "causal"), [(100, 17, 64, 32, 30, False), (149, 64, 64, 64, 64, True), (296, 16, 16, 32, 32, True), (592, 33, 40, 64, 37, False),
                                                                        (150, 70, 130, 28, 32, False), (75, 200, 200, 64, 40, True), (296, 128, 320, 64, 64, False), (98, 300, 65, 32, 25, False),
                                                                        (148, 64, 64, 64, 64, True), (300, 40, 64, 64, 50, False), (148, 16, 30, 32, 20, False), (120, 64, 33, 64, 64, False)])
def test_a_short_problem_alone_and_among_many(bh, t_q, t_k, hd, hd_v, causal):
    """The same on both sides of the rules that give short problems kernels without roles."""
    test_a_problem_alone_and_among_many(bh, t_q, t_k, hd, hd_v, causal)


@pytest.mark.parametrize(("t_q", "t_k", "hd_v", "causal"), [(130, 130, 64, True), (70, 200, 40, False), (200, 65, 100, False), (129, 129, 128, True), (33, 70, 17, False),
                                                            (70, 70, 200, False), (100, 100, 130, True)])
def test_rows_are_divided_to_the_nearest(t_q, t_k, hd_v, causal):
    """The forward's quotients (on the tensor cores, and in the tiled kernels above 128 columns) come from one reciprocal a row where the
    row's columns are of an ordinary size, from divisions where they are not. Powers of two go through everything else as they are: the same
    bits either way, so the former are rounded like the latter."""
    q, k, v, do = _problem(t_q + hd_v, 20, t_q, t_k, 32, hd_v)
    mask = np.ones((20, t_k), np.float32)
    ordinary = _step(q, k, v, do, mask, causal, 32**-0.5)[0]
    for power in (-45, 45, 100):
        scaled = _step(q, k, np.ldexp(v, power), np.zeros_like(do), mask, causal, 32**-0.5)[0]
        assert np.array_equal(np.ldexp(ordinary, power), scaled), power


@pytest.mark.parametrize(("t", "hd", "hd_v", "causal"), [(130, 32, 200, True), (130, 64, 64, True), (130, 32, 128, False), (70, 40, 130, True)])
def test_columns_far_smaller_than_their_neighbours_are_divided_to_the_nearest(t, hd, hd_v, causal):
    """Two columns of V are 2^-116 of the others (in the second run one of them is of their size): the quotients are those of the column at
    that size, bit for bit, in the tiled kernels and where the tensor cores hand items to them. V lies between 1 and 2 and scores are small, so the
    sums scale exactly."""
    q, k, v, do = _problem(t + hd_v, 64, t, t, hd, hd_v)
    v = 1 + np.abs(v) % 1
    small = np.float32(2.0**-116)
    v[..., [2, hd_v - 1]] *= small
    mixed = _step(0.5 * q, k, v, do, None, causal, hd**-0.5)[0]
    v[..., 2] /= small
    other = _step(0.5 * q, k, v, do, None, causal, hd**-0.5)[0]
    other[..., 2] *= small
    assert np.array_equal(mixed, other)


@pytest.mark.parametrize(("hd", "hd_v"), [(32, 200), (192, 96)])
def test_a_zero_keeps_its_sign(hd, hd_v):
    """Columns that the first keys take below zero and later ones, of far larger scores, scale to a zero of that sign, and of a quotient of that
    sign."""
    t_q, t_k = 70, 144  # (whole tiles of keys: a padding key would add a positive zero)
    q, k = np.ones((2, t_q, hd), np.float32), np.zeros((2, t_k, hd), np.float32)
    k[:, 128:] = 300.0
    v = np.full((2, t_k, hd_v), -1.0, np.float32)
    v[:, 128:] = -0.0
    v[:, 128:, ::2] = 1.5
    out = _step(q, k, v, np.zeros((2, t_q, hd_v), np.float32), None, False, 1.0)[0]
    assert (out[..., ::2] == 1.5).all() and (out[..., 1::2] == 0).all() and np.signbit(out[..., 1::2]).all()
