"""The fp32-arithmetic window kernels (four rows per lane group over a staged column box) and the one-pass bias gradient,
against the CPU oracle: ragged tiles, remainders of rows and columns, boxes larger than a chunk, clamped edges, causal axes,
dilation with uneven groups, GQA and the three ranks.  The split cases are as large as the kernels' size rule asks for."""
import numpy as np
import pytest
import torch

import oracle
from natten_mps_b200 import _backend, _cabi
from natten_mps_b200 import functional as F
from tests._gpu_util import check, poison, run_fused, same_finite_values

pytestmark = pytest.mark.gpu

# name, spatial, B, Hq, Hkv, kernel, dilation, causal, D
FUSED_CASES = [
    ("1d_smallest", (3,), 1, 1, 1, (2,), (1,), (False,), 32),
    ("1d_remainders", (515,), 2, 2, 1, (63,), (2,), (True,), 64),
    ("2d_tiles_plus_one", (17, 33), 1, 2, 2, (7, 7), (1, 1), (False, False), 32),
    ("2d_even_causal_dil", (23, 30), 1, 4, 2, (4, 6), (3, 2), (True, False), 32),
    ("2d_window_is_all", (9, 11), 2, 1, 1, (9, 11), (1, 1), (False, False), 128),
    ("2d_box_past_a_chunk", (40, 44), 1, 1, 1, (21, 19), (1, 1), (False, True), 128),
    ("3d_ragged", (5, 9, 14), 1, 2, 1, (3, 5, 7), (1, 1, 2), (True, False, False), 32),
    ("1d_d128", (261,), 2, 4, 2, (31,), (1,), (False,), 128),
    ("2d_d64_gqa", (21, 26), 1, 4, 2, (5, 9), (2, 1), (False, True), 64),
    ("2d_even", (23, 30), 1, 4, 2, (4, 6), (1, 1), (True, False), 32),
    ("3d_even", (5, 6, 13), 2, 4, 2, (4, 3, 2), (1, 2, 1), (False, False, False), 32),
    ("3d_even_causal", (9, 7, 10), 1, 2, 2, (2, 4, 3), (1, 1, 1), (False, True, False), 128),
    ("3d_d64", (4, 7, 11), 1, 2, 2, (3, 3, 5), (1, 2, 1), (False, True, False), 64),
]


def family(K, dil):
    """Even kernels on dilated axes stay on the general kernels."""
    return "simt" if any(k % 2 == 0 and d > 1 for k, d in zip(K, dil)) else "window"


@pytest.mark.parametrize("case", FUSED_CASES, ids=lambda c: c[0])
def test_fused_float32(case):
    _, sp, B, Hq, Hkv, K, dil, causal, D = case
    rng = np.random.default_rng(7)
    r = lambda h: rng.standard_normal((B, *sp, h, D))
    got, want = run_fused(len(sp), torch.float32, r(Hq), r(Hkv), r(Hkv), r(Hq),
                          dict(kernel_size=K, dilation=dil, is_causal=causal, return_lse=True))
    for name in ("out", "lse", "dq", "dk", "dv"):
        check(name, got[name], want[name], torch.float32)
    f = lambda h: torch.as_tensor(r(h)).float().cuda()       # (autograd runs the backward on a thread of its own)
    q, k, v, args = f(Hq), f(Hkv), f(Hkv), (K, (1,) * len(sp), dil, causal, D ** -0.5)
    out, lse = _backend.fused_forward(q, k, v, *args)
    assert _cabi.last_path() == family(K, dil)
    _backend.fused_backward(q, k, v, out, lse, f(Hq), *args)
    assert _cabi.last_path() == family(K, dil)


POISON_CASES = [c for c in FUSED_CASES if c[0] in ("1d_remainders", "2d_tiles_plus_one", "2d_box_past_a_chunk", "3d_ragged", "2d_even", "3d_d64")]


@pytest.mark.parametrize("value", [float("nan"), float("inf")], ids=["nan", "inf"])
@pytest.mark.parametrize("which", ["q", "k", "v", "dout"])
@pytest.mark.parametrize("case", POISON_CASES, ids=lambda c: c[0])
def test_fused_float32_reads_no_value_of_another_window(case, which, value):
    """Four rows share every column that is read; a NaN or Inf reaches the rows whose window holds it and no others."""
    _, sp, B, Hq, Hkv, K, dil, causal, D = case
    rng = np.random.default_rng(17)
    t = {n: rng.standard_normal((B, *sp, h, D)) for n, h in (("q", Hq), ("k", Hkv), ("v", Hkv), ("dout", Hq))}
    poison(t[which], 0, value, 0.3)
    got, want = run_fused(len(sp), torch.float32, t["q"], t["k"], t["v"], t["dout"],
                          dict(kernel_size=K, dilation=dil, is_causal=causal, return_lse=True))
    for name in ("out", "lse", "dq", "dk", "dv"):
        same_finite_values(name, got[name], want[name], torch.float32)


SPLIT_CASES = [
    ("2d_d32_ragged", (57, 61), 2, 4, 4, (7, 9), (1, 1), (False, False), 32),
    ("2d_d32_even_causal_dil", (66, 45), 2, 4, 4, (6, 12), (2, 3), (False, True), 32),
    ("1d_d32", (3001,), 3, 4, 4, (43,), (1,), (False,), 32),
    ("3d_d32", (6, 23, 25), 2, 4, 4, (3, 5, 5), (1, 1, 2), (True, False, False), 32),
    ("2d_d32_gqa", (45, 47), 2, 4, 2, (5, 3), (1, 2), (False, False), 32),
    ("2d_d32_even", (66, 45), 2, 4, 4, (6, 12), (1, 1), (False, True), 32),
    ("3d_d32_even", (7, 21, 23), 2, 4, 4, (4, 3, 4), (1, 2, 1), (False, False, True), 32),
]
# with these head dims the 16-bit types go to the tensor cores
SPLIT_FLOAT32_CASES = [
    ("1d_d64", (1999,), 1, 4, 2, (31,), (3,), (True,), 64),
    ("1d_d128", (1601,), 1, 2, 2, (43,), (1,), (False,), 128),
    ("2d_d64", (29, 31), 1, 4, 4, (7, 5), (1, 2), (False, False), 64),
    ("2d_d128", (27, 38), 2, 2, 1, (5, 9), (1, 1), (True, False), 128),
    ("3d_d64", (5, 13, 17), 2, 2, 2, (3, 5, 3), (1, 1, 2), (False, False, True), 64),
    ("3d_d128", (4, 14, 15), 1, 4, 4, (3, 3, 5), (1, 1, 1), (True, False, False), 128),
]
SPLIT_RUNS = [pytest.param(c, t, id=c[0] + "-" + str(t)[6:]) for c in SPLIT_CASES for t in (torch.float32, torch.bfloat16, torch.float16)]
SPLIT_RUNS += [pytest.param(c, torch.float32, id=c[0] + "-float32") for c in SPLIT_FLOAT32_CASES]


def split_products(q, k, v, do, w, gl, kw):
    """The six products of the split operators (logits and their gradients for `gl`, output and its for `do`), and the oracle's.
    Grouped heads exist below the public functions only."""
    n = lambda t: t.float().numpy()
    want = dict(logits=oracle.na_qk(n(q), n(k), **kw), out=oracle.na_av(n(w), n(v), **kw))
    want["dq"], want["dk"] = oracle.na_qk_backward(n(q), n(k), n(gl), **kw)
    want["dw"], want["dv"] = oracle.na_av_backward(n(w), n(v), n(do), **kw)
    if q.shape != k.shape:
        q, k, v, do, w, gl = (t.cuda() for t in (q, k, v, do, w, gl))
        args = (kw["kernel_size"], kw["dilation"], (1,) * (q.ndim - 3), kw["is_causal"])
        got = dict(logits=_backend.qk_forward(q, k, *args, None), out=_backend.av_forward(w, v, *args))
        got["dq"], got["dk"] = _backend.qk_backward(gl, q, k, *args, None)
        got["dw"], got["dv"] = _backend.av_backward(do, w, v, *args)
        return got, want
    qk, av = {1: (F.na1d_qk, F.na1d_av), 2: (F.na2d_qk, F.na2d_av), 3: (F.na3d_qk, F.na3d_av)}[q.ndim - 3]
    leaf = lambda t: t.cuda().requires_grad_(True)
    qd, kd, vd, wd = leaf(q), leaf(k), leaf(v), leaf(w)
    logits, out = qk(qd, kd, **kw), av(wd, vd, **kw)
    got = dict(logits=logits.detach(), out=out.detach())
    got["dq"], got["dk"] = torch.autograd.grad(logits, [qd, kd], gl.cuda())
    got["dw"], got["dv"] = torch.autograd.grad(out, [wd, vd], do.cuda())
    return got, want


@pytest.mark.parametrize("case,dtype", SPLIT_RUNS)
def test_split(case, dtype):
    _, sp, B, Hq, Hkv, K, dil, causal, D = case
    g = torch.Generator().manual_seed(5)
    r = lambda *s: torch.randn(*s, generator=g).to(dtype)
    q, k, v, do = r(B, *sp, Hq, D), r(B, *sp, Hkv, D), r(B, *sp, Hkv, D), r(B, *sp, Hq, D)
    w, gl = r(B, *sp, Hq, int(np.prod(K))), r(B, *sp, Hq, int(np.prod(K)))
    got, want = split_products(q, k, v, do, w, gl, dict(kernel_size=K, dilation=dil, is_causal=causal))
    for name in want:
        check(name, got[name], want[name], dtype, scale_rel=True)
    q, k, v, do, w, gl = (t.cuda() for t in (q, k, v, do, w, gl))
    args = (K, dil, (1,) * len(sp), causal)
    for call in (lambda: _backend.qk_forward(q, k, *args, None), lambda: _backend.qk_backward(gl, q, k, *args, None),
                 lambda: _backend.av_forward(w, v, *args), lambda: _backend.av_backward(do, w, v, *args)):
        call()
        assert _cabi.last_path() == family(K, dil)


@pytest.mark.parametrize("value", [float("nan"), float("inf")], ids=["nan", "inf"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("case", SPLIT_CASES, ids=lambda c: c[0])
def test_split_reads_no_value_of_another_window(case, dtype, value):
    _, sp, B, Hq, Hkv, K, dil, causal, D = case
    g = torch.Generator().manual_seed(19)
    r = lambda h, d: torch.randn(B, *sp, h, d, generator=g).to(dtype)
    q, k, v, do, w, gl = r(Hq, D), r(Hkv, D), r(Hkv, D), r(Hq, D), r(Hq, int(np.prod(K))), r(Hq, int(np.prod(K)))
    for head, (t, at) in enumerate(((q, 0.3), (k, 0.6), (v, 0.3), (do, 0.6))):
        poison(t, head % t.shape[-2], value, at)
    got, want = split_products(q, k, v, do, w, gl, dict(kernel_size=K, dilation=dil, is_causal=causal))
    for name in want:
        same_finite_values(name, got[name], want[name], dtype)


# at least as many rows as the kernels' size rule asks for
LOGIT_CASES = [((4003,), 2, (13,), (2,)), ((41, 53), 2, (7, 5), (1, 1)), ((37, 56), 2, (5, 9), (3, 2)), ((6, 19, 21), 2, (3, 5, 3), (1, 2, 1))]
LOGIT_RUNS = [(D, t) for D, t in ((32, torch.float32), (64, torch.float32), (128, torch.float32), (32, torch.bfloat16), (32, torch.float16))]


@pytest.mark.parametrize("D,dtype", LOGIT_RUNS, ids=lambda x: str(x).replace("torch.", ""))
@pytest.mark.parametrize("case", LOGIT_CASES, ids=lambda c: "x".join(map(str, c[0])))
def test_bias_added_to_the_logits(case, D, dtype):
    sp, B, K, dil = case
    g = torch.Generator().manual_seed(13)
    r = lambda *s: torch.randn(*s, generator=g).to(dtype)
    q, k, rpb = r(B, *sp, 2, D), r(B, *sp, 2, D), r(2, *[2 * x - 1 for x in K])
    fn = {1: F.na1d_qk_rpb, 2: F.na2d_qk_rpb, 3: F.na3d_qk_rpb}[len(sp)]
    got = fn(q.cuda(), k.cuda(), rpb.cuda(), K, dil, scale=D ** -0.5)
    assert _cabi.last_path() == "window"
    n = lambda t: t.double().numpy()
    want = oracle.na_qk_rpb(n(q), n(k), n(rpb), kernel_size=K, dilation=dil, scale=D ** -0.5)
    # the float32 sums, and one rounding to the tensors' type: with p significant bits (11, 8) half a unit in the last place is
    # at most 2^-p of the value
    half = {torch.float32: 0., torch.float16: 2. ** -11, torch.bfloat16: 2. ** -8}[dtype]
    err = np.abs(got.double().cpu().numpy() - want).max()
    assert err <= (1e-5 + half) * max(1., np.abs(want).max()), err


# the register part (interior positions), the table part (clamped edges, slots past the registers) and both cluster sizes
BIAS_CASES = [((95,), 12, 8, (13,), (1,)), ((40, 17), 2, 4, (7, 5), (1, 3)), ((29, 31), 1, 2, (17, 17), (1, 1)),
              ((30, 33), 1, 1, (23, 25), (1, 1)), ((5, 12, 14), 2, 2, (3, 5, 3), (1, 2, 1))]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("case", BIAS_CASES, ids=lambda c: "x".join(map(str, c[0])))
def test_bias_gradient_in_one_pass(case, dtype):
    sp, B, H, K, dil = case
    g = torch.Generator().manual_seed(11)
    r = lambda *s: torch.randn(*s, generator=g).to(dtype)
    q, k, rpb = r(B, *sp, H, 32), r(B, *sp, H, 32), r(H, *[2 * x - 1 for x in K])
    gl = r(B, *sp, H, int(np.prod(K)))
    rd = rpb.cuda().requires_grad_(True)
    fn = {1: F.na1d_qk_rpb, 2: F.na2d_qk_rpb, 3: F.na3d_qk_rpb}[len(sp)]
    (got,) = torch.autograd.grad(fn(q.cuda(), k.cuda(), rd, K, dil), [rd], gl.cuda())
    n = lambda t: t.float().numpy()
    _, _, want = oracle.na_qk_rpb_backward(n(q), n(k), n(rpb), n(gl), kernel_size=K, dilation=dil)
    check("drpb", got, want, dtype, scale_rel=True)


@pytest.mark.parametrize("inject", [2, 3], ids=["no_cluster_of_16", "no_cluster"])
def test_bias_gradient_where_the_cluster_finds_no_room(inject):
    try:
        _cabi.lib().natten_debug_wait(0, inject)
        test_bias_gradient_in_one_pass(BIAS_CASES[1], torch.float32)
    finally:
        _cabi.lib().natten_debug_wait(0, 0)


# every score far below -1e30 (a query against keys that a program pushed away); ties are exact, so the weights are 1 / n or 0
def test_scores_of_any_size():
    sp, H, D, K = (19, 23), 2, 32, (5, 7)
    q, k = np.zeros((1, *sp, H, D)), np.zeros((1, *sp, H, D))
    q[..., 0] = 1e17
    k[..., 0] = -1e17 * (1 + np.arange(19 * 23 * H).reshape(1, *sp, H) % 3)
    v = np.random.default_rng(23).standard_normal((1, *sp, H, D))
    f = lambda t: torch.as_tensor(t).float().cuda()
    for push in (1., -1.):
        out, lse = F.na2d(f(push * q), f(k), f(v), K, return_lse=True)
        want, want_lse = oracle.na_forward(push * q, k, v, K)
        check("out", out, want, torch.float32)
        check("lse", lse, want_lse, torch.float32)
    with np.errstate(all="ignore"):              # beyond float32: no key is left, 0 / 0 like torch.softmax over -inf
        assert torch.isnan(F.na2d(f(1e8 * q), f(1e8 * k), f(v), K)).all()
