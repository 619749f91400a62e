"""What the performance work of this package is measured on.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` builds what a
program has in hand before a call, ``run`` makes one pass through the public entry points, ``work`` counts the
bytes and operations a pass cannot do without and ``tolerance`` says how far another correct implementation may
be off.  Inputs are N(0, 1), like the benchmark's and the tests'.

A case is a flat dict:

    api        fused  na{1,2,3}d                                       varlen  na{1,2,3}d_varlen
               split  na{1,2,3}d_qk[_rpb] -> softmax -> na{1,2,3}d_av  module  NeighborhoodAttention{1,2,3}D
    train      forward and backward (gradients of every input) or forward only, without autograd
    dtype      float32 | float16 | bfloat16
    batch, size ("64x64"), heads, kv_heads, dim, kernel, dilation, stride ("7x7"), causal ("01": per axis)
    extra      additional key/value tokens per sample          fill  (varlen) shortest sample, percent of the extent
"""
import torch

import natten_mps_b200 as nb
from natten_mps_b200 import functional as F

_FUSED = {1: F.na1d, 2: F.na2d, 3: F.na3d}
_VARLEN = {1: F.na1d_varlen, 2: F.na2d_varlen, 3: F.na3d_varlen}
_QK = {1: F.na1d_qk, 2: F.na2d_qk, 3: F.na3d_qk}
_QK_RPB = {1: F.na1d_qk_rpb, 2: F.na2d_qk_rpb, 3: F.na3d_qk_rpb}
_AV = {1: F.na1d_av, 2: F.na2d_av, 3: F.na3d_av}
_DTYPE = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}
_WIDTH = {"float32": 4, "float16": 2, "bfloat16": 2}


def _case(name, api, train, dtype, batch, size, heads, dim, kernel, dilation=None, stride=None, causal=None,
          kv_heads=None, extra=0, fill=100, rpb=False):
    rank = size.count("x") + 1
    ones = "x".join(["1"] * rank)
    return {"name": name, "api": api, "train": train, "dtype": dtype, "batch": batch, "size": size, "heads": heads,
            "kv_heads": kv_heads or heads, "dim": dim, "kernel": kernel, "dilation": dilation or ones,
            "stride": stride or ones, "causal": causal or "0" * rank, "extra": extra, "fill": fill, "rpb": rpb}


def listed():
    return [
        # A toy or test-sized training step in the default data type: a handful of launches, all latency.
        _case("1d_f32_tiny_train", "fused", True, "float32", 2, "128", 4, 32, "7"),
        # One layer of an image backbone at batch 1, last stage: interactive inference.
        _case("2d_bf16_small_infer", "fused", False, "bfloat16", 1, "28x28", 8, 32, "7x7"),
        # An odd-sized dense-prediction input in half precision, head dim 32, rectangular window, forward only.
        _case("2d_f16_ragged_infer", "fused", False, "float16", 2, "135x241", 6, 32, "7x9"),
        # Training in the default data type (float32), the size of a backbone's first stage.
        _case("2d_f32_train", "fused", True, "float32", 4, "56x56", 4, 32, "7x7"),
        # The benchmark's workload: a bf16 training step on 64 x 64 feature maps.
        _case("2d_bf16_train", "fused", True, "bfloat16", 8, "64x64", 8, 64, "7x7"),
        # Dilated training step with a large window on 128 x 128 maps.
        _case("2d_bf16_dilated_train", "fused", True, "bfloat16", 4, "128x128", 8, 64, "13x13", dilation="2x2"),
        # Video training step, causal in time.
        _case("3d_bf16_causal_train", "fused", True, "bfloat16", 2, "16x32x32", 8, 64, "3x7x7", causal="100"),
        # Prefill of a decoder with sliding-window attention: causal, grouped heads, ragged length, forward only.
        _case("1d_bf16_causal_prefill", "fused", False, "bfloat16", 2, "8191", 16, 128, "255", causal="1", kv_heads=4),
        # Long ragged sequences with register tokens, training step.
        _case("1d_f16_varlen_train", "varlen", True, "float16", 8, "16384", 16, 128, "255", kv_heads=4, extra=16, fill=25),
        # Split operators with a relative position bias (the weights are wanted, or dropout sits on them), training step.
        _case("2d_bf16_split_rpb_train", "split", True, "bfloat16", 4, "56x56", 4, 32, "7x7", rpb=True),
        # Split operators with head dim 64 and no bias, forward only (attention maps for inspection).
        _case("2d_f16_split_infer", "split", False, "float16", 2, "61x67", 8, 64, "9x9"),
        # The module inside a network: projections, attention on strided views, gradients of the parameters.
        _case("2d_bf16_module_train", "module", True, "bfloat16", 2, "48x60", 12, 32, "7x7"),
    ]


# ---------------------------------------------------------------------------
# drawn cases
# ---------------------------------------------------------------------------
def _log(rng, lo, hi):
    """An integer of [lo, hi], spread over its logarithm; odd and even alike."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _odd(rng, lo, hi):
    return rng.randrange(lo | 1, hi + 1, 2)


def _join(values):
    return "x".join(str(v) for v in values)


_LARGEST = {}        # the listed cases' largest cost per kind, filled on first use


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def draw(rng):
    """A family of use first, then sizes over its whole range; too large ones are drawn again."""
    if not _LARGEST:
        _LARGEST["any"] = max(_cost(c) for c in listed())
        _LARGEST["float32"] = 2 * max(_cost(c) for c in listed() if c["dtype"] == "float32")
        _LARGEST["split"] = 2 * max(_cost(c) for c in listed() if c["api"] == "split")
    while True:
        c = _draw(rng)
        cost = _cost(c)
        if cost > 0.8 * _LARGEST["any"]:
            continue
        if c["dtype"] == "float32" and cost > _LARGEST["float32"]:
            continue
        if c["api"] == "split" and cost > _LARGEST["split"]:
            continue
        c.pop("name")
        return c


def _draw(rng):
    family = rng.choice(["image", "image", "image", "float32", "video", "sequence", "varlen", "split", "module"])
    train = rng.random() < 0.6
    half = rng.choice(["bfloat16", "bfloat16", "float16"])
    if family == "image":
        h = _log(rng, 14, 160)
        w = max(14, min(256, int(h * rng.choice([1, 1, 4 / 3, 16 / 9]))))
        k = _odd(rng, 3, 13)
        k2 = k if rng.random() < 0.7 else _odd(rng, 3, 13)
        d = rng.choice([1, 1, 1, 2, 3])
        d = max(1, min(d, h // k, w // k2))
        s = 2 if d == 1 and k >= 3 and rng.random() < 0.15 else 1
        heads = rng.choice([2, 3, 4, 6, 8, 12, 16])
        return _case("", "fused", train, half, _log(rng, 1, 16), _join([h, w]), heads, rng.choice([32, 32, 64, 64, 128]),
                     _join([k, k2]), dilation=_join([d, d]), stride=_join([s, s]))
    if family == "float32":
        rank = rng.choice([1, 2, 2, 3])
        if rank == 1:
            size, kernel = [_log(rng, 64, 4096)], [_odd(rng, 3, 33)]
        elif rank == 2:
            h = _log(rng, 14, 80)
            size, kernel = [h, max(14, int(h * rng.choice([1, 1.3])))], [_odd(rng, 3, 11)] * 2
        else:
            size, kernel = [_log(rng, 4, 12), _log(rng, 14, 32), _log(rng, 14, 32)], [3, _odd(rng, 3, 7), _odd(rng, 3, 7)]
        return _case("", "fused", train, "float32", _log(rng, 1, 8), _join(size), rng.choice([2, 4, 6, 8]),
                     rng.choice([32, 32, 64]), _join(kernel))
    if family == "video":
        size = [_log(rng, 4, 24), _log(rng, 14, 48), _log(rng, 14, 48)]
        kernel = [rng.choice([3, 3, min(5, size[0] | 1)]), _odd(rng, 3, 9), _odd(rng, 3, 9)]
        kernel[0] = min(kernel[0], size[0] - 1 + size[0] % 2)
        causal = rng.choice(["100", "000"])
        return _case("", "fused", train, half, _log(rng, 1, 4), _join(size), rng.choice([2, 4, 6, 8]), rng.choice([32, 64]),
                     _join(kernel), causal=causal)
    if family in ("sequence", "varlen"):
        length = _log(rng, 512, 16384)
        kernel = min(_odd(rng, 15, 511), length // 4 * 2 - 1)
        kv = rng.choice([1, 2, 4, 8])
        heads = kv * rng.choice([1, 2, 4])
        dim = rng.choice([64, 128, 128])
        if family == "varlen":
            fill = rng.randint(50, 90)
            return _case("", "varlen", train, half, _log(rng, 2, 8), str(length), heads, dim, str(kernel), kv_heads=kv,
                         extra=rng.choice([0, 0, 4, 16]), fill=fill)
        return _case("", "fused", train, half, _log(rng, 1, 4), str(length), heads, dim, str(kernel),
                     causal=rng.choice(["1", "1", "0"]), kv_heads=kv, extra=rng.choice([0, 0, 0, 8]))
    if family == "split":
        h = _log(rng, 14, 96)
        k = _odd(rng, 3, 11)
        return _case("", "split", train, half, _log(rng, 1, 8), _join([h, max(14, int(h * rng.choice([1, 1.2])))]),
                     rng.choice([2, 3, 4, 8]), rng.choice([32, 32, 64]), _join([k, k]), rpb=rng.random() < 0.5)
    h = _log(rng, 14, 80)
    heads = rng.choice([4, 6, 8, 12])
    return _case("", "module", train, half, _log(rng, 1, 8), _join([h, max(14, int(h * rng.choice([1, 1.25])))]), heads,
                 rng.choice([32, 64]), _join([_odd(rng, 3, 11)] * 2), kv_heads=rng.choice([heads, heads, heads // 2]))


# ---------------------------------------------------------------------------
# inputs and one pass
# ---------------------------------------------------------------------------
def _ints(text):
    return [int(x) for x in text.split("x")]


def _geometry(case):
    size = _ints(case["size"])
    return (len(size), size, _ints(case["kernel"]), _ints(case["dilation"]), _ints(case["stride"]),
            [c == "1" for c in case["causal"]])


def _outputs(case):
    _, size, _, _, stride, _ = _geometry(case)
    return [-(-n // s) for n, s in zip(size, stride)]


def prepare(case, seed):
    rank, size, kernel, dilation, stride, causal = _geometry(case)
    dtype, train, B = _DTYPE[case["dtype"]], case["train"], case["batch"]
    heads, kv, dim = case["heads"], case["kv_heads"], case["dim"]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, grad=train):
        t = torch.randn(*shape, device="cuda", dtype=torch.float32, generator=g).to(dtype)
        return t.requires_grad_(grad)

    state = {"case": case, "rank": rank, "kernel": tuple(kernel), "dilation": tuple(dilation), "stride": tuple(stride),
             "causal": tuple(causal)}
    if case["api"] == "module":
        channels = heads * dim
        cls = {1: nb.NeighborhoodAttention1D, 2: nb.NeighborhoodAttention2D, 3: nb.NeighborhoodAttention3D}[rank]
        module = cls(channels, heads, tuple(kernel), num_kv_heads=kv).to(device="cuda", dtype=dtype)
        with torch.no_grad():                     # the usual initialisation, from the seed
            for name, p in sorted(module.named_parameters()):
                p.copy_(torch.randn(p.shape, device="cuda", generator=g) * (channels ** -0.5 if p.ndim > 1 else 0.02))
                p.requires_grad_(train)
        x = normal(B, *size, channels)
        state.update(module=module, leaves=[x] + [p for _, p in sorted(module.named_parameters())], x=x)
        if train:
            state["dout"] = normal(B, *size, channels, grad=False)
        return state
    q, k, v = normal(B, *size, heads, dim), normal(B, *size, kv, dim), normal(B, *size, kv, dim)
    state.update(q=q, k=k, v=v, leaves=[q, k, v], extra={})
    if case["extra"]:
        ek, ev = normal(B, case["extra"], kv, dim), normal(B, case["extra"], kv, dim)
        state["extra"] = {"additional_keys": ek, "additional_values": ev}
        state["leaves"] += [ek, ev]
    if case["rpb"]:
        state["rpb"] = normal(heads, *[2 * n - 1 for n in kernel])
        state["leaves"].append(state["rpb"])
    if case["api"] == "varlen":                   # lengths as the batch's collate function left them, on the GPU
        low = [max(kk * d, n * case["fill"] // 100) for n, kk, d in zip(size, kernel, dilation)]
        lens = torch.stack([torch.randint(lo, n + 1, (B,), device="cuda", generator=g) for lo, n in zip(low, size)], dim=1)
        state["sizes"] = (lens[:, 0] if rank == 1 else lens).to(torch.int32).contiguous()
    if train:
        state["dout"] = normal(B, *_outputs(case), heads, dim, grad=False)
    return state


def _forward(state):
    case, rank = state["case"], state["rank"]
    if case["api"] == "module":
        return state["module"](state["x"])
    q, k, v, kernel, dilation = state["q"], state["k"], state["v"], state["kernel"], state["dilation"]
    if case["api"] == "fused":
        return _FUSED[rank](q, k, v, kernel_size=kernel, stride=state["stride"], dilation=dilation,
                            is_causal=state["causal"], **state["extra"])
    if case["api"] == "varlen":
        return _VARLEN[rank](q, k, v, state["sizes"], kernel_size=kernel, dilation=dilation, **state["extra"])
    scale = case["dim"] ** -0.5
    if case["rpb"]:
        logits = _QK_RPB[rank](q, k, state["rpb"], kernel, dilation, scale=scale)
    else:
        logits = _QK[rank](q, k, kernel, dilation, scale=scale)
    attn = torch.softmax(logits, dim=-1)
    out = _AV[rank](attn, v, kernel, dilation)
    return out if case["train"] else (attn, out)


def run(state):
    if not state["case"]["train"]:
        with torch.no_grad():
            return _forward(state)
    out = _forward(state)
    grads = torch.autograd.grad(out, state["leaves"], state["dout"])
    return [out.detach(), *grads]


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how exact it is
# ---------------------------------------------------------------------------
def work(case):
    """Every input read once and every output written once; 4 operations per (query, key, channel) forward and 8
    backward.  Samples of varying length are counted at their expected length (their outputs in full: the rows
    past the length are written too).  The split operators hand logits and weights to the caller: those are
    written by one operator and read by the next, forward and backward."""
    rank, size, kernel, dilation, stride, causal = _geometry(case)
    width, B, heads, kv, dim = _WIDTH[case["dtype"]], case["batch"], case["heads"], case["kv_heads"], case["dim"]
    outs = _outputs(case)
    tokens = queries = pairs = 1.0
    share = (1 + case["fill"] / 100) / 2 if case["api"] == "varlen" else 1.0
    slots = 1
    for n, o, k, d, s, c in zip(size, outs, kernel, dilation, stride, causal):
        tokens *= n
        queries *= o
        slots *= k
        pairs *= sum(min(k, p // d + 1) for p in range(0, n, s)) if c else o * k
    tokens, queries, pairs = B * tokens, B * queries, B * share * pairs * heads
    pairs += B * share * (queries / B) * case["extra"] * heads
    q_in, kv_in = tokens * share * heads * dim, tokens * share * kv * dim
    out, extra = queries * heads * dim, 2.0 * B * case["extra"] * kv * dim
    train = case["train"]
    flops = (12 if train else 4) * pairs * dim
    values = queries * share * heads * dim * (1 if not train else 2) + 2 * kv_in + out + extra   # q (and dout), k, v; out
    if train:
        values += tokens * heads * dim + 2 * tokens * kv * dim + extra                          # dq, dk, dv
    if case["api"] == "split":
        values += queries * heads * slots * (11 if train else 4)
    if case["api"] == "module":
        channels = heads * dim
        params = channels * (2 * channels + 2 * kv * dim)
        qkv = q_in + 2 * kv_in
        flops += (6 if train else 2) * tokens * params
        # x -> q, k, v -> attention -> projection, each stage's tensors written by one operator and read by the next
        values += 2 * tokens * channels + qkv + out + params
        if train:
            values += 2 * tokens * channels + 2 * qkv + 2 * out + params
    return {"bytes": values * width, "flops": flops}


def tolerance(case):
    """Two correct implementations differ by the order of their sums and, in 16 bits, by where probabilities and
    gradients are rounded on the way to the tensor cores."""
    return {"rel": {"float32": 1e-5, "float16": 2e-3, "bfloat16": 1e-2}[case["dtype"]]}
