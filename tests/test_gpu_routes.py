"""Whatever kernel family a call goes to, the general kernels agree: drawn forms of every public operator (ranks, odd and even
kernels, dilation, stride, causal axes, head counts and dims, types, layouts of the inputs), forward and every gradient."""
import random

import numpy as np
import pytest
import torch

from natten_mps_b200 import _cabi
from tests._gpu_util import AV, FUSED, QK, VARLEN
from natten_mps_b200 import functional as F

pytestmark = pytest.mark.gpu
RPB = {1: F.na1d_qk_rpb, 2: F.na2d_qk_rpb, 3: F.na3d_qk_rpb}
# two orders of fp32 sums; 16 bits: where probabilities and logit gradients are rounded on the way to the tensor cores (2-norm)
BOUND = {torch.float32: 2e-5, torch.float16: 6e-3, torch.bfloat16: 4e-2}


def layout(rng, B, sp, H, D, dtype):
    r = lambda *s: torch.randn(*s, device="cuda").to(dtype)
    return {"dense": lambda: r(B, *sp, H, D), "packed": lambda: r(B, *sp, 3, H, D)[..., 1, :, :],
            "channels": lambda: r(B, *sp, H, D + 8)[..., :D], "heads": lambda: r(B, *sp, H + 2, D)[..., 1:H + 1, :],
            "heads_first": lambda: r(B, H, *sp, D).movedim(1, -2), "misaligned": lambda: r(B, *sp, H, D + 3)[..., 1:D + 1],
            }[rng.choice(["dense"] * 5 + ["packed", "packed", "channels", "channels", "heads", "heads_first", "misaligned"])]()


def draw(rng):
    while True:
        rank = rng.choice([1, 2, 2, 3, 3])
        top = {1: 3000, 2: 70, 3: 18}[rank]
        sp = tuple(int(round(4 * (top / 4) ** rng.random())) for _ in range(rank))
        api = rng.choice(["fused", "fused", "varlen", "split", "rpb"])
        K = tuple(rng.randint(1, min(n, {1: 70, 2: 13, 3: 6}[rank])) for n in sp)
        if api == "rpb" or rng.random() < 0.6:
            K = tuple(k - 1 + k % 2 for k in K)
        if min(K) < 1 or max(K) == 1:
            continue                                             # (a window of one key: gradients of the logits are zero)
        dil = tuple(rng.randint(1, min(n // k, 9)) if rng.random() < 0.4 else 1 for n, k in zip(sp, K))
        plain = api in ("varlen", "rpb")
        st = tuple(rng.randint(1, k) if not plain and rng.random() < 0.1 else 1 for k in K)
        causal = tuple(not plain and rng.random() < 0.3 for _ in K)
        if all(k >= n for k, n in zip(K, sp)) and not any(causal) and max(st) == 1:
            continue                                             # global attention
        kv = rng.choice([1, 2, 3, 4])
        heads = kv * (1 if api in ("split", "rpb") else rng.choice([1, 1, 2, 4]))
        extra = rng.choice([0, 0, 5, 16]) if api in ("fused", "varlen") else 0
        dtype = rng.choice([torch.float32, torch.float32, torch.bfloat16, torch.float16])
        return api, sp, K, dil, st, causal, rng.choice([1, 2, 3]), heads, kv, rng.choice([20, 32, 32, 32, 48, 64, 64, 96, 128]), dtype, extra


@pytest.mark.parametrize("seed", range(8))
def test_families_agree(seed):
    rng = random.Random(seed)
    torch.manual_seed(seed)
    served = set()
    for _ in range(40):
        case = draw(rng)
        api, sp, K, dil, st, causal, B, heads, kv, D, dtype, extra = case
        rank, osp = len(sp), tuple(-(-n // s) for n, s in zip(sp, st))
        q, k, v = (layout(rng, B, sp, h, D, dtype).requires_grad_() for h in (heads, kv, kv))
        go = layout(rng, B, osp, heads, D, dtype)
        r = lambda *s: torch.randn(*s, device="cuda").to(dtype)
        ek = {n: r(B, extra, kv, D).requires_grad_() for n in ("additional_keys", "additional_values")} if extra else {}
        w, gl = r(B, *osp, heads, int(np.prod(K))).softmax(-1).requires_grad_(), r(B, *osp, heads, int(np.prod(K)))
        rpb = r(heads, *[2 * x - 1 for x in K]).requires_grad_()
        sizes = torch.tensor([[rng.randint(k * d, n) for k, d, n in zip(K, dil, sp)] for _ in range(B)], device="cuda", dtype=torch.int32)

        def run():
            if api == "split":
                logits = QK[rank](q, k, K, dil, stride=st, is_causal=causal, scale=D ** -0.5)
                out = AV[rank](w, v, K, dil, stride=st, is_causal=causal)
                return [logits, out, *torch.autograd.grad(logits, [q, k], gl), *torch.autograd.grad(out, [w, v], go)]
            if api == "rpb":
                logits = RPB[rank](q, k, rpb, K, dil, scale=D ** -0.5)
                return [logits, *torch.autograd.grad(logits, [q, k, rpb], gl)]
            if api == "varlen":
                out = VARLEN[rank](q, k, v, sizes[:, 0] if rank == 1 else sizes, kernel_size=K, dilation=dil, **ek)
            else:
                out = FUSED[rank](q, k, v, kernel_size=K, stride=st, dilation=dil, is_causal=causal, **ek)
            return [out, *torch.autograd.grad(out, [q, k, v, *ek.values()], go)]

        got = run()
        served.add(_cabi.last_path())
        try:
            _cabi.set_force("simt")
            want = run()
        finally:
            _cabi.set_force(None)
        for i, (a, b) in enumerate(zip(got, want)):
            a, b = a.detach().double(), b.detach().double()
            assert torch.equal(torch.isfinite(a), torch.isfinite(b)), (i, case)
            a, b = (torch.where(torch.isfinite(t), t, 0) for t in (a, b))
            assert (a - b).norm() <= BOUND[dtype] * b.norm().clamp_min(1e-6), (i, case)
    assert _cabi.device_status() == 0
    assert served >= {"simt", "window", "tcgen05"}
