"""Rank-3 problems with head dim 32 or 96 on the tensor-core kernels: a box of 64 channels reaches into the next
head.  Forward and backward against the oracle at one and several heads (the last head's box leaves the tensor), ragged
tiles, GQA, additional tokens, and with a neighbouring head full of NaN."""
import numpy as np
import pytest
import torch

from natten_mps_b200 import _cabi
from natten_mps_b200 import functional as F
from tests._gpu_util import check, run_fused

pytestmark = pytest.mark.gpu

# name, spatial, B, Hq, Hkv, kernel, dilation, causal, D, extra tokens
CASES = [
    ("one_head", (3, 9, 11), 1, 1, 1, (3, 5, 5), (1, 1, 1), (False, False, False), 32, 0),
    ("d32_gqa", (5, 8, 21), 2, 4, 2, (3, 3, 7), (1, 2, 1), (True, False, False), 32, 0),
    ("d32_extra", (4, 13, 10), 1, 3, 3, (3, 5, 3), (1, 1, 2), (False, True, False), 32, 5),
    ("d96", (6, 7, 19), 2, 2, 1, (5, 3, 5), (1, 1, 1), (True, False, True), 96, 0),
    ("d32_tiles", (8, 28, 29), 1, 3, 3, (3, 5, 7), (1, 1, 1), (True, False, False), 32, 0),
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: c[0])
def test_rank3_head_dim_32_and_96(case, dtype):
    _, sp, B, Hq, Hkv, K, dil, causal, D, extra = case
    rng = np.random.default_rng(3)
    r = lambda *s: rng.standard_normal(s)
    ek, ev = (r(B, extra, Hkv, D), r(B, extra, Hkv, D)) if extra else (None, None)
    got, want = run_fused(3, dtype, r(B, *sp, Hq, D), r(B, *sp, Hkv, D), r(B, *sp, Hkv, D), r(B, *sp, Hq, D),
                          dict(kernel_size=K, dilation=dil, is_causal=causal), ek, ev)
    assert _cabi.last_path() == "tcgen05"
    for name in ("out", "dq", "dk", "dv") + (("dek", "dev") if extra else ()):
        check(name, got[name], want[name], dtype, scale_rel=True)


def test_heads_stay_apart():
    q, k, v = (torch.randn(1, 4, 8, 9, 3, 32, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    with torch.no_grad():
        want = F.na3d(q, k, v, kernel_size=(3, 3, 3))
        for t in (q, k, v):
            t[..., 1, :] = float("nan")
        got = F.na3d(q, k, v, kernel_size=(3, 3, 3))
    assert torch.equal(got[..., 0, :], want[..., 0, :]) and torch.equal(got[..., 2, :], want[..., 2, :])
