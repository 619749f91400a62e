"""Split operators on tensor cores around the number of slots where their weights leave room for a third CTA on an SM (101 at head
dim 64): value product and dQ, with one chunk of keys and with several, against the general kernels."""
import math

import pytest
import torch

from natten_mps_b200 import _backend, _cabi

pytestmark = pytest.mark.gpu

# size, kernel, causal, (query heads, KV heads), dim
SHAPES = [((300,), (99,), (0,), (2, 2), 64), ((300,), (101,), (0,), (4, 2), 64), ((300,), (103,), (0,), (2, 2), 64),
          ((517,), (101,), (1,), (2, 2), 64), ((517,), (103,), (1,), (2, 1), 64), ((104,), (103,), (0,), (1, 1), 64),
          ((21, 40), (3, 33), (0, 0), (2, 2), 64), ((21, 40), (5, 21), (0, 1), (2, 2), 64), ((31, 29), (11, 11), (0, 0), (2, 1), 64),
          ((20, 33), (15, 15), (0, 0), (2, 2), 64), ((6, 13, 14), (3, 7, 5), (1, 0, 0), (2, 2), 64), ((300,), (101,), (0,), (2, 2), 128)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s[0] + s[1])) + f"d{s[-1]}")
def test_apply_around_the_third_cta(shape, dtype):
    size, kernel, causal, (hq, hkv), dim = shape
    rank, slots = len(size), math.prod(kernel)
    causal = tuple(bool(c) for c in causal)
    g = torch.Generator(device="cuda").manual_seed(slots)
    t = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k, v = (t(2, *size, h, dim).to(dtype) for h in (hq, hkv, hkv))
    attn, dlogits = torch.softmax(t(2, *size, hq, slots), dim=-1).to(dtype), t(2, *size, hq, slots).to(dtype)
    ones = (1,) * rank

    def run(path):
        try:
            _cabi.set_force(path)
            out = _backend.av_forward(attn, v, kernel, ones, ones, causal)
            assert _cabi.last_path() == {"tc": "tcgen05"}.get(path, path)
            return out, _backend.qk_backward(dlogits, q, k, kernel, ones, ones, causal, dim ** -0.5)[0]
        finally:
            _cabi.set_force(None)

    for got, want in zip(run("tc"), run("simt")):
        # weights and rows are the same 16-bit numbers on both sides, sums fp32: what differs is one rounding of the result, 2^-8
        # of its value at most in bf16; 2e-2 of the tensor's scale as in the other tests of these operators
        assert float((got.float() - want.float()).abs().max()) <= 2e-2 * max(1.0, float(want.float().abs().max()))
