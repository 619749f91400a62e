"""Split operators on tensor cores around the number of tiles where a third CTA on an SM finds one (two tiles an SM): value product,
dQ, dK and dV, with grouped heads, dilation, causal axes and several chunks, against the general kernels."""
import math

import pytest
import torch

from natten_mps_b200 import _backend, _cabi

pytestmark = pytest.mark.gpu

# size, kernel, dilation, causal, (query heads, KV heads), dim
SHAPES = [((128,), (31,), (1,), (0,), (1, 1), 64), ((128,), (63,), (2,), (1,), (2, 1), 64), ((16, 16), (7, 5), (1, 1), (0, 0), (2, 2), 64),
          ((8, 16), (7, 7), (1, 2), (0, 1), (4, 2), 64), ((4, 8, 8), (3, 5, 5), (1, 1, 1), (0, 0, 0), (2, 2), 64), ((128,), (31,), (1,), (0,), (1, 1), 128)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("an_sm", [0, 2, 3])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s[0] + s[1])) + f"d{s[-1]}")
def test_around_two_tiles_an_sm(shape, an_sm, dtype):
    size, kernel, dilation, causal, (hq, hkv), dim = shape
    causal = tuple(bool(c) for c in causal)
    tiles = math.prod(size) // 128 * hkv                 # of a sample, on the key side
    # (two an SM: the last count of the one form; the query side has the same or twice as many)
    B = max(1, an_sm * torch.cuda.get_device_properties(0).multi_processor_count // tiles)
    slots, ones = math.prod(kernel), (1,) * len(size)
    g = torch.Generator(device="cuda").manual_seed(slots)
    t = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k, v, do = (t(B, *size, h, dim).to(dtype) for h in (hq, hkv, hkv, hq))
    attn, dlogits = torch.softmax(t(B, *size, hq, slots), dim=-1).to(dtype), t(B, *size, hq, slots).to(dtype)

    def run(path):
        try:
            _cabi.set_force(path)
            out = _backend.av_forward(attn, v, kernel, dilation, ones, causal)
            assert _cabi.last_path() == {"tc": "tcgen05"}.get(path, path)
            return out, *_backend.qk_backward(dlogits, q, k, kernel, dilation, ones, causal, dim ** -0.5), *_backend.av_backward(do, attn, v, kernel, dilation, ones, causal)
        finally:
            _cabi.set_force(None)

    for got, want in zip(run("tc"), run("simt")):
        # the same 16-bit numbers on both sides, sums fp32: one rounding of the result, 2e-2 of the tensor's scale as in the other tests
        assert float((got.float() - want.float()).abs().max()) <= 2e-2 * max(1.0, float(want.float().abs().max()))
    assert _cabi.device_status() == 0
