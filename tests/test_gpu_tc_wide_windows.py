"""Windows wider than a chunk of 64 keys along the innermost axis, in images and volumes as well as in sequences: the forward's
chunks are then runs of that axis, several to a row.  Against the general kernels."""
import pytest
import torch

from natten_mps_b200 import _cabi, functional as F

pytestmark = pytest.mark.gpu

# size, kernel, dilation, causal, (query heads, KV heads), dim: two to four chunks a row, window and remainder at their edges
SHAPES = [
    ((20, 150), (3, 77), (1, 1), (0, 0), (2, 2), 64),
    ((20, 150), (3, 77), (1, 1), (0, 0), (2, 2), 128),
    ((9, 301), (5, 101), (1, 2), (0, 1), (2, 1), 64),
    ((70, 97), (65, 65), (1, 1), (0, 0), (1, 1), 64),
    ((70, 97), (65, 65), (1, 1), (1, 0), (2, 1), 128),
    ((12, 129), (1, 127), (2, 1), (0, 0), (2, 2), 32),
    ((3, 5, 140), (3, 3, 65), (1, 1, 1), (1, 0, 0), (2, 2), 64),
    ((3, 5, 140), (3, 3, 65), (1, 1, 1), (0, 0, 0), (2, 1), 128),
    ((700,), (33,), (1,), (0,), (2, 2), 64),
    ((700,), (63,), (1,), (1,), (2, 2), 128),
    ((700,), (129,), (2,), (0,), (2, 1), 64),
    ((400,), (127,), (1,), (0,), (2, 2), 96),
]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s[0] + s[1])) + f"d{s[-1]}")
@pytest.mark.parametrize("extra", [0, 70])
def test_windows_wider_than_a_chunk(shape, extra):
    size, kernel, dilation, causal, (hq, hkv), dim = shape
    g = torch.Generator(device="cuda").manual_seed(sum(size))
    t = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16).requires_grad_(True)
    q, k, v, do = t(2, *size, hq, dim), t(2, *size, hkv, dim), t(2, *size, hkv, dim), t(2, *size, hq, dim).detach()
    kw = {"additional_keys": t(2, extra, hkv, dim), "additional_values": t(2, extra, hkv, dim)} if extra else {}
    op = {1: F.na1d, 2: F.na2d, 3: F.na3d}[len(size)]

    def run(path):
        try:
            _cabi.set_force(path)
            out = op(q, k, v, kernel_size=kernel, dilation=dilation, is_causal=tuple(bool(c) for c in causal), **kw)
            assert _cabi.last_path() == {"tc": "tcgen05"}.get(path, path)
            return [out, *torch.autograd.grad(out, [q, k, v, *kw.values()], do)]
        finally:
            _cabi.set_force(None)

    for got, want in zip(run("tc"), run("simt")):
        # probabilities and results are rounded to bf16 (2^-9 each) on either side: 2e-2 of the tensor's scale, as everywhere
        assert float((got.detach().float() - want.detach().float()).abs().max()) <= 2e-2 * max(1.0, float(want.detach().float().abs().max()))


@pytest.mark.parametrize("lens", [(500, 127, 300), (128, 500, 191)])
@pytest.mark.parametrize("dim", [64, 128])
def test_windows_wider_than_a_chunk_varlen(lens, dim):
    g = torch.Generator(device="cuda").manual_seed(dim)
    t = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.float16)
    q, k, v = t(3, 500, 2, dim), t(3, 500, 2, dim), t(3, 500, 2, dim)
    for b, n in enumerate(lens):
        k[b, n:] = float("nan")                  # what lies past a sample's length must not be read
        v[b, n:] = float("nan")
    sizes = torch.tensor(lens, dtype=torch.int32, device="cuda")

    def run(path):
        try:
            _cabi.set_force(path)
            return F.na1d_varlen(q, k, v, sizes, kernel_size=127)
        finally:
            _cabi.set_force(None)

    got, want = run("tc"), run("simt")
    assert float((got.float() - want.float()).abs().max()) <= 2e-2
    for b, n in enumerate(lens):
        assert not got[b, n:].any()
