"""Tile tables of the tcgen05 forward: shapes at the edges of what the tables hold (one row per warp lane, tiles of one column,
more chunks than a row map has room for, volumes, output stride, padding tiles), against the general kernels.  These calls have few
tiles, so head dims up to 64 run the form with two score buffers; test_gpu_tc_many_tiles.py has the same shapes in the other form."""
import pytest
import torch

from natten_mps_b200 import _cabi, functional as F

pytestmark = pytest.mark.gpu



def forced(path, run):
    try:
        _cabi.set_force(path)
        return run()
    finally:
        _cabi.set_force(None)


# rank, size, kernel, dilation, stride, causal, heads, dim
SHAPES = [
    (2, (40, 40), (3, 15), (1, 1), (1, 1), (0, 0), 2, 64),       # 16 inner columns leave tiles two wide: 64 row maps
    (2, (40, 33), (1, 15), (1, 1), (1, 1), (0, 0), 2, 32),
    (2, (70, 40), (63, 9), (1, 1), (1, 1), (0, 0), 1, 64),       # more than 16 chunks: no row maps
    (2, (64, 48), (9, 9), (3, 2), (1, 1), (0, 1), 2, 64),
    (2, (37, 41), (7, 7), (1, 1), (2, 3), (0, 0), 2, 64),
    (3, (9, 17, 19), (5, 3, 7), (1, 1, 1), (1, 1, 1), (1, 0, 0), 2, 64),
    (3, (6, 12, 14), (3, 5, 5), (2, 1, 1), (1, 1, 1), (0, 0, 0), 2, 32),
    (1, (700,), (255,), (1,), (1,), (1,), 2, 128),
    (2, (30, 26), (7, 7), (1, 1), (1, 1), (0, 0), 2, 96),
]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s[1] + s[2])) + f"d{s[-1]}")
@pytest.mark.parametrize("extra", [0, 5])
def test_forward_tables(shape, extra):
    rank, size, kernel, dilation, stride, causal, heads, dim = shape
    g = torch.Generator(device="cuda").manual_seed(sum(size))
    t = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)
    q, k, v = (t(2, *size, heads, dim) for _ in range(3))
    kw = {"additional_keys": t(2, extra, heads, dim), "additional_values": t(2, extra, heads, dim)} if extra else {}
    op = {1: F.na1d, 2: F.na2d, 3: F.na3d}[rank]
    run = lambda: op(q, k, v, kernel_size=kernel, dilation=dilation, stride=stride, is_causal=tuple(bool(c) for c in causal), **kw)
    got, want = forced("tc", run), forced("simt", run)
    # probabilities and outputs are rounded to bf16 (2^-9 each): 2e-2 as everywhere
    assert float((got.float() - want.float()).abs().max()) <= 2e-2


@pytest.mark.parametrize("lens", [(300, 7, 128), (129, 300, 15)])
@pytest.mark.parametrize("dim", [64, 128])
def test_forward_tables_varlen(lens, dim):
    g = torch.Generator(device="cuda").manual_seed(dim)
    t = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.float16)
    q, k, v = t(3, 300, 4, dim), t(3, 300, 2, dim), t(3, 300, 2, dim)
    sizes = torch.tensor(lens, dtype=torch.int32, device="cuda")
    run = lambda: F.na1d_varlen(q, k, v, sizes, kernel_size=7)
    got, want = forced("tc", run), forced("simt", run)
    assert float((got.float() - want.float()).abs().max()) <= 2e-2
    for b, n in enumerate(lens):
        assert not got[b, n:].any()


# size, kernel, causal, (query heads, KV heads), dim: tiles of 2, 4 or 8 heads, ragged ends, one chunk and many
PACKED = [((200,), (15,), (0,), (4, 2), 64), ((333,), (63,), (1,), (8, 1), 128), ((700,), (255,), (0,), (4, 1), 128),
          ((129,), (33,), (1,), (6, 3), 64), ((97,), (17,), (0,), (16, 2), 32), ((23, 37), (5, 11), (0, 0), (8, 2), 64),
          ((19, 30), (9, 9), (0, 1), (4, 2), 128), ((40, 33), (3, 21), (0, 0), (8, 1), 96)]


@pytest.mark.parametrize("shape", PACKED, ids=lambda s: "x".join(map(str, s[0] + s[1] + s[3])) + f"d{s[-1]}")
@pytest.mark.parametrize("extra", [0, 5])
def test_grouped_heads_packed(shape, extra):
    size, kernel, causal, (hq, hkv), dim = shape
    g = torch.Generator(device="cuda").manual_seed(sum(size))
    t = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.float16).requires_grad_(True)
    q, k, v, do = t(2, *size, hq, dim), t(2, *size, hkv, dim), t(2, *size, hkv, dim), t(2, *size, hq, dim).detach()
    kw = {"additional_keys": t(2, extra, hkv, dim), "additional_values": t(2, extra, hkv, dim)} if extra else {}
    op = {1: F.na1d, 2: F.na2d}[len(size)]

    def run():
        out = op(q, k, v, kernel_size=kernel, is_causal=tuple(bool(c) for c in causal), **kw)
        return [out, *torch.autograd.grad(out, [q, k, v, *kw.values()], do)]

    for got, want in zip(forced("tc", run), forced("simt", run)):
        # sums of up to 16 heads x window rounded to fp16 on either side: 2e-2 of the tensor's scale
        assert float((got.float() - want.float()).abs().max()) <= 2e-2 * max(1.0, float(want.float().abs().max()))


@pytest.mark.parametrize("lens", [(300, 9, 128), (129, 300, 33)])
def test_grouped_heads_packed_varlen(lens):
    g = torch.Generator(device="cuda").manual_seed(3)
    t = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16).requires_grad_(True)
    q, k, v = t(3, 300, 8, 64), t(3, 300, 2, 64), t(3, 300, 2, 64)
    do = t(3, 300, 8, 64).detach()
    sizes = torch.tensor(lens, dtype=torch.int32, device="cuda")

    def run():
        out = F.na1d_varlen(q, k, v, sizes, kernel_size=9)
        return [out, *torch.autograd.grad(out, [q, k, v], do)]

    for got, want in zip(forced("tc", run), forced("simt", run)):
        assert float((got.float() - want.float()).abs().max()) <= 2e-2 * max(1.0, float(want.float().abs().max()))
        for b, n in enumerate(lens):
            assert not got[b, n:].any()
