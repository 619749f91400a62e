"""Forward on tensors whose axes are shorter than a tile's nominal key box, which decides how many chunks are interleaved: images and
volumes with two tiles and fewer along an axis, causal axes (whose boxes start in front of the tensor), output stride, dilation and
lengths, against the general kernels."""
import pytest
import torch

from tests.test_gpu_tc_many_tiles import compare, inputs

pytestmark = pytest.mark.gpu

# size, kernel, dilation, stride, causal, (query heads, KV heads), dim
SHAPES = [
    ((15, 7, 7), (7, 7, 5), (1, 1, 1), (1, 1, 1), (0, 0, 0), (4, 4), 32),
    ((7, 8, 7), (3, 7, 5), (1, 1, 1), (1, 1, 1), (0, 0, 0), (4, 2), 128),
    ((15, 20, 7), (5, 7, 7), (1, 1, 1), (1, 1, 1), (1, 0, 0), (2, 2), 64),
    ((6, 14, 20), (3, 7, 7), (1, 1, 1), (1, 1, 1), (0, 1, 0), (2, 2), 64),
    ((6, 32, 9), (3, 7, 7), (1, 1, 1), (1, 1, 1), (0, 0, 0), (2, 2), 64),
    ((7, 9, 30), (3, 7, 7), (2, 1, 1), (1, 1, 1), (0, 1, 0), (2, 2), 64),
    ((4, 40, 40), (3, 7, 7), (1, 1, 1), (1, 2, 3), (0, 0, 0), (2, 1), 64),
    ((8, 6, 14), (3, 5, 11), (1, 1, 1), (1, 1, 1), (0, 1, 1), (2, 2), 64),
    ((7, 7), (7, 5), (1, 1), (1, 1), (0, 0), (8, 8), 64),
    ((7, 7), (7, 7), (1, 1), (1, 1), (1, 1), (2, 2), 64),
    ((8, 24), (7, 7), (1, 1), (1, 1), (1, 0), (2, 2), 64),
    ((8, 40), (7, 13), (1, 1), (1, 1), (0, 0), (8, 2), 64),
    ((9, 24), (3, 9), (1, 1), (2, 2), (0, 0), (2, 2), 128),
    ((17, 30), (7, 7), (2, 2), (1, 1), (0, 0), (2, 2), 32),
    ((19, 30), (7, 7), (2, 1), (4, 1), (1, 0), (2, 2), 64),
    ((10, 9), (8, 6), (1, 1), (1, 1), (0, 0), (2, 2), 64),
    ((13,), (5,), (1,), (1,), (1,), (2, 2), 64),
]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s[0] + s[1])) + f"d{s[-1]}")
@pytest.mark.parametrize("B", [1, 70])
def test_forward(shape, B):
    size, kernel, dilation, stride, causal, (hq, hkv), dim = shape
    qkv, _ = inputs(B, size, hq, hkv, dim, torch.bfloat16, sum(size))
    plain = all(s == 1 for s in stride)
    compare(qkv, kernel, stride, dilation, tuple(bool(c) for c in causal), dim ** -0.5, backward=plain)


@pytest.mark.parametrize("size,kernel,sizes", [((16, 33), (7, 7), [[16, 33], [8, 9], [7, 20]]), ((9, 12, 14), (3, 7, 7), [[9, 12, 14], [3, 7, 8], [4, 9, 7]])])
def test_lengths(size, kernel, sizes):
    qkv, _ = inputs(9, size, 2, 2, 64, torch.float16, 3)
    ext = torch.tensor(sizes * 3, dtype=torch.int32, device="cuda")
    ones = (1,) * len(size)
    compare(qkv, kernel, ones, ones, (False,) * len(size), 0.125, extents=ext)
