"""Key-side boxes of the backward that are longer than the tile's extent plus the kernel: keys next to a clamped edge are read
by every query of the edge, and a tile that starts inside that range needs more column chunks than the others."""
import numpy as np
import pytest
import torch

from tests._gpu_util import check, run_fused

pytestmark = pytest.mark.gpu

# spatial, Hq, Hkv, kernel, dilation, causal, D
CASES = [((64, 64), 2, 2, (9, 13), (1, 1), (False, False), 64), ((51, 27), 4, 2, (5, 9), (1, 3), (False, False), 64),
         ((72, 20), 1, 1, (9, 7), (1, 2), (False, False), 32), ((67, 32), 1, 1, (5, 11), (1, 1), (False, False), 128),
         ((13, 14, 12), 1, 1, (5, 5, 7), (1, 1, 1), (False, False, True), 128), ((18, 20, 13), 2, 1, (3, 7, 5), (1, 1, 1), (False, False, False), 64)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])))
def test_long_key_boxes(case):
    sp, Hq, Hkv, K, dil, causal, D = case
    rng = np.random.default_rng(9)
    r = lambda h: rng.standard_normal((1, *sp, h, D))
    got, want = run_fused(len(sp), torch.bfloat16, r(Hq), r(Hkv), r(Hkv), r(Hq), dict(kernel_size=K, dilation=dil, is_causal=causal))
    for name in ("out", "dq", "dk", "dv"):
        check(name, got[name], want[name], torch.bfloat16, scale_rel=True)
