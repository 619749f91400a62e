"""Failure reporting of the tensor-core kernels, per-device launcher state, and padding hygiene.

* A barrier wait that runs out must surface as an error and must be recoverable.  The failure is
  made on the host: a test hook lets the fused forward's first barrier expect more bytes than its
  loads deliver and shortens the wait budget to a fraction of a millisecond, so the wait gives up
  (it never hangs), the kernel returns with the device's status word set, the next call raises,
  and after ``clear_status()`` the same call computes correctly again.
* A process whose first call is made under stream capture.
* One process using two GPUs in turn (skipped with a single GPU).
* Per-sample extents: whatever sits in the padding rows (NaN here) must not reach the results,
  which the reference guarantees by slicing each sample (``src/natten_mps/_core/pure.py:586-599``).
"""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import oracle
from natten_mps_b200 import _backend, _cabi, functional as F

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _case(seed=0, B=2, H=24, W=40, heads=2, D=64, dtype=torch.bfloat16, device="cuda"):
    g = torch.Generator().manual_seed(seed)
    return [torch.randn(B, H, W, heads, D, generator=g).to(dtype).to(device) for _ in range(3)]


def _oracle_out(q, k, v, K):
    f = lambda t: t.detach().float().cpu().numpy()
    return oracle.na_forward(f(q), f(k), f(v), kernel_size=K, dtype=np.float32)[0]


def test_wait_that_runs_out_is_reported_and_recoverable():
    q, k, v = _case()
    args = (q, k, v, (7, 7), (1, 1), (1, 1), (False, False), 0.125)
    L = _cabi.lib()
    try:
        L.natten_debug_wait(400_000, 1)           # ~0.2 ms budget; first barrier can never complete
        _cabi.set_force("tc")
        _backend.fused_forward(*args)
        assert _cabi.last_path() == "tcgen05"
        torch.cuda.synchronize()                  # returns: the kernel gave up instead of hanging
        assert _cabi.device_status() == -4        # NATTEN_E_DEVICE
        with pytest.raises(RuntimeError, match="bounded wait"):
            _backend.fused_forward(*args)         # the front end refuses to go on silently
    finally:
        L.natten_debug_wait(0, 0)
        _cabi.set_force(None)
        _cabi.clear_status()
    assert _cabi.device_status() == 0
    out, _ = _backend.fused_forward(*args)
    torch.cuda.synchronize()
    assert _cabi.device_status() == 0
    err = np.abs(out.float().cpu().numpy() - _oracle_out(q, k, v, 7)).max()
    assert err <= 2e-2, err


def same_after_giving_up(call):
    """The call's kernels run out of their waits, say so and return; the call after that is as good as the one before."""
    try:
        _cabi.set_force("tc")
        want = call()
        _cabi.lib().natten_debug_wait(400_000, 1)
        call()
        assert _cabi.last_path() == "tcgen05"
        torch.cuda.synchronize()
        assert _cabi.device_status() == -4
        _cabi.lib().natten_debug_wait(0, 0)
        _cabi.clear_status()
        got = call()
        torch.cuda.synchronize()
        assert _cabi.device_status() == 0
    finally:
        _cabi.lib().natten_debug_wait(0, 0)
        _cabi.set_force(None)
        _cabi.clear_status()
    for a, b in zip(got, want):
        assert (a is None and b is None) or torch.equal(a, b)


# A wait that gives up raises a flag which the CTA's other warps, each at a wait of its own, find when they next look: every role
# has to reach the end whichever of its lanes saw the flag first.
@pytest.mark.parametrize("B", [1, 24], ids=["few", "many"])
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("K,sizes", [((7, 7), None), ((3, 40), None), ((7, 7), (9, 40))], ids=["rows16", "line", "lengths"])
def test_every_role_ends_when_a_wait_runs_out(K, sizes, D, B):
    q, k, v = _case(B=B, H=24, W=48, heads=4, D=D, dtype=torch.float16)
    go = _case(seed=5, B=B, H=24, W=48, heads=4, D=D, dtype=torch.float16)[0]
    ext = None if sizes is None else torch.tensor([sizes] * B, dtype=torch.int32, device="cuda")
    args = (K, (1, 1), (1, 1), (False, False), D ** -0.5)
    same_after_giving_up(lambda: _backend.fused_forward(q, k, v, *args, extents=ext))
    out, lse = _backend.fused_forward(q, k, v, *args, extents=ext)
    same_after_giving_up(lambda: _backend.fused_backward(q, k, v, out, lse, go, *args, extents=ext))


@pytest.mark.parametrize("D,K", [(64, (7, 7)), (64, (11, 11)), (128, (7, 7))], ids=["d64", "d64_two_buffers", "d128"])
def test_every_role_of_the_split_operators_ends(D, K):
    q, k, v = _case(B=2, H=24, W=48, heads=4, D=D, dtype=torch.float16)
    geo = (K, (1, 1), (1, 1), (False, False))
    logits = _backend.qk_forward(q, k, *geo, None)
    w = torch.softmax(logits.float(), -1).half()
    same_after_giving_up(lambda: [_backend.qk_forward(q, k, *geo, None)])
    same_after_giving_up(lambda: [_backend.av_forward(w, v, *geo)])
    same_after_giving_up(lambda: _backend.qk_backward(logits, q, k, *geo, None))
    same_after_giving_up(lambda: _backend.av_backward(q, w, v, *geo))


def test_status_words_on_the_host_and_on_the_stream():
    """The word that the kernel itself writes into host memory, and the copy that a caller queues behind it."""
    q, k, v = _case(seed=1)
    L = _cabi.lib()
    word = torch.full((1,), 7, dtype=torch.int32).pin_memory()
    stream = torch.cuda.current_stream()
    try:
        assert L.natten_status_async(word.data_ptr(), stream.cuda_stream) == 0
        stream.synchronize()
        assert int(word) == 0 and L.natten_host_status(0) == 0
        L.natten_debug_wait(400_000, 1)
        F.na2d(q, k, v, 7)
        assert L.natten_status_async(word.data_ptr(), stream.cuda_stream) == 0
        stream.synchronize()
        assert int(word) != 0 and L.natten_host_status(0) != 0
    finally:
        L.natten_debug_wait(0, 0)
        _cabi.clear_status()
    assert L.natten_host_status(0) == 0


FIRST_CALL = """
import torch
from natten_mps_b200 import _cabi, functional as F
q, k, v, go = (torch.randn(1, 24, 24, 2, 64, device="cuda", dtype=torch.bfloat16) for _ in range(4))
q.requires_grad_(True)
step = lambda: torch.autograd.grad(F.na2d(q, k, v, 7), [q], go)[0]
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    got = step()
graph.replay()
torch.cuda.synchronize()
assert _cabi.last_path() == "tcgen05"
assert torch.equal(got, step())
"""


def test_first_call_of_a_process_may_be_captured():
    """The library sets itself up on first use; nothing of that may break the capture (a process of its own)."""
    done = subprocess.run([sys.executable, "-c", FIRST_CALL], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_two_devices_in_one_process():
    for dev in ("cuda:0", "cuda:1", "cuda:0"):
        q, k, v = _case(seed=3, device=dev)
        qq, kk, vv = [t.requires_grad_(True) for t in (q, k, v)]
        out = F.na2d(qq, kk, vv, 7)
        out.sum().backward()
        torch.cuda.synchronize(dev)
        assert _cabi.last_path() == "tcgen05"
        err = np.abs(out.detach().float().cpu().numpy() - _oracle_out(q, k, v, 7)).max()
        assert err <= 2e-2, (dev, err)
        assert torch.isfinite(qq.grad).all() and torch.isfinite(kk.grad).all()


@pytest.mark.parametrize("path", ["simt", "auto"])
@pytest.mark.parametrize("rank,D,dtype", [(1, 128, torch.float16), (2, 64, torch.bfloat16), (1, 32, torch.float32)],
                         ids=["1d_d128_f16", "2d_d64_bf16", "1d_d32_f32"])
def test_padding_rows_never_reach_the_results(rank, D, dtype, path):
    g = torch.Generator().manual_seed(11)
    if rank == 1:
        spatial, K, sizes = (300,), 31, [[300], [77], [200]]
    else:
        spatial, K, sizes = (20, 24), 5, [[20, 24], [9, 13], [16, 7]]
    B, Hq, Hkv = len(sizes), 4, 2
    mk = lambda h: torch.randn(B, *spatial, h, D, generator=g).to(dtype)
    q, k, v, go = mk(Hq), mk(Hkv), mk(Hkv), mk(Hq)
    f = lambda t: t.float().numpy()
    okw = dict(kernel_size=K, extents=np.asarray(sizes), dtype=np.float32)
    ref_out, ref_lse = oracle.na_forward(f(q), f(k), f(v), **okw)
    ref = (ref_out,) + oracle.na_backward(f(q), f(k), f(v), ref_out, ref_lse, f(go), **okw)[:3]
    # poison everything outside each sample's extent
    pad = torch.ones(B, *spatial, dtype=torch.bool)
    for b, ext in enumerate(sizes):
        pad[(b, *[slice(0, e) for e in ext])] = False
    for t in (q, k, v, go):
        t[pad] = float("nan")
    _cabi.set_force(path)
    try:
        leaves = [t.cuda().requires_grad_(True) for t in (q, k, v)]
        st = torch.tensor(sizes, dtype=torch.int32).cuda()
        fn = F.na1d_varlen if rank == 1 else F.na2d_varlen
        out = fn(*leaves, st[:, 0] if rank == 1 else st, K)
        grads = torch.autograd.grad(out, leaves, go.cuda())
    finally:
        _cabi.set_force(None)
    tol = 2e-2 if dtype != torch.float32 else 1e-4
    for name, got, want in zip(("out", "dq", "dk", "dv"), (out, *grads), ref):
        got = got.detach().float().cpu()
        assert torch.isfinite(got).all(), f"{name}: padding leaked into the result"
        assert float(got[pad].abs().sum()) == 0.0, f"{name}: padded rows must be exactly zero"
        err = float((got - torch.as_tensor(want)).abs().max())
        assert err <= tol * max(1.0, float(np.abs(want).max())) if dtype == torch.float32 else err <= tol, (name, err)
