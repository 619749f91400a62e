"""The module as one native call against its separate operators (what it does with a hook in place): outputs and every
gradient, packed and grouped projections, output stride, missing biases, frozen parameters, inference, a strided input."""
import pytest
import torch

import natten_mps_b200 as nb

pytestmark = pytest.mark.gpu

CASES = [("2d", nb.NeighborhoodAttention2D, (13, 17), dict(kernel_size=5)),
         ("2d_gqa", nb.NeighborhoodAttention2D, (12, 15), dict(kernel_size=(3, 5), dilation=(2, 1), num_kv_heads=2)),
         ("1d_stride", nb.NeighborhoodAttention1D, (41,), dict(kernel_size=7, stride=2, qkv_bias=False)),
         ("3d_causal", nb.NeighborhoodAttention3D, (3, 8, 9), dict(kernel_size=3, is_causal=(True, False, False), qk_scale=0.3))]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: c[0])
def test_one_call_matches_the_separate_operators(case, dtype):
    _, cls, size, kw = case
    torch.manual_seed(1)
    m = cls(128, 4, **kw).to("cuda", dtype)
    base = torch.randn(2, *size, 160, device="cuda", dtype=dtype)
    x = base[..., :128].requires_grad_(True)                     # rows are not adjacent
    frozen = m.proj.weight
    for step in ("all", "frozen", "inference"):
        frozen.requires_grad_(step == "all")
        leaves = [x] + [p for p in m.parameters() if p.requires_grad]
        got = []
        for hook in (False, True):
            h = m.proj.register_forward_hook(lambda *a: None) if hook else None
            with torch.set_grad_enabled(step != "inference"):
                y = m(x)
            assert y.requires_grad == (step != "inference")
            if step != "inference":
                names = y.grad_fn.name()
                assert ("ModuleFn" in names) != hook, names
                got.append([y, *torch.autograd.grad(y, leaves, torch.linspace(-1, 1, y.numel(), device="cuda").view_as(y).to(dtype))])
            else:
                got.append([y])
            if h is not None:
                h.remove()
        for a, b in zip(*got):
            tol = 1e-5 if dtype == torch.float32 else 1e-2
            assert a.shape == b.shape and (a.float() - b.float()).norm() <= tol * b.float().norm().clamp_min(1e-3)


@pytest.mark.parametrize("case", CASES, ids=lambda c: c[0])
def test_gradients_with_a_graph_of_their_own(case):
    """create_graph: what the separate operators allow (the attention itself is differentiable once), with the module applied
    twice so that its weights are shared and its second input depends on them."""
    _, cls, size, kw = case
    if kw.get("stride", 1) != 1:
        size = (83,)                                             # the second application needs its kernel, too
    torch.manual_seed(2)
    m = cls(64, 2, **{**kw, **({"num_kv_heads": 1} if "num_kv_heads" in kw else {})}).to("cuda", torch.float32)
    x = torch.randn(2, *size, 64, device="cuda", requires_grad=True)
    results = []
    for hook in (False, True):
        h = m.proj.register_forward_hook(lambda *a: None) if hook else None
        y = m(m(x))
        leaves = [x, *m.parameters()]
        first = torch.autograd.grad(y.square().sum(), leaves, create_graph=True)
        penalty = m(x).mul(0.5).tanh().sum()
        by_weight = torch.autograd.grad(penalty, [m.proj.weight, m.proj.bias], create_graph=True)
        second = torch.autograd.grad(sum(g.square().sum() for g in by_weight), leaves, allow_unused=True)
        results.append([*first, *second])
        if h is not None:
            h.remove()
    names = [n for n, _ in m.named_parameters()]
    for name, a, b in zip(2 * ["x", *names], *results):
        assert (a is None) == (b is None), name
        if a is not None:
            assert (a - b).norm() <= 1e-4 * b.norm().clamp_min(1e-3), name


def test_gradients_with_a_graph_refuse_a_changed_bias():
    m = nb.NeighborhoodAttention1D(64, 2, 7).to("cuda", torch.float32)
    x = torch.randn(1, 40, 64, device="cuda", requires_grad=True)
    y = m(x).sum()
    with torch.no_grad():
        m.qkv.bias.add_(1)
    torch.autograd.grad(y, x, retain_graph=True)                 # no bias is needed for this one
    with pytest.raises(RuntimeError, match="modified in place"):
        torch.autograd.grad(y, x, create_graph=True)
