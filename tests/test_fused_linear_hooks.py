"""A gated layer's hooks run, whichever way its two halves meet."""
import pytest
import torch
import torch.nn.functional as F
from torch.nn.modules.module import register_module_forward_hook

from vllm_omni_b200.diffusion.layers.linear import FusedLinear
from vllm_omni_b200.ops import gemm


def _layer():
    torch.manual_seed(0)
    return FusedLinear(16, 32, bias=False), torch.randn(5, 16).bfloat16()


def _expected(x, w):
    g, u = (x.float() @ w.float().T).split(16, -1)
    return F.silu(g) * u


def test_no_hooks_take_the_fused_call(monkeypatch):
    layer, x = _layer()
    monkeypatch.setattr(gemm, "linear_swiglu", lambda *a: "fused")
    assert layer.swiglu(x) == "fused"


@pytest.mark.parametrize("kind", ["pre", "post", "global", "forward"])
def test_hooks_run(kind):
    layer, x = _layer()
    want, handle = _expected(2 * x, layer.weight), None
    if kind == "pre":
        layer.register_forward_pre_hook(lambda m, a: (2 * a[0],))
    elif kind == "post":
        layer.register_forward_hook(lambda m, a, y: 2 * y)
    elif kind == "global":
        handle = register_module_forward_hook(lambda m, a, y: 2 * y)
    else:
        plain = layer.forward
        layer.forward = lambda t: plain(2 * t)
    try:
        y = layer.swiglu(x)
    finally:
        if handle is not None:
            handle.remove()
    # both halves and the result in bf16
    assert ((y.float() - want).abs() <= 2.0 ** -7 * want.abs() + 2.0 ** -7 * want.abs().max()).all()
    assert not torch.allclose(y.float(), _expected(x, layer.weight), rtol=0.2, atol=0.0)
