"""Products of the 32-bit path that autograd, a transform or a trace follows stay torch's operator: the framework's kernel would lose what they follow."""

import pytest
import torch

from lalamo_b200 import ops


class _NoLaunch:
    def lb_gemm_float32(self, *arguments):
        raise AssertionError("launched past torch's operators")


@pytest.fixture(autouse=True)
def no_launch(monkeypatch):
    monkeypatch.setattr(ops, "_lib", lambda: _NoLaunch())
    assert ops.float32_product_supported(8, 16, 32)


X, W = torch.randn(8, 32, generator=torch.Generator().manual_seed(1)), torch.randn(16, 32, generator=torch.Generator().manual_seed(2))


def test_forward_mode():
    value, tangent = torch.func.jvp(lambda x: ops._product(x, W), (X,), (2 * X,))
    assert torch.equal(value, X @ W.T) and torch.equal(tangent, (2 * X) @ W.T)
    with torch.autograd.forward_ad.dual_level():
        dual = ops._product(torch.autograd.forward_ad.make_dual(X, 2 * X), W)
        assert torch.equal(torch.autograd.forward_ad.unpack_dual(dual).tangent, (2 * X) @ W.T)


def test_backward():
    weight = W.clone().requires_grad_()
    ops._product(X, weight).sum().backward()
    assert torch.allclose(weight.grad, X.sum(0).expand(16, 32))


def test_vmap():
    rows = torch.stack([X, -X, 3 * X])
    assert torch.allclose(torch.func.vmap(lambda x: ops._product(x, W))(rows), rows @ W.T, atol=1e-5)


def test_traces():
    from torch.fx.experimental.proxy_tensor import make_fx

    traced = make_fx(lambda x: ops._product(x, W))(X)
    assert torch.equal(traced(2 * X), (2 * X) @ W.T)
    assert torch.equal(torch.jit.trace(lambda x: ops._product(x, W), X, check_trace=False)(2 * X), (2 * X) @ W.T)
