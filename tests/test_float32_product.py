"""Which products of the 32-bit path the framework's kernel takes: not those that autograd, a transform or a trace follows (it would lose what they follow), and
not the sizes that the library does sooner."""

import pytest
import torch

from lalamo_b200 import ops


class _NoLaunch:
    def lb_gemm_float32(self, *arguments):
        raise AssertionError("launched past torch's operators")


@pytest.fixture(autouse=True)
def no_launch(monkeypatch):
    monkeypatch.setattr(ops, "_lib", lambda: _NoLaunch())
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    assert ops.float32_product_supported(8, 16, 512)


X, W = torch.randn(8, 512, generator=torch.Generator().manual_seed(1)), torch.randn(16, 512, generator=torch.Generator().manual_seed(2))


class _OnCuda(torch.Tensor):
    """A tensor that says that it lies on a device of a certain number."""

    is_cuda = True
    device_number = 0

    def get_device(self):
        return self.device_number

    @classmethod
    def __torch_function__(cls, function, types, arguments=(), keywords=None):
        with torch._C.DisableTorchFunctionSubclass():
            return function(*arguments, **(keywords or {}))


@pytest.mark.parametrize("x_device,weight_device", [(0, 1), (1, 1)])
def test_devices(x_device, weight_device, monkeypatch):
    """The kernel runs on the current device; torch's operator on the tensors' own, if it is one."""
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    x, weight = X.as_subclass(_OnCuda), W.as_subclass(_OnCuda)
    x.device_number, weight.device_number = x_device, weight_device
    assert torch.equal(ops._product(x, weight), X @ W.T)
    x.device_number = weight.device_number = 0
    with pytest.raises(AssertionError, match="launched"):
        ops._product(x, weight)


def test_forward_mode():
    value, tangent = torch.func.jvp(lambda x: ops._product(x, W), (X,), (2 * X,))
    assert torch.equal(value, X @ W.T) and torch.equal(tangent, (2 * X) @ W.T)
    with torch.autograd.forward_ad.dual_level():
        dual = ops._product(torch.autograd.forward_ad.make_dual(X, 2 * X), W)
        assert torch.equal(torch.autograd.forward_ad.unpack_dual(dual).tangent, (2 * X) @ W.T)


def test_backward():
    weight = W.clone().requires_grad_()
    ops._product(X, weight).sum().backward()
    assert torch.allclose(weight.grad, X.sum(0).expand(16, 512))


def test_vmap():
    rows = torch.stack([X, -X, 3 * X])
    assert torch.allclose(torch.func.vmap(lambda x: ops._product(x, W))(rows), rows @ W.T, atol=1e-4)


def test_traces():
    from torch.fx.experimental.proxy_tensor import make_fx

    traced = make_fx(lambda x: ops._product(x, W))(X)
    assert torch.equal(traced(2 * X), (2 * X) @ W.T)
    assert torch.equal(torch.jit.trace(lambda x: ops._product(x, W), X, check_trace=False)(2 * X), (2 * X) @ W.T)


@pytest.mark.parametrize("taken,left", [((8, 64, 512), (8, 64, 384)), ((8, 3072, 128), (8, 2048, 256)), ((8, 64, 4096), (8, 64, 8192)), ((16, 16384, 1024), (16, 16384, 256)),
                                        ((17, 4608, 64), (17, 4608, 192)), ((32, 6144, 1024), (32, 6144, 512)), ((32, 16384, 2048), (32, 9216, 2048)), ((32, 9216, 4608), (32, 16448, 4608)),
                                        ((64, 4096, 512), (64, 4096, 384)), ((64, 4096, 1024), (64, 4608, 1024)), ((384, 1024, 1024), (400, 1024, 1024)), ((700, 8, 2048), (1000, 8, 2048)),
                                        ((5, 2048, 1024), (4, 2048, 1024)), ((8, 2048, 1024), (8, 2048, 1022))])
def test_sizes(taken, left):
    def takes(size):
        tokens, rows, width = size
        return ops.float32_product_supported(tokens, rows, width)

    assert takes(taken) and not takes(left)
