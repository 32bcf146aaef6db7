"""The Python surface as far as it goes without a GPU: the registered operators on meta tensors (shapes, autograd graph), the
modules' handling of parameters, and what importing the package loads."""
import json

import pytest

import specs


def _operands(requires_grad=True):
    """configuration, input, table and output gradient of a small dense grid, on the meta device"""
    import torch
    from qmlp import bindings
    cfg = json.dumps(specs.hashgrid(2, 3, 2, -1, 4, 16))
    enc = bindings.Encoding(cfg)
    x = torch.empty((10, 2), device="meta", requires_grad=requires_grad)
    table = torch.empty((enc.parameter_count(),), device="meta", requires_grad=requires_grad)
    return cfg, x, table, torch.empty((10, enc.num_output_channels()), device="meta")


def test_second_backward_raises():
    """The operators can be differentiated once. A second differentiation has to fail: a gradient penalty that silently
    counts as a constant trains on wrong gradients."""
    import torch
    import qmlp  # noqa: F401
    cfg, x, table, grad = _operands()
    out = torch.ops.qmlp_b200.encoding_forward(x, table, cfg)
    gx, gt = torch.autograd.grad(out, [x, table], grad, create_graph=True)
    assert gx.requires_grad and gt.requires_grad
    with pytest.raises(RuntimeError, match="differentiable"):
        (out.sum() + gx.pow(2).sum()).backward()
    a = torch.empty((4, 16), device="meta", dtype=torch.half, requires_grad=True)
    ga, = torch.autograd.grad(torch.ops.qmlp_b200.activation_forward(a, "relu").sum(), a, create_graph=True)
    with pytest.raises(RuntimeError, match="differentiable"):
        ga.sum().backward()
    # once, and without a graph of the gradient
    torch.ops.qmlp_b200.encoding_forward(x, table, cfg).backward(grad)
    assert x.grad.shape == x.shape and table.grad.shape == table.shape and not x.grad.requires_grad


def test_forward_mode_without_a_gradient():
    """The operators have no forward-mode formula: a dual tensor that requires no gradient is taken for its primal value
    (torch.func.jvp too), one that does is refused."""
    import torch
    import torch.autograd.forward_ad as fwad
    import qmlp  # noqa: F401
    cfg, x, table, grad = _operands(requires_grad=False)

    def call(a):
        return torch.ops.qmlp_b200.encoding_forward(a, table, cfg)
    with fwad.dual_level():
        out = fwad.unpack_dual(call(fwad.make_dual(x, torch.empty_like(x))))
        assert out.primal.shape == grad.shape and out.tangent is None
        with pytest.raises(RuntimeError):
            call(fwad.make_dual(x.clone().requires_grad_(True), torch.empty_like(x)))
    assert torch.func.jvp(call, (x,), (torch.empty_like(x),))[0].shape == grad.shape
