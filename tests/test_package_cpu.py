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
