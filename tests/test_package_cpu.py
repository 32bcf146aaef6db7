"""The Python surface as far as it goes without a GPU: the registered operators on meta tensors (shapes, autograd graph), the
modules' handling of parameters, and what importing the package loads."""
import json
import os
import subprocess
import sys

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


def _in_fresh_process(code, *args):
    root = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "quick-mlp_b200")
    run = subprocess.run([sys.executable, "-c", f"import sys; sys.path.insert(0, {root!r})\n" + code, *args], capture_output=True, text=True)
    assert run.returncode == 0, run.stderr[-2000:]


def test_import_loads_no_native_library():
    """Importing the package (its configurations, the stock PyTorch modules) needs none of the native libraries."""
    _in_fresh_process("""
import qmlp
from qmlp import configs
qmlp.SimulatedNetwork(configs.dumps(configs.config2()))
maps = open("/proc/self/maps").read()
assert "qmlp_calls" not in maps and "libqmlp_b200" not in maps
""")


def test_saved_graph_runs_before_any_object_exists(tmp_path):
    """A traced graph that is loaded in a process which has only imported the package: the first call of the operator loads
    its kernels, on the way to a gradient too."""
    import torch
    cfg, x, table, grad = _operands(requires_grad=False)

    class Module(torch.nn.Module):
        def forward(self, x, table):
            return torch.ops.qmlp_b200.encoding_forward(x, table, cfg)
    path = str(tmp_path / "graph.pt")
    torch.jit.save(torch.jit.trace(Module(), (x, table), check_trace=False), path)
    _in_fresh_process(f"""
import torch, qmlp
graph = torch.jit.load(sys.argv[1])
x, table = torch.empty((10, 2), device="meta", requires_grad=True), torch.empty(({table.numel()},), device="meta", requires_grad=True)
out = graph(x, table)
out.sum().backward()
assert tuple(out.shape) == {tuple(grad.shape)} and x.grad.shape == x.shape and table.grad.shape == table.shape
""", path)


def test_operators_of_other_devices_and_their_names():
    import torch
    import qmlp
    from qmlp._capi import QmlpError
    cfg, x, table, grad = _operands()
    with pytest.raises(QmlpError, match="CUDA device"):
        torch.ops.qmlp_b200.encoding_forward(torch.zeros(x.shape), torch.zeros(table.shape), cfg)
    with pytest.raises(QmlpError, match="CUDA device"):
        qmlp.ops.activation_adjoint(torch.zeros((4, 16)), torch.zeros((4, 16)), "relu")
    assert qmlp.ops.encoding_forward(x, table, cfg).shape == grad.shape
    assert torch.Tag.pt2_compliant_tag in torch.ops.qmlp_b200.encoding_forward.default.tags


class _Passed:
    """Stands for the native network: returns what forward() passes on."""
    def forward(self, x, weights, encoding_parameters):
        return x, weights, encoding_parameters


def _cpu_network(cfg):
    import torch
    import qmlp
    net = qmlp.FusedNetwork(specs.dumps(cfg), weight_dtype=torch.float32, device="cpu")
    net._network = _Passed()
    return net


def test_forward_takes_weights_that_are_no_parameter():
    """Parametrised and pruned weights, and those of a DataParallel replica, are attributes of the module but not in its
    parameter dictionary."""
    import torch
    from torch.nn.utils import parametrize, prune

    class Twice(torch.nn.Module):
        def forward(self, w):
            return 2 * w
    cfg = specs.config1()
    x = torch.zeros((4, 3))
    net = _cpu_network(cfg)
    before = net.weights.detach().clone()
    parametrize.register_parametrization(net, "weights", Twice())
    assert torch.equal(net(x)[1], 2 * before)
    net = _cpu_network(cfg)
    prune.random_unstructured(net, "weights", 0.5)
    assert torch.equal(net(x)[1], net.weights_orig * net.weights_mask)
    net = _cpu_network(cfg)
    replica = net._replicate_for_data_parallel()
    replica.weights = before
    assert replica(x)[1] is before
    net = _cpu_network(cfg)
    other = torch.zeros_like(net.weights)
    assert torch.func.functional_call(net, {"weights": other}, (x,))[1] is other


def test_module_saved_without_the_cached_shape():
    """A whole module pickled when it did not keep what forward() needs of the network."""
    import pickle
    import torch
    import qmlp
    net = qmlp.FusedNetwork(specs.dumps(specs.config3(log2_hashmap_size=12)), device="cpu")
    for name in ("_num_input_channels", "_encoding_has_parameters", "_no_encoding_parameters"):
        del net.__dict__[name]
    loaded = pickle.loads(pickle.dumps(net))
    loaded._network = _Passed()
    x = torch.zeros((4, 3))
    _, weights, encodings = loaded(x)
    assert torch.equal(weights, net.weights) and len(encodings) == 1 and torch.equal(encodings[0], net.encoding_parameters[0])
