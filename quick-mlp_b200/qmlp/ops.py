"""Registered PyTorch operators behind the stand-alone modules, so that ``FusedActivation`` and ``FusedEncoding`` can be
traced, frozen, saved and loaded with ``torch.jit`` like any other module.

The reference reaches the same by TorchScript custom classes registered in its native library (RegisterClass,
src_cpp/pytorch-bindings/src/bind_activation.cpp:82-98, bind_encoding.cpp:167-197) and its tests trace and freeze the modules
(tests_py/qmlp_tests/test_activations.py:42-57, test_encoding.py:84-106). Here the modules call operators whose only
non-tensor argument is the configuration string: a traced graph holds the string as a constant and the operator name,
and loading it needs nothing but this package imported. The operator looks the compiled object up by that string.

    activation_forward(Tensor input, str cfg) -> Tensor                          half tensors (N, C)
    activation_adjoint(Tensor input, Tensor adj_output, str cfg) -> Tensor
    encoding_forward(Tensor input, Tensor? parameters, str cfg) -> Tensor        float32 (N, C); float32 or float16 table
    encoding_adjoint(Tensor input, Tensor? parameters, Tensor adj_output, bool want_input, bool want_parameters,
                     str cfg) -> (Tensor, Tensor)

The schemas are registered here; the kernels and the autograd nodes come with the native call path (csrc/torch/calls.cpp),
which registers them for CUDA and meta tensors when it is loaded. The first object of the package loads it, not the import:
the package's plain Python (configurations, the stock PyTorch modules) works without any of the native libraries. A graph
that runs before any object exists, and tensors of other devices, end up in `_load`, which is registered under the alias
keys and therefore only reached where the native call path has no kernel of its own.
"""
import threading

import torch

from . import _capi

SCHEMAS = {
    "activation_forward": "(Tensor input, str cfg) -> Tensor",
    "activation_adjoint": "(Tensor input, Tensor adj_output, str cfg) -> Tensor",
    "encoding_forward": "(Tensor input, Tensor? parameters, str cfg) -> Tensor",
    "encoding_adjoint": "(Tensor input, Tensor? parameters, Tensor adj_output, bool want_input, bool want_parameters, str cfg) -> (Tensor, Tensor)",
}

_library = torch.library.Library("qmlp_b200", "DEF")
_inside = threading.local()


def _load(name):
    def call(*args):
        if args[0].device.type not in ("cuda", "meta") or getattr(_inside, "loading", False):
            raise _capi.QmlpError("tensor must live on a CUDA device")
        _capi.calls()
        _inside.loading = True
        try:
            return getattr(torch.ops.qmlp_b200, name)(*args)
        finally:
            _inside.loading = False
    return call


for _name, _schema in SCHEMAS.items():
    _library.define(_name + _schema, tags=(torch.Tag.pt2_compliant_tag,))
    for _key in ("CompositeExplicitAutograd", "Autograd"):
        _library.impl(_name, _load(_name), _key)

activation_forward = torch.ops.qmlp_b200.activation_forward
activation_adjoint = torch.ops.qmlp_b200.activation_adjoint
encoding_forward = torch.ops.qmlp_b200.encoding_forward
encoding_adjoint = torch.ops.qmlp_b200.encoding_adjoint
