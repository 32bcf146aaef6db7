"""Stand-alone activation and encoding as registered torch operators (``torch.ops.qmlp_b200.*``).

The reference registers TorchScript custom classes (``torch.classes.qmlp_cu.Activation / Encoding``,
src_cpp/pytorch-bindings/src/bind_activation.cpp:82-98, bind_encoding.cpp:167-197) so that its ``FusedActivation`` and
``FusedEncoding`` modules survive ``torch.jit.trace`` / ``freeze`` / ``save`` / ``load``
(tests_py/qmlp_tests/test_activations.py:42-57, test_encoding.py:84-106). Here the modules call operators whose only
non-tensor argument is the configuration string: a traced graph holds the string as a constant and the operator name,
and loading it needs nothing but this package imported. The operator looks the compiled object up by that string.

    activation_forward(Tensor input, str cfg) -> Tensor                          half tensors (N, C)
    activation_adjoint(Tensor input, Tensor adj_output, str cfg) -> Tensor
    encoding_forward(Tensor input, Tensor? parameters, str cfg) -> Tensor        float32 (N, C); float32 or float16 table
    encoding_adjoint(Tensor input, Tensor? parameters, Tensor adj_output, bool want_input, bool want_parameters,
                     str cfg) -> (Tensor, Tensor)

They are registered, with their autograd nodes, by the native call path (csrc/torch/calls.cpp).
"""
from . import _capi

_capi.calls()
