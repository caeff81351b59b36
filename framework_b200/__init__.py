"""B200-native matmul hot path of mni-ml/framework: Tensor.matmul forward/backward and
the Linear bias add, as hand-written sm_100a kernels behind a C ABI.

``framework_b200.csrc`` holds the CUDA sources and the C ABI implementation,
``framework_b200.ops`` the host-side mirror of the reference's operator interface.

The operators and the tensor object are native (lib/_host.so) and are loaded when one of them is first used, so that a
process that only wants ``framework_b200.sharding`` or ``framework_b200.shapes`` loads, and builds, nothing.
"""
import importlib

from . import _lib  # noqa: F401

_OPS = ("Linear", "adamw_step", "add", "add_backward", "bias_gelu", "bias_gelu_backward", "broadcast_shape", "clip_and_step",
        "device_status", "grad_norm", "launch_count", "matmul", "matmul_backward", "matmul_bias_gelu", "permute",
        "permute_backward", "plan_describe", "sm_reserve", "softmax", "softmax_backward")

__all__ = ["DeviceTensor", *_OPS]


def __getattr__(name):
    if name in ("ops", "tensor"):
        return importlib.import_module(f"{__name__}.{name}")
    if name not in __all__:
        raise AttributeError(f"module {__name__!r} has no attribute {name!r}")
    from . import ops, tensor
    globals()["DeviceTensor"] = tensor.DeviceTensor
    globals().update({op: getattr(ops, op) for op in _OPS})
    return globals()[name]


def __dir__():
    return sorted({*globals(), *__all__, "ops", "tensor"})
