"""Host-side mirror of the reference's operator interface for the matmul path.

Names, argument meaning and error behaviour follow src/native/src/ops/matmul.rs
and the bias branch of src/native/src/ops/elementwise.rs; every function is a thin
call into the C ABI of ``libmni_b200.so``, made by the native host side
(csrc/host/host.cpp): it checks the arguments, allocates the outputs the way the
reference's ``store.zeros`` does (uninitialised memory is fine: the kernels
overwrite every element) and names the current stream.
"""
from __future__ import annotations

from typing import Optional, Sequence, Tuple

from . import _lib
from .shapes import broadcast_shape, row_major_strides
from .tensor import DeviceTensor, _host, current_stream


def _matmul_out_shape(a: DeviceTensor, b: DeviceTensor) -> tuple:
    if a.ndim < 2 or b.ndim < 2:
        raise ValueError("matmul requires at least 2D tensors")          # ops/matmul.rs:89
    if a.shape[-1] != b.shape[-2]:
        raise ValueError(f"matmul inner dimensions must match: {a.shape[-1]} vs {b.shape[-2]}")  # :94
    return broadcast_shape(a.shape[:-2], b.shape[:-2]) + (a.shape[-2], b.shape[-1])


def matmul(a: DeviceTensor, b: DeviceTensor, bias: Optional[DeviceTensor] = None, *, flags: int = 0,
           out: Optional[DeviceTensor] = None) -> DeviceTensor:
    """``ops::matmul::matmul`` (ops/matmul.rs:83-197).  ``bias`` fuses the Linear bias add."""
    return _host.matmul(a, b, bias, flags, out)


def matmul_backward(grad: DeviceTensor, a: DeviceTensor, b: DeviceTensor, *, flags: int = 0,
                    need_da: bool = True, need_db: bool = True, want_dbias: bool = False,
                    da: Optional[DeviceTensor] = None, db: Optional[DeviceTensor] = None,
                    dbias: Optional[DeviceTensor] = None):
    """``ops::matmul::matmul_backward`` (ops/matmul.rs:225-255) -> (grad_a, grad_b[, dbias])."""
    return _host.matmul_backward(grad, a, b, flags, need_da, need_db, want_dbias, da, db, dbias)


def add(a: DeviceTensor, b: DeviceTensor) -> DeviceTensor:
    """Bias branch of ``ops::elementwise::add`` (ops/elementwise.rs:105-130): [.., N] + [N]."""
    return _host.add(a, b)


def add_backward(grad: DeviceTensor, a_shape: Sequence[int], b_shape: Sequence[int], *,
                 flags: int = 0) -> Tuple[DeviceTensor, DeviceTensor]:
    """``add_backward`` for the bias branch (ops/elementwise.rs:213-231) -> (grad_a, grad_bias)."""
    return _host.add_backward(grad, a_shape, b_shape, flags)


def bias_gelu(x: DeviceTensor, bias: DeviceTensor) -> DeviceTensor:
    """``ops::fused::bias_gelu`` (ops/fused.rs:279-314): gelu(x + bias) with bias over the last dim."""
    return _host.bias_gelu(x, bias)


def bias_gelu_backward(grad: DeviceTensor, x: DeviceTensor, bias: DeviceTensor, *,
                       flags: int = 0) -> Tuple[DeviceTensor, DeviceTensor]:
    """``ops::fused::bias_gelu_backward`` (ops/fused.rs:354-392) -> (dx, dbias)."""
    return _host.bias_gelu_backward(grad, x, bias, flags)


def matmul_bias_gelu(a: DeviceTensor, b: DeviceTensor, bias: DeviceTensor, *, flags: int = 0,
                     want_pre: bool = True) -> Tuple[Optional[DeviceTensor], DeviceTensor]:
    """matmul followed by bias_gelu in one GEMM launch -> (pre = a.b or None, out = gelu(pre + bias))."""
    return _host.matmul_bias_gelu(a, b, bias, flags, want_pre)


def softmax(a: DeviceTensor, dim: int = -1) -> DeviceTensor:
    """``ops::norm::softmax`` (ops/norm.rs:52-89).  A strided input is gathered first, as the reference's
    ``dev_ptr`` read assumes row-major data."""
    return _host.softmax(a, dim)


def softmax_backward(grad: DeviceTensor, out: DeviceTensor, dim: int = -1) -> DeviceTensor:
    """``ops::norm::softmax_backward`` (ops/norm.rs:125-163) from the saved forward output."""
    return _host.softmax_backward(grad, out, dim)


def _grad_sumsq(grads: Sequence[DeviceTensor]) -> "torch.Tensor":
    """Squared global gradient norm as a one-element f64 device tensor (no host read)."""
    import torch
    sumsq = torch.empty(1, dtype=torch.float64, device=grads[0].storage.device)
    _host.grad_norm_sq(grads, sumsq.data_ptr())
    return sumsq


def grad_norm(grads: Sequence[DeviceTensor]) -> float:
    """``ops::optimizer::grad_norm`` (ops/optimizer.rs:126-171): sqrt of the f64 sum of squares, as f32."""
    if not grads:
        return 0.0
    import numpy as np
    return float(np.sqrt(np.float32(_grad_sumsq(grads).item())))


def adamw_step(param: DeviceTensor, m: DeviceTensor, v: DeviceTensor, grad: DeviceTensor, *, lr: float,
               beta1: float = 0.9, beta2: float = 0.999, eps: float = 1e-8, weight_decay: float = 0.0,
               step: int = 1, grad_sumsq=None, max_grad_norm: float = 0.0, write_clipped_grad: bool = True) -> None:
    """``ops::optimizer::adamw_step`` for one parameter (ops/optimizer.rs:67-120): in-place update.
    ``grad_sumsq`` (a one-element f64 device tensor) with ``max_grad_norm`` > 0 applies the clip of
    ``clip_and_step`` inside the same pass."""
    if not (param.is_contiguous() and m.is_contiguous() and v.is_contiguous() and grad.is_contiguous()):
        raise ValueError("adamw_step needs contiguous tensors")
    if not (param.size == m.size == v.size == grad.size):
        raise ValueError("param, m, v and grad must have the same size")
    sq = grad_sumsq.data_ptr() if grad_sumsq is not None else None
    _lib.check(_lib.lib().mni_b200_adamw_step(param.ptr, m.ptr, v.ptr, grad.ptr, param.size, lr, beta1, beta2, eps,
                                              weight_decay, int(step), sq, max_grad_norm,
                                              1 if write_clipped_grad else 0, current_stream()))


def clip_and_step(params: Sequence[DeviceTensor], ms: Sequence[DeviceTensor], vs: Sequence[DeviceTensor],
                  grads: Sequence[DeviceTensor], *, lr: float, beta1: float = 0.9, beta2: float = 0.999,
                  eps: float = 1e-8, weight_decay: float = 0.0, step: int = 1, max_grad_norm: float = 0.0) -> float:
    """``ops::optimizer::clip_and_step`` (ops/optimizer.rs:247-276): global-norm clip and AdamW over all
    parameters; returns the norm before clipping.  The call waits for the norm alone: the step it has queued by
    then may still run, in stream order with whatever follows."""
    if not params:
        return 0.0
    if len(params) == len(ms) == len(vs) == len(grads):
        return _host.clip_and_step(params, ms, vs, grads, lr, beta1, beta2, eps, weight_decay, int(step), max_grad_norm)
    # more gradients than parameters (or the other way round): the norm is over all of them, the step over the pairs
    import numpy as np
    sumsq = _grad_sumsq(grads)
    for p, m, v, g in zip(params, ms, vs, grads):
        adamw_step(p, m, v, g, lr=lr, beta1=beta1, beta2=beta2, eps=eps, weight_decay=weight_decay, step=step,
                   grad_sumsq=sumsq, max_grad_norm=max_grad_norm)
    return float(np.sqrt(np.float32(sumsq.item())))


def permute(a: DeviceTensor, dims: Sequence[int]) -> DeviceTensor:
    """``ops::layout::permute``: a stride-only view sharing the storage (what the reference's CPU backend
    does, ops/layout.rs:112-134); the matmul kernels read it in place."""
    return a.permute(dims)


def permute_backward(grad: DeviceTensor, dims: Sequence[int], orig_shape: Sequence[int]) -> DeviceTensor:
    """``ops::layout::permute_backward`` (ops/layout.rs:198-212): the gradient of the permuted tensor, put
    back into the original layout -- one device gather of the inverse-permuted view."""
    return _host.permute_backward(grad, dims, orig_shape)


class Linear:
    """``Linear`` of src/nn.ts:8-26 over device tensors: y = x.W + b with W [in, out].

    ``forward`` runs the drop-in sequence (matmul, then the stand-alone bias add, the
    two N-API calls of nn.ts:24); ``forward_fused`` folds the bias into the GEMM epilogue.
    """

    def __init__(self, weight: DeviceTensor, bias: DeviceTensor):
        if weight.ndim != 2 or bias.shape != (weight.shape[1],):
            raise ValueError("weight must be [in, out] and bias [out]")
        self.weight = weight
        self.bias = bias

    def forward(self, x: DeviceTensor) -> DeviceTensor:
        return add(matmul(x, self.weight), self.bias)

    def forward_fused(self, x: DeviceTensor, flags: int = 0) -> DeviceTensor:
        return matmul(x, self.weight, self.bias, flags=flags)

    def backward(self, x: DeviceTensor, dy: DeviceTensor, flags: int = 0):
        """-> (dx, dW, db): add_backward then matmul_backward, with dbias fused into one call."""
        dx, dw, dbias = matmul_backward(dy, x, self.weight, flags=flags, want_dbias=True)
        return dx, dw, dbias


def sm_reserve(sms: int) -> None:
    """Keeps `sms` SMs out of the tensor-core kernels' grids (0 = none): room for a collective that runs beside them."""
    _lib.check(_lib.lib().mni_b200_sm_reserve(int(sms)))


def device_status() -> int:
    """Synchronises the current stream; raises if a kernel recorded a bounded-wait timeout."""
    import ctypes as C
    detail = C.c_uint32(0)
    _lib.check(_lib.lib().mni_b200_device_status(current_stream(), C.byref(detail)))
    return int(detail.value)


def launch_count() -> int:
    return int(_lib.lib().mni_b200_launch_count())


def plan_describe(a_shape: Sequence[int], b_shape: Sequence[int], *, a_strides: Optional[Sequence[int]] = None,
                  b_strides: Optional[Sequence[int]] = None, backward: int = 0, flags: int = 0,
                  sm_count: int = 148) -> list:
    """The launches ``matmul`` (backward=0) or ``matmul_backward`` (1; 2 = with the bias gradient) would make for
    operands of these shapes and element strides (row-major when not given) on a device with `sm_count` SMs:
    one line of text per launch.  Needs no device -- the planner is host arithmetic."""
    import ctypes as C
    va = _lib.make_view(256, a_shape, a_strides if a_strides is not None else row_major_strides(a_shape))
    vb = _lib.make_view(256, b_shape, b_strides if b_strides is not None else row_major_strides(b_shape))
    buf = C.create_string_buffer(8192)
    _lib.check(_lib.lib().mni_b200_plan_describe(C.byref(va), C.byref(vb), int(backward), int(flags), int(sm_count),
                                                 buf, len(buf)))
    return buf.value.decode().splitlines()
