"""Device tensor with the reference's data model: storage + shape + element strides.

Mirrors ``GpuTensor`` of src/native/src/tensor.rs:63-73.  ``permute`` is a
stride-only view (what the reference's CPU backend does, ops/layout.rs:112-134;
its CUDA backend materialises instead, :137-156) so that strided operands reach
the matmul kernels through TMA descriptors without a copy.  PyTorch is used only
to own device memory and to name the current stream.
"""
from __future__ import annotations

import copyreg
from typing import Sequence

import numpy as np
import torch

from . import _lib, build
from .shapes import row_major_strides, shape_size  # noqa: F401

_host = build.load_host()


def current_stream() -> int:
    """Address of the current CUDA stream of the current device."""
    return _host.current_stream()


class DeviceTensor(_host.Tensor):
    """f32 tensor on the current CUDA device: flat `storage`, `shape`, element `strides`.

    ``DeviceTensor(storage, shape, strides=None)``; the object itself, with `size`, `ndim`, `ptr`,
    `is_contiguous()`, `permute(dims)` and `contiguous()`, is native (csrc/host/host.cpp)."""

    __slots__ = ()

    # -- construction ------------------------------------------------------
    @staticmethod
    def empty(shape: Sequence[int], device=None) -> "DeviceTensor":
        return _host.empty(shape, device)

    @staticmethod
    def from_numpy(a: np.ndarray, device=None) -> "DeviceTensor":
        """Tensor.fromFloat32 (src/tensor.ts:72-75): host f32 data -> contiguous device tensor."""
        a = np.ascontiguousarray(a, dtype=np.float32)
        flat = torch.from_numpy(a.reshape(-1))
        return DeviceTensor(flat.to(device or "cuda"), a.shape)

    @staticmethod
    def from_torch(t: torch.Tensor) -> "DeviceTensor":
        """Wraps a CUDA f32 torch tensor (any strides) without copying."""
        if t.dtype != torch.float32 or not t.is_cuda:
            raise TypeError("need a float32 CUDA tensor")
        base = t.untyped_storage()
        flat = torch.empty(0, dtype=torch.float32, device=t.device).set_(
            base, t.storage_offset(), (max(_span(t), 1),), (1,))
        return DeviceTensor(flat, tuple(t.shape), tuple(t.stride()))

    # -- copies and checkpoints --------------------------------------------
    def __reduce_ex__(self, protocol):
        """copy.copy shares the storage; copy.deepcopy and pickle (torch.save) carry it.  The state is the one a Python class
        with these three slots has, (instance dictionary or None, slot values), so that files of either kind load."""
        if protocol < 2:
            return super().__reduce_ex__(protocol)           # refused, as for any class with slots
        names = ["storage", "shape", "strides", *copyreg._slotnames(type(self))]
        slots = {name: getattr(self, name) for name in names if getattr(self, name, None) is not None}
        return copyreg.__newobj__, (type(self),), (getattr(self, "__dict__", None) or None, slots)

    def view_struct(self) -> "_lib.View":
        return _lib.make_view(self.ptr, self.shape, self.strides)

    # -- layout ops (ops/layout.rs) ------------------------------------------
    def narrow(self, dim: int, start: int, length: int) -> "DeviceTensor":
        """The sub-tensor [start, start + length) of dimension `dim`, as a view of the same storage (pointer
        offset + same strides): how row or column panels of an operand reach the kernels without a copy."""
        d = dim + self.ndim if dim < 0 else dim
        if not (0 <= d < self.ndim and 0 <= start and length >= 0 and start + length <= self.shape[d]):
            raise ValueError(f"narrow({dim}, {start}, {length}) out of range for shape {self.shape}")
        shape = list(self.shape)
        shape[d] = length
        return DeviceTensor(self.storage[start * self.strides[d]:], shape, self.strides)

    def view(self, shape: Sequence[int]) -> "DeviceTensor":
        """ops/layout.rs:80-89: reshape of the contiguous data (shares storage when already contiguous)."""
        if shape_size(shape) != self.size:
            raise ValueError(f"cannot view {self.shape} as {tuple(shape)}")
        return DeviceTensor(self.contiguous().storage, shape)

    # -- host transfer -----------------------------------------------------
    def numpy(self) -> np.ndarray:
        """toFloat32 (tensor.rs:364-387): logical contents, row-major."""
        c = self.contiguous()
        return c.storage[: max(c.size, 0)].cpu().numpy().reshape(c.shape).copy()

    def torch_view(self) -> torch.Tensor:
        """The same memory as a strided torch tensor (for harness comparisons)."""
        return torch.as_strided(self.storage, self.shape, self.strides)


def _span(t: torch.Tensor) -> int:
    if t.numel() == 0:
        return 0
    return 1 + sum((s - 1) * st for s, st in zip(t.shape, t.stride()))


_host.setup(DeviceTensor, lambda: _host.bind(_lib.addresses()), _lib.raise_status, lambda a, b: _product_shape(a, b))


def _product_shape(a, b) -> tuple:
    from .ops import _matmul_out_shape
    return _matmul_out_shape(a, b)
