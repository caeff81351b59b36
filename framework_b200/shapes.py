"""Shape arithmetic of the operators: plain Python, no native code."""
from __future__ import annotations

from typing import Sequence


def broadcast_shape(a: Sequence[int], b: Sequence[int]) -> tuple:
    """utils.rs:3-20.  Raises where the reference panics."""
    nd = max(len(a), len(b))
    out = []
    for i in range(nd):
        da = 1 if i < nd - len(a) else a[i - (nd - len(a))]
        db = 1 if i < nd - len(b) else b[i - (nd - len(b))]
        if da == db:
            out.append(da)
        elif da == 1:
            out.append(db)
        elif db == 1:
            out.append(da)
        else:
            raise ValueError(f"shapes {list(a)} and {list(b)} are not broadcastable")
    return tuple(out)


def row_major_strides(shape: Sequence[int]) -> tuple:
    """tensor.rs:7-17 compute_strides."""
    st, acc = [], 1
    for s in reversed(shape):
        st.append(acc)
        acc *= int(s)
    return tuple(reversed(st))


def shape_size(shape: Sequence[int]) -> int:
    n = 1
    for s in shape:
        n *= int(s)
    return n
