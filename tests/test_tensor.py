"""The tensor object: copies and pickles."""
import copy
import copyreg
import io
import pickle

import numpy as np
import pytest


def _module():
    from framework_b200 import tensor
    return tensor


def test_state_has_the_form_of_a_class_with_slots():
    tensor = _module()
    t = tensor.DeviceTensor.__new__(tensor.DeviceTensor)
    t.shape, t.strides = (2, 3), (1, 2)
    assert t.__reduce_ex__(2) == (copyreg.__newobj__, (tensor.DeviceTensor,), (None, {"shape": (2, 3), "strides": (1, 2)}))
    for u in (copy.copy(t), copy.deepcopy(t), pickle.loads(pickle.dumps(t))):
        assert type(u) is tensor.DeviceTensor and u.shape == (2, 3) and u.strides == (1, 2) and not u.is_contiguous()
    with pytest.raises(TypeError):
        pickle.dumps(t, 0)


def test_state_of_a_subclass():
    class Named(_module().DeviceTensor):     # what a subclass may add: a slot and an instance dictionary
        __slots__ = ("tag", "__dict__")

    cls = Named
    t = cls.__new__(cls)
    t.shape, t.strides, t.tag, t.note = (4,), (1,), "a", [1]
    u = copy.deepcopy(t)
    assert type(u) is cls and (u.shape, u.tag, u.note) == ((4,), "a", [1]) and u.note is not t.note


@pytest.mark.gpu
def test_copies_and_checkpoints_keep_layout_and_contents(F):
    import torch
    a = np.random.default_rng(0).standard_normal((3, 5, 7)).astype(np.float32)
    t = F.DeviceTensor.from_numpy(a).permute((2, 0, 1))
    want = a.transpose(2, 0, 1)
    shallow, deep = copy.copy(t), copy.deepcopy(t)
    assert shallow.ptr == t.ptr and deep.ptr != t.ptr
    file = io.BytesIO()
    torch.save({"w": t, "again": t}, file)
    file.seek(0)
    loaded = torch.load(file, weights_only=False)
    assert loaded["w"] is loaded["again"]
    for u in (shallow, deep, pickle.loads(pickle.dumps(t)), loaded["w"]):
        assert u.shape == t.shape and u.strides == t.strides and np.array_equal(u.numpy(), want)
    deep.storage.zero_()
    assert np.array_equal(t.numpy(), want)


@pytest.mark.gpu
def test_fewer_strides_than_dimensions(F):
    """A dimension without a stride is not advanced along; there is nothing to permute it with."""
    import torch
    flat = torch.arange(16, dtype=torch.float32, device="cuda")
    t = F.DeviceTensor(flat, (4, 4), (1,))
    assert np.array_equal(t.contiguous().numpy(), np.repeat(np.arange(4, dtype=np.float32)[:, None], 4, 1))
    with pytest.raises(IndexError):
        t.permute((1, 0))
    u = F.DeviceTensor(flat, (16,))
    u.shape = (4, 4)                    # the strides are those of before
    assert not u.is_contiguous()
    with pytest.raises(IndexError):
        u.permute((1, 0))
    u.strides = (4, 1)
    assert u.is_contiguous() and np.array_equal(u.numpy(), flat.cpu().numpy().reshape(4, 4))


@pytest.mark.gpu
def test_dimensions_and_shapes_that_are_no_integers(F):
    t, y = F.DeviceTensor.empty((2, 3)), F.DeviceTensor.empty((2, 3))
    for dims in ((1.5, 0), (1.0, 0.0), ("1", "0"), (None, 0)):
        with pytest.raises(TypeError):
            t.permute(dims)
        with pytest.raises(TypeError):
            F.permute_backward(t, dims, (3, 2))
    assert t.permute((np.int64(1), 0)).shape == (3, 2)
    assert F.permute_backward(t, (1, 0), (3.0, 2)).shape == (3, 2)
    with pytest.raises(ValueError):
        F.permute_backward(t, (1, 0), (3.5, 2))
    assert F.add_backward(y, (2.0, 3), (3,))[0].shape == (2, 3)
    with pytest.raises(NotImplementedError):
        F.add_backward(y, (2.5, 3), (3,))
