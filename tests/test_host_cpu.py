"""CPU: what the native operator front end refuses, before it touches a device."""
import pytest


@pytest.fixture(scope="module")
def F():
    from framework_b200 import build
    build.build_library()
    import framework_b200
    return framework_b200


def bare(F, shape):
    """A tensor with a shape and no storage: enough for the checks that come before the device."""
    t = F.DeviceTensor.__new__(F.DeviceTensor)
    t.shape = shape
    t.strides = F.tensor.row_major_strides(t.shape)
    return t


class NoTruth:
    def __bool__(self):
        raise RuntimeError("no truth value")


@pytest.mark.parametrize("flags", [None, 1.0, "1"])
def test_flags_that_are_no_number(F, flags):
    x, w, y, b = bare(F, (4, 3)), bare(F, (3, 2)), bare(F, (4, 2)), bare(F, (2,))
    launches = F.launch_count()
    for call in (lambda: F.matmul(x, w, flags=flags), lambda: F.matmul_backward(y, x, w, flags=flags),
                 lambda: F.matmul_bias_gelu(x, w, b, flags=flags), lambda: F.add_backward(y, (4, 2), (2,), flags=flags),
                 lambda: F.bias_gelu_backward(y, y, b, flags=flags)):
        with pytest.raises(TypeError):
            call()
    assert F.launch_count() == launches


def test_switches_without_a_truth_value(F):
    x, w, y, b = bare(F, (4, 3)), bare(F, (3, 2)), bare(F, (4, 2)), bare(F, (2,))
    for kw in ("need_da", "need_db", "want_dbias"):
        with pytest.raises(RuntimeError, match="no truth value"):
            F.matmul_backward(y, x, w, **{kw: NoTruth()})
    with pytest.raises(RuntimeError, match="no truth value"):
        F.matmul_bias_gelu(x, w, b, want_pre=NoTruth())


def test_tensor_without_storage(F):
    """An object that was never initialised has no `storage`: every use says so, none ends the process."""
    t, v = bare(F, (4, 4)), bare(F, (4,))
    uses = [lambda: t.storage, lambda: t.ptr, lambda: t.permute((1, 0)), lambda: t.numpy(), lambda: F.matmul(t, t),
            lambda: F.matmul_backward(t, t, t), lambda: F.matmul_bias_gelu(t, t, v), lambda: F.add(t, v),
            lambda: F.add_backward(t, (4, 4), (4,)), lambda: F.bias_gelu(t, v), lambda: F.bias_gelu_backward(t, t, v),
            lambda: F.softmax(t), lambda: F.softmax_backward(t, t), lambda: F.permute_backward(t, (1, 0), (4, 4)),
            lambda: F.clip_and_step([t], [t], [t], [t], lr=1e-3)]
    for use in uses:
        with pytest.raises(AttributeError, match="storage"):
            use()


def test_no_device_is_an_error_not_an_abort(F):
    import torch
    if torch.cuda.is_available():
        pytest.skip("there is a device")
    for use in (lambda: F.device_status(), lambda: F.tensor.current_stream(), lambda: F.DeviceTensor.empty((2, 2))):
        with pytest.raises(RuntimeError):
            use()
