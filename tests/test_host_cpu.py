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
