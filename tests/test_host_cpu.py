"""CPU: what the native operator front end refuses, before it touches a device."""
import threading
import time

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


def test_one_of_several_compiles_the_extension(monkeypatch, tmp_path):
    from framework_b200 import build
    monkeypatch.setattr(build, "HOST_PATH", str(tmp_path / "lib" / "_host.so"))
    runs = []

    def compiler(cmd, **kw):
        runs.append(cmd)
        time.sleep(0.2)
        open(cmd[cmd.index("-o") + 1], "w").close()
    monkeypatch.setattr(build.subprocess, "check_call", compiler)
    threads = [threading.Thread(target=build.build_host) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(runs) == 1 and not build.host_is_stale()
    build.build_host(force=True)
    assert len(runs) == 2


def test_no_compiler_is_an_import_error(monkeypatch, tmp_path):
    from framework_b200 import build
    monkeypatch.setattr(build, "HOST_PATH", str(tmp_path / "lib" / "_host.so"))

    def no_compiler(cmd, **kw):
        raise FileNotFoundError(2, "No such file or directory", cmd[0])
    monkeypatch.setattr(build.subprocess, "check_call", no_compiler)
    with pytest.raises(ImportError, match="framework_b200.build"):
        build.load_host()


def test_names_of_the_package():
    import subprocess
    import sys
    from conftest import ROOT
    code = """
import sys
import framework_b200 as F
assert "framework_b200.ops" not in sys.modules and {"matmul", "DeviceTensor", "ops"} <= set(dir(F))
assert F.matmul is F.ops.matmul and F.DeviceTensor is F.tensor.DeviceTensor and F.broadcast_shape((2, 1), (3,)) == (2, 3)
from framework_b200 import *
assert all(name in globals() for name in F.__all__)
try:
    F.nothing
except AttributeError as e:
    assert "nothing" in str(e)
else:
    raise AssertionError
"""
    subprocess.run([sys.executable, "-c", code], check=True, cwd=ROOT)
