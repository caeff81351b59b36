"""GPU parity of the bias + GELU widening: the stand-alone kernels and the GEMM epilogue that fuses
matmul -> bias_gelu, against the CPU oracle (ops/fused.rs:251-277, :317-352 restated in C)."""
import numpy as np
import pytest

from conftest import rel_fro, tol_3xtf32

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def F():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    import framework_b200 as F
    F._lib.lib()
    return F


def _dev(F, arr):
    return F.DeviceTensor.from_numpy(arr)


@pytest.mark.parametrize("shape", [(64, 128), (33, 30), (4, 5, 96), (1, 7)])
def test_bias_gelu_forward_and_backward(F, oracle, shape):
    rng = np.random.default_rng(sum(shape))
    x = (2.0 * rng.standard_normal(shape)).astype(np.float32)
    bias = rng.standard_normal(shape[-1], dtype=np.float32)
    g = rng.standard_normal(shape, dtype=np.float32)
    H = oracle.HostTensor.from_array
    ref = oracle.bias_gelu(H(x), H(bias)).numpy()
    got = F.bias_gelu(_dev(F, x), _dev(F, bias)).numpy()
    # tanhf of the device and of the host libm differ by a few ulp
    assert float(np.max(np.abs(got - ref))) <= 2e-6 * (1.0 + float(np.abs(x).max() + np.abs(bias).max()))
    rdx, rdb = oracle.bias_gelu_backward(H(g), H(x), H(bias))
    dx, db = F.bias_gelu_backward(_dev(F, g), _dev(F, x), _dev(F, bias))
    F.device_status()
    assert float(np.max(np.abs(dx.numpy() - rdx.numpy()))) <= 4e-6 * float(np.abs(g).max()) * 1.2
    rows = int(np.prod(shape[:-1]))
    assert float(np.max(np.abs(db.numpy() - rdb.numpy()))) <= 1e-5 * rows * float(np.abs(g).max()) * 1.2


@pytest.mark.parametrize("m,k,n,flags_name", [(384, 256, 512, None), (200, 100, 72, None), (130, 64, 30, None),
                                              (4, 256, 512, None), (256, 2048, 256, "split")])
def test_matmul_with_bias_gelu_epilogue(F, oracle, m, k, n, flags_name):
    """Fused path (aligned, no split-K) and the two-kernel route it falls back to must both match
    matmul followed by bias_gelu on the CPU."""
    rng = np.random.default_rng(m + k + n)
    a = rng.standard_normal((m, k), dtype=np.float32)
    w = (0.05 * rng.standard_normal((k, n))).astype(np.float32)
    bias = (0.1 * rng.standard_normal(n)).astype(np.float32)
    H = oracle.HostTensor.from_array
    rpre = oracle.matmul(H(a), H(w))
    rout = oracle.bias_gelu(rpre, H(bias)).numpy()
    flags = F._lib.force_split_k(3) | F._lib.FORCE_TENSOR_PATH if flags_name == "split" else 0
    pre, out = F.matmul_bias_gelu(_dev(F, a), _dev(F, w), _dev(F, bias), flags=flags)
    F.device_status()
    bound = tol_3xtf32(k, a, w)
    assert float(np.max(np.abs(pre.numpy() - rpre.numpy()))) <= bound
    assert float(np.max(np.abs(out.numpy() - rout))) <= 1.2 * bound + 4e-6
    _, out_only = F.matmul_bias_gelu(_dev(F, a), _dev(F, w), _dev(F, bias), flags=flags, want_pre=False)
    F.device_status()
    assert np.array_equal(out_only.numpy(), out.numpy())


def test_batched_broadcast_weight_with_gelu(F, oracle):
    """Config 4's shape family at reduced size: [B, M, K] . [K, N] + b, GELU."""
    rng = np.random.default_rng(5)
    a = rng.standard_normal((3, 160, 96), dtype=np.float32)
    w = (0.02 * rng.standard_normal((96, 256))).astype(np.float32)
    bias = (0.02 * rng.standard_normal(256)).astype(np.float32)
    H = oracle.HostTensor.from_array
    rpre = oracle.matmul(H(a), H(w))
    rout = oracle.bias_gelu(rpre, H(bias)).numpy()
    pre, out = F.matmul_bias_gelu(_dev(F, a), _dev(F, w), _dev(F, bias))
    F.device_status()
    assert pre.shape == (3, 160, 256)
    assert float(np.max(np.abs(out.numpy() - rout))) <= 1.2 * tol_3xtf32(96, a, w) + 4e-6


def _exact(v):
    v = v.astype(np.float64)
    u2 = 2 * 0.7978845608028654 * (v + 0.044715 * v ** 3)
    s = 1 / (1 + np.exp(-u2))
    return u2, v * s, s + v * s * (1 / (1 + np.exp(u2))) * 2 * 0.7978845608028654 * (1 + 3 * 0.044715 * v ** 2)


def _gelu_and_derivative(F, v):
    n = 1024
    x = F.DeviceTensor.from_numpy(v.reshape(-1, n))
    zero, one = (F.DeviceTensor.from_numpy(np.full(s, c, np.float32)) for s, c in (((n,), 0), (x.shape, 1)))
    return F.bias_gelu(x, zero).numpy().ravel(), F.bias_gelu_backward(one, x, zero)[0].numpy().ravel()


def test_gelu_is_as_exact_as_the_tanh_form_in_single_precision(F):
    """Normally distributed inputs, error in the 2-norm against float64: 0.5 v (1 + tanhf(u)) and its derivative in f32 are off
    by 3.84e-8 and 4.50e-8."""
    v = np.random.default_rng(0).standard_normal(1 << 20).astype(np.float32)
    _, gelu, grad = _exact(v)
    got, dgot = _gelu_and_derivative(F, v)
    assert rel_fro(got, gelu) <= 3.84e-8 and rel_fro(dgot, grad) <= 4.50e-8


def test_gelu_pointwise(F):
    """Positive v: the rounding of the result, and the error of e = exp(-2u) < 1, two units and more where e is small, in
    1 + e: three units of 2^-24 together.  Negative v: the error of the exponential, (2 + 1.2 |2u|) units, and of 2u itself, two
    roundings times |2u|.  The derivative is s plus v s (1 - s) 2u', |v 2u'| <= 3 |2u|, with such an error in each factor."""
    v = np.linspace(-10, 10, 1 << 20).astype(np.float32)
    u2, gelu, grad = _exact(v)
    got, dgot = _gelu_and_derivative(F, v)
    relative = np.where(v >= 0, 3 * 2.0 ** -24, (4 + 3.2 * np.abs(u2)) * 2.0 ** -23)
    assert np.all(np.abs(got - gelu) <= relative * np.abs(gelu) + 1e-37)
    terms = np.where(v >= 0, 1.2, np.exp(np.minimum(u2, 0)) * (1 + 3 * np.abs(u2)))
    assert np.all(np.abs(dgot - grad) <= 2 * relative * terms + 1e-36)


def test_gelu_of_extreme_inputs(F):
    v = np.zeros(1024, np.float32)
    v[:9] = [np.inf, -np.inf, np.nan, 1e13, -1e13, 3e38, -3e38, 88, -88]
    got, dgot = _gelu_and_derivative(F, v)
    assert got[0] == np.inf and np.isnan(got[1]) and np.isnan(got[2])       # as 0.5 v (1 + tanh u) gives them
    assert np.array_equal(got[3:9], np.maximum(v[3:9], 0))
    assert list(dgot[[3, 4, 7, 8]]) == [1, 0, 1, 0] and np.all(np.isnan(dgot[:3]))
    assert not got[9:].any() and np.all(dgot[9:] == 0.5)
