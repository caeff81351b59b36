"""The warp-level streaming kernels of a few rows: edges of tiles, slices and strips, aligned and unaligned weights, weights
seen through a transposing view, bias and accumulation, against float64 inside guard zones."""
import numpy as np
import pytest

from conftest import Guarded, regression_bound_3xtf32, rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n", [(9, 4096, 2404), (15, 1000, 2500), (1, 65, 2433), (16, 31, 33), (3, 1024, 129), (12, 33, 4096),
                                   (10, 2401, 2390), (5, 16384, 2370), (9, 64, 32), (2, 1, 1)])
@pytest.mark.parametrize("transposed", [False, True])
def test_few_rows_forward_and_backward(F, m, k, n, transposed):
    rng = np.random.default_rng([m, k, n])
    x, dy = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((m, n)).astype(np.float32)
    w, bias = rng.standard_normal((k, n)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    t = F.DeviceTensor.from_numpy
    wd = t(np.ascontiguousarray(w.T)).permute((1, 0)) if transposed else t(w)
    x64, w64, dy64 = (a.astype(np.float64) for a in (x, w, dy))
    c0 = [rng.standard_normal(s).astype(np.float32) for s in ((m, n), (m, k), (k, n))]
    for accumulate in (False, True):
        y, dx, dw = (Guarded(F, c.shape, init=c if accumulate else None) for c in c0)
        flags = (F._lib.ACCUMULATE_C | F._lib.ACCUMULATE_DA | F._lib.ACCUMULATE_DB) if accumulate else 0
        F.matmul(t(x), wd, t(bias), out=y.tensor, flags=flags)
        F.matmul_backward(t(dy), t(x), wd, da=dx.tensor, db=dw.tensor, flags=flags)
        F.device_status()
        for got, want, c, length in ((y, x64 @ w64 + bias, c0[0], k), (dx, dy64 @ w64.T, c0[1], n), (dw, x64.T @ dy64, c0[2], m)):
            got.check(fully_written=not accumulate)
            ref = want + (c if accumulate else 0)
            assert rel_fro(got.tensor.numpy(), ref) <= regression_bound_3xtf32(length), (accumulate, length)


def test_few_rows_plans(F):
    """Which calls stream the weight: few rows that the FFMA kernels do not take, enough outputs for the strips or a short
    contraction; 16 aligned rows are the tensor path's."""
    def kernel(m, k, n):
        return F.plan_describe((m, k), (k, n))[0]
    assert "few rows" in kernel(9, 4096, 4096) and "few rows" in kernel(16, 4096, 4093) and "few rows" in kernel(9, 1000, 4001)
    assert "skinny" in kernel(3, 4096, 4096)
    assert "tensor" in kernel(16, 4096, 4096) and "tensor" in kernel(9, 8192, 512)


@pytest.mark.parametrize("m,k,n", [(2, 97, 130), (7, 129, 1001), (16, 70, 63), (13, 1030, 2434), (4, 33, 4100)])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_few_rows_units_from_before_a_row(F, m, k, n, offset):
    """Rows at every shift against the 16-byte units that they are copied in; NaNs around the operands must not leak in."""
    rng = np.random.default_rng([m, k, n, offset])

    def inside(a, at):
        buf = np.full(a.size + 8, np.nan, np.float32)
        buf[at:at + a.size] = a.ravel()
        return F.DeviceTensor(F.DeviceTensor.from_numpy(buf).torch_view()[at:at + a.size], a.shape)

    x, dy = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((m, n)).astype(np.float32)
    w = rng.standard_normal((k, n)).astype(np.float32)
    x64, w64, dy64 = (a.astype(np.float64) for a in (x, w, dy))
    for transposed in (False, True):
        wd = inside(np.ascontiguousarray(w.T), offset).permute((1, 0)) if transposed else inside(w, offset)
        y = F.matmul(inside(x, (offset + 1) % 4), wd)
        dx, dw = F.DeviceTensor.empty((m, k)), Guarded(F, (k, n), misalign=offset)
        F.matmul_backward(inside(dy, (offset + 2) % 4), inside(x, (offset + 1) % 4), wd, da=dx, db=dw.tensor)
        F.device_status()
        dw.check("dw")
        dw = dw.tensor
        for got, want, length in ((y, x64 @ w64, k), (dx, dy64 @ w64.T, n), (dw, x64.T @ dy64, m)):
            assert rel_fro(got.numpy(), want) <= regression_bound_3xtf32(length)


def test_weight_gradient_of_more_slabs_than_a_grid_has(F):
    """9 rows in slabs of 512 weight rows: the first length past 65535 slabs."""
    import torch
    k = 65535 * 512 + 1
    gen = torch.Generator(device="cuda").manual_seed(1)
    x, dy = torch.randn((9, k), generator=gen, device="cuda"), torch.randn((9, 1), generator=gen, device="cuda")
    dw = Guarded(F, (k, 1))
    t = F.DeviceTensor.from_torch
    F.matmul_backward(t(dy), t(x), F.DeviceTensor.empty((k, 1)), need_da=False, db=dw.tensor)
    F.device_status()
    dw.check("dw")
    want = (x * dy).sum(0, dtype=torch.float64)
    got = dw.tensor.storage.double()
    assert float((got - want).norm() / want.norm()) <= regression_bound_3xtf32(9)
    assert float((got - want)[-600:].abs().max()) <= 1e-5


@pytest.mark.parametrize("m,k,n", [(1, 4096, 2044), (1, 4096, 2048), (5, 2099, 4000), (8, 65, 129060), (3, 16421, 516)])
def test_weight_written_by_the_kernel_before(F, m, k, n):
    """A long weight's first rows are asked into L2 before the kernel before has ended; what that kernel writes there is what the
    product reads.  Sizes on both sides of the rule, ragged slices and strips."""
    rng = np.random.default_rng([m, k, n])
    x = rng.standard_normal((m, k)).astype(np.float32)
    t = F.DeviceTensor.from_numpy
    xd, w, y = t(x), F.DeviceTensor.empty((k, n)), Guarded(F, (m, n))
    for turn in range(4):
        u, v = rng.standard_normal((k, 3)).astype(np.float32), rng.standard_normal((3, n)).astype(np.float32)
        ud, vd = t(u), t(v)
        F.matmul(ud, vd, out=w)
        F.matmul(xd, w, out=y.tensor)
        F.device_status()
        y.check(fully_written=True)
        want = x.astype(np.float64) @ w.numpy().astype(np.float64)
        assert rel_fro(y.tensor.numpy(), want) <= regression_bound_3xtf32(k), turn


@pytest.mark.parametrize("k,n", [(4097, 2048), (33, 2052), (35, 508), (31, 516), (2, 2044), (16, 4), (2100, 4100), (4741, 2052), (9490, 516)])
@pytest.mark.parametrize("m", range(1, 9))
def test_input_gradient_steps_and_what_is_left_of_a_row(F, m, k, n):
    """Each row count's own kernel: whole steps of 512 columns, none, a last part; odd weight rows; short and long rows; two and
    three blocks per SM."""
    rng = np.random.default_rng([m, k, n])
    x, dy, w = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (m, n), (k, n)))
    t = F.DeviceTensor.from_numpy
    c = rng.standard_normal((m, k)).astype(np.float32)
    for accumulate in (False, True):
        dx = Guarded(F, (m, k), init=c if accumulate else None)
        flags = F._lib.FORCE_SKINNY_PATH | (F._lib.ACCUMULATE_DA if accumulate else 0)
        F.matmul_backward(t(dy), t(x), t(w), da=dx.tensor, need_db=False, flags=flags)
        F.device_status()
        dx.check(fully_written=not accumulate)
        want = dy.astype(np.float64) @ w.astype(np.float64).T + (c if accumulate else 0)
        assert rel_fro(dx.tensor.numpy(), want) <= regression_bound_3xtf32(n), accumulate
