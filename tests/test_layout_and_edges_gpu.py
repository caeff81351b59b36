"""Forms of the memory-bound kernels at the sizes where they change or can go wrong: gathers of permuted views, column
sums with their copy, the bias pass, softmax rows that are not 16-byte aligned, and products whose output rows are not."""
import numpy as np
import pytest

from conftest import Guarded, regression_bound_3xtf32, rel_fro

pytestmark = pytest.mark.gpu


def _rng(*key):
    return np.random.default_rng(list(key))


@pytest.mark.parametrize("shape,dims", [
    ((2, 5, 3, 64), (0, 2, 1, 3)),          # rows of 16-byte units
    ((2, 7, 3, 65), (0, 2, 1, 3)),          # odd rows: an element per unit
    ((2, 3, 65, 33), (0, 1, 3, 2)),         # transposing tiles, both extents past a tile's edge
    ((3, 64, 32), (0, 2, 1)),               # exactly one tile each
    ((2, 3, 8, 130), (0, 3, 1, 2)),         # tiles with dimensions between
    ((130, 7), (1, 0)),                     # too narrow for tiles
    ((5, 1, 9), (2, 1, 0)), ((1, 1, 1), (2, 0, 1)), ((4, 6), (0, 1))])
def test_gather_of_permuted_views(F, shape, dims):
    a = _rng(1, *shape).standard_normal(shape).astype(np.float32)
    view = F.DeviceTensor.from_numpy(a).permute(dims)
    want = np.ascontiguousarray(a.transpose(dims))
    out = Guarded(F, want.shape)
    F._lib.check(F._lib.lib().mni_b200_contiguous(view.view_struct(), out.tensor.ptr, 0))
    out.check("gather")
    assert np.array_equal(out.tensor.numpy(), want)
    assert np.array_equal(view.contiguous().numpy(), want)
    back = F.permute_backward(F.DeviceTensor.from_numpy(want), dims, shape)
    assert np.array_equal(back.numpy(), a)


@pytest.mark.parametrize("shape,dims", [
    ((7, 5, 3), (1, 0, 2)),                 # rows of 3 in units of 4, a remainder of 1
    ((3, 5, 2), (1, 0, 2)), ((9, 7, 1, 5), (1, 0, 2, 3)), ((2, 3), (1, 0)), ((31, 3, 17), (2, 1, 0)),
    ((150, 333, 65), (1, 0, 2)),            # two units per thread, the last one partial
    ((4, 12, 640, 79), (0, 2, 1, 3)),
    ((8, 400, 12, 64), (0, 2, 1, 3))])      # two aligned units per thread
def test_gather_in_units_across_rows(F, shape, dims):
    a = _rng(7, *shape).standard_normal(shape).astype(np.float32)
    view = F.DeviceTensor.from_numpy(a).permute(dims)
    want = np.ascontiguousarray(a.transpose(dims))
    for misalign in (0, 1):
        out = Guarded(F, want.shape, misalign=misalign)
        F._lib.check(F._lib.lib().mni_b200_contiguous(view.view_struct(), out.tensor.ptr, 0))
        out.check("gather")
        assert np.array_equal(out.tensor.numpy(), want)


@pytest.mark.parametrize("rows,n,misalign", [(1, 1, 0), (63, 4, 0), (65, 130, 0), (64, 128, 0), (1000, 516, 0), (129, 260, 1),
                                             (777, 131, 0), (5000, 33, 0), (40, 200_000, 0)])
def test_bias_add_and_its_backward(F, rows, n, misalign):
    rng = _rng(2, rows, n)
    y, b = rng.standard_normal((rows, n)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    dy = Guarded(F, (rows, n), init=y, misalign=misalign)
    bias = F.DeviceTensor.from_numpy(b)
    lib, check = F._lib.lib(), F._lib.check
    out = Guarded(F, (rows, n), misalign=misalign)
    check(lib.mni_b200_add_bias(dy.tensor.ptr, bias.ptr, out.tensor.ptr, rows, n, 0))
    out.check("bias add")
    assert np.array_equal(out.tensor.numpy(), y + b)
    copy, sums = Guarded(F, (rows, n), misalign=misalign), Guarded(F, (n,))
    check(lib.mni_b200_add_bias_bwd(dy.tensor.ptr, copy.tensor.ptr, sums.tensor.ptr, rows, n, 0, 0))
    copy.check("copy of dy")
    sums.check("column sums")
    assert np.array_equal(copy.tensor.numpy(), y)
    exact = y.astype(np.float64).sum(0)
    bound = 1e-6 * np.sqrt(rows) * np.abs(y).max() + 1e-6
    assert np.max(np.abs(sums.tensor.numpy() - exact)) <= bound * 8
    check(lib.mni_b200_add_bias_bwd(dy.tensor.ptr, None, sums.tensor.ptr, rows, n, F._lib.ACCUMULATE_DBIAS, 0))
    assert np.max(np.abs(sums.tensor.numpy() - 2 * exact)) <= bound * 16


@pytest.mark.parametrize("length", [31, 33, 333, 511, 1023, 1025, 2047])
def test_softmax_rows_of_odd_length(F, length):
    rng = _rng(3, length)
    x, dy = (rng.standard_normal((19, length)).astype(np.float32) * 3 for _ in range(2))
    e = np.exp(x.astype(np.float64) - x.max(-1, keepdims=True))
    p = e / e.sum(-1, keepdims=True)
    got = F.softmax(F.DeviceTensor.from_numpy(x))
    assert np.max(np.abs(got.numpy() - p)) <= 4e-7 + 4e-6 * p.max()
    s = got.numpy().astype(np.float64)
    want = s * (dy - (dy * s).sum(-1, keepdims=True))
    dx = F.softmax_backward(F.DeviceTensor.from_numpy(dy), got)
    assert np.max(np.abs(dx.numpy() - want)) <= 1e-6 * (1 + np.abs(want).max())


@pytest.mark.parametrize("m,k,n,batch,flags", [
    (130, 64, 257, (), 0), (70, 40, 333, (3,), 0),           # one piece, rows of 257 / 333 floats
    (256, 1700, 301, (), 0),                                 # pieces added to unaligned rows
    (300, 512, 129, (), 3 << 16), (64, 260, 777, (2,), 2 << 16)])   # split contraction, padded partials
@pytest.mark.parametrize("accumulate", [False, True])
def test_products_with_unaligned_output_rows(F, m, k, n, batch, flags, accumulate):
    rng = _rng(4, m, k, n)
    a, b = rng.standard_normal(batch + (m, k)).astype(np.float32), rng.standard_normal(batch + (k, n)).astype(np.float32)
    bias, c0 = rng.standard_normal(n).astype(np.float32), rng.standard_normal(batch + (m, n)).astype(np.float32)
    want = a.astype(np.float64) @ b.astype(np.float64) + bias + (c0 if accumulate else 0)
    out = Guarded(F, want.shape, init=c0 if accumulate else None)
    F.matmul(F.DeviceTensor.from_numpy(a), F.DeviceTensor.from_numpy(b), F.DeviceTensor.from_numpy(bias), out=out.tensor,
             flags=flags | F._lib.FORCE_TENSOR_PATH | (F._lib.ACCUMULATE_C if accumulate else 0))
    F.device_status()
    out.check("product", fully_written=not accumulate)
    assert rel_fro(out.tensor.numpy(), want) <= regression_bound_3xtf32(k)


@pytest.mark.parametrize("m,k,n,batch", [
    (2048, 416, 3072, ()),        # 96 tiles of 256 x 256: 22 of them cut into three units
    (2000, 420, 3001, ()),        # ragged edges, unaligned rows
    (2304, 2048, 2050, ()),       # 81 tiles: 7 cut into four units of 512
    (512, 700, 1000, (12,))])     # batched
@pytest.mark.parametrize("mode", ["plain", "accumulate", "gelu", "single pass"])
def test_last_wave_cut_into_units(F, m, k, n, batch, mode):
    """After a whole round, the tiles of a half-empty last wave are computed by several units each, and a finish kernel adds
    their partial tiles with everything the epilogue does to a whole one."""
    rng = _rng(5, m, k, n)
    a, b = rng.standard_normal(batch + (m, k)).astype(np.float32), rng.standard_normal(batch + (k, n)).astype(np.float32)
    bias, c0 = rng.standard_normal(n).astype(np.float32), rng.standard_normal(batch + (m, n)).astype(np.float32)
    ad, bd, biasd = (F.DeviceTensor.from_numpy(x) for x in (a, b, bias))
    assert "tail_ways=0" not in F.plan_describe(a.shape, b.shape)[0]
    want = a.astype(np.float64) @ b.astype(np.float64)
    if mode == "gelu":
        pre, got = F.matmul_bias_gelu(ad, bd, biasd)
        F.device_status()
        assert rel_fro(pre.numpy(), want) <= regression_bound_3xtf32(k)
        v = want + bias
        want = 0.5 * v * (1 + np.tanh(0.7978845608028654 * (v + 0.044715 * v ** 3)))
        assert rel_fro(got.numpy(), want) <= regression_bound_3xtf32(k)
        return
    out = Guarded(F, want.shape, init=c0 if mode == "accumulate" else None)
    flags = {"plain": 0, "accumulate": F._lib.ACCUMULATE_C, "single pass": F._lib.PRECISION_TF32}[mode]
    F.matmul(ad, bd, biasd, out=out.tensor, flags=flags)
    F.device_status()
    out.check("product", fully_written=mode != "accumulate")
    want = want + bias + (c0 if mode == "accumulate" else 0)
    assert rel_fro(out.tensor.numpy(), want) <= (2e-3 if mode == "single pass" else regression_bound_3xtf32(k))


@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (9, 8, 7), (31, 33, 32), (32, 64, 32), (33, 65, 31), (64, 128, 5), (100, 300, 120),
                                   (320, 9, 320), (192, 192, 192), (5, 100, 1000)])
@pytest.mark.parametrize("layout", ["plain", "a transposed", "b transposed", "dc transposed"])
def test_small_products_in_one_launch(F, m, k, n, layout):
    """Plain f32 tiles: edges of the 32 x 32 tile and of the 8 x 8 contraction steps, every side a transposing view, bias,
    accumulation, all three gradients in one launch."""
    rng = _rng(6, m, k, n)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    g, bias = rng.standard_normal((m, n)).astype(np.float32), rng.standard_normal(n).astype(np.float32)

    def dev(x, transposed):
        t = F.DeviceTensor.from_numpy
        return t(np.ascontiguousarray(x.T)).permute((1, 0)) if transposed else t(x)
    ad, bd, gd = dev(a, layout[0] == "a"), dev(b, layout[0] == "b"), dev(g, layout[0] == "d")
    a64, b64, g64 = (x.astype(np.float64) for x in (a, b, g))
    c0 = [rng.standard_normal(s).astype(np.float32) for s in ((m, n), (m, k), (k, n), (n,))]
    lib = F._lib
    for accumulate in (False, True):
        y, da, db, dbias = (Guarded(F, c.shape, init=c if accumulate else None) for c in c0)
        F.matmul(ad, bd, F.DeviceTensor.from_numpy(bias), out=y.tensor, flags=lib.ACCUMULATE_C if accumulate else 0)
        F.matmul_backward(gd, ad, bd, da=da.tensor, db=db.tensor, dbias=dbias.tensor, want_dbias=True,
                          flags=lib.ACCUMULATE_DA | lib.ACCUMULATE_DB | lib.ACCUMULATE_DBIAS if accumulate else 0)
        F.device_status()
        for got, want, c in zip((y, da, db, dbias), (a64 @ b64 + bias, g64 @ b64.T, a64.T @ g64, g64.sum(0)), c0):
            got.check(fully_written=not accumulate)
            assert rel_fro(got.tensor.numpy(), want + (c if accumulate else 0)) <= regression_bound_3xtf32(max(m, k, n))


@pytest.mark.parametrize("n,misalign", [(2 ** 31 - 5, 1), (2 ** 31 + 3, 0)])
def test_bias_rows_past_the_flat_index(F, n, misalign):
    """A row whose elements a 32-bit index does not count, added in place."""
    import torch
    y, bias = torch.rand(n + 8, device="cuda"), torch.empty(n, device="cuda")
    bias.copy_(y[misalign:misalign + n])
    F._lib.check(F._lib.lib().mni_b200_add_bias(y.data_ptr() + 4 * misalign, bias.data_ptr(), y.data_ptr() + 4 * misalign, 1, n, 0))
    torch.cuda.synchronize()
    step = 1 << 28
    for at in range(0, n, step):
        assert torch.equal(y[misalign + at:misalign + min(n, at + step)], 2 * bias[at:at + step]), at


def test_a_call_honours_a_switch_however_many_are_set(F, monkeypatch):
    x, w, dy = (F.DeviceTensor.from_numpy(np.ones(s, np.float32)) for s in ((32, 64), (64, 32), (32, 32)))

    def launches():
        before = F.launch_count()
        F.matmul_backward(dy, x, w)
        return F.launch_count() - before
    assert launches() == 1                       # both products in one f32 kernel
    for i in range(60):
        monkeypatch.setenv(f"MNI_B200_UNUSED_{i}", "1")
    monkeypatch.setenv("MNI_B200_TINY", "0")
    assert launches() >= 2


@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (9, 8, 7), (31, 33, 32), (33, 65, 129), (8, 128, 1024), (320, 320, 64), (3, 70, 517)])
@pytest.mark.parametrize("want_pre", [False, True])
def test_small_products_with_gelu_in_one_launch(F, m, k, n, want_pre):
    rng = _rng(8, m, k, n)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32) / np.sqrt(k).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32)
    launches = F.launch_count()
    pre, out = F.matmul_bias_gelu(*(F.DeviceTensor.from_numpy(x) for x in (a, b, bias)), want_pre=want_pre)
    F.device_status()
    assert F.launch_count() - launches == 1
    want = a.astype(np.float64) @ b.astype(np.float64)
    assert (pre is not None) == want_pre and (not want_pre or rel_fro(pre.numpy(), want) <= regression_bound_3xtf32(k))
    v = want + bias
    assert rel_fro(out.numpy(), 0.5 * v * (1 + np.tanh(0.7978845608028654 * (v + 0.044715 * v ** 3)))) <= regression_bound_3xtf32(k)


@pytest.mark.parametrize("m,k,n", [(9, 40, 7000), (700, 40, 900), (8, 96, 7900), (8, 100, 8300), (4, 64, 8000), (5, 65, 33)])
def test_products_around_the_limits_of_the_small_kernel(F, m, k, n):
    """Either side of the tile limits, eager and captured, whose limits differ: the same products."""
    import torch
    rng = _rng(9, m, k, n)
    a, b, g = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (k, n), (m, n)))
    ad, bd, gd = (F.DeviceTensor.from_numpy(x) for x in (a, b, g))
    a64, b64, g64 = (x.astype(np.float64) for x in (a, b, g))
    outs = [Guarded(F, s) for s in ((m, n), (m, k), (k, n), (n,))]

    def call():
        F.matmul(ad, bd, out=outs[0].tensor)
        F.matmul_backward(gd, ad, bd, da=outs[1].tensor, db=outs[2].tensor, dbias=outs[3].tensor, want_dbias=True)

    def check():
        F.device_status()
        for got, want in zip(outs, (a64 @ b64, g64 @ b64.T, a64.T @ g64, g64.sum(0))):
            got.check()
            assert rel_fro(got.tensor.numpy(), want) <= regression_bound_3xtf32(max(m, k, n))
    call()
    check()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    for o in outs:
        o.tensor.storage.zero_()
    graph.replay()
    check()


@pytest.mark.parametrize("m,k,n,batch", [
    (2048, 3072, 1280, ()),       # 40 tiles of 256 x 256 on 74 pairs, no whole round: cut into three units each
    (1530, 4100, 2047, ()),       # 48, ragged edges, unaligned rows
    (2040, 3080, 3500, ())])      # 112: one round and 38 tiles cut into three
@pytest.mark.parametrize("mode", ["plain", "accumulate", "gelu"])
def test_long_contractions_cut_into_several_rounds_of_units(F, m, k, n, batch, mode):
    rng = _rng(10, m, k, n)
    a, b = rng.standard_normal(batch + (m, k)).astype(np.float32), rng.standard_normal(batch + (k, n)).astype(np.float32)
    b /= np.sqrt(k).astype(np.float32)
    bias, c0 = rng.standard_normal(n).astype(np.float32), rng.standard_normal(batch + (m, n)).astype(np.float32)
    ad, bd, biasd = (F.DeviceTensor.from_numpy(x) for x in (a, b, bias))
    assert "tail_ways=0" not in F.plan_describe(a.shape, b.shape)[0]
    want = a.astype(np.float64) @ b.astype(np.float64)
    if mode == "gelu":
        pre, got = F.matmul_bias_gelu(ad, bd, biasd)
        F.device_status()
        # one accumulator holds a unit's whole share of the contraction here: 2.35e-9 an element and pass of it
        assert rel_fro(pre.numpy(), want) <= regression_bound_3xtf32(k) + 7.1e-9 * k / 3
        v = want + bias
        assert rel_fro(got.numpy(), 0.5 * v * (1 + np.tanh(0.7978845608028654 * (v + 0.044715 * v ** 3)))) <= regression_bound_3xtf32(k) + 7.1e-9 * k / 3
        return
    out = Guarded(F, want.shape, init=c0 if mode == "accumulate" else None)
    F.matmul(ad, bd, biasd, out=out.tensor, flags=F._lib.ACCUMULATE_C if mode == "accumulate" else 0)
    F.device_status()
    out.check("product", fully_written=mode != "accumulate")
    assert rel_fro(out.tensor.numpy(), want + bias + (c0 if mode == "accumulate" else 0)) <= regression_bound_3xtf32(k)
