"""GPU: large products from 16-bit planes of their operands (half.cu and the f16 variants of the tensor-core kernel).

MNI_B200_HALF=1 takes every product there that can go, so that the edges of tiles, of k-blocks and of pieces are reached at small
sizes.  Reference: float64.  Bounds: hi and lo keep 22 bits of each operand and the dropped lo x lo is 2^-24, together below 4e-7
of a product's norm; the f32 accumulate of the f16 pipe loses up to 0.75e-9 per element of a chain of at most 4608 (measured, K =
4096: 3.1e-6).  Three bf16 planes keep 24 bits.  In single-pass mode f16 rounds to 11 bits: 2^-12 at most, per operand."""
import ctypes as C

import numpy as np
import pytest

from conftest import Guarded, rel_fro

pytestmark = pytest.mark.gpu


def _bound(k, single=False):
    return 6e-4 if single else 5e-7 + 1e-9 * min(k, 4608)


@pytest.fixture
def planes(monkeypatch):
    monkeypatch.setenv("MNI_B200_HALF", "1")


SHAPES = [
    # m, k, n, batch, weight shared
    (256, 192, 256, (), False),           # whole tiles
    (129, 130, 131, (), False),           # a little more than a block in every dimension
    (500, 333, 777, (), False),           # nothing aligned
    (384, 4160, 512, (), False),          # a unit of just more than a chain
    (300, 9300, 260, (), False),          # split contraction, several pieces a unit
    (2560, 5000, 2560, (), False),        # many tiles of two pieces
    (2048, 416, 3072, (), False),         # a last wave cut into units
    (300, 200, 260, (5,), False),
    (256, 192, 320, (2, 3), True),        # the weight gradient sums over the batch
]


@pytest.mark.parametrize("m,k,n,batch,shared,bt", [s + (bt,) for s in SHAPES for bt in (False, True) if not bt or s[0] * s[2] < 4e6])
@pytest.mark.parametrize("single", [False, True])
def test_forward_and_gradients(F, planes, m, k, n, batch, shared, bt, single):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m + k + n)
    def normal(*s):
        return torch.randn(s, generator=gen, device="cuda")
    wb = () if shared else batch
    x, w, dy, bias = normal(*batch, m, k), normal(*wb, *((n, k) if bt else (k, n))), normal(*batch, m, n), normal(n)
    wv = w.transpose(-1, -2) if bt else w
    t = F.DeviceTensor.from_torch
    dw_view = t(w).permute(tuple(range(len(wb))) + (len(wb) + 1, len(wb))) if bt else t(w)
    flags = F._lib.PRECISION_TF32 if single else 0
    y = Guarded(F, batch + (m, n), init=np.ones(batch + (m, n), np.float32))
    F.matmul(t(x), dw_view, t(bias), out=y.tensor, flags=flags | F._lib.ACCUMULATE_C)
    add = bt                                      # one of the two layouts accumulates onto ones
    da, db, dbias = (Guarded(F, s, init=np.ones(s, np.float32) if add else None) for s in (batch + (m, k), wb + (k, n), (n,)))
    F.matmul_backward(t(dy), t(x), dw_view, want_dbias=True, da=da.tensor, db=db.tensor, dbias=dbias.tensor,
                      flags=flags | (F._lib.ACCUMULATE_DA | F._lib.ACCUMULATE_DB | F._lib.ACCUMULATE_DBIAS if add else 0))
    F.device_status()
    product = x.double() @ wv.double()
    want = {"y": product + bias.double() + 1, "da": dy.double() @ wv.double().transpose(-1, -2),
            "db": x.double().transpose(-1, -2) @ dy.double(), "dbias": dy.double().reshape(-1, n).sum(0)}
    if shared:
        want["db"] = want["db"].sum(tuple(range(len(batch))))
    fold = int(np.prod(batch)) if shared else 1
    for got, name, length in ((y, "y", k), (da, "da", n), (db, "db", m * fold), (dbias, "dbias", 0)):
        got.check(name, fully_written=name != "y" and not add)
        assert rel_fro(got.tensor.numpy(), want[name].cpu().numpy() + (1 if add and name != "y" else 0)) <= (1e-6 if name == "dbias" else _bound(length, single)), name


@pytest.mark.parametrize("n,misalign,want_pre", [(512, 0, True), (512, 0, False), (500, 0, True), (501, 1, True)])
def test_gelu_epilogue_and_unaligned_outputs(F, planes, n, misalign, want_pre):
    rng = np.random.default_rng(n)
    a, w, bias = (rng.standard_normal(s).astype(np.float32) for s in ((600, 300), (300, n), (n,)))
    w /= np.sqrt(np.float32(300))
    t = F.DeviceTensor.from_numpy
    pre, out = F.matmul_bias_gelu(t(a), t(w), t(bias), want_pre=want_pre)
    plain = Guarded(F, (600, n), misalign=misalign)
    F.matmul(t(a), t(w), t(bias), out=plain.tensor)
    F.device_status()
    want = a.astype(np.float64) @ w
    plain.check("product")
    assert rel_fro(plain.tensor.numpy(), want + bias) <= _bound(300)
    v = want + bias
    assert rel_fro(out.numpy(), 0.5 * v * (1 + np.tanh(0.7978845608028654 * (v + 0.044715 * v ** 3)))) <= _bound(300)
    assert (pre is not None) == want_pre and (pre is None or rel_fro(pre.numpy(), want) <= _bound(300))


def _ranges():
    rng = np.random.default_rng(1)
    m, k, n = 300, 512, 272
    x, w = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    def put(a, at, v):
        a = a.copy()
        a[at] = v
        return a
    spread = np.logspace(-12, 0, k).astype(np.float32)
    few = np.logspace(-4, 0, k).astype(np.float32)
    eye = np.eye(k, n, dtype=np.float32)
    return {
        "small": (x * np.float32(1e-30), w), "large": (x * np.float32(1e30), w * np.float32(1e-20)),
        "subnormal": (x * np.float32(1e-39), w), "largest": (np.full((m, k), 3.4e38, np.float32), eye),
        "row": (put(x, 5, x[5] * np.float32(1e-12)), w), "column": (x, put(w, (slice(None), 7), w[:, 7] * np.float32(1e-12))),
        "contraction": (x * spread, w / spread[:, None]), "contraction within range": (x * few, w / few[:, None]),
        "outlier": (put(x, (3, 4), 1e8), w), "zeros": (x * 0, w), "zero rows": (put(x, slice(10, 200), 0), w),
        "exponents": (np.sign(x) * np.exp2(-40 * rng.random((m, k))).astype(np.float32), eye),
        "infinity": (put(x, (3, 4), np.inf), w), "nan": (x, put(w, (3, 4), np.nan)),
    }


def _sparse():
    """Small numbers in a row, a column or a matrix of few non-zeros, or beside large ones that meet zeros."""
    rng = np.random.default_rng(2)
    m, k, n = 300, 512, 272
    x, w = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, n)).astype(np.float32)
    cases = {}
    for count, scale in ((1, 1e-8), (8, 1e-9), (8, 1e-12), (15, 1e-13), (100, 1e-7)):
        a, b = x.copy(), w.copy()
        a[5] = 0
        b[:, 7] = 0
        for c0 in range(0, k, 256):
            at = c0 + rng.permutation(256)[:count]
            a[5, at], b[at, 7] = x[5, at] * np.float32(scale), w[at, 7] * np.float32(scale)
        cases[f"row of {count} at {scale:g}"], cases[f"column of {count} at {scale:g}"] = (a, w), (x, b)
    a, b = x.copy(), w.copy()
    a[5] *= np.float32(1e-10)
    a[5, ::256] = 1
    b[::256] = 0
    cases["row behind ones"] = (a, b)
    a, b = x.copy(), w.copy()
    b[:, 7] *= np.float32(1e-10)
    b[::16, 7] = 1
    a[:, ::16] = 0
    cases["column behind ones"] = (a, b)
    a, b = x.copy(), w.copy()
    a[5] = 0
    a[5, 3], a[5, 7], b[3] = 1, 1e-10, 0
    cases["one behind a one"] = (a, b)
    long = rng.standard_normal((2048, n)).astype(np.float32)
    for scale in (1e-6, 1e-8, 1e-12):                # none of the diagonal is among the samples that the scale comes from
        cases[f"diagonal {scale:g}"] = (np.eye(2048, dtype=np.float32) * np.float32(scale), long)
    cases["diagonal of many sizes"] = (np.diag(np.logspace(-14, 0, 2048).astype(np.float32)), long)
    return cases


@pytest.mark.parametrize("name", list(_ranges()))
@pytest.mark.parametrize("single", [False, True])
def test_any_range_of_values(F, planes, monkeypatch, name, single):
    """Row by row and column by column: what f16 does not hold goes through bf16 planes.  Infinities and NaN as from f32 operands."""
    x, w = _ranges()[name]
    t = F.DeviceTensor.from_numpy
    flags = F._lib.PRECISION_TF32 if single else 0
    got = F.matmul(t(x), t(w), flags=flags).numpy()
    F.device_status()
    monkeypatch.setenv("MNI_B200_HALF", "0")
    general = F.matmul(t(x), t(w), flags=flags).numpy()
    finite = np.isfinite(general)
    assert np.array_equal(finite, np.isfinite(got))
    if not finite.all():
        return
    _by_rows_and_columns(got, x.astype(np.float64) @ w.astype(np.float64), single)


def _by_rows_and_columns(got, want, single):
    """Single pass: 2^-12 of every operand's element and a sum's rounding; else 2^-22 and that: 2e-6 at K = 512."""
    for axis in (-1, -2):
        error = np.sqrt(((got - want) ** 2).sum(axis))
        assert (error <= (1e-3 if single else 2e-6) * np.sqrt((want ** 2).sum(axis))).all(), axis


@pytest.mark.parametrize("name", list(_sparse()))
@pytest.mark.parametrize("single", [False, True])
def test_rows_and_columns_of_few_small_numbers(F, planes, name, single):
    x, w = _sparse()[name]
    t = F.DeviceTensor.from_numpy
    got = F.matmul(t(x), t(w), flags=F._lib.PRECISION_TF32 if single else 0).numpy()
    F.device_status()
    _by_rows_and_columns(got, x.astype(np.float64) @ w.astype(np.float64), single)


@pytest.mark.parametrize("single", [False, True])
def test_small_columns_beside_ordinary_ones_of_the_next_matrix(F, planes, single):
    """A block of the pass takes ten tiles of 16 rows here and a matrix has four: no matrix has a block of its own."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(3)
    x, dy = (torch.randn(s, generator=gen, device="cuda") for s in ((555, 64, 200), (555, 64, 136)))
    for b in range(555):
        x[b, :, b % 200] *= 1e-12
    t = F.DeviceTensor.from_torch
    _, dw = F.matmul_backward(t(dy), t(x), t(torch.zeros(555, 200, 136, device="cuda")), need_da=False,
                              flags=F._lib.PRECISION_TF32 if single else 0)
    F.device_status()
    _by_rows_and_columns(dw.numpy(), (x.double().transpose(1, 2) @ dy.double()).cpu().numpy(), single)


@pytest.mark.parametrize("single", [False, True])
def test_ordinary_values_stay_in_f16(F, planes, single):
    """The verdict of the pass, which follows the blocks' words at the start of the scratch: what f16 holds is not sent to the
    planes that take longer; a scattering of more small elements than a sixteenth is."""
    import torch
    rng = np.random.default_rng(6)
    def normal(*s):
        return rng.standard_normal(s).astype(np.float32)
    x, w = normal(1000, 700), normal(700, 520)
    half_off = np.where(normal(1000, 700) > 0, x, 0).astype(np.float32)
    cases = {"normal": (x, w), "uniform": (rng.random((1000, 700), np.float32), w), "halves": (half_off, w), "narrow": (normal(1000, 257), normal(257, 520)),
             "few": (np.where(rng.random((1000, 700)) < 0.02, x, 0).astype(np.float32), w), "one hot": (np.eye(700, dtype=np.float32)[rng.integers(0, 700, 1000)], w),
             "gelu": (0.5 * x * (1 + np.tanh(0.7978845608 * (x + 0.044715 * x ** 3))), w * np.float32(0.02)), "scaled rows": (x * np.float32(10) ** rng.uniform(-3, 1, (1000, 1)).astype(np.float32), w)}
    lib, room = F._lib.lib(), 64 << 20
    buf = torch.empty(room, dtype=torch.uint8, device="cuda")
    F._lib.check(lib.mni_b200_workspace_set(C.c_void_p(buf.data_ptr()), room))
    scattered = x.copy()
    scattered[np.add.outer(np.arange(1000), np.arange(700)) % 11 == 0] *= np.float32(1e-9)      # nowhere a fifth of a row or column
    try:
        for name, (a, b) in {**cases, "scattered": (scattered, w)}.items():
            a, b = F.DeviceTensor.from_numpy(np.ascontiguousarray(a, np.float32)), F.DeviceTensor.from_numpy(b)
            F.matmul(a, b, flags=F._lib.PRECISION_TF32 if single else 0)
            F.device_status()
            blocks = min(148 * 3, sum(-(-r // 16) * -(-(-(-c // 64) * 64) // 512) for r, c in (a.shape, b.shape)))
            words = buf[:4 * (blocks + 1)].view(torch.int32)
            assert int(words[blocks]) == (name == "scattered") and bool(words.any()) == (name == "scattered"), name
    finally:
        F._lib.check(lib.mni_b200_workspace_set(None, 0))


@pytest.mark.parametrize("at", ["left", "right", "both"])
@pytest.mark.parametrize("single", [False, True])
def test_infinities_as_from_f32_operands(F, planes, monkeypatch, at, single):
    """Against finite numbers of one bf16 and of more, of either sign, zero, and an infinity: the same infinities, the same NaN."""
    rng = np.random.default_rng(7)
    x, w = (rng.standard_normal(s).astype(np.float32) for s in ((300, 320), (320, 272)))
    w[4, :4], x[:4, 5] = (1, -2, 0, 1e-30), (1, -2, 0, 1e-30)
    if at != "right":
        x[10, 4], x[11, 4] = np.inf, -np.inf
    if at != "left":
        w[5, 20], w[5, 21] = np.inf, -np.inf
    if at == "both":
        w[4, 30], w[4, 31] = np.inf, -np.inf
    t = F.DeviceTensor.from_numpy
    flags = F._lib.PRECISION_TF32 if single else 0
    got = F.matmul(t(x), t(w), flags=flags).numpy()
    F.device_status()
    monkeypatch.setenv("MNI_B200_HALF", "0")
    general = F.matmul(t(x), t(w), flags=flags).numpy()
    assert np.array_equal(np.isnan(general), np.isnan(got)) and not np.isfinite(general).all()
    infinite = np.isinf(general)
    assert np.array_equal(infinite, np.isinf(got)) and np.array_equal(general[infinite], got[infinite])
    assert infinite.any() == single                  # in three passes inf - inf is what is left of one


def test_without_scratch_for_the_planes_the_product_comes_from_f32(F, planes, monkeypatch):
    """A buffer that the general path fits in and the planes do not, and a capture that may not grow the library's own."""
    import torch
    rng = np.random.default_rng(9)
    a, b, g = (rng.standard_normal(s).astype(np.float32) for s in ((512, 512), (512, 512), (512, 512)))
    t = F.DeviceTensor.from_numpy
    ad, bd, gd = t(a), t(b), t(g)
    want = {"y": a.astype(np.float64) @ b, "da": g.astype(np.float64) @ b.T, "db": a.T.astype(np.float64) @ g}
    lib, general = F._lib.lib(), 32 << 20
    buf = torch.empty(general + 256, dtype=torch.uint8, device="cuda")
    small = t(rng.standard_normal((4096, 4096)).astype(np.float32))
    F._lib.check(lib.mni_b200_workspace_set(C.c_void_p((buf.data_ptr() + 255) // 256 * 256), general))
    try:
        y, (da, db) = F.matmul(ad, bd), F.matmul_backward(gd, ad, bd)
        launches = F.launch_count()
        F.matmul(small, small)                       # its planes need 200 MB
        assert F.launch_count() - launches <= 2      # the product and a finish
        F.device_status()
    finally:
        F._lib.check(lib.mni_b200_workspace_set(None, 0))
    for got, name in ((y, "y"), (da, "da"), (db, "db")):
        assert rel_fro(got.numpy(), want[name]) <= 5e-6, name
    F._lib.check(lib.mni_b200_release())
    monkeypatch.setenv("MNI_B200_HALF", "0")
    F.matmul(small, small)                           # scratch for this, eagerly
    monkeypatch.setenv("MNI_B200_HALF", "1")
    out, stream = F.DeviceTensor.empty((4096, 4096)), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            F.matmul(small, small, out=out)
    F.matmul(small, small)                           # its planes make the library's scratch grow: the graph keeps its own
    out.torch_view().zero_()
    graph.replay()
    F.device_status()
    s = small.torch_view().double()
    assert float((out.torch_view().double() - s @ s).norm() / (s @ s).norm()) <= 2e-5


def test_capture_before_there_is_any_scratch(F):
    """The first call after a release is a captured one: it allocates nothing, and needs nothing from f32 operands."""
    import torch
    x, w, out = (F.DeviceTensor.from_torch(torch.randn(s, device="cuda")) for s in ((4096, 1024), (1024, 4096), (4096, 4096)))
    F._lib.check(F._lib.lib().mni_b200_release())
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            F.matmul(x, w, out=out)
    graph.replay()
    F.device_status()
    want = x.torch_view().double() @ w.torch_view().double()
    assert float((out.torch_view().double() - want).norm() / want.norm()) <= 2e-5


@pytest.fixture
def little_memory():
    """All of the device's memory but 80 MB taken, until release() is called."""
    import torch
    hog = []
    def take():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        hog.append(torch.empty(torch.cuda.mem_get_info()[0] - (80 << 20), dtype=torch.uint8, device="cuda"))
    def release():
        hog.clear()
        torch.cuda.empty_cache()
    yield take, release
    release()


@pytest.mark.parametrize("recorded", [False, True])
def test_planes_that_do_not_fit_leave_the_scratch_there_was(F, little_memory, recorded):
    """A small call that has run can be captured, although a larger one found no memory for its planes in between."""
    import torch
    x, w, out = (F.DeviceTensor.from_torch(torch.randn(s, device="cuda")) for s in ((8192, 1024), (1024, 8192), (8192, 8192)))
    a, c = (F.DeviceTensor.from_torch(torch.randn(512, 512, device="cuda")) for _ in range(2))
    want = a.torch_view().double() @ a.torch_view().double()
    F._lib.check(F._lib.lib().mni_b200_release())
    def small():
        F.matmul(a, a, out=c)                        # four splits, in scratch
    def capture(call):
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            with torch.cuda.graph(graph, stream=stream):
                call()
        return graph
    small()
    capture(c.torch_view().zero_)                    # what torch needs for its first capture
    first = capture(small) if recorded else None
    little_memory[0]()
    launches = F.launch_count()
    F.matmul(x, w, out=out)                          # planes of 100 MB
    assert F.launch_count() - launches == 1
    for graph in (first, capture(small)):
        if graph is not None:
            c.torch_view().zero_()
            graph.replay()
            F.device_status()
            assert float((c.torch_view().double() - want).norm() / want.norm()) <= 5e-6


def test_planes_are_tried_again_once_there_is_memory(F, little_memory):
    import torch
    x, w, out = (F.DeviceTensor.from_torch(torch.randn(s, device="cuda")) for s in ((8192, 1024), (1024, 8192), (8192, 8192)))
    F._lib.check(F._lib.lib().mni_b200_release())
    def launches():
        before = F.launch_count()
        F.matmul(x, w, out=out)
        return F.launch_count() - before
    little_memory[0]()
    assert (launches(), launches()) == (1, 1)
    little_memory[1]()
    assert (launches(), launches()) == (3, 3)        # two passes over the operands and the product
    F.device_status()


def test_queried_scratch_holds_the_planes(F, planes):
    import torch
    rng = np.random.default_rng(4)
    a, b, g = (F.DeviceTensor.from_numpy(rng.standard_normal(s).astype(np.float32)) for s in ((700, 333), (333, 500), (700, 500)))
    lib, need = F._lib.lib(), C.c_size_t(0)
    F._lib.check(lib.mni_b200_workspace_query(a.view_struct(), b.view_struct(), 0, C.byref(need)))
    buf = torch.full((need.value + 4352,), 0x5A, dtype=torch.uint8, device="cuda")
    base = (buf.data_ptr() + 255) // 256 * 256
    F._lib.check(lib.mni_b200_workspace_set(C.c_void_p(base), need.value))
    try:
        before = F.launch_count()
        F.matmul(a, b)
        assert F.launch_count() - before >= 3         # the passes over the operands, the product
        F.matmul_backward(g, a, b, want_dbias=True)
        F.device_status()
    finally:
        F._lib.check(lib.mni_b200_workspace_set(None, 0))
    assert bool((buf[base - buf.data_ptr() + need.value:] == 0x5A).all())


@pytest.mark.parametrize("shape", [(1024, 512, 768), (2048, 768, 3072), (512, 320, 512, 3)])
@pytest.mark.parametrize("exchanged,off", [(False, 0), (False, 1), (True, 0), (True, 1)])
def test_queried_scratch_serves_every_view_of_the_gradient(F, monkeypatch, shape, exchanged, off):
    """The call takes the same launches from a buffer of the queried size as from the library's own scratch."""
    import torch
    (m, k, n), lead = shape[:3], shape[3:]
    x, w = (F.DeviceTensor.from_torch(torch.randn(s, device="cuda")) for s in (lead + (m, k), lead + (k, n)))
    size = m * n * int(np.prod(lead))
    g = F.DeviceTensor(torch.randn(size + off, device="cuda")[off:], lead + ((n, m) if exchanged else (m, n)))
    if exchanged:
        g = g.permute(tuple(range(len(lead))) + (len(lead) + 1, len(lead)))
    def launches(**kw):
        before = F.launch_count()
        F.matmul_backward(g, x, w, **kw)
        return F.launch_count() - before
    lib, need = F._lib.lib(), C.c_size_t(0)
    wanted = [dict(want_dbias=True), dict(), dict(need_da=False, want_dbias=True), dict(need_db=False)]
    for half in ("0", "1", None):
        monkeypatch.setenv("MNI_B200_HALF", half) if half else monkeypatch.delenv("MNI_B200_HALF")
        own = [launches(**kw) for kw in wanted]
        F._lib.check(lib.mni_b200_workspace_query(x.view_struct(), w.view_struct(), 0, C.byref(need)))
        buf = torch.empty(need.value + 256, dtype=torch.uint8, device="cuda")
        F._lib.check(lib.mni_b200_workspace_set(C.c_void_p((buf.data_ptr() + 255) // 256 * 256), need.value))
        try:
            assert [launches(**kw) for kw in wanted] == own, half
        finally:
            F.device_status()
            F._lib.check(lib.mni_b200_workspace_set(None, 0))


@pytest.mark.parametrize("flags", [0, 1])
def test_wait_limit_runs_out_then_the_library_recovers(F, planes, monkeypatch, flags):
    """As test_timeout_gpu.py does for the other variants: a stage that is armed and never filled."""
    rng = np.random.default_rng(5)
    a, b = (rng.standard_normal((512, 512), dtype=np.float32) for _ in range(2))
    ad, bd = F.DeviceTensor.from_numpy(a), F.DeviceTensor.from_numpy(b)
    F.device_status()
    monkeypatch.setenv("MNI_B200_WAIT_CYCLES", "2000000")
    monkeypatch.setenv("MNI_B200_TEST_WITHHOLD_KBLOCK", "3")
    F.matmul(ad, bd, flags=flags)
    with pytest.raises(F._lib.MniError) as ei:
        F.device_status()
    assert ei.value.status == 8
    monkeypatch.delenv("MNI_B200_TEST_WITHHOLD_KBLOCK")
    monkeypatch.delenv("MNI_B200_WAIT_CYCLES")
    out = F.matmul(ad, bd, flags=flags)
    assert F.device_status() == 0
    assert rel_fro(out.numpy(), a.astype(np.float64) @ b) <= _bound(512, flags == 1)


def test_replayed_graph_looks_at_the_values_each_time(F, planes):
    """Scale and range are found on the device: a graph replayed with other values in the same buffers is right for those."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(8)
    x, w = torch.randn(300, 500, generator=gen, device="cuda"), torch.randn(500, 400, generator=gen, device="cuda")
    xt, wt, out = F.DeviceTensor.from_torch(x), F.DeviceTensor.from_torch(w), F.DeviceTensor.empty((300, 400))
    F.matmul(xt, wt, out=out)                        # scratch
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            F.matmul(xt, wt, out=out)
    first = x.clone()
    spread = torch.logspace(-15, 10, 500, device="cuda")
    for value in (first, first * 1e-20, first * spread, first * 1e25, first):
        x.copy_(value)
        graph.replay()
        F.device_status()
        want = x.double() @ w.double()
        assert float((out.torch_view().double() - want).norm() / want.norm()) <= _bound(500)
