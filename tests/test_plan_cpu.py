"""CPU: the launch planner, pinned at the benchmark configurations.

Which kernel a product takes -- tile width, CTA pairing, the A operand from tensor memory, the split of the
contraction, the cut or balanced tail, how many SMs two side-by-side products get, streaming kernels for few rows,
pieces of a long contraction -- is host arithmetic over shapes, strides and the SM count, so it is checked here
without a device through `mni_b200_plan_describe`.  The pins are the plans the measured numbers were taken
with: a change of the planner that moves one of them is a performance change and must be re-measured.  (The
reference has no counterpart: it hands every product to cuBLAS, ops/matmul.rs:145-190.)"""
import re

import pytest


@pytest.fixture(scope="module")
def plan():
    from framework_b200 import build, ops
    build.build_library()
    return ops.plan_describe


def fields(line):
    """'grad_a: tensor m=512 n=64 ...' -> ('grad_a', 'tensor', {'m': 512, ...})"""
    label, rest = line.split(": ", 1)
    kind = rest.split(" ", 1)[0]
    return label, kind, {k: int(v) for k, v in re.findall(r"(\w+)=(-?\d+)", rest)}


def by_label(lines):
    out = {}
    for line in lines:
        if ": " in line:
            label, kind, f = fields(line)
            out.setdefault(label, []).append((kind, f, line))
    return out


def tensor_plan(lines, label):
    entries = [e for e in by_label(lines)[label] if e[0] == "tensor"]
    assert len(entries) == 1, lines
    return entries[0][1]


def test_default_benchmark_shape_whole_and_as_an_eighth(plan):
    """[64,1024,768] x [768,3072]: 256-wide CTA pairs on every SM; the weight gradient folds the batches into the
    contraction and splits it two ways (72 units on 72 pairs), summed in pieces of about 1024."""
    for batches in (64, 8):
        fwd = tensor_plan(plan((batches, 1024, 768), (768, 3072)), "forward")
        assert (fwd["bn"], fwd["bk"], fwd["pair"], fwd["tmem_a"], fwd["splits"], fwd["grid"]) == (256, 16, 1, 0, 1, 148)
        assert fwd["batch"] == batches and fwd["pieces"] == 1
        bwd = plan((batches, 1024, 768), (768, 3072), backward=1)
        da, dw = tensor_plan(bwd, "grad_a"), tensor_plan(bwd, "grad_b")
        assert (da["m"], da["n"], da["k"], da["batch"], da["pieces"]) == (1024, 768, 3072, batches, 3)
        assert (dw["m"], dw["n"], dw["k"], dw["batch"], dw["fold"]) == (768, 3072, 1024, 1, batches)
        assert (dw["splits"], dw["grid"]) == (2, 144)
        assert dw["pieces"] == batches // 2                  # (batches * 1024 / 2) / 1024
        assert not any("side by side" in line for line in bwd)        # large products run one after the other
        # whole: 768 pair-tiles = 10.4 rounds, the ragged wave is left alone; an eighth: 96 tiles on 74 pairs
        # would be two rounds at 0.65 -> the last wave's 22 tiles are cut
        assert da["tail"] == (1 if batches == 8 else 0) and da["grid"] == 148


def test_reserved_sms_shrink_the_grid(plan):
    """What the step driver reserves for the collective comes out of the persistent grid, in whole pairs."""
    for sms, grid in ((148, 148), (146, 146), (132, 132)):
        assert tensor_plan(plan((64, 1024, 768), (768, 3072), sm_count=sms), "forward")["grid"] == grid


def test_linear_layer(plan):
    """x[4096,1024] . W[1024,4096] + b: one round of pair tiles; the bias gradient's column sums go beside the
    products; both gradients contract over 4096 in four pieces."""
    fwd = tensor_plan(plan((4096, 1024), (1024, 4096)), "forward")
    assert (fwd["bn"], fwd["pair"], fwd["splits"], fwd["tail"], fwd["pieces"]) == (256, 1, 1, 0, 1)
    bwd = plan((4096, 1024), (1024, 4096), backward=2)
    assert any(line.startswith("grad_bias: column sums") and "side stream" in line for line in bwd)
    for label in ("grad_a", "grad_b"):
        g = tensor_plan(bwd, label)
        assert (g["bn"], g["pair"], g["splits"], g["pieces"], g["grid"]) == (256, 1, 1, 4, 128)


def test_attention_shapes_strided_key_and_narrow_outputs(plan):
    """S = Q.K^T with K read through its strides (no gather), O = S.V with 64-wide tiles and A from tensor
    memory; the two gradients of each run side by side on half of the SMs; dK^T (64 rows) is computed with
    the operands exchanged."""
    q, kt = (8, 12, 512, 64), (8, 12, 64, 512)
    s_fwd = plan(q, kt, b_strides=(393216, 32768, 1, 64))
    assert not any("gather" in line for line in s_fwd)
    f = tensor_plan(s_fwd, "forward")
    assert (f["bn"], f["pair"], f["batch"], f["k"], f["grid"]) == (256, 1, 96, 64, 148)
    s_bwd = plan(q, kt, b_strides=(393216, 32768, 1, 64), backward=1)
    assert any("side by side" in line for line in s_bwd)
    dq, dkt = tensor_plan(s_bwd, "grad_a"), tensor_plan(s_bwd, "grad_b")
    assert (dq["bn"], dq["tmem_a"], dq["grid"], dq["exchanged"]) == (64, 1, 74, 0)
    assert (dkt["bn"], dkt["tmem_a"], dkt["grid"], dkt["exchanged"]) == (64, 1, 74, 1)
    o_fwd = tensor_plan(plan((8, 12, 512, 512), (8, 12, 512, 64)), "forward")
    assert (o_fwd["bn"], o_fwd["tmem_a"], o_fwd["pair"], o_fwd["splits"], o_fwd["grid"]) == (64, 1, 0, 1, 148)
    assert o_fwd["mma_n"] == 64
    o_bwd = plan((8, 12, 512, 512), (8, 12, 512, 64), backward=1)
    ds, dv = tensor_plan(o_bwd, "grad_a"), tensor_plan(o_bwd, "grad_b")
    assert (ds["bn"], ds["pair"], ds["grid"]) == (256, 1, 74)
    assert (dv["bn"], dv["tmem_a"], dv["grid"]) == (64, 1, 74)


def test_small_square_is_split_over_the_gpu(plan):
    """512^3 has 8 tiles of 128 x 256: the cost model picks narrow tiles and a 4-way split instead."""
    f = tensor_plan(plan((512, 512), (512, 512)), "forward")
    assert (f["bn"], f["tmem_a"], f["splits"], f["grid"]) == (64, 1, 4, 128)
    bwd = plan((512, 512), (512, 512), backward=1)
    assert any("side by side" in line for line in bwd)
    for label in ("grad_a", "grad_b"):
        g = tensor_plan(bwd, label)
        assert g["splits"] * (512 // 128) * (512 // g["bn"]) == g["grid"] <= 74


def test_long_contraction_is_summed_in_pieces(plan):
    f = tensor_plan(plan((8192, 8192), (8192, 8192)), "forward")
    assert (f["bn"], f["pair"], f["splits"], f["grid"], f["pieces"]) == (256, 1, 1, 148, 8)


def test_few_rows_take_the_streaming_kernels(plan):
    """M = 1, 4 at K = N = 4096: all three products stream the weight through CUDA-core kernels; at 16 rows the
    tensor path takes over, forward and input gradient with the operands exchanged."""
    for rows in (1, 4):
        fwd = plan((rows, 4096), (4096, 4096))
        assert fwd == ["forward: streaming (skinny) forward kernel"]
        bwd = by_label(plan((rows, 4096), (4096, 4096), backward=1))
        assert bwd["grad_a"][0][0] == "streaming" and bwd["grad_b"][0][0] == "streaming"
    f = tensor_plan(plan((16, 4096), (4096, 4096)), "forward")
    assert (f["exchanged"], f["m"], f["n"], f["bn"], f["tmem_a"], f["splits"]) == (1, 4096, 16, 64, 1, 4)
    assert f["mma_n"] == 16                              # a 64-wide tile over 16 columns multiplies 16
    bwd = plan((16, 4096), (4096, 4096), backward=1)
    assert tensor_plan(bwd, "grad_a")["exchanged"] == 1
    dw = tensor_plan(bwd, "grad_b")
    assert (dw["m"], dw["n"], dw["k"], dw["bn"], dw["pair"]) == (4096, 4096, 16, 256, 1)


def test_flags_and_undescribable_views(plan):
    """The single-pass flag reaches the plan; a view whose matrix dims both have a stride other than one cannot be
    described to TMA and is gathered first; a forced split is honoured."""
    from framework_b200 import _lib
    f = tensor_plan(plan((1024, 1024), (1024, 1024), flags=_lib.PRECISION_TF32 | _lib.FORCE_TENSOR_PATH), "forward")
    assert f["single_pass"] == 1 and f["bk"] == 32
    strided = plan((256, 256), (256, 256), a_strides=(512, 2))
    assert any("gather of a strided operand" in line for line in strided)
    assert tensor_plan(plan((256, 256), (256, 256), flags=_lib.force_split_k(3)), "forward")["splits"] == 3


def test_mma_width_follows_the_output_width(plan):
    """Lone-CTA tiles wider than the output: MMAs in units of 16 columns for a K-major B (here b is given
    transposed, so its rows are contiguous along the contraction), whole 32-float chunks for an MN-major one."""
    from framework_b200 import _lib
    t = _lib.FORCE_TENSOR_PATH
    k_major = {n: tensor_plan(plan((128, 256), (256, n), b_strides=(1, 256), flags=t), "forward")["mma_n"]
               for n in (8, 16, 24, 40, 64, 100)}
    assert k_major == {8: 16, 16: 16, 24: 32, 40: 48, 64: 64, 100: 64}      # 100 columns: two 64-wide tiles
    mn_major = {n: tensor_plan(plan((128, 256), (256, n), flags=t), "forward")["mma_n"] for n in (8, 40, 64, 100)}
    assert mn_major == {8: 32, 40: 64, 64: 64, 100: 64}
    # CTA pairs keep full-width MMAs
    wide = tensor_plan(plan((32768, 256), (256, 200), flags=t), "forward")
    assert (wide["bn"], wide["pair"], wide["mma_n"]) == (256, 1, 256)


@pytest.mark.parametrize("flags", [0, 1])
def test_exchanged_operands_keep_to_the_plans_that_store_transposed(plan, monkeypatch, flags):
    """Few rows and many columns are computed as C^T.  At a forced width of 256 that is a 256-wide pair problem, but the split
    tail and the running sum store no transposed patches: neither may be planned, whatever the last wave and the contraction."""
    monkeypatch.setenv("MNI_B200_BN", "256")
    from framework_b200 import _lib
    for m, k, n in ((48, 512, 20480), (64, 2048, 20000), (32, 8192, 4096), (32, 8000, 32768), (17, 256, 19200)):
        f = tensor_plan(plan((m, k), (k, n), flags=flags | _lib.FORCE_TENSOR_PATH), "forward")
        assert (f["exchanged"], f["bn"], f["pair"], f["tail_ways"], f["running"]) == (1, 256, 1, 0, 0), f
    plain = tensor_plan(plan((8192, 8192), (8192, 8192), flags=flags), "forward")
    assert (plain["exchanged"], plain["running"]) == (0, 1)
    cut = tensor_plan(plan((2048, 768), (768, 3072), flags=flags), "forward")
    assert (cut["exchanged"], cut["tail_ways"]) == (0, 3)


def test_long_contractions_over_a_ragged_wave_are_cut(plan):
    """A partly filled wave of 256-wide pairs, alone or last, is cut into units where the contraction is long enough to pay for
    adding them; the grid is then full.  Narrow tiles in a few long rounds are split."""
    def f(m, k, n, batch=(), **kw):
        return tensor_plan(plan(batch + (m, k), batch + (k, n), **kw), "forward")
    for m, k, n, ways in ((2048, 4096, 1280, 5), (1536, 8192, 2048, 3), (1280, 8192, 2560, 4), (2048, 3072, 3584, 3)):
        p = f(m, k, n)
        assert (p["bn"], p["pair"], p["splits"], p["tail_ways"], p["grid"], p["running"]) == (256, 1, 1, ways, 148, 0), p
    for m, k, n in ((2048, 2048, 3584), (2048, 1024, 3584), (4096, 1024, 4096), (8192, 8192, 8192), (2048, 2048, 1280)):
        assert f(m, k, n)["tail_ways"] == 0, (m, k, n)
    assert f(2048, 8192, 3584, flags=1)["tail_ways"] == 0
    assert f(384, 4096, 64, (100,))["splits"] > 1 and f(384, 512, 64, (100,))["splits"] == 1


def test_nine_to_fifteen_rows_against_aligned_weights(plan):
    """The warp-level kernels take them with short contractions, or up to 16 M elements with as many outputs as the contraction
    is long; the tensor path streams larger weights better, and then takes both gradients."""
    for k, n, fwd, dx in ((1024, 4096, True, False), (4096, 4096, True, True), (2792, 3880, True, False), (8192, 8192, False, False),
                          (4096, 12000, False, False), (6000, 3000, False, False), (8191, 8191, True, True)):
        assert ("few rows" in plan((9, k), (k, n))[0]) == fwd, (k, n)
        b = by_label(plan((9, k), (k, n), backward=1))
        assert ("few rows" in b["grad_a"][0][2]) == dx and "streaming" in b["grad_b"][0][2], (k, n)


def test_streamed_gradients_that_fill_the_memory_run_in_turn(plan):
    def beside(m, k, n):
        return any("side" in line for line in plan((m, k), (k, n), backward=1))
    for shape, want in (((1, 4096, 4096), True), ((4, 8192, 8192), True), ((1, 8192, 8192), False), ((9, 4096, 4096), False),
                        ((12, 4096, 12000), False), ((9, 1024, 4096), True), ((15, 4096, 4096), True)):
        assert beside(*shape) == want, shape


def test_a_wave_beside_another_product_is_left_whole(plan):
    """24 pair tiles on half of the device, the other half busy with grad_a."""
    b = plan((19, 104, 1847), (1847, 661), b_strides=(1, 1847), backward=1)
    assert any("side by side" in line for line in b)
    assert tensor_plan(b, "grad_b")["tail_ways"] == 0


def test_small_products_are_those_of_few_tiles(plan):
    """The one-launch f32 kernel takes calls of at most 900 tiles of 32 x 32 (two gradients 1200), and of few rows only where the streaming kernels,
    which read the weight in 16-byte units, do not do better."""
    def small(m, k, n, backward=0):
        return all("small f32 kernel" in line for line in plan((m, k), (k, n), backward=backward))
    for shape in ((32, 64, 32), (128, 128, 128), (192, 192, 192), (9, 8, 7), (700, 3, 1000), (8, 8, 4512), (8, 90, 1656), (2, 8, 3568), (1, 1, 1)):
        assert small(*shape), shape
    for shape in ((2048, 1, 4096), (100000, 2, 40), (65536, 128, 1), (9, 1, 900000), (1024, 8, 1024), (4096, 4, 512),      # tiles
                  (1, 128, 65536), (1, 64, 131072), (8, 16, 65536), (1, 128, 1024), (8, 8, 37266), (1, 8, 19862), (256, 512, 64), (8, 128, 8192)):
        assert not small(*shape), shape
    for shape in ((32, 64, 32), (8, 12704, 8), (4, 4096, 64), (100, 1, 300), (13, 5616, 99)):
        assert small(*shape, backward=2), shape
    for shape in ((1, 65536, 128), (300, 27000, 1), (1, 131072, 64), (8, 65536, 16)):
        assert not small(*shape, backward=2), shape


def test_staging_patches_are_one_or_two(plan, monkeypatch):
    """A patch per epilogue warp more costs pipeline stages; any other number than two leaves the default."""
    def stages():
        return tensor_plan(plan((4096, 1024), (1024, 4096)), "forward")["stages"]
    default = stages()
    for value, same in (("1", True), ("2", False), ("3", True), ("4", True), ("8", True)):
        monkeypatch.setenv("MNI_B200_EPI_PATCHES", value)
        assert (stages() == default) == same, value


@pytest.mark.parametrize("others", [0, 46, 47, 48, 60])
def test_a_switch_counts_however_many_are_set(plan, monkeypatch, others):
    for i in range(others):
        monkeypatch.setenv(f"MNI_B200_UNUSED_{i}", "1")
    monkeypatch.setenv("MNI_B200_BN", "64")
    assert tensor_plan(plan((4096, 1024), (1024, 4096)), "forward")["bn"] == 64
    monkeypatch.delenv("MNI_B200_BN")
    assert tensor_plan(plan((4096, 1024), (1024, 4096)), "forward")["bn"] == 256


def test_errors_are_the_calls_own(plan):
    from framework_b200 import _lib
    with pytest.raises(_lib.MniError) as ei:
        plan((2, 3), (4, 2))
    assert ei.value.status == 2 and "inner dimensions must match" in ei.value.message
    with pytest.raises(_lib.MniError) as ei:
        plan((2, 3), (3, 2), sm_count=0)
    assert ei.value.status == 4
