"""CPU: which calls are computed from 16-bit planes of their operands, and how their units are dealt out.  (The reference hands
every product to cuBLAS, ops/matmul.rs:145-190.)"""
import re

import pytest

from framework_b200 import _lib


@pytest.fixture(scope="module")
def plan():
    from framework_b200 import build, ops
    build.build_library()
    return ops.plan_describe


def planes(lines):
    return [{k: int(v) for k, v in re.findall(r"(\w+)=(-?\d+)", line)} for line in lines if ": planes " in line]


@pytest.mark.parametrize("a,b,flags,forward,backward", [
    ((4096, 1024), (1024, 4096), 0, 1, 2), ((64, 1024, 768), (768, 3072), 0, 1, 2), ((8192, 8192), (8192, 8192), 1, 1, 2),
    ((2048, 768), (768, 3072), 0, 0, 2),                                           # both gradients pay, the forward does not
    ((8192, 8192), (8192, 512), 0, 0, 2), ((256, 8192), (8192, 8192), 0, 0, 0),    # operands too large for the work
    ((1024, 1024), (1024, 1024), 0, 0, 0), ((8, 12, 512, 64), (8, 12, 64, 512), 0, 0, 0), ((16, 4096), (4096, 4096), 0, 0, 0),
    ((4096, 1024), (1024, 4096), _lib.FORCE_TENSOR_PATH, 0, 0), ((4096, 1024), (1024, 4096), _lib.force_split_k(2), 0, 0)])
def test_calls_from_16_bit_planes(plan, a, b, flags, forward, backward):
    """The plan names the f32 path first, which serves where there is no scratch for the planes."""
    for backward_call, want in ((0, forward), (1, backward)):
        lines = plan(a, b, flags=flags, backward=backward_call)
        assert len(planes(lines)) == want, lines
        kinds = ["planes" if ": planes " in line else "f32" if ": tensor " in line else
                 "instead" if "with scratch for 16-bit operands" in line else "" for line in lines]
        named = [kind for kind in kinds if kind]
        if want:
            assert named == ["f32"] * named.count("f32") + ["instead"] + ["planes"] * want and named[0] == "f32", lines
        else:
            assert set(named) <= {"f32"}, lines


@pytest.mark.parametrize("m,k,n", [(2048, 3072, 768), (1000, 1333, 2777), (700, 5000, 3000), (4096, 4096, 4096), (8192, 768, 3072)])
@pytest.mark.parametrize("sms", [148, 132, 66])
def test_units_fill_the_pairs(plan, monkeypatch, m, k, n, sms):
    """Splits and cuts stay within the contraction, only the launch's last product is cut, and few tiles are made into more units."""
    monkeypatch.setenv("MNI_B200_HALF", "1")
    for backward in (0, 1):
        got = planes(plan((m, k), (k, n), backward=backward, sm_count=sms))
        assert len(got) == 1 + backward
        units = 0
        for i, p in enumerate(got):
            tiles = -(-p["m"] // 256) * -(-p["n"] // 256)
            assert p["k"] / max(p["splits"], p["tail_ways"], 1) >= 256 and (p["tail_ways"] == 0 or i == len(got) - 1)
            assert p["splits"] == 1 or p["tail_ways"] == 0
            units += tiles * p["splits"]
        cut = got[-1]["tail_ways"]
        units += (units % (sms // 2)) * (cut - 1) if cut else 0
        assert all(p["grid"] == 2 * min(units, sms // 2) for p in got)
