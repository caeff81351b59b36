"""CPU: the benchmark's host logic -- work per configuration, sharding of the workloads, the `config` object both
arms print, and the sizing of the CPU samples."""
import importlib.util
import os

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_algorithmic_flops_per_configuration(bench):
    """fwd + bwd = 3 GEMMs of 2*M*N*K per batch (6 for the attention-shaped configuration)."""
    want = {"c1": 0.805e9, "c2": 103.08e9, "c3": 19.33e9, "c4": 927.7e9, "c5a": 3298.5e9,
            "c5b1": 0.1007e9, "c5b4": 0.4027e9, "c5b16": 1.611e9}
    for name, flops in want.items():
        assert abs(bench.WORKLOADS[name].flops - flops) / flops < 1e-3, name
    assert bench.WORKLOADS["c3"].out_shape == (8, 12, 512, 512)
    assert bench.WORKLOADS["c3"].b_logical == (8, 12, 64, 512)          # K^T through the permute view
    assert bench.WORKLOADS["c4"].out_shape == (64, 1024, 3072)


def test_sharding_of_the_workloads(bench):
    c4, c5a, c2 = (bench.WORKLOADS[n] for n in ("c4", "c5a", "c2"))
    assert bench.shard_workload(c4, 3, 8).a_shape == (8, 1024, 768)
    assert bench.shard_workload(c4, 0, 8).b_shape == (768, 3072)          # the weight is replicated
    assert bench.shard_workload(c5a, 7, 8).a_shape == (1024, 8192)
    assert bench.shard_workload(c2, 1, 8).a_shape == c2.a_shape            # weak scaling: a full shard per rank
    assert sum(bench.shard_workload(c4, r, 8).flops for r in range(8)) == c4.flops
    assert bench.scaling_label(c4) == "strong" and bench.scaling_label(c2) == "weak"


def test_both_arms_print_the_same_config(bench):
    for name in ("c1", "c2", "c4", "c5a", "softmax", "adamw"):
        for world in (1, 8):
            a = bench.config_dict(bench.WORKLOADS[name], world, "3xtf32")
            b = bench.config_dict(bench.WORKLOADS[name], world, "3xtf32")
            assert a == b and a["workload"].startswith(name + ":")
    assert "NCCL reduce" in bench.config_dict(bench.WORKLOADS["c4"], 8, "3xtf32")["parallelism"]
    assert bench.config_dict(bench.WORKLOADS["c4"], 1, "3xtf32")["parallelism"] == "single GPU"


def test_pipe_of_a_call_is_asked_of_the_library(bench, monkeypatch):
    """By the results with and without 16-bit planes, however many launches a call makes; the caller's switch is put back."""
    import torch
    out = [torch.zeros(4), torch.zeros(2)]
    def planes():
        out[1].fill_(1.0 if os.environ.get("MNI_B200_HALF") == "0" else 1.0 + 2.0 ** -20)
    for chosen in (None, "1"):
        monkeypatch.setenv("MNI_B200_HALF", chosen) if chosen else monkeypatch.delenv("MNI_B200_HALF", raising=False)
        assert bench.product_pipe(planes, out) == "f16"
        assert bench.product_pipe(lambda: out[0].fill_(3.0), out) == "tf32"
        assert os.environ.get("MNI_B200_HALF") == chosen


def test_cpu_samples_are_bounded_leading_slices(bench):
    c4 = bench.WORKLOADS["c4"]
    small, what = bench.cpu_sample_workload(c4, budget_gflop=150.0)
    assert small.a_shape[1:] == c4.a_shape[1:] and 1 <= small.a_shape[0] < 64 and small.flops <= 150e9
    assert "leading" in what
    whole, what = bench.cpu_sample_workload(bench.WORKLOADS["c1"], budget_gflop=150.0)
    assert whole.a_shape == (512, 512) and what == "whole step"


def test_reference_arm_loads_no_native_code_of_the_package(bench):
    """What the reference arm takes from the package -- shapes and shards of the workloads -- maps none of its libraries."""
    import subprocess
    import sys
    code = """
import importlib.util, sys
spec = importlib.util.spec_from_file_location("bench_module", "bench.py")
bench = importlib.util.module_from_spec(spec)
spec.loader.exec_module(bench)
for wl in bench.WORKLOADS.values():
    bench.config_dict(wl, 8, "f32")
    shard = bench.shard_workload(wl, 1, 8)
    if wl.kind not in ("softmax", "adamw"):
        shard.out_shape, shard.batch, shard.flops, bench.cpu_sample_workload(wl, budget_gflop=150.0)
assert "framework_b200.sharding" in sys.modules
maps = open("/proc/self/maps").read()
assert "framework_b200" not in maps, [line for line in maps.splitlines() if "framework_b200" in line]
"""
    subprocess.run([sys.executable, "-c", code], check=True, cwd=ROOT)
