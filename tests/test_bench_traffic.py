"""The DRAM traffic that bench.py prints beside the tv row is the traffic of the kernel that runs."""
import os
import re

import bench

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_the_profiled_kernel_is_the_one_that_runs(monkeypatch):
    monkeypatch.delenv("NESSI_TV_KERNEL", raising=False)
    name = bench.TV_PROFILE["fp64"]
    kernel = open(os.path.join(ROOT, "profiles", name)).readline().split()[1]
    source = open(os.path.join(ROOT, "nessi_b200", "csrc", "nessi_gpu.cu")).read()
    assert re.search(r"\b%s<S, VIE><<<" % kernel, source)  # launched for FP64 steps
    assert 0.9 < bench.tv_traffic_ratio("fp64") < 1.5


def test_no_ratio_where_another_kernel_runs(monkeypatch):
    monkeypatch.delenv("NESSI_TV_KERNEL", raising=False)
    assert bench.tv_traffic_ratio("mixed") is None
    monkeypatch.setenv("NESSI_TV_KERNEL", "stream")
    assert bench.tv_traffic_ratio("fp64") is None
