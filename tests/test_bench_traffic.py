"""The DRAM traffic that bench.py prints beside its FP32 and FP64 workloads is
that of the kernel it names, from a committed capture of that kernel (no GPU)."""
import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402


@pytest.mark.parametrize("real_bytes", [4, 8])
@pytest.mark.parametrize("ms", [[3.0, 1.0, 1.0, 0.0], [1.0, 3.0, 1.0, 0.0], [1.0, 1.0, 3.0, 0.0]])
def test_traffic_is_of_the_kernel_named(real_bytes, ms):
    n = 4096
    r = bench.roofline_of(ms, [4, 4, 4, 0], n, real_bytes, bench.pass_tag(n, real_bytes), 6793.4, "measured")
    kernel = r["kernel"].split()[0]
    path, _, of = r["traffic_source"].partition(" (ncu, ")
    assert of.rstrip(")") == kernel
    with open(os.path.join(ROOT, path)) as f:
        entry = json.load(f)[kernel[:7]]
    assert entry["kernel"] == kernel and r["traffic"] == entry["dram_read"] + entry["dram_write"]


def test_which_passes_run():
    assert [bench.pass_tag(n, 4) for n in (1024, 2048, 8192)] == ["fp32", "fp32_lean", "fp32_lean"]
    assert bench.pass_tag(4096, 8) == "fp64"
