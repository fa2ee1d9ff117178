"""The bench's roofline reads the DRAM traffic of each step kernel it names from
the profile summary of that kernel."""

import importlib.util
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("kernel,key", [
    ("fwdv_kernel", "small_case_dram_bytes_per_cell_per_step"),
    ("adjv_kernel", "small_case_dram_bytes_per_cell_per_step"),
    ("fwd2_step_kernel", "pec_257_dram_bytes_per_cell_per_step_one_step"),
    ("fwd2_step_kernel", "pec_257_dram_bytes_per_cell_per_step_two_step"),
])
def test_named_kernels_have_a_traffic_figure(kernel, key):
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    assert 30.0 < bench._traffic_per_cell(kernel, key) < 200.0
