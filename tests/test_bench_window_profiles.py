"""The windowed descent's figures that bench.py reads from the committed ncu summaries, and that each summary of a descent names
a command that still reaches its kernel (CPU only)."""
import math
import os
import re
import sys

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, REPO)

import bench  # noqa: E402


@pytest.mark.parametrize("name,key,low,high", [
    ("k_descent_window_large", "warp_inst_per_move_per_block", 1000, 100000),
    ("k_descent_window_large", "dram_bytes_per_launch", 1e8, 1e12),
    ("k_descent_window_wide3", "warp_inst_per_move_per_block", 1000, 100000),
    ("k_descent_window_wide3", "dram_bytes_per_launch", 1e8, 1e12)])
def test_profile_figure_present(name, key, low, high):
    value = bench.profiled_value(name, key)
    assert value is not None and low <= value <= high, (name, key, value)


# vertices a unit of gain width above which each kernel's graphs keep it
@pytest.mark.parametrize("name,units", [
    ("k_descent_large", 1150), ("k_descent_cluster_large", 1150), ("k_descent_wide3_sparse_n65536", 1500),
    ("k_descent_incremental_regs_n14486_k53", None)])
def test_recipe_of_a_replaced_kernel_uses_a_sparse_graph(name, units):
    with open(os.path.join(REPO, "profiles", name + ".txt")) as fh:
        runs = re.findall(r"cli --n (\d+) --density ([0-9.]+) --k (\d+)", fh.read())
    assert len(runs) == 2 and runs[0] == runs[1]
    n, p, k = int(runs[0][0]), float(runs[0][1]), int(runs[0][2])
    width = 2.8 * math.sqrt(n * p * (1 - p) / k)
    assert n > units * width if units else (k > 32 and width < 4)
