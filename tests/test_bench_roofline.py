"""The benchmark's roofline figures from profiles of each layout (no GPU)."""
import importlib.util
import os

import pytest

spec = importlib.util.spec_from_file_location("bench", os.path.join(os.path.dirname(__file__), os.pardir, "bench.py"))
bench = importlib.util.module_from_spec(spec)
spec.loader.exec_module(bench)


def test_kernel_bound_is_the_longer_floor():
    # one multiply-add per double read: FP64 at 1.25 TFLOP/s takes longer than 6.8 TB/s
    assert bench.kernel_bound("k_border_cg", 2e9, 8e9, 1.25, 6800) == "fp64"
    assert bench.kernel_bound("k_spmv_jcp", 2e9, 16e9, 1.25, 6800) == "hbm"
    assert bench.kernel_bound("k_prepare", 0.0, 16e9, 1.25, 6800) == "hbm"
    assert bench.kernel_bound("k_border_update<4>", 64e9, 16e9, 1.25, 6800) == "hbm"


def test_solve_work_of_each_layout():
    # {kernel: (launches, ms, flops, bytes)}
    queues = {"k_front_small": (3, 1.0, 5e9, 0.0), "k_trsv_fwd": (10, 1.0, 2e9, 8e9), "k_trsv_bwd": (10, 1.0, 2e9, 8e9)}
    w = bench.solve_work(queues, 100.0, 2.0, 50)
    assert w["pairs"] == 108 and w["factor"] == 5e9
    assert w["fp64"] == pytest.approx(5e9 + 108 * 0.4e9) and w["solve_bytes"] == pytest.approx(108 * 1.6e9)
    blocks = {"k_border_update<4>": (3, 1.0, 7e9, 1e9), "k_border_update<1>": (2, 1.0, 1e9, 1e9),
              "k_border_once": (8, 1.0, 8e8, 3.2e9), "k_border_cg": (2, 1.0, 1e10, 4e10)}
    w = bench.solve_work(blocks, 100.0, 2.0, 50)
    assert w["pairs"] == 108 and w["factor"] == 8e9
    assert w["fp64"] == pytest.approx(108 * 1e8) and w["solve_bytes"] == pytest.approx(108 * 4e8)
    del blocks["k_border_cg"]
    blocks["k_schur_cg<4>"] = (2, 1.0, 1e9, 4e9)
    w = bench.solve_work(blocks, 100.0, 2.0, 50)
    assert w["pairs"] == 4 and w["fp64"] == pytest.approx(4 * 1e8 + 104 * 2 * 2500)
    assert bench.solve_work({"k_prepare": (1, 1.0, 0.0, 0.0)}, 1.0, 1.0, 5) is None
