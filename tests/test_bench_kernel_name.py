"""The bench line names the kernel that its FP64 figure was measured on."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


def test_fp64_kernel_of_the_bench_line():
    import bench
    assert bench.fp64_kernel(32 ** 4, 152, True, 18) == "or_fx_kernel<4>"
    assert bench.fp64_kernel(2 * 64 * 152, 152, True, 12) == "or_fx_quad_kernel<4>"
    assert bench.fp64_kernel(2 * 64 * 152 + 2, 152, True, 12) == "or_fx_kernel<4>"
    assert bench.fp64_kernel(32 ** 4, 152, False, 18) == "or_halfsweep_kernel<double,18,4>"
