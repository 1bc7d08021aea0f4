"""The roofline that bench.py prints is a fraction of something the kernel uses:
HBM for the kernels that move the state every step, the FP32 rate for the on-chip
kernel (whose algorithmic bytes never leave the SMs and passed the copy rate)."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def test_on_chip_kernel_is_held_against_the_fp32_rate():
    import bench
    pts, seconds = 119.7e9, 1.0                 # 64 RTM shots of 481 x 1281, on chip
    r = bench.kernel_roof("resident", pts, 57.7 * pts, seconds, 6772.9, 80.5)
    assert r["bound"] == "fp32" and r["unit"] == "TFLOP/s" and r["peak"] == 80.5
    assert abs(r["frac"] - 137 * 119.7e9 / 80.5e12) < 1e-3 and r["frac"] < 1


def test_step_kernels_are_held_against_hbm():
    import bench
    for kernel in ("tma", "tma_narrow", "tma2", "direct"):
        r = bench.kernel_roof(kernel, 92.9e9, 57.7 * 92.9e9, 1.0, 6772.9, 80.5)
        assert r["bound"] == "hbm" and r["unit"] == "GB/s" and abs(r["frac"] - 0.791) < 2e-3


def test_fp32_peak_of_the_gpu():
    import bench
    assert 10 < bench.fp32_peak(2070.0) < 200
