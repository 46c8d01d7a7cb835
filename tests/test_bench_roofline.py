"""The roof that bench.py divides by is that of the memory the run's kernel reads its
operands from."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


def test_operand_roofline():
    staged = bench.operand_roofline(8, 30_000.0, 37_500.0, None)
    assert staged["bound"] == "smem" and staged["peak"] == 37_500.0
    assert staged["frac"] == 0.8
    tmem = bench.operand_roofline(9, 54_000.0, 37_500.0, {"sm_mhz": 1500.0})
    assert tmem["bound"] == "tmem"
    assert abs(tmem["peak"] - 136 * 4 * 148 * 1.5) < 1e-6  # GB/s at 1.5 GHz
    assert tmem["frac"] == 54_000.0 / tmem["peak"] < 1.0
