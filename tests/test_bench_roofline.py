"""bench.py's HBM fractions: of the bytes a launch moves, never above the peak
for what one round over HBM a step would have moved."""
import os
import sys
from types import SimpleNamespace

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402

PEAK = 6784.2


def test_many_steps_a_launch_take_the_profiled_bytes():
    """25 points 1024^3 at 469 Gpts/s: 16 bytes a step would be 1.1 of the peak."""
    info = SimpleNamespace(bytes_per_point=16.0, temporal_block=1)
    pts, steps = 1024 ** 3, 50
    ms = pts * steps / 469e9 * 1e3
    r = bench.wave_roofline(info, "wave25_1024", pts, steps, ms, 1, PEAK)
    assert 8.0 < r["bytes_per_point"] < 16.0
    assert abs(r["frac"] - r["bytes_per_point"] * 469 / PEAK) < 1e-9 and r["frac"] < 1.0
    assert abs(r["one_round"]["frac"] - 16 * 469 / PEAK) < 1e-9
    # orders and plane sizes without a committed profile have no fraction rather than a wrong one
    for workload in ("wave7_1024", "wave25_528"):
        assert bench.wave_roofline(info, workload, pts, steps, ms, 1, PEAK)["frac"] is None


def test_single_steps_and_fused_passes_take_the_algorithmic_bytes():
    pts, steps, ms = 1024 ** 3, 40, 100.0
    one = bench.wave_roofline(SimpleNamespace(bytes_per_point=16.0, temporal_block=1), "wave25_1024", pts, steps, ms,
                              steps, PEAK)
    two = bench.wave_roofline(SimpleNamespace(bytes_per_point=10.0, temporal_block=2), "wave25_1024", pts, steps, ms,
                              20, PEAK)
    rate = pts * steps / 0.1 / 1e9
    assert abs(one["frac"] - 16 * rate / PEAK) < 1e-9 and "one_round" not in one
    assert abs(two["frac"] - 10 * rate / PEAK) < 1e-9 and "one_round" not in two
