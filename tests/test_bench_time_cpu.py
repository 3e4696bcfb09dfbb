"""The benchmark's longest side leg must not cost the run its line (no GPU)."""
import bench


def test_the_tight_leg_gives_way_to_the_line():
    ran = []
    assert bench.tight_in_time(bench.TIGHT_LATEST_S - 1.0, lambda: ran.append(1) or {"batched_value": 1.0}) == {"batched_value": 1.0}
    out = bench.tight_in_time(bench.TIGHT_LATEST_S + 1.0, lambda: ran.append(2))
    assert set(out) == {"skipped"} and ran == [1]
