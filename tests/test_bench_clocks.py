"""Clock samples of bench.py's timed region: a region of a few milliseconds has some."""
import time

import bench


def test_short_regions_are_sampled():
    calls = []

    def read():
        calls.append(time.perf_counter())
        if len(calls) == 2:
            raise OSError("a failed read")
        return 1900.0 + len(calls) % 2, 1965.0, ["sw_power_cap"] if len(calls) == 3 else []

    with bench.ClockSampler(read) as clocks:
        t0 = time.perf_counter()
        time.sleep(0.015)
        t1 = time.perf_counter()
    s = clocks.summary(None)
    inside = sum(t0 <= c <= t1 for c in calls)
    assert inside >= 3
    assert s["samples"] == len(calls) - 1 and 1900.0 <= s["sm_mhz"] <= 1901.0
    assert s["sm_max_mhz"] == 1965.0 and s["reasons"] == ["sw_power_cap"]


def test_without_a_reader_the_summary_has_its_keys():
    with bench.ClockSampler() as clocks:
        pass
    s = clocks.summary(None)
    assert set(s) == {"sm_mhz", "sm_max_mhz", "reasons", "samples"}
