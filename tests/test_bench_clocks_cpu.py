"""The benchmark's clock sampler against a stand-in for NVML: its line carries clocks however slow the queries are."""
import importlib
import os
import sys
import time
import types

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


def _nvml(init_s, query_s, mhz, reasons):
    m = types.ModuleType("pynvml")
    m.NVML_CLOCK_SM = 1
    m.nvmlInit = lambda: time.sleep(init_s)
    m.nvmlDeviceGetHandleByIndex = lambda i: i
    m.nvmlDeviceGetMaxClockInfo = lambda h, c: 1965

    def clock(h, c):
        time.sleep(query_s)
        return mhz
    m.nvmlDeviceGetClockInfo = clock
    m.nvmlDeviceGetCurrentClocksEventReasons = lambda h: reasons
    return m


@pytest.mark.parametrize("init_s,query_s", [(0.0, 0.0), (0.4, 0.0), (0.2, 0.1)])
def test_a_timed_region_of_milliseconds_has_clock_samples(monkeypatch, init_s, query_s):
    """NVML that takes longer to come up than warm-up and timed region together, and queries longer than the region."""
    monkeypatch.setitem(sys.modules, "pynvml", _nvml(init_s, query_s, 1500, 0x4))
    bench = importlib.import_module("bench")
    sampler = bench.ClockSampler(0)
    sampler.start()
    time.sleep(0.05)
    lo = sampler.mark()
    time.sleep(0.016)
    got = sampler.stop(lo, sampler.mark())
    assert got["samples"] >= 1 and got["sm_mhz"] == 1500.0 and got["sm_max_mhz"] == 1965.0 and got["reasons"] == ["sw_power_cap"]


def test_samples_from_outside_the_timed_region_do_not_count(monkeypatch):
    nvml = _nvml(0.0, 0.001, 1500, 0)
    monkeypatch.setitem(sys.modules, "pynvml", nvml)
    bench = importlib.import_module("bench")
    sampler = bench.ClockSampler(0)
    sampler.start()
    time.sleep(0.05)
    nvml.nvmlDeviceGetClockInfo = lambda h, c: 1965
    time.sleep(0.05)
    lo = sampler.mark()
    time.sleep(0.05)
    hi = sampler.mark()
    nvml.nvmlDeviceGetClockInfo = lambda h, c: 300
    time.sleep(0.05)
    got = sampler.stop(lo, hi)
    assert got["sm_mhz"] == 1965.0 and got["samples"] >= 5
