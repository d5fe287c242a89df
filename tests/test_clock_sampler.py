"""bench.py's clock record covers a timed region of a tenth of a second: sampled
from a stand-in for NVML, with the reasons that were active at any sample."""
import sys
import time
import types


def test_short_region_is_sampled(monkeypatch):
    import bench

    clocks = iter([1000] + [1965] * 1000)
    reasons = iter([0, 0x4] + [0x1] * 1000)
    nv = types.SimpleNamespace(
        NVML_CLOCK_SM=1, nvmlInit=lambda: None, nvmlDeviceGetHandleByIndex=lambda i: i,
        nvmlDeviceGetMaxClockInfo=lambda d, k: 1965, nvmlDeviceGetClockInfo=lambda d, k: next(clocks),
        nvmlDeviceGetCurrentClocksEventReasons=lambda d: next(reasons))
    monkeypatch.setitem(sys.modules, "pynvml", nv)
    with bench.ClockSampler(0) as clk:
        time.sleep(0.1)
    s = clk.summary()
    assert s["samples"] >= 2 and s["sm_mhz"] == 1965.0 and s["sm_max_mhz"] == 1965.0
    assert s["reasons"] == ["sw_power_cap"]


def test_without_nvml_the_record_says_so(monkeypatch):
    import bench

    monkeypatch.setitem(sys.modules, "pynvml", None)
    with bench.ClockSampler(0) as clk:
        pass
    assert clk.summary() == {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
