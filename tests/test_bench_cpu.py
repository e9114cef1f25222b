"""The benchmark's clock samples, on a stand-in for NVML."""
import sys
import time
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))

import bench  # noqa: E402


class FakeNvml:
    """Answers a query in 2 ms, as a loaded driver does."""

    def __init__(self, reasons=0):
        self.reasons = reasons

    def nvmlInit_v2(self):
        return 0

    def nvmlDeviceGetHandleByUUID(self, uuid, handle):
        return 1

    def nvmlDeviceGetHandleByIndex_v2(self, index, handle):
        return 0

    def nvmlDeviceGetMaxClockInfo(self, handle, kind, out):
        out._obj.value = 1965
        return 0

    def nvmlDeviceGetClockInfo(self, handle, kind, out):
        time.sleep(0.002)
        out._obj.value = 1900
        return 0

    def nvmlDeviceGetCurrentClocksThrottleReasons(self, handle, out):
        out._obj.value = self.reasons
        return 0


def test_a_region_of_twenty_steps_is_sampled():
    with bench.ClockSampler(0, FakeNvml(0x4 | 0x20)) as clk:
        clk.wait_first(lambda: time.sleep(0.001))
        time.sleep(0.013)
    got = clk.summary()
    assert got["samples"] >= 2 and got["sm_mhz"] == 1900 and got["sm_max_mhz"] == 1965
    assert got["reasons"] == ["sw_power_cap", "sw_thermal_slowdown"]


def test_no_reason_and_no_nvml():
    with bench.ClockSampler(0, FakeNvml()) as clk:
        time.sleep(0.01)
    assert clk.summary()["reasons"] == []

    class Broken(FakeNvml):
        def nvmlInit_v2(self):
            return 9

    with bench.ClockSampler(0, Broken()) as clk:
        clk.wait_first(lambda: time.sleep(0.001))
    assert clk.summary() == {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
