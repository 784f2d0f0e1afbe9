"""Host-side pieces of bench.py that need no GPU: the clock sampler's windowing and the byte counts of the sumcheck's launches."""
import importlib.util
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
spec = importlib.util.spec_from_file_location("bench_under_test", os.path.join(ROOT, "bench.py"))
bench = importlib.util.module_from_spec(spec)
spec.loader.exec_module(bench)


class _FakeProc:
    def terminate(self):
        pass

    def wait(self, timeout=None):
        return 0


def _row(sm, power_cap="Not Active"):
    return ["0", str(sm), "1965", "500.0", "0x0", "Not Active", "Not Active", "Not Active", power_cap]


def _sampler(rows):
    s = bench.ClockSampler(0)
    s.proc = _FakeProc()
    s.rows = list(rows)
    return s


def test_clock_sampler_uses_the_timed_window():
    s = _sampler([_row(1000), _row(1000), _row(1965), _row(1950), _row(1965), _row(1200)])
    out = s.stop(2, 5)
    assert out["samples"] == 3 and out["sm_mhz"] == 1965.0 and out["sm_max_mhz"] == 1965.0
    assert out["window"] == "timed region" and out["reasons"] == []


def test_clock_sampler_falls_back_to_all_samples_and_reports_reasons():
    s = _sampler([_row(1900), _row(1800, "Active")])
    out = s.stop(2, 2)                      # nothing arrived inside the window
    assert out["samples"] == 2 and out["window"] == "warm-up and timed region"
    assert out["reasons"] == ["sw_power_cap"]


def test_clock_sampler_without_nvidia_smi():
    s = bench.ClockSampler(0)
    assert s.stop()["reasons"] == ["nvidia-smi unavailable"]


def test_launch_bytes_add_up_to_the_schedule_of_each_form():
    for n, split, words in ((28, False, 48), (28, True, 56), (15, False, 48), (14, False, 80)):
        per = bench.schedule_bytes(n, n + 2, split)
        assert bench.schedule_total(n, split) == words
        assert words - 1 < sum(per) / (1 << n) <= words           # the last rounds are what is left of the geometric sum
        named = bench.schedule_kernels(n, split)
        prof = [1.0] * 5
        for i in range(4):
            prof[i] = 9.0
            r = bench.sumcheck_roofline(n, prof, 6434.8, "t", 2 if split else 1)
            prof[i] = 1.0
            assert r["kernel"].startswith(named[i][0] if i < len(named) else "sc_round_kernel") and f": {per[i]} bytes" in r["kernel"]
