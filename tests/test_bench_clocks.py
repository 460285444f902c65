"""bench.py's clock sampler against a stand-in for nvidia-smi: a sample counts
for a timed region only if its query began before the region's end."""
import os
import stat
import sys
import time

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
QUERY = 0.08  # seconds that the stand-in's query takes, and its interval between queries

FAKE = f"""#!{sys.executable}
import os, time
while True:
    busy = os.path.exists({{flag!r}})  # read when the query begins
    time.sleep({QUERY})
    print("0, %d, 1965, 500, 0x0, Not Active, Not Active, Not Active, Not Active" % (1900 if busy else 300), flush=True)
    time.sleep({QUERY})
"""


@pytest.fixture
def sampler(tmp_path, monkeypatch):
    sys.path.insert(0, REPO)
    import bench
    flag, smi = tmp_path / "busy", tmp_path / "nvidia-smi"
    smi.write_text(FAKE.format(flag=str(flag)))
    smi.chmod(smi.stat().st_mode | stat.S_IXUSR)
    monkeypatch.setenv("PATH", f"{tmp_path}:{os.environ['PATH']}")
    monkeypatch.setattr(bench.ClockSampler, "EVERY_MS", int(QUERY * 1000), raising=False)

    def region(seconds):
        with bench.ClockSampler(0) as clk:
            flag.touch()
            time.sleep(seconds)
            flag.unlink()
        return clk.summary()

    return region


def test_a_region_shorter_than_the_interval_takes_no_idle_sample(sampler):
    assert sampler(0.01)["sm_mhz"] in (None, 1900.0)


def test_a_query_in_flight_at_the_region_s_end_counts(sampler):
    s = sampler(0.12)  # the query of 80 to 160 ms
    assert s["sm_mhz"] == 1900.0 and s["sm_max_mhz"] == 1965.0


def test_long_regions_are_sampled_throughout(sampler):
    s = sampler(0.6)
    assert s["sm_mhz"] == 1900.0 and 2 <= s["samples"] <= 5
