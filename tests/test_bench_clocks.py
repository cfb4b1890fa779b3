"""bench.py's clock sampler around timed regions shorter than nvidia-smi's start,
with a stand-in for nvidia-smi."""
import os
import stat
import time

import pytest

import bench

ROW = "0, {mhz}, 1965, 200.0, 0x0, Not Active, Not Active, Not Active, {cap}"


def _fake(tmp_path, monkeypatch, body):
    exe = tmp_path / "nvidia-smi"
    exe.write_text("#!/bin/sh\n" + body)
    exe.chmod(exe.stat().st_mode | stat.S_IXUSR)
    monkeypatch.setenv("PATH", f"{tmp_path}{os.pathsep}{os.environ['PATH']}")


@pytest.mark.parametrize("start", [0.0, 0.5])
def test_short_region_has_a_sample(tmp_path, monkeypatch, start):
    """The row from before the region is left out, one from its end is there."""
    _fake(tmp_path, monkeypatch, f"sleep {start}\necho '{ROW.format(mhz=120, cap='Active')}'\n"
          f"while true; do sleep 0.1; echo '{ROW.format(mhz=1900, cap='Not Active')}'; done\n")
    with bench.ClockSampler(0) as clk:
        pass
    s = clk.summary()
    assert s["sm_mhz"] == 1900.0 and s["sm_max_mhz"] == 1965.0 and s["reasons"] == []
    assert s["samples"] >= 1 and clk.proc.poll() is not None
    assert not os.path.exists(clk.path)


@pytest.mark.parametrize("body", ["exit 1\n", "echo 'No devices were found'\n"])
def test_no_rows_do_not_hold_the_bench_up(tmp_path, monkeypatch, body):
    _fake(tmp_path, monkeypatch, body)
    t0 = time.monotonic()
    with bench.ClockSampler(0) as clk:
        pass
    assert time.monotonic() - t0 < bench.ClockSampler.WAIT_S
    assert clk.summary() == {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
