"""The clock record of a benchmark line holds samples of the timed region on, not of the settling before it."""
import datetime
import os
import sys

import pytest

from conftest import ROOT

sys.path.insert(0, ROOT)
import bench  # noqa: E402

ROW = "%s, %d, 2070, %.1f, 0x0, %s, Not Active, Not Active, Not Active\n"


@pytest.fixture
def sampler(tmp_path):
    s = bench.ClockSampler(0)
    s.path = str(tmp_path / "clocks.csv")
    return s


def _write(s, since):
    at = lambda ms: (since + datetime.timedelta(milliseconds=ms)).strftime("%Y/%m/%d %H:%M:%S.%f")[:-3]
    with open(s.path, "w") as f:
        f.write("timestamp, clocks.sm [MHz], ...\n")
        f.write(ROW % (at(-5000), 900, 300.0, "Active"))     # while the scene settled
        f.write(ROW % (at(-1), 1000, 900.0, "Active"))
        f.write(ROW % (at(1), 1990, 500.0, "Not Active"))
        f.write(ROW % (at(201), 2010, 510.0, "Not Active"))
        f.write("2026/")                                     # cut off


def test_rows_from_the_mark_on(sampler):
    sampler.mark()
    _write(sampler, sampler.since)
    rows = sampler.rows(open(sampler.path))
    assert [r[0] for r in rows] == [1990.0, 2010.0]
    assert not any(v.lower() == "active" for r in rows for v in r[3])


def test_record_of_a_run(sampler, monkeypatch):
    """start, mark and stop with a stand-in for nvidia-smi."""
    class Proc:
        def __init__(self, cmd, stdout=None, **kw):
            assert cmd[0] == "nvidia-smi" and any(c.startswith("--query-gpu=timestamp,") for c in cmd)
        terminate = wait = kill = lambda self, **kw: None

    monkeypatch.setattr(bench.subprocess, "Popen", Proc)
    monkeypatch.setattr(bench.time, "sleep", lambda s: _write(sampler, sampler.since))
    sampler.start()
    sampler.mark()
    got = sampler.stop()
    assert got["samples"] == 2 and got["reasons"] == [] and got["sm_mhz"] == 2000.0 and got["power_w_max"] == 510.0
    os.remove(sampler.path)
