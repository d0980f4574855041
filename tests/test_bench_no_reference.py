"""bench.py where the reference library is not built (its sources are not on the
host): the CPU baseline says why it is missing, the measurement stands."""
import json
import sys

import pytest

import bench
import oracle


@pytest.fixture
def no_reference(monkeypatch):
    monkeypatch.setattr(oracle, "ref_available", lambda: False)


def test_reference_arm_prints_why(no_reference, monkeypatch, capsys):
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--gpus", "1"])
    bench.main()
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "not built" in line["unavailable"]


def test_sections_keep_their_result(no_reference):
    def tasks(size):
        raise AssertionError("no sample is made for a path that cannot run")
    r = bench.cpu_sampled_baseline(tasks, (20, 100))
    assert set(r) == {"unavailable"} and "not built" in r["unavailable"]


def test_available_is_what_the_baseline_loads(monkeypatch):
    for built, want in ((set(), False), ({"libqldref.so"}, True), ({"libqldref_blis.so"}, True)):
        monkeypatch.setattr(oracle.os.path, "exists",
                            lambda p, built=built: p.rsplit("/", 1)[-1] in built)
        assert oracle.ref_available() is want
