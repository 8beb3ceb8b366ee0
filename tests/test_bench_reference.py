"""bench.py where the reference's own library is not built: its arm and the entries that run it
say so, and the rest of the line does not depend on them."""
import json
import os
import sys

import pytest

import bench
import oracle.pyoracle as pyoracle


@pytest.fixture(autouse=True)
def no_reference(monkeypatch):
    monkeypatch.setattr(pyoracle, "REF_LIB", os.path.join(os.path.dirname(__file__), "absent.so"))


def test_entries_say_unavailable():
    for entry in (bench.reference_gpu_baseline(64, 1, 2), bench.accuracy_full_run(64, 1, 0, 1)):
        assert list(entry) == ["unavailable"] and "not built" in entry["unavailable"]


def test_reference_arm_says_unavailable(monkeypatch, capsys):
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--gpus", "1", "--steps", "2", "--warmup", "3"])
    bench.main()
    line = json.loads(capsys.readouterr().out.strip().splitlines()[-1])
    assert line["impl"] == "reference" and "not built" in line["unavailable"] and "value" not in line
