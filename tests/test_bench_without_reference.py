"""bench.py where the reference's own CPU code has not been built (oracle/_ref):
the GPU line keeps its rows, and the reference arm says why it has none."""
import json
import os
import sys

import pytest

import common as C

sys.path.insert(0, C.ROOT)
sys.path.insert(0, os.path.join(C.ROOT, "oracle"))
import bench  # noqa: E402
import ref_cpu as R  # noqa: E402


class NoContext:
    def close(self):
        pass


@pytest.fixture
def run(monkeypatch, tmp_path, capsys):
    monkeypatch.setattr(R, "REF_DIR", str(tmp_path))

    def main(*argv):
        monkeypatch.setattr(sys, "argv", ["bench.py", *argv])
        bench.main()
        return json.loads(capsys.readouterr().out.strip().splitlines()[-1])

    return main


def test_the_gpu_line_is_printed(run, monkeypatch):
    measured = {"metric": bench.METRIC, "value": 2.0, "unit": bench.UNIT, "e2e": {"value": 1.0}}
    monkeypatch.setattr(bench, "run_ours", lambda args, dist: (dict(measured), NoContext()))
    line = run("--steps", "1", "--warmup", "1")
    assert {k: line[k] for k in measured} == measured
    assert "oracle/_ref" in line["cpu_baseline"]["unavailable"]
    assert "summary" in line and "gpu_over_cpu" not in line


def test_the_reference_arm_says_why(run):
    line = run("--impl", "reference", "--steps", "1", "--warmup", "1")
    assert line["impl"] == "reference" and "oracle/_ref" in line["unavailable"] and "value" not in line


def test_a_failure_of_the_gpu_run_is_not_hidden(run, monkeypatch):
    def broken(args, dist):
        raise RuntimeError("no GPU")

    monkeypatch.setattr(bench, "run_ours", broken)
    with pytest.raises(RuntimeError, match="no GPU"):
        run("--steps", "1", "--warmup", "1")
