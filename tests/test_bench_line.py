"""The default bench line survives a leg that fails: the leg's key holds the
error, its process's messages reach stderr, every other key is there.  Host
only: the timed run is replaced by a record of the same form."""
import json
import sys
from pathlib import Path

import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))
import bench  # noqa: E402


def _record(args, rank, world, local_rank):
    call = {"key": "C2C:4096:256:f", "config": "1", "passes": "", "ms": 0.005, "flop": 6.3e7, "alg_bytes": 1.7e7,
            "launches": 1, "ms_hot": 0.005, "copies": 1, "copy_ms": 0.004}
    return {"total_ms": 0.1, "calls": [call], "clocks": {}, "check": None, "cufft": {},
            "e2e": {"ms_per_step": 1.0, "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 1}}


def _run(monkeypatch, capfd, **legs):
    monkeypatch.setattr(bench, "run_ours", _record)
    monkeypatch.setattr(bench, "run_batched", lambda *a: {"metric": "batched", "value": 1.0, "n_gpus": 1})
    monkeypatch.setattr(bench, "run_precision", lambda *a: {"metric": "precision"})
    for name, leg in legs.items():
        monkeypatch.setattr(bench, name, leg)
    monkeypatch.setattr(bench, "cpu_baseline", lambda *a: {})
    monkeypatch.setattr(bench, "cpu_baseline_fp64", lambda *a: {})
    monkeypatch.setattr(sys, "argv", ["bench.py", "--steps", "1", "--warmup", "3"])
    for v in ("RANK", "LOCAL_RANK", "WORLD_SIZE"):
        monkeypatch.delenv(v, raising=False)
    assert bench.main() == 0
    out, err = capfd.readouterr()
    return json.loads(out.strip().splitlines()[-1]), err


def test_child_that_exits_non_zero(monkeypatch, capfd, tmp_path):
    child = tmp_path / "python"
    child.write_text("#!/bin/sh\necho why it failed >&2\nexit 1\n")
    child.chmod(0o755)
    monkeypatch.setattr(bench.sys, "executable", str(child))
    line, err = _run(monkeypatch, capfd)
    assert "status 1" in line["serving"]["error"] and "why it failed" in err
    assert line["value"] > 0 and line["batched_uneven"]["value"] == 1.0 and line["precision_mode"]
    assert line["e2e"]["value"] > 0


@pytest.mark.parametrize("name", ["run_batched", "run_precision"])
def test_leg_that_raises(monkeypatch, capfd, name):
    def fail(*a):
        raise RuntimeError("no leg")

    monkeypatch.setattr(bench, "serving_in_child", lambda args: {"metric": "serving", "value": 2.0})
    line, err = _run(monkeypatch, capfd, **{name: fail})
    key = {"run_batched": "batched_uneven", "run_precision": "precision_mode"}[name]
    assert line[key]["error"] == "RuntimeError: no leg" and "no leg" in err
    assert line["serving"]["value"] == 2.0
