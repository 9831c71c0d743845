"""The counters file behind the bench's roofline holds figures of the logs it was made from and of nothing else."""
import importlib.util
import json
import os

import pytest

from conftest import ROOT


@pytest.fixture()
def bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def log(path, rows):
    with open(path, "w") as f:
        f.write("==PROF== not a row\n")
        f.write('"ID","Kernel Name","Metric Name","Metric Unit","Metric Value"\n')
        for name, unit, value in rows:
            f.write('"0","void mm16_kernel<1>(MmParams)","%s","%s","%s"\n' % (name, unit, value))
    return str(path)


def test_traffic_of_another_capture_is_dropped(bench, tmp_path, monkeypatch):
    path = tmp_path / "counters.json"
    path.write_text(json.dumps({"kernel": "old", "command": "c", "command_traffic": "t", "dram_bytes_per_launch_8192cubed": 1,
                                "metrics": {"dram__bytes_read.sum_8192cubed": 1.0}, "captured_at": "8192^3 (DRAM traffic)"}))
    monkeypatch.setattr(bench, "COUNTERS_PATH", str(path))
    per_mac = log(tmp_path / "a.csv", [("smsp__inst_executed.sum", "inst", "4,000"), ("sm__inst_executed_pipe_alu.sum", "inst", "2000")])
    c = bench.record_counters(per_mac, 32, None, "note")
    assert c["inst_per_mac"] == pytest.approx(4000 * 32 / 32 ** 3, abs=1e-3) and c["command"] == "c" and "mm16_kernel" in c["kernel"]
    assert "dram_bytes_per_launch_8192cubed" not in c and "command_traffic" not in c
    assert not any("8192" in k for k in c["metrics"])
    assert json.loads(path.read_text()) == c and bench.load_counters()["constants_stale"] is False
    path.write_text(json.dumps(dict(c, command_traffic="t")))
    traffic = log(tmp_path / "b.csv", [("dram__bytes_read.sum", "Gbyte", "1.5"), ("dram__bytes_write.sum", "Mbyte", "500")])
    c = bench.record_counters(per_mac, 32, traffic, "note")
    assert c["dram_bytes_per_launch_8192cubed"] == 2_000_000_000 and c["command_traffic"] == "t"


def test_reference_arm_never_times_the_oracle(bench, monkeypatch, capsys):
    import argparse

    import oracle.build_ref

    monkeypatch.setattr(oracle.build_ref, "load_ref", lambda name: None)
    monkeypatch.setattr(bench, "cpu_baseline", lambda *a: pytest.fail("the oracle was timed as the reference"))
    assert bench.run_reference(argparse.Namespace(gpus=1, steps=1, warmup=0)) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
