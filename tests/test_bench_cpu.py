"""The benchmark's reference arm, without a GPU."""
import json


def test_reference_arm_without_the_original_solver(monkeypatch, capsys):
    """Without the original solver's binary the arm says so: no other code's speed
    goes under its name."""
    import argparse

    import bench
    monkeypatch.setattr(bench, "run_reference_cpu", lambda steps: None)
    monkeypatch.setattr(bench, "run_oracle_cpu", lambda steps: (1.0, 1))
    bench.reference_arm(argparse.Namespace(steps=2, warmup=3, gpus=1), 0, 1)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
