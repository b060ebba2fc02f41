"""CPU test of bench.py's reference arm where the reference is not built: one line that
says so and no number (the repository's own C restatement is not the reference)."""
import argparse
import json


def test_reference_arm_without_the_reference(monkeypatch, capsys):
    import bench
    import oracle
    monkeypatch.setattr(oracle, "reference_available", lambda: False)
    args = argparse.Namespace(gpus=1, steps=1, warmup=3, n=10**5)
    assert bench.run_reference(args, 0, 1) == 0
    lines = capsys.readouterr().out.splitlines()
    assert len(lines) == 1
    d = json.loads(lines[0])
    assert set(d) == {"impl", "unavailable"} and d["impl"] == "reference" and "\n" not in d["unavailable"]
