"""The reference arm of the benchmark times the reference's own program or says
why it cannot: the oracle's restatement never stands in for it."""
import argparse
import json


def test_unavailable_without_the_reference_binary(monkeypatch, capsys):
    import bench
    from oracle import cpu_baseline as B
    from oracle import oracle as O
    monkeypatch.setattr(O, "harness_available", lambda: False)
    monkeypatch.setattr(B, "port_rate", lambda *a, **k: {"value": 1.0, "cores": 1, "kind": "port", "sample": ""})
    bench.reference_arm(argparse.Namespace(steps=4, warmup=1), 0, 1)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "value" not in line
    assert "not built" in line["unavailable"]
