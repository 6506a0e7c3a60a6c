"""bench.py's reference arm without the reference."""
import argparse
import json
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_is_unavailable_without_the_reference(monkeypatch, capsys):
    """Where the reference's own library is not built, the arm says so; it never times this repository's C restatement
    under the name of the reference."""
    monkeypatch.syspath_prepend(ROOT)
    import bench
    import oracle
    monkeypatch.setattr(oracle, "ref", lambda: None)
    monkeypatch.setattr(oracle, "port", lambda: (_ for _ in ()).throw(AssertionError("the restatement was asked for")))
    bench.run_reference(argparse.Namespace(workload="c1", size=None, steps=1, warmup=0, gpus=1))
    line = json.loads(capsys.readouterr().out.strip())
    assert line.keys() == {"impl", "unavailable"} and line["impl"] == "reference" and line["unavailable"]
