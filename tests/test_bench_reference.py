"""bench.py's reference arm on a machine without the reference."""
import argparse
import json
import os


def test_reference_arm_says_when_the_reference_is_not_built(monkeypatch, capsys, tmp_path):
    import bench
    from oracle import refbridge
    monkeypatch.setattr(refbridge, "LIB", os.path.join(tmp_path, "libmaosref.so"))
    monkeypatch.delenv("RANK", raising=False)
    args = argparse.Namespace(gpus=1, steps=1, warmup=1, cpu_seconds=1.0)
    assert bench.run_reference(args) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"]
