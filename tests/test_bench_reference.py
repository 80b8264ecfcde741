"""The build and bench.py's reference arm on a machine without the reference."""
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


def test_build_without_the_reference_sources(monkeypatch, tmp_path):
    """An empty directory in the place of the reference's sources is no reason to fail."""
    import __graft_entry__ as entry
    from maos_b200 import build, native
    built = []
    monkeypatch.setenv("MAOS_REF", str(tmp_path))
    monkeypatch.setattr(build, "build", lambda **kw: built.append(kw))
    monkeypatch.setattr(native, "load", lambda: None)
    entry.build()
    assert built == [{"force": True, "verbose": True}]
