"""Without the reference's sources the bench's reference arm says so in its one line and ends well."""
import json
import os
import sys
import types

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_without_the_reference(monkeypatch, capsys, tmp_path):
    monkeypatch.syspath_prepend(ROOT)
    import bench
    import oracle as orc
    monkeypatch.setattr(orc, "REF_LIB", str(tmp_path / "absent.so"))
    monkeypatch.delenv("RANK", raising=False)
    bench.run_reference_arm(types.SimpleNamespace(workload="glycine128", gpus=1, steps=3, warmup=3))
    line = json.loads(capsys.readouterr().out.strip())
    assert line["impl"] == "reference" and line["unavailable"]
