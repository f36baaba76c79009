"""
The reference arm of bench.py on the CPU: where the reference is not installed it says so, and nothing of this
repository is timed in its place.
"""

import json
import types


def test_reference_arm_without_the_reference(monkeypatch, capsys):
    import bench
    monkeypatch.setattr(bench, "reference_diffraction", lambda: None)
    bench.run_reference(types.SimpleNamespace(gpus=1, steps=1, warmup=0), 0)
    line = json.loads(capsys.readouterr().out.strip().splitlines()[-1])
    assert set(line) == {"impl", "unavailable"} and line["impl"] == "reference"
