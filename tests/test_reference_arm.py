"""bench.py --impl reference times the reference's own kernels or says that they are not there: the oracle's
restatement of them is never reported as the reference."""
import json
import sys
from pathlib import Path
from types import SimpleNamespace

import pytest

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))


@pytest.mark.parametrize("kind", ["port", "reference"])
def test_reference_arm_is_the_reference_or_unavailable(kind, monkeypatch, capsys):
    import bench
    monkeypatch.setattr(bench, "build_scene", lambda seed: SimpleNamespace(n_particles=10, n_walls=5))
    monkeypatch.setattr(bench, "ref_kind", lambda spec, V: (SimpleNamespace(step=lambda: None), kind))
    assert bench.reference_arm(SimpleNamespace(steps=2, warmup=1, gpus=1)) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference"
    assert ("value" in line) == (kind == "reference") and ("unavailable" in line) == (kind == "port")
