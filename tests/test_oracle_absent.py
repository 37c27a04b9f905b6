"""What runs beside the oracle goes on where its library has not been built: the
benchmark's reference arms answer that they are unavailable, the VCA line has no CPU
figure, and the smoke check compares with the oracle's record."""
import argparse
import json

import numpy as np
import pytest


@pytest.fixture
def absent(monkeypatch, tmp_path):
    from oracle import ref, refpath
    monkeypatch.setattr(ref, "LIB_PATH", str(tmp_path / "none.so"))
    monkeypatch.setattr(refpath, "reference_root", lambda required=False: None)


def test_reference_arms_answer_unavailable(absent, capsys):
    import bench
    bench.run_reference(argparse.Namespace(steps=2, warmup=1, gpus=1, no_secondary=False), 1, 0)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"]
    assert "\n" not in line["unavailable"]
    assert bench.batch_line("batch", 2, 0, 1, 1, "reference")["unavailable"]
    assert bench.vca_reference_sample() is None


def test_smoke_has_the_record_of_its_problem(absent):
    import __graft_entry__ as entry
    from oracle import port
    from pyqcm_b200 import workloads as W
    prob = W.chain8()
    sector, e, z, G = entry._recorded(prob, "chain8_L")
    assert sector == "R0:N8:S0:1"
    assert np.allclose(z, W.matsubara(256), rtol=1e-14) and G.shape == (256, 8, 8)
    assert abs(e - port.solve(prob)["E0"]) < 1e-9 * abs(e)
