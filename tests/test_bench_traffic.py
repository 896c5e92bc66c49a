"""The bench line's DRAM traffic is that of the kernel that ran, or none."""
import json
from types import SimpleNamespace

import pytest

import bench


@pytest.mark.parametrize("counted,batch,precision,want", [(1e11, 148, "c128", 5e10), (1.1e11, 148, "c128", 5e10),
                                                          (1.9e11, 148, "c128", None), (0.0, 148, "c128", None),
                                                          (1e11, 64, "c128", None), (1e11, 148, "c64", None)])
def test_traffic_of_this_kernel_and_workload(monkeypatch, tmp_path, counted, batch, precision, want):
    f = tmp_path / "t.json"
    d = dict(chi=256, precision="c128", batch=148, jacobi_precondition="on", dram_bytes_per_launch=5e10,
             counted_bytes_per_launch=1e11)
    f.write_text(json.dumps(d))
    monkeypatch.setattr(bench, "TRAFFIC", str(f))
    args = SimpleNamespace(chi=256, precision=precision, precondition="on")
    assert bench.captured_traffic(args, batch, counted) == want
    del d["counted_bytes_per_launch"]  # a capture that does not say what its kernel counted
    f.write_text(json.dumps(d))
    assert bench.captured_traffic(args, batch, counted) is None


def test_no_capture_no_traffic(monkeypatch, tmp_path):
    monkeypatch.setattr(bench, "TRAFFIC", str(tmp_path / "absent.json"))
    assert bench.captured_traffic(SimpleNamespace(chi=256, precision="c128", precondition="on"), 148, 1e11) is None
