"""bench.py where the library was built without the reference sources: it
renders with the generated psi table, says so, and leaves out the reference's
CPU baseline instead of stopping."""
import os
import types

import numpy as np
import pytest

import bench
import oracle
import vfray_b200 as vb


@pytest.fixture
def no_table(monkeypatch):
    def absent():
        raise vb.VfrError(vb._lib.VFR_ERR_IO, "file error")

    monkeypatch.setattr(vb, "reference_psi_table", absent)


def test_generated_table_is_used_and_named(no_table):
    sp = dict(name="tiny", desc="", jobs=[(0, None, 8, 8)], tf=None, meshes=[])
    wl = bench.prepare_ours(sp)
    assert np.array_equal(wl["psi"], vb.psi_table())
    cfg = bench.workload_config(wl, 1, "ref")
    assert cfg["psi_table"].startswith("generated") and "psiGammaTable512.h" not in cfg["psi_table"]


def test_a_named_file_is_not_called_the_reference_table(tmp_path, monkeypatch):
    path = tmp_path / "other.bin"
    table = (vb.psi_table() * np.float32(0.5)).astype(np.float32)
    table.tofile(path)
    monkeypatch.setitem(os.environ, "VFRAY_PSI_TABLE", str(path))
    psi, name = bench.bench_psi_table()
    assert np.array_equal(psi, table) and "other.bin" in name and "psiGammaTable512.h" not in name


def test_cpu_baseline_without_the_reference_build(monkeypatch):
    monkeypatch.setattr(oracle, "ref_available", lambda kind: False)
    wl = dict(meshes=[], jobs=[], tf=None)
    assert "unavailable" in bench.cpu_baseline(wl, 1.0)
    out = bench.run_reference(types.SimpleNamespace(), 0)
    assert out["impl"] == "reference" and "unavailable" in out
