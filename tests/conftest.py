import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

GOLDEN = os.path.join(ROOT, "tests", "golden")
GOLDEN_CASES = ["convex6_rot", "carved10_rot", "convex5_axis", "single_tet", "cfg0_convex24"]


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")
    config.addinivalue_line("markers", "slow: longer CPU test")


def has_reference_table():
    """The reference's psi table beside the library, or a file the caller names."""
    return "VFRAY_PSI_TABLE" in os.environ or os.path.exists(
        os.path.join(ROOT, "vfray_b200", "data", "psiGammaTable512.bin"))


def pytest_collection_modifyitems(items):
    if has_reference_table():
        return
    for item in items:
        if getattr(item, "originalname", "") == "test_reference_psi_table_is_the_default":
            item.add_marker(pytest.mark.skip(reason="library built without the reference's psi table"))


@pytest.fixture(scope="session", autouse=True)
def default_psi_table(tmp_path_factory):
    """Where the library was built without the reference sources it has no
    default psi table, and a caller that passes none is refused.  GPU tests
    that compare the library with itself or with the oracle hold for any
    table: they, and the driver they start, get the generated one as the
    default."""
    import torch

    if has_reference_table() or not torch.cuda.is_available():
        yield
        return
    import vfray_b200 as vb

    path = tmp_path_factory.mktemp("psi") / "generated.bin"
    vb.psi_table().tofile(path)
    os.environ["VFRAY_PSI_TABLE"] = str(path)
    yield
    del os.environ["VFRAY_PSI_TABLE"]


def has_reference_sources():
    import oracle

    return os.path.isdir(oracle.REF_SOURCES)


def load_golden(name):
    """A golden case with its inputs (regenerated from seeds where the
    fixture stores only a checksum) and the reference outputs."""
    import vfray_b200 as vb
    from tests.golden.make_golden import checksum, make_inputs

    d = dict(np.load(os.path.join(GOLDEN, f"{name}.npz")))
    d["name"] = name
    d["W"], d["H"], d["n_ext"] = int(d["W"]), int(d["H"]), int(d["n_ext"])
    d["psi"] = vb.psi_table()
    assert checksum(d["psi"]) == str(d["psi_sha256"]), "generated psi table drifted"
    if "vert" not in d:
        vert, tet, tf = make_inputs(name)
        p = vb.prepare(vert, tet)
        d.update(vert=p["vert"], tet=p["tet"], con=p["con"], extf=p["extf"], tf=tf)
        assert np.array_equal(p["lmt"], d["lmt"])
    assert checksum(d["vert"], d["tet"], d["con"], d["extf"], d["tf"]) == str(d["input_sha256"])
    return d


@pytest.fixture(scope="session")
def oracle_lib():
    import oracle

    return oracle.Oracle()


@pytest.fixture(scope="session")
def renderer():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import vfray_b200 as vb

    r = vb.Renderer(0)
    yield r
    r.close()
