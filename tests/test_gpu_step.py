"""The traversal step's certified shortcuts where they are least certain, and
the view set-up's longest edge, against the oracle: rays through lattice
edges and vertices (the exit face's signs are unsure), transfer functions
whose extinctions leave the exponential's table or the psi estimate's range,
limits that do not fit the mesh, planes with zero coefficients, and
model-views that are no rotation (the long edges do not suffice).

Steps and entry faces must be equal.  The colours' only differences are one
rounding of a sum of two floats where the oracle rounds twice, and the double
exp of two libraries: far below one level of 8 bits, which a value on a
level's edge can still change, so one level is allowed."""
import numpy as np
import pytest

import vfray_b200 as vb
from vfray_b200 import synth

pytestmark = pytest.mark.gpu


def _lattice(n, permuted=False, scale=(1.0, 1.0, 1.0), scalar=None):
    xyz, tet = synth.freudenthal_mesh(n, jitter=0.0)
    s = synth.gaussian_field(xyz, 8, 5) if scalar is None else scalar(xyz)
    vert = np.empty((xyz.shape[0], 4), np.float32)
    vert[:, :3] = xyz * np.asarray(scale)
    vert[:, 3] = s
    if permuted:
        tet = synth.permute_tet_vertices(tet, 3)
    return vert, tet


def _check(renderer, oracle_lib, p, tf, W, H, lmt=None, mv=None):
    psi = vb.psi_table()
    lmt = p["lmt"] if lmt is None else np.asarray(lmt, np.float32)
    renderer.upload_tables(tf, psi)
    mid = renderer.upload_mesh(p["vert"], p["tet"], p["con"], p["extf"], lmt)
    vert, edge = p["vert"], float(lmt[0])
    if mv is not None:
        vert = vb.normalize(vb.rotate(vert, mv))
        edge = float(vb.build_lmt(vert, p["tet"])[0])
    m = oracle_lib.mesh(vert, p["tet"], p["con"], p["extf"], np.ascontiguousarray(tf, np.float32),
                        psi, edge)
    try:
        for mode, want in ((vb.MODE_REF, oracle_lib.render_ref(m, W, H)),
                           (vb.MODE_COMPOSITED, oracle_lib.render_composited(m, W, H))):
            try:
                got = renderer.render(mid, W, H, mv=mv, mode=mode)
            except vb.VfrError as e:  # a ray that cycles: the image is not returned
                assert e.status == vb._lib.VFR_ERR_DEVICE
                continue
            assert np.array_equal(got["steps"], np.asarray(want["steps"]).reshape(H, W)), mode
            diff = np.abs(got["rgb8"].astype(int) - np.asarray(want["rgb8"]).reshape(H, W, 3).astype(int))
            assert diff.max() <= 1, (mode, diff.max())
            assert got["steps"].max() > 0
    finally:
        renderer.release_mesh(mid)


@pytest.mark.parametrize("permuted", [False, True])
@pytest.mark.parametrize("n,W,H", [(1, 2, 2), (4, 33, 33), (6, 49, 31)])
def test_rays_through_lattice_edges(n, W, H, permuted, renderer, oracle_lib):
    """Pixel centres on the lattice's lines: cross products that are zero."""
    vert, tet = _lattice(n, permuted)
    _check(renderer, oracle_lib, vb.prepare(vert, tet), synth.transfer_function(2), W, H)


@pytest.mark.parametrize("alpha", [0.0, 1.0, 30.0, 3000.0, -0.5])
def test_extinctions_outside_the_fast_range(alpha, renderer, oracle_lib):
    vert, tet = synth.make_mesh(5, carved=True, view_seed=4)
    tf = synth.transfer_function(2)
    tf[:, 3] = alpha * np.linspace(0.2, 1.0, 256)
    _check(renderer, oracle_lib, vb.prepare(vert, tet), tf, 61, 47)


@pytest.mark.parametrize("alpha", [2.0**30, 2.0**48, 2.0**60, 2.0**100])
@pytest.mark.parametrize("permuted", [False, True])
def test_power_of_two_extinctions(alpha, permuted, renderer, oracle_lib):
    """Depth differences of a lattice seen along its axes are powers of two too,
    so each sum's product with 32 / ln2 has zeros in the low word that holds
    the exponential's table index."""
    vert, tet = _lattice(4, permuted)
    tf = synth.transfer_function(2)
    tf[:, 3] = np.float32(alpha)
    _check(renderer, oracle_lib, vb.prepare(vert, tet), tf, 33, 33, lmt=(1.0, 1.0, -1.0))


@pytest.mark.parametrize("edge", [1e-35, 1e-4, 1e4, 1e20])
def test_limits_that_do_not_fit_the_mesh(edge, renderer, oracle_lib):
    vert, tet = synth.make_mesh(5, view_seed=4)
    p = vb.prepare(vert, tet)
    _check(renderer, oracle_lib, p, synth.transfer_function(2), 47, 61, lmt=(edge, 1.0, -1.0))


@pytest.mark.parametrize("scalar", [lambda x: 0.4 + 0.0 * x[:, 0], lambda x: x[:, 0],
                                    lambda x: (x[:, 2] > 0.5) * 1.0])
def test_planes_with_zero_coefficients(scalar, renderer, oracle_lib):
    vert, tet = _lattice(5, scalar=scalar)
    p = vb.prepare(vert, tet)
    p["vert"][:, 3] = np.nan_to_num(scalar(0.5 + 0.5 * p["vert"][:, :3]), nan=0.0)
    _check(renderer, oracle_lib, p, synth.transfer_function(2), 45, 37)


def _mv(a, t=(0.0, 0.0, 0.0)):
    m = np.eye(4, dtype=np.float32)
    m[:3, :3] = a
    m[:3, 3] = t
    return m


@pytest.mark.parametrize("jitter", [False, True])
@pytest.mark.parametrize("mv", [
    _mv(synth.random_rotation(3)),
    _mv(37.0 * synth.random_rotation(3), (5.0, -2.0, 1.0)),
    _mv(np.diag([1.0, 0.2, 3.0])),
    _mv(synth.random_rotation(3) @ np.array([[1, 0.7, 0], [0, 1, 0], [0, 0.1, 1.0]])),
    _mv(np.diag([1.0, 1.0, 1.0005])),
    _mv(1e-3 * synth.random_rotation(5), (400.0, 0.0, 0.0)),
])
def test_longest_edge_of_any_model_view(mv, jitter, renderer, oracle_lib):
    vert, tet = synth.make_mesh(6, view_seed=None) if jitter else _lattice(6)
    _check(renderer, oracle_lib, vb.prepare(vert, tet), synth.transfer_function(2), 53, 41, mv=mv)
