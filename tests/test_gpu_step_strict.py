"""The step's uncertain inputs (see test_gpu_step.py) with nothing left out: a
device status is accepted only if it is the cycle's alone and the oracle stops
a ray there too, and then, as always, every pixel's steps and float colours
are compared.

Steps are equal.  A step's colour differs from the oracle's by at most one
rounding of the channel's sum and one of zeta (the double exp of two
libraries), so a pixel's channels by 2^-22 of their magnitude per step."""
import re

import numpy as np
import pytest

import vfray_b200 as vb
from tests.test_gpu_step import _lattice, _mv
from vfray_b200 import batch as vbatch
from vfray_b200 import synth

pytestmark = pytest.mark.gpu


def _run(renderer, mid, W, H, mv, mode):
    """(steps, rgba, device status) of one batched view."""
    for _ in range(4):  # composited lists are sized by a first run
        B = vbatch.BatchRenderer(renderer, [(mid, mv, W, H)], mode=mode, graph=False)
        try:
            B.run()
            status = 0
            try:
                B.stats()
            except vb.VfrError as e:
                if "overflowed" in str(e):
                    continue
                status = int(re.search(r"device status 0x([0-9a-f]+)", str(e)).group(1), 16)
            steps, rgba = np.empty(W * H, np.uint32), np.empty(W * H * 4, np.float32)
            B.read(steps=steps, rgba=rgba)
            return steps, rgba.reshape(-1, 4), status
        finally:
            B.close()
    raise AssertionError("entry lists kept overflowing")


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
        for mode, o in ((vb.MODE_REF, oracle_lib.render_ref(m, W, H)),
                        (vb.MODE_COMPOSITED, oracle_lib.render_composited(m, W, H))):
            steps, rgba, status = _run(renderer, mid, W, H, mv, mode)
            want = np.asarray(o["steps"]).reshape(-1)
            assert status in (0, vb.VFR_DEV_CYCLE), (mode, status)
            assert (status != 0) == bool((want > 4095).any()), (mode, status, want.max())
            assert want.max() > 0 and np.array_equal(steps, want), mode
            ref = np.asarray(o["rgba"]).reshape(-1, 4)
            ok = np.isfinite(ref).all(1)
            assert np.array_equal(np.isfinite(rgba).all(1), ok)
            limit = want[:, None] * 2.0**-22 * np.maximum(1.0, np.abs(ref))
            assert np.all(np.abs(rgba[ok] - ref[ok]) <= limit[ok]), mode
    finally:
        renderer.release_mesh(mid)


@pytest.mark.parametrize("permuted", [False, True])
@pytest.mark.parametrize("n,W,H", [(1, 2, 2), (4, 33, 33), (6, 49, 31), (8, 65, 65)])
def test_rays_through_lattice_edges(n, W, H, permuted, renderer, oracle_lib):
    vert, tet = _lattice(n, permuted)
    _check(renderer, oracle_lib, vb.prepare(vert, tet), synth.transfer_function(2), W, H)


@pytest.mark.parametrize("alpha", [0.0, 1.0, 12.0, 30.0, 3000.0, 2.0**48, 2.0**100])
@pytest.mark.parametrize("lattice", [False, True])
def test_extinctions_of_any_size(alpha, lattice, renderer, oracle_lib):
    vert, tet = _lattice(4) if lattice else synth.make_mesh(5, carved=True, view_seed=4)
    tf = synth.transfer_function(2)
    tf[:, 3] = np.float32(alpha)
    _check(renderer, oracle_lib, vb.prepare(vert, tet), tf, 61, 47)


@pytest.mark.parametrize("decay", [20.0, 60.0, 120.0, 200.0])
@pytest.mark.parametrize("mv", [None, _mv(synth.random_rotation(3))])
def test_scalars_of_many_magnitudes(decay, mv, renderer, oracle_lib):
    """A field with tails: planes whose scalar coefficients are as small as
    floats go, down to zero."""
    vert, tet = synth.make_mesh(7, carved=True, view_seed=4)
    x = vert[:, :3].astype(np.float64)
    p = vb.prepare(vert, tet)
    p["vert"][:, 3] = np.exp(-decay * ((x - x.mean(0)) ** 2).sum(1)).astype(np.float32)
    _check(renderer, oracle_lib, p, synth.transfer_function(2, cutoff=0.0), 61, 47, mv=mv)


@pytest.mark.parametrize("scalar", [lambda x: 0.4 + 0.0 * x[:, 0], lambda x: x[:, 0],
                                    lambda x: np.maximum(0.0, 1 - 3 * ((x - 0.5) ** 2).sum(1)),
                                    lambda x: (x[:, 2] > 0.5) * 1.0])
@pytest.mark.parametrize("alpha", [0.6, 25.0])
def test_planes_with_zero_coefficients(scalar, alpha, renderer, oracle_lib):
    vert, tet = _lattice(5, scalar=scalar)
    p = vb.prepare(vert, tet)
    p["vert"][:, 3] = np.nan_to_num(scalar(0.5 + 0.5 * p["vert"][:, :3]), nan=0.0)
    tf = synth.transfer_function(2)
    tf[:, 3] *= np.float32(alpha)
    _check(renderer, oracle_lib, p, tf, 45, 37)
