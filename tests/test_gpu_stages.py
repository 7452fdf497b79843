"""The three stage calls in the orders a program may make them: a projection
repeated on the same visible faces, before or after a traversal, starts from
those faces alone, so its images, step counts and ray counts are those of a
fresh sequence (whole numbers and floats of the same kernels, compared
exactly)."""
import numpy as np
import pytest

import vfray_b200 as vb
from vfray_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(renderer):
    renderer.upload_tables(synth.transfer_function(2), vb.psi_table())
    p = vb.prepare(*synth.make_mesh(9, carved=True, view_seed=6))
    mid = renderer.upload_mesh(p["vert"], p["tet"], p["con"], p["extf"], p["lmt"])
    yield mid, p["extf"].shape[0]
    renderer.release_mesh(mid)


def _fresh(renderer, scene, W, H):
    mid, n_ext = scene
    vis, _ = renderer.find_visible(mid, n_ext)
    bbox, writer = renderer.project(mid, W, H, len(vis))
    return bbox, writer, renderer.traverse(mid, W, H)


def _same(got, want):
    for k in ("rgb8", "rgba", "steps"):
        assert np.array_equal(got[k], want[k]), k
    for k in ("num_vis", "num_rays", "num_steps", "device_status"):
        assert got["stats"][k] == want["stats"][k], k
    assert want["stats"]["num_rays"] > 0


@pytest.mark.parametrize("sizes", [
    [(64, 48), (200, 150)],                        # the second larger: buffers grow
    [(200, 150), (64, 48), (200, 150)],
    [(33, 47), (33, 47)],
])
@pytest.mark.parametrize("walk_each", [True, False])
def test_projection_repeated_on_the_same_visible_faces(sizes, walk_each, renderer, scene):
    mid, n_ext = scene
    want = [_fresh(renderer, scene, W, H) for W, H in sizes]
    vis, _ = renderer.find_visible(mid, n_ext)
    for k, (W, H) in enumerate(sizes):
        bbox, writer = renderer.project(mid, W, H, len(vis))
        assert np.array_equal(bbox, want[k][0]) and np.array_equal(writer, want[k][1])
        if walk_each or k == len(sizes) - 1:
            _same(renderer.traverse(mid, W, H), want[k][2])


def test_traversal_needs_a_projection_of_its_own(renderer, scene):
    mid, n_ext = scene
    want = _fresh(renderer, scene, 40, 30)[2]
    with pytest.raises(vb.VfrError) as e:
        renderer.traverse(mid, 40, 30)  # its rays are consumed
    assert e.value.status == vb._lib.VFR_ERR_STATE
    vis, _ = renderer.find_visible(mid, n_ext)
    with pytest.raises(vb.VfrError):
        renderer.traverse(mid, 40, 30)  # no projection yet
    renderer.project(mid, 40, 30, len(vis))
    with pytest.raises(vb.VfrError) as e:
        renderer.project(mid, 1, 30, len(vis))  # refused before it touches the projection
    assert e.value.status == vb._lib.VFR_ERR_INVALID
    _same(renderer.traverse(mid, 40, 30), want)
