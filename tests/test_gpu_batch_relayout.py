"""A batch whose job list changes: another list runs as that list whether or
not it is captured again, and a list that is refused leaves the batch, its
captured graph and its outputs as they were."""
import numpy as np
import pytest

import vfray_b200 as vb
from vfray_b200 import batch as vbatch
from vfray_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(renderer):
    renderer.upload_tables(synth.transfer_function(2), vb.psi_table())
    ids = []
    for n, carved in ((9, True), (6, False)):
        p = vb.prepare(*synth.make_mesh(n, carved=carved, view_seed=None))
        ids.append(renderer.upload_mesh(p["vert"], p["tet"], p["con"], p["extf"], p["lmt"]))
    yield ids
    for m in ids:
        renderer.release_mesh(m)


def _read(B, jobs):
    rgb = np.empty(sum(W * H for _, _, W, H in jobs) * 3, np.uint8)
    B.read(rgb8=rgb)
    at = np.cumsum([0] + [W * H * 3 for _, _, W, H in jobs])
    return [rgb[at[k]:at[k + 1]].reshape(H, W, 3) for k, (_, _, W, H) in enumerate(jobs)]


def _lists(ids):
    v = synth.orbit_views(8, seed=3)
    return [
        [(ids[k % 2], v[k], 48 + 8 * k, 40) for k in range(8)],
        [(ids[1], v[1], 130, 70), (ids[0], None, 33, 65)],  # fewer, other sizes
        [(ids[0], v[k % 8], 40, 40) for k in range(12)],
        [(ids[0], v[(k + 3) % 8], 40, 40) for k in range(12)],  # other cameras only
        [(ids[0], v[k % 8], 40, 39) for k in range(12)],  # the same tiles, other pixels
    ]


@pytest.mark.parametrize("mode", [vb.MODE_REF, vb.MODE_COMPOSITED])
@pytest.mark.parametrize("capture", ["first", "each", "never"])
def test_another_list_of_jobs(mode, capture, renderer, scene):
    lists = _lists(scene)
    B = vbatch.BatchRenderer(renderer, lists[0], mode=mode)
    try:
        for k, jobs in enumerate(lists + lists[::-1]):
            if k:
                B.set_jobs(jobs)
            if capture == "each" or (capture == "first" and k == 0):
                B.prepare()
            B.run()
            B.stats()
            got = _read(B, jobs)
            for g, (mid, mv, W, H) in zip(got, jobs):
                want = renderer.render(mid, W, H, mv=mv, mode=mode, rgba=False, steps=False)["rgb8"]
                assert np.array_equal(g, want), (k, W, H)
    finally:
        B.close()


@pytest.mark.parametrize("graph", [False, True])
def test_refused_list_leaves_the_batch_as_it_was(graph, renderer, scene):
    jobs = _lists(scene)[0]
    bad = [(scene[0], None, 1, 64)]
    B = vbatch.BatchRenderer(renderer, jobs, graph=graph)
    try:
        B.prepare()
        B.run()
        want = _read(B, jobs)
        for refused in (bad, jobs * 4 + bad, [(12345, None, 32, 32)] * 40):
            with pytest.raises(vb.VfrError):
                B.set_jobs(refused)
            B.run()
            B.stats()
            assert all(np.array_equal(a, b) for a, b in zip(_read(B, jobs), want))
    finally:
        B.close()
    with pytest.raises(vb.VfrError):
        vbatch.BatchRenderer(renderer, bad)
