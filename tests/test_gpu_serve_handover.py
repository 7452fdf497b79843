"""How the request server hands finished images to their callers: in pieces,
one large image after another.  Sizes lie at the edges of a piece (1 MiB of
RGB8), a burst of large images is not finished all at once at its end, and
small images of the same burst do not wait for it."""
import numpy as np
import pytest

import vfray_b200 as vb
from vfray_b200 import serve, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(renderer):
    renderer.upload_tables(synth.transfer_function(2), vb.psi_table())
    p = vb.prepare(*synth.make_mesh(6, carved=True, view_seed=None))
    mid = renderer.upload_mesh(p["vert"], p["tet"], p["con"], p["extf"], p["lmt"])
    yield mid, synth.orbit_views(8, seed=3)
    renderer.release_mesh(mid)


# below, at and above one piece, a few pieces and a byte or so more
SIZES = [(32, 32), (591, 591), (593, 589), (592, 592), (1024, 683), (1031, 1033), (2048, 1024)]


def test_images_of_any_number_of_pieces(renderer, scene):
    mid, views = scene
    reqs = [(W, H, views[k % 8]) for k, (W, H) in enumerate(SIZES * 3)]
    alone = [renderer.render(mid, W, H, mv=mv, rgba=False, steps=False)["rgb8"] for W, H, mv in reqs]
    with serve.Server(renderer, budget_bytes=4 << 30) as S:
        tickets = [S.submit(mid, W, H, mv=mv) for W, H, mv in reqs]
        for k, t in enumerate(tickets):
            assert np.array_equal(S.wait(t, timeout_ms=60000)[0], alone[k]), reqs[k][:2]


def test_large_images_finish_one_after_another(renderer, scene):
    """12 images of 12 MB, rendered faster than they are copied.  Handed over
    in turn, the one in the middle of the burst is done halfway through the
    copying; handed over together, all are done in its last twelfth.  The
    limit between the two allows for the start of the copying."""
    mid, views = scene
    small = 64
    with serve.Server(renderer, budget_bytes=8 << 30) as S:
        ratio, waited = [], []
        for _ in range(3):
            big = [S.submit(mid, 2048, 2048, mv=views[k % 8]) for k in range(12)]
            little = [S.submit(mid, small, small, mv=views[k % 8]) for k in range(12)]
            info = [S.wait(t, timeout_ms=60000)[1] for t in big]
            info_s = [S.wait(t, timeout_ms=60000)[1] for t in little]
            ready = min(i["t_ready_ms"] for i in info)
            done = sorted(i["t_done_ms"] for i in info)
            ratio.append((done[5] - ready) / (done[-1] - ready))
            waited.append(max(i["t_done_ms"] - i["t_ready_ms"] for i in info_s)
                          / (done[-1] - ready))
        assert min(ratio) < 0.75, ratio
        assert min(waited) < 0.5, waited
