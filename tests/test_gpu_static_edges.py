"""vfr_find_visible_static at the edges of its blocks of 256 faces and warps of
32, and at the most faces it takes: each face's verdict stands alone, so a list
cut short or repeated has the full list's verdicts in its own order (whole
numbers, compared exactly)."""
import ctypes as C

import numpy as np
import pytest

import vfray_b200 as vb
from vfray_b200 import _lib, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_ext", [0, 1, 31, 32, 33, 255, 256, 257, 511, 65536, 65537, 1 << 18])
def test_visible_faces_of_any_list_length(n_ext, renderer):
    import torch

    vert, tet = synth.make_mesh(9, carved=True, view_seed=6)
    p = vb.prepare(vert, tet)
    faces = p["extf"].shape[0]
    mid = renderer.upload_mesh(p["vert"], p["tet"], p["con"], p["extf"], p["lmt"])
    seen, _ = renderer.find_visible(mid, faces)
    renderer.release_mesh(mid)
    verdict = np.zeros(faces, bool)
    verdict[seen] = True
    pick = np.arange(n_ext) % faces
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    v, t = dev(p["vert"]), dev(p["tet"].view(np.int32))
    f = dev(p["extf"].view(np.int32)[pick] if n_ext else np.zeros((1, 2), np.int32))
    out = torch.full((n_ext + 1,), -7, dtype=torch.int32, device="cuda")
    count = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    want = np.flatnonzero(verdict[pick]) if n_ext else np.empty(0, int)
    ptr = lambda x: C.c_void_p(x.data_ptr())  # noqa: E731
    for _ in range(3):  # back to back: a call must not start on the last one's scratch
        assert vb.load().vfr_find_visible_static(
            ptr(v), v.shape[0], ptr(t), t.shape[0], ptr(f), n_ext, ptr(out), ptr(count),
            C.c_void_p(torch.cuda.current_stream().cuda_stream)) == _lib.VFR_OK
    assert int(count.item()) == len(want)
    got = out.cpu().numpy()
    assert np.array_equal(got[:len(want)], want)
    assert np.all(got[len(want):] == -7)  # nothing past the list
