"""launches_per_run counts what a run launches: compared with the kernels that
torch's profiler sees in one run of the library's own stream."""
import numpy as np
import pytest

import vfray_b200 as vb
from vfray_b200 import batch as vbatch
from vfray_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [vb.MODE_REF, vb.MODE_COMPOSITED])
@pytest.mark.parametrize("views,W,H,use_mv", [
    (1, 64, 48, False), (1, 64, 48, True),  # every fold
    (1, 1500, 1100, True),                  # the ray list is more than one wave
    (64, 96, 96, True), (300, 33, 33, True),  # more and more of the others
])
def test_count_of_one_run(mode, views, W, H, use_mv, renderer):
    import torch
    from torch.profiler import ProfilerActivity, profile

    renderer.upload_tables(synth.transfer_function(2), vb.psi_table())
    p = vb.prepare(*synth.make_mesh(9, carved=True, view_seed=6))
    mid = renderer.upload_mesh(p["vert"], p["tet"], p["con"], p["extf"], p["lmt"])
    mvs = synth.orbit_views(views, seed=3)
    B = vbatch.BatchRenderer(renderer, [(mid, mv if use_mv else None, W, H) for mv in mvs],
                             mode=mode, graph=False)
    try:
        assert B.launches_per_run() == 0
        B.run()
        renderer.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            B.run()
            renderer.synchronize()
            torch.cuda.synchronize()
        seen = [e.name for e in prof.events() if "vfr::" in e.name]
        if not seen:
            pytest.skip("the profiler reports no kernels here")
        assert B.launches_per_run() == len(seen), seen
    finally:
        B.close()
        renderer.release_mesh(mid)
