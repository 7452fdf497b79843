"""The checked build and a vertex id that is out of range before the mesh's
first view with a model-view: the mesh's edges are listed then, so their ids
are met there first.  It comes back as VFR_DEV_RANGE like any other, and the
context stays usable.  In a process of its own, so that the checked library is
the only one loaded there."""
import json
import os
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import ctypes as C, json, os, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from vfray_b200 import _lib
lib = _lib.load(os.path.join(sys.argv[1], "vfray_b200", "libvfray_b200_checked.so"))
lib.vfr_checked_set_id.restype = C.c_int
lib.vfr_checked_set_id.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_uint64, C.c_uint32]
import vfray_b200 as vb
from vfray_b200 import synth
p = vb.prepare(*synth.make_mesh(7, carved=True, view_seed=4))
mv = synth.orbit_views(3, seed=3)[1]
out = {"errors": []}
with vb.Renderer(0) as r:
    r.upload_tables(synth.transfer_function(2), vb.psi_table())
    up = lambda: r.upload_mesh(p["vert"], p["tet"], p["con"], p["extf"], p["lmt"])
    m = up()
    want = r.render(m, 48, 40, mv=mv)
    r.release_mesh(m)
    nV = len(p["vert"])
    for corner, bad in ((0, nV), (3, nV + 1000), (2, 0xffffffff)):
        m = up()
        _lib.check(lib.vfr_checked_set_id(r.h, m, 1, 4 * (len(p["tet"]) // 2) + corner, bad))
        for again in range(2):
            try:
                r.render(m, 48, 40, mv=mv)
                out["errors"].append("none")
            except vb.VfrError as e:
                out["errors"].append(str(e))
        r.release_mesh(m)
    m = up()
    got = r.render(m, 48, 40, mv=mv)
    out["after"] = all(bool(np.array_equal(got[k], want[k])) for k in ("rgb8", "rgba", "steps"))
print(json.dumps(out), flush=True)
"""


def test_bad_vertex_id_before_the_first_rotated_view():
    p = subprocess.run([sys.executable, "-c", SCRIPT, ROOT], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-3000:]
    out = json.loads(p.stdout.strip().splitlines()[-1])
    assert len(out["errors"]) == 6 and all("status 0x4 " in e for e in out["errors"]), out
    assert out["after"]
