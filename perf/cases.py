"""Benchmark cases of the render path, through the package's public entry points.

Each case is one thing a program does with this package, at the sizes it does
it: single views into device or host memory, the driver's three stage calls,
batches of views over one mesh or many, the frame loop that changes cameras
and reads images back, the request server, and stage (a) on the caller's own
buffers.  Meshes are the seeded synthetic ones of ``vfray_b200.synth`` (a cube
of n^3 cells split into tetrahedra, optionally carved so that rays leave and
re-enter it); the seed moves its vertices, its scalar field, the carving, the
transfer function and every camera.

``listed()`` gives the named cases, ``draw(rng)`` another one of the same
ranges, ``prepare`` the state a program keeps, ``run`` one pass, ``work`` the
bytes and operations a pass cannot do without, and ``exact`` the float results
of a pass in 64 bits where that is quick.
"""
import ctypes
import math

import numpy as np
import torch

import vfray_b200 as vb
from vfray_b200 import synth
from vfray_b200.batch import BatchRenderer, job
from vfray_b200.serve import Server


def listed():
    return [
        # interactive preview while the user drags: the smallest call, all latency
        dict(name="preview", kind="view", n=16, carved=True, W=128, H=128, mode="ref"),
        # the reference driver's own sequence on a mesh as stored: the three
        # stage calls with every intermediate result read back to the host
        dict(name="stages", kind="stages", n=24, carved=False, W=512, H=512),
        # one still frame of an interactive viewer, RGB8 into pinned host memory
        dict(name="frame_host", kind="frame", n=32, carved=True, W=637, H=483, mode="ref"),
        # one frame for further processing on the device (float colour, steps)
        dict(name="view_device", kind="view", n=64, carved=True, W=1024, H=768, mode="ref"),
        # a view in which rays re-enter a non-convex mesh: depth-ordered segments
        dict(name="view_composited", kind="view", n=48, carved=True, W=801, H=600,
             mode="composited"),
        # a large still of a mesh whose records do not fit in L2
        dict(name="still_2048", kind="view", n=96, carved=True, W=2048, H=2048, mode="ref"),
        # an orbit animation: 64 views in one captured batch (the package's headline)
        dict(name="orbit", kind="orbit", n=64, carved=True, views=64, W=512, H=512, mode="ref"),
        # the same kind of batch in composited mode, at a ragged size
        dict(name="orbit_composited", kind="orbit", n=40, carved=True, views=24, W=500, H=375,
             mode="composited"),
        # offline rendering of many meshes at many sizes in one uneven batch
        dict(name="mixed", kind="mixed", nmin=16, nmax=64, meshes=5, jobs=96, res=128, mode="ref"),
        # a frame loop: new cameras in, a few views rendered, images out, every step
        dict(name="frame_loop", kind="loop", n=32, carved=True, views=8, W=512, H=512,
             mode="ref"),
        # a burst of requests to the render server, images of several sizes
        dict(name="served", kind="served", nmin=16, nmax=48, meshes=4, jobs=24, res=256,
             mode="ref"),
        # visible faces on the caller's own device buffers, nothing allocated
        dict(name="visible_static", kind="static", n=48, carved=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["view", "view", "view", "stages", "frame", "orbit", "orbit", "mixed", "loop",
                       "served", "static"])
    n = _log_int(rng, 12, 64)
    carved = rng.random() < 0.8
    mode = "composited" if rng.random() < 0.35 else "ref"
    W, H = _log_int(rng, 90, 1400), _log_int(rng, 90, 1400)
    if kind == "static":
        return dict(kind=kind, n=n, carved=carved)
    if kind == "stages":
        return dict(kind=kind, n=n, carved=False, W=W, H=H)  # the driver's meshes are convex
    if kind in ("view", "frame"):
        return dict(kind=kind, n=n, carved=carved, W=W, H=H, mode=mode)
    if kind in ("orbit", "loop"):
        # at most a third of the listed orbit's pixels, which bounds the cost
        most = max(2, min(48 if kind == "orbit" else 12, int(64 * 512 * 512 / 3 / (W * H))))
        return dict(kind=kind, n=n, carved=carved, views=_log_int(rng, 2, most), W=W, H=H, mode=mode)
    nmin = _log_int(rng, 12, 24)
    return dict(kind=kind, nmin=nmin, nmax=_log_int(rng, nmin, 56), meshes=rng.randint(2, 5),
                jobs=_log_int(rng, 4, 40), res=rng.choice([96, 128, 200]), mode=mode)


# ------------------------------------------------------------------ inputs

_MODES = {"ref": vb.MODE_REF, "composited": vb.MODE_COMPOSITED}


def _mesh(n, carved, seed):
    vert, tet = synth.make_mesh(n, carved=carved, view_seed=seed + 3, jitter_seed=seed,
                                scalar_seed=seed + 1, carve_seed=seed + 4)
    return vb.prepare(vert, tet)


def _sizes(case):
    """Cells per side of each mesh of a many-mesh case."""
    k = case["meshes"]
    step = (case["nmax"] / case["nmin"]) ** (1.0 / max(1, k - 1))
    return [int(round(case["nmin"] * step ** i)) for i in range(k)]


def _jobs(case):
    """(mesh index, W, H) of each job: sizes res to 8 res (requests: to 4 res),
    every third one not square."""
    top = 3 if case["kind"] == "served" else 4
    out = []
    for i in range(case["jobs"]):
        w = case["res"] << ((i * 5 + i // 7) % top)
        out.append(((i * 3 + i // 4) % case["meshes"], w, w if i % 3 else w * 3 // 4 + 1))
    return out


def _rotation(seed):
    return synth._mv(synth.random_rotation(seed))


def _tables(seed):
    return synth.transfer_function(seed + 2), vb.psi_table()


def _outputs(pixels):
    return dict(rgb8=torch.empty(pixels, 3, dtype=torch.uint8, device="cuda"),
                rgba=torch.empty(pixels, 4, dtype=torch.float32, device="cuda"),
                steps=torch.empty(pixels, dtype=torch.int32, device="cuda"))


def _renderer(seed, meshes):
    r = vb.Renderer(0)
    r.upload_tables(*_tables(seed))
    ids = [r.upload_mesh(p["vert"], p["tet"], p["con"], p["extf"], p["lmt"]) for p in meshes]
    return r, ids


def prepare(case, seed):
    seed = 1000 * (int(seed) % 100003)
    kind = case["kind"]
    many = kind in ("mixed", "served")
    if many:
        meshes = [_mesh(n, True, seed + 10 * i) for i, n in enumerate(_sizes(case))]
    else:
        meshes = [_mesh(case["n"], case["carved"], seed)]
    p = meshes[0]
    if kind == "static":
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        n_ext = p["extf"].shape[0]
        room = 32 * case["n"] ** 2  # the caller's list: its pool's size, for any mesh of this n
        return dict(case=case, lib=vb.load(), vert=dev(p["vert"]), tet=dev(p["tet"].view(np.int32)),
                    extf=dev(p["extf"].view(np.int32)), n_ext=n_ext,
                    vis=torch.full((room,), -1, dtype=torch.int32, device="cuda"),
                    count=torch.zeros(1, dtype=torch.int32, device="cuda"))
    r, ids = _renderer(seed, meshes)
    s = dict(case=case, r=r, ids=ids, n_ext=p["extf"].shape[0], mv=_rotation(seed + 7),
             mode=_MODES[case.get("mode", "ref")])
    if kind == "view":
        s["out"] = _outputs(case["W"] * case["H"])
    elif kind == "frame":
        s["rgb8"] = torch.empty(case["H"], case["W"], 3, dtype=torch.uint8, pin_memory=True).numpy()
    elif kind == "orbit":
        px = case["W"] * case["H"]
        s["out"] = _outputs(case["views"] * px)
        part = lambda k: {q: t[k * px:(k + 1) * px] for q, t in s["out"].items()}  # noqa: E731
        cams = synth.orbit_views(case["views"], seed + 7)
        s["batch"] = BatchRenderer(r, [job(ids[0], case["W"], case["H"], mv=m, **part(k))
                                       for k, m in enumerate(cams)], mode=s["mode"])
    elif kind == "loop":
        cams = synth.orbit_views(case["views"], seed + 7)
        s["cams"] = torch.from_numpy(cams).pin_memory()
        s["rgb8"] = torch.empty(case["views"], case["H"], case["W"], 3, dtype=torch.uint8,
                                pin_memory=True)
        s["batch"] = BatchRenderer(r, [(ids[0], m, case["W"], case["H"]) for m in cams],
                                   mode=s["mode"])
    elif kind == "mixed":
        js = _jobs(case)
        at = np.concatenate([[0], np.cumsum([w * h for _, w, h in js])])
        s["out"] = _outputs(int(at[-1]))
        s["batch"] = BatchRenderer(
            r, [job(ids[m], w, h, mv=_rotation(seed + 20 + i),
                    **{q: t[at[i]:at[i + 1]] for q, t in s["out"].items()})
                for i, (m, w, h) in enumerate(js)], mode=s["mode"])
    elif kind == "served":
        s["reqs"] = [(ids[m], w, h, _rotation(seed + 20 + i), np.empty((h, w, 3), np.uint8))
                     for i, (m, w, h) in enumerate(_jobs(case))]
        s["server"] = Server(r, budget_bytes=2 << 30)
        # a program that renders bursts beside other GPU work lets the GPU go
        # as soon as a burst is done
        s["server"].set_idle(400000, 0)
    if "batch" in s:
        # composited lists are sized by a first run: a batch that reports an
        # overflow is laid out again with the room it asked for
        b = s["batch"]
        for _ in range(4):
            b.run()
            try:
                b.stats()
                break
            except vb.VfrError:
                b.close()
                jobs, mode = b.jobs, b.mode
                b = s["batch"] = BatchRenderer(r, jobs, mode=mode)
        b.prepare()
    elif kind == "view" and case["mode"] == "composited":
        for _ in range(4):
            run(s)
            try:
                r.device_status()
                break
            except vb.VfrError:
                continue
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "view":
        o = s["out"]
        s["r"].render_device(s["ids"][0], case["W"], case["H"], mv=s["mv"], mode=s["mode"], **o)
        return o
    if kind == "orbit" or kind == "mixed":
        s["batch"].run()
        return s["out"]
    if kind == "loop":
        s["batch"].run_host(s["rgb8"], cameras=s["cams"])
        return s["rgb8"]
    if kind == "frame":
        s["r"].render_into_host(s["ids"][0], case["W"], case["H"], s["rgb8"], mv=s["mv"],
                                mode=s["mode"])
        return s["rgb8"]
    if kind == "stages":
        r, mid = s["r"], s["ids"][0]
        vis, face_data = r.find_visible(mid, s["n_ext"])
        bbox, writer = r.project(mid, case["W"], case["H"], len(vis))
        out = r.traverse(mid, case["W"], case["H"])
        return dict(vis=vis, face_data=face_data, bbox=bbox, writer=writer, rgb8=out["rgb8"],
                    rgba=out["rgba"], steps=out["steps"])
    if kind == "served":
        sv = s["server"]
        tickets = [sv.submit(m, w, h, mv=mv, mode=s["mode"], out=out)
                   for m, w, h, mv, out in s["reqs"]]
        return [sv.wait(t)[0] for t in tickets]
    # stage (a) on the caller's buffers: the C ABI's own entry point
    p = ctypes.c_void_p
    rc = s["lib"].vfr_find_visible_static(
        p(s["vert"].data_ptr()), s["vert"].shape[0], p(s["tet"].data_ptr()), s["tet"].shape[0],
        p(s["extf"].data_ptr()), s["n_ext"], p(s["vis"].data_ptr()), p(s["count"].data_ptr()),
        p(torch.cuda.current_stream().cuda_stream))
    if rc:
        raise RuntimeError("vfr_find_visible_static: %d" % rc)
    return dict(vis=s["vis"], count=s["count"])


# ------------------------------------------------------------------ work

def work(case):
    """Each mesh read once per pass (32 bytes per tet, 16 per vertex, 8 per
    external face), each output written once (3 + 16 + 4 bytes per pixel, 3
    where only RGB8 is asked for); about 180 operations per tet a ray walks
    through.  A framed cube covers about 0.55 of the image; a ray walks about
    1.7 n tets of a carved mesh to its first exit, 2 n with its re-entries,
    3 n of a convex one."""
    kind = case["kind"]

    def mesh_bytes(n, carved):
        keep = 0.85 if carved else 1.0
        return 6 * n ** 3 * keep * 32 + (n + 1) ** 3 * 0.87 * 16 + 12 * n * n * (1.3 if carved else 1) * 8

    if kind == "static":
        n_ext = 12 * case["n"] ** 2 * (1.3 if case["carved"] else 1.0)
        return {"bytes": n_ext * (8 + 16 + 16 + 2), "flops": n_ext * 60}
    per_ray = {"ref": 1.7, "composited": 2.0}[case.get("mode", "ref")]
    if kind in ("mixed", "served"):
        ns, js = _sizes(case), _jobs(case)
        pixels = sum(w * h for _, w, h in js)
        steps = sum(0.55 * w * h * per_ray * ns[m] for m, w, h in js)
        mesh = sum(mesh_bytes(n, True) for n in ns)
    else:
        pixels = case["W"] * case["H"] * case.get("views", 1)
        steps = 0.55 * pixels * (per_ray if case["carved"] else 3.0) * case["n"]
        mesh = mesh_bytes(case["n"], case["carved"])
    out = 3 if kind in ("frame", "loop", "served") else 23
    return {"bytes": mesh + out * pixels, "flops": 180 * steps}


# ------------------------------------------------------------------ exact

def _planes64(a, b, c):
    """z(x, y) and s(x, y) through three vertices: ([..., 3], [..., 3])."""
    c1 = b[..., 1] - c[..., 1]
    c0 = b[..., 0] - c[..., 0]
    cross = b[..., 0] * c[..., 1] - b[..., 1] * c[..., 0]
    det = a[..., 0] * c1 - a[..., 1] * c0 + cross
    det = torch.where(det.abs() < 1e-12, torch.full_like(det, 1e-12), det)
    out = []
    for k in (2, 3):
        t = (a[..., k], b[..., k], c[..., k])
        mx = t[1] - t[2]
        my = t[1] * c[..., 1] - b[..., 1] * t[2]
        mz = b[..., 0] * t[2] - t[1] * c[..., 0]
        out.append(torch.stack([(t[0] * c1 - a[..., 1] * mx + my) / det,
                                (a[..., 0] * mx - t[0] * c0 + mz) / det,
                                (-a[..., 0] * my - a[..., 1] * mz + t[0] * cross) / det], -1))
    return out


def _at(plane, x, y):
    return x * plane[..., 0] + y * plane[..., 1] + plane[..., 2]


def _inside(a, b, c, x, y, slack):
    """Whether (x, y) lies in the projected triangle; degenerate ones hold nothing."""
    v1, v2 = b[..., :2] - a[..., :2], c[..., :2] - a[..., :2]
    cr = v1[..., 0] * v2[..., 1] - v1[..., 1] * v2[..., 0]
    sg = torch.where(cr < 0, -1.0, 1.0)
    px, py = x - a[..., 0], y - a[..., 1]
    c1 = sg * (v1[..., 0] * py - v1[..., 1] * px)
    c2 = sg * (px * v2[..., 1] - py * v2[..., 0])
    return (cr.abs() >= 1e-12) & (c1 >= 0) & (c2 >= 0) & (c1 + c2 <= cr.abs() + slack)


def _view64(p, tf, psi, mv, W, H, composited):
    """One view in 64 bits: (face planes [nExt, 6], colour [W * H, 4])."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    as_t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a)).to(dev).to(d)  # noqa: E731
    f8, i8 = torch.float64, torch.int64
    v = as_t(p["vert"], f8)
    tet, con = as_t(p["tet"].view(np.int32), i8), as_t(p["con"].view(np.int32), i8)
    extf = as_t(p["extf"].view(np.int32), i8)
    tf, psi = as_t(tf, f8), as_t(psi, f8)
    max_edge = float(p["lmt"][0])
    if mv is not None:  # rotate, normalise, longest edge of the view
        m = as_t(mv, f8)
        xyz = v[:, :3] @ m[:3, :3].T + m[:3, 3]
        lo, hi = xyz.min(0).values, xyz.max(0).values
        cen = (lo + hi) / 2
        sc, s = v[:, 3], 1.0 / (hi - cen).max()
        v = torch.cat([(xyz - cen) * s, ((sc - sc.min()) / (sc.max() - sc.min()))[:, None]], 1)
        q = v[:, :3]
        max_edge = max(float((q[tet[:, i]] - q[tet[:, j]]).square().sum(1).max().sqrt())
                       for i in range(4) for j in range(i))
    # visible faces: the opposite vertex lies in front of the face's plane or on it
    corner = lambda t, k: torch.gather(tet[t], 1, (k & 3)[:, None])[:, 0]  # noqa: E731
    et, ef = extf[:, 0], extf[:, 1]
    a, b, c, o = (v[corner(et, ef + k)] for k in range(4))
    pz, ps = _planes64(a, b, c)
    hidden = _at(pz, o[:, 0], o[:, 1]) < o[:, 2]
    ps[hidden, 0] = -1.0
    planes = torch.cat([pz, ps], 1)
    vis = torch.nonzero(~hidden)[:, 0]
    # (face, pixel) pairs of the visible faces' pixel boxes
    tri = torch.stack([a[vis], b[vis], c[vis]], 1)
    px = ((W - 1.0) * (tri[..., 0] + 1.0) / 2.0).to(i8).clamp(0, W - 1)
    py = ((H - 1.0) * (tri[..., 1] + 1.0) / 2.0).to(i8).clamp(0, H - 1)
    x0, x1, y0, y1 = px.amin(1), px.amax(1), py.amin(1), py.amax(1)
    bw = x1 - x0 + 1
    count = bw * (y1 - y0 + 1)
    pix, face, ez, es = [], [], [], []
    for lo in range(0, vis.numel(), 20000):
        n = count[lo:lo + 20000]
        k = torch.repeat_interleave(torch.arange(lo, lo + n.numel(), device=dev), n)
        r = torch.arange(k.numel(), device=dev) - torch.repeat_interleave(n.cumsum(0) - n, n)
        x, y = x0[k] + r % bw[k], y0[k] + r // bw[k]
        ox, oy = 2.0 * x / (W - 1.0) - 1.0, 2.0 * y / (H - 1.0) - 1.0
        f = vis[k]
        s = _at(ps[f], ox, oy)
        ok = _inside(tri[k, 0], tri[k, 1], tri[k, 2], ox, oy, 0.0) & (s >= 0) & (s <= 1)
        pix.append((y * W + x)[ok])
        face.append(f[ok])
        ez.append(_at(pz[f], ox, oy)[ok])
        es.append(s[ok])
    pix, face, ez, es = (torch.cat(q) for q in (pix, face, ez, es))
    if composited:  # every entry, per pixel front to back
        o = torch.argsort(-ez, stable=True)
        o = o[torch.argsort(pix[o], stable=True)]
    else:  # the last visible face in order
        o = torch.argsort(pix * (extf.shape[0] + 1) + face)
        last = torch.ones_like(o, dtype=torch.bool)
        last[:-1] = pix[o][1:] != pix[o][:-1]
        o = o[last]
    pix, face, ez, es = pix[o], face[o], ez[o], es[o]
    image = torch.zeros(W * H, 4, dtype=f8, device=dev)
    image[:, 3] = 1.0  # transparency, until the end
    rays, length = torch.unique_consecutive(pix, return_counts=True)
    first = length.cumsum(0) - length
    leave = torch.full((rays.numel(),), math.inf, dtype=f8, device=dev)
    for seg in range(int(length.max()) if rays.numel() else 0):
        at = torch.nonzero((length > seg))[:, 0]
        at = at[ez[first[at] + seg] <= leave[at]]
        e = first[at] + seg
        x, y = rays[at] % W, rays[at] // W
        ox, oy = 2.0 * x / (W - 1.0) - 1.0, 2.0 * y / (H - 1.0) - 1.0
        t, f, z = et[face[e]].clone(), ef[face[e]].clone(), ez[e].clone()
        back = (255 * es[e]).to(i8).clamp(0, 255)
        who, last_z = at, z.clone()
        col = image[rays[at]]
        for _ in range(4096):
            if not who.numel():
                break
            q = v[tet[t]]  # [rays, 4, 4]
            pick = lambda k: torch.gather(q, 1, (k & 3)[:, None, None].expand(-1, 1, 4))[:, 0]  # noqa: E731
            ex = torch.full_like(t, -1)
            for i in (3, 2, 1):
                hit = _inside(pick(f + i), pick(f + i + 1), pick(f + i + 2), ox, oy, 1e-12)
                ex = torch.where(hit, (f + i) & 3, ex)
            go = ex >= 0
            exs = ex.clamp(min=0)
            nz, ns = _planes64(pick(exs), pick(exs + 1), pick(exs + 2))
            zn, sn = _at(nz, ox, oy), _at(ns, ox, oy)
            go &= (sn >= -1e-7) & (sn <= 1 + 1e-7)
            sn = sn.clamp(0, 1)
            front = (255 * sn).to(i8).clamp(0, 255)
            dz = (z - zn).abs() / max_edge
            cf, cb = tf[front], tf[back]
            tau_f, tau_b = cf[:, 3] * dz, cb[:, 3] * dz
            zeta = torch.exp(-0.5 * (tau_f + tau_b))
            gi = ((tau_f / (1 + tau_f) + 0.5 / 512) * 512).to(i8).clamp(0, 511)
            gj = ((tau_b / (1 + tau_b) + 0.5 / 512) * 512).to(i8).clamp(0, 511)
            w = psi[gi, gj]
            new = cf[:, :3] * (1 - w)[:, None] + cb[:, :3] * (w - zeta)[:, None] + zeta[:, None] * col[:, :3]
            col = torch.where(go[:, None], torch.cat([new, (col[:, 3] * zeta)[:, None]], 1), col)
            last_z = torch.where(go, zn, last_z)
            nxt = torch.gather(con[t], 1, exs[:, None])[:, 0]
            on = go & (nxt != t)
            if not bool(on.all()):  # rays that end here
                done = ~on
                image[rays[who[done]]] = col[done]
                leave[who[done]] = last_z[done]
            nf = (con[nxt] == t[:, None]).to(i8).argmax(1)
            t, f, z, back = nxt[on], nf[on], zn[on], front[on]
            ox, oy, who, col, last_z = ox[on], oy[on], who[on], col[on], last_z[on]
    image[:, :3] = image[:, :3].clamp(max=1.0)
    image[:, 3] = 1.0 - image[:, 3]
    return planes.cpu(), image.cpu()


def exact(case, seed):
    """Float outputs of the single-view cases in 64 bits; the other cases hold
    many views (seconds each) or return whole numbers and bytes only."""
    kind = case["kind"]
    if kind not in ("view", "stages"):
        return None
    seed = 1000 * (int(seed) % 100003)
    p = _mesh(case["n"], case["carved"], seed)
    tf, psi = _tables(seed)
    mv = None if kind == "stages" else _rotation(seed + 7)
    planes, image = _view64(p, tf, psi, mv, case["W"], case["H"], case.get("mode") == "composited")
    if kind == "view":
        return dict(rgb8=None, rgba=image, steps=None)
    return dict(vis=None, face_data=planes.numpy(), bbox=None, writer=None, rgb8=None,
                rgba=image.reshape(case["H"], case["W"], 4).numpy(), steps=None)
