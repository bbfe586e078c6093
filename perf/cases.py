"""The workloads this library is timed on, and what they compute in 64 bits.

Seven kinds of call, each through the public entry points (``mrfmap_gb300.lib``
and ``mrfmap_gb300.warmstart``):

score    the log-likelihood image and sum of a depth image at a pose, image
         and results on the device: the inner call of a pose search
render   an evaluation image of a map at a pose, host arrays in and out
infer    BP iterations on a map whose incidence lists are built
map      a map from host depth images to host log-odds: create, add the views,
         build, iterate, read back
stream   a walk: every frame is added, a few incremental iterations run, the
         frame that leaves the keyframe window is retired
predict  the warm-start network's log-odds of a map's bricks
train    one training step of that network: loss, gradients, updated weights

Maps are compared by their total log-odds (brick slots in order, zeros behind
them, so that the arrays of one workload have one size); BP runs are kept to
view counts and schedules that settle: where the iterations still oscillate,
a last-bit difference grows until it says nothing.

``exact`` restates the computations with torch in 64 bits on the traversal's
specified fp32 geometry (separately rounded operations in a fixed order).
"""
import math

import numpy as np
import torch

from mrfmap_gb300 import lib, synthetic, warmstart
from mrfmap_gb300.params import MapParams

FREE, RETURN, NO_RETURN = 1e-4, 1e-3, 10.0  # belief clamp, likelihood floor, range without a return


def listed():
    return [
        # a pose search against a coarse map on a low-resolution stream: the smallest call
        dict(name="score_160x120_4cm", kind="score", rows=120, cols=160, res=0.04, field="loaded"),
        # the same at full resolution in the map that BP at 1 cm left
        dict(name="score_640x480_1cm", kind="score", rows=480, cols=640, res=0.01, field="bp"),
        # the depth image a map expects at a pose, as an evaluation asks for it
        dict(name="render_320x240_2cm", kind="render", rows=240, cols=320, res=0.02, field="loaded", mode=0),
        # the reference's schedule on a small room: launches and latency
        dict(name="infer_5x160x120_4cm", kind="infer", views=5, rows=120, cols=160, res=0.04, scenes=0, iters=10),
        # the headline map's resolution and iterations, with a window of 8 keyframes
        dict(name="infer_8x640x480_1cm", kind="infer", views=8, rows=480, cols=640, res=0.01, scenes=0, iters=20),
        # several scenes of mixed image sizes in one map, all views of an iteration at once
        dict(name="infer_8scenes_32_2cm", kind="infer", views=4, rows=480, cols=640, res=0.02, scenes=8, iters=10),
        # a small map from images to log-odds: host work, copies and synchronisations
        dict(name="map_5x160x120_4cm", kind="map", views=5, rows=120, cols=160, res=0.04, iters=10, full_ray=True),
        # the reference's viewer configuration: 12 keyframes, bricks around the returns only, 3 iterations
        dict(name="map_12x640x480_2cm", kind="map", views=12, rows=480, cols=640, res=0.02, iters=3, full_ray=False),
        # the large map from images to log-odds
        dict(name="map_8x640x480_1cm", kind="map", views=8, rows=480, cols=640, res=0.01, iters=20, full_ray=True),
        # 16 frames of a walk with a window of 8 keyframes
        dict(name="stream_16x640x480_2cm", kind="stream", frames=16, window=8, rows=480, cols=640, res=0.02, iters=5),
        # the network on the bricks of a ten-view 2 cm map
        dict(name="predict_18432", kind="predict", bricks=18432),
        # a training step at the training's batch size
        dict(name="train_512", kind="train", bricks=512),
    ]


def _spread(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["score", "render", "infer", "infer", "map", "stream", "predict", "train"])
    if kind in ("predict", "train"):
        return dict(kind=kind, bricks=int(_spread(rng, 37, 18432 if kind == "predict" else 2048)))
    rows = int(_spread(rng, 61, 480))
    cols = min(640, int(rows * rng.uniform(1.2, 1.5)))
    if kind in ("score", "render"):
        res = round(_spread(rng, 0.02, 0.05), 3)
        c = dict(kind=kind, rows=rows, cols=cols, res=res, field="loaded")
        return dict(c, mode=rng.choice([0, 0, 1, 2, 3])) if kind == "render" else c
    if kind == "stream":
        return dict(kind=kind, frames=rng.randint(3, 14), window=rng.randint(2, 8), rows=rows, cols=cols,
                    res=round(_spread(rng, 0.02, 0.05), 3), iters=rng.randint(1, 5))
    if kind == "map":
        return dict(kind=kind, views=rng.randint(1, 8), rows=rows, cols=cols, res=round(_spread(rng, 0.012, 0.05), 3),
                    iters=rng.randint(1, 12), full_ray=rng.random() < 0.5)
    if rng.random() < 0.3:
        return dict(kind=kind, views=rng.randint(2, 4), rows=rows, cols=cols, res=round(_spread(rng, 0.02, 0.04), 3),
                    scenes=rng.randint(2, 8), iters=rng.randint(1, 10))
    return dict(kind=kind, views=rng.randint(2, 8), rows=rows, cols=cols, res=round(_spread(rng, 0.012, 0.05), 3),
                scenes=0, iters=rng.randint(2, 20))


# ---- inputs ------------------------------------------------------------------

def _params(case, dims):
    f = 525.0 * case["cols"] / 640
    p = MapParams(res=case["res"], dims=tuple(dims), rows=case["rows"], cols=case["cols"], fx=f, fy=f,
                  cx=case["cols"] / 2, cy=case["rows"] / 2, prior=0.1, max_iters=case.get("iters", 1))
    return synthetic.sensor_params(p)


def _depth(scene, cam, pose, seed, max_range=5.0):
    """z-depth of the scene's room, boxes and spheres with the sensor's noise and dropouts (on the device)."""
    rows, cols, fx, fy, cx, cy = cam
    t64 = dict(device="cuda", dtype=torch.float64)
    xs = (torch.arange(cols, **t64) + 0.5 - cx) / fx
    ys = (torch.arange(rows, **t64) + 0.5 - cy) / fy
    P = torch.tensor(np.asarray(pose), **t64)
    rc = torch.stack(torch.broadcast_tensors(xs[None, :], ys[:, None], torch.ones(rows, cols, **t64)), -1)
    d = (rc @ P[:3, :3].T).reshape(-1, 3)
    o = P[:3, 3]
    inv = 1.0 / d
    room = torch.tensor(scene.room, **t64)
    t = torch.maximum((room[:3] - o) * inv, (room[3:] - o) * inv).amin(1)
    for b in torch.tensor(np.asarray(scene.boxes), **t64):
        lo, hi = (b[:3] - o) * inv, (b[3:] - o) * inv
        tn, tf = torch.minimum(lo, hi).amax(1), torch.maximum(lo, hi).amin(1)
        t = torch.where((tn <= tf) & (tn > 0), torch.minimum(t, tn), t)
    for s in torch.tensor(np.asarray(scene.spheres).reshape(-1, 4), **t64):
        oc = o - s[:3]
        a, b, c = (d * d).sum(1), 2 * d @ oc, oc @ oc - s[3] ** 2
        disc = b * b - 4 * a * c
        tn = (-b - disc.clamp(min=0).sqrt()) / (2 * a)
        t = torch.where((disc >= 0) & (tn > 0), torch.minimum(t, tn), t)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    z = t + torch.randn(t.shape, generator=g, **t64) * (0.002 + 0.0012 * t * t)
    z[torch.rand(t.shape, generator=g, device="cuda") < 0.02] = 0.0
    z[z > max_range] = 0.0
    return z.float().reshape(rows, cols)


def _views(case, seed):
    """(params, views): views of a room, of the batch's scenes or of a walk, each a dict of pose, depth (device),
    camera and, in a batch, the scene's brick box."""
    if case["kind"] == "stream":
        w = synthetic.walk_room(seed, n_frames=case["frames"], rows=case["rows"], cols=case["cols"], res=case["res"])
        p = w.params
        cam = (p.rows, p.cols, p.fx, p.fy, p.cx, p.cy)
        return p, [dict(pose=P, cam=cam, depth=d) for P, d in
                   zip(w.poses, synthetic.render_frames_torch(w, range(case["frames"])))]
    if case.get("scenes"):
        r, c = case["rows"], case["cols"]
        b = synthetic.batch_scenes(seed, n_scenes=case["scenes"], views_per_scene=case["views"], res=case["res"],
                                   sizes=((r // 4, c // 4), (r // 2, c // 2), (r, c)))
        depths = synthetic.render_batch_torch(b, range(len(b.poses)))
        return b.params, [dict(pose=P, cam=k, depth=d, box=b.boxes[s]) for P, k, d, s in
                          zip(b.poses, b.cams, depths, b.scene_of)]
    n = case.get("views", 4)
    w = synthetic.full_room(seed, n_frames=n, rows=24, cols=32, res=case["res"])
    p = _params(case, w.params.dims)
    cam = (p.rows, p.cols, p.fx, p.fy, p.cx, p.cy)
    return p, [dict(pose=P, cam=cam, depth=_depth(w.scene, cam, P, seed * 131 + k)) for k, P in enumerate(w.poses)]


def _field(case, seed):
    """An occupancy map to load, as points (voxel units) and occupancies, with the view to score in it: the free
    space of a room at small probabilities, its surfaces a few voxels thick at large ones."""
    p, views = _views(dict(case, views=1), seed)
    scene = synthetic.full_room(seed, n_frames=1, rows=24, cols=32, res=case["res"]).scene
    n = [int(round(d / p.res)) for d in p.dims]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 7)
    ax = [torch.arange(k, device="cuda", dtype=torch.float32) + 0.5 for k in n]
    v = torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    w = v * p.res - torch.tensor([p.dims[0] / 2, p.dims[1] / 2, 0.0], device="cuda")
    far = torch.full((len(v),), 1e9, device="cuda")  # signed distance to the nearest surface, inside negative
    for b in torch.tensor(np.asarray(scene.boxes), device="cuda", dtype=torch.float32):
        far = torch.minimum(far, torch.maximum(b[:3] - w, w - b[3:]).amax(1))
    for s in torch.tensor(np.asarray(scene.spheres), device="cuda", dtype=torch.float32):
        far = torch.minimum(far, (w - s[:3]).norm(dim=1) - s[3])
    room = torch.tensor(scene.room, device="cuda", dtype=torch.float32)
    far = torch.minimum(far, torch.minimum(w - room[:3], room[3:] - w).amin(1))
    known = far > -2 * p.res
    far, v = far[known], v[known]
    u = torch.rand(far.shape, generator=g, device="cuda")
    occ = torch.where(far < p.res, 0.3 + 0.6999 * u, torch.pow(10.0, -4.0 + 2.0 * u * u))
    return p, views[0], v, occ


def _bricks_input(case, seed):
    """Features, targets and weights of a map's bricks: mostly free or unseen voxels, surfaces in some."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n = case["bricks"]
    r = lambda *s: torch.rand(s, generator=g, device="cuda")  # noqa: E731
    seen = (r(n, 1) < 0.8).float() * (r(n, 512) < 0.9).float()
    near = (r(n, 1) < 0.4).float() * (r(n, 512) < 0.3).float() * seen
    feat = torch.stack([near * r(n, 512), seen * torch.log1p(30 * r(n, 512)), near * torch.log1p(200 * r(n, 512)),
                        near * torch.log1p(10 * r(n, 512))], -1).contiguous()
    target = (seen * (-9.0 + 4 * r(n, 512)) + near * 12 * r(n, 512)).contiguous()
    return feat, target, seen.contiguous()


# ---- the calls -----------------------------------------------------------------

def _add(m, v):
    if "box" in v:
        _, _, fx, fy, cx, cy = v["cam"]
        return m.add_view_box(v["pose"], v["host"], fx, fy, cx, cy, *v["box"])
    return m.add_view(v["pose"], v["host"])


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("predict", "train"):
        feat, target, weight = _bricks_input(case, seed)
        net = warmstart.WarmNet.load_file(warmstart.DEFAULT_WEIGHTS)
        net.predict(feat)  # the workspace
        return dict(case, net=net, feat=feat, target=target, weight=weight, norm=float(weight.sum()))
    if kind in ("score", "render") and case["field"] == "loaded":
        p, view, points, occ = _field(case, seed)
        m = lib.MRFMap(p, activation=lib.ACT_ENDPOINT)
        m.load_map(points.cpu().numpy(), occ.cpu().numpy())
        return dict(case, m=m, pose=view["pose"], depth=view["depth"], host=view["depth"].cpu().numpy(),
                    image=torch.empty_like(view["depth"]), sum=torch.empty(1, device="cuda"))
    p, views = _views(case, seed)
    for v in views:
        v["host"] = v["depth"].cpu().pin_memory().numpy()
    if kind in ("map", "stream"):
        for v in views:
            del v["depth"]
        return dict(case, params=p, views=views, out=_outputs(case, p))
    m = lib.MRFMap(p, activation=lib.ACT_FULL_RAY)
    scored = views.pop() if kind in ("score", "render") else None
    for v in views:
        _add(m, v)
    if scored is not None:
        m.infer(iters=5)
        return dict(case, m=m, pose=scored["pose"], depth=scored["depth"], host=scored["host"],
                    image=torch.empty_like(scored["depth"]), sum=torch.empty(1, device="cuda"))
    flags = lib.JACOBI if case["scenes"] else 0
    m.infer(iters=4, flags=flags)  # the lists
    return dict(case, m=m, flags=flags, out=_outputs(case, p))


def _most_bricks(case, p):
    if case["kind"] == "stream":
        return 40000 + 6000 * case["frames"]
    if case.get("scenes"):
        return 40000 * case["scenes"]
    return math.prod(int(math.ceil(d / p.res) + 16) // 8 for d in p.dims)


def _outputs(case, p):
    """Pinned host arrays for brick centres and log-odds, as a program that reads maps again and again keeps them."""
    n = _most_bricks(case, p)
    return dict(centres=torch.zeros(n, 3, pin_memory=True).numpy(), logodds=torch.zeros(n, 512, pin_memory=True).numpy())


def _read(m, out):
    n = m.num_bricks
    lib._check(lib.load().mrf_read_bricks(m.handle, lib._fp(out["centres"]), None, n))
    lib._check(lib.load().mrf_read_logodds(m.handle, lib._fp(out["logodds"]), n))
    return out


def run(s):
    kind = s["kind"]
    if kind == "score":
        s["m"].likelihood_device(s["pose"], s["depth"].data_ptr(), s["image"].data_ptr(), s["sum"].data_ptr())
        return dict(image=s["image"], sum=s["sum"])
    if kind == "render":
        image, score, counts = s["m"].render(s["mode"], s["pose"], s["host"])
        return dict(image=image, score=score, counts=counts)
    if kind == "infer":
        s["m"].reset_state()
        s["m"].infer(iters=s["iters"], flags=s["flags"])
        return _read(s["m"], s["out"])
    if kind == "map":
        m = lib.MRFMap(s["params"], activation=lib.ACT_FULL_RAY if s["full_ray"] else lib.ACT_ENDPOINT)
        for v in s["views"]:
            _add(m, v)
        m.infer(iters=s["iters"])
        _read(m, s["out"])
        m.close()
        return s["out"]
    if kind == "stream":
        m = lib.MRFMap(s["params"], activation=lib.ACT_FULL_RAY)
        for k, v in enumerate(s["views"]):
            _add(m, v)
            if k >= s["window"]:
                m.retire_view(k - s["window"])
            m.infer(iters=s["iters"], flags=lib.INCREMENTAL)
        _read(m, s["out"])
        m.close()
        return s["out"]
    net = s["net"]
    if kind == "predict":
        return net.predict(s["feat"])
    loss = net.gradients(s["feat"], s["target"], s["weight"], s["norm"])
    net.adam()
    return dict(loss=loss, grads=net.grads, params=net.params)


def work(case):
    """Bytes and operations a pass cannot do without.  BP, per iteration: a 12-byte read (pair, length, cavity
    term) per voxel a ray crosses and a 4-byte message written and read per voxel of its depth window."""
    kind = case["kind"]
    if kind in ("predict", "train"):
        macs = 512 * 27 * (4 * 16 + 16 * 16 + 16)
        n = case["bricks"]
        return dict(bytes=n * 512 * 4 * (5 if kind == "predict" else 6), flops=2 * macs * n * (1 if kind == "predict" else 3))
    pix = case["rows"] * case["cols"]
    cells = 36.0 * 3 / case["res"] ** 3 * 4  # the room's voxels, 4 bytes each
    cross = 1.5 * 3.2 / case["res"]  # voxels a ray crosses: mean range, and the grid's angle
    if kind in ("score", "render"):
        return dict(bytes=8 * pix + min(cells, 4 * pix * cross), flops=20 * pix * cross)
    n = case.get("frames") or case["views"] * max(1, case["scenes"] if "scenes" in case else 1)
    if case.get("scenes"):
        pix = pix / 8
    window = 1.5 * 0.4 / case["res"]  # inside the sensor's depth window
    live = sum(min(k + 1, case["window"]) for k in range(n)) if kind == "stream" else n
    bp = case["iters"] * live * pix * (12 * cross + 8 * window)
    build = 0 if kind == "infer" else n * pix * (4 + 12 * cross)
    return dict(bytes=bp + build + min(cells, n * pix * cross * 4),
                flops=case["iters"] * live * pix * cross * 10 + (0 if kind == "infer" else n * pix * cross * 20))


# ---- the same in 64 bits ---------------------------------------------------------

class _Exact:
    """A map on a dense voxel grid: traversal in the specified fp32 operations, everything else in 64 bits."""

    def __init__(self, p):
        f = np.float32
        self.p, self.res = p, f(p.res)
        g = [f(d) / self.res for d in p.dims]
        self.nb = [(int(math.ceil(x)) + 8) // 8 for x in g]
        self.hi = [float(x) for x in g]
        self.off = [f(p.dims[0]) * f(0.5) / self.res, f(p.dims[1]) * f(0.5) / self.res, f(0)]
        self.sigma = [float(f(x)) for x in p.const_sigmasq_poly]
        self.size = [8 * k for k in self.nb]
        self.active = torch.zeros(math.prod(self.nb), dtype=torch.bool, device="cuda")
        self.order = []  # bricks in slot order, one tensor an activation
        self.lp = math.log(p.prior) - math.log(1 - p.prior)
        self.L = torch.full((math.prod(self.size),), self.lp, dtype=torch.float64, device="cuda")
        self.views = []

    def poly(self, s):
        c = self.sigma
        return ((s * s) * c[2] + s * c[1]) + c[0]

    def commit(self, flags):
        new = flags & ~self.active
        self.active |= new
        self.order.append(new.nonzero().reshape(-1))

    def mark(self, flags, pv, lo=(0, 0, 0), hi=None):
        """The bricks within a voxel of the points pv [n, 3]."""
        hi = hi or self.nb
        v = pv.floor().long()
        ends = [[((v[:, a] + e) // 8).clamp(lo[a], hi[a] - 1) for e in (-1, 1)] for a in range(3)]
        for k in range(8):
            b = [ends[a][(k >> a) & 1] for a in range(3)]
            flags[(b[0] * self.nb[1] + b[1]) * self.nb[2] + b[2]] = True

    def rays(self, view):
        f, (rows, cols, fx, fy, cx, cy) = np.float32, view["cam"]
        P = [float(x) for x in np.asarray(view["pose"], f).reshape(-1)]
        x = torch.arange(cols, device="cuda", dtype=torch.float32) + 0.5
        y = torch.arange(rows, device="cuda", dtype=torch.float32) + 0.5
        rx = (2.0 * (x / torch.full_like(x, cols)) - 1.0) * float(f(cx) / f(fx))
        ry = (2.0 * (y / torch.full_like(y, rows)) - 1.0) * float(f(cy) / f(fy))
        ry, rx = torch.meshgrid(ry, rx, indexing="ij")
        rx, ry = rx.reshape(-1), ry.reshape(-1)
        dw = [(rx * P[4 * a] + ry * P[4 * a + 1]) + P[4 * a + 2] for a in range(3)]
        n = ((dw[0] * dw[0] + dw[1] * dw[1]) + dw[2] * dw[2]).sqrt()
        d = torch.stack([k / n for k in dw])
        o = torch.tensor([[float(f(P[4 * a + 3]) / self.res + self.off[a])] for a in range(3)], device="cuda")
        mult = ((d[0] * P[2] + d[1] * P[6]) + d[2] * P[10]).abs() * float(self.res)
        return o, d, mult

    def walk(self, view):
        """The voxels of every ray in step: (voxel coordinates [3, n], length, entry and exit parameter, alive)."""
        o, d, _ = self.rays(view)
        box = view.get("box", ((0, 0, 0), self.nb))
        lo, hi = (torch.tensor([[8.0 * k] for k in b], device="cuda") for b in box)
        inv = torch.where(d != 0, torch.ones_like(d) / d, torch.zeros_like(d))
        a, b = (lo - o) * inv, (hi - o) * inv
        inf = torch.full_like(d, math.inf)
        tn = torch.where(d != 0, torch.minimum(a, b), -inf).amax(0).clamp(min=0)
        tf = torch.where(d != 0, torch.maximum(a, b), inf).amin(0)
        alive = (tn < tf) & ((d != 0) | ((o >= lo) & (o < hi))).all(0)
        v = torch.minimum(torch.maximum((o + tn * d).floor(), lo), hi - 1)
        step, tprev = torch.sign(d), tn
        while bool(alive.any()):
            for _ in range(16):
                t = torch.where(step > 0, ((v + 1) - o) * inv, torch.where(step < 0, (v - o) * inv, inf))
                ax = torch.where((t[0] <= t[1]) & (t[0] <= t[2]), 0, torch.where(t[1] <= t[2], 1, 2))[None]
                te = t.gather(0, ax)[0]
                yield v, (te - tprev).clamp(min=0), tprev, te, alive
                tprev = torch.maximum(tprev, te)
                v = v.scatter_add(0, ax, step.gather(0, ax))
                alive = alive & ((v >= lo) & (v < hi)).all(0)

    def brick(self, v, alive):
        b = (v * 0.125).floor().long().clamp(min=0)
        lin = (b[0].clamp(max=self.nb[0] - 1) * self.nb[1] + b[1].clamp(max=self.nb[1] - 1)) * self.nb[2] \
            + b[2].clamp(max=self.nb[2] - 1)
        return torch.where(alive, lin, torch.full_like(lin, -1))

    def voxel(self, v):
        w = [v[a].long().clamp(0, self.size[a] - 1) for a in range(3)]
        return (w[0] * self.size[1] + w[1]) * self.size[2] + w[2]

    def activate(self, view, full_ray):
        rows, cols, fx, _, cx, cy = view["cam"]
        f, d = np.float32, view["depth"].reshape(-1)
        P = [float(x) for x in np.asarray(view["pose"], f).reshape(-1)]
        flags = torch.zeros_like(self.active)
        lo, hi = view.get("box", ((0, 0, 0), self.nb))
        x = torch.arange(cols, device="cuda", dtype=torch.float32).repeat(rows)
        y = torch.arange(rows, device="cuda", dtype=torch.float32).repeat_interleave(cols)
        z = d / torch.full_like(d, fx)
        X, Y = z * (x - float(f(cx))), z * (y - float(f(cy)))
        pv = torch.stack([(((X * P[4 * a] + Y * P[4 * a + 1]) + d * P[4 * a + 2]) + P[4 * a + 3])
                          * float(f(1) / self.res) + float(self.off[a]) for a in range(3)], 1)
        gate = [min(self.hi[a], 8.0 * hi[a]) for a in range(3)]
        ok = (d > 0) & torch.stack([(pv[:, a] >= 8.0 * lo[a]) & (pv[:, a] < gate[a]) for a in range(3)]).all(0)
        self.mark(flags, pv[ok], lo, hi)
        if full_ray:
            mult = self.rays(view)[2]
            cur = torch.full(d.shape, -1, dtype=torch.long, device="cuda")
            s_last, going = torch.zeros_like(d), d > 0
            for v, _, _, te, alive in self.walk(view):
                lin = self.brick(v, alive)
                new = going & alive & (lin != cur)
                going = going & ~(new & (cur >= 0) & (s_last > d + 3.0 * self.poly(s_last)))
                flags[lin[new & going]] = True
                cur = torch.where(new, lin, cur)
                s_last = torch.where(alive, te * mult, s_last)
        self.commit(flags)

    def trace(self, view):
        """The lists of a view, rays in columns, steps in rows."""
        d, mult = view["depth"].reshape(-1), self.rays(view)[2]
        cur = torch.full(d.shape, -1, dtype=torch.long, device="cuda")
        none = torch.full_like(cur, -1)
        opened, pre, post = torch.zeros_like(d, dtype=torch.bool), d > 0, d > 0
        s_last, start, r0, k = torch.zeros_like(d), none.clone(), none.clone(), 0
        vox, length, mu, inpost = [], [], [], []

        def close(ended):
            nonlocal pre, post
            rhs = d + 3.0 * self.poly(s_last)
            post = post & ~(ended & (s_last >= rhs))
            pre = pre & ~(ended & (s_last > rhs))

        for v, l, _, te, alive in self.walk(view):
            lin = self.brick(v, alive)
            close(opened & (lin != cur))
            opened = opened & (lin == cur)
            cur = lin
            here = alive & pre & self.active[lin.clamp(min=0)]
            s = te * mult
            start = torch.where(here & ~opened, torch.full_like(start, k), start)
            x = (d - s).abs() / (3.0 * self.poly(s))
            hit = here & (0.5 * (x * x) <= 87.0)
            r0 = torch.where(hit & (r0 < 0), start, r0)
            s6 = 3.0 * (self.sigma[0] + self.sigma[1] * s.double() + self.sigma[2] * s.double() ** 2)
            m = 0.398942 / s6 * torch.exp(-0.5 * ((d.double() - s.double()) / s6) ** 2)
            vox.append(torch.where(here, self.voxel(v), none).int())
            length.append(torch.where(here, l, torch.zeros_like(l)))
            mu.append(torch.where(hit, m, torch.zeros_like(m)))
            inpost.append(here & post)
            opened = opened | here
            s_last = torch.where(here, s, s_last)
            k += 1
        ran = pre & opened  # lists that end at the volume's face
        gate = (d > 0) & pre & (s_last > 0) & (d > s_last)
        if bool(ran.any()):
            close(ran)
            gate &= pre
        first = torch.where(r0 >= 0, r0, start)
        some = torch.stack([(x >= 0).any() for x in vox]).cpu().numpy().nonzero()[0]
        n = int(some[-1]) + 1 if len(some) else 1
        view.update(vox=torch.stack(vox[:n]), l=torch.stack(length[:n]).double(), mu=torch.stack(mu[:n]),
                    post=torch.stack(inpost[:n]), first=first, gate=gate)
        keep = view["vox"] >= 0
        view["at"] = torch.where(keep, view["vox"], 0).long()
        cum = torch.zeros_like(self.L).index_add_(0, view["at"][view["post"]], view["l"][view["post"]])
        view["pairs"] = (cum.float() > 0.1).nonzero().reshape(-1)
        view["cum"] = cum[view["pairs"]]
        view["m"] = torch.zeros_like(view["cum"])

    def update(self, view):
        """The view's new messages from the present log-odds."""
        eta = self.L.clone()
        eta[view["pairs"]] -= view["m"]
        q = (1.0 / (1.0 + torch.exp(eta))).clamp(FREE, 1 - FREE)[view["at"]]
        A = torch.cumsum(view["l"] * torch.log(q), 0)
        start = (view["first"] - 1).clamp(min=0)[None]
        A0 = torch.where(view["first"] > 0, A.gather(0, start)[0], torch.zeros_like(A[0]))
        steps = torch.arange(len(A), device="cuda")[:, None]
        T = torch.where(steps >= view["first"], torch.exp(A - A0) * (1 - q) * view["mu"], 0.0).sum(0)
        T = T + torch.where(view["gate"], torch.exp(A[-1] - A0), 0.0)
        vmu = torch.exp(A) * view["mu"] * view["post"]
        tau = vmu * (1 - q)
        F = torch.cumsum(tau, 0) - tau
        mu1, mu0 = F + vmu, F + ((T - F) - tau) / q
        p = (mu1 / (mu1 + mu0 + 1e-7)).clamp(FREE, 1 - FREE)
        acc = torch.zeros_like(self.L).index_add_(0, view["at"][view["post"]], (p * view["l"])[view["post"]])
        a = (acc[view["pairs"]] / view["cum"]).clamp(FREE, 1 - FREE)
        return torch.log(a) - torch.log(1 - a)

    def infer(self, views, iters, jacobi=False):
        for _ in range(iters):
            held = []
            for v in views:
                new = self.update(v)
                held.append((v, new))
                if not jacobi:
                    self.L[v["pairs"]] += new - v["m"]
                    v["m"] = new
            for v, new in held if jacobi else ():
                self.L[v["pairs"]] += new - v["m"]
                v["m"] = new

    def read(self, most):
        lin = torch.cat(self.order)
        b = torch.stack([lin // (self.nb[1] * self.nb[2]), lin // self.nb[2] % self.nb[1], lin % self.nb[2]], 1)
        e = torch.arange(8, device="cuda")
        local = torch.stack(torch.meshgrid(e, e, e, indexing="ij"), -1).reshape(1, 512, 3)
        at = self.voxel((8 * b[:, None] + local).permute(2, 0, 1))
        rows = [(8.0 * b + 4.0).double(), self.L[at]]
        c, lo = (torch.cat([r, r.new_zeros(most - len(r), r.shape[1])]) for r in rows)
        return dict(centres=c, logodds=lo)

    def look(self, view, belief, render):
        """The log-likelihood image of a view in a belief field, or the depth it expects."""
        d, mult = view["depth"].reshape(-1), self.rays(view)[2]
        o = self.rays(view)[0].double()
        P = [float(x) for x in np.asarray(view["pose"], np.float32).reshape(-1)]
        D = d.double()
        A, V = torch.zeros_like(D), torch.ones_like(D)
        total, prev = torch.zeros_like(D), torch.zeros_like(D)
        cur = torch.full(d.shape, -1, dtype=torch.long, device="cuda")
        opened = torch.zeros_like(d, dtype=torch.bool)
        begun = opened.clone()

        def density(s):
            s6 = 3.0 * (self.sigma[0] + self.sigma[1] * s + self.sigma[2] * s * s)
            return 0.398942 / s6 * torch.exp(-0.5 * ((D - s) / s6) ** 2)

        for v, l, tin, te, alive in self.walk(view):
            lin = self.brick(v, alive)
            opened = opened & (lin == cur)
            cur = lin
            here = alive & self.active[lin.clamp(min=0)]
            prev = torch.where(here & ~begun, (tin * mult).double(), prev)
            begun, opened = begun | here, opened | here
            p = torch.where(here, belief[self.voxel(v)], 0.0)
            dA = torch.log1p(-p) * torch.where(here, l, torch.zeros_like(l)).double()
            A = A + dA
            w, V = -V * torch.expm1(dA), torch.exp(A)
            if render:
                c = v.double() - o
                total = total + w * ((c[0] * P[2] + c[1] * P[6]) + c[2] * P[10]).abs() * float(self.res)
                continue
            s = te * mult
            near = (s - d).abs() <= 3.0 * self.poly(s)
            s = s.double()
            pz = torch.where(near, (1 - RETURN) * 0.5 * (density(s) + density(prev)), RETURN)
            total = total + torch.where(here & (te * mult >= 0.1), w * pz, 0.0)
            prev = torch.where(here, s, prev)
        if render:
            return total / (1 - V + FREE)
        total = total + V * torch.where(D >= NO_RETURN, 1 - RETURN, RETURN)
        return torch.where(d > 0, torch.log(total), 0.0)


def _exact_net(case, seed):
    feat, target, weight = _bricks_input(case, seed)
    P = torch.from_numpy(np.fromfile(warmstart.DEFAULT_WEIGHTS, dtype=np.float32)).cuda()
    x = P.double().requires_grad_(case["kind"] == "train")
    at, layers = 0, []
    for ci, co in ((4, 16), (16, 16), (16, 1)):
        w, at = x[at:at + 27 * ci * co].reshape(3, 3, 3, ci, co).permute(4, 3, 0, 1, 2), at + 27 * ci * co
        layers.append((w, x[at:at + co]))
        at += co
    n = case["bricks"]
    out = []
    for k in range(0, n, 1024):
        h = feat[k:k + 1024].double().reshape(-1, 8, 8, 8, 4).permute(0, 4, 1, 2, 3)
        for i, (w, b) in enumerate(layers):
            h = torch.nn.functional.conv3d(h, w, b, padding=1)
            h = torch.relu(h) if i < 2 else h
        y = h.reshape(-1, 512)
        if case["kind"] == "train":
            loss = (weight[k:k + 1024].double() * (y - target[k:k + 1024].double()) ** 2).sum() / float(weight.sum())
            loss.backward(retain_graph=True)
            y = loss.detach()
        out.append(y)
    if case["kind"] == "predict":
        return torch.cat(out)
    g = x.grad
    return dict(loss=torch.stack(out).sum().reshape(1), grads=g, params=x.detach() - 1e-3 * g / (g.abs() + 1e-8))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("predict", "train"):
        return _exact_net(case, seed)
    if kind in ("score", "render"):
        if case["field"] != "loaded" or case.get("mode"):
            return None
        p, view, points, occ = _field(case, seed)
        e = _Exact(p)
        flags = torch.zeros_like(e.active)
        e.mark(flags, points)
        e.commit(flags)
        belief = torch.zeros_like(e.L)
        belief[e.voxel(points.floor().T)] = occ.double()
        if kind == "render":
            return dict(image=e.look(view, belief, True).reshape(p.rows, p.cols), score=None, counts=None)
        image = e.look(view, belief, False)
        return dict(image=image.reshape(p.rows, p.cols), sum=image.sum().reshape(1))
    n = case.get("frames") or case["views"] * max(1, case.get("scenes", 0))
    steps = 1.6 * 8.0 / case["res"]
    if n * case["rows"] * case["cols"] * steps / (8 if case.get("scenes") else 1) > 1.2e9 or n * steps > 12000:
        return None  # over 20 seconds
    p, views = _views(case, seed)
    e = _Exact(p)
    if kind == "stream":
        for k, v in enumerate(views):
            e.activate(v, True)
            e.trace(v)
            if k >= case["window"]:
                views[k - case["window"]] = None
            e.infer([w for w in views[:k + 1] if w is not None], case["iters"])
    else:
        for v in views:
            e.activate(v, case.get("full_ray", True))
        for v in views:
            e.trace(v)
        e.infer(views, case["iters"], jacobi=bool(case.get("scenes")))
    return e.read(_most_bricks(case, p))
