"""Workloads of the hybrid kd-tree Gaussian ray tracer, through its public entry points.

Each case names one kind of use (``KINDS``) with its sizes.  Scenes follow
the two distributions of the render benchmark (``uniform``: 100k Gaussians in
the unit cube; ``cluster``: 1M Gaussians in anisotropic clusters plus a shell
with a heavy tail of needle-like ones); the frames run from 256x256 to
1920x1080, with odd sizes among the drawn ones.

``exact`` is a float64 restatement of the rendering equations in torch (ray
set-up, kd-tree walk, max-response test, front-to-back compositing, mirror
and glass bounces), written from the formulas and sharing nothing with the
library but the inputs: the records and the tree that the library built.
"""
import importlib
import math

import numpy as np
import torch

_PKG = "3dgrt_kdtree_gb300"
RESOLUTIONS = ((256, 256), (640, 480), (1280, 720), (1920, 1080))

KINDS = ("plain", "fast", "batch", "packed", "hybrid", "trace", "build", "open", "serve")


def listed():
    return [
        # the drop-in call on a preview frame, with the alpha and depth planes a compositor asks for
        {"name": "plain_256", "kind": "plain", "scene": "uniform", "n": 100_000, "w": 256, "h": 256, "planes": True},
        # the drop-in call at the headline size: the 1M-Gaussian scene, one full-HD frame
        {"name": "plain_1080p", "kind": "plain", "scene": "cluster", "n": 1_000_000, "w": 1920, "h": 1080,
         "planes": False},
        # the smallest call: a thumbnail of a small scene through the one-view fast call
        {"name": "fast_thumb", "kind": "fast", "scene": "uniform", "n": 5_000, "w": 161, "h": 99, "planes": True},
        # an interactive viewer: one VGA frame of a mid-size scene per call
        {"name": "fast_vga", "kind": "fast", "scene": "cluster", "n": 100_000, "w": 640, "h": 480, "planes": False},
        # the headline frame in the batching form
        {"name": "batch_1080p", "kind": "batch", "scene": "cluster", "n": 1_000_000, "views": 1, "w": 1920, "h": 1080},
        # a dataset render: 16 views at four resolutions, one call (w = 0: the mixed resolutions)
        {"name": "batch_mixed", "kind": "batch", "scene": "cluster", "n": 300_000, "views": 16, "w": 0, "h": 0},
        # the capacity form (BF16 / FP16 arrays), four full-HD views
        {"name": "packed_4x1080p", "kind": "packed", "scene": "cluster", "n": 300_000, "views": 4, "w": 1920,
         "h": 1080},
        # secondary rays: two spheres (glass, mirror) and a mirror mesh of 320 triangles
        {"name": "hybrid_720p", "kind": "hybrid", "scene": "cluster", "n": 100_000, "w": 1280, "h": 720, "tris": 320},
        # a burst of twelve one-view VGA requests to the serving loop, frames into page-locked host memory
        {"name": "serve_12", "kind": "serve", "scene": "cluster", "n": 100_000, "w": 640, "h": 480, "requests": 12},
        # a tree for a small object and for a capture
        {"name": "build_10k", "kind": "build", "scene": "uniform", "n": 10_000},
        {"name": "build_500k", "kind": "build", "scene": "cluster", "n": 500_000},
        # a capture opened (upload of both default forms) and its first preview frame drawn
        {"name": "open_200k", "kind": "open", "scene": "cluster", "n": 200_000, "w": 256, "h": 256},
        # the debug counters (render_trace, the plain kernel with counters) are left to draw()
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def frame(lo=8_000, hi=1_000_000):
        pixels, ratio = logint(lo, hi), rng.uniform(0.75, 1.9)
        w = max(16, int(math.sqrt(pixels * ratio)))
        return w, max(16, pixels // w)

    kind = rng.choice(KINDS)
    scene = rng.choice(("uniform", "cluster"))
    n = logint(3_000, 200_000)
    w, h = frame()
    if kind in ("plain", "fast"):
        return {"kind": kind, "scene": scene, "n": n, "w": w, "h": h, "planes": rng.random() < 0.5}
    if kind in ("batch", "packed"):
        w, h = frame(8_000, 500_000)
        return {"kind": kind, "scene": scene, "n": n, "views": rng.randint(1, 9), "w": w, "h": h}
    if kind == "hybrid":
        w, h = frame(8_000, 500_000)
        return {"kind": kind, "scene": scene, "n": n, "w": w, "h": h, "tris": rng.choice((0, 2, 20, 80, 320))}
    if kind == "trace":
        w, h = frame(8_000, 300_000)
        return {"kind": kind, "scene": scene, "n": n, "w": w, "h": h}
    if kind == "build":
        # above 30k the unit cube's Gaussians overlap so much that its tree is all duplicates
        return {"kind": kind, "scene": scene, "n": logint(3_000, 300_000 if scene == "cluster" else 30_000)}
    if kind == "open":
        w, h = frame(8_000, 100_000)
        return {"kind": kind, "scene": scene, "n": n, "w": w, "h": h}
    w, h = frame(8_000, 200_000)
    return {"kind": "serve", "scene": scene, "n": logint(3_000, 100_000), "w": w, "h": h, "requests": rng.randint(3, 12)}


# ------------------------------------------------------------------ inputs
def _lib():
    p = importlib.import_module(_PKG)
    return p.renderer, p.kdtree, p.scenes


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _records(scene, n, seed):
    """(n, 64) float32 activated records on the device (the library's record
    layout: position, opacity, scale, k_scale, quaternion w x y z, SH)."""
    g = torch.Generator(device=_dev()).manual_seed(seed * 7919 + 17)

    def normal(*s):
        return torch.randn(*s, generator=g, device=_dev())

    def uniform(lo, hi, *s):
        return torch.rand(*s, generator=g, device=_dev()) * (hi - lo) + lo

    rec = torch.zeros(n, 64, device=_dev())
    if scene == "uniform":
        rec[:, 0:3] = uniform(-0.5, 0.5, n, 3)
        log_scale = normal(n, 3) * 0.5 + math.log(0.01)
        logit = normal(n)
    else:
        k, n_shell = 64, n // 5
        centres, axes = uniform(-1, 1, k, 3), uniform(0.02, 0.2, k, 3)
        rot = torch.linalg.qr(normal(k, 3, 3).cpu())[0].to(rec.device)
        cid = torch.randint(0, k, (n,), generator=g, device=_dev())
        pos = centres[cid] + ((normal(n, 3) * axes[cid])[:, None, :] * rot[cid]).sum(2)
        shell = torch.nn.functional.normalize(normal(n, 3), dim=1) * (1.5 + 0.01 * normal(n, 1))
        on_shell = (torch.arange(n, device=_dev()) * n_shell // n) != ((torch.arange(n, device=_dev()) + 1) * n_shell // n)
        rec[:, 0:3] = torch.where(on_shell[:, None], shell, pos)
        log_scale = normal(n, 3) * 0.7 + math.log(0.005)
        half = 0.5 * math.log(10.0) * uniform(2.0, 3.4, n) * (uniform(0, 1, n) < 0.05)
        log_scale[:, 0] += half
        log_scale[:, 2] -= half
        logit = normal(n) * 1.2 + 0.5
    rec[:, 3] = torch.sigmoid(logit)
    rec[:, 4:7] = torch.exp(log_scale)
    rec[:, 7] = 1.0
    rec[:, 8:12] = torch.nn.functional.normalize(normal(n, 4), dim=1)
    rec[:, 12:15] = normal(n, 3) * 0.2 + 0.5
    rec[:, 15:60] = normal(n, 45) * 0.05
    return rec


def _cameras(case, seed):
    """[(camera, w, h)] of a case: eyes around the scene, looking near its middle."""
    _, _, scenes = _lib()
    rng = np.random.default_rng(seed * 31 + 5)
    count = case.get("views", case.get("requests", 1))
    out = []
    for i in range(count):
        w, h = (case["w"], case["h"]) if case["w"] else RESOLUTIONS[i * len(RESOLUTIONS) // count]
        d = rng.normal(size=3) * (1.0, 0.4, 1.0)
        d /= np.linalg.norm(d)
        r = rng.uniform(1.3, 2.2) if case["scene"] == "uniform" else rng.uniform(2.0, 3.5)
        cam = scenes.look_at(d * r, target=rng.uniform(-0.1, 0.1, 3), fovy=60.0, aspect=w / h)
        out.append((cam, w, h))
    return out


def _mesh(count, seed):
    """(count, 9) float32 triangles: 0, a quad, or an icosphere of 20 * 4^k."""
    if count == 0:
        return np.zeros((0, 9), np.float32)
    if count == 2:
        a, b, c, d = (-0.9, -0.9, -0.6), (0.9, -0.9, -0.6), (0.9, 0.9, -0.6), (-0.9, 0.9, -0.6)
        return np.array([a + b + c, a + c + d], np.float32)
    p = (1 + 5 ** 0.5) / 2
    v = [(-1, p, 0), (1, p, 0), (-1, -p, 0), (1, -p, 0), (0, -1, p), (0, 1, p), (0, -1, -p), (0, 1, -p), (p, 0, -1),
         (p, 0, 1), (-p, 0, -1), (-p, 0, 1)]
    f = [(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (1, 5, 9), (5, 11, 4), (11, 10, 2), (10, 7, 6),
         (7, 1, 8), (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5), (2, 4, 11), (6, 2, 10), (8, 6, 7),
         (9, 8, 1)]
    t = np.array(v, np.float64)[np.array(f)]
    while len(t) < count:
        a, b, c = t[:, 0], t[:, 1], t[:, 2]
        ab, bc, ca = (a + b) / 2, (b + c) / 2, (c + a) / 2
        t = np.concatenate([np.stack(x, 1) for x in ((a, ab, ca), (ab, b, bc), (ca, bc, c), (ab, bc, ca))])
    t /= np.linalg.norm(t, axis=2, keepdims=True)
    at = np.random.default_rng(seed * 13 + 3).uniform(-0.3, 0.3, 3)
    return (t * 0.35 + at).reshape(-1, 9).astype(np.float32)


def _scene_inputs(case, seed):
    """Records on the device, as the caller's host array, and their tree."""
    _, kdtree, _ = _lib()
    rec = _records(case["scene"], case["n"], seed)
    host = rec.cpu().numpy()
    return rec, host, kdtree.build(host, device="cuda" if rec.is_cuda else "cpu")


def _planes(pixels, extra):
    return [torch.zeros(pixels * 3, device=_dev())] + [torch.zeros(pixels, device=_dev()) for _ in range(extra)]


def prepare(case, seed):
    F, _, _ = _lib()
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "build":
        # the caller's arrays for any tree of this many Gaussians (other seeds give other sizes)
        s["host"] = _records(case["scene"], case["n"], seed).cpu().numpy()
        s["nodes"] = np.zeros(16 * case["n"], np.int32)
        s["offsets"] = np.zeros(64 * case["n"], np.int32)
        return s
    rec, host, tree = _scene_inputs(case, seed)
    cams = s["cams"] = _cameras(case, seed)
    if kind == "open":
        s["rec"], s["tree"], s["out"] = rec, tree, _planes(case["w"] * case["h"], 0)
        return s
    if kind == "serve":
        s["server"] = F.Server(hbm_budget_bytes=8 << 30, arena_bytes=64 << 20)
        s["slot"] = s["server"].add_scene(tree, host)
        s["requests"] = [F.make_views([c])[0] for c in cams]
        s["out"] = [torch.zeros(w * h * 3).pin_memory() for _, w, h in cams]
        return s
    forms = {"plain": F.FORM_EXACT, "trace": F.FORM_EXACT, "hybrid": F.FORM_EXACT, "fast": F.FORM_FAST,
             "batch": F.FORM_FAST, "packed": F.FORM_PACKED}[kind]
    s["scene"] = F.Scene.from_device(tree, rec, forms=forms)
    if kind in ("batch", "packed"):
        s["views"], pixels, _ = F.make_views(cams)
        s["out"] = _planes(pixels, 2)
        s["cfg"] = None
        if kind == "packed":
            s["cfg"] = F.BatchConfig.default()
            s["cfg"].precision = 1
        return s
    _, w, h = cams[0]
    if kind == "trace":
        s["out"] = _planes(w * h, 2) + [torch.zeros(w * h * 56, dtype=torch.uint8, device=_dev())]
    else:
        s["out"] = _planes(w * h, 2 if case.get("planes") else 0)
    if kind == "hybrid":
        s["secondary"] = F.Secondary(F.demo_spheres(), _mesh(case["tris"], seed), F.mesh_material_default())
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "build":
        _, kdtree, _ = _lib()
        t = kdtree.build(s["host"], device="cuda")
        s["nodes"][:t.nodes.size] = t.nodes.reshape(-1).view(np.int32)
        s["offsets"][:t.offsets.size] = t.offsets.view(np.int32)
        return {"nodes": s["nodes"], "offsets": s["offsets"], "aabb": t.aabb, "valid": t.valid,
                "sizes": np.array([t.n_nodes, t.offsets.size, t.depth, t.n_leaves, t.max_leaf])}
    cam, w, h = s["cams"][0]
    if kind == "open":
        F, _, _ = _lib()
        scene = F.Scene.from_device(s["tree"], s["rec"])
        scene.render_fast(cam, w, h, s["out"][0])
        scene.close()
        return s["out"]
    if kind == "serve":
        tickets = [s["server"].submit(s["slot"], v, 1, o) for v, o in zip(s["requests"], s["out"])]
        for t in tickets:
            status, _ = s["server"].wait(t)
            if status != 0:
                raise RuntimeError("request ended with status %d" % status)
        return s["out"]
    out = s["out"]
    if kind == "plain":
        s["scene"].render(cam, w, h, *out)
    elif kind == "fast":
        s["scene"].render_fast(cam, w, h, *out)
    elif kind == "hybrid":
        s["scene"].render_hybrid(cam, w, h, s["secondary"], out[0])
    elif kind == "trace":
        s["scene"].render_trace(cam, w, h, out[0], out[1], out[2], out[3])
    else:
        s["scene"].render_batch(s["views"], len(s["cams"]), out[0], out[1], out[2], cfg=s["cfg"])
    return out


def _rays(case):
    if case["kind"] == "build":
        return 0
    count = case.get("views", case.get("requests", 1))
    sizes = [(case["w"], case["h"]) if case["w"] else RESOLUTIONS[i * len(RESOLUTIONS) // count] for i in range(count)]
    return sum(w * h for w, h in sizes)


def work(case):
    """Bytes read and written once and arithmetic of one pass.  A tree of
    these scenes has about 2 nodes (8 B) and 25 leaf IDs (4 B) per Gaussian;
    a ray meets about 80 nodes, 20 accepted hits (60 operations each to test)
    and 11 composited ones (160 with their degree-3 colour)."""
    n, rays, kind = case["n"], _rays(case), case["kind"]
    tree = n * (2 * 8 + 25 * 4)
    if kind == "build":
        # position, scale, opacity and quaternion in, the tree out; one SAH
        # score (about 40 operations) for each of some 60 edges per level
        return {"bytes": 44 * n + tree, "flops": 60.0 * 40 * 24 * n}
    flops = rays * (80 * 4 + 20 * 60 + 11 * 160.0)
    planes = {"trace": 76, "batch": 20, "packed": 20}.get(kind, 20 if case.get("planes") else 12)
    if kind == "open":
        # records and tree in, the plain and fast forms' arrays out
        return {"bytes": 256 * n + tree + n * (64 + 192 + 4) + tree + 25 * n * 48 + 12 * rays, "flops": flops + 300.0 * n}
    seen = min(256 * n + tree, rays * 14_000)  # a frame cannot read more than its rays meet
    return {"bytes": seen + planes * rays, "flops": flops}


# ------------------------------------------------------------------ float64
_SH = [0.28209479177387814, 0.4886025119029199, 1.0925484305920792, 0.31539156525252005, 0.5462742152960396,
       0.5900435899266435, 2.890611442640554, 0.4570457994644658, 0.3731763325901154, 1.445305721320277]


def _basis(d):
    """(m, 16) real spherical harmonics of bands 0 to 3 at unit directions d."""
    x, y, z = d.unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    c = _SH
    return torch.stack([
        torch.full_like(x, c[0]), -c[1] * y, c[1] * z, -c[1] * x, c[2] * x * y, -c[2] * y * z,
        c[3] * (2 * zz - xx - yy), -c[2] * x * z, c[4] * (xx - yy), -c[5] * y * (3 * xx - yy), c[6] * x * y * z,
        -c[7] * y * (4 * zz - xx - yy), c[8] * z * (2 * zz - 3 * xx - 3 * yy), -c[7] * x * (4 * zz - xx - yy),
        c[9] * z * (xx - yy), -c[5] * x * (xx - 3 * yy)], 1)


class _Exact:
    """The scene in float64: tree arrays, M = diag(1/s) R^T and mu per Gaussian."""

    def __init__(self, rec, tree):
        f = torch.float64
        dev = rec.device
        nodes = torch.from_numpy(tree.nodes.astype(np.int64)).to(dev)
        self.leaf = (nodes[:, 0] & 7) == 3
        self.hi = nodes[:, 0] >> 3
        self.axis = nodes[:, 0] & 3
        self.lo = nodes[:, 1]
        self.split = torch.from_numpy(np.ascontiguousarray(tree.nodes[:, 1]).view(np.float32).astype(np.float64)).to(dev)
        self.ids = torch.from_numpy(tree.offsets.astype(np.int64)).to(dev)
        self.box = torch.from_numpy(tree.aabb.astype(np.float64)).to(dev)
        self.mu, self.opacity = rec[:, 0:3].to(f), rec[:, 3].to(f)
        w, x, y, z = rec[:, 8:12].to(f).unbind(1)
        rt = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y + w * z), 2 * (x * z - w * y),
                          2 * (x * y - w * z), 1 - 2 * (x * x + z * z), 2 * (y * z + w * x),
                          2 * (x * z + w * y), 2 * (y * z - w * x), 1 - 2 * (x * x + y * y)], 1).view(-1, 3, 3)
        self.m = rt / rec[:, 4:7].to(f)[:, :, None]
        self.sh = rec[:, 12:60]

    def colour(self, gid, basis):
        sh = self.sh[gid].to(torch.float64)
        rest = sh[:, 3:].view(-1, 3, 15)
        c = basis[:, :1] * sh[:, :3] + (rest * basis[:, None, 1:]).sum(2) + 0.5
        return c.clamp_min(0.0)

    def blend(self, ray, gid, t, gray, basis, acc):
        """Composite hits (sorted by ray, then t) front to back into acc
        (r, g, b, opacity, depth); a ray stops once its opacity passes 0.99."""
        first = torch.ones_like(ray, dtype=torch.bool)
        first[1:] = ray[1:] != ray[:-1]
        at = torch.arange(ray.numel(), device=ray.device)
        rank = at - torch.cummax(torch.where(first, at, 0), 0)[0]
        resp = torch.exp(-0.0555555555556 * gray * gray)
        alpha = torch.clamp_max(self.opacity[gid] * resp, 0.99)
        keep = (resp >= 0.0113) & (alpha >= 1.0 / 255.0)
        for k in range(int(rank.max()) + 1 if rank.numel() else 0):
            sel = torch.nonzero(keep & (rank == k))[:, 0]
            sel = sel[acc[ray[sel], 3] <= 0.99]
            r, w = ray[sel], alpha[sel] * (1 - acc[ray[sel], 3])
            add = torch.cat([self.colour(gid[sel], basis[r]) * w[:, None], w[:, None], (t[sel] * w)[:, None]], 1)
            acc[r] += add

    def trace(self, o, d, max_t, acc):
        """Walk the tree front to back for rays (o, d) up to max_t, adding to acc in place."""
        inv = 1.0 / d
        a, b = (self.box[:3] - o) * inv, (self.box[3:] - o) * inv
        near = torch.minimum(a, b).amax(1).clamp_min(float(np.float32(1e-2)))
        far = torch.maximum(a, b).amin(1)
        live = (far >= near) & (far >= 0)
        far = torch.minimum(far, max_t)
        live &= (near <= far) & (acc[:, 3] < 0.99)
        ray = torch.nonzero(live)[:, 0]  # rays on the way, compacted as they end
        basis = _basis(d)
        near, far, end = near[ray], far[ray], far[ray]
        cur = torch.zeros_like(ray)
        sp = torch.zeros_like(ray)
        depth = 40
        st_id = torch.zeros(ray.numel(), depth, dtype=torch.int64, device=ray.device)
        st_t = torch.zeros(ray.numel(), depth, dtype=torch.float64, device=ray.device)
        while ray.numel():
            inner = torch.nonzero(~self.leaf[cur])[:, 0]
            while inner.numel():
                c, ax, r = cur[inner], self.axis[cur[inner]], ray[inner]
                iv = inv[r].gather(1, ax[:, None])[:, 0]
                ts = (self.split[c] - o[r].gather(1, ax[:, None])[:, 0]) * iv
                neg = torch.signbit(iv).long()
                child, nr, fr = self.hi[c], near[inner], far[inner]
                both = (nr < ts) & (ts < fr)
                b = inner[both]
                st_id[b, sp[b]] = (child + (neg ^ 1))[both]
                st_t[b, sp[b]] = fr[both]
                sp[b] += 1
                far[b] = ts[both]
                cur[inner] = child + (neg ^ (ts <= nr).long())
                inner = inner[~self.leaf[cur[inner]]]
            # every (ray, candidate) of the leaves, and the accepted ones in (ray, t) order
            count = self.hi[cur]
            who = torch.repeat_interleave(torch.arange(ray.numel(), device=ray.device), count)
            start = torch.cumsum(count, 0) - count
            gid = self.ids[self.lo[cur][who] + torch.arange(who.numel(), device=ray.device) - start[who]]
            hits = []
            for k in range(0, who.numel(), 4_000_000):
                w, g = who[k:k + 4_000_000], gid[k:k + 4_000_000]
                r, m = ray[w], self.m[g]
                gd = (m * d[r][:, None, :]).sum(2)
                ng = (m * (self.mu[g] - o[r])[:, None, :]).sum(2)
                q = (gd * gd).sum(1)
                t = (gd * ng).sum(1) / q
                gray = torch.linalg.cross(gd, ng).square().sum(1) / q
                ok = torch.nonzero((t >= near[w]) & (t < far[w]) & (gray < 8))[:, 0]
                hits.append((w[ok], g[ok], t[ok], gray[ok]))
            if hits:
                w, g, t, gray = (torch.cat(x) for x in zip(*hits))
                by_t = torch.sort(t, stable=True)[1]
                order = by_t[torch.sort(w[by_t], stable=True)[1]]
                self.blend(ray[w[order]], g[order], t[order], gray[order], basis, acc)
            go = torch.nonzero((acc[ray, 3] < 0.99) & (far < end) & (sp > 0))[:, 0]
            ray, end, near, sp, st_id, st_t = ray[go], end[go], far[go], sp[go] - 1, st_id[go], st_t[go]
            cur = st_id.gather(1, sp[:, None])[:, 0]
            far = st_t.gather(1, sp[:, None])[:, 0]


def _primary(cam, w, h, dev):
    """(origins, directions) of a frame in image rows from the bottom up, the output order."""
    f = torch.float64
    pos, u, v, n = (torch.tensor([float(np.float32(x)) for x in a], dtype=f, device=dev)
                    for a in (cam.pos, cam.uaxis, cam.vaxis, cam.naxis))
    height = 2 * cam.near_c * math.tan(cam.fovy * math.pi / 360.0)
    width = height * cam.aspect
    start = pos - n * cam.near_c - u * (width / 2) + v * (height / 2)
    y = torch.arange(h - 1, -1, -1, dtype=f, device=dev).repeat_interleave(w) + 0.5
    x = torch.arange(w, dtype=f, device=dev).repeat(h) + 0.5
    d = start + u * (x * (width / w))[:, None] - v * (y * (height / h))[:, None] - pos
    return pos.expand_as(d).contiguous(), torch.nn.functional.normalize(d, dim=1)


def _closest(o, d, spheres, tris, mirror):
    """Closest secondary primitive of every ray: t (1e8: none), normal, front side, material row."""
    t = torch.full((o.shape[0],), 1e8, dtype=torch.float64, device=o.device)
    n = torch.zeros_like(o)
    mat = torch.zeros(o.shape[0], 6, dtype=torch.float64, device=o.device)
    for centre, radius, m in spheres:
        oc = o - centre
        b, c = 2 * (oc * d).sum(1), (oc * oc).sum(1) - radius * radius
        disc = b * b - 4 * c
        sq = disc.clamp_min(0).sqrt()
        root = torch.where((-b - sq) / 2 < 1e-5, (-b + sq) / 2, (-b - sq) / 2)
        hit = (disc >= 0) & (root > 1e-5) & (root < t)
        t = torch.where(hit, root, t)
        n = torch.where(hit[:, None], (o + d * root[:, None] - centre) / radius, n)
        mat = torch.where(hit[:, None], m, mat)
    for v0, v1, v2 in tris:
        e1, e2 = v1 - v0, v2 - v0
        hv = torch.linalg.cross(d, e2.expand_as(d))
        a = (hv * e1).sum(1)
        s = o - v0
        u = (s * hv).sum(1) / a
        q = torch.linalg.cross(s, e1.expand_as(s))
        v = (d * q).sum(1) / a
        tt = (q * e2).sum(1) / a
        hit = (a.abs() >= 1e-5) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (tt > 1e-5) & (tt < t)
        t = torch.where(hit, tt, t)
        n = torch.where(hit[:, None], torch.nn.functional.normalize(torch.linalg.cross(e1, e2), dim=0), n)
        mat = torch.where(hit[:, None], mirror, mat)
    front = (d * n).sum(1) <= 0
    return t, torch.where(front[:, None], n, -n), front, mat


def _exact_hybrid(E, cam, w, h, spheres, tris, mirror):
    o, d = _primary(cam, w, h, E.mu.device)
    fin = torch.zeros_like(o)
    through = torch.ones_like(o)
    acc = torch.zeros(o.shape[0], 5, dtype=torch.float64, device=o.device)
    at = torch.arange(o.shape[0], device=o.device)
    for bounce in range(5):
        t, n, front, mat = _closest(o, d, spheres, tris, mirror)
        part = acc[at]
        E.trace(o, d, t, part)
        acc[at] = part
        thr = through[at]
        f = fin[at] + thr * part[:, :3]
        thr = thr * (1 - part[:, 3:4])
        kind = mat[:, 0]
        go = (t < 1e8) & ~(thr < 0.01).all(1)
        mirrored, glass = go & (kind == 1), go & (kind == 2)
        solid = go & (kind == 0)
        p, cos = o + d * t[:, None], -(n * d).sum(1)
        refl = torch.nn.functional.normalize(d + 2 * n * cos[:, None], dim=1)
        eta = torch.where(front, 1 / mat[:, 2].clamp_min(1e-30), mat[:, 2])
        sin2 = eta * eta * (1 - cos * cos)
        bent = d * eta[:, None] + n * (eta * cos - (1 - sin2).clamp_min(0).sqrt())[:, None]
        inside = glass & (sin2 <= 1)
        f = f + torch.where(solid[:, None], thr * mat[:, 3:], 0.0)
        if bounce == 0:
            f = f + torch.where(mirrored[:, None], thr * (1 - mat[:, 1:2]) * mat[:, 3:], 0.0)
        thr = torch.where(mirrored[:, None], thr * mat[:, 1:2], torch.where(glass[:, None], thr * mat[:, 3:], thr))
        o = torch.where(inside[:, None], p - n * 1e-4, p + n * 1e-4)
        d = torch.where(inside[:, None], torch.nn.functional.normalize(bent, dim=1), refl)
        fin[at], through[at] = f, thr
        keep = mirrored | glass
        at, o, d = at[keep], o[keep], d[keep]
        if not at.numel():
            break
    return fin.clamp_max(1.0).reshape(-1)


def exact(case, seed):
    """What run() returns, in float64; None for trees (whole numbers) and for
    frames of more than 2.5M rays, which take longer than the timed work."""
    kind = case["kind"]
    if kind == "build" or _rays(case) > 2_500_000:
        return None
    F, _, _ = _lib()
    rec, _, tree = _scene_inputs(case, seed)
    E = _Exact(rec, tree)
    cams = _cameras(case, seed)
    if kind == "hybrid":
        def row(m):
            return torch.tensor([m.material, m.reflectivity, m.ior, *m.color], dtype=torch.float64, device=rec.device)

        spheres = [(torch.tensor(list(s.center), dtype=torch.float64, device=rec.device), float(s.radius),
                    row(s.material)) for s in F.demo_spheres()]
        tris = torch.from_numpy(_mesh(case["tris"], seed).astype(np.float64)).to(rec.device).view(-1, 3, 3)
        return [_exact_hybrid(E, *cams[0], spheres, tris, row(F.mesh_material_default()))]
    frames = []
    for cam, w, h in cams:
        o, d = _primary(cam, w, h, rec.device)
        acc = torch.zeros(w * h, 5, dtype=torch.float64, device=rec.device)
        E.trace(o, d, torch.full((w * h,), math.inf, dtype=torch.float64, device=rec.device), acc)
        frames.append(acc)
    if kind == "serve":
        return [a[:, :3].reshape(-1) for a in frames]
    a = torch.cat(frames)
    planes = [a[:, :3].reshape(-1), a[:, 3].contiguous(), a[:, 4].contiguous()]
    if kind in ("batch", "packed"):
        return planes
    if kind == "trace":
        return planes + [None]
    return planes if case.get("planes") else planes[:1]
