"""The renderer's work, as its users' programs call it, for timing.

A case is one call (or one whole render) through the package's public entry
points; `listed()` names the ones that are always timed, `draw()` gives more of
the same ranges.  Scenes are the repository's own procedural ones (the Cornell
box, the displaced icosphere, the mixed-material scene, the sky-lit room, the
batched requests) and a field of spheres; they stand for the model files that a
program has loaded, so a scene depends on its size alone, while cameras, rays,
samples, seeds and network weights come from the case's seed.

Kinds of case:
  hits     closest hits of rays in device memory (`trace_closest_device`)
  hosthits closest hits of rays in numpy arrays (`trace_closest`)
  render   a whole render: initialize, render_until_done, the image read back
  preview  a progressive frame: re_start, a few steps, the image read back
  guided   a whole render with a trained, frozen path-guiding network
  batch    uneven render requests sharing one path pool
  infer    the guiding network over rows of vertices
  train    one training step of the guiding network (gradients, then Adam)
"""
from __future__ import annotations

import math

import numpy as np
import torch

import raccoongpurender_gb300 as rg
from raccoongpurender_gb300 import materials, scenes

FLT_MAX = 3.4028234663852886e38
TAN_22_5 = 0.41421356237309503

# Host scenes with their trees, one per kind and size: a program loads its model once.
_scenes: dict = {}


def listed() -> list:
    return [
        # a mouse pick or a probe of a few hundred rays in a mid-size model: the smallest call
        dict(name="hits_pick", kind="hits", level=5, rays="random", n=1000, reorder=0, normals=1),
        # primary visibility of a 2048 x 2048 camera over 1.31M triangles
        dict(name="hits_camera", kind="hits", level=8, rays="camera", n=2048 * 2048, reorder=0, normals=0),
        # ambient or bounce rays without any order, as a baker casts them
        dict(name="hits_random", kind="hits", level=8, rays="random", n=4_000_001, reorder=0, normals=0),
        # the same rays with the library's sort switched on
        dict(name="hits_random_sorted", kind="hits", level=8, rays="random", n=4_000_001, reorder=1, normals=0),
        # a tool that has its rays in numpy arrays
        dict(name="hits_host", kind="hosthits", level=7, n=1_000_000),
        # the small whole render: thumbnails, unit tests, look-up renders
        dict(name="render_cornell", kind="render", scene="cornell", level=0, w=256, h=256, spp=4, depth=5,
             paths=1 << 18, image="sums"),
        # the final-quality frame: 1.31M triangles, mixed materials, sky, volume
        dict(name="render_mixed_1080p", kind="render", scene="mixed", level=8, w=1920, h=1080, spp=64, depth=8,
             paths=1 << 24, image="color"),
        # an interactive viewer's frame after the camera moved: spheres and sky, a few bounces of a small pool
        dict(name="preview_spheres", kind="preview", scene="spheres", level=0, w=1280, h=720, steps=12,
             paths=1 << 20),
        # the next frame of an animation, guided by the network that earlier frames trained
        dict(name="guided_room", kind="guided", level=4, w=640, h=360, spp=16, depth=8, paths=1 << 21),
        # a render service's queue: requests of 64 to 512 pixels a side, 1 to 32 samples, 1k to 150k triangles
        dict(name="batch_8", kind="batch", requests=8, max_side=512, max_spp=32, max_tris=150_000, paths=1 << 21),
        # the guiding network alone, forward
        dict(name="guide_infer", kind="infer", n=1 << 18),
        # ... and backward: a training step on one batch
        dict(name="guide_train", kind="train", n=1 << 18),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pool(rng, samples: int, most: int) -> int:
    """A resident path pool that goes through `samples` paths in at most 24 fillings."""
    return _log_int(rng, max(1 << 14, samples // 24), most)


def draw(rng) -> dict:
    kind = rng.choice(["hits", "hits", "hosthits", "render", "render", "preview", "guided", "batch", "infer", "train"])
    if kind == "hits":
        return dict(kind=kind, level=rng.randint(3, 8), rays=rng.choice(["camera", "random"]),
                    n=_log_int(rng, 100, 4_000_000), reorder=rng.choice([0, 0, 1]), normals=rng.choice([0, 0, 1]))
    if kind == "hosthits":
        return dict(kind=kind, level=rng.randint(4, 8), n=_log_int(rng, 500, 2_000_000))
    if kind == "render":
        scene = rng.choice(["cornell", "mixed", "room", "spheres"])
        w, h = _log_int(rng, 48, 1920), _log_int(rng, 48, 1080)
        spp = _log_int(rng, 1, max(1, min(64, 60_000_000 // (w * h))))
        return dict(kind=kind, scene=scene, level=rng.randint(4, 8) if scene == "mixed" else 4, w=w, h=h, spp=spp,
                    depth=rng.randint(3, 10), paths=_pool(rng, w * h * spp, 1 << 24),
                    image=rng.choice(["color", "sums"]))
    if kind == "preview":
        scene = rng.choice(["cornell", "mixed", "room", "spheres"])
        return dict(kind=kind, scene=scene, level=rng.randint(4, 7) if scene == "mixed" else 4,
                    w=_log_int(rng, 160, 1920), h=_log_int(rng, 120, 1080), steps=rng.randint(1, 24),
                    paths=_log_int(rng, 1 << 15, 1 << 22))
    if kind == "guided":
        w, h, spp = _log_int(rng, 80, 960), _log_int(rng, 60, 540), _log_int(rng, 2, 24)
        return dict(kind=kind, level=4, w=w, h=h, spp=spp, depth=rng.randint(4, 8),
                    paths=_pool(rng, w * h * spp, 1 << 22))
    if kind == "batch":
        return dict(kind=kind, requests=rng.randint(2, 12), max_side=_log_int(rng, 96, 512),
                    max_spp=_log_int(rng, 2, 32), max_tris=_log_int(rng, 2000, 150_000),
                    paths=_log_int(rng, 1 << 17, 1 << 22))
    return dict(kind=kind, n=_log_int(rng, 100, 1 << 20))


# ------------------------------------------------------------------ scenes
def _sphere_field():
    """600 spheres of the full-render material mix on a ground quad, under the sky."""
    rng = np.random.default_rng(17)
    r = rng.uniform(0.05, 0.3, 600)
    p = np.stack([rng.uniform(-5, 5, 600), r - 1.2, rng.uniform(-5, 5, 600), r], 1).astype(np.float32)
    gp = np.array([[-12, -1.2, -12], [12, -1.2, -12], [12, -1.2, 12], [-12, -1.2, 12]], np.float32)
    gi = scenes.orient(gp, np.array([[0, 1, 2], [0, 2, 3]], np.uint32), np.array([0, -5, 0], np.float32), True)
    return gp, gi, p, materials.random_mix(600, rng)


def _scene(kind: str, level: int):
    """(SceneManager with its tree, camera dict, triangles) of one size."""
    key = (kind, level)
    if key not in _scenes:
        sm = rg.SceneManager()
        if kind == "sphere":
            mesh = scenes.displaced_icosphere(level)
            sm.addPolymesh(mesh.points, mesh.indices, np.repeat(materials.as_array(mesh.materials[:1]), mesh.ntris))
            cam = None
            lo, hi = mesh.points.min(0), mesh.points.max(0)
            extra = (mesh.points, mesh.indices, lo, hi)
        elif kind == "cornell":
            mesh, cam, extra = scenes.cornell_box(), scenes.cornell_camera(), None
            sm.addMesh(mesh)
        elif kind == "spheres":
            gp, gi, sp, mats = _sphere_field()
            sm.addPolymesh(gp, gi, [materials.lambertian(r=(0.6, 0.6, 0.6))] * len(gi))
            sm.addSpheres(sp, mats)
            sm.setEnvmap(scenes.sky_envmap(512, 256))
            cam, extra = dict(eye=(0.0, 1.2, 6.5), target=(0.0, -0.8, 0.0), up=(0.0, 1.0, 0.0), vfov=45.0), None
        else:
            mesh, env, cam = scenes.mixed_scene(level) if kind == "mixed" else scenes.sky_room(level)
            extra = None
            sm.addMesh(mesh)
            sm.setEnvmap(env)
        sm.buildBVH()
        _scenes[key] = (sm, cam, extra)
    return _scenes[key]


def _batch(case):
    """The requests of the batched workload, scaled: (SceneManager, camera dict, spp) each."""
    key = ("batch", case["requests"], case["max_side"], case["max_spp"], case["max_tris"])
    if key not in _scenes:
        rng = np.random.default_rng(21)
        out, env = [], scenes.sky_envmap(512, 256)
        for i in range(case["requests"]):
            side = int(round(math.exp(rng.uniform(math.log(64), math.log(case["max_side"])))))
            spp = int(round(math.exp(rng.uniform(0.0, math.log(case["max_spp"])))))
            tris = int(round(math.exp(rng.uniform(math.log(1000), math.log(case["max_tris"])))))
            mesh, cam = scenes.request_scene(tris, rng, i % 2 == 1)
            sm = rg.SceneManager()
            sm.addMesh(mesh)
            sm.setEnvmap(env)
            sm.buildBVH()
            out.append((sm, dict(cam, w=side, h=side), spp, mesh.ntris))
        _scenes[key] = out
    return _scenes[key]


def _camera(cam: dict, rng, w: int, h: int):
    """The scene's camera, moved a little by the seed."""
    eye = np.asarray(cam["eye"], np.float64) + rng.uniform(-0.04, 0.04, 3)
    return rg.camera_look_at(tuple(eye), cam["target"], cam["up"], cam["vfov"], w, h)


# ------------------------------------------------------------------ inputs
def _unit(g, n: int) -> torch.Tensor:
    v = torch.randn((n, 3), generator=g, device="cuda")
    return v / v.norm(dim=1, keepdim=True).clamp_min(1e-6)


def _rays(case, seed: int):
    """Seven device arrays: origins, directions, far clip."""
    _, _, (_, _, lo, hi) = _scene("sphere", case["level"])
    n = case["n"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case.get("rays") == "camera":
        # pixel-centre rays of a pinhole camera, in raster order, the first n of a square image
        side = int(math.ceil(math.sqrt(n)))
        rng = np.random.default_rng(seed)
        eye = np.array([0.0, 0.35, 3.0]) + rng.uniform(-0.05, 0.05, 3)
        fwd = -eye / np.linalg.norm(eye)
        right = np.cross(fwd, [0.0, 1.0, 0.0])
        right /= np.linalg.norm(right)
        up = np.cross(right, fwd)
        to = lambda v: torch.tensor(v, dtype=torch.float64, device="cuda")  # noqa: E731
        i = torch.arange(n, device="cuda")
        x = (((i % side).double() + 0.5) / side - 0.5) * 2.0 * TAN_22_5
        y = (0.5 - ((i // side).double() + 0.5) / side) * 2.0 * TAN_22_5
        d = to(fwd) + x[:, None] * to(right) + y[:, None] * to(up)
        d = (d / d.norm(dim=1, keepdim=True)).float()
        o = to(eye).float().expand(n, 3)
        tmax = torch.full((n,), FLT_MAX, device="cuda")
    else:
        lo_t, hi_t = torch.tensor(lo, device="cuda"), torch.tensor(hi, device="cuda")
        o = lo_t + (hi_t - lo_t) * torch.rand((n, 3), generator=g, device="cuda")
        d = _unit(g, n)
        tmax = torch.full((n,), 8.0, device="cuda")  # a far clip well outside the model
    return [o[:, k].contiguous() for k in range(3)] + [d[:, k].contiguous() for k in range(3)] + [tmax]


def _weights(seed: int):
    """A network with the magnitudes of a trained one: He-uniform layers, small biases, zero padding."""
    rng = np.random.default_rng(seed)
    w = np.zeros((5, 64, 64), np.float32)
    b = np.zeros((5, 64), np.float32)
    for layer in range(5):
        fi, fo = (36 if layer == 0 else 64), (41 if layer == 4 else 64)
        lim = math.sqrt(6.0 / fi) * (0.5 if layer == 4 else 1.0)
        w[layer, :fi, :fo] = rng.uniform(-lim, lim, (fi, fo))
        b[layer, :fo] = rng.uniform(-0.1, 0.1, fo)
    return w, b


def _samples(n: int, seed: int) -> torch.Tensor:
    """Rows of 16 floats: vertex, normal, outgoing and incident direction, weight, BSDF pdf, two spare."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = torch.zeros((n, 16), device="cuda")
    s[:, 0:3] = torch.rand((n, 3), generator=g, device="cuda") * 2.0 - 1.0
    nrm, wo, wi = _unit(g, n), _unit(g, n), _unit(g, n)
    wo = torch.where((wo * nrm).sum(1, keepdim=True) < 0, -wo, wo)
    s[:, 3:6], s[:, 6:9], s[:, 9:12] = nrm, wo, wi
    s[:, 12] = torch.exp(torch.randn(n, generator=g, device="cuda") - 0.5)  # radiance x cos / pdf: log-normal
    s[:, 13] = (wi * nrm).sum(1).clamp_min(0.0) / math.pi
    return s


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    st = dict(case=case)
    if kind in ("hits", "hosthits"):
        sm, _, _ = _scene("sphere", case["level"])
        lane = rg.WavefrontLane(0, 1 << 12)
        lane.setup(sm)
        rays = _rays(case, seed)
        if kind == "hits":
            n = case["n"]
            lane.set_trace_reorder(case["reorder"])
            st.update(rays=rays, ptrs=[a.data_ptr() for a in rays], stream=torch.cuda.Stream(),
                      prim=torch.empty(n, dtype=torch.int32, device="cuda"), t=torch.empty(n, device="cuda"),
                      ng=torch.empty((n, 3), device="cuda") if case["normals"] else None)
        else:
            st.update(rays=[a.cpu().numpy() for a in rays])
        st.update(lane=lane)
    elif kind in ("render", "preview", "guided"):
        sm, cam, _ = _scene("room" if kind == "guided" else case["scene"], case["level"])
        lane = rg.WavefrontLane(0, case["paths"])
        lane.setup(sm)
        if kind == "guided":
            guide = rg.Guide(0, train=0)
            guide.set_weights(*_weights(seed + 5))
            lane.set_guide(guide)
            st.update(guide=guide)
        kw = dict(seed_offset=int(rng.integers(1, 1 << 31)))
        if kind != "preview":
            kw.update(spp=case["spp"], max_depth=case["depth"])
        st.update(lane=lane, camera=_camera(cam, rng, case["w"], case["h"]), config=rg.render_config(**kw))
    elif kind == "batch":
        b = rg.Batch(0, case["paths"])
        for sm, cam, spp, _ in _batch(case):
            b.add(sm, _camera(cam, rng, cam["w"], cam["h"]),
                  rg.render_config(spp=spp, max_depth=8, seed_offset=int(rng.integers(1, 1 << 31))))
        st.update(batch=b)
    else:
        guide = rg.Guide(0)
        guide.set_weights(*_weights(seed + 5))
        guide.set_bounds((-1, -1, -1), (1, 1, 1))
        n = case["n"]
        st.update(guide=guide, rows=_samples(n, seed), stream=torch.cuda.Stream())
        if kind == "infer":
            st.update(out=torch.empty((n, rg.Guide.ROW_OUTPUTS), device="cuda"))
        else:
            st.update(grads=torch.empty(rg.Guide.N_PARAMS, device="cuda"))
    torch.cuda.synchronize()
    return st


def run(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "hits":
        st["lane"].trace_closest_device(st["ptrs"], case["n"], st["prim"].data_ptr(), st["t"].data_ptr(),
                                        st["ng"].data_ptr() if st["ng"] is not None else 0,
                                        st["stream"].cuda_stream)
        out = dict(prim=st["prim"], t=st["t"])
        if st["ng"] is not None:
            out["ng"] = st["ng"]
        return out
    if kind == "hosthits":
        prim, t = st["lane"].trace_closest(st["rays"])
        return dict(prim=prim, t=t)
    if kind == "preview":
        st["lane"].re_start(st["camera"], st["config"])
        st["lane"].step(case["steps"])
        return dict(color=st["lane"].finalize_color())
    if kind in ("render", "guided"):
        lane = st["lane"]
        lane.initialize(st["camera"], st["config"])
        lane.render_until_done()
        if case.get("image") == "sums":
            return dict(sums=lane.accumulation())
        return dict(color=lane.finalize_color())
    if kind == "batch":
        b = st["batch"]
        b.run(order=rg.ORDER_SHORTEST_FIRST)
        return [b.color(i) for i in range(case["requests"])]
    if kind == "infer":
        st["guide"].infer_device(st["rows"].data_ptr(), case["n"], st["out"].data_ptr(), st["stream"].cuda_stream)
        return dict(out=st["out"])
    loss = st["guide"].train_device(st["rows"].data_ptr(), case["n"], weight_scale=1.0 / case["n"],
                                    grads_ptr=st["grads"].data_ptr(), stream=st["stream"].cuda_stream)
    return dict(loss=loss, grads=st["grads"])


# ------------------------------------------------------------------ work
def _ray_flops(prims: float) -> float:
    """A closest hit: a walk down a binary tree over leaves of about three
    primitives, two boxes a node (18 operations each), four primitive tests (45)."""
    return 1.2 * max(1.0, math.log2(max(2.0, prims / 3.0))) * 36.0 + 4 * 45.0


def _tree_bytes(prims: float) -> float:
    return 48.0 * prims + 64.0 * prims / 3.0


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("hits", "hosthits"):
        n, prims = case["n"], 20 * 4 ** case["level"]
        per = 36 + (12 if case.get("normals") else 0)
        return dict(bytes=per * n + min(_tree_bytes(prims), n * 1700.0), flops=n * _ray_flops(prims))
    if kind in ("render", "preview", "guided"):
        scene = "room" if kind == "guided" else case["scene"]
        prims = dict(cornell=36, spheres=602, room=20 * 4 ** 4, mixed=20 * 4 ** case["level"])[scene]
        npix = case["w"] * case["h"]
        # extension rays: a path has about three segments in these scenes
        rays = case["paths"] * case["steps"] if kind == "preview" else 3.0 * npix * case["spp"]
        per = _ray_flops(prims) + 300.0 + (34304.0 if kind == "guided" else 0.0)
        return dict(bytes=_tree_bytes(prims) + npix * (32.0 if case.get("image") == "sums" else 36.0), flops=rays * per)
    if kind == "batch":
        total_b = total_f = 0.0
        for _, cam, spp, tris in _batch(case):
            npix = cam["w"] * cam["h"]
            total_b += _tree_bytes(tris) + 36.0 * npix
            total_f += 3.0 * npix * spp * (_ray_flops(tris) + 300.0)
        return dict(bytes=total_b, flops=total_f)
    n, macs = case["n"], 36 * 64 + 3 * 64 * 64 + 64 * 41
    params = 4 * rg.Guide.N_PARAMS
    if kind == "infer":
        return dict(bytes=n * (36 + 192) + params, flops=2.0 * macs * n)
    # samples in; weights, both moments and gradients through Adam
    return dict(bytes=n * 56 + 8 * params, flops=6.0 * macs * n)


# ------------------------------------------------------------------ 64 bits
def _exact_t(case, seed: int):
    """The closest hits' distances by testing every triangle in 64 bits (Moller-Trumbore)."""
    _, _, (pts, idx, _, _) = _scene("sphere", case["level"])
    r = [a.double() for a in _rays(case, seed)]
    o, d, t = torch.stack(r[0:3], 1), torch.stack(r[3:6], 1), r[6].clone()
    P = torch.tensor(pts, device="cuda").double()
    T = P[torch.tensor(idx.astype(np.int64), device="cuda")]
    v0, e1, e2 = T[:, 0], T[:, 1] - T[:, 0], T[:, 2] - T[:, 0]
    step = max(1, (1 << 24) // case["n"])
    for a in range(0, v0.shape[0], step):
        b1, b2 = e1[None, a:a + step], e2[None, a:a + step]
        pv = torch.linalg.cross(d[:, None], b2)
        det = (b1 * pv).sum(-1)
        inv = 1.0 / det
        tv = o[:, None] - v0[None, a:a + step]
        u = (tv * pv).sum(-1) * inv
        qv = torch.linalg.cross(tv, b1.expand_as(tv))
        v = (d[:, None] * qv).sum(-1) * inv
        tt = (b2 * qv).sum(-1) * inv
        hit = (det.abs() >= 1e-8) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (tt >= 0)
        t = torch.minimum(t, torch.where(hit, tt, torch.full_like(tt, math.inf)).amin(1))
    return t


def _exact_net(rows: torch.Tensor, W, b):
    """The network's 41 outputs in 64 bits; its inputs' coordinates lie in the unit box."""
    x = rows[:, 0:9].double()
    v = 0.5 * (x + 1.0)
    feats = torch.stack([torch.sin(math.pi * v), torch.cos(math.pi * v), torch.sin(2 * math.pi * v),
                         torch.cos(2 * math.pi * v)], 2).reshape(-1, 36)
    h = torch.nn.functional.pad(feats, (0, 28))
    for layer in range(5):
        h = h @ W[layer] + b[layer]
        if layer < 4:
            h = torch.relu(h)
    return h


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "hits" and case["rays"] == "random" and case["n"] * 20 * 4 ** case["level"] <= 2_000_000_000:
        return dict(prim=None, t=_exact_t(case, seed), ng=None)
    if kind not in ("infer", "train"):
        return None
    w, b = _weights(seed + 5)
    W = torch.tensor(w, device="cuda").double().requires_grad_(kind == "train")
    B = torch.tensor(b, device="cuda").double().requires_grad_(kind == "train")
    rows = _samples(case["n"], seed)
    if kind == "infer":
        out = _exact_net(rows, W, B)
        out[:, 41:] = 0.0
        return dict(out=out[:, :rg.Guide.ROW_OUTPUTS].contiguous())
    total = 0.0
    for a in range(0, case["n"], 1 << 17):
        s = rows[a:a + (1 << 17)]
        o = _exact_net(s, W, B)
        wi, wt, pb = s[:, 9:12].double(), s[:, 12].double() / case["n"], s[:, 13].double()
        vec = torch.stack([o[:, 0:8], o[:, 8:16], o[:, 16:24]], 2)
        norm = vec.norm(dim=2)
        mu = vec / norm[..., None]
        kappa = torch.clamp(torch.nn.functional.softplus(o[:, 24:32]) + 0.01, max=5000.0)
        pi = torch.softmax(5.0 * torch.tanh(o[:, 32:40] / 5.0), 1)
        f = kappa / (2 * math.pi * -torch.expm1(-2 * kappa)) * torch.exp(kappa * ((mu * wi[:, None]).sum(2) - 1.0))
        q = (pi * f).sum(1)
        nll = -(wt * torch.log(q)).sum()
        share = 0.05 + 0.9 * torch.sigmoid(o[:, 40])
        sel = torch.log(share * q.detach() + (1.0 - share) * pb)
        sel = -(wt * torch.where(pb > 0, sel, torch.zeros_like(sel))).sum()
        pull = (wt[:, None] * 0.01 * (norm - 1.0) ** 2).sum()
        (nll + sel + pull).backward()
        total += float(nll.detach())
    return dict(loss=total, grads=torch.cat([W.grad.reshape(-1), B.grad.reshape(-1)]))
