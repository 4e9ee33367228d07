"""Workloads of the renderer, measured through its public entry points.

Three kinds of call, which are what programs use the library for:

* ``render``: one frame or one progressive step: the film is cleared, ``c2g_render`` traces a range of samples of
  every pixel, and the film's sums and weights come back to page-locked host memory (the loop of a viewer or of an
  offline frame).  Scenes are the package's own generators at sizes from a thumbnail to 1920 x 1080; path tracer,
  direct lighting and guided path tracer; Halton, Default and Stratified samplers; BVH and Brute semantics.
* ``rays``: ray queries (closest hit, or any hit on a segment) against a loaded scene, on device arrays or on host
  arrays, as a baking or visibility tool calls them.
* ``batch``: several jobs rendered together by ``Batch.run`` in its default mode (one graph launch).
* ``gradient``: the guiding network's forward and backward pass on an explicit sample batch.

Every scene, ray set, network and sample range comes from the seed.
"""
import ctypes
import json
import math
import shutil
import tempfile

import numpy as np
import torch

from crystal2_gb300 import Batch, Context, scenes
from crystal2_gb300 import native as N

INTEGRATORS = {"path": N.INTEGRATOR_PATH, "direct": N.INTEGRATOR_DIRECT, "guided": N.INTEGRATOR_GUIDED}

# Approximate rays per camera path (extension, shadow and MIS rays together) of each scene: they only scale work().
RAYS_PER_PATH = {"cornell": 9.0, "material": 22.0, "yard": 6.0, "many": 6.5, "slit": 14.0}
TRIANGLES = {"cornell": 14, "material": 24, "yard": 6}
NETWORK = ((80, 64), (64, 64), (64, 64), (64, 48))  # layer shapes of the guiding network
GUIDE_BOX = ((-5.0, 0.0, -5.0), (5.0, 4.0, 6.0))


def listed():
    return [
        # a material preview: a thumbnail at one sample per pixel, redrawn on each edit; latency counts
        dict(name="thumbnail", kind="render", scene="cornell", width=64, height=64, spp=1, depth=8, integrator="path", sampler="Halton", accel="BVH"),
        # the Cornell box at its usual size: a complete small frame
        dict(name="cornell_frame", kind="render", scene="cornell", width=256, height=256, spp=64, depth=8, integrator="path", sampler="Halton", accel="BVH"),
        # every material, curved lights and a point light; odd frame size, stratified samples, exact shadow tests
        dict(name="materials_odd", kind="render", scene="material", width=201, height=149, spp=9, depth=8, integrator="path", sampler="Stratified", accel="Brute"),
        # textures and skybox under direct lighting: a layout preview
        dict(name="direct_yard", kind="render", scene="yard", width=320, height=240, spp=4, depth=6, integrator="direct", sampler="Halton", accel="BVH"),
        # the headline frame: two million triangles, 1080p, one 16-sample step
        dict(name="many_1080p", kind="render", scene="many", size=20, width=1920, height=1080, spp=16, depth=16, integrator="path", sampler="Halton", accel="BVH"),
        # an interactive step on a smaller scene of that family, with the plain random sampler
        dict(name="many_interactive", kind="render", scene="many", size=8, width=640, height=360, spp=2, depth=16, integrator="path", sampler="Default", accel="BVH"),
        # the slit-lit glossy room, path traced: long paths in a closed room
        dict(name="slit_plain", kind="render", scene="slit", size=192, width=960, height=540, spp=8, depth=12, integrator="path", sampler="Halton", accel="Brute"),
        # the same room guided: inference at every level, then Adam steps on the wave's records
        dict(name="slit_guided", kind="render", scene="slit", size=192, width=640, height=360, spp=8, depth=12, integrator="guided", sampler="Halton", accel="Brute"),
        # closest hits of device-resident rays, half coherent and half random
        dict(name="rays_closest", kind="rays", tris=1 << 16, rays=1 << 21, any_hit=False, host=False),
        # a visibility query of an odd number of host rays
        dict(name="rays_visible", kind="rays", tris=1 << 12, rays=10007, any_hit=True, host=True),
        # a handful of jobs of mixed sizes rendered together
        dict(name="batch_jobs", kind="batch", jobs=8, side=192, spp=16),
        # one gradient of the guiding network
        dict(name="guide_gradient", kind="gradient", samples=1 << 17),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "render", "rays", "batch", "gradient"])
    if kind == "rays":
        return dict(kind=kind, tris=_log(rng, 1 << 8, 1 << 16), rays=_log(rng, 1000, 1 << 21), any_hit=rng.random() < 0.5, host=rng.random() < 0.4)
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(2, 12), side=_log(rng, 64, 256), spp=rng.choice([4, 8, 16]))
    if kind == "gradient":
        return dict(kind=kind, samples=_log(rng, 1 << 8, 1 << 18))
    scene = rng.choice(["cornell", "material", "yard", "many", "many", "slit", "slit"])
    paths = math.exp(rng.uniform(math.log(4096), math.log(8 << 20)))  # camera paths of the pass
    spp = rng.choice([1, 2, 3, 4, 8, 16])
    pixels = max(2048.0, min(paths / spp, 1920 * 1080.0))
    aspect = rng.uniform(1.0, 1.8)
    c = dict(kind=kind, scene=scene, width=max(8, int(round(math.sqrt(pixels * aspect)))), height=max(8, int(round(math.sqrt(pixels / aspect)))), spp=spp,
             depth=rng.choice([5, 8, 12, 16]), integrator=rng.choice(["path", "path", "path", "direct", "guided" if scene == "slit" else "path"]),
             sampler=rng.choice(["Halton", "Halton", "Default", "Stratified"]), accel="Brute" if scene == "slit" else rng.choice(["BVH", "Brute"]))
    if c["sampler"] == "Stratified":
        c["spp"] = {2: 1, 3: 4, 8: 9}.get(spp, spp)  # a square number of samples per pixel
    if scene == "many":
        c["size"] = rng.randint(4, 16)
    if scene == "slit":
        c["size"] = rng.choice([64, 97, 128, 192])
    return c


def _set_config(path, sampler, accel, seed):
    with open(path) as fh:
        cfg = json.load(fh)
    cfg["Acceleration"] = accel
    cfg["Integrator"]["Sampler"] = {"Type": sampler, "Seed": int(seed)}
    with open(path, "w") as fh:
        json.dump(cfg, fh)


def _scene_files(d, case, seed):
    w, h, spp, depth, scene = case["width"], case["height"], case["spp"], case["depth"], case["scene"]
    if scene == "cornell":
        cp, sp = scenes.cornell_variant(d, seed=seed, width=w, height=h, spp=spp, depth=depth)
    elif scene == "material":
        cp, sp = scenes.material_box(d, width=w, height=h, spp=spp, depth=depth)
    elif scene == "yard":
        cp, sp = scenes.textured_yard(d, width=w, height=h, spp=spp, depth=depth, seed=seed)
    elif scene == "many":
        cp, sp = scenes.many_material(d, width=w, height=h, spp=spp, depth=depth, seed=seed, n_grid=case["size"])
    else:
        cp, sp = scenes.slit_room(d, width=w, height=h, spp=spp, depth=depth, seed=seed, hf_res=case["size"])
    _set_config(cp, case["sampler"], case["accel"], seed & 0x7FFF)
    return cp, sp


def _load(case, seed, make):
    d = tempfile.mkdtemp(prefix="c2g_cases_")
    try:
        ctx = Context(0)
        ctx.load(*make(d), tree=N.TREE_SAH)
        return ctx
    finally:
        shutil.rmtree(d, ignore_errors=True)


def _network(seed):
    """Weights of the guiding network, He-uniform with a small output layer, as a program that keeps them has."""
    rng = np.random.default_rng(seed)
    parts = []
    for i, (k, n) in enumerate(NETWORK):
        w = rng.uniform(-1, 1, (k, n)) * math.sqrt(6.0 / k) * (0.1 if i == 3 else 1.0)
        b = rng.uniform(-0.05, 0.05, n)
        if i == 3:
            w[:, N.GUIDE_OUTPUTS:] = 0
            b[N.GUIDE_OUTPUTS:] = 0
        parts += [w.ravel(), b]
    return np.concatenate(parts).astype(np.float32)


class _Film:
    """Page-locked host buffers of one film."""

    def __init__(self, w, h):
        self.t = (torch.zeros((h, w, 3), dtype=torch.float32, pin_memory=True), torch.zeros((h, w), dtype=torch.float32, pin_memory=True))
        self.rgb, self.weight = (x.numpy() for x in self.t)

    def read(self, ctx):
        ctx.check(N.load_library().c2g_film_download(ctx.handle, N.fptr(self.rgb), N.fptr(self.weight)))


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([seed & 0x7FFFFFFF, 11])
    if kind == "render":
        ctx = _load(case, seed, lambda d: _scene_files(d, case, seed & 0x7FFFFFFF))
        p = ctx.render_params()
        p.integrator = INTEGRATORS[case["integrator"]]
        p.sample_begin = 0 if case["sampler"] == "Stratified" else int(rng.integers(0, 4096))
        p.sample_count = case["spp"]
        s = {"kind": kind, "ctx": ctx, "p": p, "film": _Film(case["width"], case["height"])}
        if case["integrator"] == "guided":
            ctx.guide_config(1e-3, 0.7, 0, 16)  # a resumed frame: the network is used from the first wave on
            ctx.guide_levels(0)
            ctx.guide_batch(1 << 18, 4)
            ctx.guide_regularize(200.0, 20.0, 2000.0)
            ctx.guide_reset(*GUIDE_BOX, seed=seed)
            s["net"] = _network(seed)
        return s
    if kind == "rays":
        def soup(d):
            return scenes.tri_soup(d, n_tris=case["tris"], seed=seed & 0x7FFFFFFF)
        ctx = _load(case, seed, soup)
        n = case["rays"]
        o, v = scenes.microbench_rays(n, seed=seed & 0xFFFF)
        tmax = (rng.random(n) * 2.0).astype(np.float32)
        s = {"kind": kind, "ctx": ctx, "n": n, "any": case["any_hit"], "host": case["host"]}
        if case["host"]:
            s.update(o=o, d=v, tmax=tmax)
        else:
            dev = torch.device("cuda", 0)
            s.update(o=torch.from_numpy(o).to(dev), d=torch.from_numpy(v).to(dev), tmax=torch.from_numpy(tmax).to(dev),
                     obj=torch.empty(n, dtype=torch.int32, device=dev), t=torch.empty(n, dtype=torch.float32, device=dev))
        return s
    if kind == "batch":
        b, ctxs, films = Batch(0), [], []
        for j in range(case["jobs"]):
            side = max(16, int(case["side"] * (0.5, 1.0, 0.75)[j % 3]))
            scene = "cornell" if j % 2 == 0 else "many"
            c = dict(scene=scene, size=4, width=side, height=side, spp=case["spp"], depth=8, sampler="Halton", accel="BVH")
            ctx = _load(c, seed, lambda d: _scene_files(d, c, (seed + 101 * j) & 0x7FFFFFFF))
            p = ctx.render_params()
            p.sample_count = case["spp"]
            b.add(ctx, p)
            ctxs.append(ctx)
            films.append(_Film(side, side))
        return {"kind": kind, "batch": b, "ctxs": ctxs, "films": films}
    ctx = _load(case, seed, lambda d: scenes.cornell(d, width=16, height=16, spp=1, depth=2))
    ctx.guide_reset(*GUIDE_BOX, seed=seed)
    ctx.guide_set_params(_network(seed))
    return {"kind": kind, "ctx": ctx, "samples": _samples(case, seed)}


def _samples(case, seed):
    rng = np.random.default_rng([seed & 0x7FFFFFFF, 5])
    m = case["samples"]
    lo, hi = np.array(GUIDE_BOX[0]), np.array(GUIDE_BOX[1])

    def unit():
        v = rng.normal(size=(m, 3))
        return v / np.linalg.norm(v, axis=1, keepdims=True)

    x = lo + (hi - lo) * rng.random((m, 3))
    w, pb = rng.exponential(1.0, (m, 1)), 0.05 + 1.95 * rng.random((m, 1))
    return np.concatenate([x, unit(), unit(), unit(), w, pb], axis=1).astype(np.float32)


def run(s):
    kind = s["kind"]
    if kind == "render":
        ctx = s["ctx"]
        if "net" in s:
            ctx.guide_set_params(s["net"])
        ctx.film_clear()
        ctx.render(s["p"])
        s["film"].read(ctx)
        out = {"rgb": s["film"].rgb, "weight": s["film"].weight}
        if "net" in s:
            out["params"] = ctx.guide_params()
        return out
    if kind == "rays":
        ctx = s["ctx"]
        if s["host"]:
            return ctx.trace_rays(s["o"], s["d"], any_hit=s["any"], tmax=s["tmax"] if s["any"] else None)

        def p(x):
            return ctypes.c_void_p(x.data_ptr()) if x is not None else None
        ctx.check(N.load_library().c2g_trace_rays_dev(ctx.handle, s["n"], p(s["o"]), p(s["d"]), None, p(s["tmax"]) if s["any"] else None, None,
                                                      int(s["any"]), p(s["obj"]), None if s["any"] else p(s["t"]), None))
        return (s["obj"],) if s["any"] else (s["obj"], s["t"])
    if kind == "batch":
        for ctx in s["ctxs"]:
            ctx.film_clear()
        s["batch"].run()
        for ctx, film in zip(s["ctxs"], s["films"]):
            film.read(ctx)
        return [(f.rgb, f.weight) for f in s["films"]]
    g, loss = s["ctx"].guide_gradient(s["samples"])
    return {"grad": g, "loss": loss}


def _traced(rays, tris):
    """Bytes and operations that many rays need: the ray and its hit, the scene once, and per ray one box test per
    level of a balanced four-wide tree (4 boxes of 18 operations) and two triangle tests of 50."""
    levels = max(1.0, math.log(max(2.0, tris / 2.0), 4))
    return dict(bytes=rays * 40.0 + tris * 64.0, flops=rays * (levels * 72.0 + 100.0))


def work(case):
    kind = case["kind"]
    if kind == "render":
        tris = TRIANGLES.get(case["scene"]) or (case["size"] ** 2 * 5120 if case["scene"] == "many" else 2 * case["size"] ** 2)
        paths = case["width"] * case["height"] * case["spp"]
        rays = paths * RAYS_PER_PATH[case["scene"]] * (0.5 if case["integrator"] == "direct" else 1.0)
        w = _traced(rays, tris)
        flops = w["flops"] + rays * 100.0  # shading, spread over the rays
        if case["integrator"] == "guided":
            flops += paths * 3.0 * 2 * sum(k * n for k, n in NETWORK)
        return dict(bytes=tris * 64.0 + case["width"] * case["height"] * 16.0, flops=flops)
    if kind == "rays":
        return _traced(case["rays"], case["tris"])
    if kind == "batch":
        paths = case["jobs"] * (0.75 * case["side"]) ** 2 * case["spp"]
        return dict(bytes=paths / case["spp"] * 16.0, flops=paths * 7.0 * 500.0)
    m = case["samples"]
    return dict(bytes=m * 56.0 + 2 * 4.0 * N.GUIDE_PARAMS, flops=3.0 * 2 * m * sum(k * n for k, n in NETWORK))


def exact(case, seed):
    """Only the network's gradient has a value in 64 bits; a film is a sum over paths whose branches follow the
    renderer's own float arithmetic, and so are hit records on shared edges."""
    if case["kind"] != "gradient":
        return None
    dev = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
    flat = torch.from_numpy(_network(seed)).double().to(dev).requires_grad_(True)
    s = torch.from_numpy(_samples(case, seed)).to(dev)
    lo = torch.tensor(GUIDE_BOX[0], dtype=torch.float64, device=dev)
    hi = torch.tensor(GUIDE_BOX[1], dtype=torch.float64, device=dev)
    loss_sum, weight_sum = 0.0, 0.0
    for part in s.double().split(1 << 15):
        x, nrm, wo, wi, w, pb = part.split([3, 3, 3, 3, 1, 1], dim=1)
        p = ((x - lo) / (hi - lo)).clamp(0, 1)
        ang = math.pi * p[:, :, None] * (2.0 ** torch.arange(12, dtype=torch.float64, device=dev))
        h = torch.cat([torch.stack([ang.sin(), ang.cos()], dim=3).reshape(len(part), 72), nrm, wo, torch.zeros(len(part), 2, dtype=torch.float64, device=dev)], dim=1)
        at = 0
        for i, (k, n) in enumerate(NETWORK):
            h = h @ flat[at:at + k * n].reshape(k, n) + flat[at + k * n:at + k * n + n]
            at += k * n + n
            h = h.relu() if i < 3 else h
        o = h[:, :40].reshape(-1, 8, 5)
        mu = torch.nn.functional.normalize(o[:, :, :3], dim=2)
        kappa = (torch.nn.functional.softplus(o[:, :, 3]) + 0.05).clamp(max=500.0)
        cosine = (mu * wi[:, None, :]).sum(2)
        vmf = kappa / (2 * math.pi * -torch.expm1(-2 * kappa)) * torch.exp(kappa * (cosine - 1))
        q = (o[:, :, 4].softmax(1) * vmf).sum(1)
        c = 0.05 + 0.75 * torch.sigmoid(h[:, 40])
        nll = (w[:, 0] * -torch.log((1 - c) * pb[:, 0] + c * q)).sum()
        nll.backward()
        loss_sum += float(nll.detach())
        weight_sum += float(w.sum())
    return {"grad": flat.grad.cpu().numpy(), "loss": loss_sum / weight_sum}
