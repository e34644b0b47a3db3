"""Measured workloads of the renderer: what a program asks of it, from one
picking query to the full terrain frame, through the public entry points
(kazen_proto_gb300.api and, for device-resident buffers it has no wrapper
for, the C ABI that api binds).

A case is a dict of plain values; `kind` selects how it is prepared and run:
  rays      closest-hit or any-hit queries against a triangle soup
  li        radiance of a batch of camera rays (PathIntegrator.Li)
  frame     one image (Renderer.render)
  batch     many jobs in one call (render_batch)
  guided    one image guided by a given network (render_guided)
  train     one training step of the guiding network: loss and gradient
  closures  evaluation and sampling of a batch of closure lobes
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from kazen_proto_gb300 import _native as N
from kazen_proto_gb300 import api, scenes


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # a viewport's pick: a few rays in host arrays, the answer needed at once
        {"name": "pick", "kind": "rays", "query": "closest", "mem": "host", "tris": 20_000, "rays": 64},
        # a simulation's or baker's incoherent closest hits, resident on the device (the traversal benchmark)
        {"name": "closest_incoherent", "kind": "rays", "query": "closest", "mem": "device", "tris": 1 << 20,
         "rays": 1 << 24},
        # visibility of an odd number of segments in a smaller model
        {"name": "any_odd", "kind": "rays", "query": "any", "mem": "device", "tris": 250_001, "rays": 3_000_017},
        # a host integrator that hands its own camera rays over in batches
        {"name": "li_batch", "kind": "li", "scene": "terrain", "detail": 256, "rays": 65_537, "depth": 5},
        # an interactive preview: small, few samples, textures, normals, mixtures, point light, environment
        {"name": "preview", "kind": "frame", "scene": "studio", "detail": 2, "width": 97, "height": 65, "spp": 4,
         "depth": 6},
        # the small box scene, the workload of the CPU renderer
        {"name": "box_frame", "kind": "frame", "scene": "box", "detail": 0, "width": 256, "height": 256, "spp": 16,
         "depth": 5},
        # a look-development frame: every closure family in mixtures, textured and smooth-shaded
        {"name": "materials_frame", "kind": "frame", "scene": "studio", "detail": 4, "width": 641, "height": 359,
         "spp": 16, "depth": 6},
        # the headline frame
        {"name": "terrain_frame", "kind": "frame", "scene": "terrain", "detail": 1024, "width": 1920, "height": 1080,
         "spp": 64, "depth": 8},
        # a queue of uneven jobs (previews, material variants) in one call
        {"name": "batch_jobs", "kind": "batch", "jobs": 24, "tris_lo": 20_000, "tris_hi": 200_000, "res_hi": 256},
        # a frame with learned guiding, the network trained before
        {"name": "guided_frame", "kind": "guided", "width": 512, "height": 512, "spp": 8, "depth": 10},
        # one step of the guiding network's training at its stated batch
        {"name": "guide_train", "kind": "train", "rows": 1 << 18},
        # closures evaluated and sampled for a host's own integrator or a material check, kinds in arbitrary order
        {"name": "closures", "kind": "closures", "lobes": 1_000_003, "mix": "all"},
    ]


def _log_int(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n))


def draw(rng):
    kind = rng.choice(["rays", "rays", "rays", "li", "frame", "frame", "frame", "batch", "guided", "train", "closures"])
    if kind == "rays":
        mem = rng.choice(["host", "device", "device"])
        return {"kind": kind, "query": rng.choice(["closest", "any"]), "mem": mem,
                "tris": _log_int(rng, 2_000, 1 << 20), "rays": _log_int(rng, 1, 4096 if mem == "host" else 1 << 24)}
    if kind == "li":
        return {"kind": kind, "scene": rng.choice(["box", "studio", "terrain"]), "detail": rng.randint(2, 4),
                "rays": _log_int(rng, 1_000, 2_000_000), "depth": rng.randint(3, 8)}
    if kind == "frame":
        scene = rng.choice(["box", "studio", "terrain"])
        return {"kind": kind, "scene": scene,
                "detail": _log_int(rng, 64, 512) if scene == "terrain" else rng.randint(2, 4),
                "width": _log_int(rng, 48, 1600), "height": _log_int(rng, 48, 1000),
                "spp": rng.choice([1, 2, 4, 8, 16, 16, 32]), "depth": rng.randint(3, 8)}
    if kind == "batch":
        lo = _log_int(rng, 5_000, 50_000)
        return {"kind": kind, "jobs": rng.randint(3, 24), "tris_lo": lo, "tris_hi": lo * 4,
                "res_hi": rng.choice([64, 128, 256])}
    if kind == "guided":
        return {"kind": kind, "width": _log_int(rng, 64, 600), "height": _log_int(rng, 64, 600),
                "spp": rng.choice([1, 4, 8, 16]), "depth": rng.randint(4, 12)}
    if kind == "train":
        return {"kind": kind, "rows": _log_int(rng, 1_000, 1 << 20)}
    return {"kind": kind, "lobes": _log_int(rng, 1_000, 4_000_000), "mix": rng.choice(["all", "principled", "rough"])}


# ---------------------------------------------------------------- scenes
def _camera(cam, seed):
    """The scene's camera, moved a little by the seed."""
    r = np.random.default_rng(seed)
    d = r.uniform(-0.01, 0.01, 3)
    return api.Camera(eye=tuple(float(a + b) for a, b in zip(cam.eye, d)), lookat=cam.lookat, up=cam.up, fov=cam.fov)


def _studio(subdiv, seed):
    """The box room with textured walls and smooth spheres of mixed materials,
    an area light, a point light and an environment seen through the open side."""
    r = np.random.default_rng(seed)
    d = scenes.SceneDesc()
    img = r.uniform(0.1, 0.9, (33, 65, 3)).astype(np.float32)
    sky = r.uniform(0.2, 1.0, (16, 32, 3)).astype(np.float32)
    d.textures = [api.checker_texture(5.0, 5.0, (0.8, 0.75, 0.7), (0.25, 0.3, 0.35)), api.image_texture(img),
                  api.image_texture(sky)]
    c = lambda lo, hi: tuple(float(v) for v in r.uniform(lo, hi, 3))  # noqa: E731
    a = lambda lo=0.08, hi=0.5: float(r.uniform(lo, hi))  # noqa: E731
    rough = lambda: [api.diffuse(tuple(0.5 * v for v in c(0.3, 0.9))),  # noqa: E731
                     api.microfacet("beckmann", a(), eta=1.5, weight=c(0.05, 0.2))]
    plastic = lambda: [api.principle_diffuse(c(0.2, 0.7)), api.principle_retro(a(0.2, 0.9), c(0.1, 0.3)),  # noqa: E731
                       api.principle_specular((0.04, 0.04, 0.04), a(), 1.5, 0.0, (0.6, 0.6, 0.6)),
                       api.principle_sheen(1.0, c(0.0, 0.2)), api.principle_clearcoat(a(0.1, 0.6), (0.25, 0.25, 0.25))]
    kinds = [rough, plastic, lambda: [api.microfacet("ggx", a(), eta=0.66, refract=2)],
             lambda: [api.conductor_ggx(c(0.5, 1.0), a())], lambda: [api.dielectric(1.5, 1.0)],
             lambda: [api.diffuse(c(0.2, 0.8))], lambda: [api.mirror(c(0.7, 0.95))],
             lambda: [api.microfacet("ggx", a(), eta=1.5, weight=c(0.3, 0.9)), api.diffuse(c(0.1, 0.4))]]
    walls = [((0, 0, 0), (0, 0, 1), (1, 0, 0), api.textured(api.diffuse((0.8, 0.8, 0.8)), 0)),
             ((0, 1, 0), (1, 0, 0), (0, 0, 1), api.diffuse((0.7, 0.7, 0.7))),
             ((0, 0, 1), (0, 1, 0), (1, 0, 0), api.textured(api.diffuse((0.9, 0.9, 0.9)), 1)),
             ((0, 0, 0), (0, 1, 0), (0, 0, 1), api.diffuse((0.6, 0.1, 0.1))),
             ((1, 0, 0), (0, 0, 1), (0, 1, 0), api.diffuse((0.1, 0.5, 0.1)))]
    uv = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], np.float32)
    for p0, e1, e2, lobe in walls:
        v, i = scenes.quad(p0, e1, e2)
        d.materials.append(api.material([lobe]))
        d.add(v, i, len(d.materials) - 1, uv=uv)
    sv, sf = scenes.icosphere(subdiv)
    for k in range(24):
        d.materials.append(api.material(kinds[k % len(kinds)]()))
        rad = np.float32(r.uniform(0.05, 0.11))
        pos = r.uniform((0.12, 0.1, 0.15), (0.88, 0.75, 0.9)).astype(np.float32)
        d.add((sv * rad + pos).astype(np.float32), sf, len(d.materials) - 1, normals=sv if k % 4 else None)
    d.materials.append(api.material([], Le=(14.0, 12.0, 9.0)))
    v, i = scenes.quad((0.35, 0.995, 0.35), (0.3, 0, 0), (0, 0, 0.3))
    d.add(v, i, len(d.materials) - 1, is_light=True)
    d.point_lights = [((0.2, 0.85, 0.1), (0.05, 0.05, 0.06))]
    d.env, d.env_texture = (0.4, 0.45, 0.5), 2
    d.camera = api.Camera(eye=(0.5, 0.5, -1.2), lookat=(0.5, 0.45, 0.5), up=(0, 1, 0), fov=42.0)
    return d


def _scene(case, seed):
    if case["scene"] == "box":
        return scenes.box_scene()
    if case["scene"] == "studio":
        return _studio(case["detail"], seed)
    if case["detail"] < 16:  # a small terrain for rays of a host integrator
        return scenes.terrain_scene(cells=64 * case["detail"], n_spheres=16, subdiv=2, seed=seed)
    return scenes.terrain_scene(cells=case["detail"], seed=seed)


def _soup(case, seed):
    return scenes.triangle_soup(case["tris"], seed)


def _rays(case, seed):
    return scenes.soup_rays(case["rays"], seed + 1)


def _camera_rays(cam, n, seed):
    """n rays of a host's camera: jittered positions in scanline order."""
    r = np.random.default_rng(seed)
    w = max(1, int(math.sqrt(n * 16 / 9)))
    h = (n + w - 1) // w
    k = np.arange(n)
    t = math.tan(math.radians(cam.fov) / 2)
    x = (2 * (k % w + r.random(n)) / w - 1) * t
    y = (1 - 2 * (k // w + r.random(n)) / h) * t * h / w
    eye, look, up = (np.array(v, np.float64) for v in (cam.eye, cam.lookat, cam.up))
    z = (eye - look) / np.linalg.norm(eye - look)
    xa = np.cross(up, z)
    xa /= np.linalg.norm(xa)
    return api.make_rays(eye, x[:, None] * xa + y[:, None] * np.cross(z, xa) - z)


def _on_device(records):
    return torch.from_numpy(records.view(np.float32).reshape(len(records), -1)).cuda()


# ---------------------------------------------------------------- closures and guiding inputs
_PRINCIPLED, _ROUGH = (8, 17, 18, 19, 20), (0, 3, 4, 5, 6, 7, 8)


def _lobes(case, seed):
    """Lobes of the closure kinds a mix names, in arbitrary order, with
    directions on both sides, and the uniforms to sample them with."""
    r = np.random.default_rng(seed)
    n = case["lobes"]
    kinds = {"all": np.arange(21), "principled": np.array(_PRINCIPLED), "rough": np.array(_ROUGH)}[case["mix"]]
    kind = kinds[r.integers(0, len(kinds), n)]
    a, b = r.uniform(0.05, 1.0, n), r.uniform(0.05, 1.0, n)
    eta, x = r.uniform(0.3, 2.5, n), r.uniform(0.05, 0.9, n)
    rgb = r.uniform(0.0, 1.0, (n, 3))
    ids = np.array([N.KZ_CLOSURE_DIFFUSE, N.KZ_CLOSURE_KP_MIRROR, N.KZ_CLOSURE_KP_DIELECTRIC, N.KZ_CLOSURE_KP_GLOSS,
                    N.KZ_CLOSURE_KP_GLOSS, N.KZ_CLOSURE_KP_GLASS, N.KZ_CLOSURE_KP_GLASS, N.KZ_CLOSURE_CONDUCTOR_GGX,
                    N.KZ_CLOSURE_KP_PRINCIPLE_SPECULAR_REFL, N.KZ_CLOSURE_PHONG, N.KZ_CLOSURE_WARD,
                    N.KZ_CLOSURE_WARD, N.KZ_CLOSURE_REFLECTION, N.KZ_CLOSURE_REFRACTION, N.KZ_CLOSURE_TRANSPARENT,
                    N.KZ_CLOSURE_TRANSLUCENT, N.KZ_CLOSURE_KP_MICROFACET, N.KZ_CLOSURE_KP_PRINCIPLE_DIFFUSE,
                    N.KZ_CLOSURE_KP_PRINCIPLE_RETRO, N.KZ_CLOSURE_KP_PRINCIPLE_SHEEN,
                    N.KZ_CLOSURE_KP_PRINCIPLE_CLEARCOAT], np.uint32)
    lobes = np.zeros(n, N.LOBE_DTYPE)
    lobes["closure_id"] = ids[kind]
    lobes["weight"] = 1.0
    p = np.zeros((n, 12))

    def put(k, cols):
        m = kind == k
        for j, v in cols.items():
            p[m, j] = v[m] if isinstance(v, np.ndarray) else v

    up = {0: 0.0, 1: 1.0, 2: 0.0}
    for k in (0, 9, 10, 11, 12, 13, 17, 18, 19, 20):
        put(k, up)
    put(2, {0: 1.1 + 0.9 * x, 1: 1.0})
    for k, dist, same, refract in ((3, 0, False, 0), (4, 1, False, 0), (5, 0, True, 1), (6, 1, True, 2)):
        put(k, {0: dist, 2: 1.0, 4: 1.0, 7: a, 8: a if same else b, 9: eta, 10: refract})
    put(7, {0: rgb[:, 0], 1: rgb[:, 1], 2: rgb[:, 2], 3: a, 4: a})
    put(8, {0: rgb[:, 0], 1: rgb[:, 1], 2: rgb[:, 2], 4: 1.0, 6: a, 7: a, 8: eta, 9: x})
    put(9, {3: 1.0 + 100.0 * x})
    put(10, {3: 1.0, 6: a, 7: a})
    put(11, {3: 1.0, 6: a, 7: b})
    put(12, {3: eta})
    put(13, {3: eta})
    put(16, {0: a, 1: 1.1 + 0.9 * x, 2: 1.0, 3: b})
    for k in (18, 19, 20):
        put(k, {3: x})
    lobes["params"] = p.astype(np.float32)

    def directions():
        d = r.standard_normal((n, 3))
        d[:, 1] = np.where(r.random(n) < 0.8, np.abs(d[:, 1]), d[:, 1])
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        return d.astype(np.float32)

    u = r.random((n, 3)).astype(np.float32)
    return kind, lobes, directions(), directions(), np.minimum(u, np.float32(1.0 - 2.0 ** -24))


_LAYERS = ((64, 51), (64, 64), (64, 64), (40, 64))


def _network(seed):
    """Weights of the guiding network, exact in BF16, in the layout of kz_guide_set_params."""
    r = np.random.default_rng(seed + 77)
    out = []
    for k, (rows, fan) in enumerate(_LAYERS):
        w = np.zeros((rows, 64))
        w[:, :fan] = r.uniform(-1, 1, (rows, fan)) * (math.sqrt(6 / fan) if k < 3 else 0.5 * math.sqrt(3 / fan))
        out += [w.reshape(-1), r.uniform(-0.1, 0.1, rows)]
    return torch.from_numpy(np.concatenate(out)).to(torch.bfloat16).float().numpy()


def _samples(case, seed):
    """Radiance samples: position, weight, normal, direction (12 floats a row)."""
    r = np.random.default_rng(seed)
    n = case["rows"]
    s = np.zeros((n, 12), np.float32)
    s[:, 0:3] = r.random((n, 3))
    s[:, 3] = np.exp(r.normal(0.0, 1.0, n)).clip(0.0, 20.0)
    s[:, 4 + r.integers(0, 3)] = 1.0
    d = r.standard_normal((n, 3)) + np.array([0.5, 1.0, 0.0])
    s[:, 8:11] = d / np.linalg.norm(d, axis=1, keepdims=True)
    return s


# ---------------------------------------------------------------- prepare / run
def prepare(case, seed):
    kind, st = case["kind"], {"case": case}
    if kind == "rays":
        st["scene"] = scenes.soup_desc(_soup(case, seed)).build()
        rays = _rays(case, seed)
        if case["mem"] == "host":
            st["rays"] = rays
        else:
            n = case["rays"]
            st["rays"] = _on_device(rays)
            if case["query"] == "any":
                st["out"] = torch.empty(n, dtype=torch.uint8, device="cuda")
            else:
                f = lambda t: torch.empty(n, dtype=t, device="cuda")  # noqa: E731
                st["out"] = {"t": f(torch.float32), "prim_id": f(torch.int32), "geom_id": f(torch.int32),
                             "u": f(torch.float32), "v": f(torch.float32)}
    elif kind == "li":
        d = _scene(case, seed)
        st["scene"] = d.build()
        st["integrator"] = api.PathIntegrator(max_depth=case["depth"], seed=seed)
        st["integrator"].setup(st["scene"])
        st["rays"] = _on_device(_camera_rays(_camera(d.camera, seed), case["rays"], seed))
    elif kind == "frame":
        d = _scene(case, seed)
        st["scene"], st["camera"] = d.build(), _camera(d.camera, seed)
        st["renderer"] = api.Renderer(spp=case["spp"], max_depth=case["depth"], seed=seed)
        # an interactive loop's own buffer, reused for each frame
        st["out"] = torch.empty((case["height"], case["width"], 3), pin_memory=True)
    elif kind == "batch":
        res = tuple(r for r in (32, 64, 128, 256) if r <= case["res_hi"])
        # the queue's sizes belong to the case, its models and random streams to the seed
        jobs = scenes.batch_jobs(case["jobs"], 5, (case["tris_lo"], case["tris_hi"]), res, (4, 16), (4, 8))
        for k, j in enumerate(jobs):
            j["desc_args"], j["seed"] = (j["desc_args"][0], seed * 1000 + k), seed + k
        st["jobs"] = scenes.build_batch_scenes(jobs, workers=16)
        st["cfg"] = api.batch_config()
    elif kind == "guided":
        d = scenes.slit_room_scene(seed=seed)
        st["scene"], st["camera"] = d.build(), _camera(d.camera, seed)
        st["guide"] = api.Guide(seed=1)
        st["guide"].set_params(_network(seed))
        st["cfg"] = api.guide_config(train=False)
        st["seed"] = seed
    elif kind == "train":
        st["guide"] = api.Guide(seed=1)
        st["guide"].set_params(_network(seed))
        st["samples"] = torch.from_numpy(_samples(case, seed)).cuda()
    else:
        _, lobes, wi, wo, u = _lobes(case, seed)
        dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
        st.update(lobes=_on_device(lobes), wi=dev(wi), wo=dev(wo), u=dev(u))
        n = case["lobes"]
        f = lambda *s: torch.empty(s, device="cuda")  # noqa: E731
        st["out"] = {"f": f(n, 3), "pdf": f(n), "s_wo": f(n, 3), "s_weight": f(n, 3), "s_pdf": f(n),
                     "s_flags": torch.empty(n, dtype=torch.uint8, device="cuda")}
    return st


def _p(t):
    return C.c_void_p(t.data_ptr())


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "rays":
        s = st["scene"]
        query = s.intersect if case["query"] == "closest" else s.occluded
        if case["mem"] == "host":
            return query(st["rays"])
        out = query(st["rays"], out=st["out"])
        s.synchronize()  # the results are complete (and the status known) after this call only
        return out
    if kind == "li":
        return st["integrator"].Li(st["rays"])
    if kind == "frame":
        return st["renderer"].render(st["scene"], st["camera"], case["width"], case["height"], out=st["out"])
    if kind == "batch":
        return api.render_batch(st["jobs"], st["cfg"])[0]
    if kind == "guided":
        return api.render_guided(st["scene"], st["guide"], st["camera"], case["width"], case["height"], case["spp"],
                                 case["depth"], seed=st["seed"], gcfg=st["cfg"])[0]
    if kind == "train":
        loss, grad = C.c_float(), np.empty(N.KZ_GUIDE_PARAMS, np.float32)
        N.check(N.lib().kz_guide_train_step(st["guide"].handle, _p(st["samples"]), case["rows"], 1e-3, 0,
                                            C.byref(loss), grad.ctypes.data_as(C.c_void_p), N.KZ_MEM_DEVICE))
        return {"loss": loss.value, "grad": grad}
    n, o = case["lobes"], st["out"]
    N.check(N.lib().kz_closure_eval_batch(_p(st["lobes"]), _p(st["wi"]), _p(st["wo"]), n, N.KZ_CONVENTION_INTEGRATOR,
                                          _p(o["f"]), _p(o["pdf"]), N.KZ_MEM_DEVICE))
    N.check(N.lib().kz_closure_sample_batch(_p(st["lobes"]), _p(st["wi"]), _p(st["u"]), n, _p(o["s_wo"]),
                                            _p(o["s_weight"]), _p(o["s_pdf"]), _p(o["s_flags"]), N.KZ_MEM_DEVICE))
    return o


# ---------------------------------------------------------------- what a pass cannot do without
def _ray_flops(tris):
    """One ray: eight boxes a level of an 8-wide tree, and four triangle tests."""
    return 8 * 18 * max(1.0, math.log(max(tris, 8), 8)) + 4 * 50


def work(case):
    kind = case["kind"]
    if kind == "rays":
        per = 32 + (20 if case["query"] == "closest" else 1)
        return {"bytes": per * case["rays"] + 36 * case["tris"], "flops": case["rays"] * _ray_flops(case["tris"])}
    if kind in ("li", "frame"):
        tris = {"box": 36, "studio": 12 + 24 * 20 * 4 ** case["detail"]}.get(case["scene"])
        if tris is None:
            cells = case["detail"] if case["detail"] >= 16 else 64 * case["detail"]
            tris = 2 * cells * cells + (64 * 1280 if case["detail"] >= 16 else 16 * 320)
        paths = case["rays"] if kind == "li" else case["width"] * case["height"] * case["spp"]
        io = 44 * paths if kind == "li" else 12 * case["width"] * case["height"]
        # about 2.5 vertices a path: an extension ray, a shadow ray and some 300 operations of shading each
        return {"bytes": io + 36 * tris, "flops": paths * 2.5 * (2 * _ray_flops(tris) + 300)}
    if kind == "batch":
        tris = (case["tris_lo"] + case["tris_hi"]) / 2
        res = [r for r in (32, 64, 128, 256) if r <= case["res_hi"]]
        px = sum(r * r for r in res) / len(res)
        return {"bytes": case["jobs"] * (36 * tris + 12 * px),
                "flops": case["jobs"] * px * 10 * 2 * (2 * _ray_flops(tris) + 300)}
    if kind == "guided":
        px, tris = case["width"] * case["height"], 50 + 32 * 320
        return {"bytes": 12 * px + 36 * tris + 4 * N.KZ_GUIDE_PARAMS,
                "flops": px * case["spp"] * 6 * (2 * _ray_flops(tris) + 1200 + 2 * 14016)}
    if kind == "train":
        return {"bytes": 48 * case["rows"] + 8 * N.KZ_GUIDE_PARAMS, "flops": case["rows"] * 6 * 14016}
    # a lobe's 64 bytes and directions read by each of the two calls, their outputs written
    return {"bytes": case["lobes"] * (88 + 16 + 88 + 29), "flops": case["lobes"] * 400}


# ---------------------------------------------------------------- 64-bit values
def exact(case, seed):
    """run()'s outputs in 64 bits. None where there is no such value: an image
    is the sum of paths that branch on comparisons (which triangle, which lobe,
    roulette), so another rounding takes other paths; and None where testing
    every ray against every triangle would take too long."""
    kind = case["kind"]
    if kind == "rays" and case["query"] == "closest" and case["rays"] * case["tris"] <= 10 ** 9:
        return _exact_rays(_soup(case, seed), _rays(case, seed))
    if kind == "train":
        return _exact_train(_samples(case, seed), _network(seed))
    if kind == "closures":
        return _exact_closures(*_lobes(case, seed))
    return None


def _f64(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda().double()


def _exact_rays(soup, rays):
    tri = _f64(soup).view(-1, 3, 3)
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    r = _f64(rays.view(np.float32).reshape(len(rays), 8))
    ts, us, vs = [], [], []
    step = max(1, 20_000_000 // len(tri))
    for k in range(0, len(r), step):
        o, d = r[k:k + step, None, 0:3], r[k:k + step, None, 4:7]
        p = torch.linalg.cross(d.expand(-1, len(tri), -1), e2[None].expand(d.shape[0], -1, -1))
        det = (p * e1).sum(-1)
        s = o - v0
        u = (s * p).sum(-1) / det
        q = torch.linalg.cross(s, e1[None].expand_as(s))
        v = (d * q).sum(-1) / det
        t = (q * e2).sum(-1) / det
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > r[k:k + step, None, 3]) & (t <= r[k:k + step, None, 7])
        best, at = torch.where(ok, t, torch.full_like(t, math.inf)).min(1)
        hit = torch.isfinite(best)
        pick = lambda x: torch.where(hit, x.gather(1, at[:, None])[:, 0], torch.zeros_like(best))  # noqa: E731
        ts.append(best)
        us.append(pick(u))
        vs.append(pick(v))
    return {"t": torch.cat(ts), "prim_id": None, "geom_id": None, "u": torch.cat(us), "v": torch.cat(vs)}


def _exact_train(samples, params):
    """Mean of weight * -log q over the rows and its gradient, without the
    kernels' BF16 roundings of the activations."""
    p = _f64(params).requires_grad_()
    n = len(samples)
    total = 0.0
    for k in range(0, n, 1 << 17):
        s = _f64(samples[k:k + (1 << 17)])
        x = s[:, 0:3]
        arg = x[:, :, None] * (2.0 ** torch.arange(8, device=x.device).double()) * math.pi
        h = torch.cat([torch.stack([arg.sin(), arg.cos()], -1).flatten(1), s[:, 4:7],
                       torch.zeros(len(s), 13, device=x.device, dtype=torch.float64)], 1)
        at = 0
        for j, (rows, _) in enumerate(_LAYERS):
            w, b = p[at:at + rows * 64].view(rows, 64), p[at + rows * 64:at + rows * 65]
            at += rows * 65
            h = h @ w.T + b
            h = h.relu() if j < 3 else h
        h = h.view(-1, 8, 5)
        mu = torch.nn.functional.normalize(h[:, :, 0:3] - x[:, None], dim=-1)
        kappa = (0.05 + torch.nn.functional.softplus(h[:, :, 3])).clamp(max=2000.0)
        logv = kappa.log() - math.log(2 * math.pi) - torch.log1p(-torch.exp(-2 * kappa)) \
            + kappa * ((mu * s[:, None, 8:11]).sum(-1) - 1)
        loss = -(s[:, 3] * torch.logsumexp(torch.log_softmax(h[:, :, 4], 1) + logv, 1)).sum() / n
        loss.backward()
        total += float(loss.detach())
    return {"loss": total, "grad": p.grad}


# The lobes in 64 bits, in the local frame (y up): value times |cos(wo)| and
# the solid-angle pdf, and the sampled direction, as the path loop uses them.
def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


def _refl(wi, m):
    return 2 * _dot(wi, m)[:, None] * m - wi


def _fresnel(eta, c):
    """Unpolarised reflectance, eta = outside over inside along the incident side."""
    ct = (1 - (1 - c * c) * eta * eta).clamp(min=0).sqrt()
    rp, rs = (c - eta * ct) / (c + eta * ct), (ct - eta * c) / (ct + eta * c)
    return torch.where((1 - c * c) * eta * eta > 1, torch.ones_like(c), 0.5 * (rp * rp + rs * rs))


class _Facets:
    """A GGX or Beckmann distribution: D, Smith's Lambda, the visible-normal pdf."""

    def __init__(self, beckmann, ax, ay):
        self.beckmann, self.ax, self.ay = beckmann, ax, ay

    def D(self, m):
        x = ((m[:, 0] / self.ax) ** 2 + (m[:, 2] / self.ay) ** 2) / m[:, 1] ** 2
        v = torch.exp(-x) / math.pi if self.beckmann else 1 / (math.pi * (1 + x) ** 2)
        return v / (m[:, 1] ** 4 * self.ax * self.ay)

    def lam(self, w):
        a = ((w[:, 0] * self.ax) ** 2 + (w[:, 2] * self.ay) ** 2).sqrt() / w[:, 1].abs()
        if not self.beckmann:
            return 0.5 * ((1 + a * a).sqrt() - 1)
        a = 1 / a
        return torch.where(a < 1.6, (1 - 1.259 * a + 0.396 * a * a) / (3.535 * a + 2.181 * a * a), torch.zeros_like(a))

    def pdf(self, wi, m):
        return _dot(wi, m).abs() * self.D(m) / ((1 + self.lam(wi)) * wi[:, 1].abs())

    def sample(self, wi, u1, u2):
        if not self.beckmann:
            v = _unit(torch.stack([self.ax * wi[:, 0], self.ay * wi[:, 2], wi[:, 1]], -1))
            t1 = torch.stack([-v[:, 1], v[:, 0], torch.zeros_like(u1)], -1)
            t1 = t1 / t1.norm(dim=-1, keepdim=True)
            t2 = torch.linalg.cross(v, t1)
            r, phi = u1.sqrt(), 2 * math.pi * u2
            a, s = r * phi.cos(), 0.5 * (1 + v[:, 2])
            b = (1 - s) * (1 - a * a).sqrt() + s * r * phi.sin()
            h = t1 * a[:, None] + t2 * b[:, None] + v * (1 - a * a - b * b).clamp(min=0).sqrt()[:, None]
            return _unit(torch.stack([self.ax * h[:, 0], h[:, 2].clamp(min=0), self.ay * h[:, 1]], -1))
        ws = _unit(torch.stack([wi[:, 0] * self.ax, wi[:, 1], wi[:, 2] * self.ay], -1))
        ct = ws[:, 1]
        st = (1 - ct * ct).clamp(min=0).sqrt()
        steep = ct > 0.99999
        c = torch.where(steep, torch.full_like(ct, 0.99999), ct)
        s = torch.where(steep, (1 - c * c).sqrt(), st)
        tan, cot = s / c, c / s
        top, k = torch.erf(cot), tan / math.sqrt(math.pi)
        z = 1 + top + k * torch.exp(-cot * cot)
        uu = u1.clamp(1e-7, 1 - 1e-7)
        lo, hi = torch.full_like(top, -1.0), top.clone()
        for _ in range(80):  # the visible slope's distribution, inverted by bisection
            mid = 0.5 * (lo + hi)
            e = torch.erfinv(mid.clamp(-1 + 1e-16, 1 - 1e-16))
            above = (1 + mid + k * torch.exp(-e * e)) / z > uu
            lo, hi = torch.where(above, lo, mid), torch.where(above, mid, hi)
        sx, sy = torch.erfinv(0.5 * (lo + hi)), torch.erfinv(2 * u2.clamp(1e-7, 1 - 1e-7) - 1)
        r, phi = (-torch.log((1 - u1).clamp(min=1e-12))).sqrt(), 2 * math.pi * u2
        sx, sy = torch.where(steep, r * phi.cos(), sx), torch.where(steep, r * phi.sin(), sy)
        phi = torch.atan2(ws[:, 2], ws[:, 0])
        rx, ry = phi.cos() * sx - phi.sin() * sy, phi.sin() * sx + phi.cos() * sy
        return _unit(torch.stack([-rx * self.ax, torch.ones_like(rx), -ry * self.ay], -1))


def _facets(kind, p):
    if kind in (3, 4, 5, 6):
        return _Facets(kind in (4, 6), p[:, 7], p[:, 8]), p[:, 9]
    return _Facets(False, p[:, 3], p[:, 4]) if kind == 7 else _Facets(False, p[:, 6], p[:, 7]), p[:, 8]


def _walter_g1(m, v, alpha):
    b = v[:, 1] / (alpha * (1 - v[:, 1] ** 2).clamp(min=0).sqrt())
    g = (3.535 * b + 2.181 * b * b) / (1 + 2.276 * b + 2.577 * b * b)
    return torch.where(_dot(v, m) / v[:, 1] <= 0, torch.zeros_like(b), torch.where(b >= 1.6, torch.ones_like(b), g))


def _value(kind, p, wi, wo):
    """(f * |cos wo| (n, 3), pdf) of one kind."""
    n = len(p)
    zero = torch.zeros(n, device=p.device, dtype=torch.float64)
    ci, co = wi[:, 1], wo[:, 1]
    both = (ci > 0) & (co > 0)
    h = _unit(wi + wo)
    cd = _dot(wo, h)
    grey = lambda v: v[:, None].expand(-1, 3)  # noqa: E731
    if kind == 0:
        f = co.clamp(min=0) / math.pi
        return grey(f), f
    if kind in (1, 2, 12, 13, 14):
        return grey(zero), zero
    if kind in (3, 4, 7, 8):
        mf, eta = _facets(kind, p)
        d = mf.D(h)
        g = 1 / (1 + mf.lam(wi) + mf.lam(wo))
        pdf = mf.pdf(wi, h) / (4 * cd.abs())
        if kind == 7:
            f = (d * g / (4 * ci * co))[:, None] * (p[:, 0:3] + (1 - p[:, 0:3]) * ((1 - cd) ** 5)[:, None])
        elif kind == 8:
            r0 = ((1 - eta) / (1 + eta)) ** 2
            s = (r0 + (1 - r0) * (1 - cd) ** 5)[:, None]
            f = ((d.clamp(max=4) * g / (4 * ci * co))[:, None] * (p[:, 0:3] + (1 - p[:, 0:3]) * s)).clamp(max=1)
        else:
            f = grey(d * g * _fresnel(eta, cd) / (4 * ci * co))
        return torch.where(both[:, None], f * co[:, None], zero[:, None]), torch.where(both, pdf, zero)
    if kind in (5, 6):
        mf, eta = _facets(kind, p)
        eta = torch.where(ci < 0, 1 / eta, eta)
        same = ci * co >= 0
        m = torch.where(same[:, None], h, _unit(wi + eta[:, None] * wo))
        m = torch.where((~same & (m[:, 1] < 0))[:, None], -m, m)
        cmi, cmo = _dot(wi, m), _dot(wo, m)
        F, D, G = _fresnel(eta, cmi), mf.D(m), 1 / (1 + mf.lam(wi) + mf.lam(wo))
        den = cmi + eta * cmo
        refl_f, refl_p = F * D * G / (4 * ci * co).abs(), mf.pdf(wi, m) / (4 * cmi.abs())
        # the transmitted value carries its denominator to the fourth power
        tran_f = (cmi * cmo / (ci * co)).abs() * D * G * (1 - F) * eta ** 2 / den ** 4
        tran_f = torch.where(den ** 2 < 1e-6, zero, tran_f)
        tran_p = torch.where(den.abs() < 1e-6, zero, cmo.abs() * (eta / den) ** 2 * mf.pdf(wi, m))
        f = torch.where(same, refl_f, tran_f) * co.abs()
        return grey(f), torch.where(same, refl_p * F, tran_p * (1 - F))
    if kind == 9:
        e = p[:, 3]
        c = _dot(_refl(wi, torch.tensor([[0.0, 1.0, 0.0]], device=p.device).double().expand(n, 3)), wo)
        lobe = c.clamp(min=0) ** e / (2 * math.pi)
        ok = both & (c > 0)
        return grey(torch.where(ok, (e + 2) * lobe * co, zero)), torch.where(ok, (e + 1) * lobe, zero)
    if kind in (10, 11):
        ax, ay = p[:, 6], p[:, 7]
        k = torch.exp(-((h[:, 0] / ax) ** 2 + (h[:, 2] / ay) ** 2) / h[:, 1] ** 2) / (4 * math.pi * ax * ay)
        f = torch.where(both, k * co / (ci * co).clamp(min=1e-300).sqrt(), zero)
        return grey(f), torch.where(both, k / (_dot(h, wi) * h[:, 1] ** 3), zero)
    if kind == 15:
        f = torch.where(ci * co < 0, co.abs() / math.pi, zero)
        return grey(f), f
    if kind == 16:
        al, kd = p[:, 0], p[:, 3]
        c, s2 = h[:, 1], 1 - h[:, 1] ** 2
        D = torch.exp(-(s2 / c ** 2) / al ** 2) / (math.pi * al ** 2 * c ** 3)
        F = _fresnel(p[:, 2] / p[:, 1], cd)
        G = _walter_g1(h, wi, al) * _walter_g1(h, wo, al)
        f = (kd / math.pi + (1 - kd) * D * F * G / (4 * ci * co * c)) * co
        return grey(torch.where(both, f, zero)), torch.where(both, (1 - kd) * D / (4 * cd) + kd * co / math.pi, zero)
    pdf = torch.where(both, co / math.pi, zero)
    fl, fv = (1 - co) ** 5, (1 - ci) ** 5
    if kind == 17:
        f = (1 - 0.5 * fl) * (1 - 0.5 * fv) / math.pi * co
    elif kind == 18:
        rr = 2 * p[:, 3] * cd * cd
        f = rr * (fl + fv + fl * fv * (rr - 1)) / math.pi * co
    elif kind == 19:
        f = p[:, 3] * (1 - cd) ** 5 * co
    else:
        a2 = p[:, 3] ** 2
        D = (a2 - 1) / (math.pi * a2.log() * (1 + (a2 - 1) * h[:, 1] ** 2))
        g1 = lambda c: 2 / (1 + (1 + 0.0625 * (1 - c * c) / (c * c)).sqrt())  # noqa: E731
        f = 0.25 * D * (0.04 + 0.96 * (1 - cd) ** 5) * g1(ci) * g1(co) / (4 * ci)
        pdf = torch.where(both, D * h[:, 1] / (4 * cd), zero)
    return grey(torch.where(both, f, zero)), pdf


def _refract(wi, up, eta):
    """Transmission of wi through the surface whose unit normal `up` lies on
    wi's side, eta = this side over the other; the second result says whether there is any."""
    c = _dot(wi, up)
    c2 = 1 - (1 - c * c) * eta * eta
    return -eta[:, None] * wi + (eta * c - c2.clamp(min=0).sqrt())[:, None] * up, c2 > 0


def _sampled(kind, p, wi, u):
    """(wo, valid, delta) of one kind."""
    n, ci = len(p), wi[:, 1]
    y = torch.tensor([[0.0, 1.0, 0.0]], device=p.device).double().expand(n, 3)
    side = torch.where(ci < 0, -1.0, 1.0)[:, None].double()
    yes = torch.ones(n, device=p.device, dtype=torch.bool)
    u0, u1, u2 = u[:, 0], u[:, 1], u[:, 2]
    polar = lambda st, ct, phi: torch.stack([st * phi.cos(), ct, st * phi.sin()], -1)  # noqa: E731
    cosine = polar(u0.sqrt(), (1 - u0).clamp(min=0).sqrt(), 2 * math.pi * u1)
    if kind in (0, 15, 17, 18, 19):
        return (cosine * torch.stack([torch.ones_like(ci), -side[:, 0], torch.ones_like(ci)], -1) if kind == 15
                else cosine), yes, False
    if kind in (1, 12):
        return _refl(wi, y), yes if kind == 1 else ci > 0, True
    if kind == 2:
        eta = torch.where(ci > 0, p[:, 1] / p[:, 0], p[:, 0] / p[:, 1])
        F = _fresnel(eta, ci.abs())
        t, ok = _refract(wi, y * side, eta)
        return torch.where((u0 < F)[:, None], _refl(wi, y), t), (u0 < F) | ok, True
    if kind == 13:
        t, ok = _refract(wi, y * side, torch.where(ci < 0, p[:, 3], 1 / p[:, 3]))
        return torch.where(ok[:, None], t, torch.zeros_like(t)), ok, True
    if kind == 14:
        return -wi, yes, True
    if kind in (3, 4, 7, 8):
        wo = _refl(wi, _facets(kind, p)[0].sample(wi, u0, u1))
        return wo, (ci > 0) & (wo[:, 1] > 0), False
    if kind in (5, 6):
        mf, eta = _facets(kind, p)
        eta = torch.where(ci < 0, 1 / eta, eta)
        m = mf.sample(wi * side, u0, u1)
        c = _dot(m, wi)
        reflect = u2 < _fresnel(eta, c)
        e = torch.where(c < 0, 1 / eta, eta)
        c2 = 1 - (1 - c * c) * e * e
        t = m * (-c * e + torch.where(c >= 0, 1.0, -1.0) * c2.clamp(min=0).sqrt())[:, None] + wi * e[:, None]
        t = torch.where((c2 > 0)[:, None], t, torch.zeros_like(t))
        wo = torch.where(reflect[:, None], _refl(wi, m), t / t.norm(dim=-1, keepdim=True).clamp(min=1e-300))
        same = ci * wo[:, 1] > 0
        return wo, torch.where(reflect, same, (c2 > 0) & ~same), False
    if kind == 9:
        R = _refl(wi, y)
        sg = torch.where(R[:, 2] >= 0, 1.0, -1.0).double()
        a = -1 / (sg + R[:, 2])
        b = R[:, 0] * R[:, 1] * a
        b1 = torch.stack([1 + sg * R[:, 0] ** 2 * a, sg * b, -sg * R[:, 0]], -1)
        b2 = torch.stack([b, sg + R[:, 1] ** 2 * a, -R[:, 1]], -1)
        ct = u1 ** (1 / (p[:, 3] + 1))
        st, phi = (1 - ct * ct).clamp(min=0).sqrt(), 2 * math.pi * u0
        wo = b1 * (st * phi.cos())[:, None] + b2 * (st * phi.sin())[:, None] + R * ct[:, None]
        return wo, (ci > 0) & (wo[:, 1] > 0), False
    phi = 2 * math.pi * u0
    if kind in (10, 11):
        px, pz = p[:, 6] * phi.cos(), p[:, 7] * phi.sin()
        k = (px * px + pz * pz).sqrt()
        px, pz = px / k, pz / k
        t = (-torch.log1p(-u1) / ((px / p[:, 6]) ** 2 + (pz / p[:, 7]) ** 2)).sqrt()
        ct = 1 / (1 + t * t).sqrt()
        wo = _refl(wi, torch.stack([t * ct * px, ct, t * ct * pz], -1))
    elif kind == 16:
        t = (-p[:, 0] ** 2 * torch.log1p(-u1)).sqrt()
        ct = 1 / (1 + t * t).sqrt()
        wo = torch.where((u2 >= 1 - p[:, 3])[:, None], cosine, _refl(wi, polar(t * ct, ct, phi)))
    else:
        a2 = p[:, 3] ** 2
        ct = ((1 - a2 ** (1 - u1)) / (1 - a2)).clamp(min=0).sqrt()
        wo = _refl(wi, polar((1 - ct * ct).clamp(min=0).sqrt(), ct, phi))
    return wo, (ci > 0) & (wo[:, 1] > 0), False


def _exact_closures(kind, lobes, wi, wo, u):
    p, wi, wo, u = _f64(lobes["params"]), _f64(wi), _f64(wo), _f64(u)
    n = len(kind)
    z = lambda *s: torch.zeros(s, device=p.device, dtype=torch.float64)  # noqa: E731
    out = {"f": z(n, 3), "pdf": z(n), "s_wo": z(n, 3), "s_weight": z(n, 3), "s_pdf": z(n), "s_flags": None}
    for k in range(21):
        at = torch.from_numpy(np.flatnonzero(kind == k)).to(p.device)
        if not len(at):
            continue
        pk, ik = p[at], wi[at]
        out["f"][at], out["pdf"][at] = _value(k, pk, ik, wo[at])
        w, valid, delta = _sampled(k, pk, ik, u[at])
        f, pdf = _value(k, pk, ik, w)
        valid = valid & (delta | (pdf > 0))
        # a lobe that takes no light from below returns no direction there
        above = (ik[:, 1] > 0) | (k not in (3, 4, 7, 8, 9, 10, 11, 12, 16, 20))
        out["s_wo"][at] = torch.where(above[:, None], w, torch.zeros_like(w))
        out["s_weight"][at] = torch.where(valid[:, None], torch.ones_like(f) if delta else f / pdf[:, None], torch.zeros_like(f))
        out["s_pdf"][at] = torch.where(valid, pdf, torch.zeros_like(pdf))
    return out
