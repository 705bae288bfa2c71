"""What a user of this library has it do, as cases that can be timed: renders
in the plain and the wavefront form from previews to full frames, a batch of
subsurface and media scenes, black-hole and wormhole images, geodesic and
closest-hit queries on ray batches, gradients of an image loss and Metropolis
light transport.  The scenes are the library's own seeded builders; a case's
seed moves its meshes, media, albedos, rays and random streams.

A case is a dict with "kind" (what is called) and the kind's sizes; images
come back whole as the calls return them."""
import math

import numpy as np
import torch

from prender_gb300 import _abi as A
from prender_gb300 import gpu, scenes
from prender_gb300.scene import Camera, Material, RenderSettings, Scene

MODES = {"plain": A.PR_MODE_MEGAKERNEL, "wavefront": A.PR_MODE_WAVEFRONT}

# path segments (extension and shadow rays) per camera path, as the renderer
# counts them on these scenes; a segment takes about SEGMENT_FLOPS: some three
# wide nodes of eight boxes, two triangles and its share of the shading
SEGMENTS = {"spheres": 9, "diffuse": 29, "glass": 41, "phong": 29, "ward": 29, "media": 34}
SEGMENT_FLOPS = 700
# one Cash-Karp attempt: five geodesic evaluations and the step's combinations
STEP_FLOPS = 630


def listed():
    return [
        # a thumbnail of the sphere Cornell box in the default (plain) form: the smallest call, all latency
        {"name": "preview_spheres", "kind": "render", "scene": "spheres", "form": "plain", "width": 64, "height": 48,
         "samples": 1, "supersamples": 2},
        # the edupt sphere scene at its usual size, as `prender scene.txt` renders it (plain form, no next-event estimation)
        {"name": "spheres_plain", "kind": "render", "scene": "spheres", "form": "plain", "width": 256, "height": 192,
         "samples": 4, "supersamples": 2},
        # a triangle mesh with next-event estimation in the plain form, odd image sides
        {"name": "mesh_plain", "kind": "render", "scene": "diffuse", "form": "plain", "width": 321, "height": 243,
         "samples": 4, "supersamples": 2, "subdiv": 5},
        # the full frame of the benchmark: 1024 x 768, 64 samples a pixel, 327,680 triangles, wavefront form
        {"name": "mesh_wavefront", "kind": "render", "scene": "diffuse", "form": "wavefront", "width": 1024,
         "height": 768, "samples": 16, "supersamples": 2, "subdiv": 7},
        # a glass mesh (paths split in branches) at draft quality, wavefront form
        {"name": "glass_wavefront", "kind": "render", "scene": "glass", "form": "wavefront", "width": 512,
         "height": 384, "samples": 4, "supersamples": 2, "subdiv": 6},
        # many variants in one call: media around a subsurface (directional dipole) mesh, uneven sizes
        {"name": "media_batch", "kind": "batch", "form": "wavefront", "jobs": 6, "side_min": 96, "side_max": 320,
         "samples": 4, "supersamples": 2, "subdiv": 5},
        # black-hole frames at two spins with a textured accretion disk, mixed precision, one batch
        {"name": "kerr_frames", "kind": "kerr_frames", "jobs": 2, "width": 512, "height": 256, "max_steps": 4000},
        # the reference-arithmetic FP64 geodesics of a camera's rays
        {"name": "kerr_trace", "kind": "kerr_trace", "spin": 0.6, "width": 192, "height": 96, "max_steps": 4000},
        # a wormhole view with objects on both sides, FP64 geodesics
        {"name": "wormhole", "kind": "wormhole", "width": 128, "height": 96, "supersamples": 2, "max_steps": 300},
        # the backward direction: d(loss)/d(albedo, emission) of an image of eight materials
        {"name": "adjoint", "kind": "adjoint", "width": 256, "height": 256, "samples": 4, "supersamples": 2,
         "subdiv": 5},
        # Metropolis light transport on the sphere Cornell box with next-event estimation
        {"name": "metropolis", "kind": "metropolis", "width": 96, "height": 72, "samples": 8, "mutation": 16.0},
        # bit-exact closest hits of a batch of random rays in a mesh scene
        {"name": "first_hit", "kind": "first_hit", "rays": 262144, "subdiv": 5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render"] * 6 + ["batch", "kerr_frames", "kerr_trace", "wormhole", "adjoint", "metropolis",
                                        "first_hit"])
    if kind == "render":
        form = rng.choice(["plain", "wavefront"])
        scene = rng.choice(["spheres", "diffuse", "diffuse", "glass", "phong", "ward", "media"])
        c = {"kind": kind, "scene": scene, "form": form, "width": _log(rng, 48, 800)}
        c["height"] = max(33, int(c["width"] * rng.uniform(0.55, 1.0)))
        c["supersamples"] = rng.choice([1, 2, 2])
        # camera samples: up to 1.2 M in the plain form, 5 M in the wavefront form
        most = (1.2e6 if form == "plain" else 5.0e6) / (c["width"] * c["height"] * c["supersamples"] ** 2)
        c["samples"] = max(1, min(rng.choice([1, 2, 4, 16]), int(most)))
        if scene != "spheres":
            c["subdiv"] = rng.randint(3, 7)
        return c
    if kind == "batch":
        lo = _log(rng, 32, 128)
        return {"kind": kind, "form": rng.choice(["wavefront", "wavefront", "plain"]), "jobs": rng.randint(2, 7),
                "side_min": lo, "side_max": lo + rng.randint(1, 120), "samples": rng.choice([1, 2, 4]),
                "supersamples": 2, "subdiv": rng.randint(3, 5)}
    if kind == "kerr_frames":
        w = _log(rng, 64, 512)
        return {"kind": kind, "jobs": rng.randint(1, 3), "width": w, "height": max(32, w // 2 + rng.randint(-3, 3)),
                "max_steps": rng.choice([2000, 4000])}
    if kind == "kerr_trace":
        w = _log(rng, 48, 256)
        return {"kind": kind, "spin": rng.choice([0.0, 0.3, 0.6, 0.9, 0.999]), "width": w,
                "height": max(24, w // 2 + rng.randint(-3, 3)), "max_steps": rng.choice([500, 2000, 4000])}
    if kind == "wormhole":
        w = _log(rng, 32, 160)
        return {"kind": kind, "width": w, "height": max(24, int(w * rng.uniform(0.6, 0.9))),
                "supersamples": rng.choice([1, 2]), "max_steps": rng.choice([150, 300])}
    if kind == "adjoint":
        w = _log(rng, 64, 256)
        return {"kind": kind, "width": w, "height": max(48, w - rng.randint(0, 17)), "samples": rng.choice([1, 2, 4]),
                "supersamples": 2, "subdiv": rng.randint(3, 5)}
    if kind == "metropolis":
        w = _log(rng, 32, 128)
        return {"kind": kind, "width": w, "height": max(24, int(0.75 * w)), "samples": rng.randint(2, 8),
                "mutation": rng.choice([4.0, 8.0, 16.0])}
    return {"kind": kind, "rays": _log(rng, 1000, 400000) | 1, "subdiv": rng.randint(3, 6)}


class State:
    """A context with an uploaded scene (or scene objects) and the call's
    other inputs; gives its GPU memory back when dropped."""

    def __init__(self, kind):
        self.kind = kind
        self.ctx = gpu.Context(0)
        self.objs = []

    def __del__(self):
        for o in getattr(self, "objs", []):
            o.release()
        if hasattr(self, "ctx"):
            self.ctx.close()


def _render_scene(c, seed):
    w, h, n, ss = c["width"], c["height"], c["samples"], c["supersamples"]
    if c["scene"] == "spheres":
        s = scenes.cornell_spheres(w, h, n, ss, seed=seed)
    elif c["scene"] == "media":
        rng = np.random.default_rng(seed)
        s = scenes.media_cornell(w, h, n, ss, sigma_s=float(rng.uniform(0.02, 0.1)), g=float(rng.uniform(-0.3, 0.6)),
                                 subdiv=c["subdiv"], seed=seed)
    else:
        s = scenes.mesh_cornell(w, h, n, ss, subdiv=c["subdiv"], material=c["scene"], seed=seed)
    s.settings.mode = MODES[c["form"]]
    return s


def _batch_scenes(c, seed):
    sides = sorted({c["side_min"] + (c["side_max"] - c["side_min"]) * k // 4 for k in range(5)})
    ss = scenes.media_batch(n=c["jobs"], seed=seed, sizes=sides, samples=c["samples"], supersamples=c["supersamples"],
                            subdiv=c["subdiv"])
    # the sides of the batch are the case's, not the seed's
    for k, s in enumerate(ss):
        s.camera.width = s.camera.height = sides[(3 * k + 1) % len(sides)]
        s.settings.mode = MODES[c["form"]]
    return ss


def _kerr_scenes(c, seed):
    out = []
    for j in range(c["jobs"]):
        s = scenes.kerr_accretion(a=(0.6, 0.999)[j % 2], width=c["width"], height=c["height"],
                                  max_steps=c["max_steps"], precision=A.PR_KERR_FP32,
                                  texture=scenes.celestial_texture(1024, 512, stars=10000, seed=seed),
                                  disk_texture=scenes.accretion_texture(512, 512, seed=seed), disk_seed=seed + 1)
        s.settings.seed = seed
        s.settings.tent_filter = 1
        out.append(s)
    return out


def _sky(h, w, rng, base):
    y, x = np.mgrid[0:h, 0:w]
    img = np.zeros((h, w, 3))
    img[..., 0] = base[0] + 60 * np.sin(x * 6.2832 / w * 4)
    img[..., 1] = base[1] + 60 * np.cos(y * 6.2832 / h * 3)
    img[..., 2] = base[2] + 40 * ((x // 8 + y // 8) % 2)
    return np.clip(img + rng.integers(-10, 11, (h, w, 3)), 0, 255).astype(np.uint8)


def _wormhole_scene(c, seed):
    rng = np.random.default_rng(seed)
    s = Scene()
    s.camera = Camera(position=(0.0, 0.5, 12.0), dir=(0.0, -0.02, -1.0), up=(0.0, 1.0, 0.0), angle=60,
                      width=c["width"], height=c["height"])
    s.settings = RenderSettings(samples=1, supersamples=c["supersamples"], tent_filter=1, depth=4, nee=0, seed=seed)
    out = (0.0, 0.0, 3.0e6)
    s.set_wormhole((0.0, 0.0, 0.0), out, rho=1.3, a=0.5, w=0.05, max_steps=c["max_steps"],
                   textures=(_sky(64, 128, rng, (120, 140, 200)), _sky(64, 128, rng, (200, 120, 60))),
                   texture_coef=(1.0, 1.5))
    s.add_sphere((3.5, 0.0, -3.0), 1.0, Material.diffuse((0.1, 0.1, 0.1), (2.0, 1.5, 0.5)))
    s.add_sphere((-3.0, -1.5, 1.0), 1.2, Material.diffuse((0.7, 0.7, 0.7)))
    s.add_sphere((out[0] + 1.5, out[1], out[2] - 4.0), 1.0, Material.diffuse((0.1, 0.1, 0.1), (0.5, 2.0, 1.0)))
    s.add_sphere((out[0] - 2.0, out[1] + 1.0, out[2] - 6.0), 1.5, Material.mirror((0.9, 0.9, 0.9)))
    return s


def _hit_scene(c, seed):
    return scenes.mesh_cornell(64, 48, 1, 1, subdiv=c["subdiv"], seed=seed)


def _hit_rays(c, seed):
    """half the rays anywhere in the box, half aimed at the icosphere"""
    n = c["rays"]
    v = _hit_scene(c, seed).meshes[1].vertices
    lo, hi = (2, 1, 1), (98, 80, 249)
    return np.concatenate([scenes.random_rays(lo, hi, n - n // 2, seed=seed),
                           scenes.rays_toward(v, lo, hi, n // 2, seed=seed + 1)])


def prepare(case, seed):
    c = case
    st = State(c["kind"])
    if c["kind"] in ("batch", "kerr_frames"):
        ss = _batch_scenes(c, seed) if c["kind"] == "batch" else _kerr_scenes(c, seed)
        st.objs = [st.ctx.scene_object(s) for s in ss]
        st.outs = [torch.empty((s.camera.height, s.camera.width, 3), dtype=torch.float32, device="cuda:0") for s in ss]
        st.jobs = list(zip(st.objs, st.outs))
        return st
    if c["kind"] == "render":
        st.scene = _render_scene(c, seed)
    elif c["kind"] == "kerr_trace":
        st.scene = scenes.kerr_lensing(a=c["spin"], width=c["width"], height=c["height"], max_steps=c["max_steps"])
        st.rays = scenes.camera_rays(st.scene, jitter_seed=seed + 1)
    elif c["kind"] == "wormhole":
        st.scene = _wormhole_scene(c, seed)
    elif c["kind"] == "adjoint":
        st.scene = scenes.diff_cornell(c["width"], c["height"], c["samples"], c["supersamples"], subdiv=c["subdiv"],
                                       seed=seed)
        # d(loss)/d(image) of a squared difference from a target: signed, of the image's own size
        rng = np.random.default_rng(seed + 1)
        st.dl = rng.normal(scale=0.1, size=(c["height"], c["width"], 3)).astype(np.float32)
    elif c["kind"] == "metropolis":
        st.scene = scenes.cornell_spheres(c["width"], c["height"], c["samples"], 1, seed=seed)
        s = st.scene.settings
        s.mode, s.mutation, s.pre_sample, s.nee = A.PR_MODE_MLT, c["mutation"], 0.4, 1
    else:
        st.scene = _hit_scene(c, seed)
        st.rays = _hit_rays(c, seed)
    st.ctx.upload(st.scene)
    if c["kind"] == "first_hit":
        st.ctx.qbvh(2)  # the exact trees, which the context builds once per scene on their first use
    return st


def run(state):
    if state.kind in ("batch", "kerr_frames"):
        state.ctx.render_batch(state.jobs)
        return state.outs
    if state.kind == "kerr_trace":
        return state.ctx.kerr_trace(state.rays)
    if state.kind == "adjoint":
        return state.ctx.render_adjoint(state.dl)
    if state.kind == "first_hit":
        return state.ctx.first_hit(state.rays)
    return state.ctx.render()


def work(case):
    """Image, rays, results and the scene's triangles once; the arithmetic from
    the segments or steps that the scenes take per path or ray."""
    c = case
    tris = 20 * 4 ** c.get("subdiv", 0)
    scene_bytes = 48 * tris + 80 * tris // 5
    px = c.get("width", 0) * c.get("height", 0)
    if c["kind"] == "render":
        paths = px * c["samples"] * c["supersamples"] ** 2
        return {"bytes": 12 * px + (0 if c["scene"] == "spheres" else scene_bytes),
                "flops": paths * SEGMENTS[c["scene"]] * SEGMENT_FLOPS}
    if c["kind"] == "batch":
        px = sum(s.camera.width ** 2 for s in _batch_scenes(dict(c, subdiv=0), 0))
        paths = px * c["samples"] * c["supersamples"] ** 2
        return {"bytes": 12 * px + c["jobs"] * scene_bytes, "flops": paths * 36 * SEGMENT_FLOPS}
    if c["kind"] == "kerr_frames":  # near the hole some 60 FP64 steps, then FP32 ones
        return {"bytes": c["jobs"] * (12 * px + 3 * 1024 * 512 + 4 * 512 * 512),
                "flops": c["jobs"] * px * 0.12 * c["max_steps"] * STEP_FLOPS}
    if c["kind"] == "kerr_trace":  # about a fifth of the rays escape and run all their steps
        return {"bytes": px * (48 + 72), "flops": px * 0.18 * c["max_steps"] * STEP_FLOPS}
    if c["kind"] == "wormhole":
        return {"bytes": 12 * px, "flops": px * c["supersamples"] ** 2 * 0.8 * c["max_steps"] * STEP_FLOPS}
    if c["kind"] == "adjoint":
        paths = px * c["samples"] * c["supersamples"] ** 2
        return {"bytes": 12 * px + scene_bytes, "flops": paths * 30 * SEGMENT_FLOPS}
    if c["kind"] == "metropolis":
        return {"bytes": 12 * px, "flops": px * c["samples"] * (c["mutation"] + 0.4) * 25 * SEGMENT_FLOPS}
    return {"bytes": c["rays"] * (48 + 16) + scene_bytes, "flops": c["rays"] * 6000}


def exact(case, seed):
    """Closest hits by brute force over every triangle in 64 bits.  The other
    kinds have no such value within reach: a path's or a geodesic's branches
    (roulette, light choice, step control, capture) follow the arithmetic of
    the tracer, and thousands of serial steps a ray take minutes this way."""
    if case["kind"] != "first_hit":
        return None
    dev = "cuda:0"
    s = _hit_scene(case, seed)
    rays = torch.from_numpy(_hit_rays(case, seed)).to(dev)
    d = rays[:, 3:]
    o = rays[:, :3] + 1.0e-6 * d  # distances count from the origin pushed 1e-6 along the ray
    best = torch.full((len(rays),), math.inf, dtype=torch.float64, device=dev)
    cross, dot = torch.linalg.cross, lambda a, b: (a * b).sum(-1)  # noqa: E731
    for m in s.meshes:
        tri = torch.from_numpy(np.asarray(m.vertices, np.float32)[np.asarray(m.faces)].astype(np.float64)).to(dev)
        v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
        n = cross(e1, e2)
        w = cross(v0, e1), cross(e2, v0)
        step = max(1, 12_000_000 // len(tri))
        for i in range(0, len(rays), step):
            oi, di = o[i:i + step], d[i:i + step]
            m_ = cross(oi, di)  # the ray's moment: u, v and t as products of ray and triangle vectors
            det = -(di @ n.T)
            t = (oi @ n.T - dot(n, v0)) / det
            u = (m_ @ e2.T - di @ w[1].T) / det
            v = (-(m_ @ e1.T) - di @ w[0].T) / det
            bad = (det.abs() <= 1.0e-7) | (u < 0) | (v < 0) | (u + v > 1) | ~(t > 1.0e-6)
            best[i:i + step] = torch.minimum(best[i:i + step], t.masked_fill_(bad, math.inf).amin(1))
    for e in s.entities:
        if e.type != A.PR_ENT_UVPLANE:
            continue
        p, U, V = (torch.tensor(x, dtype=torch.float64, device=dev) for x in (e.p, e.u, e.v))
        n = cross(U, V)
        n = n / n.norm()
        t = ((p - o) @ n) / (d @ n)
        rel = o + t[:, None] * d - p
        lu, lv = U.norm(), V.norm()
        u, v = rel @ U / lu / lu, rel @ V / lv / lv  # the plane's extent rule: coordinate / length against the length
        bad = (u < 0) | (u > lu) | (v < 0) | (v > lv) | ~(t >= 1.0e-6)
        best = torch.minimum(best, t.masked_fill(bad, math.inf))
    best = torch.where(torch.isinf(best), torch.full_like(best, -1.0), best)
    return {"entity": None, "prim": None, "t": best.cpu().numpy()}
