"""The work whose speed this library is judged by, as a caller's program does it.

A case is one call (or the few calls that belong together) through the public
entry points of xyz_b200.api and xyz_b200.diff.  The listed cases run from an
interactive preview and a few thousand rays, where launches and latency count,
to the large-mesh render; the sizes are those of the benchmark's workloads and
of the tests.  `draw` gives other sizes of the same ranges, odd ones among them.
"""

import functools
import math

import numpy as np
import torch

from xyz_b200 import api, diff, scenes

ROOM_CAMERA = ((0.0, 1.5, 1.2), (0.0, 1.1, -2.0), 60.0)  # the guiding workload's view
GUIDE_LAYERS = (192, 64, 64, 64, 64)


def listed():
    return [
        # a picking or visibility query of a host program: a few thousand rays, latency only
        {"name": "hits_small", "kind": "hits", "level": 0, "rays": 4096},
        # batch closest hit on the 1M-triangle mesh: half camera rays, half cosine bounces from their hits
        {"name": "hits_mesh", "kind": "hits", "level": 7, "rays": 4194304},
        # an interactive preview frame: 64 x 64, 1 sample, mirror and metal boxes, thin lens, default depth
        {"name": "preview", "kind": "render", "scene": "specular", "level": 0, "width": 64, "height": 64, "spp": 1,
         "depth": 15, "spectral": "off"},
        # the small configuration: Cornell room, 256 x 256, 16 spp, 4 hero wavelengths in 380-720 nm, depth 8
        {"name": "cornell_spectral", "kind": "render", "scene": "cornell", "level": 0, "width": 256, "height": 256,
         "spp": 16, "depth": 8, "spectral": "continuous"},
        # the headline configuration: 984,322 triangles, 1024 x 1024, 64 spp, depth 10, leaves of at most 4
        {"name": "mesh_1m", "kind": "render", "scene": "mesh", "level": 7, "width": 1024, "height": 1024, "spp": 64,
         "depth": 10, "spectral": "off"},
        # a frame of an animation: host arrays in, tree built, film read back into host memory (247,042 triangles)
        {"name": "frame", "kind": "frame", "level": 6, "width": 517, "height": 389, "spp": 8, "depth": 10},
        # a pass of the guided tracer on the indirect-lit room, on the benchmark's 32 spread rows
        {"name": "guided", "kind": "guided", "level": 5, "wall": 32, "width": 1024, "rows": 32, "spp": 64, "depth": 10},
        # the guide's network on caller-supplied points: outputs, and the gradient of one training batch
        {"name": "guide_net", "kind": "net", "rows": 16384},
        # a differentiable-rendering step through autograd: 512 x 512, 32 spp and a 32-spp adjoint, depth 6
        {"name": "adjoint", "kind": "adjoint", "level": 4, "wall": 20, "width": 512, "height": 512, "spp": 32, "depth": 6},
        # a pass of the importance-driven tracer (the reference's own guide), 100,000 particles
        {"name": "importon", "kind": "importon", "level": 5, "wall": 32, "width": 1024, "rows": 16, "spp": 16,
         "depth": 10, "particles": 100000},
        # many scenes of uneven size in one launch
        {"name": "batch", "kind": "batch", "jobs": 8, "tris": 1000, "top_tris": 200000, "size": 128, "top_size": 512,
         "spp": 16, "depth": 8},
        # the film's way out: Radiance pixels and tone-mapped BMP rows of a full-HD frame
        {"name": "film_out", "kind": "film", "width": 1920, "height": 1080, "op": "reinhard_white"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hits", "render", "render", "render", "frame", "guided", "net", "adjoint", "importon", "batch", "film"])
    if kind == "hits":
        return {"kind": kind, "level": rng.choice([0, 3, 5, 6, 7]), "rays": _log(rng, 1000, 4000000)}
    if kind == "render":
        scene = rng.choice(["cornell", "specular", "checker", "mesh", "mesh"])
        return {"kind": kind, "scene": scene, "level": rng.randint(4, 7) if scene == "mesh" else 0,
                "width": _log(rng, 48, 1024), "height": _log(rng, 48, 1024), "spp": _log(rng, 1, 48),
                "depth": rng.randint(3, 15 if scene != "mesh" else 10),
                "spectral": "off" if scene == "specular" else rng.choice(["off", "off", "binned", "continuous"])}
    if kind == "frame":
        return {"kind": kind, "level": rng.randint(3, 7), "width": _log(rng, 64, 1024), "height": _log(rng, 64, 768),
                "spp": _log(rng, 1, 16), "depth": rng.randint(4, 10)}
    if kind == "guided":
        return {"kind": kind, "level": rng.randint(4, 6), "wall": rng.randint(8, 40), "width": _log(rng, 128, 1024),
                "rows": rng.randint(4, 32), "spp": _log(rng, 4, 64), "depth": rng.randint(4, 10)}
    if kind == "net":
        return {"kind": kind, "rows": _log(rng, 100, 65536)}
    if kind == "adjoint":
        return {"kind": kind, "level": rng.randint(2, 4), "wall": rng.randint(5, 20), "width": _log(rng, 64, 512),
                "height": _log(rng, 64, 512), "spp": _log(rng, 2, 32), "depth": rng.randint(3, 6)}
    if kind == "importon":
        return {"kind": kind, "level": rng.randint(4, 6), "wall": rng.randint(8, 40), "width": _log(rng, 128, 1024),
                "rows": rng.randint(4, 16), "spp": _log(rng, 2, 16), "depth": rng.randint(4, 10),
                "particles": _log(rng, 10000, 300000)}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(2, 12), "tris": 1000, "top_tris": _log(rng, 4000, 300000), "size": _log(rng, 64, 160),
                "top_size": _log(rng, 160, 512), "spp": _log(rng, 4, 24), "depth": rng.randint(4, 8)}
    return {"kind": kind, "width": _log(rng, 64, 3840), "height": _log(rng, 64, 2160),
            "op": rng.choice(["film", "linear", "reinhard", "reinhard_white"])}


# ------------------------------------------------------------------ scenes
@functools.lru_cache(maxsize=2)
def _mesh(level, seed):
    """The large-mesh workload's scene at a level; XYZ albedos only."""
    return scenes.spheres_scene(level=level, n_spheres=3, seed=seed % 9973)


@functools.lru_cache(maxsize=2)
def _room(level, wall, seed):
    return scenes.occluded_room(level=level, wall_n=wall, seed=seed % 9973)


def _xyz_only(sd):
    import dataclasses
    return dataclasses.replace(sd, albedo_spd=None, light_power_spd=None)


def _scene(case, seed):
    name = case.get("scene", "mesh")
    if name == "cornell":
        return scenes.cornell_box()
    if name == "specular":
        return scenes.cornell_specular(shininess=20.0 + seed % 50, pinhole=False)
    if name == "checker":
        return scenes.color_checker_room()
    sd = _mesh(case["level"], seed)
    return sd if case.get("spectral", "off") != "off" else _xyz_only(sd)


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _camera_rays(cam, n, gen):
    """n pinhole rays through random points of a square image of `cam`, as rows o.xyz, tmin, d.xyz, tmax."""
    eye = torch.tensor(cam.eye, dtype=torch.float64, device="cuda")
    fwd = torch.tensor(cam.at, dtype=torch.float64, device="cuda") - eye
    fwd = fwd / fwd.norm()
    right = torch.linalg.cross(fwd, torch.tensor([0.0, 1.0, 0.0], dtype=torch.float64, device="cuda"))
    right = right / right.norm()
    up = torch.linalg.cross(right, fwd)
    u = torch.rand((n, 2), generator=gen, device="cuda", dtype=torch.float64) - 0.5
    d = _unit(cam.film_size * (u[:, :1] * right + u[:, 1:] * up) + cam.focal_length * fwd)
    r = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    r[:, 0:3] = eye.float()
    r[:, 3] = 1e-5
    r[:, 4:7] = d.float()
    r[:, 7] = float("inf")
    return r


def _bounce_rays(sd, prim, hits, n, gen):
    """n rays that leave hit points of `prim` in cosine-weighted directions about the hit triangle's normal."""
    code = hits[:, 3].contiguous().view(torch.int32)
    hit = torch.nonzero(code >= 0)[:, 0]
    sel = hit[torch.randint(0, hit.numel(), (n,), generator=gen, device="cuda")]
    pos = torch.from_numpy(sd.positions).cuda().double()
    tri = torch.from_numpy(sd.tris).cuda().long()[(code[sel] >> 1).long()]
    a, b, c = pos[tri[:, 0]], pos[tri[:, 1]], pos[tri[:, 2]]
    ng = _unit(torch.linalg.cross(c - a, b - a))
    din = prim[sel, 4:7].double()
    ng = torch.where((ng * din).sum(1, keepdim=True) > 0, -ng, ng)
    d = _unit(ng + _unit(torch.randn((n, 3), generator=gen, device="cuda", dtype=torch.float64)))
    r = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    r[:, 0:3] = (prim[sel, 0:3].double() + hits[sel, 0:1].double() * din).float()
    r[:, 3] = 1e-5
    r[:, 4:7] = d.float()
    r[:, 7] = float("inf")
    return r


def _net_inputs(case, seed):
    """Parameters like those of a partly trained guide, points of the room, and training rows
    (point, normal, direction, weight F / q)."""
    rng = np.random.default_rng(seed)
    p = []
    for l, k in enumerate(GUIDE_LAYERS):
        scale = math.sqrt(2.0 / k) * (0.6 if l == 4 else 1.0)
        p += [rng.normal(0.0, scale, k * 64), rng.normal(0.0, 0.05, 64)]
    p = np.concatenate(p).astype(np.float32)
    n = case.get("rows", 0)
    lo, hi = np.array([-2.0, 0.0, -2.0]), np.array([2.0, 3.0, 2.0])
    nrm = rng.normal(size=(n, 3))
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    dire = rng.normal(size=(n, 3))
    dire = nrm + dire / np.linalg.norm(dire, axis=1, keepdims=True)
    dire /= np.linalg.norm(dire, axis=1, keepdims=True)
    w = rng.lognormal(-1.0, 1.0, size=(n, 1))
    rec = np.concatenate([rng.uniform(lo, hi, size=(n, 3)), nrm, dire, w], axis=1).astype(np.float32)
    return p, rec


# ------------------------------------------------------------------ state
def prepare(case, seed):
    kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if kind == "hits":
        sd = scenes.cornell_box() if case["level"] == 0 else _xyz_only(_mesh(case["level"], seed))
        s = api.Scene(sd, leaf_max_tris=4)
        n = case["rays"]
        prim = _camera_rays(sd.camera, n - n // 2, gen)
        hits = torch.empty((prim.shape[0], 4), dtype=torch.float32, device="cuda")
        s.trace_device(prim, hits)
        rays = torch.cat([prim, _bounce_rays(sd, prim, hits, n // 2, gen)]).contiguous()
        return {"kind": kind, "scene": s, "rays": rays, "hits": torch.empty((n, 4), dtype=torch.float32, device="cuda")}
    if kind == "render":
        sd = _scene(case, seed)
        return {"kind": kind, "scene": api.Scene(sd, leaf_max_tris=4), "camera": sd.camera, "case": case, "seed": seed}
    if kind == "frame":
        sd = _xyz_only(_mesh(case["level"], seed))
        film = np.zeros((case["height"], case["width"], 3), np.float32)
        return {"kind": kind, "data": sd, "film": film, "case": case, "seed": seed}
    if kind in ("guided", "importon"):
        s = api.Scene(_room(case["level"], case["wall"], seed))
        step = 1024 // case["rows"]
        state = {"kind": kind, "scene": s, "camera": scenes.Camera.with_fov(*ROOM_CAMERA, pinhole=True), "case": case,
                 "seed": seed, "rows": (step // 2, step * case["rows"], step)}
        if kind == "guided":
            state["guide"] = api.Guide(s, guide_bounces=9, train_bounces=5, seed=seed)
            state["guide"].set_params(_net_inputs({}, seed)[0])
        else:
            state["map"] = api.Importons(s, particles=case["particles"], seed=seed)
        return state
    if kind == "net":
        p, rec = _net_inputs(case, seed)
        s = api.Scene(scenes.occluded_room(level=1, wall_n=2, seed=seed % 9973))
        g = api.Guide(s)
        g.set_params(p)
        rec = torch.from_numpy(rec).cuda()
        return {"kind": kind, "guide": g, "features": rec[:, :6].contiguous(), "records": rec}
    if kind == "adjoint":
        ds = scenes.diff_scene(level=case["level"], wall_n=case["wall"], seed=seed % 9973)
        s = api.Scene(ds.scene)
        r = diff.Renderer(s, ds.scene.camera, case["width"], case["height"], case["spp"], seed=seed % (1 << 31), max_depth=case["depth"])
        target = r(torch.from_numpy(ds.target_albedo).cuda(), torch.from_numpy(ds.target_emission).cuda()).detach()
        albedo = torch.from_numpy(ds.albedo).cuda().requires_grad_()
        emission = torch.from_numpy(ds.emission).cuda().requires_grad_()
        return {"kind": kind, "renderer": r, "albedo": albedo, "emission": emission, "target": target}
    if kind == "batch":
        jobs, n = [], case["jobs"]
        for k in range(n):
            f = k / max(1, n - 1)
            tris = int(case["tris"] * (case["top_tris"] / case["tris"]) ** f)
            # sizes run against the triangle counts and back, so that neither grows with the other
            res = int(case["size"] * (case["top_size"] / case["size"]) ** (((3 * k) % n) / max(1, n - 1)))
            sd = scenes.batch_scene(2 * (seed % 9973) + k, target_tris=tris)
            jobs.append(api.BatchJob(api.Scene(sd), sd.camera, res, res, case["spp"], seed=k, max_depth=case["depth"]))
        return {"kind": kind, "batch": api.Batch(jobs), "jobs": jobs}
    # a film as a render of 16 spp leaves it: sums over a wide range of brightness, black pixels among them
    h, w = case["height"], case["width"]
    lum = torch.exp(2.0 * torch.randn((h, w, 1), generator=gen, device="cuda"))
    film = 16.0 * lum * (0.7 + 0.3 * torch.rand((h, w, 3), generator=gen, device="cuda"))
    film[torch.rand((h, w), generator=gen, device="cuda") < 0.02] = 0.0
    return {"kind": kind, "film": film.contiguous(), "op": case["op"]}


def run(state):
    kind = state["kind"]
    if kind == "hits":
        s, hits = state["scene"], state["hits"]
        s.trace_device(state["rays"], hits)
        return {"t": hits[:, 0], "f": hits[:, 1], "g": hits[:, 2], "code": hits.view(torch.int32)[:, 3]}
    if kind == "net":
        g = state["guide"]
        return {"outputs": g.forward(state["features"]),
                "gradient": g.gradient(state["records"], 1.0 / state["records"].shape[0])}
    if kind == "adjoint":
        a, e = state["albedo"], state["emission"]
        a.grad = e.grad = None
        image = state["renderer"](a, e)
        loss = ((image - state["target"]) ** 2).mean()
        loss.backward()
        return {"loss": loss.detach(), "image": image.detach(), "albedo": a.grad, "emission": e.grad}
    if kind == "batch":
        state["batch"].launch()
        return [j.film for j in state["jobs"]]
    if kind == "film":
        film = state["film"]
        return {"rgbe": api.encode_rgbe(film, 1.0 / 16.0), "bmp": api.tonemap(film, 1.0 / 16.0, op=state["op"], rgb=True)}
    c = state["case"]
    if kind == "frame":
        with api.Scene(state["data"]) as s:
            return s.render(state["data"].camera, c["width"], c["height"], c["spp"], seed=state["seed"],
                            max_depth=c["depth"], film=state["film"])
    if kind == "render":
        return state["scene"].render(state["camera"], c["width"], c["height"], c["spp"], seed=state["seed"],
                                     max_depth=c["depth"], spectral=c["spectral"])
    tracer = state["guide"] if kind == "guided" else state["map"]
    return tracer.render(state["camera"], c["width"], 1024, c["spp"], seed=state["seed"], max_depth=c["depth"],
                         rows=state["rows"])


# ------------------------------------------------------------------ work
def _tris(case):
    if case["kind"] in ("guided", "importon"):
        return 2 * 20 * 4 ** case["level"] + 14 * case["wall"] ** 2 + 50
    if case["kind"] == "adjoint":
        return 3 * 20 * 4 ** case["level"] + 10 * case["wall"] ** 2 + 32
    return 3 * 20 * 4 ** case["level"] + 1282 if case["level"] else 36


def work(case):
    """Inputs read and outputs written once; the operations of a closest-hit
    answer are taken as one triangle test (50) and of a path vertex as 200."""
    kind = case["kind"]
    if kind == "hits":
        return {"bytes": 48 * case["rays"] + 36 * _tris(case), "flops": 50 * case["rays"]}
    if kind == "net":
        # forward 54,272 operations per row, and forward, input deltas and weight gradients for a training row
        return {"bytes": case["rows"] * (24 + 256 + 40) + 3 * 4 * api.GUIDE_PARAMS, "flops": case["rows"] * 4 * 54272}
    if kind == "film":
        return {"bytes": case["width"] * case["height"] * (2 * 12 + 4 + 3), "flops": 100 * case["width"] * case["height"]}
    if kind == "batch":
        n, side = case["jobs"], case["size"] * case["top_size"]
        return {"bytes": n * (36 * case["tris"] + 12 * side), "flops": n * side * case["spp"] * 300}
    if kind in ("guided", "importon"):
        paths = case["width"] * case["rows"] * case["spp"]
        net = 54272 * 3 if kind == "guided" else 16 * 3
        return {"bytes": 84 * _tris(case) + 12 * case["width"] * case["rows"], "flops": paths * (900 + net)}
    px = case["width"] * case["height"]
    passes = 2 if kind == "adjoint" else 1
    return {"bytes": 84 * _tris(case) + 12 * px * passes, "flops": passes * px * case["spp"] * 300}


# ------------------------------------------------------------------ 64 bits
def _exact_hits(case, seed):
    """Closest hits of the small scene by testing every triangle in 64 bits."""
    sd = scenes.cornell_box()
    rays = prepare(case, seed)["rays"].double()
    pos, tri = torch.from_numpy(sd.positions).cuda().double(), torch.from_numpy(sd.tris).cuda().long()
    v0, e1, e2 = pos[tri[:, 0]], pos[tri[:, 1]] - pos[tri[:, 0]], pos[tri[:, 2]] - pos[tri[:, 0]]
    n = torch.linalg.cross(e2, e1)
    best = torch.full((rays.shape[0],), math.inf, dtype=torch.float64, device="cuda")
    bf, bg = torch.zeros_like(best), torch.zeros_like(best)
    o, d = rays[:, 0:3], rays[:, 4:7]
    for k in range(tri.shape[0]):
        det = (d * n[k]).sum(1)
        vmo = v0[k] - o
        t = (vmo * n[k]).sum(1) / det
        c = torch.linalg.cross(d, vmo)
        f, g = (c * e2[k]).sum(1) / det, -(c * e1[k]).sum(1) / det
        ok = (det.abs() > 1e-6) & (t >= rays[:, 3]) & (t < best) & (f >= 0) & (g >= 0) & (f + g <= 1)
        best, bf, bg = torch.where(ok, t, best), torch.where(ok, f, bf), torch.where(ok, g, bg)
    return {"t": torch.where(best.isinf(), 0.0, best), "f": bf, "g": bg, "code": None}


def _exact_net(case, seed):
    """The guide's network and its training gradient in 64 bits: one-blob
    encoding (32 Gaussian bins per input, zero beyond 4.5 sigma), four ReLU
    layers, and -w log p(direction) of the 8-lobe von Mises-Fisher mixture."""
    p, rec = _net_inputs(case, seed)
    sd = scenes.occluded_room(level=1, wall_n=2, seed=seed % 9973)
    with api.Scene(sd) as s:
        st = s.stats()
    lo = torch.tensor(st["bounds_min"], dtype=torch.float64, device="cuda")
    hi = torch.tensor(st["bounds_max"], dtype=torch.float64, device="cuda")
    rec = torch.from_numpy(rec).cuda().double()
    par = torch.from_numpy(p).cuda().double().requires_grad_()
    u = 32.0 * torch.cat([(rec[:, 0:3] - lo) / (hi - lo), (rec[:, 3:6] + 1.0) * 0.5], 1).clamp(0.0, 1.0)
    d = u[:, :, None] - (torch.arange(32, dtype=torch.float64, device="cuda") + 0.5)
    a = torch.where(d.abs() <= 4.5, torch.exp(-0.5 * d * d), 0.0).reshape(rec.shape[0], 192)
    at = 0
    for l, k in enumerate(GUIDE_LAYERS):
        a = a @ par[at:at + 64 * k].view(k, 64) + par[at + 64 * k:at + 64 * k + 64]
        a = torch.relu(a) if l < 4 else a
        at += 64 * k + 64
    lk = a[:, 8:16].clamp(-5.0, 8.0)
    kap = lk.exp()
    mu = a[:, 16:40].reshape(-1, 8, 3)
    mu = mu / torch.sqrt((mu * mu).sum(2, keepdim=True) + 1e-12)
    dot = (mu * rec[:, None, 6:9]).sum(2)
    lv = lk - math.log(2.0 * math.pi) - torch.log(-torch.expm1(-2.0 * kap)) + kap * (dot - 1.0)
    logp = torch.logsumexp(torch.log_softmax(a[:, 0:8], 1) + lv, 1)
    loss = -(rec[:, 9] * logp).sum() / rec.shape[0]
    (grad,) = torch.autograd.grad(loss, par)
    return {"outputs": a.detach(), "gradient": grad}


def exact(case, seed):
    if case["kind"] == "hits" and case["level"] == 0:
        return _exact_hits(case, seed)
    if case["kind"] == "net":
        return _exact_net(case, seed)
    return None
