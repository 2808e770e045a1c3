"""The wide tree the traversal walks against the kd-tree it is derived from.

CPU: the tree's builder and box test, compiled for the host, against a test of
every triangle (tests/cpp/wide_check.cpp).  GPU: counting calls walk the
kd-tree, so the same rays and the same render through both must agree in every
bit (the wide traversal hands rays whose answer rounding could decide to the
kd-tree, so no tolerance applies)."""

import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_host_walk_finds_the_closest_hit(tmp_path):
    exe = str(tmp_path / "wide_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "wide_check.cpp"),
                    os.path.join(ROOT, "xyz_b200", "csrc", "kdbuild_host.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def _soup(n, size, seed):
    from xyz_b200 import scenes
    rng = np.random.default_rng(seed)
    pos = (rng.uniform(-1, 1, (n, 1, 3)) + size * rng.uniform(-1, 1, (n, 3, 3))).astype(np.float32).reshape(-1, 3)
    lit = np.zeros(2, np.int32)
    lit[1] = 1
    mat = np.zeros(n, np.int32)
    mat[-1] = 1
    return scenes.SceneData(pos, np.arange(3 * n, dtype=np.int32).reshape(-1, 3), mat,
                            np.full((2, 3), 0.5, np.float32), lit, np.ones(3, np.float32))


def _scenes():
    from xyz_b200 import scenes
    coincident = _soup(1, 0.5, 7)
    coincident.tris = np.tile(coincident.tris, (300, 1))
    coincident.tri_mat = np.ones(300, np.int32)
    return {"one": _soup(1, 0.5, 1), "nine": _soup(9, 0.5, 2), "soup": _soup(3000, 0.05, 3), "coincident": coincident,
            "cornell": scenes.cornell_box(), "mesh": scenes.spheres_scene(level=4, seed=3),
            "room": scenes.occluded_room(level=3, wall_n=8), "boxes": scenes.batch_scene(2, target_tris=6000)}


def _rays(sd, n, seed):
    """Rays at triangle insides, edges and vertices from in and around the box,
    axis-parallel rays, short intervals, and rays the wide tree cannot serve
    (far origins, long and short directions)."""
    rng = np.random.default_rng(seed)
    lo, hi = sd.positions.min(0).astype(np.float64), sd.positions.max(0).astype(np.float64)
    o = lo + (hi - lo) * rng.uniform(-0.6, 1.6, (n, 3)) + 1e-3 * rng.normal(size=(n, 3))
    t = sd.positions[sd.tris[rng.integers(0, sd.tris.shape[0], n)]].astype(np.float64)
    w = rng.dirichlet((1.0, 1.0, 1.0), n)
    w[: n // 4, 2] = 0.0                     # on an edge
    w[n // 8: n // 4, 1] = 0.0               # on a vertex
    w /= w.sum(1, keepdims=True)
    p = (w[:, :, None] * t).sum(1)
    d = p - o
    k = n // 2
    d[k: k + n // 8] = 0.0                   # axis-parallel through such points
    d[np.arange(k, k + n // 8), rng.integers(0, 3, n // 8)] = rng.choice([-1.0, 1.0], n // 8)
    o[k: k + n // 8] = p[k: k + n // 8] - 0.7 * d[k: k + n // 8]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o[-n // 16:] = p[-n // 16:] - 300.0 * d[-n // 16:]
    scale = np.ones((n, 1))
    scale[-n // 8: -n // 16] = rng.choice([1e-4, 0.03, 3.0, 1e3], (n // 16, 1))
    r = np.empty((n, 8), np.float32)
    r[:, 0:3] = o
    r[:, 3] = 1e-5
    r[:, 4:7] = d * scale
    r[:, 7] = np.inf
    m = slice(3 * n // 4 - n // 16, 3 * n // 4)  # intervals that end or start at the hit
    dist = np.linalg.norm(p[m] - o[m], axis=1).astype(np.float32)
    r[m, 7] = dist
    r[m, 3][::2] = dist[::2]
    return r


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["one", "nine", "soup", "coincident", "cornell", "mesh", "room", "boxes"])
@pytest.mark.parametrize("build", [dict(), dict(leaf_max_tris=1), dict(builder="host", leaf_max_tris=4)])
def test_hits_equal_the_kd_tree(name, build):
    import torch
    from xyz_b200 import api
    sd = _scenes()[name]
    rays = torch.from_numpy(_rays(sd, 1 << 16, 11)).cuda()
    with api.Scene(sd, **build) as s:
        a, b = (torch.empty((rays.shape[0], 4), dtype=torch.float32, device="cuda") for _ in range(2))
        s.trace_device(rays, a)
        c = s.trace_device(rays, b, counted=True)
    assert c["hits"] > 0
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("name,spectral", [("cornell", "off"), ("mesh", "off"), ("boxes", "off"), ("mesh", "binned")])
def test_film_equals_the_kd_tree(name, spectral):
    """Extension and shadow rays of a whole render (profile=2 counts, on the kd-tree)."""
    import torch
    from xyz_b200 import api
    sd = _scenes()[name]
    with api.Scene(sd) as s:
        films = [s.render(sd.camera, 96, 80, 8, seed=5, max_depth=8, profile=p, spectral=spectral) for p in (0, 2)]
    assert float(films[0].sum()) > 0
    assert torch.equal(films[0], films[1])
