"""The wide tree's answers where rounding decides: rays aimed at and beside the
edges of slivers, on the CPU against a host kd loop (tests/cpp/wide_kd_check.cpp)
and on the GPU against counting calls, which walk the kd-tree.  Equal in every bit."""

import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("wide") / "wide_kd_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "wide_kd_check.cpp"),
                    os.path.join(ROOT, "xyz_b200", "csrc", "kdbuild_host.cpp"), "-o", exe], check=True)

    def run(scene, rays, kind):
        r = subprocess.run([exe, scene, str(rays), kind], capture_output=True, text=True, check=True)
        return [float(x) for x in r.stdout.split()]
    return run


@pytest.mark.parametrize("scene", ["sliver:1e-2", "sliver:1e-3", "sliver:1e-4", "sliver:1e-5", "soup:0.1", "boxes"])
def test_answers_beside_edges(check, scene):
    rays, hits, unsettled, differ = check(scene, 200000, "edge")[:4]
    assert hits > rays / 10 and unsettled < rays / 1000
    assert differ == 0


def test_answers_in_the_planes_of_triangles(check):
    """Rays between two points of a face of a box, large enough that rounding keeps
    the determinant above the triangle test's limit: what the test then accepts
    are the triangles that the kd loop's cells hold."""
    rays, hits, _, differ = check("turned", 200000, "plane")[:4]
    assert hits > rays / 2 and differ == 0


def scene_of(pos):
    """A scene of loose triangles, the last of them a light."""
    from xyz_b200 import scenes
    n = pos.shape[0]
    mat = np.zeros(n, np.int32)
    mat[-1] = 1
    return scenes.SceneData(pos.reshape(-1, 3).astype(np.float32), np.arange(3 * n, dtype=np.int32).reshape(-1, 3), mat,
                            np.full((2, 3), 0.5, np.float32), np.array([0, 1], np.int32), np.ones(3, np.float32))


def slivers(width, seed=1, n=200):
    rng = np.random.default_rng(seed)
    c, a = rng.uniform(-1, 1, (n, 3)), rng.normal(size=(n, 3))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    b = np.cross(a, rng.normal(size=(n, 3)))
    b /= np.linalg.norm(b, axis=1, keepdims=True)
    l, s = rng.uniform(0.3, 1.0, (2, n, 1))
    return np.stack([c, c + l * a, c + l * s * a + width * l * b], 1)


def edge_rays(pos, n, seed):
    """Rays at points 1e-7 to 1e-1 of a triangle inside or beyond one of its edges."""
    rng = np.random.default_rng(seed)
    t = pos[rng.integers(0, pos.shape[0], n)].astype(np.float64)
    k = rng.integers(0, 3, n)
    i = np.arange(n)
    a, b, c = t[i, k], t[i, (k + 1) % 3], t[i, (k + 2) % 3]
    e = a + rng.uniform(0, 1, (n, 1)) * (b - a)
    p = e + 10.0 ** rng.uniform(-7, -1, (n, 1)) * np.where(rng.random((n, 1)) < 0.75, 1, -1) * (e - c)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    size = 0.5 * np.ptp(pos.reshape(-1, 3), axis=0).max()
    r = np.empty((n, 8), np.float32)
    r[:, 0:3] = p - d * size * 10.0 ** rng.uniform(-1.5, 0.5, (n, 1))
    r[:, 3] = 1e-5
    r[:, 4:7] = d
    r[:, 7] = np.inf
    return r


def compare(sd, rays, **build):
    """Hits of the rays by the wide tree and by the kd-tree; returns the number of hits."""
    import torch
    from xyz_b200 import api
    rays = torch.from_numpy(rays).cuda()
    with api.Scene(sd, **build) as s:
        a, b = (torch.empty((rays.shape[0], 4), dtype=torch.float32, device="cuda") for _ in range(2))
        s.trace_device(rays, a)
        c = s.trace_device(rays, b, counted=True)
    same = (a.view(torch.int32) == b.view(torch.int32)).all(1)
    assert bool(same.all()), int((~same).sum())
    return c["hits"]


@pytest.mark.gpu
@pytest.mark.parametrize("width", [1e-2, 1e-3, 1e-4, 1e-5])
@pytest.mark.parametrize("builder", ["device", "host"])
def test_sliver_hits_equal_the_kd_tree(width, builder):
    pos = slivers(width).astype(np.float32)
    assert compare(scene_of(pos), edge_rays(pos, 1 << 20, 3), builder=builder) > 1 << 17


# ---- coordinates that are large beside the triangles
@pytest.mark.parametrize("scene", ["terrain:0", "terrain:1000", "terrain:10000", "ground:10", "ground:1000", "ground:3000"])
def test_work_does_not_depend_on_the_coordinates(check, scene):
    """Wherever the triangles lie a ray meets fewer than half the nodes that it
    meets in the kd-tree, and not many more triangles (at 10,000 the corners are
    rounded to a tenth of a triangle, which the kd-tree's splits suffer from too)."""
    differ, nodes, tests, kd_nodes, kd_tests = check(scene, 30000, "local")[3:]
    assert differ == 0
    assert nodes < 0.5 * kd_nodes
    assert tests < 1.5 * kd_tests


@pytest.mark.parametrize("scene", ["terrain:0", "terrain:10000", "ground:300", "ground:3000"])
def test_answers_at_large_coordinates(check, scene):
    rays, hits, unsettled, differ = check(scene, 100000, "edge")[:4]
    assert hits > rays / 2 and unsettled < rays / 100
    assert differ == 0


def test_rays_from_far_beyond_the_scene(check):
    """Rays up to 30,000 scene sizes away keep the kd-tree's work: the tree's boxes,
    widened by the distance, would no longer separate the triangles."""
    rays, hits, _, differ, _, tests, _, kd_tests = check("terrain:0", 100000, "far")
    assert hits > rays / 2 and differ == 0
    assert tests < 1.5 * kd_tests


def terrain(n, at):
    x = np.linspace(-1, 1, n + 1)
    X, Z = np.meshgrid(x, x, indexing="ij")
    Y = 0.1 * np.sin(7 * X) * np.cos(5 * Z) + 0.004 * np.random.default_rng(5).normal(size=X.shape)
    P = np.stack([X + at, Y, Z + at], -1)
    a, b, c, d = P[:-1, :-1], P[1:, :-1], P[1:, 1:], P[:-1, 1:]
    return np.concatenate([np.stack(t, 2).reshape(-1, 3, 3) for t in ((a, b, c), (a, c, d))])


def ground(h):
    q = [(-h, -1, -h), (h, -1, -h), (h, -1, h), (-h, -1, h)]
    return np.concatenate([terrain(100, 0.0), np.array([[q[0], q[1], q[2]], [q[0], q[2], q[3]]], np.float64)])


@pytest.mark.gpu
@pytest.mark.parametrize("pos", [terrain(100, 1000.0), terrain(100, 10000.0), ground(300.0), ground(3000.0)],
                         ids=["terrain1000", "terrain10000", "ground300", "ground3000"])
def test_hits_equal_the_kd_tree_at_large_coordinates(pos):
    pos = pos.astype(np.float32)
    rays = edge_rays(pos, 1 << 19, 4)
    m = rays.shape[0] // 2  # the other half from nearby
    near = rays[m:, 0:3] + rays[m:, 4:7] * (0.9 * np.linalg.norm(rays[m:, 0:3] - pos.reshape(-1, 3).mean(0), axis=1))[:, None]
    rays[m:, 0:3] = near
    assert compare(scene_of(pos), rays) > 1 << 16


# ---- rays whose direction is not of unit length, or has no extent along an axis
@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-3, 0.03, 3.0, 1e4, None])
def test_directions_of_any_length(scale):
    pos = np.concatenate([slivers(1e-2), terrain(40, 0.0)]).astype(np.float32)
    rays = edge_rays(pos, 1 << 18, 5)
    s = scale if scale else 10.0 ** np.random.default_rng(1).uniform(-8, 8, (rays.shape[0], 1))
    rays[:, 4:7] *= s
    # (the triangle test bounds d . n from below, so short directions hit little)
    assert compare(scene_of(pos), rays) > (0 if not scale or scale < 0.1 else 1 << 15)


@pytest.mark.gpu
@pytest.mark.parametrize("extra", [-1, 0, 33])
@pytest.mark.parametrize("share", [1.0, 0.9])
def test_queues_of_axis_parallel_rays(extra, share):
    """Queues around the size from which the kd-tree's own kernel follows, all
    or most of whose rays have no extent along two axes."""
    import torch
    n = 2 * 8 * 128 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    pos = terrain(60, 0.0).astype(np.float32)
    rng = np.random.default_rng(6)
    rays = edge_rays(pos, n, 7)
    flat = rng.random(n) < share
    d = np.zeros((n, 3), np.float32)
    d[np.arange(n), rng.integers(0, 3, n)] = rng.choice([-1.0, 1.0], n)
    p = rays[:, 0:3] + rays[:, 4:7] * np.linalg.norm(rays[:, 0:3], axis=1, keepdims=True)
    rays[flat, 4:7] = d[flat]
    rays[flat, 0:3] = (p - d)[flat]
    assert compare(scene_of(pos), rays) > 1 << 14


@pytest.mark.gpu
def test_intervals_that_are_no_interval():
    """tmin or tmax not a number (which the triangle test lets pass), negative tmin,
    empty intervals, an infinite tmin."""
    pos = np.concatenate([slivers(1e-2), terrain(40, 0.0)]).astype(np.float32)
    rays = edge_rays(pos, 1 << 17, 8)
    k = np.arange(rays.shape[0]) % 8
    rays[k == 0, 7] = np.nan
    rays[k == 1, 3] = np.nan
    rays[k == 2, 3] = -np.inf
    rays[k == 3, 3] = -3.0
    rays[k == 4, 7] = 0.0
    rays[k == 5, 3] = np.inf
    rays[k == 6, 3:8:4] = np.nan
    assert compare(scene_of(pos), rays) > 1 << 14


@pytest.mark.gpu
@pytest.mark.parametrize("side", [7, 60])
def test_far_rays_hit_as_in_the_kd_tree(side):
    """Rays from 10 to 10,000 scene sizes at a terrain they meet at all slopes, some
    so small that the triangle test's error exceeds the triangles."""
    pos = terrain(side, 0.0).astype(np.float32)
    rng = np.random.default_rng(9)
    n = 1 << 21
    t = pos[rng.integers(0, pos.shape[0], n)].astype(np.float64)
    d = rng.normal(size=(n, 3)) * [1.0, 0.05, 1.0]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.empty((n, 8), np.float32)
    rays[:, 0:3] = (rng.dirichlet([1, 1, 1], n)[..., None] * t).sum(1) - d * 2.0 * 10.0 ** rng.uniform(1, 4, (n, 1))
    rays[:, 3], rays[:, 4:7], rays[:, 7] = 1e-5, d, np.inf
    assert compare(scene_of(pos), rays) > 1 << 19


@pytest.mark.gpu
@pytest.mark.parametrize("extra", [-1, 0, 1])
@pytest.mark.parametrize("triangles", [64, 65])
def test_queues_of_tiny_scenes(triangles, extra):
    """Queues around the size from which scenes of up to 64 triangles take the
    kd-tree's kernel, and scenes around that number."""
    import torch
    pos = slivers(0.3, n=triangles).astype(np.float32)
    n = 9 * 128 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    assert compare(scene_of(pos), edge_rays(pos, n, 10)) > n // 8
