"""Importon queries in a scene whose cells are as small as the rounding of its
coordinates: the cells around a point then span five rows and more."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,ext,radius", [(83215.87, 133235.12, 0.008815357), (-1484.9487, 4663.99, 0.00031954632),
                                           (0.0, 40.0, 0.1)])
@pytest.mark.parametrize("axis", [1, 2])
def test_histogram_counts_every_row(lo, ext, radius, axis):
    """All importons and points on a line along `axis`, seen from above: the last
    cumulative count is 256 and the number of importons within the radius."""
    import torch
    from xyz_b200 import api, scenes
    f = np.float32
    rng = np.random.default_rng(2)
    n = 20000
    z = (lo + ext * rng.uniform(0.9, 1.0, n)).astype(f)
    near = (z + radius * rng.uniform(-1.2, 1.2, n)).astype(f)
    z, near = np.clip(z, f(lo), f(lo + ext)), np.clip(near, f(lo), f(lo + ext))
    up = 3 - axis  # the shading normal
    lengthwise, normal, other = np.eye(3, dtype=f)[axis], np.eye(3, dtype=f)[up], np.eye(3, dtype=f)[0]
    ends = np.array([f(lo), f(lo + ext)])
    pos = np.stack([ends[[0, 1, 0]][:, None] * lengthwise, ends[[1, 0, 1]][:, None] * lengthwise])
    pos[:, 1] += f(0.25) * f(radius) * other
    sd = scenes.SceneData(pos.reshape(-1, 3).astype(f), np.arange(6, dtype=np.int32).reshape(-1, 3),
                          np.array([0, 1], np.int32), np.full((2, 3), 0.5, f), np.array([0, 1], np.int32), np.ones(3, f))
    imp = np.concatenate([near[:, None] * lengthwise, np.tile(-normal, (n, 1))], 1)
    frames = np.concatenate([z[:, None] * lengthwise, np.tile(np.concatenate([lengthwise, other, normal]), (n, 1))], 1)
    s = np.sort(near)
    d = lambda k: (s[np.clip(k, 0, n - 1)] - z).astype(f)
    want = np.zeros(n)
    first = np.searchsorted(s, z - 3 * radius)
    for k in range(int((np.searchsorted(s, z + 3 * radius) - first).max()) + 1):
        want += ((d(first + k) * d(first + k)).astype(f) < f(radius) * f(radius)) & (first + k < n)
    with api.Scene(sd) as scene, api.Importons(scene, importons=imp.astype(f), radius=radius) as m:
        got = m.query(torch.from_numpy(np.ascontiguousarray(frames, f)).cuda()).cpu().numpy()
    assert want.max() > 1
    assert np.array_equal(got[:, -1], 256 + want)
