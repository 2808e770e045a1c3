"""The device builder's small nodes (one warp each) against the host builder."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(n, flat, seed):
    """n triangles; flat: all in the plane z = 0 on a coarse lattice, so that an
    axis has no extent, many costs tie and many references lie on planes."""
    from xyz_b200 import scenes
    rng = np.random.default_rng(seed)
    if flat:
        c = rng.integers(0, 8, (n, 1, 3)).astype(np.float32) / 8.0
        pos = c + np.array([[0, 0, 0], [0.125, 0, 0], [0, 0.125, 0]], np.float32)
        pos[..., 2] = 0.0
    else:
        pos = rng.uniform(-1.0, 1.0, (n, 1, 3)) + rng.normal(scale=0.05, size=(n, 3, 3))
    mat = np.zeros(n, np.int32)
    mat[:2] = 1
    return scenes.SceneData(pos.reshape(-1, 3).astype(np.float32), np.arange(3 * n, dtype=np.int32).reshape(n, 3),
                            mat, np.array([[0.5] * 3, [0.0] * 3], np.float32), np.array([0, 1], np.int32),
                            np.ones(3, np.float32))


# references of a warp's batch (64) and of the rule that gives a node to CTAs
# (512); one, two and three planes of 32 lanes' worth of bins, and their edges
@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("bins", [2, 3, 32, 33, 34, 63, 64])
@pytest.mark.parametrize("n", [2, 33, 64, 65, 511, 512, 1300])
def test_small_nodes_equal_host_tree(n, bins, flat):
    from xyz_b200 import api
    kw = dict(bins=bins, leaf_max_tris=1, empty_bonus=0.2)
    sd = _soup(n, flat, seed=n + bins)
    with api.Scene(sd, builder="host", **kw) as a, api.Scene(sd, builder="device", **kw) as b:
        (na, ra), (nb, rb) = a.tree(), b.tree()
    assert np.array_equal(na, nb)
    assert np.array_equal(ra, rb)
