"""An adjoint whose primal waves start with a launch per bounce and end in the
one-launch kernel: that kernel writes the rest of the records which the replay
reads.  The same paths in waves that run in one launch from the first bounce on,
and one at a time, give the same gradients."""

import pytest

pytestmark = pytest.mark.gpu

ONE_LAUNCH = 1 << 17  # waves (or what is left of them) of at most so many rays


@pytest.mark.parametrize("kind", ["box", "mesh", "room"])
@pytest.mark.parametrize("size,depth", [((640, 480, 1), 10), ((333, 251, 3), 8), ((512, 300, 2), 15)])
def test_gradients_equal_those_of_small_waves(kind, size, depth):
    import torch
    from xyz_b200 import api, scenes
    w, h, spp = size
    if kind == "room":
        ds = scenes.diff_scene(level=2, wall_n=5, seed=3)
        sd = ds.scene
    else:
        sd = scenes.cornell_box() if kind == "box" else scenes.spheres_scene(level=3, n_spheres=3, seed=1)
    gen = torch.Generator("cuda").manual_seed(1)
    d_film = torch.rand((h, w, 3), generator=gen, device="cuda")
    with api.Scene(sd) as s:
        assert w * h * spp > ONE_LAUNCH
        s.render(sd.camera, w, h, spp, seed=3, max_depth=depth, profile=2)
        rays = [int(x) for x in s.render_profile()["ext_rays_by_iter"]]
        even = [b for b in range(4, depth - 3, 2) if rays[b] <= ONE_LAUNCH]
        assert even and rays[even[0]] > 0, rays  # a bounce at which the kernel takes over
        got = s.adjoint(sd.camera, w, h, spp, d_film, max_depth=depth, seed=3)
        small = s.adjoint(sd.camera, w, h, spp, d_film, max_depth=depth, seed=3, wave_paths=ONE_LAUNCH)
        tiny = s.adjoint(sd.camera, w, h, spp, d_film, max_depth=depth, seed=3, wave_paths=30000)
    # sums of up to 2^22 terms in another order: 2^-24 times the square root of
    # their number, and a margin of 8
    for other in (small, tiny):
        for a, b in zip(got, other):
            assert float(b.abs().max()) > 0
            assert torch.allclose(a, b, rtol=1e-3, atol=1e-5 * float(b.abs().max()))
