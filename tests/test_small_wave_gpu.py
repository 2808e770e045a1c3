"""Waves of at most 2^17 paths run all their bounces in one launch, and larger
ones the bounces after that few rays are left; profiled renders launch every
bounce's kernels.  Same film, same counters."""

import pytest

pytestmark = pytest.mark.gpu


# one path; fewer paths than CTAs, one more, uneven shares; the rule's last size
# and the first beyond it; a wave taken over when it has thinned out; several waves
# in a call
@pytest.mark.parametrize("depth", [1, 2, 15])
@pytest.mark.parametrize("shape", [(1, 1, 1, 0), (37, 16, 1, 0), (593, 1, 1, 0), (97, 61, 3, 0), (512, 256, 1, 0),
                                   (43691, 3, 1, 0), (640, 480, 2, 0), (97, 61, 3, 5000)])
@pytest.mark.parametrize("kind", ["box", "specular", "mesh", "binned", "continuous"])
def test_one_launch_gives_the_film_and_counters_of_many(kind, shape, depth):
    import torch
    from xyz_b200 import api, scenes
    w, h, spp, wave = shape
    mode = kind if kind in ("binned", "continuous") else "off"
    sd = {"specular": scenes.cornell_specular,
          "mesh": lambda: scenes.spheres_scene(level=3, n_spheres=3, seed=1)}.get(kind, scenes.cornell_box)()
    with api.Scene(sd) as s:
        films, counts = [], []
        for profile in (0, 1):
            films.append(s.render(sd.camera, w, h, spp, seed=5, max_depth=depth, profile=profile, wave_paths=wave,
                                  spectral=mode))
            c = s.render_counters()
            counts.append([c[k] for k in ("paths", "extension_rays", "shadow_rays", "shadow_hits_visible", "waves")])
    assert counts[0] == counts[1] and counts[0][1] >= w * h * spp
    assert torch.equal(films[0], films[1])
