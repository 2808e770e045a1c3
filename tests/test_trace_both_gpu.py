"""Shadow rays share a launch with the next bounce's extension rays, as one
queue in waves of at most 2^18 paths and one after the other in larger ones;
profiled renders launch them apart.  All give the same film, for every mode."""

import pytest

pytestmark = pytest.mark.gpu

SMALL, LARGE = (64, 48, 5), (600, 440, 1)  # 15,360 and 264,000 paths


@pytest.mark.parametrize("size", [SMALL, LARGE])
@pytest.mark.parametrize("depth", [1, 2, 6])
@pytest.mark.parametrize("kind", ["plain", "specular", "spectral", "guided", "importon", "noalloc"])
def test_launches_do_not_change_the_film(kind, size, depth):
    import torch
    from xyz_b200 import api, scenes
    w, h, spp = size
    sd = {"specular": scenes.cornell_specular, "guided": lambda: scenes.occluded_room(level=2, wall_n=6),
          "importon": lambda: scenes.occluded_room(level=2, wall_n=6)}.get(kind, scenes.cornell_box)()
    kw = dict(seed=2, max_depth=depth)
    with api.Scene(sd) as s:
        if kind == "guided":
            with api.Guide(s, guide_bounces=3) as g:
                films = [g.render(sd.camera, w, h, spp, profile=p, **kw) for p in (0, 1)]
        elif kind == "importon":
            with api.Importons(s, particles=2000) as m:
                films = [m.render(sd.camera, w, h, spp, profile=p, **kw) for p in (0, 1)]
        elif kind == "noalloc":
            films = [torch.zeros((h, w, 3), device="cuda") for _ in range(2)]
            s.render_noalloc(sd.camera, w, h, spp, films[0], **kw)
            s.render(sd.camera, w, h, spp, film=films[1], profile=1, **kw)
        else:
            mode = "continuous" if kind == "spectral" else "off"
            films = [s.render(sd.camera, w, h, spp, profile=p, spectral=mode, **kw) for p in (0, 1)]
        counts = s.render_counters()
    assert counts["paths"] == w * h * spp
    assert float(films[0].sum()) > 0 or kind in ("guided", "importon")
    assert torch.equal(films[0], films[1])


def test_counters_are_the_same_in_one_launch_and_apart():
    from xyz_b200 import api, scenes
    sd = scenes.cornell_box()
    with api.Scene(sd) as s:
        got = []
        for p in (0, 1):
            s.render(sd.camera, 80, 60, 4, seed=3, max_depth=7, profile=p)
            c = s.render_counters()
            got.append([c[k] for k in ("paths", "extension_rays", "shadow_rays", "shadow_hits_visible", "waves")])
    assert got[0] == got[1] and got[0][3] > 0
