"""The spectral film kernel adds a pixel's samples in order, eight at a time:
the film of n samples equals the sum of the films of its single samples added
one after another, at sample and pixel counts around the kernel's groups."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp", [1, 7, 8, 9, 17])
@pytest.mark.parametrize("size", [(1, 1), (31, 1), (33, 3)])
@pytest.mark.parametrize("mode,hero", [("continuous", 4), ("binned", 1)])
def test_film_is_the_ordered_sum_of_its_samples(spp, size, mode, hero):
    import torch
    from xyz_b200 import api, scenes
    sd = scenes.cornell_box()
    w, h = size
    kw = dict(seed=4, max_depth=4, spectral=mode, hero_wavelengths=hero)
    with api.Scene(sd) as s:
        whole = s.render(sd.camera, w, h, spp, **kw)
        step = torch.zeros((h, w, 3), dtype=torch.float32, device="cuda")
        for k in range(spp):
            s.render(sd.camera, w, h, 1, spp_offset=k, film=step, accumulate=True, **kw)
    assert np.isfinite(whole.cpu().numpy()).all() and float(whole.sum()) > 0 or w * h == 1
    assert torch.equal(whole, step)
