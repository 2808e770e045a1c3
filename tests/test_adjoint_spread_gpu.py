"""The emission gradient is summed 256 bytes apart per material where that is
small enough: few materials, narrower strides, and more than 2^22 materials'
worth of floats (the caller's array itself) give the same gradients on the same
paths, added to what the arrays hold."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [0, 2000, (1 << 18) + 3, (1 << 21) + 3])
def test_gradient_does_not_depend_on_the_layout(extra):
    import dataclasses
    import torch
    from xyz_b200 import api, scenes
    sd = scenes.cornell_box()
    d_film = torch.rand((40, 52, 3), generator=torch.Generator("cuda").manual_seed(1), device="cuda")
    nm = sd.albedo_xyz.shape[0]
    out = []
    for pad in (0, extra):
        s2 = dataclasses.replace(
            sd, albedo_xyz=np.concatenate([sd.albedo_xyz, np.full((pad, 3), 0.5, np.float32)]),
            is_light=np.concatenate([sd.is_light, np.zeros(pad, np.int32)]), albedo_spd=None, light_power_spd=None)
        with api.Scene(s2) as s:
            # gradients add to what the arrays hold
            a = torch.full((nm + pad, 3), 0.25, device="cuda")
            e = torch.full((nm + pad,), 0.5, device="cuda")
            s.adjoint(sd.camera, 52, 40, 8, d_film, max_depth=5, seed=3, d_albedo=a, d_emission=e)
            out.append((a[:nm].cpu(), e[:nm].cpu(), a[nm:].cpu(), e[nm:].cpu()))
    (a0, e0, _, _), (a1, e1, ra, re) = out
    # float sums of up to 16,640 paths in another order: 2^-24 times the square
    # root of the terms, and a margin of 8
    assert float((e0 - 0.5).abs().max()) > 0
    assert torch.allclose(e0, e1, rtol=6e-5, atol=1e-5) and torch.allclose(a0, a1, rtol=6e-5, atol=1e-5)
    assert (ra == 0.25).all() and (re == 0.5).all()
