"""Tone-mapped bytes at the byte thresholds: the fast arithmetic may only decide
where its error cannot.  The oracle is the operator in 64 bits; a byte may differ
from it only where the operator's own 32-bit arithmetic (a few roundings and a
power of 4 ulp; the film operator's 1 - e^-x with 2 ulp) reaches the threshold."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def operator(op, light, e, w):
    if op == "linear":
        return e * light
    if op == "film":
        return -np.expm1(-e * light)
    return e * light * (1.0 + (light / (w * w) if op == "reinhard_white" else 0.0)) / (1.0 + light)


def inverse(op, v, e, w):
    if op == "linear":
        return v / e
    if op == "film":
        return -np.log1p(-np.minimum(v, 1.0 - 1e-9)) / e
    if op == "reinhard":
        return v / (e - v)
    a, b, c = e / (w * w), e - v, -v
    return (-b + np.sqrt(b * b - 4 * a * c)) / (2 * a)


def bytes_of(light, op, e, g_src, g_dst, w):
    import torch
    from xyz_b200 import api
    n = -(-light.size // 3072) * 3072
    film = np.zeros(n, F)
    film[:light.size] = light
    out = api.tonemap(torch.from_numpy(film.reshape(-1, 1024, 3)).cuda(), 1.0, op=op, exposure=float(e), white=float(w),
                      src_gamma=g_src, dst_gamma=g_dst)
    return out.cpu().numpy().reshape(-1, 3)[:, ::-1].reshape(-1)[:light.size]


def check(light, op, e, g_src, g_dst, w):
    got = bytes_of(light, op, e, g_src, g_dst, w).astype(np.float64)
    g = float(F(F(g_src) / F(g_dst)))
    v = operator(op, light.astype(np.float64), float(F(e)), float(F(w)))
    dv = v * 8 * 2.0 ** -24 + (1.3 * 2.0 ** -23 if op == "film" else 0.0)
    power = 5 * 2.0 ** -23
    p, least, most = (256.0 * np.maximum(x, 0.0) ** g for x in (v, v - dv, v + dv))
    least, most = least * (1 - power), most * (1 + power)
    lo, hi = np.clip(np.floor(least), 0, 255), np.clip(np.floor(most), 0, 255)
    bad = (got < lo) | (got > hi)
    assert not bad.any(), (light[bad][:4], got[bad][:4], p[bad][:4])
    return most - least


@pytest.mark.parametrize("gamma", [(1.0, 2.2), (1.0, 1.0), (2.2, 1.0), (1.0, 8.0), (14.0, 1.0)])
@pytest.mark.parametrize("op,e,w", [("film", 1.0, 0.0), ("film", 0.02, 0.0), ("linear", 0.3, 0.0), ("reinhard", 1.7, 0.0),
                                    ("reinhard_white", 1.0, 2.5), ("reinhard_white", 0.8, 40.0)])
def test_bytes_at_the_thresholds(op, e, w, gamma):
    g = float(F(F(gamma[0]) / F(gamma[1])))
    d = 10.0 ** np.linspace(-7.5, -2.0, 120)
    v = ((np.arange(1, 256) / 256.0) ** (1.0 / g))[:, None] * (1.0 + np.concatenate([-d, [0.0], d]))
    light = inverse(op, v.reshape(-1), float(F(e)), float(F(w)) if w else 1.0).astype(F)
    light = light[np.isfinite(light) & (light > 0)]
    width = check(light, op, e, *gamma, w)
    if gamma != (1.0, 8.0):  # (there the film operator's cancellation reaches most thresholds)
        assert (width < 0.02).mean() > 0.6


@pytest.mark.parametrize("white", [1.5e19, 3e14, 1e-18])
def test_white_points_whose_square_leaves_the_range(white):
    light = np.exp(np.linspace(np.log(1e-9), np.log(5e37), 30000)).astype(F)
    check(light, "reinhard_white", 0.4, 1.0, 1.0, white)
