"""Film kernels at the sizes and alignments where their four-pixel groups and
wide accesses end: narrow and ragged widths, films and outputs that start off a
16-byte (or 4-byte) border, padding bytes, infinities and NaN; against the C
oracle (Radiance bytes equal; tone-mapped bytes at most 1 apart, nearly all
equal, as expf / powf of device and host may differ in the last bit)."""

import numpy as np
import pytest

from tests.helpers import ensure_port

pytestmark = pytest.mark.gpu


def _film(h, w, seed, special):
    rng = np.random.default_rng(seed)
    f = (4.0 * rng.lognormal(0.0, 2.0, (h, w, 1)) * rng.uniform(0.5, 1.0, (h, w, 3))).astype(np.float32)
    f[rng.random((h, w)) < 0.1] = 0.0
    if special:
        flat = f.reshape(-1)
        flat[rng.integers(0, flat.size, 6)] = [np.inf, -np.inf, np.nan, -1.0, 1e-38, 3e38]
    return f


@pytest.mark.parametrize("w", [1, 2, 3, 4, 5, 7, 8, 130, 516])
@pytest.mark.parametrize("offset", [0, 1])
def test_shapes_and_alignments(w, offset):
    import torch
    from xyz_b200 import api
    P = ensure_port()
    h = 5
    L = api.load_library()
    for seed, special in ((w, False), (w + 1, True)):
        host = _film(h, w, seed, special)
        store = torch.empty(h * w * 3 + offset, dtype=torch.float32, device="cuda")
        film = store[offset:].view(h, w, 3)
        film.copy_(torch.from_numpy(host))
        for xyze in (False, True):
            got = api.encode_rgbe(film, 0.25, xyze=xyze).cpu().numpy()
            fin = host if not xyze else np.where(np.isfinite(host).all(-1, keepdims=True), host, 1.0)
            want = P.encode_rgbe(np.ascontiguousarray(fin), np.float32(0.25), xyze)
            if xyze:  # a non-finite maximum has no defined exponent
                keep = np.isfinite(host).all(-1)
                assert np.array_equal(got[keep], want[keep])
            else:
                assert np.array_equal(got, want)
        if special:
            continue
        for op in ("film", "reinhard_white"):
            want = P.tonemap(host, scale=0.25, op=api.TONEMAP_OPS[op], rgb=True).astype(np.int32)
            stride = (3 * w + 3) & ~3
            for shift in (0, 1):  # an output off a word border is written by bytes
                out = torch.full((h * stride + 8,), 0x5A, dtype=torch.uint8, device="cuda")
                word = torch.zeros(1, dtype=torch.int32, device="cuda")
                tp = api.TonemapParams()
                import ctypes as C
                L.xyzgpu_tonemap_params_default(C.byref(tp))
                tp.scale, tp.op, tp.rgb = 0.25, api.TONEMAP_OPS[op], 1
                assert L.xyzgpu_film_tonemap(film.data_ptr(), w, h, C.byref(tp), out.data_ptr() + shift,
                                             word.data_ptr(), None) == 0
                torch.cuda.synchronize()
                o = out.cpu().numpy()
                assert (o[:shift] == 0x5A).all() and (o[shift + h * stride:] == 0x5A).all()
                g = o[shift: shift + h * stride].reshape(h, stride).astype(np.int32)
                assert (g[:, 3 * w:] == 0).all()
                assert g.shape == want.shape
                assert np.abs(g - want).max() <= 1
                assert (g == want).mean() >= 0.99
