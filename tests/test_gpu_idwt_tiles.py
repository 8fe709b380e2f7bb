"""The allocation-free inverse DWT at the edges of its 64x64 and 32x32 tiles, against whole-line
lifting in numpy with the same separately rounded float32 operations (tolerance 0): levels of
one sample, of one tile and a bit, levels on either side of the small-tile rule, several tiles a
CTA, odd strides."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
C97 = [np.float32(c) for c in (0.44350685204397, 0.88291107553093, -0.05298011857296, -1.58613434205992)]


def _line(v, rev):
    """Inverse lifting along the last axis of interleaved lines."""
    n = v.shape[-1]
    if n < 2:
        return v
    x = v.copy()

    def at(i):
        i = abs(i)
        return x[..., 2 * (n - 1) - i if i >= n else i]

    def step(first, update):
        new = {i: update(x[..., i], at(i - 1), at(i + 1)) for i in range(first, n, 2)}
        for i, val in new.items():
            x[..., i] = val
    if rev:
        step(0, lambda s, a, b: s - ((a + b + 2) >> 2))
        step(1, lambda s, a, b: s + ((a + b) >> 1))
    else:
        for k, c in enumerate(C97):
            step(k & 1, lambda s, a, b: s - c * (a + b))
    return x


def _reference(coef, rw, rh, rev):
    klo = np.float32(1.23017410558578)
    ll = coef[:rh[0], :rw[0]]
    for r in range(1, len(rw)):
        w, h, lw, lh = rw[r], rh[r], rw[r - 1], rh[r - 1]
        if not rev and r > 1:
            ll = ll * (klo * klo)
        p = np.empty((h, w), coef.dtype)
        p[0::2, 0::2], p[0::2, 1::2] = ll, coef[:lh, lw:w]
        p[1::2, 0::2], p[1::2, 1::2] = coef[lh:h, :lw], coef[lh:h, lw:w]
        p = _line(p, rev)
        ll = np.ascontiguousarray(_line(np.ascontiguousarray(p.T), rev).T)
    return ll


@pytest.mark.parametrize("rev", [0, 1])
@pytest.mark.parametrize("w,h,levels", [(1, 1, 2), (1, 70, 3), (70, 1, 3), (3, 5, 2), (31, 33, 1), (32, 64, 5), (64, 64, 1),
                                        (65, 63, 2), (129, 200, 3), (500, 389, 2), (1000, 777, 5), (2049, 1030, 6),
                                        (4096, 65, 1)])
def test_tile_edges(pkg, rev, w, h, levels):
    import torch
    from jpeg2000_decoder_b200 import native
    rng = np.random.default_rng(w * 7 + h)
    tc = native.TileComp()
    tc.w, tc.h, tc.levels = w, h, levels
    rw, rh = [w], [h]
    for _ in range(levels):
        rw.insert(0, (rw[0] + 1) // 2)
        rh.insert(0, (rh[0] + 1) // 2)
    for r in range(levels + 1):
        tc.res_w[r], tc.res_h[r] = rw[r], rh[r]
    coef = rng.integers(-500, 500, (h, w)).astype(np.int32) if rev else (rng.standard_normal((h, w)) * 100).astype(np.float32)
    want = _reference(coef, rw, rh, rev)
    src = torch.from_numpy(coef).cuda()
    pad = 3
    out = torch.full((h, w + pad), -7, dtype=src.dtype, device="cuda")
    rc = native.lib().j2k_gpu_tile_idwt_noalloc(ctypes.byref(tc), rev, 0, ctypes.c_void_p(src.data_ptr()),
                                                ctypes.c_void_p(out.data_ptr()), w + pad,
                                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    got = out.cpu().numpy()
    assert np.array_equal(got[:, :w].view(np.int32), want.view(np.int32))
    assert (got[:, w:] == -7).all()
