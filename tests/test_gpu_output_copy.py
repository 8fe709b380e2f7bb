"""Pictures on either side of the size from which the copy into pageable memory is threaded, with
a last piece that is not whole, equal the copy into page-locked memory (the driver's own)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(2389, 2341), (2363, 2366)])  # 16.78 MB: just above and just below 16 MiB
def test_pageable_copy_equals_pinned(pkg, w, h):
    import torch
    from jpeg2000_decoder_b200 import native, synth
    img = np.tile(synth.fields_and_edges(5, 256, 256), (1, 10, 10))[:, :h, :w]
    cs = native.encode(np.ascontiguousarray(img), 8, reversible=0, levels=3, num_layers=1, layer_bpp=[0.3], tile_w=1024,
                       tile_h=1024, guard_bits=1)
    plan = native.Plan(cs)
    ctx = native.GpuContext(0)
    try:
        ctx.begin()
        slot = ctx.add(plan, native.FMT_24BITS_RGB)
        ctx.launch()
        n = w * h * 3
        pinned = torch.empty(n, dtype=torch.uint8, pin_memory=True)
        ctx.output_async(slot, pinned.data_ptr(), n)
        assert ctx.sync() == 0
        want = pinned.numpy()
        for _ in range(2):
            assert np.array_equal(ctx.output(slot), want)
        odd = np.empty(n + 1, np.uint8)  # a destination off the word
        assert native.lib().j2k_gpu_output_copy(ctx.h, slot, ctypes.c_void_p(odd.ctypes.data + 1), n) == 0
        assert np.array_equal(odd[1:], want)
    finally:
        ctx.close()


def test_service_copy_equals_view(pkg):
    """The service's copy of a result above that size equals its page-locked original."""
    from jpeg2000_decoder_b200 import native, synth
    img = np.tile(synth.fields_and_edges(6, 256, 256), (1, 10, 10))[:, :2341, :2389]
    cs = native.encode(np.ascontiguousarray(img), 8, reversible=0, levels=3, num_layers=1, layer_bpp=[0.3], tile_w=1024,
                       tile_h=1024, guard_bits=1)
    srv = native.Server(0)
    try:
        rid = srv.submit(cs, native.FMT_24BITS_RGB)
        got = srv.result(rid)
        rc, view = srv.view(rid)
        assert rc == 0 and got.size == 2341 * 2389 * 3 and np.array_equal(got, view)
        srv.release(rid)
    finally:
        srv.close()
