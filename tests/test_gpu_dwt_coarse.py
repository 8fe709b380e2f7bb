"""Both ways to run the coarse DWT levels (dwt_coarse 1: one shared-memory kernel, 2: a launch per
level) against the oracle, tolerance 0: every golden stream, odd and tiny pictures, and tiles one
sample high or wide, 5/3 (also with the reference's column end) and 9/7."""
import os

import numpy as np
import pytest

import oracle_util
from conftest import ROOT

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(ROOT, "tests", "golden")


def _check(ctx, cs, flags):
    from jpeg2000_decoder_b200 import native
    plan = native.Plan(cs)
    fmt = native.FMT_32BITS_4COMPONENTS if plan.info.ncomp == 1 else (
        native.FMT_48BITS_RGB if plan.info.bitdepth > 8 else native.FMT_24BITS_RGB)
    _, want, _ = oracle_util.oracle_decode(plan, fmt, ref_compat=1 if flags & native.FLAG_REF_COMPAT else 0)
    # the fused last level, and levels and output apart
    for keep in (0, native.FLAG_KEEP_COMPONENTS):
        out, rc, bad, _ = ctx.decode(cs, fmt, flags | keep)
        assert rc == native.J2K_OK and bad == 0
        assert np.array_equal(out, want), (flags, keep)


@pytest.fixture(params=[1, 2])
def coarse_ctx(gpu_ctx, request):
    gpu_ctx.set_tuning(dwt_coarse=request.param)
    yield gpu_ctx
    gpu_ctx.set_tuning()


@pytest.mark.parametrize("flags", [0, 1])
@pytest.mark.parametrize("name", sorted(n for n in os.listdir(GOLDEN) if n.endswith(".j2k")))
def test_golden_streams(coarse_ctx, name, flags):
    with open(os.path.join(GOLDEN, name), "rb") as f:
        _check(coarse_ctx, f.read(), flags)


@pytest.mark.parametrize("reversible", [0, 1])
@pytest.mark.parametrize("w,h,levels,tile", [(1, 1, 1, 0), (1, 70, 3, 0), (70, 1, 3, 0), (3, 5, 2, 0), (33, 31, 4, 0),
                                             (64, 65, 5, 0), (129, 127, 6, 0), (65, 129, 3, 64), (129, 64, 5, 32),
                                             (200, 97, 2, 32)])
def test_geometries(coarse_ctx, w, h, levels, tile, reversible):
    from jpeg2000_decoder_b200 import native, synth
    img = np.ascontiguousarray(synth.fields_and_edges(w + h, max(h, 16), max(w, 16))[:, :h, :w])
    kw = dict(tile_w=tile, tile_h=tile) if tile else {}
    cs = native.encode(img, 8, reversible=reversible, levels=levels, num_layers=1, layer_bpp=[0 if reversible else 4], **kw)
    for flags in ((0, 1) if reversible else (0,)):
        _check(coarse_ctx, cs, flags)
