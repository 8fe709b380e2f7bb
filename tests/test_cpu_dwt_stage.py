"""The window staging of the inverse DWT (csrc/dwt_kernel.cuh), built for the host: every address
that it reads lies inside the level, and every position that feeds an output holds the sample
that the whole-sample symmetric extension gives."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

EDGES = (1, 2, 3, 4, 5, 31, 32, 33, 63, 64, 65, 66, 67, 68, 69, 127, 128, 129, 197)


@pytest.fixture(scope="module")
def stage(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    so = str(tmp_path_factory.mktemp("dwtstage") / "libdwt_stage_host.so")
    subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-w", "-o", so,
                    os.path.join(ROOT, "tests", "dwt_stage_host.cpp")], check=True)
    lib = ctypes.CDLL(so)
    lib.dwt_stage_host_outside.restype = ctypes.c_int64
    return lib


@pytest.mark.parametrize("tile", [64, 32])
def test_reads_stay_inside_the_level(stage, tile):
    """Lines of 1 to 200 samples across and down, lines of one sample and tile edges among them; a
    row that ends with the buffer (a tile-component one sample wide or high)."""
    bad = [(w, h) for a in range(1, 201) for e in EDGES for w, h in ((a, e), (e, a))
           if stage.dwt_stage_host_outside(tile, w, h)]
    assert not bad, bad[:20]
    for w, h in ((4096, 1), (1, 4096), (100000, 1), (1, 20001)):
        assert stage.dwt_stage_host_outside(tile, w, h) == 0, (w, h)


def _line(origin, count, n):
    """Position on the interleaved line of each window position, by reflection at both ends."""
    p = np.arange(origin - 4, origin - 4 + count)
    if n == 1:
        return np.zeros(count, np.int64)
    p = np.abs(p) % (2 * (n - 1))
    return np.where(p >= n, 2 * (n - 1) - p, p)


@pytest.mark.parametrize("tile", [64, 32])
@pytest.mark.parametrize("w,h", [(1, 1), (1, 70), (70, 1), (2, 2), (3, 5), (31, 33), (64, 64), (65, 63), (130, 200), (129, 68)])
def test_window_holds_the_extended_samples(stage, tile, w, h):
    lw, lh, stride, stride_ll = (w + 1) // 2, (h + 1) // 2, w + 3, (w + 1) // 2 + 2
    out = np.empty((tile + 8, tile + 8), np.int32)
    for oy in range(0, h, tile):
        for ox in range(0, w, tile):
            n = stage.dwt_stage_host_window(tile, w, h, stride, stride_ll, ox, oy, out.ctypes.data_as(ctypes.c_void_p))
            assert n == tile + 8 and (out >= 0).all()
            xs, ys = _line(ox, n, w), _line(oy, n, h)
            ll = ((xs & 1) == 0)[None, :] & ((ys & 1) == 0)[:, None]
            sx, sy = (xs >> 1) + (xs & 1) * lw, (ys >> 1) + (ys & 1) * lh
            want = (ll.astype(np.int64) << 30) + (sy[:, None] << 15) + sx[None, :]
            # positions up to four past the end feed outputs, on a line of one sample only its own
            ux = np.arange(ox - 4, ox - 4 + n) <= w + 3 if w > 1 else np.arange(ox - 4, ox - 4 + n) == 0
            uy = np.arange(oy - 4, oy - 4 + n) <= h + 3 if h > 1 else np.arange(oy - 4, oy - 4 + n) == 0
            used = uy[:, None] & ux[None, :]
            assert np.array_equal(out[used], want[used]), (ox, oy)
