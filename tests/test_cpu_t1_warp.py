"""The one-block-per-warp Tier-1 decoder (csrc/t1_kernel.cuh), built for the host with its 32
lanes as fibers, against the reference's Tier-1 digests and the oracle, block by block: both
kernel forms, every mode switch, all block shapes, cut and corrupted segments."""
import ctypes
import hashlib
import json
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle_util
from conftest import ROOT

GOLDEN = os.path.join(ROOT, "tests", "golden")


@pytest.fixture(scope="module")
def warp(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    so = str(tmp_path_factory.mktemp("t1warp") / "libt1_warp_host.so")
    subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-w", "-U_FORTIFY_SOURCE", "-o", so,
                    os.path.join(ROOT, "tests", "t1_warp_host.cpp")], check=True)
    return ctypes.CDLL(so)


def _block(lib, cb, data, seglens, latency):
    out = np.zeros(cb.w * cb.h, np.int32)
    rc = lib.t1_warp_host_block(ctypes.byref(cb), data, seglens, latency, out.ctypes.data_as(ctypes.c_void_p))
    return rc, out


def _check(lib, cs, most=None):
    """The first `most` blocks of a codestream (all when None): rows of both forms against the
    oracle."""
    from jpeg2000_decoder_b200 import native
    plan = native.Plan(cs)
    cbs = plan.cblks()
    n = plan.info.num_cblks
    for i in range(n if most is None else min(n, most)):
        orc, want = oracle_util.oracle_block(plan, i)
        for latency in (0, 1):
            rc, out = _block(lib, cbs[i], plan.bytes_ptr(), plan.seglens_ptr(), latency)
            assert rc == orc and np.array_equal(out, want), ("block", i, latency)
    return n


@pytest.mark.parametrize("name", [k for k, v in json.load(open(os.path.join(GOLDEN, "golden.json"))).items()
                                  if "reference_t1_sha256_16" in v])
def test_matches_reference_golden(pkg, warp, name):
    from jpeg2000_decoder_b200 import native
    g = json.load(open(os.path.join(GOLDEN, "golden.json")))[name]
    with open(os.path.join(GOLDEN, name), "rb") as f:
        plan = native.Plan(f.read())
    cbs = plan.cblks()
    for i in range(plan.info.num_cblks):
        rc, out = _block(warp, cbs[i], plan.bytes_ptr(), plan.seglens_ptr(), i & 1)
        assert rc == 0
        assert hashlib.sha256(out.tobytes()).hexdigest()[:16] == g["reference_t1_sha256_16"][i], (name, i)


@pytest.mark.parametrize("mode", [0x00, 0x01, 0x02, 0x03, 0x04, 0x05, 0x08, 0x10, 0x20, 0x2E, 0x3F])
def test_mode_switches(pkg, warp, mode):
    """Bypass, context reset, per-pass termination, stripe-causal contexts, predictable
    termination, segmentation symbols and combinations."""
    from jpeg2000_decoder_b200 import native, synth
    img = synth.fractal_rgb(13, 70, 133, bitdepth=12)
    cs = native.encode(img, 12, reversible=1, levels=3, cbw_exp=5, cbh_exp=5, num_layers=3, layer_bpp=[1, 3, 0],
                       mode=mode)
    assert _check(warp, cs) > 0


@pytest.mark.parametrize("cw,ch", [(6, 6), (6, 4), (4, 6), (3, 3), (6, 2), (2, 6), (5, 6), (2, 2)])
def test_block_shapes(pkg, warp, cw, ch):
    """Blocks from 4x4 to 64x64 with ragged edges (one and two chunks, partial stripes), 5/3 and
    9/7."""
    from jpeg2000_decoder_b200 import native, synth
    img = synth.fractal_rgb(14, 67, 131)
    for kw in (dict(reversible=0, layer_bpp=[1, 4]), dict(reversible=1, layer_bpp=[1, 0])):
        assert _check(warp, native.encode(img, 8, levels=2, cbw_exp=cw, cbh_exp=ch, num_layers=2, **kw)) > 0


@pytest.mark.parametrize("mode", [0x00, 0x01, 0x05])
def test_cut_and_corrupted_segments(pkg, warp, mode):
    """Segments cut at every length class, 0xFF runs, bytes 0x80..0x8F after 0xFF (the carry of
    the bit-stuffing rule) and 0x90.. (markers): the decoder's registers hold more code than
    the reference's, and must still see each byte when the reference does."""
    from jpeg2000_decoder_b200 import native, synth
    img = synth.fields_and_edges(15, 64, 64)[:1]
    plan = native.Plan(native.encode(img, 8, reversible=1, levels=1, cbw_exp=5, cbh_exp=5, num_layers=1, layer_bpp=[0],
                                     mode=mode))
    rng = np.random.default_rng(16)
    cbs = plan.cblks()
    size = int(plan.info.coded_bytes)
    good = np.ctypeslib.as_array((ctypes.c_uint8 * size).from_address(plan.bytes_ptr().value)).copy()
    for trial in range(120):
        cb = cbs[int(rng.integers(0, plan.info.num_cblks))]
        if cb.data_len < 8:
            continue
        data = np.zeros(size + 16, np.uint8)
        data[:size] = good
        a = cb.data_off
        kind = trial % 4
        if kind == 0:    # cut (and, with several segments, a table that asks for too much)
            cb = type(cb).from_buffer_copy(cb)
            cb.data_len = int(rng.integers(0, cb.data_len))
        elif kind == 1:  # stuffed carries and markers
            for _ in range(6):
                at = a + int(rng.integers(0, cb.data_len - 1))
                data[at] = 0xFF
                data[at + 1] = int(rng.integers(0x70, 0xA0))
        elif kind == 2:  # a run of 0xFF
            at = a + int(rng.integers(0, cb.data_len))
            data[at:min(at + 5, a + cb.data_len)] = 0xFF
        else:            # noise rich in 0xFF
            n = cb.data_len
            noise = rng.integers(0, 256, n, dtype=np.uint8)
            noise[rng.random(n) < 0.2] = 0xFF
            data[a:a + n] = noise
        out = np.zeros(cb.w * cb.h, np.int32)
        orc = oracle_util.orc().oracle_t1_block(ctypes.byref(cb), data.ctypes.data_as(ctypes.c_void_p), plan.seglens_ptr(),
                                                out.ctypes.data_as(ctypes.c_void_p))
        for latency in (0, 1):
            rc, got = _block(warp, cb, data.ctypes.data_as(ctypes.c_void_p), plan.seglens_ptr(), latency)
            assert rc == orc, (trial, kind, latency)
            assert np.array_equal(got, out), (trial, kind, latency)


def test_random_configurations(pkg, warp):
    import tier2_streams as ts
    for i, (kw, depth, h, w) in enumerate(ts.random_cases(2027, 12)):
        _, cs = ts.random_case_stream(2027, i, kw, depth, h, w)
        _check(warp, cs, most=12)


@pytest.mark.parametrize("latency", [0, 1])
def test_symbols_around_stuffed_bytes(warp, latency):
    """Encoded symbols come back where 0xFF bytes and carries into the byte after them are
    common: a carry must not be compared before it is due, nor a bit be missing between the two
    symbols of a pair."""
    carries = 0
    for seed in range(1, 601):
        c = ctypes.c_int()
        n = seed if seed < 40 else 200000
        assert warp.t1_warp_host_symbols(seed * 7919 + 1, n, 5 if seed % 8 == 0 else n + 1, latency, ctypes.byref(c)) == 0
        carries += c.value
    assert carries > 250000
