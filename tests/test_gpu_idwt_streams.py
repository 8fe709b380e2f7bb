"""The allocation-free inverse DWT where its callers run it: captured into a graph that is replayed
on new coefficients, on a stream that may use only some of the SMs, and behind work of the same and
of other streams that is still running when the call is made.  The values are those of a call on an
idle stream, bit for bit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tile(w, h, levels):
    from jpeg2000_decoder_b200 import native
    tc = native.TileComp()
    tc.w, tc.h, tc.levels = w, h, levels
    for r in range(levels, -1, -1):
        tc.res_w[r], tc.res_h[r] = w, h
        w, h = (w + 1) // 2, (h + 1) // 2
    return tc


def _call(tc, rev, src, out, stream):
    from jpeg2000_decoder_b200 import native
    return native.lib().j2k_gpu_tile_idwt_noalloc(ctypes.byref(tc), rev, 0, ctypes.c_void_p(src.data_ptr()),
                                                  ctypes.c_void_p(out.data_ptr()), tc.w, ctypes.c_void_p(stream))


def _coefficients(seed, tc, rev):
    import torch
    rng = np.random.default_rng(seed)
    c = rng.integers(-500, 500, (tc.h, tc.w)).astype(np.int32)
    return torch.from_numpy(c if rev else c.astype(np.float32) / 7).cuda()


SHAPES = [(1000, 777, 5), (70, 1, 3), (2049, 1030, 6), (65, 63, 1)]


@pytest.mark.parametrize("rev", [0, 1])
@pytest.mark.parametrize("w,h,levels", SHAPES)
def test_captured_call_replays_on_new_coefficients(pkg, rev, w, h, levels):
    import torch
    tc = _tile(w, h, levels)
    inputs = [_coefficients(s, tc, rev) for s in range(3)]
    want = []
    for c in inputs:
        out = torch.empty_like(c)
        assert _call(tc, rev, c, out, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        want.append(out.cpu().numpy())
    src, out = inputs[0].clone(), torch.zeros_like(inputs[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert _call(tc, rev, src, out, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert not out.any()  # recorded, not run
    for k in (1, 2, 0):
        src.copy_(inputs[k])
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().view(np.int32), want[k].view(np.int32)), k


@pytest.mark.parametrize("rev", [0, 1])
def test_stream_of_a_few_sms(pkg, rev):
    """A green context of 16 SMs: the levels' CTAs run there in turn."""
    import torch
    drv = pytest.importorskip("cuda.bindings.driver")
    torch.cuda.init()

    def ck(r):
        assert r[0] == drv.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else r[1:]
    dev = ck(drv.cuDeviceGet(torch.cuda.current_device()))
    sms = ck(drv.cuDeviceGetDevResource(dev, drv.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups = ck(drv.cuDevSmResourceSplitByCount(1, sms, 0, 16))[0]
    desc = ck(drv.cuDevResourceGenerateDesc(groups[:1], 1))
    green = ck(drv.cuGreenCtxCreate(desc, dev, drv.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = ck(drv.cuGreenCtxStreamCreate(green, drv.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    try:
        for w, h, levels in SHAPES:
            tc = _tile(w, h, levels)
            src = _coefficients(w, tc, rev)
            want, out = torch.empty_like(src), torch.zeros_like(src)
            assert _call(tc, rev, src, want, torch.cuda.current_stream().cuda_stream) == 0
            torch.cuda.synchronize()
            assert _call(tc, rev, src, out, int(stream)) == 0
            ck(drv.cuStreamSynchronize(stream) + (None,))
            assert np.array_equal(out.cpu().numpy().view(np.int32), want.cpu().numpy().view(np.int32)), (w, h)
    finally:
        drv.cuStreamDestroy(stream)
        drv.cuGreenCtxDestroy(green)


@pytest.mark.parametrize("behind", ["same stream", "event", "legacy stream"])
@pytest.mark.parametrize("rev", [0, 1])
@pytest.mark.parametrize("w,h,levels", SHAPES)
def test_coefficients_that_are_still_being_written(pkg, rev, w, h, levels, behind):
    """The call sees what earlier work writes to its coefficients, and what follows it sees its
    result: work enqueued on the same stream, work of another stream joined by an event, and work
    of a blocking stream, which the legacy default stream waits for."""
    import torch
    rt = pytest.importorskip("cuda.bindings.runtime")
    tc = _tile(w, h, levels)
    new, old = _coefficients(5, tc, rev), _coefficients(6, tc, rev)
    want = torch.empty_like(new)
    assert _call(tc, rev, new, want, 0) == 0
    torch.cuda.synchronize()
    src, out, after = old.clone(), torch.zeros_like(new), torch.zeros_like(new)
    torch.cuda.synchronize()
    err, other = rt.cudaStreamCreate()  # a blocking stream
    assert err == rt.cudaError_t.cudaSuccess
    writer = torch.cuda.ExternalStream(int(other))
    caller = torch.cuda.default_stream() if behind == "legacy stream" else torch.cuda.Stream()
    if behind == "same stream":
        writer = caller
    with torch.cuda.stream(caller):
        after.fill_(1)  # a kernel right before the call
    with torch.cuda.stream(writer):
        torch.cuda._sleep(4000000)  # about 2 ms
        src.copy_(new)
        if behind == "event":
            done = torch.cuda.Event()
            done.record(writer)
    if behind == "event":
        caller.wait_event(done)
    assert _call(tc, rev, src, out, caller.cuda_stream) == 0
    with torch.cuda.stream(caller):
        after.copy_(out)
    torch.cuda.synchronize()
    assert np.array_equal(after.cpu().numpy().view(np.int32), want.cpu().numpy().view(np.int32))
    rt.cudaStreamDestroy(other)
