"""Workloads of the decoder as its users run them, for timing.

Each case is one whole call through a public entry point on host codestreams (host Tier-2,
copies in, device decode, copy of the picture back), as the decoder's callers make it, or,
for the allocation-free inverse DWT, one call on device buffers.  Codestreams are written by
the package's own encoder from seeded synthetic pictures with the parameters of the
benchmark's configurations (smooth fields with edges and sensor noise, sums of sinusoids,
1/f noise), drawn on the GPU so that a state is made quickly.

kind     entry point
decode   GpuContext.decode: one picture, host to host
api      bmi_decoder_decode / bmi_decoder_result / bmi_decoder_release (BMI::Decoder)
reduced  Plan(discard_levels=...) + a one-picture batch: a picture at 1/2^n size
batch    a batch of frames: Plan on host threads, one launch, output copies behind it
serve    Server.submit ... result ... release: a burst of mixed requests
idwt     j2k_gpu_tile_idwt_noalloc: one tile-component between device buffers
"""
import ctypes
import importlib.util
import math
import os
import random
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    name = "jpeg2000_decoder_b200"
    if name not in sys.modules:
        path = os.path.join(ROOT, "jpeg2000-decoder_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(path, "__init__.py"),
                                                      submodule_search_locations=[path])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


_package()
from jpeg2000_decoder_b200 import native  # noqa: E402

# bpp 0 is lossless 5/3 (RCT on three components), anything else 9/7 (ICT) at that rate;
# bypass adds BYPASS + RESET, 32x32 blocks, RPCL order and eight layers
PICTURE = dict(width=0, height=0, ncomp=3, depth=8, bpp=0.0, tile=0, layers=1, bypass=False, content="fields")


def _picture(name, kind, width, height, **kw):
    return dict(PICTURE, name=name, kind=kind, width=width, height=height, **kw)


def listed():
    return [
        # the smallest request of a serving mix: a 256x256 preview
        _picture("call_rgb256_lossy", "decode", 256, 256, bpp=1.0),
        # one gray 512x512 lossless picture (the plain single-picture configuration)
        _picture("call_gray512_lossless", "decode", 512, 512, ncomp=1, content="waves"),
        # an odd-sized 12-bit photograph, packed into 48-bit RGB
        _picture("call_ragged_12bit_lossy", "decode", 1021, 677, depth=12, bpp=2.0),
        # a 1080p lossless picture through the drop-in decoder API
        _picture("api_rgb1080_lossless", "api", 1920, 1080),
        # one 2048x2048 RGB picture at about 1 bpp
        _picture("call_rgb2048_lossy", "decode", 2048, 2048, bpp=1.0),
        # a 2K 12-bit lossless master with coding bypass: uneven bit-planes, small blocks
        _picture("call_2k_12bit_bypass", "decode", 2048, 1080, depth=12, bypass=True, content="fractal"),
        # one 4K 12-bit distribution picture
        _picture("call_uhd_12bit_lossy", "decode", 4096, 2160, depth=12, bpp=1.5),
        # browsing: the 2048x2048 picture at an eighth of its size
        _picture("reduced_rgb2048", "reduced", 2048, 2048, bpp=1.0, discard=3),
        # batched video: 32 1080p frames, tiled, three quality layers
        _picture("batch_video_1080p", "batch", 1920, 1080, bpp=2.0, tile=512, layers=3, frames=32, distinct=8),
        # a burst of requests of mixed size, depth and wavelet through the service
        dict(name="serve_mixed_burst", kind="serve", requests=24, distinct=6, max_height=2160),
        # reconstruction alone, between device buffers: a 4K luma plane, a small ragged tile
        dict(name="idwt97_uhd_plane", kind="idwt", width=4096, height=2160, levels=5, bpp=1.0),
        dict(name="idwt53_ragged_tile", kind="idwt", width=1000, height=777, levels=5, bpp=0.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "api", "reduced", "batch", "serve", "idwt"])
    if kind == "idwt":
        return dict(kind=kind, width=_log_int(rng, 64, 4096), height=_log_int(rng, 64, 2160),
                    levels=rng.randint(1, 6), bpp=rng.choice([0.0, 1.0]))
    if kind == "serve":
        n = rng.randint(4, 24)
        return dict(kind=kind, requests=n, distinct=min(n, rng.randint(2, 8)), max_height=rng.choice([512, 1080, 2160]))
    lossy = rng.random() < 0.5
    c = dict(PICTURE, kind=kind, width=_log_int(rng, 96, 4096), height=_log_int(rng, 96, 2160),
             ncomp=rng.choice([1, 3, 3, 3]), depth=rng.choice([8, 8, 12]),
             bpp=round(rng.uniform(0.5, 2.0), 2) if lossy else 0.0, content=rng.choice(["fields", "fields", "waves", "fractal"]))
    if kind == "batch":
        c.update(width=_log_int(rng, 256, 1920), height=_log_int(rng, 256, 1080), ncomp=3, tile=rng.choice([0, 512]),
                 layers=3 if lossy else 1, frames=rng.randint(2, 16 if lossy else 6), distinct=2)
    elif kind == "reduced":
        c.update(discard=rng.randint(1, 3))
    elif not lossy and rng.random() < 0.3:
        c.update(depth=12, bypass=True, ncomp=3, width=min(c["width"], 2048), height=min(c["height"], 1080))
    return c


# ------------------------------------------------------------------ inputs -------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _image(seed, width, height, ncomp, depth, content, sigma=4.0):
    """(ncomp, height, width) uint16 picture on the host."""
    rng, gen = random.Random(int(seed)), _generator(seed)
    y = torch.arange(height, device="cuda", dtype=torch.float32)[:, None]
    x = torch.arange(width, device="cuda", dtype=torch.float32)[None, :]
    out = torch.full((ncomp, height, width), 128.0, device="cuda")
    if content == "waves":  # eight sinusoids of 8 to 256 pixels' period
        sigma = 8.0
        for _ in range(8):
            px, py = rng.uniform(8, 256), rng.uniform(8, 256)
            out += rng.uniform(8, 24) * torch.sin(2 * math.pi * (x / px + y / py) + rng.uniform(0, 2 * math.pi))
    elif content == "fractal":  # 1/f amplitude spectrum over the whole range
        sigma = 0.0
        fy = torch.fft.fftfreq(height, device="cuda")[:, None]
        fx = torch.fft.rfftfreq(width, device="cuda")[None, :]
        f2 = fx * fx + fy * fy
        f2[0, 0] = 1.0
        for c in range(ncomp):
            spec = torch.randn((2,) + f2.shape, generator=gen, device="cuda") / f2.sqrt()
            spec[:, 0, 0] = 0
            img = torch.fft.irfft2(torch.complex(spec[0], spec[1]), s=(height, width))
            out[c] = 127.5 + img * (127.5 / (2.6 * img.std().clamp_min(1e-9)))
    else:  # smooth colour fields, rectangles with sharp edges
        for c in range(ncomp):
            for _ in range(4):
                kx, ky = (rng.uniform(0.5, 3.0) * 2 * math.pi / n for n in (width, height))
                out[c] += rng.uniform(10, 40) * torch.sin(kx * x + ky * y + rng.uniform(0, 2 * math.pi))
        for _ in range(max(4, min(60, (width * height) >> 14))):
            x0, y0 = rng.randrange(width), rng.randrange(height)
            rw, rh = rng.randint(width // 40 + 1, width // 4 + 2), rng.randint(height // 40 + 1, height // 4 + 2)
            step = rng.uniform(20, 200) * rng.choice([-1, 1])
            for c in range(ncomp):
                out[c, y0:y0 + rh, x0:x0 + rw] += step * rng.uniform(0.5, 1.0)
    if sigma:
        out += sigma * torch.randn(out.shape, generator=gen, device="cuda")
    scale = (1 << depth) / 256.0
    out = (out * scale).round().clamp(0, (1 << depth) - 1)
    return out.to(torch.int32).cpu().numpy().astype(np.uint16)


def _levels(width, height, most):
    n = 0
    while n < most and min(width, height) >> (n + 1) >= 8:
        n += 1
    return n


def _encode(case, img):
    w, h = case["width"], case["height"]
    if case["bypass"]:
        return native.encode(img, case["depth"], reversible=1, levels=_levels(w, h, 6), cbw_exp=5, cbh_exp=5, num_layers=8,
                             layer_bpp=[0.5, 1, 2, 3, 4, 6, 8, 0], progression=2, mode=0x03)
    p = dict(reversible=0 if case["bpp"] else 1, levels=_levels(w, h, 5), cbw_exp=6, cbh_exp=6, num_layers=case["layers"])
    top = case["bpp"]
    p["layer_bpp"] = [top / 2 ** (case["layers"] - 1 - k) for k in range(case["layers"])]
    if case["bpp"]:
        p["guard_bits"] = 1
    if case["tile"]:
        p.update(tile_w=case["tile"], tile_h=case["tile"])
    return native.encode(img, case["depth"], **p)


def _format(case):
    if case["ncomp"] == 1:
        return native.FMT_32BITS_4COMPONENTS if case["depth"] <= 8 else native.FMT_64BITS_4COMPONENTS
    return native.FMT_24BITS_RGB if case["depth"] <= 8 else native.FMT_48BITS_RGB


SERVE_SIZES = [(256, 256), (512, 512), (1024, 1024), (1920, 1080), (4096, 2160)]


def _serve_requests(case, seed):
    """Distinct requests of the serving mix: every size in turn, half lossless 8-bit, half 8- or
    12-bit at 0.5 to 2 bpp (the 4K ones lossy)."""
    rng, mix = random.Random(int(seed)), random.Random(5)
    sizes = [s for s in SERVE_SIZES if s[1] <= case["max_height"]]
    for i in range(case["distinct"]):
        w, h = sizes[i % len(sizes)]
        lossy = h > 1080 or mix.random() < 0.5
        depth = mix.choice([8, 12]) if lossy else 8
        yield _picture("", "serve", w, h, depth=depth, bpp=rng.uniform(0.5, 2.0) if lossy else 0.0)


def _resolutions(case):
    w, h = [case["width"]], [case["height"]]
    for _ in range(_levels(case["width"], case["height"], case["levels"])):
        w.append((w[-1] + 1) // 2)
        h.append((h[-1] + 1) // 2)
    return w[::-1], h[::-1]


def _coefficients(case, seed):
    """A tile-component's coefficients in the Mallat layout: an LL band with the picture's
    range and Laplacian detail bands that fall off with the frequency."""
    gen = _generator(seed)
    rw, rh = _resolutions(case)
    n = len(rw) - 1
    u = torch.rand((case["height"], case["width"]), generator=gen, device="cuda") - 0.5
    out = -u.sign() * torch.log1p(-2 * u.abs().clamp_max(0.4999999)) * 1.5
    for r in range(n - 1, -1, -1):
        out[:rh[r], :rw[r]] *= 2.0
    ll = torch.rand((rh[0], rw[0]), generator=gen, device="cuda") * 255 - 128
    out[:rh[0], :rw[0]] = ll
    return out.round().to(torch.int32) if not case["bpp"] else out


# ------------------------------------------------------------------ program state ------
# What a program makes once and keeps: a decoder context, the drop-in decoder, the service.
_kept = {}


def _context():
    if "ctx" not in _kept:
        _kept["ctx"] = native.GpuContext(0)
    return _kept["ctx"]


def _server():
    if "server" not in _kept:
        _kept["server"] = native.Server(0)
    return _kept["server"]


def _threads():
    if "threads" not in _kept:
        _kept["threads"] = ThreadPoolExecutor(max_workers=min(16, os.cpu_count() or 1))
    return _kept["threads"]


def _api():
    if "api" not in _kept:
        lib = native.lib()
        if lib.bmi_decoder_init(1, 4) != 0:
            raise RuntimeError("bmi_decoder_init failed")
        _kept["api"] = lib
    return _kept["api"]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "idwt":
        coef = _coefficients(case, seed)
        rw, rh = _resolutions(case)
        tc = native.TileComp()
        tc.w, tc.h, tc.levels = case["width"], case["height"], len(rw) - 1
        for r in range(len(rw)):
            tc.res_w[r], tc.res_h[r] = rw[r], rh[r]
        return dict(kind=kind, tc=tc, reversible=0 if case["bpp"] else 1, coef=coef, out=torch.empty_like(coef))
    if kind == "serve":
        server = _server()
        cases = list(_serve_requests(case, seed))
        streams = list(_threads().map(
            lambda k: _encode(cases[k], _image(seed * 31 + k, cases[k]["width"], cases[k]["height"], 3, cases[k]["depth"], "fields")),
            range(len(cases))))
        queue = [k % len(streams) for k in range(case["requests"])]
        random.Random(case["requests"]).shuffle(queue)
        return dict(kind=kind, server=server, queue=[(streams[k], _format(cases[k])) for k in queue])
    if kind == "batch":
        # one scene, drifting a few pixels a frame, fresh noise on every frame
        margin = 16
        base = _image(seed, case["width"] + margin, case["height"] + margin, 3, case["depth"], case["content"], sigma=0.0)
        gen, rng = _generator(seed + 1), random.Random(int(seed))
        frames = []
        for _ in range(case["distinct"]):
            x, y = rng.randrange(margin), rng.randrange(margin)
            f = torch.from_numpy(base[:, y:y + case["height"], x:x + case["width"]].astype(np.float32)).cuda()
            f += 3.0 * (1 << case["depth"]) / 256.0 * torch.randn(f.shape, generator=gen, device="cuda")
            frames.append(f.round().clamp(0, (1 << case["depth"]) - 1).to(torch.int32).cpu().numpy().astype(np.uint16))
        streams = list(_threads().map(lambda f: _encode(case, f), frames))
        fmt = _format(case)
        size = case["width"] * case["height"] * native.FMT_BYTES[fmt]
        out = torch.empty((case["frames"], size), dtype=torch.uint8, pin_memory=True)
        return dict(kind=kind, ctx=_context(), threads=_threads(), streams=[streams[k % len(streams)] for k in range(case["frames"])],
                    fmt=fmt, out=out, size=size)
    stream = _encode(case, _image(seed, case["width"], case["height"], case["ncomp"], case["depth"], case["content"]))
    state = dict(kind=kind, stream=stream, fmt=_format(case))
    if kind == "api":
        state["api"] = _api()
    else:
        state["ctx"] = _context()
    if kind == "reduced":
        state["discard"] = min(case["discard"], _levels(case["width"], case["height"], 5))
    return state


def run(state):
    kind = state["kind"]
    if kind == "decode":
        out, rc, _, _ = state["ctx"].decode(state["stream"], state["fmt"])
        return [out, rc]
    if kind == "api":
        lib, ms, size = state["api"], ctypes.c_double(), ctypes.c_int()
        lib.bmi_decoder_set_job(state["fmt"], -1, 0, -1)
        handle = lib.bmi_decoder_decode(state["stream"], len(state["stream"]), ctypes.byref(ms))
        ptr = lib.bmi_decoder_result(handle, ctypes.byref(size))
        out = np.ctypeslib.as_array((ctypes.c_uint8 * size.value).from_address(ptr)).copy()
        lib.bmi_decoder_release(handle)
        return out
    if kind == "reduced":
        ctx = state["ctx"]
        plan = native.Plan(state["stream"], discard_levels=state["discard"])
        ctx.begin()
        slot = ctx.add(plan, state["fmt"])
        ctx.launch()
        return [ctx.sync(), ctx.output(slot)]
    if kind == "batch":
        ctx = state["ctx"]
        plans = list(state["threads"].map(native.Plan, state["streams"]))
        ctx.begin()
        slots = [ctx.add(p, state["fmt"]) for p in plans]
        ctx.launch()
        base = state["out"].data_ptr()
        for k, slot in enumerate(slots):
            ctx.output_async(slot, base + k * state["size"], state["size"])
        return [ctx.sync(), state["out"]]
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(cs, fmt) for cs, fmt in state["queue"]]
        outs = []
        for i in ids:
            outs.append(server.result(i))
            server.release(i)
        return outs
    rc = native.lib().j2k_gpu_tile_idwt_noalloc(
        ctypes.byref(state["tc"]), state["reversible"], 0, ctypes.c_void_p(state["coef"].data_ptr()),
        ctypes.c_void_p(state["out"].data_ptr()), state["tc"].w, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc != 0:
        raise RuntimeError("j2k_gpu_tile_idwt_noalloc: %d" % rc)
    return state["out"]


# ------------------------------------------------------------------ work and values ----
def _picture_work(case, scale=1.0):
    """Coded bytes in, packed pixels out; lifting (9/7: 8 operations a sample and direction over
    all levels, 5/3: 4) and the component transform."""
    px = case["width"] * case["height"] * scale
    lossless_bpp = case["ncomp"] * case["depth"] * 0.7
    coded = px * (case["bpp"] or lossless_bpp) / 8
    samples = px * case["ncomp"]
    return coded + px * native.FMT_BYTES[_format(case)], samples * (8 if case["bpp"] else 4) * 2 * 4 / 3 + px * 8


def work(case):
    kind = case["kind"]
    if kind == "idwt":
        n = case["width"] * case["height"]
        return {"bytes": 8 * n, "flops": n * (8 if case["bpp"] else 4) * 2 * 4 / 3}
    if kind == "serve":
        w = [_picture_work(c) for c in _serve_requests(case, 0)]
        share = case["requests"] / len(w)
        return {"bytes": share * sum(b for b, _ in w), "flops": share * sum(f for _, f in w)}
    scale = 1.0 / 4 ** case["discard"] if kind == "reduced" else 1.0
    b, f = _picture_work(case, scale)
    return {"bytes": b * case.get("frames", 1), "flops": f * case.get("frames", 1)}


def exact(case, seed):
    """The reconstructed plane in 64 bits (inverse lifting of T.800 Annex F on whole lines); the
    packed pictures are bytes and have to be equal, so they need no such value."""
    if case["kind"] != "idwt":
        return None
    rw, rh = _resolutions(case)
    n = len(rw) - 1
    coef = _coefficients(case, seed)
    x = coef.to(torch.float64 if case["bpp"] else torch.int64)

    def line(v):  # inverse lifting along the last axis of an interleaved plane
        size = v.shape[-1]
        if size < 2:
            return v
        even, odd = v[..., 0::2].clone(), v[..., 1::2].clone()

        def near_odd():  # the odd neighbours left and right of each even sample
            right = odd if odd.shape[-1] == even.shape[-1] else torch.cat([odd, odd[..., -1:]], -1)
            left = torch.cat([odd[..., :1], odd], -1)[..., :even.shape[-1]]
            return left, right

        def near_even():  # the even neighbours of each odd sample
            right = torch.cat([even[..., 1:], even[..., -1:]], -1)[..., :odd.shape[-1]]
            return even[..., :odd.shape[-1]], right

        if case["bpp"]:
            for step, c in enumerate((0.44350685204397, 0.88291107553093, -0.05298011857296, -1.58613434205992)):
                a, b = near_odd() if step % 2 == 0 else near_even()
                if step % 2 == 0:
                    even = even - c * (a + b)
                else:
                    odd = odd - c * (a + b)
        else:
            a, b = near_odd()
            even = even - ((a + b + 2) >> 2)
            a, b = near_even()
            odd = odd + ((a + b) >> 1)
        out = torch.empty_like(v)
        out[..., 0::2], out[..., 1::2] = even, odd
        return out

    ll = x[:rh[0], :rw[0]]
    for r in range(1, n + 1):
        lh, lw, h, w = rh[r - 1], rw[r - 1], rh[r], rw[r]
        if case["bpp"] and r > 1:
            ll = ll * 1.23017410558578 ** 2
        plane = torch.empty((h, w), dtype=x.dtype, device=x.device)
        plane[0::2, 0::2], plane[0::2, 1::2] = ll, x[:lh, lw:w]
        plane[1::2, 0::2], plane[1::2, 1::2] = x[lh:h, :lw], x[lh:h, lw:w]
        plane = line(plane)
        ll = line(plane.transpose(0, 1).contiguous()).transpose(0, 1).contiguous()
    return ll if case["bpp"] else ll.to(torch.int32)
