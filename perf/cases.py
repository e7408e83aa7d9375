"""The performance cases: what a program that uses libbh.so has it do, through its public entry points.

A case is a dict with a `kind` (which entry point) and its sizes and options; `prepare` makes what a
program holds before the call, `run` is one call (a frame, a batch, a training run), `work` the bytes
and operations the call cannot do without, `exact` the same outputs in 64-bit arithmetic where such
values exist.

Rendered samples (`accum`) and bytes have no 64-bit value: the sky, the disk texture and the dither are
FP32 hashes of lattice cells, so a wider type would draw another picture, and a ray near the photon
sphere turns its last bits into its outcome.  The same holds for a ray set and for weights trained on it.
"""
import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "black-hole_b200"))

from bhrt import lib, scenes  # noqa: E402
from bhrt.abi import (BH_PREC_FP32, BH_PREC_MIXED, DERIVE_REQ_DTYPE, DERIVED_DTYPE, BHView)  # noqa: E402
from bhrt.device import Frame  # noqa: E402

SCHW, RN, KERR, KN = 0, 1, 2, 3


def listed():
    return [
        # the smallest call of an interactive viewer: a thumbnail while the camera is dragged (fast preset);
        # latency and launches count
        dict(name="frame_thumb_128x72", kind="frame", width=128, height=72, model=KN, spin=0.8, charge=0.3,
             dist=25.0, elevation=15.0, fov=45.0, preset="fast", bloom=True, spots=True, accum_mode=0,
             sample=0, precision=0),
        # one sample of a progressive render of a charged hole in a window of odd size, high quality
        dict(name="frame_rn_1283x719_accum", kind="frame", width=1283, height=719, model=RN, spin=0.0, charge=0.5,
             dist=15.0, elevation=15.0, fov=60.0, preset="high", bloom=True, spots=False, accum_mode=1,
             sample=5, precision=0),
        # the ordinary full-HD animation frame
        dict(name="frame_kerr_1080p", kind="frame", width=1920, height=1080, model=KERR, spin=0.9, charge=0.0,
             dist=20.0, elevation=10.0, fov=45.0, preset="balanced", bloom=True, spots=True, accum_mode=0,
             sample=0, precision=0),
        # the headline workload's frame: 4K Kerr-Newman orbit
        dict(name="frame_kn_4k", kind="frame", width=3840, height=2160, model=KN, spin=0.8, charge=0.3,
             dist=25.0, elevation=15.0, fov=45.0, preset="balanced", bloom=True, spots=True, accum_mode=0,
             sample=0, precision=0),
        # mixed precision on the near-extremal sweep's middle frame
        dict(name="frame_mixed_kn_4k", kind="frame", width=3840, height=2160, model=KN, spin=0.998, charge=0.05,
             dist=12.0, elevation=45.0, fov=50.0, preset="balanced", bloom=True, spots=True, accum_mode=0,
             sample=0, precision=1),
        # many views of mixed sizes and families in one call
        dict(name="batch_48_views", kind="batch", views=48),
        # the anchored surrogate frame of the headline scene (the form that takes any camera)
        dict(name="surrogate_frame_4k", kind="surrogate", width=3840, height=2160, model=KN, spin=0.8, charge=0.3,
             dist=25.0, elevation=15.0, fov=45.0, stride=8),
        # fused inference of the surrogate network for two million rays, a ragged count
        dict(name="forward_2m", kind="forward", rays=2_000_003),
        # training steps at the batch size the network is trained with
        dict(name="train_16384", kind="train", batch=16384, steps=16),
        # the RK4-traced ray set the network is trained on: 4096 rays of each view
        dict(name="generate_96_views", kind="generate", views=96, rays=4096),
        # display pass of an existing 4K accumulation buffer (exposure or bloom changed by the user)
        dict(name="post_4k", kind="post", width=3840, height=2160, bloom=True),
        # black-hole parameters of a parameter sweep derived on the device
        dict(name="derive_13824", kind="derive", count=13824),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _hole(rng):
    """A black hole of the batched workload's parameter box."""
    model = rng.randrange(4)
    while True:
        a, q = rng.uniform(-0.998, 0.998), rng.uniform(0.0, 0.6)
        if a * a + q * q <= 0.98:
            break
    return model, (a if model >= KERR else 0.0), (q if model in (RN, KN) else 0.0)


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "mixed", "batch", "surrogate", "forward", "train", "generate",
                       "post", "derive"])
    if kind == "batch":
        return dict(kind=kind, views=_log_int(rng, 3, 48))
    if kind == "forward":
        return dict(kind=kind, rays=_log_int(rng, 1000, 4_000_000))
    if kind == "train":
        return dict(kind=kind, batch=128 * _log_int(rng, 8, 192), steps=rng.randint(6, 16))
    if kind == "generate":
        return dict(kind=kind, views=_log_int(rng, 4, 96), rays=_log_int(rng, 256, 8192))
    if kind == "derive":
        return dict(kind=kind, count=_log_int(rng, 16, 16384))
    top = {"frame": 3840, "mixed": 1920, "surrogate": 3840, "post": 3840}[kind]
    width = _log_int(rng, {"frame": 96, "mixed": 160, "surrogate": 320, "post": 96}[kind], top)
    height = max(32, min(int(width * rng.choice([9 / 16, 9 / 16, 3 / 4, 0.42])), top * 9 // 16))
    if kind == "post":
        return dict(kind=kind, width=width, height=height, bloom=rng.random() < 0.75)
    model, a, q = _hole(rng)
    scene = dict(width=width, height=height, model=model, spin=a, charge=q, dist=rng.uniform(6.0, 60.0),
                 elevation=rng.uniform(2.0, 88.0), fov=rng.uniform(30.0, 90.0))
    if kind == "surrogate":
        return dict(kind=kind, stride=rng.choice([4, 8, 8]), **scene)
    mode = rng.choice([0, 0, 1, 2])
    return dict(kind="frame", preset=rng.choice(["fast", "balanced", "balanced", "high" if width <= 1920 else "fast"]),
                bloom=rng.random() < 0.75, spots=rng.random() < 0.5, accum_mode=mode,
                sample=rng.randint(0, 40) if mode else 0, precision=1 if kind == "mixed" else 0, **scene)


# ---- inputs -----------------------------------------------------------------------------------------------

def _scene(case, seed):
    """The case's view; the seed moves the camera round the hole and sets the disk time."""
    r = random.Random(1000003 * seed + 17)
    P = scenes.scene(lib.derive, case["model"], case["spin"], case["charge"], case["width"], case["height"],
                     case["dist"], case["elevation"], case["fov"], az_deg=r.uniform(0.0, 360.0),
                     preset=case.get("preset", "balanced"), hot_spots=case.get("spots", True),
                     bloom=case.get("bloom", True), disk_time=r.uniform(0.0, 4.0))
    P.accumMode, P.sampleIndex = case.get("accum_mode", 0), case.get("sample", 0)
    return P


def _batch_views(count, seed):
    """Views of the batched workload's parameter box, their sizes and holes by their number alone; the seed
    moves the cameras and sets the disk times."""
    layout, r, views = random.Random(1234), random.Random(1000003 * seed + 19), []
    for _ in range(count):
        w, h = layout.choice(scenes.BATCH_RESOLUTIONS)
        model, a, q = _hole(layout)
        dist, inc, fov = layout.uniform(6.0, 60.0), layout.uniform(2.0, 88.0), layout.uniform(30.0, 90.0)
        views.append(scenes.scene(lib.derive, model, a, q, w, h, dist, 90.0 - inc, fov, az_deg=r.uniform(0.0, 360.0),
                                  hot_spots=layout.random() < 0.5, disk_time=r.uniform(0.0, 4.0)))
    return views


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 7)
    return g


def _hdr_image(width, height, seed):
    """An accumulation buffer like a rendered one: dark sky, sparse stars, a bright disk band."""
    g = _generator(seed)
    x = torch.empty((height, width, 4), dtype=torch.float32, device="cuda")
    x[..., :3] = 0.002 + 0.03 * torch.rand((height, width, 3), generator=g, device="cuda")
    star = torch.rand((height, width, 1), generator=g, device="cuda")
    x[..., :3] += torch.where(star > 0.996, 6.0 * (star - 0.996) / 0.004, torch.zeros_like(star))
    lo, hi = int(height * 0.42), max(int(height * 0.58), int(height * 0.42) + 1)
    x[lo:hi, width // 4: max(3 * width // 4, width // 4 + 1), :3] += \
        4.0 * torch.rand((hi - lo, max(3 * width // 4, width // 4 + 1) - width // 4, 3), generator=g, device="cuda") ** 3
    x[..., 3] = 1.0
    return x


def _net_inputs(rays, seed):
    """Camera-basis unit directions within 45 degrees of the axis and one scene's inputs per 4096 rays."""
    g = _generator(seed)
    x = torch.zeros((rays, 8), dtype=torch.float32, device="cuda")
    d = torch.rand((rays, 2), generator=g, device="cuda") * 2 - 1
    v = torch.cat([d, torch.ones((rays, 1), device="cuda")], 1)
    x[:, :3] = v / v.norm(dim=1, keepdim=True)
    views = -(-rays // 4096)
    x[:, 3:7] = (torch.rand((views, 4), generator=g, device="cuda") * 2 - 1).repeat_interleave(4096, 0)[:rays]
    return x


def _net_params(seed):
    """A network's parameter vector: four 256 x 256 layers and the 16 x 256 head, each followed by its biases."""
    rng = np.random.default_rng(seed + 11)
    parts = []
    for out in (256, 256, 256, 256, 16):
        lim = math.sqrt(6.0 / (256 + out))
        parts += [rng.uniform(-lim, lim, out * 256), rng.uniform(-0.05, 0.05, out)]
    return np.concatenate(parts).astype(np.float32)


def _derive_requests(count, seed):
    rng = np.random.default_rng(seed + 13)
    r = np.zeros(count, DERIVE_REQ_DTYPE)
    r["model"] = rng.integers(0, 4, count)
    r["M"] = rng.uniform(0.3, 1.5, count)
    r["aStar"] = rng.uniform(-0.998, 0.998, count)
    r["q"] = rng.uniform(0.0, 0.6, count)
    return r


class _Net:
    """A surrogate handle, released with the object."""

    def __init__(self, seed):
        self.L = lib.load()
        self.h = C.c_void_p()
        lib.check(self.L.bhSurrogateCreate(C.byref(self.h), C.c_uint(seed & 0x7FFFFFFF)), "bhSurrogateCreate")

    def __del__(self):
        if self.h:
            self.L.bhSurrogateDestroy(self.h)


class _DeviceArray:
    """Device memory of a handle, seen as a tensor while the handle lives."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f4", "version": 2}


def _p(t):
    return C.c_void_p(t.data_ptr())


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def prepare(case, seed):
    kind = case["kind"]
    L = lib.load()
    s = dict(kind=kind, L=L)
    if kind in ("frame", "surrogate"):
        s["P"] = _scene(case, seed)
        s["frame"] = Frame(case["width"], case["height"])
        if case.get("sample", 0):
            s["frame"].accum.copy_(_hdr_image(case["width"], case["height"], seed))
        s["precision"] = BH_PREC_MIXED if case.get("precision", 0) else BH_PREC_FP32
        if kind == "surrogate":
            s["net"] = _Net(seed)
            lib.check(L.bhSurrogateSetAnchors(s["net"].h, case["stride"], 0, C.c_float(1e-4), C.c_float(0.5)),
                      "bhSurrogateSetAnchors")
    elif kind == "batch":
        views = _batch_views(case["views"], seed)
        pixels = [P.width * P.height for P in views]
        half = [((P.width + 1) // 2) * ((P.height + 1) // 2) for P in views]
        s["out"] = torch.zeros((sum(pixels), 4), dtype=torch.uint8, device="cuda")
        s["accum"] = torch.zeros((sum(pixels), 4), dtype=torch.float32, device="cuda")
        s["bloomA"] = torch.zeros((sum(half), 4), dtype=torch.float32, device="cuda")
        s["bloomB"] = torch.zeros((sum(half), 4), dtype=torch.float32, device="cuda")
        s["views"], s["n"] = (BHView * len(views))(), len(views)
        at = ah = 0
        for v, P, n, m in zip(s["views"], views, pixels, half):
            v.params = P
            v.out, v.accum = s["out"].data_ptr() + 4 * at, s["accum"].data_ptr() + 16 * at
            v.bloomA, v.bloomB = s["bloomA"].data_ptr() + 16 * ah, s["bloomB"].data_ptr() + 16 * ah
            at, ah = at + n, ah + m
    elif kind == "forward":
        s["net"] = _Net(seed)
        params = _net_params(seed)
        lib.check(L.bhSurrogateSetParams(s["net"].h, params.ctypes.data_as(C.c_void_p)), "bhSurrogateSetParams")
        s["in"] = _net_inputs(case["rays"], seed)
        s["out"] = torch.zeros((case["rays"], 16), dtype=torch.float32, device="cuda")
    elif kind == "train":
        s["net"] = _Net(seed)
        lib.check(L.bhSurrogateGenerate(s["net"].h, C.c_longlong(16 * 4096), 16, C.c_uint(seed & 0x7FFFFFFF)),
                  "bhSurrogateGenerate")
        s["batch"], s["steps"], s["seed"] = case["batch"], case["steps"], seed & 0x7FFFFFFF
        s["loss"] = np.zeros((case["steps"], 5), np.float32)
        s["params"] = np.zeros(L.bhSurrogateParamCount(), np.float32)
    elif kind == "generate":
        s["net"] = _Net(seed)
        s["views"], s["rays"], s["seed"] = case["views"], case["views"] * case["rays"], seed & 0x7FFFFFFF
    elif kind == "post":
        s["P"] = scenes.scene(lib.derive, KN, 0.8, 0.3, case["width"], case["height"], 25.0, 15.0, 45.0,
                              bloom=case["bloom"])
        s["frame"] = Frame(case["width"], case["height"])
        s["frame"].accum.copy_(_hdr_image(case["width"], case["height"], seed))
    else:
        r = _derive_requests(case["count"], seed)
        s["requests"] = torch.from_numpy(r.view(np.uint8).reshape(-1)).cuda()
        s["derived"] = torch.zeros(case["count"] * DERIVED_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
        s["n"] = case["count"]
    return s


# ---- one pass ---------------------------------------------------------------------------------------------

def run(s):
    kind, L = s["kind"], s["L"]
    if kind == "frame":
        f = s["frame"]
        f.pipeline(s["P"], s["precision"])
        return dict(out=f.out, accum=f.accum, bloomA=f.bloomA, bloomB=f.bloomB)
    if kind == "surrogate":
        f = s["frame"]
        lib.check(L.bhSurrogateRender(s["net"].h, _p(f.out), _p(f.accum), _p(f.bloomA), _p(f.bloomB),
                                      C.byref(s["P"]), _stream()), "bhSurrogateRender")
        return dict(out=f.out, accum=f.accum, bloomA=f.bloomA, bloomB=f.bloomB)
    if kind == "batch":
        lib.check(L.bhRenderBatch(s["views"], s["n"], _stream()), "bhRenderBatch")
        return dict(out=s["out"], accum=s["accum"], bloomA=s["bloomA"], bloomB=s["bloomB"])
    if kind == "forward":
        lib.check(L.bhSurrogateForward(s["net"].h, _p(s["in"]), _p(s["out"]), s["in"].shape[0], 1, _stream()),
                  "bhSurrogateForward")
        return s["out"]
    if kind == "train":
        lib.check(L.bhSurrogateTrain(s["net"].h, s["steps"], s["batch"], C.c_float(2e-3), C.c_uint(s["seed"]),
                                     s["loss"].ctypes.data_as(C.c_void_p)), "bhSurrogateTrain")
        lib.check(L.bhSurrogateGetParams(s["net"].h, s["params"].ctypes.data_as(C.c_void_p)), "bhSurrogateGetParams")
        return dict(loss=s["loss"], params=s["params"])
    if kind == "generate":
        lib.check(L.bhSurrogateGenerate(s["net"].h, C.c_longlong(s["rays"]), s["views"], C.c_uint(s["seed"])),
                  "bhSurrogateGenerate")
        x, t, n = C.c_void_p(), C.c_void_p(), C.c_longlong()
        lib.check(L.bhSurrogateDataset(s["net"].h, C.byref(x), C.byref(t), C.byref(n)), "bhSurrogateDataset")
        # copies: the ray set goes with the handle
        return dict(inputs=torch.as_tensor(_DeviceArray(x.value, (n.value, 8)), device="cuda").clone(),
                    targets=torch.as_tensor(_DeviceArray(t.value, (n.value, 8)), device="cuda").clone())
    if kind == "post":
        f = s["frame"]
        f.post(s["P"])
        return dict(out=f.out, bloomA=f.bloomA, bloomB=f.bloomB)
    lib.check(L.bhDeriveBatch(_p(s["requests"]), _p(s["derived"]), s["n"], _stream()), "bhDeriveBatch")
    d = s["derived"].view(torch.float32).view(-1, 9)
    return dict(radii=d[:, 0:6], isco=d[:, 6], flags=s["derived"].view(torch.int32).view(-1, 9)[:, 7:9],
                requests=s["requests"].view(torch.float32).view(-1, 5)[:, 1:4])


# ---- what one pass cannot do without ------------------------------------------------------------------------

# Operations of an RK4 step (Kerr family, spherical family) and the mean steps of a ray at the balanced
# preset on the headline scene; the step count goes with 1 / dPhi.
_STEP_FLOPS = {False: 115.0, True: 420.0}
_STEPS = 196.0
_NET_FLOPS = 2.0 * (4 * 256 * 256 + 256 * 16)


def _trace_flops(pixels, model, preset="balanced"):
    return pixels * _STEPS * scenes.PRESETS["balanced"][0] / scenes.PRESETS[preset][0] * _STEP_FLOPS[model >= KERR]


def _post_bytes(pixels, bloom):
    """Accumulation read, RGBA8 written; with bloom the two half-resolution images written."""
    return pixels * (16 + 4 + (8 if bloom else 0))


def work(case):
    kind = case["kind"]
    if kind in ("frame", "surrogate"):
        n = case["width"] * case["height"]
        flops = _trace_flops(n, case["model"], case.get("preset", "balanced"))
        if kind == "surrogate":
            flops /= case["stride"] ** 2      # the anchors; how much of the rest is traced is the scene's
        return dict(bytes=n * (16 if not case.get("sample", 0) else 32) + _post_bytes(n, case.get("bloom", True)),
                    flops=flops)
    if kind == "batch":
        views = _batch_views(case["views"], 0)
        return dict(bytes=sum(P.width * P.height * 44 for P in views),
                    flops=sum(_trace_flops(P.width * P.height, P.model) for P in views))
    if kind == "forward":
        return dict(bytes=case["rays"] * (32 + 64), flops=case["rays"] * _NET_FLOPS)
    if kind == "train":
        params = 4 * 256 * 257 + 16 * 257
        return dict(bytes=case["steps"] * (case["batch"] * 64 + params * 4 * 7),
                    flops=case["steps"] * case["batch"] * 3 * _NET_FLOPS)
    if kind == "generate":
        n = case["views"] * case["rays"]
        return dict(bytes=n * 64, flops=_trace_flops(n, KERR) / 2 + _trace_flops(n, SCHW) / 2)
    if kind == "post":
        n = case["width"] * case["height"]
        return dict(bytes=_post_bytes(n, case["bloom"]), flops=n * 150)
    # 12000 radii of the numeric ISCO scan at most, 30 operations each
    return dict(bytes=case["count"] * 56, flops=case["count"] * 10000 * 30)


# ---- 64-bit values ------------------------------------------------------------------------------------------

_GAUSS9 = (0.02907, 0.06794, 0.12458, 0.17925, 0.20236, 0.17925, 0.12458, 0.06794, 0.02907)


def _blur(x, dim):
    """9-tap Gaussian along `dim`, clamped to the edge; channels last."""
    n = x.shape[dim]
    at = torch.arange(n, device=x.device)
    y = torch.zeros_like(x)
    for k, w in enumerate(_GAUSS9):
        y += w * x.index_select(dim, (at + k - 4).clamp(0, n - 1))
    return y


def _exact_post(case, seed):
    if not case["bloom"]:
        return None          # bytes, and two buffers that are not written
    x = _hdr_image(case["width"], case["height"], seed)[..., :3].double()
    x = torch.cat([x, x[-1:]], 0) if x.shape[0] % 2 else x
    x = torch.cat([x, x[:, -1:]], 1) if x.shape[1] % 2 else x
    half = (x[0::2, 0::2] + x[0::2, 1::2] + x[1::2, 0::2] + x[1::2, 1::2]) * 0.25
    lum = 0.2126 * half[..., 0] + 0.7152 * half[..., 1] + 0.0722 * half[..., 2]
    t = ((lum - 0.95) / (2.2 - 0.95)).clamp(0, 1)
    bright = half * (t * t * (3 - 2 * t))[..., None]
    h = _blur(bright, 1)
    v = _blur(h, 0)
    one = torch.ones_like(h[..., :1])
    return dict(out=None, bloomA=torch.cat([v, one], -1), bloomB=torch.cat([h, one], -1))


def _exact_forward(case, seed):
    p = torch.from_numpy(_net_params(seed)).cuda().double()
    x = _net_inputs(case["rays"], seed)
    w = math.pi * torch.pow(2.0, 0.5 * torch.arange(16, device="cuda", dtype=torch.float64))
    out = torch.empty((case["rays"], 16), dtype=torch.float64, device="cuda")
    for at in range(0, case["rays"], 1 << 18):
        v = x[at:at + (1 << 18), :7].double()
        a = v[:, :, None] * w
        h = torch.cat([torch.stack([a.sin(), a.cos()], -1).flatten(1), v,
                       torch.zeros((v.shape[0], 25), device="cuda", dtype=torch.float64)], 1)
        k = 0
        for n in (256, 256, 256, 256, 16):
            h = h @ p[k:k + n * 256].view(n, 256).T + p[k + n * 256:k + n * 257]
            k += n * 257
            if n == 256:
                h = 0.5 * h * (1 + torch.tanh(math.sqrt(2 / math.pi) * (h + 0.044715 * h ** 3)))
        out[at:at + (1 << 18)] = h
    return out


def _exact_derive(case, seed):
    """Horizons, photon orbit and ergosphere in closed form.  The ISCO has none here: it is the radius of a
    numeric scan whose energies differ by less than an FP32 ulp near their minimum."""
    r = _derive_requests(case["count"], seed)
    kerr, charged = r["model"] >= KERR, (r["model"] % 2) == 1
    M, a, q = (r[k].astype(np.float64) for k in ("M", "aStar", "q"))
    a = np.clip(a, -0.995, 0.995)
    ae, qe = np.where(kerr, a, 0.0), np.where(charged, q, 0.0)
    s2 = ae * ae + qe * qe
    k = np.where(s2 > 0.995, np.sqrt(0.995 / np.maximum(s2, 1e-30)), 1.0)
    ae, qe = ae * k, qe * k
    a, q = np.where(kerr, ae, a), np.where(charged, qe, q)
    A, Q = ae * M, qe * M
    root = np.sqrt(np.maximum(M * M - A * A - Q * Q, 0))
    rs = 0.5 * (3 * M + np.sqrt(9 * M * M - 8 * Q * Q))
    rk = 2 * M * (1 + np.cos(2 / 3 * np.arccos(np.clip(-ae, -1, 1))))
    w = qe * qe
    rot = np.where(r["model"] == KN, np.where(np.abs(ae) < 1e-5, rs, (1 - 0.35 * w) * rk + 0.35 * w * rs), rk)
    photon = np.where(kerr, np.maximum(rot, 1.02 * (M + root)), rs)
    radii = np.stack([A, Q, M + root, M - root, photon, M + np.sqrt(M * M - Q * Q)], 1)
    return dict(radii=radii, isco=None, flags=None, requests=np.stack([M, a, q], 1))


def exact(case, seed):
    if case["kind"] == "post":
        return _exact_post(case, seed)
    if case["kind"] == "forward":
        return _exact_forward(case, seed)
    if case["kind"] == "derive":
        return _exact_derive(case, seed)
    return None
