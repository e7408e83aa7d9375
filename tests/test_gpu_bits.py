"""Results whose bits are pinned: frames of every family and precision, a batch, ray sets, derivation, the display
pass and the forward passes.  The digests were taken from the library before its kernels were rearranged (guarded
RK4 steps only, every disk chord sampled, one launch a view, the whole ISCO scan, outputs through buffers), so they
hold what the comments call "the same bits".  They go with the compiler: after a change of nvcc, or of a result on
purpose, take them anew from a library whose results are known to be right (run this file, which prints them)."""
import ctypes as C
import hashlib
import json
import os
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path[:0] = [os.path.join(os.path.dirname(HERE), p) for p in ("black-hole_b200", "oracle", "tests")]

import pytest  # noqa: E402

from bhrt import lib, scenes  # noqa: E402
from bhrt.abi import (BH_PREC_FP32, BH_PREC_FP64, BH_PREC_MIXED, DERIVE_REQ_DTYPE, DERIVED_DTYPE,  # noqa: E402
                      BHView)

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(HERE, "golden", "bits.json")

# model, a*, q, distance, elevation, field of view, disk, step budget, naked
FRAMES = {
    "schwarzschild": (0, 0.0, 0.0, 12.0, 20.0, 60.0, True, 0, False),
    "rn": (1, 0.0, 0.5, 15.0, 15.0, 60.0, True, 0, False),
    "kerr": (2, 0.9, 0.0, 20.0, 10.0, 45.0, True, 0, False),
    "kerr_axis": (2, 0.9, 0.0, 12.0, 89.5, 50.0, True, 0, False),
    "kerr_no_disk": (2, -0.7, 0.0, 6.0, 60.0, 70.0, False, 0, False),
    "kn": (3, 0.8, 0.3, 25.0, 15.0, 45.0, True, 0, False),
    "kn_extremal_close": (3, 0.998, 0.05, 4.0, 30.0, 80.0, True, 0, False),
    "kn_budget": (3, -0.7, 0.4, 6.0, 60.0, 50.0, True, 41, False),
    "kerr_naked": (2, 1.05, 0.0, 10.0, 30.0, 50.0, True, 0, True),
}


def _sha(*arrays):
    h = hashlib.sha256()
    for a in arrays:
        h.update(np.ascontiguousarray(a).tobytes())
    return h.hexdigest()[:32]


def _frame(name, precision, w=240, h=137):
    import torch
    from bhrt.device import Frame
    model, a, q, dist, el, fov, disk, steps, naked = FRAMES[name]
    if precision == BH_PREC_FP64:
        w, h = 48, 27
    P = scenes.scene(lib.derive, model, a, q, w, h, dist, el, fov, disk=disk, allow_naked=naked)
    if steps:
        P.maxSteps = steps
    f = Frame(w, h)
    f.pipeline(P, precision)
    torch.cuda.synchronize()
    return _sha(f.out.cpu().numpy(), f.accum.cpu().numpy(), f.bloomA.cpu().numpy(), f.bloomB.cpu().numpy())


def _probe(precision):
    from bhrt.device import probe_grid
    P = scenes.scene(lib.derive, 3, 0.8, 0.3, 96, 54, 12.0, 80.0, 60.0)
    return _sha(probe_grid(P, 96, 54, precision))


def _batch():
    import torch
    views, bufs = (BHView * len(FRAMES))(), []
    for v, (name, (model, a, q, dist, el, fov, disk, steps, naked)) in zip(views, FRAMES.items()):
        w, h = 96 + 8 * len(bufs), 54 + 5 * len(bufs)
        P = scenes.scene(lib.derive, model, a, q, w, h, dist, el, fov, disk=disk, allow_naked=naked)
        if steps:
            P.maxSteps = steps
        b = [torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda"), torch.zeros((h, w, 4), device="cuda")]
        b += [torch.zeros(((h + 1) // 2, (w + 1) // 2, 4), device="cuda") for _ in range(2)]
        v.params, v.out, v.accum, v.bloomA, v.bloomB = P, *[t.data_ptr() for t in b]
        bufs.append(b)
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.load().bhRenderBatch(views, len(views), s) == 0
    torch.cuda.synchronize()
    return _sha(*[t.cpu().numpy() for b in bufs for t in b])


def _accumulated():
    import torch
    from bhrt.device import Frame
    P = scenes.scene(lib.derive, 1, 0.0, 0.5, 203, 119, 15.0, 15.0, 60.0)
    f = Frame(203, 119)
    for k in range(3):
        P.accumMode, P.sampleIndex = 1, k
        f.pipeline(P)
    torch.cuda.synchronize()
    return _sha(f.out.cpu().numpy(), f.accum.cpu().numpy())


def _derive():
    import torch
    rng = np.random.default_rng(5)
    r = np.zeros(3000, DERIVE_REQ_DTYPE)
    r["model"], r["M"] = rng.integers(0, 4, 3000), rng.uniform(0.3, 1.5, 3000)
    r["aStar"], r["q"], r["allowNaked"] = rng.uniform(-1.4, 1.4, 3000), rng.uniform(0, 0.9, 3000), rng.integers(0, 2, 3000)
    req = torch.from_numpy(r.view(np.uint8).copy()).cuda()
    out = torch.zeros(3000 * DERIVED_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.load().bhDeriveBatch(C.c_void_p(req.data_ptr()), C.c_void_p(out.data_ptr()), 3000, s) == 0
    torch.cuda.synchronize()
    return _sha(out.cpu().numpy(), req.cpu().numpy())


def _net(what):
    from test_gpu_surrogate import Net, _inputs
    net = Net(7)
    try:
        if what == "rays":
            n = 24 * 5000
            assert net.L.bhSurrogateGenerate(net.h, C.c_longlong(n), 24, C.c_uint(3)) == 0
            x, t = np.zeros((n, 8), np.float32), np.zeros((n, 8), np.float32)
            assert net.L.bhSurrogateDatasetCopy(net.h, x.ctypes.data_as(C.c_void_p), t.ctypes.data_as(C.c_void_p),
                                                C.c_longlong(0), C.c_longlong(n)) == 0
            return _sha(x, t)
        return _sha(net.forward(_inputs(5000, 8), what == "fused"))
    finally:
        net.close()


CASES = {"frame_%s_%s" % (n, p): (lambda n=n, k=k: _frame(n, k))
         for n in FRAMES for p, k in (("fp32", BH_PREC_FP32), ("mixed", BH_PREC_MIXED), ("fp64", BH_PREC_FP64))}
CASES.update({"probe_fp32": lambda: _probe(BH_PREC_FP32), "probe_mixed": lambda: _probe(BH_PREC_MIXED),
              "batch": _batch, "accumulated": _accumulated, "derive": _derive, "rays": lambda: _net("rays"),
              "forward_fused": lambda: _net("fused"), "forward_training_form": lambda: _net("training")})


@pytest.mark.parametrize("name", CASES)
def test_bits(cuda, name):
    with open(GOLDEN) as f:
        assert CASES[name]() == json.load(f)[name]


if __name__ == "__main__":
    import torch
    torch.cuda.init()
    print(json.dumps({n: c() for n, c in CASES.items()}, indent=1))
