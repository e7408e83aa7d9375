"""The device's ISCO scan (exact radius sequences, coarse pass and window) against
the host's full running-sum scan: the same radius, bit for bit, over masses whose
scans start and end in different binades, near-extremal holes and naked ones."""
import ctypes as C

import numpy as np
import pytest

from bhrt import lib
from bhrt.abi import DERIVE_REQ_DTYPE, DERIVED_DTYPE

pytestmark = pytest.mark.gpu


def _requests(kind, n=700):
    rng = np.random.default_rng({"box": 1, "extremal": 2, "masses": 3, "naked": 4}[kind])
    r = np.zeros(n, DERIVE_REQ_DTYPE)
    r["model"] = rng.integers(0, 4, n)
    r["M"] = 0.5
    r["aStar"], r["q"] = rng.uniform(-0.998, 0.998, n), rng.uniform(0.0, 0.6, n)
    if kind == "extremal":
        r["aStar"] = rng.choice([-1.0, 1.0], n) * (0.995 - 10.0 ** rng.uniform(-7, -1, n))
        r["q"] = 10.0 ** rng.uniform(-4, -0.2, n)
    if kind == "masses":     # 2^k, just below and above it, and anything between
        r["M"] = np.concatenate([2.0 ** rng.integers(-12, 12, n // 2) * rng.choice([1.0, 1 - 2e-7, 1 + 2e-7], n // 2),
                                 10.0 ** rng.uniform(-5, 5, n - n // 2)])
    if kind == "naked":
        r["allowNaked"] = 1
        r["aStar"], r["q"] = rng.uniform(-1.5, 1.5, n), rng.uniform(0.0, 1.5, n)
    return r


@pytest.mark.parametrize("kind", ["box", "extremal", "masses", "naked"])
def test_isco_scan_equals_running_sum(cuda, kind):
    import torch
    req = _requests(kind)
    n = len(req)
    want = np.array([lib.derive(int(r["model"]), float(r["M"]), float(r["aStar"]), float(r["q"]),
                                bool(r["allowNaked"]))[0].rIsco for r in req], np.float32)
    dreq = torch.from_numpy(req.view(np.uint8).copy()).cuda()
    dout = torch.zeros(n * DERIVED_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.load().bhDeriveBatch(C.c_void_p(dreq.data_ptr()), C.c_void_p(dout.data_ptr()), n, s) == 0
    torch.cuda.synchronize()
    got = dout.cpu().numpy().view(DERIVED_DTYPE)["rIsco"]
    bad = np.nonzero(got.view(np.uint32) != want.view(np.uint32))[0]
    assert bad.size == 0, [(req[i], got[i], want[i]) for i in bad[:5]]
