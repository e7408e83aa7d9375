"""Device derivation over the whole range of masses: the host's values bit for bit (rPhoton of the Kerr family
within its ulps) also where M^2 overflows, where energies leave the normal range and where the scan starts inside
the horizon."""
import ctypes as C

import numpy as np
import pytest

from bhrt import lib
from bhrt.abi import DERIVE_REQ_DTYPE, DERIVED_DTYPE

pytestmark = pytest.mark.gpu


def _derive(req):
    import torch
    dreq = torch.from_numpy(req.view(np.uint8).copy()).cuda()
    dout = torch.zeros(len(req) * DERIVED_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.load().bhDeriveBatch(C.c_void_p(dreq.data_ptr()), C.c_void_p(dout.data_ptr()), len(req), s) == 0
    torch.cuda.synchronize()
    return dout.cpu().numpy().view(DERIVED_DTYPE)


@pytest.mark.parametrize("low, high", [(-37.0, -16.0), (-16.0, -10.0), (-10.0, -5.0), (5.0, 18.0), (18.0, 19.3),
                                       (19.3, 37.0)])
def test_extreme_masses_equal_host(cuda, low, high):
    rng = np.random.default_rng(int(low * 10) + 1000)
    n = 400
    r = np.zeros(n, DERIVE_REQ_DTYPE)
    r["model"] = rng.integers(0, 4, n)
    r["M"] = 10.0 ** rng.uniform(low, high, n)
    r["aStar"], r["q"] = rng.uniform(-0.998, 0.998, n), rng.uniform(0.0, 0.6, n)
    r["allowNaked"][::5] = 1
    r["aStar"][::5] *= 1.4
    got = _derive(r)
    for i, (x, g) in enumerate(zip(r, got)):
        want = lib.derive(int(x["model"]), float(x["M"]), float(x["aStar"]), float(x["q"]), bool(x["allowNaked"]))[0]
        for f in ("a", "Q", "rPlus", "rMinus", "rErgo", "rIsco", "clamped", "naked"):
            assert np.array_equal(np.float32(g[f]), np.float32(getattr(want, f)), equal_nan=True), (i, f, x, g)


def test_a_scan_past_the_largest_float_ends(cuda):
    """12 M overflows: the radii end with the largest finite one."""
    r = np.zeros(4, DERIVE_REQ_DTYPE)
    r["model"], r["M"], r["aStar"] = range(4), 3e38, 0.5
    assert (_derive(r)["clamped"] == 0).all()
