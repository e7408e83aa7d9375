"""Mixed-precision frames.  The tile kernel keeps a warp's lanes waiting at the polar cap and takes their FP64
passages together; the refill-queue kernel (refillMin < 32) takes each ray's by itself.  Both against each other and
against the all-FP64 frame: the spin axis in view, a near-extremal hole, budgets that end inside a passage or just
after one, and frames of 1, 2, 8 and 32 rays a warp."""
import numpy as np
import pytest

import parity
from bhrt import lib, scenes
from bhrt.abi import BH_KERR, BH_KERR_NEWMAN, BH_PREC_FP64, BH_PREC_MIXED

pytestmark = pytest.mark.gpu

SCENES = {"axis": (BH_KERR, 0.9, 0.0, 89.5, 0), "near_axis": (BH_KERR_NEWMAN, 0.8, 0.3, 80.0, 0),
          "near_extremal": (BH_KERR_NEWMAN, 0.998, 0.05, 45.0, 0), "budget_24": (BH_KERR, 0.9, 0.0, 89.5, 24),
          "budget_37": (BH_KERR, 0.9, 0.0, 88.0, 37), "budget_90": (BH_KERR_NEWMAN, 0.8, 0.3, 85.0, 90)}
SIZES = [(64, 64), (128, 96), (320, 180), (640, 360)]       # 1, 2, 8 and 32 rays a warp


def _frame(P, w, h, precision):
    import torch
    from bhrt.device import Frame
    f = Frame(w, h)
    f.pipeline(P, precision)
    torch.cuda.synchronize()
    return f.out.cpu().numpy(), f.accum.cpu().numpy()


@pytest.mark.parametrize("size", SIZES, ids=["%dx%d" % s for s in SIZES])
@pytest.mark.parametrize("name", SCENES)
def test_mixed_frame(cuda, name, size):
    model, a, q, el, steps = SCENES[name]
    w, h = size
    P = scenes.scene(lib.derive, model, a, q, w, h, 25.0, el, 50.0, bloom=False)
    if steps:
        P.maxSteps = steps
    rgba, acc = _frame(P, w, h, BH_PREC_MIXED)
    again = _frame(P, w, h, BH_PREC_MIXED)
    assert np.array_equal(acc.view(np.uint32), again[1].view(np.uint32)) and np.array_equal(rgba, again[0])
    before = lib.get_tuning(1)
    try:
        lib.set_tuning(1, 16, before[1])
        single, _ = _frame(P, w, h, BH_PREC_MIXED)
    finally:
        lib.set_tuning(1, *before)
    # the bars of the FP32 comparison of these two kernels
    s = parity.compare_rgba(rgba, single)
    assert s["alpha_ok"] and s["lsb1_frac"] >= 0.9995 and s["exact_frac"] >= 0.99, s
    # FP32 steps against FP64 ones: 99 % of escape directions within 1e-4 rad where the outcome is the same, a few
    # per cent of the pixels on an outcome's edge or behind a star's
    s = parity.compare_rgba(rgba, _frame(P, w, h, BH_PREC_FP64)[0])
    assert s["lsb1_frac"] >= 0.95, s
