"""Frames small enough that a warp takes fewer than 32 rays at a time (every width
the launch rule picks, and sizes on both sides of its limits), against the same
views in a batch, which always takes whole tiles: the batch suite's bars."""
import ctypes as C

import pytest

import parity
from bhrt import lib, scenes
from bhrt.abi import BH_KERR_NEWMAN, BH_REISSNER_NORDSTROM, BHView

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,a", [(BH_REISSNER_NORDSTROM, 0.0), (BH_KERR_NEWMAN, 0.7)])
@pytest.mark.parametrize("size", [(1, 1), (33, 7), (128, 64), (136, 64), (256, 128), (213, 121), (512, 256), (520, 257)])
def test_small_frame_equals_batch(cuda, model, a, size):
    import torch
    from bhrt.device import Frame
    w, h = size
    P = scenes.scene(lib.derive, model, a, 0.3, w, h, 12.0, 20.0, 60.0)
    frame, other = Frame(w, h), Frame(w, h)
    frame.pipeline(P)
    v = (BHView * 1)()
    v[0].params = P
    v[0].out, v[0].accum = other.out.data_ptr(), other.accum.data_ptr()
    v[0].bloomA, v[0].bloomB = other.bloomA.data_ptr(), other.bloomB.data_ptr()
    assert lib.load().bhRenderBatch(v, 1, C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    s = parity.compare_rgba(frame.out.cpu().numpy(), other.out.cpu().numpy())
    assert s["lsb1_frac"] == 1.0 and s["exact_frac"] >= 0.999, s
