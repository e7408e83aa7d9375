"""Batches of one or both metric families on every kind of stream: the second family's launch
starts in the first one's tail, and what follows on the stream sees both families' frames."""
import ctypes as C

import pytest

from bhrt import lib, scenes
from bhrt.abi import BH_KERR, BH_KERR_NEWMAN, BH_REISSNER_NORDSTROM, BH_SCHWARZSCHILD, BHView

pytestmark = pytest.mark.gpu

MODELS = {"rotating": (BH_KERR, BH_KERR_NEWMAN), "spherical": (BH_SCHWARZSCHILD, BH_REISSNER_NORDSTROM),
          "both": (BH_KERR, BH_SCHWARZSCHILD, BH_KERR_NEWMAN, BH_REISSNER_NORDSTROM)}


@pytest.mark.parametrize("which", sorted(MODELS))
@pytest.mark.parametrize("stream", ["null", "legacy", "per thread", "own"])
def test_batch_on_every_stream(cuda, which, stream):
    import torch
    from bhrt.device import Frame
    own = torch.cuda.Stream()
    s = {"null": 0, "legacy": 1, "per thread": 2, "own": own.cuda_stream}[stream]
    L = lib.load()
    views = (BHView * len(MODELS[which]))()
    frames, ones = [], []
    for v, m in zip(views, MODELS[which]):
        P = scenes.scene(lib.derive, m, 0.8, 0.3, 640, 360, 12.0, 20.0, 60.0)
        frames.append(Frame(640, 360))
        ones.append(Frame(640, 360))
        v.params = P
        v.out, v.accum = frames[-1].out.data_ptr(), frames[-1].accum.data_ptr()
        v.bloomA, v.bloomB = frames[-1].bloomA.data_ptr(), frames[-1].bloomB.data_ptr()
        one = (BHView * 1)()
        one[0].params = P
        one[0].out, one[0].accum = ones[-1].out.data_ptr(), ones[-1].accum.data_ptr()
        one[0].bloomA, one[0].bloomB = ones[-1].bloomA.data_ptr(), ones[-1].bloomB.data_ptr()
        assert L.bhRenderBatch(one, 1, C.c_void_p(own.cuda_stream)) == 0
        torch.cuda.synchronize()
    for _ in range(3):
        assert L.bhRenderBatch(views, len(views), C.c_void_p(s)) == 0
    torch.cuda.synchronize()
    # the same kernels on the same tiles: the same bytes
    for a, b in zip(frames, ones):
        assert torch.equal(a.out, b.out) and torch.equal(a.accum, b.accum)
