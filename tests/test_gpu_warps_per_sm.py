"""Frame sizes on both sides of the limits at which the launch leaves SMs with fewer warps:
the same bytes as with the number of blocks an SM given."""
import pytest

from bhrt import lib, scenes
from bhrt.abi import BH_KERR_NEWMAN, BH_REISSNER_NORDSTROM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,model,a", [(0, BH_REISSNER_NORDSTROM, 0.0), (1, BH_KERR_NEWMAN, 0.7)])
@pytest.mark.parametrize("size", [(128, 128), (136, 128), (512, 256), (520, 256), (1024, 256), (1032, 256), (1024, 512), (1031, 515), (2048, 512), (2056, 512)])
def test_frame_does_not_depend_on_blocks_per_sm(cuda, family, model, a, size):
    import torch
    from bhrt.device import Frame
    w, h = size
    L = lib.load()
    P = scenes.scene(lib.derive, model, a, 0.3, w, h, 12.0, 20.0, 60.0)
    outs = []
    try:
        for blocks in (0, 1, 64):
            L.bhSetTuning(family, 32, blocks)
            f = Frame(w, h)
            f.pipeline(P)
            torch.cuda.synchronize()
            outs.append(f.out.clone())
    finally:
        L.bhSetTuning(family, 32, 0)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
