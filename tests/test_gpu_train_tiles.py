"""The training kernels at the edges of their tiles: one 128-ray tile, batches that do not
divide into the weight gradients' shares, and forward passes with a ragged last tile."""
import ctypes as C

import numpy as np
import pytest

import sg_oracle as SG
from test_gpu_surrogate import Net, _features, _inputs, _ptr, _targets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 129, 1000])
def test_forward_tiles_match_the_fused_kernel(cuda, n):
    net = Net(11)
    try:
        inp = _inputs(n, 12)
        net.forward(_inputs(2048, 13), False)      # leaves other values in the rows past n
        got, want = net.forward(inp, False), net.forward(inp, True)
        # the same BF16 operands, FP32 sums in another order
        assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max() + 1e-6
    finally:
        net.close()


@pytest.mark.parametrize("n", [128, 384, 896, 1920, 4224])
def test_gradients_of_uneven_batches_match_oracle(cuda, n):
    import torch
    net = Net(17)
    try:
        p = net.params()
        rng = np.random.default_rng(3)
        p[SG.HIDDEN * SG.HID:] += rng.normal(scale=0.05, size=p.size - SG.HIDDEN * SG.HID).astype(np.float32)
        for l in range(SG.HIDDEN):
            p[l * SG.HID + 65536:(l + 1) * SG.HID] = rng.normal(scale=0.1, size=256)
        net.set_params(p)
        inp = _inputs(n, 18)
        tgt = _targets(inp, 19)
        x, t = (torch.as_tensor(v, device="cuda") for v in (inp, tgt))
        g = np.zeros(net.count, dtype=np.float32)
        loss = np.zeros(5, dtype=np.float32)
        assert net.L.bhSurrogateGradients(net.h, _ptr(x), _ptr(t), n, g.ctypes.data_as(C.c_void_p),
                                          loss.ctypes.data_as(C.c_void_p)) == 0
        want, wloss = SG.gradients(_features(inp), p, inp.astype(np.float64), tgt.astype(np.float64))
        # BF16 operands and activations in four layers each way: the bounds of the 256-ray test
        assert np.allclose(loss, wloss, rtol=2e-2, atol=1e-4)
        for l in range(SG.HIDDEN + 1):
            w0, w1 = l * SG.HID, l * SG.HID + (65536 if l < SG.HIDDEN else 16 * 256)
            b1 = w1 + (256 if l < SG.HIDDEN else 16)
            for a, b in ((w0, w1), (w1, b1)):
                assert np.linalg.norm(g[a:b] - want[a:b]) < 5e-2 * np.linalg.norm(want[a:b]), (l, a)
    finally:
        net.close()
