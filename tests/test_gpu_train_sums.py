"""The sums of a training step: in a fixed order, over accumulators of at most 512 rays, and carried
from step to step (hashed rows, gradients, Adam, repacked weights)."""
import ctypes as C
import math

import numpy as np
import pytest

from test_gpu_surrogate import Net, _inputs, _ptr, _targets

pytestmark = pytest.mark.gpu

BATCHES = [128, 1280, 16384, 19072]      # one tile, uneven shares, full shares, more tiles than SMs


def _gradients(net, x, t, n):
    g = np.zeros(net.count, dtype=np.float32)
    loss = np.zeros(5, dtype=np.float32)
    assert net.L.bhSurrogateGradients(net.h, _ptr(x), _ptr(t), n, g.ctypes.data_as(C.c_void_p),
                                      loss.ctypes.data_as(C.c_void_p)) == 0
    return g, loss


def _train(net, steps, batch, lr, seed):
    loss = np.zeros((steps, 5), dtype=np.float32)
    assert net.L.bhSurrogateTrain(net.h, steps, batch, C.c_float(lr), C.c_uint(seed),
                                  loss.ctypes.data_as(C.c_void_p)) == 0
    return loss


def _generate(net, rays=16384, views=8, seed=5):
    assert net.L.bhSurrogateGenerate(net.h, C.c_longlong(rays), views, C.c_uint(seed)) == 0


@pytest.mark.parametrize("batch", BATCHES)
def test_training_repeats_bit_for_bit(cuda, batch):
    runs = []
    for _ in range(2):
        net = Net(21)
        try:
            _generate(net)
            loss = [_train(net, 4, batch, 2e-3, 9), _train(net, 3, batch, 1e-3, 10)]
            runs.append(np.concatenate([net.params()] + [v.ravel() for v in loss]))
        finally:
            net.close()
    assert np.isfinite(runs[0]).all()
    assert np.array_equal(runs[0].view(np.uint32), runs[1].view(np.uint32))


def _in_order(blocks):
    """Shares of 512 rays (float32 each): some consecutive ones a part, added in float32; 14 parts at most, added in
    float64 and rounded once."""
    parts = min(len(blocks), 14)
    total = np.zeros_like(blocks[0], dtype=np.float64)
    for y in range(parts):
        part = None
        for k in range(len(blocks) * y // parts, len(blocks) * (y + 1) // parts):
            part = blocks[k] if part is None else part + blocks[k]
        total += part.astype(np.float64)
    return total.astype(np.float32)


@pytest.mark.parametrize("blocks", [2, 32])
def test_a_batch_is_the_sum_of_its_512_ray_blocks(cuda, blocks):
    """512 and `blocks` are powers of two, so the blocks' loss gradients are the batch's, scaled exactly; the
    batch's gradient is then the sum, in its fixed order, of the blocks' gradients, each of one accumulator."""
    import torch
    net = Net(23)
    try:
        n = 512 * blocks
        inp = _inputs(n, 24)
        tgt = _targets(inp, 25)
        x, t = (torch.as_tensor(v, device="cuda") for v in (inp, tgt))
        g, loss = _gradients(net, x, t, n)
        parts = [_gradients(net, x[k:k + 512].contiguous(), t[k:k + 512].contiguous(), 512) for k in range(0, n, 512)]
        assert np.array_equal(g, _in_order([p[0] / np.float32(blocks) for p in parts]))
        assert np.array_equal(loss, _in_order([p[1] * np.float32(512) for p in parts]) / np.float32(n))
    finally:
        net.close()


def _rows(batch, N, seed):
    """Rows of the ray set that the batch's rays take: the hash of the training kernel."""
    with np.errstate(over="ignore"):
        u = np.uint32
        h = (np.arange(batch, dtype=u) * u(0x9E3779B1)) ^ u(seed)
        h ^= h >> u(16); h *= u(0x7FEB352D); h ^= h >> u(15); h *= u(0x846CA68B); h ^= h >> u(16)
        h2 = h * u(0x2C1B3C6D) + u(0x297A2D39)
        h2 ^= h2 >> u(15)
    return ((h.astype(np.uint64) << np.uint64(32)) | h2.astype(np.uint64)) % np.uint64(N)


@pytest.mark.parametrize("batch", BATCHES)
def test_training_is_its_steps_taken_one_by_one(cuda, batch):
    """bhSurrogateTrain against a replay: the rows gathered on the host, bhSurrogateGradients, Adam in numpy, the
    weights set in a second handle.  The first step's loss is the same bits; Adam in numpy rounds differently by some
    ulps, which turn a few BF16 roundings of the weights in the steps after."""
    import torch
    steps, lr, seed, N = 4, 2e-3, 11, 16384
    net, ref = Net(31), Net(31)
    try:
        _generate(net, N)
        x, t = np.zeros((N, 8), np.float32), np.zeros((N, 8), np.float32)
        assert net.L.bhSurrogateDatasetCopy(net.h, x.ctypes.data_as(C.c_void_p), t.ctypes.data_as(C.c_void_p),
                                            C.c_longlong(0), C.c_longlong(N)) == 0
        p = net.params()
        start = p.copy()
        loss = _train(net, steps, batch, lr, seed)
        m, v = np.zeros(p.size), np.zeros(p.size)
        for k in range(steps):
            at = _rows(batch, N, (seed * 0x9E3779B1 + k * 0x632BE5AB) & 0xFFFFFFFF).astype(np.int64)
            ref.set_params(p)
            g, want = _gradients(ref, torch.as_tensor(x[at], device="cuda"), torch.as_tensor(t[at], device="cuda"), batch)
            if k == 0:
                assert np.array_equal(loss[0], want)
            # a relative 1e-3: some hundred of 266,000 weights off by a BF16 ulp (2^-9) move a loss term by less
            assert np.allclose(loss[k], want, rtol=1e-3, atol=1e-6), k
            m, v = 0.9 * m + 0.1 * g.astype(np.float64), 0.999 * v + 0.001 * g.astype(np.float64) ** 2
            lrT = lr * (0.05 + 0.95 * 0.5 * (1 + math.cos(math.pi * k / (steps - 1))))
            p = (p - lrT * (m / (1 - 0.9 ** (k + 1))) / (np.sqrt(v / (1 - 0.999 ** (k + 1))) + 1e-8)).astype(np.float32)
        # a step left out, taken twice or on other rows moves most parameters by its whole length
        got = net.params()
        moved = np.linalg.norm(p - start)
        assert np.linalg.norm(got - p) < 1e-2 * moved
    finally:
        net.close()
        ref.close()
