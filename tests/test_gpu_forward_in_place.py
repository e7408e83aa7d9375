"""bhSurrogateForward in the training form with outputs that overlap the inputs: the inputs' values count, wherever
the outputs lie."""
import pytest

from test_gpu_surrogate import Net, _inputs, _ptr, _stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [127, 70000])
@pytest.mark.parametrize("out_at, in_at", [(0, 0), (0, 8), (0, 15), (4, 0)])       # in floats of n
def test_outputs_over_inputs(cuda, n, out_at, in_at):
    import torch
    net = Net(41)
    try:
        inp = _inputs(n, 42)
        want = torch.as_tensor(net.forward(inp, False))
        buf = torch.zeros(24 * n, dtype=torch.float32, device="cuda")
        x, y = buf[in_at * n:(in_at + 8) * n], buf[out_at * n:(out_at + 16) * n]
        for _ in range(3):
            x.copy_(torch.as_tensor(inp).reshape(-1))
            assert net.L.bhSurrogateForward(net.h, _ptr(x), _ptr(y), n, 0, _stream()) == 0
            torch.cuda.synchronize()
            assert torch.equal(y.cpu().view(n, 16), want)
    finally:
        net.close()
