"""The two post-processing launches overlap: the same bytes on the null stream, on a stream of its
own, back to back over one set of buffers, and replayed from a captured graph."""
import ctypes as C

import pytest

from bhrt import lib, scenes
from bhrt.abi import BH_KERR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bloom", [True, False])
@pytest.mark.parametrize("size", [(1, 1), (65, 17), (640, 359)])
def test_post_on_streams_and_in_a_graph(cuda, size, bloom):
    import torch
    from bhrt.device import Frame
    w, h = size
    P = scenes.scene(lib.derive, BH_KERR, 0.8, 0.0, w, h, 12.0, 20.0, 60.0, bloom=bloom)
    L = lib.load()
    images = [torch.rand((h, w, 4), generator=torch.Generator().manual_seed(k)).cuda() * 4 for k in (1, 2)]

    def post(f, s):
        assert L.bhPostProcess(C.c_void_p(f.out.data_ptr()), C.c_void_p(f.accum.data_ptr()),
                               C.c_void_p(f.bloomA.data_ptr()), C.c_void_p(f.bloomB.data_ptr()), C.byref(P),
                               C.c_void_p(s)) == 0

    want = []
    for im in images:
        f = Frame(w, h)
        f.accum.copy_(im.view_as(f.accum))
        torch.cuda.synchronize()
        post(f, 0)
        torch.cuda.synchronize()
        want.append((f.out.clone(), f.bloomA.clone(), f.bloomB.clone()))
    f = Frame(w, h)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        for k in (0, 1, 0, 1):      # no synchronisation between the images
            f.accum.copy_(images[k].view_as(f.accum))
            post(f, side.cuda_stream)
    torch.cuda.synchronize()
    got = (f.out.clone(), f.bloomA.clone(), f.bloomB.clone())
    assert all(torch.equal(a, b) for a, b in zip(got, want[1]) if bloom or a is got[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        f.accum.copy_(images[0].view_as(f.accum))
        post(f, torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(f.out, want[0][0])
