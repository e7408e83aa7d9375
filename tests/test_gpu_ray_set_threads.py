"""Ray sets generated while another thread queues frames of the same handle, and two handles trained at once: the
results are those of the calls by themselves."""
import ctypes as C
import threading

import numpy as np
import pytest

from bhrt import lib, scenes
from bhrt.abi import BH_KERR_NEWMAN
from test_gpu_surrogate import Net, _ptr

pytestmark = pytest.mark.gpu


def _together(*calls):
    errors = []

    def guarded(call):
        try:
            call()
        except BaseException as e:      # noqa: BLE001 -- handed to the test's thread
            errors.append(e)
    threads = [threading.Thread(target=guarded, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_generate_beside_frames_of_the_same_handle(cuda):
    import torch
    from bhrt.device import Frame
    net = Net(51)
    w, h, rays, views = 640, 360, 64 * 2048, 64
    try:
        P = scenes.scene(lib.derive, BH_KERR_NEWMAN, 0.8, 0.3, w, h, 25.0, 15.0, 45.0)
        # cell gate on: the frame forks to the handle's stream and joins it
        assert net.L.bhSurrogateSetAnchors(net.h, 8, 1, C.c_float(1e-4), C.c_float(0.5)) == 0
        f, stream = Frame(w, h), torch.cuda.Stream()

        def frame():
            assert net.L.bhSurrogateRender(net.h, _ptr(f.out), _ptr(f.accum), _ptr(f.bloomA), _ptr(f.bloomB),
                                           C.byref(P), C.c_void_p(stream.cuda_stream)) == 0

        def ray_set():
            x, t = np.zeros((rays, 8), np.float32), np.zeros((rays, 8), np.float32)
            assert net.L.bhSurrogateGenerate(net.h, C.c_longlong(rays), views, C.c_uint(7)) == 0
            assert net.L.bhSurrogateDatasetCopy(net.h, x.ctypes.data_as(C.c_void_p), t.ctypes.data_as(C.c_void_p),
                                                C.c_longlong(0), C.c_longlong(rays)) == 0
            return x, t

        frame()
        torch.cuda.synchronize()
        image = f.out.clone()
        want = ray_set()
        sets = []

        def frames():
            for _ in range(60):
                frame()
                stream.synchronize()

        _together(frames, lambda: sets.extend(ray_set() for _ in range(6)))
        torch.cuda.synchronize()
        assert torch.equal(f.out, image)
        for x, t in sets:
            assert np.array_equal(x, want[0]) and np.array_equal(t, want[1])
    finally:
        net.close()


def test_two_handles_trained_at_once(cuda):
    def train(net):
        loss = np.zeros((6, 5), np.float32)
        assert net.L.bhSurrogateTrain(net.h, 6, 4096, C.c_float(2e-3), C.c_uint(3), loss.ctypes.data_as(C.c_void_p)) == 0
        return np.concatenate([net.params(), loss.ravel()])

    def handle():
        net = Net(61)
        assert net.L.bhSurrogateGenerate(net.h, C.c_longlong(8192), 8, C.c_uint(5)) == 0
        return net
    nets = [handle() for _ in range(3)]
    try:
        want, got = train(nets[0]), {}
        _together(lambda: got.update(a=train(nets[1])), lambda: got.update(b=train(nets[2])))
        assert np.array_equal(got["a"], want) and np.array_equal(got["b"], want)
    finally:
        for net in nets:
            net.close()
