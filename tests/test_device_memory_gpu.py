"""Device memory across layers, sequence lengths and streams: what one use leaves serves the next."""
import ctypes as C
import gc

import numpy as np
import pytest
import torch

from boat_b200 import capi, rng
from boat_b200.host import Attention, DeviceBuffer, EncoderBlock, Tensor, check

pytestmark = pytest.mark.gpu


def free_bytes(lib):
    check(lib.boat_cuda_sync(), "sync")
    return torch.cuda.mem_get_info()[0]


def test_new_blocks_live_on_what_the_last_one_left(gpu_lib):
    """Twenty encoder blocks, one after another, each created, stepped and dropped."""
    B, S, d, nh, dev = 4, 384, 512, 8, capi.DEVICE_CUDA
    x, t = (Tensor.from_numpy(rng.normal(31, i, (B, S, d)), dev, bf16=True) for i in range(2))
    used, free, ref = [], [], None
    for i in range(20):
        block = EncoderBlock(d, nh)
        for j, layer in enumerate((block.fc1, block.fc2)):
            w = Tensor(gpu_lib.boat_dense_layer_get_weight(layer.h), own=False)
            w.set(rng.normal(32, j, w.shape, 0.02))
        for n in Attention.PARAMS[:4]:
            block.attn.param(n).set(rng.normal(33, ord(n[-1]), (d, d), 0.02))
        out, dx = block.step(x, t)
        got = out.numpy()
        ref = got if ref is None else ref
        assert np.array_equal(got, ref)
        del block, out, dx, w
        gc.collect()
        used.append(gpu_lib.boat_cuda_bytes_in_use())
        free.append(free_bytes(gpu_lib))
    assert len(set(used)) == 1
    assert len(set(free[1:])) == 1


def test_steps_of_changing_lengths_settle(gpu_lib):
    d, nh, dev = 256, 4, capi.DEVICE_CUDA
    layer = Attention(d, nh, causal=True)
    layer.to_device(dev)
    lengths = [40 + 97 * ((7 * i) % 10) for i in range(10)]
    x = {S: Tensor.from_numpy(rng.normal(34, S, (8, S, d)), dev, bf16=True) for S in lengths}
    first, free = {}, []
    for _ in range(5):
        for S in lengths:
            out = layer.forward(x[S])
            layer.backward(x[S])
            got = out.numpy()
            assert np.array_equal(got, first.setdefault(S, got))
        free.append(free_bytes(gpu_lib))
    assert free[2] == free[3] == free[4]


def test_blocks_follow_the_library_stream(gpu_lib):
    """Blocks freed on one stream are not handed out on another."""
    n = 3 << 20
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    try:
        check(gpu_lib.boat_cuda_set_stream(a.cuda_stream))
        p = DeviceBuffer(n)
        was = p.p.value
        p.free()
        check(gpu_lib.boat_cuda_set_stream(b.cuda_stream))
        q = DeviceBuffer(n)
        assert q.p.value != was
        q.free()
        check(gpu_lib.boat_cuda_set_stream(a.cuda_stream))
        r = DeviceBuffer(n)
        assert r.p.value == was
        r.free()
        layer = Attention(64, 4)
        layer.to_device(capi.DEVICE_CUDA)
        x = Tensor.from_numpy(rng.normal(35, 0, (2, 50, 64)), capi.DEVICE_CUDA)
        on_a = layer.forward(x).numpy()
    finally:
        check(gpu_lib.boat_cuda_sync())
        check(gpu_lib.boat_cuda_set_stream(None))
    assert np.array_equal(layer.forward(x).numpy(), on_a)


def test_blocks_of_a_captured_stream_belong_to_the_graph(gpu_lib):
    """y += 2 * (x * x) through a block that is allocated and freed inside the capture, replayed between other work."""
    n = 100000
    x = rng.normal(36, 0, (n,))
    dx, dy, s = DeviceBuffer.from_numpy(x), DeviceBuffer.from_numpy(np.zeros(n, np.float32)), torch.cuda.Stream()
    outside = DeviceBuffer(4 * n)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    try:
        check(gpu_lib.boat_cuda_set_stream(s.cuda_stream))
        with torch.cuda.graph(graph, stream=s):
            t = DeviceBuffer(4 * n)
            check(gpu_lib.boat_cuda_mul(t.p, dx.p, dx.p, n))
            check(gpu_lib.boat_cuda_axpy(dy.p, t.p, C.c_float(2.0), n))
            t.free()
            assert gpu_lib.boat_cuda_free(outside.p) != 0          # was not allocated in the capture
    finally:
        check(gpu_lib.boat_cuda_set_stream(None))
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        other = DeviceBuffer.from_numpy(np.full(n, 7.0, np.float32))
        assert (other.numpy((n,)) == 7.0).all()
        other.free()
    want = np.zeros(n, np.float32)
    for _ in range(3):
        want = want + np.float32(2.0) * (x * x)
    assert np.array_equal(dy.numpy((n,)), want)
    outside.free()
    del graph
