"""Work of the program's own on the library's stream, between calls of the library: it sees what the call before has written, and
the call behind sees what it has written."""
import threading

import numpy as np
import pytest
import torch

from boat_b200 import capi, rng
from boat_b200.host import Attention, DeviceBuffer, Tensor, check

pytestmark = pytest.mark.gpu
B, S, D, NH = 4, 128, 256, 4


class _Memory:
    """A library tensor's memory for torch."""

    def __init__(self, t):
        self.__cuda_array_interface__ = {"shape": t.shape, "typestr": "<f4", "data": (t.data_ptr, False), "version": 2}


def _torch(t):
    return torch.as_tensor(_Memory(t), device="cuda")


def _train(mma, wait, steps=8):
    """Steps of a layer whose weights, input and upstream gradient torch kernels write between the library's calls; no call of either
    is followed by a wait unless `wait`."""
    layer = Attention(D, NH, causal=True)
    layer.to_device(capi.DEVICE_CUDA)
    layer.set_precision(mma)
    for i, name in enumerate(Attention.PARAMS):
        p = layer.param(name)
        p.set(rng.normal(41, i, p.shape, 0.06))
    x, g = (Tensor.from_numpy(rng.normal(42, i, (B, S, D)), capi.DEVICE_CUDA) for i in range(2))
    settle = torch.cuda.synchronize if wait else lambda: None
    settle()
    kept = []
    for _ in range(steps):
        out = layer.forward(x)
        settle()
        _torch(g).mul_(0.9).add_(_torch(out), alpha=0.1)
        settle()
        grads = layer.backward(g)
        settle()
        for name in Attention.PARAMS:
            _torch(layer.param(name)).sub_(_torch(layer.param("grad_" + name)), alpha=1e-3)
        _torch(x).add_(_torch(grads[0]), alpha=1e-2)
        settle()
        kept.append((out, grads))
    result = [x.numpy(), g.numpy(), kept[-1][0].numpy()] + [layer.param(n).numpy() for n in Attention.PARAMS]
    layer.free()
    return result


def _on(lib, stream, f):
    if stream is None:
        return f()
    try:
        check(lib.boat_cuda_set_stream(stream.cuda_stream))
        with torch.cuda.stream(stream):
            return f()
    finally:
        torch.cuda.synchronize()
        check(lib.boat_cuda_set_stream(None))


@pytest.mark.parametrize("mma", [capi.MMA_FP32, capi.MMA_TF32], ids=["fp32", "tf32"])
@pytest.mark.parametrize("own", [False, True], ids=["default stream", "a stream of its own"])
def test_kernels_of_the_program_between_two_calls(gpu_lib, mma, own):
    torch.cuda.synchronize()
    stream = torch.cuda.Stream() if own else None
    got, want = (_on(gpu_lib, stream, lambda: _train(mma, wait)) for wait in (False, True))
    for a, b in zip(got, want):
        assert np.isfinite(a).all() and a.tobytes() == b.tobytes()


PER_THREAD = 2          # cudaStreamPerThread


@pytest.mark.parametrize("per_thread", [False, True], ids=["one stream", "a stream per thread"])
def test_two_threads(gpu_lib, per_thread):
    want = _train(capi.MMA_FP32, True)
    got = {}

    def work(i):
        with torch.cuda.stream(torch.cuda.ExternalStream(PER_THREAD) if per_thread else torch.cuda.default_stream()):
            got[i] = _train(capi.MMA_FP32, False)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    try:
        check(gpu_lib.boat_cuda_set_stream(PER_THREAD if per_thread else None))
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        torch.cuda.synchronize()
        check(gpu_lib.boat_cuda_set_stream(None))
    for i in range(2):
        for a, b in zip(got[i], want):
            assert a.tobytes() == b.tobytes()


def test_a_capture_within_a_sequence(gpu_lib):
    """Products into a graph between eager ones, some of either independent of one another; the graph runs at the end."""
    n, stream, graph = 192, torch.cuda.Stream(), torch.cuda.CUDAGraph()
    host = [rng.normal(43, i, (n, n)) / np.float32(14) for i in range(3)]

    def play():
        x, w, v = (DeviceBuffer.from_numpy(a) for a in host)
        out = [DeviceBuffer(n * n * 4) for _ in range(6)]
        gemm = lambda c, a, b: check(gpu_lib.boat_cuda_gemm(capi.MMA_FP32, 0, 0, n, n, n, a.p, n, b.p, n, capi.CUDA_F32, c.p, n,  # noqa: E731
                                                            capi.CUDA_F32, None))
        gpu_lib.boat_cuda_launches_begin()
        gemm(out[0], x, w)
        with torch.cuda.graph(graph, stream=stream):
            gemm(out[1], v, out[2])
            gemm(out[3], v, w)
        gemm(out[2], out[0], w)
        gemm(out[4], x, x)
        gemm(out[5], out[2], out[4])
        gpu_lib.boat_cuda_launches_end()
        graph.replay()
        return [b.numpy((n, n)) for b in out]

    got = _on(gpu_lib, stream, play)
    x, w, v = (a.astype(np.float64) for a in host)
    want = [x @ w, v @ (x @ w @ w), x @ w @ w, v @ w, x @ x, (x @ w @ w) @ (x @ x)]
    for a, b in zip(got, want):
        # sums of n products in FP32, three deep: 3 * sqrt(n) * 2^-24 of the norms in the mean, with a margin of ten
        assert np.linalg.norm(a - b) <= 30 * np.sqrt(n) * 2.0**-24 * np.linalg.norm(b)
    del graph
