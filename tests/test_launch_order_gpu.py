"""Work of the program's own on the library's stream, between calls of the library: it sees what the call before has written, and
the call behind sees what it has written."""
import ctypes as C
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


class _Draws:
    """A random sequence over every kernel that names its memory, within one sequence of launches, with launches that name none, copies and
    memsets between: windows of few arenas, which overlap in part, so that most neighbours depend on each other - read after write, write
    after read, write after write.  Products of long contractions, whose pieces are added in an order that varies, have operands of
    small integers: their sums are exact in every order."""

    T = 4096                                         # a contraction that is cut in pieces: clear, products, sums of the pieces

    def __init__(self, lib, mma, n, seed, wait):
        self.lib, self.mma, self.n, self.wait = lib, mma, n, wait
        self.pick = np.random.default_rng(seed)
        self.bf = mma == capi.MMA_BF16
        self.ty, self.es = (capi.CUDA_BF16, 2) if self.bf else (capi.CUDA_F32, 4)
        normal = lambda i, *s: rng.normal(50 + seed, i, s)  # noqa: E731
        make = lambda a: DeviceBuffer.from_numpy(rng.bf16_round(a) if self.bf else a, bf16=self.bf)  # noqa: E731
        self.fresh = normal(0, 4 * n, n) / np.float32(np.sqrt(n))
        self.small = np.rint(np.clip(normal(1, 4 * self.T, n), -2, 2)).astype(np.float32)
        self.wide, self.whole = DeviceBuffer.from_numpy(self.fresh), DeviceBuffer.from_numpy(self.small)
        self.a, self.w = make(normal(2, 5 * n, n)), make(self.fresh)                 # results of products; their second operands
        self.tall = make(self.small[:3 * self.T])                                    # operands of the long products
        self.dw, self.db = (DeviceBuffer.from_numpy(np.zeros(3 * n * c, np.float32)) for c in (n, 1))
        self.param = DeviceBuffer.from_numpy(np.zeros(2 * n * n, np.float32))
        self.f32 = DeviceBuffer.from_numpy(normal(3, 4 * n, n))
        self.vec = DeviceBuffer.from_numpy(np.concatenate([normal(4, 4 * n) / np.float32(np.sqrt(n)), np.zeros(8 * n, np.float32)]))
        self.ran = set()

    def at(self, buf, row, es=None):
        return C.c_void_p(buf.p.value + int(row) * self.n * (es or self.es))

    def rows(self, of, count, written=1):
        """Starts of `count` windows of n rows in `of` * n rows, in steps of an eighth; the first `written` meet no other."""
        n, steps = self.n, 8 * (of - 1) + 1
        while True:
            r = [int(x) * n // 8 for x in self.pick.integers(steps, size=count)]
            if all(abs(r[i] - r[j]) >= n for i in range(written) for j in range(count) if i != j):
                return r

    def step(self):
        lib, n, ty, mma, at, pick, T = self.lib, self.n, self.ty, self.mma, self.at, self.pick, self.T
        table = lambda *p: (C.c_void_p * len(p))(*[x.value for x in p])  # noqa: E731
        sizes = lambda *s: (C.c_int64 * len(s))(*s)  # noqa: E731
        f = C.c_float
        what = str(pick.choice(["gemm", "fused", "grouped", "sum", "long", "short", "grads", "convert", "cast", "round", "lincomb", "axpy", "scale", "sgd", "norm",
                                "colsum", "tall", "memset", "copy", "mul"]))
        if what == "gemm":
            z, x = self.rows(5, 2)
            rc = lib.boat_cuda_gemm(mma, 0, int(pick.integers(2)), n, n, n, at(self.a, x), n, at(self.w, self.rows(4, 1)[0]), n, ty, at(self.a, z), n, ty, self.vec.p)
        elif what == "fused":
            z, aux, x = self.rows(5, 3, 2)
            e = int(pick.integers(1, 4))
            rc = lib.boat_cuda_gemm_fused(mma, e, 0, int(e == 2), n, n, n, at(self.a, x), n, at(self.w, self.rows(4, 1)[0]), n, ty, at(self.a, z), n, None, at(self.a, aux))
        elif what in ("grouped", "sum"):
            z, y, x, u = self.rows(5, 4, 2)
            first, second = table(at(self.a, x), at(self.a, u)), table(*(at(self.w, r) for r in self.rows(4, 2, 0)))
            if what == "grouped":
                rc = lib.boat_cuda_gemm_grouped(mma, 0, 0, 2, n, n, n, first, n, second, n, ty, table(at(self.a, z), at(self.a, y)), n, ty, None)
            else:
                rc = lib.boat_cuda_gemm_sum(mma, 0, 1, 2, n, n, n, first, n, second, n, ty, at(self.a, z), n, ty)
        elif what in ("long", "short"):
            k, add = (T if what == "long" else n), int(pick.integers(2))
            groups = 1 if add else int(pick.integers(1, 3))
            x = [at(self.tall, int(pick.integers(2 * 8 + 1)) * T // 8) for _ in range(2 * groups)]
            r = self.rows(3, groups, groups)
            db = table(*(C.c_void_p(self.db.p.value + 4 * v) for v in r)) if pick.integers(2) else None
            rc = lib.boat_cuda_weight_grads(mma, groups, n, n, k, table(*x[:groups]), table(*x[groups:]), ty, table(*(at(self.dw, v, 4) for v in r)), db, add)
        elif what == "grads":                        # dX over one of the windows, dW into FP32 memory
            if mma != capi.MMA_FP32:
                return
            (z, x), (dw, w) = self.rows(5, 2), self.rows(4, 2)
            rc = lib.boat_cuda_linear_grads(mma, 1, n, n, n, table(at(self.a, x)), table(at(self.a, x)), table(at(self.w, w)), table(at(self.a, z)),
                                            table(at(self.f32, dw, 4)), None)
        elif what == "convert":
            to = capi.CUDA_BF16 if self.bf else capi.CUDA_F32_TF32
            rc = lib.boat_cuda_convert_multi(table(*(at(self.w, v) for v in self.rows(4, 2, 2))), to, table(*(at(self.wide, v, 4) for v in self.rows(4, 2, 0))),
                                             sizes(n * n, n * n), 2)
        elif what == "cast":
            r, q = self.rows(5, 1)[0], self.rows(4, 1)[0]
            back = self.bf and pick.integers(2)
            rc = (lib.boat_cuda_cast(at(self.f32, q, 4), capi.CUDA_F32, at(self.a, r), ty, n * n) if back else
                  lib.boat_cuda_cast(at(self.a, r), ty, at(self.wide, q, 4), capi.CUDA_F32, n * n))
        elif what == "round":
            z, x = self.rows(4, 2)
            rc = lib.boat_cuda_round_tf32(at(self.f32, z, 4), at(self.f32, x, 4), n * n)
        elif what == "lincomb":
            z, x, y = self.rows(5, 3)
            rc = lib.boat_cuda_lincomb(at(self.a, z), at(self.a, x), f(0.6), at(self.a, y), f(-0.4), ty, n * n)
        elif what in ("axpy", "scale"):
            z, x = int(pick.integers(n + 1)), self.rows(3, 1)[0]
            rc = getattr(lib, "boat_cuda_" + what)(at(self.param, z, 4), at(self.dw, x, 4), f(0.5), n * n)
        elif what == "sgd":
            rc = lib.boat_cuda_sgd_clear(table(at(self.param, 0, 4), at(self.param, n, 4)), table(*(at(self.dw, v, 4) for v in self.rows(3, 2, 2))), f(0.25),
                                         sizes(n * n, n * n - 4), 2)
        elif what == "norm":
            z, x = self.rows(5, 2)
            v = lambda i: C.c_void_p(self.vec.p.value + 4 * n * int(i))  # noqa: E731
            rc = lib.boat_cuda_layernorm_fwd(at(self.a, x), ty, n, n, v(pick.integers(4)), v(pick.choice([0, 1, 8, 10])), f(1e-5), at(self.a, z), v(6), v(7))
        elif what == "colsum":                       # into biases of LayerNorm
            x = self.rows(5, 2, 0)
            rc = lib.boat_cuda_colsum_multi(table(at(self.a, x[0]), at(self.a, x[1])), ty, n, n, table(*(C.c_void_p(self.vec.p.value + 4 * n * i) for i in (8, 10))), 2)
        elif what == "tall":                         # other integers under the long products
            z, x = (int(pick.integers(2 * 8 + 1)) * T // 8 for _ in range(2))
            rc = lib.boat_cuda_cast(at(self.tall, z), ty, at(self.whole, x, 4), capi.CUDA_F32, T * n) if self.bf else \
                lib.boat_cuda_scale(at(self.tall, z), at(self.whole, x, 4), f(1.0), T * n)
        elif what == "memset":
            rc = lib.boat_cuda_memset(at(self.dw, self.rows(3, 1)[0], 4), 0, n * n * 4)
        elif what == "copy":
            z, x = self.rows(5, 2)
            rc = lib.boat_cuda_memcpy_d2d(at(self.a, z), at(self.a, x), n * n * self.es)
        else:                                        # a kernel that names nothing
            z, x = self.rows(4, 2)
            rc = lib.boat_cuda_mul(at(self.f32, z, 4), at(self.f32, x, 4), at(self.wide, x, 4), n * n)
        if rc != 13 or what not in ("sum", "grads"):
            check(rc, what)
            self.ran.add(what)
        if self.wait:
            check(lib.boat_cuda_sync(), "sync")

    def play(self, steps):
        check(self.lib.boat_cuda_sync(), "sync")
        self.lib.boat_cuda_launches_begin()
        try:
            for _ in range(steps):
                self.step()
        finally:
            self.lib.boat_cuda_launches_end()
        check(self.lib.boat_cuda_sync(), "sync")
        n = self.n
        return dict(a=self.a.numpy((5 * n, n), bf16=self.bf), w=self.w.numpy((4 * n, n), bf16=self.bf), dw=self.dw.numpy((3 * n, n)), db=self.db.numpy((3 * n,)),
                    param=self.param.numpy((2 * n, n)), f32=self.f32.numpy((4 * n, n)), vec=self.vec.numpy((12 * n,)))


@pytest.mark.parametrize("mma", [capi.MMA_FP32, capi.MMA_TF32, capi.MMA_BF16], ids=["fp32", "tf32", "bf16"])
@pytest.mark.parametrize("n", [64, 128, 256])
@pytest.mark.parametrize("seed", [0, 1])
def test_every_kernel_that_names_its_memory(gpu_lib, mma, n, seed):
    """Run beside one another they give the bits of the same calls with a wait after each."""
    got, want = (_Draws(gpu_lib, mma, n, seed, wait) for wait in (False, True))
    a, b = got.play(240), want.play(240)
    # the sum of products is the tensor cores', which take 128 rows and more; both gradients in one launch are for small FP32 problems
    assert len(want.ran) == 18 + (mma != capi.MMA_FP32 and n >= 128) + (mma == capi.MMA_FP32 and n == 64)
    for k in a:
        assert np.isfinite(b[k]).all() and a[k].tobytes() == b[k].tobytes(), k


@pytest.mark.parametrize("mma", [capi.MMA_TF32, capi.MMA_BF16], ids=["tf32", "bf16"])
@pytest.mark.parametrize("add", [0, 1])
def test_captured_weight_gradients_in_pieces(gpu_lib, mma, add):
    """The sums of the pieces wait in memory of the launch, within a graph in memory of the graph: exact sums at every replay."""
    n, T, bf, stream, graph = 128, 6000, mma == capi.MMA_BF16, torch.cuda.Stream(), torch.cuda.CUDAGraph()
    make = lambda i: np.rint(np.clip(rng.normal(60, i, (T, n)), -2, 2)).astype(np.float32)  # noqa: E731
    x, dy = make(0), make(1)
    dx, ddy = (DeviceBuffer.from_numpy(t, bf16=bf) for t in (x, dy))
    dw, db = DeviceBuffer.from_numpy(np.ones((n, n), np.float32)), DeviceBuffer.from_numpy(np.ones(n, np.float32))
    one = lambda b: (C.c_void_p * 1)(b.p.value)  # noqa: E731

    def play():
        with torch.cuda.graph(graph, stream=stream):
            check(gpu_lib.boat_cuda_weight_grads(mma, 1, n, n, T, one(dx), one(ddy), capi.CUDA_BF16 if bf else capi.CUDA_F32, one(dw), one(db), add))
        for _ in range(3):
            graph.replay()

    torch.cuda.synchronize()
    _on(gpu_lib, stream, play)
    times, first = (3, 1) if add else (1, 0)
    assert np.array_equal(dw.numpy((n, n)), first + times * (x.T @ dy)) and np.array_equal(db.numpy((n,)), first + times * dy.sum(0))
    del graph
