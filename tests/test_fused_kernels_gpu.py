"""GPU tests of the fused kernels and of the branches of their dispatch, at the sizes where they change,
against numpy in float64."""
import ctypes as C
import math

import numpy as np
import pytest

from boat_b200 import capi, rng
from boat_b200.host import Attention, DeviceBuffer, Tensor, Variable, check
from gpu_driver import gpu_step
from test_kernels_gpu import Shifted, rel, run_core, run_gemm

pytestmark = pytest.mark.gpu


def _table(bufs):
    return (C.c_void_p * len(bufs))(*[b.p.value for b in bufs])


def _bf(seed, stream, shape, scale=1.0):
    return rng.bf16_round(rng.normal(seed, stream, shape) * np.float32(scale))


_erf = np.vectorize(math.erf, otypes=[np.float64])


def _gelu(x):
    return 0.5 * x * (1 + _erf(x / math.sqrt(2)))


def _gelu_grad(x):
    return 0.5 * (1 + _erf(x / math.sqrt(2))) + x * np.exp(-0.5 * x * x) / math.sqrt(2 * math.pi)


# one tile, ragged rows and columns, K tails, many tiles; the last two are not for the tensor cores
@pytest.mark.parametrize("shape", [(128, 64, 64), (333, 136, 200), (700, 768, 72), (2100, 520, 256), (40, 24, 16), (130, 70, 64)])
@pytest.mark.parametrize("epilogue", [1, 2, 3], ids=["gelu", "gelu_grad", "add"])
def test_gemm_epilogues(gpu_lib, shape, epilogue):
    M, N, K = shape
    tb = epilogue == 2
    a, b = _bf(1, 0, (M, K)), _bf(1, 1, (N, K) if tb else (K, N), 1 / math.sqrt(K))
    aux, bias = _bf(1, 2, (M, N)), None if tb else rng.normal(1, 3, (N,))
    da, db, daux = (DeviceBuffer.from_numpy(t, bf16=True) for t in (a, b, aux))
    dbias = DeviceBuffer.from_numpy(bias) if bias is not None else None
    dc = DeviceBuffer(M * N * 2)
    check(gpu_lib.boat_cuda_gemm_fused(capi.MMA_BF16, epilogue, 0, int(tb), M, N, K, da.p, K, db.p, K if tb else N, capi.CUDA_BF16,
                                       dc.p, N, dbias.p if dbias else None, daux.p), "gemm_fused")
    check(gpu_lib.boat_cuda_sync(), "sync")
    z = a.astype(np.float64) @ (b.T if tb else b).astype(np.float64) + (0 if bias is None else bias)
    got = dc.numpy((M, N), bf16=True).astype(np.float64)
    if epilogue == 3:
        assert rel(got, z + aux) <= 5e-3
        return
    # Element by element: one BF16 rounding (half of 2^-7), two where separate passes store the product in between (the
    # shapes that are not for the tensor cores), FP32 sums (1e-5 of the largest), 3e-7 of the erf formula.  The tanh
    # approximation of GELU, off by 2 % at -2.5, fails this.
    if epilogue == 1:
        kept = daux.numpy((M, N), bf16=True).astype(np.float64)
        assert rel(kept, z) <= 3e-3
        want, slack = _gelu(kept), 3e-7 * np.abs(kept)
    else:
        want, slack = z * _gelu_grad(aux.astype(np.float64)), 1e-5 * np.abs(z).max()
    roundings = 2 if epilogue == 2 and (M < 128 or N % 8) else 1
    assert (np.abs(got - want) <= roundings * 1.01 * 2.0 ** -8 * np.abs(want) + slack).all()


# The operand of the epilogue comes through one shared-memory box per warp, asked for again as soon as it has been read: many
# tiles per CTA, many times, the same bits each time.
@pytest.mark.parametrize("epilogue", [2, 3], ids=["gelu_grad", "add"])
def test_gemm_epilogue_operand_boxes_are_read_in_time(gpu_lib, epilogue):
    M, N, K, tb = 8192, 1024, 256, epilogue == 2
    da, db, daux = (DeviceBuffer.from_numpy(_bf(11, i, sh), bf16=True) for i, sh in enumerate([(M, K), (N, K) if tb else (K, N), (M, N)]))
    dc, first = DeviceBuffer(M * N * 2), None
    for _ in range(300):
        check(gpu_lib.boat_cuda_gemm_fused(capi.MMA_BF16, epilogue, 0, int(tb), M, N, K, da.p, K, db.p, K if tb else N, capi.CUDA_BF16,
                                           dc.p, N, None, daux.p), "gemm_fused")
        check(gpu_lib.boat_cuda_sync(), "sync")
        got = dc.numpy((M, N), bf16=True)
        first = got if first is None else first
        assert (got == first).all()


@pytest.mark.parametrize("shape", [(128, 64, 64), (333, 768, 96), (2000, 320, 200)])
@pytest.mark.parametrize("groups", [1, 2, 3])
def test_gemm_sum_of_products(gpu_lib, shape, groups):
    M, N, K = shape
    a, b = [_bf(2, g, (M, K)) for g in range(groups)], [_bf(3, g, (N, K)) for g in range(groups)]
    da, db = [DeviceBuffer.from_numpy(t, bf16=True) for t in a], [DeviceBuffer.from_numpy(t, bf16=True) for t in b]
    dc = DeviceBuffer(M * N * 4)
    check(gpu_lib.boat_cuda_gemm_sum(capi.MMA_BF16, 0, 1, groups, M, N, K, _table(da), K, _table(db), K, capi.CUDA_BF16, dc.p, N,
                                     capi.CUDA_F32), "gemm_sum")
    check(gpu_lib.boat_cuda_sync(), "sync")
    assert rel(dc.numpy((M, N)), sum(x.astype(np.float64) @ y.astype(np.float64).T for x, y in zip(a, b))) <= 1e-5
    assert gpu_lib.boat_cuda_gemm_sum(capi.MMA_FP32, 0, 1, groups, M, N, K, _table(da), K, _table(db), K, capi.CUDA_F32, dc.p, N,
                                      capi.CUDA_F32) == 13


# FP32 results of few tiles and a long K are cut along K and added into a cleared output: the one output there is, and
# of it the rows of the result alone.  The inputs are BF16 values, exact in either arithmetic.
@pytest.mark.parametrize("mma", [capi.MMA_BF16, capi.MMA_TF32], ids=["bf16", "tf32"])
@pytest.mark.parametrize("M,N,K,pad", [(128, 2048, 2048, 0), (333, 192, 2048, 64), (200, 256, 3072, 0)])
def test_gemm_sum_of_products_with_split_k(gpu_lib, mma, M, N, K, pad):
    bf, groups, ldc = mma == capi.MMA_BF16, 3, N + pad
    a, b = [_bf(2, g, (M, K)) for g in range(groups)], [_bf(3, g, (N, K), 1 / math.sqrt(K)) for g in range(groups)]
    da, db = [DeviceBuffer.from_numpy(t, bf16=bf) for t in a], [DeviceBuffer.from_numpy(t, bf16=bf) for t in b]
    dc = DeviceBuffer.from_numpy(np.full((M, ldc), np.nan, np.float32))
    check(gpu_lib.boat_cuda_gemm_sum(mma, 0, 1, groups, M, N, K, _table(da), K, _table(db), K, capi.CUDA_BF16 if bf else capi.CUDA_F32,
                                     dc.p, ldc, capi.CUDA_F32), "gemm_sum")
    check(gpu_lib.boat_cuda_sync(), "sync")
    got = dc.numpy((M, ldc))
    assert rel(got[:, :N], sum(x.astype(np.float64) @ y.astype(np.float64).T for x, y in zip(a, b))) <= 1e-5
    assert np.isnan(got[:, N:]).all()


# one CTA's tiles of every width, a pair's, and the split of FP32 results with its remainders
@pytest.mark.parametrize("shape", [(128, 64, 64), (129, 200, 64), (1300, 768, 200), (2300, 1100, 136), (4096, 2304, 64)])
@pytest.mark.parametrize("layout", [(0, 0), (0, 1)], ids=["nn", "nt"])
def test_gemm_tile_shapes(gpu_lib, shape, layout):
    got, ref = run_gemm(gpu_lib, capi.MMA_BF16, *layout, *shape, out_bf16=True)
    assert rel(got, ref) <= 3e-3


@pytest.mark.parametrize("shape", [(256, 192, 3000), (512, 512, 1500), (768, 520, 5000)])
def test_gemm_split_of_fp32_results(gpu_lib, shape):
    got, ref = run_gemm(gpu_lib, capi.MMA_BF16, 1, 0, *shape, bias=False)
    assert rel(got, ref) <= 1e-5


@pytest.mark.parametrize("bf", [False, True], ids=["fp32", "bf16"])
@pytest.mark.parametrize("shape", [(64, 64, 200), (136, 72, 333), (256, 512, 3000)])
def test_weight_grads_accumulate(gpu_lib, bf, shape):
    I, O, T = shape
    make = _bf if bf else (lambda s, i, sh: rng.normal(s, i, sh))
    x, dy = make(4, 0, (T, I)), make(4, 1, (T, O))
    w0, b0 = rng.normal(4, 2, (I, O)), rng.normal(4, 3, (O,))
    dx, ddy = DeviceBuffer.from_numpy(x, bf16=bf), DeviceBuffer.from_numpy(dy, bf16=bf)
    dw, db = DeviceBuffer.from_numpy(w0), DeviceBuffer.from_numpy(b0)
    check(gpu_lib.boat_cuda_weight_grads(capi.MMA_BF16 if bf else capi.MMA_FP32, 1, I, O, T, _table([dx]), _table([ddy]),
                                         capi.CUDA_BF16 if bf else capi.CUDA_F32, _table([dw]), _table([db]), 1), "weight_grads")
    check(gpu_lib.boat_cuda_sync(), "sync")
    assert rel(dw.numpy((I, O)), w0 + x.astype(np.float64).T @ dy.astype(np.float64)) <= 1e-5
    assert np.abs(db.numpy((O,)) - (b0 + dy.astype(np.float64).sum(0))).max() <= 1e-6 * np.abs(dy).sum(0).max()


# one tile, remainders in each direction, K in pieces, every tile shape, CTA pairs, more tiles than SMs
@pytest.mark.parametrize("mma", [capi.MMA_BF16, capi.MMA_TF32], ids=["bf16", "tf32"])
@pytest.mark.parametrize("I,O,T,groups", [(128, 64, 64, 1), (136, 72, 333, 3), (520, 200, 1000, 2), (256, 512, 3000, 3), (2048, 1032, 700, 1),
                                          (1024, 1024, 2500, 3)])
def test_weight_grads_with_column_sums(gpu_lib, mma, I, O, T, groups):
    bf = mma == capi.MMA_BF16
    make = _bf if bf else (lambda s, i, sh: rng.normal(s, i, sh))
    x, dy = [make(5, g, (T, I)) for g in range(groups)], [make(6, g, (T, O)) for g in range(groups)]
    dx, ddy = ([DeviceBuffer.from_numpy(t, bf16=bf) for t in ts] for ts in (x, dy))
    dw = [DeviceBuffer.from_numpy(np.full((I, O), np.nan, np.float32)) for _ in range(groups)]
    db = [DeviceBuffer.from_numpy(np.full((O,), np.nan, np.float32)) for _ in range(groups)]
    check(gpu_lib.boat_cuda_weight_grads(mma, groups, I, O, T, _table(dx), _table(ddy), capi.CUDA_BF16 if bf else capi.CUDA_F32,
                                         _table(dw), _table(db), 0), "weight_grads")
    check(gpu_lib.boat_cuda_sync(), "sync")
    for g in range(groups):
        y = dy[g].astype(np.float64)
        assert rel(dw[g].numpy((I, O)), x[g].astype(np.float64).T @ y) <= (1e-5 if bf else 5e-3)
        # FP32 sums of T terms in some order: random roundings of partial sums no larger than the sum of the magnitudes
        # grow like sqrt(T) half units; four times that
        assert (np.abs(db[g].numpy((O,)) - y.sum(0)) <= 4 * math.sqrt(T) * 2.0 ** -25 * np.abs(y).sum(0)).all()


# column sums over K in pieces: few and many of them, groups, CTA pairs, ragged columns, added to what is there
@pytest.mark.parametrize("mma", [capi.MMA_BF16, capi.MMA_TF32], ids=["bf16", "tf32"])
@pytest.mark.parametrize("I,O,T,groups,add", [(1024, 1024, 8000, 3, 0), (128, 64, 20000, 1, 0), (256, 520, 9001, 1, 1), (1024, 1024, 8000, 1, 1),
                                              (1024, 4096, 4096, 1, 1)])
def test_column_sums_have_the_same_bits_every_time(gpu_lib, mma, I, O, T, groups, add):
    bf = mma == capi.MMA_BF16
    make = _bf if bf else (lambda s, i, sh: rng.normal(s, i, sh))
    x, dy = [make(9, g, (T, I)) for g in range(groups)], [make(10, g, (T, O)) for g in range(groups)]
    dx, ddy = ([DeviceBuffer.from_numpy(t, bf16=bf) for t in ts] for ts in (x, dy))
    dw, first = DeviceBuffer(groups * I * O * 4), rng.normal(11, 0, (O,))
    outs = [DeviceBuffer.from_numpy(first) for _ in range(24 * groups)]
    for i in range(0, 24 * groups, groups):
        check(gpu_lib.boat_cuda_weight_grads(mma, groups, I, O, T, _table(dx), _table(ddy), capi.CUDA_BF16 if bf else capi.CUDA_F32,
                                             (C.c_void_p * groups)(*[dw.p.value + g * I * O * 4 for g in range(groups)]), _table(outs[i:i + groups]),
                                             add), "weight_grads")
    check(gpu_lib.boat_cuda_sync(), "sync")
    for g in range(groups):
        got = [b.numpy((O,)) for b in outs[g::groups]]
        y = dy[g].astype(np.float64)
        want, size = y.sum(0) + (first if add else 0), np.abs(y).sum(0) + np.abs(first)
        assert (np.abs(got[0] - want) <= 4 * math.sqrt(T) * 2.0 ** -25 * size).all()         # as above
        assert all(np.array_equal(got[0], b) for b in got)


@pytest.mark.parametrize("n", [1, 4, 1023, 4096, 100003])
def test_elementwise_over_several_arrays(gpu_lib, n):
    a = [rng.normal(5, i, (n,)) for i in range(4)]
    y = DeviceBuffer.from_numpy(a[0])
    x = [DeviceBuffer.from_numpy(t) for t in a[1:]]
    check(gpu_lib.boat_cuda_add_n(y.p, _table(x), 3, n), "add_n")
    want = ((a[0] + a[1]) + a[2]) + a[3]
    assert np.array_equal(y.numpy((n,)), want)
    sizes = (C.c_int64 * 2)(n, (n + 1) // 2)
    w, g = [DeviceBuffer.from_numpy(t) for t in a[:2]], [DeviceBuffer.from_numpy(t) for t in a[2:]]
    check(gpu_lib.boat_cuda_axpy_multi(_table(w), _table(g), C.c_float(-0.5), sizes, 2), "axpy_multi")
    assert np.array_equal(w[0].numpy((n,)), a[0] - np.float32(0.5) * a[2])
    check(gpu_lib.boat_cuda_sgd_clear(_table(w), _table(g), C.c_float(0.25), sizes, 2), "sgd_clear")
    h = sizes[1]
    assert np.array_equal(w[1].numpy((n,))[:h], (a[1] - np.float32(0.5) * a[3])[:h] - np.float32(0.25) * a[3][:h])
    assert np.array_equal(w[1].numpy((n,))[h:], a[1][h:])
    assert not g[0].numpy((n,)).any() and not g[1].numpy((n,))[:h].any() and np.array_equal(g[1].numpy((n,))[h:], a[3][h:])


@pytest.mark.parametrize("nbytes", [4, 16, 4096 + 16, 1000004, 256 * 1024, 256 * 1024 + 16])
def test_stage_copy(gpu_lib, nbytes):
    src = rng.normal(6, 0, (nbytes // 4,))
    up, down = (gpu_lib.boat_cuda_host_alloc(nbytes) for _ in range(2))
    dev = DeviceBuffer(nbytes)
    C.memmove(up, src.ctypes.data, nbytes)
    check(gpu_lib.boat_cuda_stage_copy(dev.p, up, nbytes, 0), "up")
    check(gpu_lib.boat_cuda_stage_copy(down, dev.p, nbytes, 1), "down")
    check(gpu_lib.boat_cuda_sync(), "sync")
    assert C.string_at(down, nbytes) == src.tobytes()
    for p in (up, down):
        gpu_lib.boat_cuda_host_free(p)


# rows of less than a warp's width, the widths with registers of their own, and one beyond them
@pytest.mark.parametrize("bf", [False, True], ids=["fp32", "bf16"])
@pytest.mark.parametrize("rows,cols", [(1, 8), (37, 100), (333, 768), (1000, 1024), (50, 4096), (9, 5000)])
def test_layernorm_rows_and_residual_gradient(gpu_lib, bf, rows, cols):
    make = _bf if bf else (lambda s, i, sh: rng.normal(s, i, sh))
    x, dy, add = make(7, 0, (rows, cols)), make(7, 1, (rows, cols)), make(7, 2, (rows, cols))
    gamma, beta = 1 + rng.normal(7, 3, (cols,)) * np.float32(0.1), rng.normal(7, 4, (cols,))
    ty = capi.CUDA_BF16 if bf else capi.CUDA_F32
    es = 2 if bf else 4
    dx_, ddy, dadd = (DeviceBuffer.from_numpy(t, bf16=bf) for t in (x, dy, add))
    dg, dbt = DeviceBuffer.from_numpy(gamma), DeviceBuffer.from_numpy(beta)
    y, dx = DeviceBuffer(rows * cols * es), DeviceBuffer(rows * cols * es)
    mean, rstd, dgam, dbet = (DeviceBuffer(4 * n) for n in (rows, rows, cols, cols))
    check(gpu_lib.boat_cuda_layernorm_fwd(dx_.p, ty, rows, cols, dg.p, dbt.p, C.c_float(1e-5), y.p, mean.p, rstd.p), "fwd")
    X, G = x.astype(np.float64), dy.astype(np.float64)
    mu = X.mean(1, keepdims=True)
    rs = 1 / np.sqrt(X.var(1, keepdims=True) + 1e-5)
    hat = (X - mu) * rs
    tol = 8e-3 if bf else 2e-6
    assert rel(y.numpy((rows, cols), bf16=bf), hat * gamma + beta) <= tol
    p = G * gamma
    ref = (p - p.mean(1, keepdims=True) - hat * (p * hat).mean(1, keepdims=True)) * rs
    for res, want in ((None, ref), (dadd.p, ref + add)):
        check(gpu_lib.boat_cuda_layernorm_bwd_add(ddy.p, dx_.p, ty, rows, cols, dg.p, mean.p, rstd.p, res, dx.p, dgam.p, dbet.p), "bwd")
        check(gpu_lib.boat_cuda_sync(), "sync")
        assert rel(dx.numpy((rows, cols), bf16=bf), want) <= tol
        assert np.abs(dgam.numpy((cols,)) - (G * hat).sum(0)).max() <= 1e-5 * np.abs(G * hat).sum(0).max()
        assert np.abs(dbet.numpy((cols,)) - G.sum(0)).max() <= 1e-5 * np.abs(G).sum(0).max()


@pytest.mark.parametrize("bf", [False, True], ids=["fp32", "bf16"])
@pytest.mark.parametrize("cols", [768, 5000])
@pytest.mark.parametrize("which", ["x", "y", "dy", "dx", "gamma", "all"])
def test_layernorm_of_arrays_off_alignment(gpu_lib, bf, cols, which):
    rows, ty, tol = 37, capi.CUDA_BF16 if bf else capi.CUDA_F32, 8e-3 if bf else 2e-6
    make = _bf if bf else (lambda s, i, sh: rng.normal(s, i, sh))
    x, g, gamma = make(7, 0, (rows, cols)), make(7, 1, (rows, cols)), 1 + rng.normal(7, 3, (cols,)) * np.float32(0.1)
    d = {n: Shifted(gpu_lib, (rows, cols), bf, int(which in (n, "all")), v) for n, v in dict(x=x, dy=g, y=None, dx=None).items()}
    dg = Shifted(gpu_lib, (cols,), False, int(which in ("gamma", "all")), gamma)
    mean, rstd, dgam, dbet = (DeviceBuffer(4 * n) for n in (rows, rows, cols, cols))
    check(gpu_lib.boat_cuda_layernorm_fwd(d["x"].p, ty, rows, cols, dg.p, None, C.c_float(1e-5), d["y"].p, mean.p, rstd.p), "fwd")
    check(gpu_lib.boat_cuda_layernorm_bwd(d["dy"].p, d["x"].p, ty, rows, cols, dg.p, mean.p, rstd.p, d["dx"].p, dgam.p, dbet.p), "bwd")
    check(gpu_lib.boat_cuda_sync(), "sync")
    X, G = x.astype(np.float64), g.astype(np.float64)
    rs = 1 / np.sqrt(X.var(1, keepdims=True) + 1e-5)
    hat, p = (X - X.mean(1, keepdims=True)) * rs, G * gamma
    assert rel(d["y"].numpy(), hat * gamma) <= tol
    assert rel(d["dx"].numpy(), (p - p.mean(1, keepdims=True) - hat * (p * hat).mean(1, keepdims=True)) * rs) <= tol
    assert np.abs(dgam.numpy((cols,)) - (G * hat).sum(0)).max() <= 1e-5 * np.abs(G * hat).sum(0).max()


# more work than SMs: every CTA of the persistent kernels takes several items, unevenly long ones when causal
@pytest.mark.parametrize("hs,units,S", [(64, 170, 300), (128, 100, 520)])
@pytest.mark.parametrize("causal", [False, True], ids=["full", "causal"])
def test_attention_core_with_several_items_per_cta(gpu_lib, hs, units, S, causal):
    got, ref = run_core(gpu_lib, capi.MMA_BF16, units, S, hs, causal)
    for key in ("o", "dq", "dk", "dv"):
        assert rel(got[key], ref[key]) <= 2e-2, key


# one tile, K split over a cluster with CTAs left over in the last one, ragged and unaligned sizes, the largest taken
@pytest.mark.parametrize("T,I,O,groups", [(8, 32, 32, 1), (128, 64, 64, 3), (200, 40, 72, 2), (33, 13, 9, 3), (300, 64, 32, 4), (640, 96, 64, 1)])
def test_linear_grads_in_one_launch(gpu_lib, T, I, O, groups):
    x, dy, w = ([rng.normal(9, 10 * k + g, s) for g in range(groups)] for k, s in enumerate([(T, I), (T, O), (I, O)]))
    dx, ddy, dw_ = ([DeviceBuffer.from_numpy(t) for t in ts] for ts in (x, dy, w))
    got, want = ([[DeviceBuffer.from_numpy(np.full(s, np.nan, np.float32)) for _ in range(groups)] for s in ((T, I), (I, O), (O,))] for _ in range(2))
    check(gpu_lib.boat_cuda_linear_grads(capi.MMA_FP32, groups, T, I, O, _table(dx), _table(ddy), _table(dw_), *map(_table, got)), "linear_grads")
    check(gpu_lib.boat_cuda_weight_grads(capi.MMA_FP32, groups, I, O, T, _table(dx), _table(ddy), capi.CUDA_F32, _table(want[1]), _table(want[2]), 0), "dw")
    check(gpu_lib.boat_cuda_gemm_grouped(capi.MMA_FP32, 0, 1, groups, T, I, O, _table(ddy), O, _table(dw_), O, capi.CUDA_F32, _table(want[0]), I,
                                         capi.CUDA_F32, None), "dx")
    check(gpu_lib.boat_cuda_sync(), "sync")
    for a, b, shape in zip(got, want, ((T, I), (I, O), (O,))):
        for g in range(groups):
            assert a[g].numpy(shape).tobytes() == b[g].numpy(shape).tobytes()
    assert rel(got[0][0].numpy((T, I)), dy[0].astype(np.float64) @ w[0].astype(np.float64).T) <= 1e-6
    # larger problems, and other arithmetic, are two launches
    assert gpu_lib.boat_cuda_linear_grads(capi.MMA_FP32, 1, 100000, I, O, _table(dx), _table(ddy), _table(dw_), *map(_table, got)) == 13
    assert gpu_lib.boat_cuda_linear_grads(capi.MMA_TF32, 1, T, I, O, _table(dx), _table(ddy), _table(dw_), *map(_table, got)) == 13


# Within a sequence of launches, kernels that name their memory run beside one another when they touch nothing of each other's: one over
# few buffers, where most neighbours do depend on each other - read after write, write after read, write after write, over
# windows that overlap in part - gives the bits of the same sequence with a wait after every call.
@pytest.mark.parametrize("mma", [capi.MMA_FP32, capi.MMA_BF16], ids=["fp32", "bf16"])
@pytest.mark.parametrize("n", [64, 256])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_kernels_beside_one_another(gpu_lib, mma, n, seed):
    bf = mma == capi.MMA_BF16
    ty, es, count = (capi.CUDA_BF16, 2, 5) if bf else (capi.CUDA_F32, 4, 5)
    first = rng.normal(8, seed, (count * n, n)) / np.float32(math.sqrt(n))

    def play(wait):
        pick = np.random.default_rng(seed)
        block = DeviceBuffer.from_numpy(_bf(8, seed, (count * n, n), 1 / math.sqrt(n)) if bf else first, bf16=bf)
        wide, grads = DeviceBuffer.from_numpy(first), DeviceBuffer(n * n * 4)
        at = lambda rows: C.c_void_p(block.p.value + rows * n * es)
        gpu_lib.boat_cuda_launches_begin()
        for _ in range(80):
            # n rows each, from any eighth of the block: neighbours overlap in part
            x, y, z = (int(r) * n // 8 for r in pick.choice(8 * (count - 1) + 1, 3, replace=False))
            if abs(z - x) < n or abs(z - y) < n:            # a result over its own operand is no valid call
                z = (max(x, y) + n) if max(x, y) + 2 * n <= count * n else min(x, y) - n
                if z < 0 or abs(z - x) < n or abs(z - y) < n:
                    continue
            what = int(pick.integers(6))
            if what < 3:
                check(gpu_lib.boat_cuda_gemm(mma, int(what == 2), int(what == 1), n, n, n, at(x), n, at(y), n, ty, at(z), n, ty, None), "gemm")
            elif what < 4 and not bf:                       # fresh values, so that products of products stay in range
                check(gpu_lib.boat_cuda_lincomb(at(z), C.c_void_p(wide.p.value + x * n * 4), C.c_float(0.75), C.c_void_p(wide.p.value + y * n * 4),
                                                C.c_float(-0.5), ty, n * n), "lincomb")
            elif bf:
                check(gpu_lib.boat_cuda_cast(at(z), ty, C.c_void_p(wide.p.value + x * n * 4), capi.CUDA_F32, n * n), "cast")
            else:
                check(gpu_lib.boat_cuda_weight_grads(mma, 1, n, n, n, (C.c_void_p * 1)(at(x).value), (C.c_void_p * 1)(at(y).value), ty,
                                                     _table([grads]), None, 0), "dw")
            if wait:
                check(gpu_lib.boat_cuda_sync(), "sync")
        gpu_lib.boat_cuda_launches_end()
        check(gpu_lib.boat_cuda_sync(), "sync")
        return block.numpy((count * n, n), bf16=bf), grads.numpy((n, n))

    (a, ga), (b, gb) = play(False), play(True)
    assert np.isfinite(b).mean() > 0.5
    assert a.tobytes() == b.tobytes() and (bf or ga.tobytes() == gb.tobytes())


# the staged TF32 backward: one key tile, two, the first that waits for a buffer used before, a remainder of one row
@pytest.mark.parametrize("units,S", [(3, 40), (150, 256), (40, 385), (20, 1025)])
@pytest.mark.parametrize("causal", [False, True], ids=["full", "causal"])
def test_tf32_attention_core_over_its_buffers(gpu_lib, units, S, causal):
    got, ref = run_core(gpu_lib, capi.MMA_TF32, units, S, 64, causal)
    for key in ("o", "dq", "dk", "dv"):
        assert rel(got[key], ref[key]) <= 5e-3, key


# results written to page-locked memory, packed and separate copies, chunks of more than one batch entry
@pytest.mark.parametrize("B,S,H,nh", [(2, 4, 32, 4), (3, 40, 128, 4), (5, 61, 256, 8), (6, 700, 256, 8)])
def test_host_tensors_give_the_results_of_cuda_tensors(gpu_lib, B, S, H, nh):
    n = lambda i, *s: rng.normal(8, i, s)  # noqa: E731
    x = n(0, B, S, H)
    inp = {"q": x, "k": x, "v": x, "w": [n(1 + i, H, H) / np.float32(math.sqrt(H)) for i in range(4)],
           "b": [n(5 + i, H) for i in range(4)], "dout": n(9, B, S, H)}
    host, cuda = (gpu_step(inp, nh, True, device=d, lr=0.1) for d in (capi.DEVICE_CPU, capi.DEVICE_CUDA))
    for k in ("out", "dq", "dk", "dv"):
        assert rel(host[k], cuda[k]) <= 1e-6, k
    for k in ("dw", "db", "w_after"):
        for i in range(4):
            assert rel(host[k][i], cuda[k][i]) <= 1e-6 or np.abs(host[k][i]).max() <= 1e-5, (k, i)


def test_self_attention_gradient_is_the_sum_of_three(gpu_lib):
    B, S, H, nh = 2, 50, 64, 4
    layer = Attention(H, nh, causal=True)
    layer.to_device(capi.DEVICE_CUDA)
    x, g = rng.normal(9, 0, (B, S, H)), rng.normal(9, 1, (B, S, H))
    grads = []
    for distinct in (False, True):
        t = [Variable(Tensor.from_numpy(x, capi.DEVICE_CUDA)) for _ in range(3 if distinct else 1)]
        q, k, v = t if distinct else t * 3
        r = q.attention(layer, k, v) + q
        r.backward(Tensor.from_numpy(g, capi.DEVICE_CUDA))
        grads.append(sum(u.grad.numpy().astype(np.float64) for u in t))
    assert rel(grads[0], grads[1]) <= 1e-6
