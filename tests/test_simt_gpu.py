"""GPU tests of the CUDA-core kernels at the sizes where their tiles, splits and vector paths change,
against numpy in float64."""
import ctypes as C

import numpy as np
import pytest

from boat_b200 import capi, rng
from boat_b200.host import DeviceBuffer, check
from test_kernels_gpu import LAYOUTS, rel, run_core, run_gemm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", LAYOUTS + [(1, 1)], ids=["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("shape", [(33, 31, 4), (64, 64, 1000), (65, 68, 129), (100, 257, 600), (2000, 1100, 70)])
def test_exact_gemm_tiles_and_splits(gpu_lib, layout, shape):
    M, N, K = shape
    got, ref = run_gemm(gpu_lib, capi.MMA_FP32, layout[0], layout[1], M, N, K)
    assert rel(got, ref) <= 1e-5


@pytest.mark.parametrize("mma", [capi.MMA_FP32, capi.MMA_BF16], ids=["fp32", "bf16"])
@pytest.mark.parametrize("shape", [(32, 32, 8), (48, 40, 131), (128, 64, 3000)])
@pytest.mark.parametrize("groups", [1, 3])
def test_weight_grads(gpu_lib, mma, shape, groups):
    I, O, T = shape
    bf = mma == capi.MMA_BF16
    f = rng.bf16_round if bf else (lambda a: a)
    x = [f(rng.normal(31, i, (T, I))) for i in range(groups)]
    dy = [f(rng.normal(32, i, (T, O))) for i in range(groups)]
    dx, ddy = ([DeviceBuffer.from_numpy(a, bf16=bf) for a in t] for t in (x, dy))
    dw, db = [DeviceBuffer(I * O * 4) for _ in range(groups)], [DeviceBuffer(O * 4) for _ in range(groups)]
    tab = lambda bufs: (C.c_void_p * groups)(*[b.p.value for b in bufs])  # noqa: E731
    check(gpu_lib.boat_cuda_weight_grads(mma, groups, I, O, T, tab(dx), tab(ddy), capi.CUDA_BF16 if bf else capi.CUDA_F32,
                                         tab(dw), tab(db), 0), "weight_grads")
    check(gpu_lib.boat_cuda_sync(), "sync")
    for g in range(groups):
        assert rel(dw[g].numpy((I, O)), x[g].astype(np.float64).T @ dy[g].astype(np.float64)) <= 1e-5
        assert np.abs(db[g].numpy((O,)) - dy[g].astype(np.float64).sum(0)).max() <= 1e-6 * np.abs(dy[g]).sum(0).max()


@pytest.mark.parametrize("S,hs", [(1, 8), (5, 5), (63, 16), (64, 20), (65, 32), (130, 33), (200, 64), (129, 100), (70, 128)])
@pytest.mark.parametrize("causal", [False, True], ids=["full", "causal"])
def test_exact_attention_core_edges(gpu_lib, S, hs, causal):
    got, ref = run_core(gpu_lib, capi.MMA_FP32, 3, S, hs, causal)
    for key in ("o", "dv") if S == 1 else ("o", "dq", "dk", "dv"):      # one key: dq and dk vanish
        assert rel(got[key], ref[key]) <= 1e-5, key


# delta made by the CTAs or by a pass of its own: the last and first numbers of units, tiles and head sizes of either (148 SMs)
@pytest.mark.parametrize("units,S,hs", [(591, 6, 16), (592, 6, 16), (295, 65, 16), (296, 65, 16), (5, 128, 64), (5, 128, 65), (5, 129, 16)])
def test_attention_backward_with_delta_of_either_kind(gpu_lib, units, S, hs):
    got, ref = run_core(gpu_lib, capi.MMA_FP32, units, S, hs, True)
    for key in ("dq", "dk", "dv"):
        assert rel(got[key], ref[key]) <= 1e-5, key


@pytest.mark.parametrize("S,hs", [(70, 16), (129, 32), (66, 80)])
def test_cuda_core_attention_on_bf16_storage(gpu_lib, S, hs):
    got, ref = run_core(gpu_lib, capi.MMA_BF16, 2, S, hs, True)
    for key in ("o", "dq", "dk", "dv"):
        assert rel(got[key], ref[key]) <= 2e-2, key
