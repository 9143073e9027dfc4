// attn_tc.cu - host side of the tcgen05 attention-core kernels: shape support, tensor maps,
// launches.  The kernels themselves are in attn_fwd_tc.cuh, attn_bwd_tc.cuh (BF16 storage) and
// attn_bwd_tf32_tc.cuh (FP32 storage).
#include "attn_bwd_tc.cuh"
#include "attn_bwd_tf32_tc.cuh"
#include <stdlib.h>

namespace boatcu {

using namespace attn_tc;

namespace {

template <typename T, int HS>
int launch_fwd(int64_t units, int64_t S, int causal, float scale, const void* Q, const void* K, const void* V,
               void* O, float* lse) {
    using C = FwdCfg<T, HS>;
    CUtensorMap mq, mk, mv;
    if (int rc = make_tensor_map_unit_tiles(&mq, Q, C::ES, units, S, HS, kTile)) return rc;
    if (int rc = make_tensor_map_unit_tiles(&mk, K, C::ES, units, S, HS, kTile)) return rc;
    // V is read by the tensor core along its contiguous head dimension: FP32 needs the
    // 32-byte-unit swizzle for that
    if (int rc = make_tensor_map_unit_tiles(&mv, V, C::ES, units, S, HS, kTile, C::TF32)) return rc;
    FwdParams p;
    p.O = O;
    p.lse = lse;
    p.S = (int)S;
    p.units = (int)units;
    p.causal = causal;
    p.scale = scale;
    p.wide = ((uintptr_t)O & 31) == 0;
    p.status = kernel_status_ptr();
    // units whose K and V (2 * S * hs elements each) together take about a third of L2
    const int64_t group = (40ll << 20) / (2 * S * HS * (int64_t)C::ES);
    p.group = (int)(group < 1 ? 1 : (group > units ? units : group));
    {
        // BOAT_FWD_GROUP=n in the environment overrides the group size; it is read at every launch so
        // that a test can run a small problem in several groups, the first of them short
        const char* e = getenv("BOAT_FWD_GROUP");
        const int n = e ? atoi(e) : 0;
        if (n >= 1) p.group = n > (int)units ? (int)units : n;
    }
    auto kern = attn_fwd_tc_kernel<T, HS>;
    static bool configured = false;
    if (!configured) {
        BOATCU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
        configured = true;
    }
    const int64_t grid = units * ((ceil_div(S, kTile) + 1) / 2);      // one CTA per pair of query tiles
    ProfileScope prof("attn_fwd_tc");
    BOATCU_RUN(kern, (unsigned)grid, kFwdThreads, C::SMEM, mq, mk, mv, p);
    BOATCU_LAUNCH_OK("attn_fwd_tc");
    return 0;
}

}  // namespace

bool attn_tc_supported(int mma, int64_t units, int64_t S, int64_t hs, int io_type) {
    if (S < 1 || units * ceil_div(S, kTile) * kTile > 0x7fffffffLL) return false;
    if (mma == BOAT_MMA_BF16) return io_type == BOAT_CUDA_BF16 && (hs == 64 || hs == 128);
    if (mma == BOAT_MMA_TF32) return io_type == BOAT_CUDA_F32 && hs == 64;
    return false;
}

int attn_fwd_tc(int mma, int64_t units, int64_t S, int64_t hs, int causal, float scale, const void* Q, const void* K,
                const void* V, int io_type, void* O, float* lse) {
    (void)io_type;
    if (int rc = ensure_init()) return rc;
    if (mma == BOAT_MMA_BF16) {
        if (hs == 64) return launch_fwd<__nv_bfloat16, 64>(units, S, causal, scale, Q, K, V, O, lse);
        return launch_fwd<__nv_bfloat16, 128>(units, S, causal, scale, Q, K, V, O, lse);
    }
    return launch_fwd<float, 64>(units, S, causal, scale, Q, K, V, O, lse);
}

namespace {

template <int HS>
int launch_bwd(int64_t units, int64_t S, int causal, float scale, const void* Q, const void* K, const void* V,
               const void* O, const void* dO, const float* lse, void* dQ, void* dK, void* dV, float* dq_accum,
               float* stats2) {
    using C = BwdCfg<HS>;
    CUtensorMap mq, mk, mv, mdo, mdq;
    const int64_t n_tiles = ceil_div(S, kTile);
    const int64_t stat_rows = units * n_tiles * kTile;        // the statistics are padded to whole tiles
    if (int rc = make_tensor_map_unit_tiles(&mq, Q, 2, units, S, HS, kTile)) return rc;
    if (int rc = make_tensor_map_unit_tiles(&mk, K, 2, units, S, HS, kTile)) return rc;
    if (int rc = make_tensor_map_unit_tiles(&mv, V, 2, units, S, HS, kTile)) return rc;
    if (int rc = make_tensor_map_unit_tiles(&mdo, dO, 2, units, S, HS, kTile)) return rc;
    if (int rc = make_tensor_map_units(&mdq, dq_accum, 4, units, S, HS, 32)) return rc;   // FP32 reduce-add target
    const size_t n = (size_t)units * (size_t)S * HS;
    BwdParams p;
    p.lse2 = stats2;
    p.delta2 = stats2 + stat_rows;
    p.dq_accum = dq_accum;
    p.dK = dK;
    p.dV = dV;
    p.S = (int)S;
    p.units = (int)units;
    p.causal = causal;
    // units whose dQ (FP32), Q, dO, K and V - 16 bytes per element of the unit - share L2 at a time
    const int64_t unit_bytes = S * HS * 16;
    int64_t group = (64ll << 20) / unit_bytes;
    p.group = (int)(group < 1 ? 1 : (group > units ? units : group));
    p.scale = scale;
    p.status = kernel_status_ptr();
    auto kern = attn_bwd_tc_kernel<HS>;
    static bool configured = false;
    if (!configured) {
        BOATCU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
        configured = true;
    }
    {
        ProfileScope prof("attn_delta");
        if (int rc = attn_bwd_prepare(dO, O, lse, units, S, n_tiles * kTile, HS, scale, stats2 + stat_rows, stats2, dq_accum)) return rc;
    }
    {
        ProfileScope prof("attn_bwd_tc");
        const int64_t grid = units * n_tiles;           // one CTA per walk; those on the SMs take the others over
        BOATCU_RUN(kern, (unsigned)grid, kBwdThreads, C::SMEM, mq, mk, mv, mdo, mdq, p);
        BOATCU_LAUNCH_OK("attn_bwd_tc");
        // the summed FP32 contributions become the BF16 output
        if (int rc = boat_cuda_cast(dQ, BOAT_CUDA_BF16, dq_accum, BOAT_CUDA_F32, (int64_t)n)) return rc;
    }
    return 0;
}

// FP32 storage, TF32 arithmetic, head size 64: one launch of CTAs over key tiles (dK, dV) and CTAs over
// query tiles (dQ); no scratch beyond delta.
int launch_bwd_tf32(int64_t units, int64_t S, int causal, float scale, const void* Q, const void* K, const void* V,
                    const void* dO, const float* lse, const float* delta, void* dQ, void* dK, void* dV) {
    using C = Bwd32Cfg;
    constexpr int HS = kBwd32HS, SMEM = C::SMEM;
    Bwd32Maps m;
    // the same matrices with both shared-memory layouts: 16-byte swizzle units for operands read
    // along hs, 32-byte units for operands read along their rows
    if (int rc = make_tensor_map_unit_tiles(&m.q, Q, 4, units, S, HS, kTile)) return rc;
    if (int rc = make_tensor_map_unit_tiles(&m.q_mn, Q, 4, units, S, HS, kTile, true)) return rc;
    if (int rc = make_tensor_map_unit_tiles(&m.k, K, 4, units, S, HS, kTile)) return rc;
    if (int rc = make_tensor_map_unit_tiles(&m.k_mn, K, 4, units, S, HS, kTile, true)) return rc;
    if (int rc = make_tensor_map_unit_tiles(&m.v, V, 4, units, S, HS, kTile)) return rc;
    if (int rc = make_tensor_map_unit_tiles(&m.dout, dO, 4, units, S, HS, kTile)) return rc;
    if (int rc = make_tensor_map_unit_tiles(&m.dout_mn, dO, 4, units, S, HS, kTile, true)) return rc;
    Bwd32Params p;
    p.lse = lse;
    p.delta = delta;
    p.dQ = (float*)dQ;
    p.dK = (float*)dK;
    p.dV = (float*)dV;
    p.S = (int)S;
    p.units = (int)units;
    p.causal = causal;
    p.scale = scale;
    p.status = kernel_status_ptr();
    static bool configured = false;     // per process = per device: the library binds to one device
    if (!configured) {
        BOATCU_CHECK(cudaFuncSetAttribute(attn_bwd_tf32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        configured = true;
    }
    const unsigned grid = (unsigned)(2 * units * ceil_div(S, kTile));
    ProfileScope prof("attn_bwd_tc");
    BOATCU_RUN(attn_bwd_tf32_kernel, grid, kBwd32Threads, SMEM, m, p);
    BOATCU_LAUNCH_OK("attn_bwd_tf32");
    return 0;
}

}  // namespace

// Scratch of the BF16 tensor-core backward: the FP32 accumulation buffer of dQ, then the two
// pre-scaled statistics per row, padded to whole 128-row tiles of every unit.  (The first part is a
// multiple of 256 bytes, the parts of the second of 512.)
size_t attn_bwd_tc_scratch_bytes(int mma, int64_t units, int64_t S, int64_t hs) {
    if (mma != BOAT_MMA_BF16) return 0;
    const size_t stat_rows = (size_t)units * (size_t)ceil_div(S, kTile) * kTile;
    return (size_t)units * (size_t)S * (size_t)hs * sizeof(float) + 2 * stat_rows * sizeof(float);
}

int attn_bwd_tc(int mma, int64_t units, int64_t S, int64_t hs, int causal, float scale, const void* Q, const void* K,
                const void* V, const void* O, const void* dO, const float* lse, const float* delta, int io_type, void* dQ,
                void* dK, void* dV, void* scratch, size_t scratch_bytes) {
    if (int rc = ensure_init()) return rc;
    if (mma == BOAT_MMA_BF16) {
        if (scratch_bytes < attn_bwd_tc_scratch_bytes(mma, units, S, hs))
            return set_error(12, "attention backward: scratch too small for the dQ accumulation buffer");
        float* stats2 = (float*)scratch + (size_t)units * (size_t)S * (size_t)hs;
        if (hs == 64)
            return launch_bwd<64>(units, S, causal, scale, Q, K, V, O, dO, lse, dQ, dK, dV, (float*)scratch, stats2);
        return launch_bwd<128>(units, S, causal, scale, Q, K, V, O, dO, lse, dQ, dK, dV, (float*)scratch, stats2);
    }
    (void)io_type;
    return launch_bwd_tf32(units, S, causal, scale, Q, K, V, dO, lse, delta, dQ, dK, dV);
}

}  // namespace boatcu
