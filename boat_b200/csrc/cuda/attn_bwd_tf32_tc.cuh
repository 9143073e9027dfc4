// attn_bwd_tf32_tc.cuh - fused attention backward on tcgen05 for FP32 storage (kind::tf32, FP32
// accumulation), head size 64.
//
// Replaces attention_backward (reference src/layers/attention.c:1388-1534) for FP32 tensors:
// the probabilities are rebuilt from the saved log-sum-exp tile by tile, and P and dS stay in
// TF32 (never BF16), so the result holds the 5e-3 tolerance of TF32 arithmetic.
//
// Two kinds of CTA.  The BF16 backward keeps dS^T in shared memory because dQ = dS.K
// wants dS with queries on the M side while dK = dS^T.Q wants it with keys on the M side; an
// FP32 dS^T tile is 64 KB and does not fit beside double-staged FP32 Q/dO tiles.  Splitting the
// work by output removes the tile altogether - each product then takes its left operand
// straight from tensor memory, exactly where the softmax warps wrote it:
//
//   dQ          CTA = one 128-row query tile, walks the key tiles (like the forward)
//       S  = Q.K^T, dP = dO.V^T             both operands from shared memory
//       dS = P*(dP - delta)/sqrt(hs)        softmax warps, thread = query row, written over S
//       dQ += dS.K                          A = dS from tensor memory, B = K with hs on the N side
//   dK, dV      CTA = one 128-row key tile, walks the query tiles that see it
//       S^T = K.Q^T, dP^T = V.dO^T
//       P^T over S^T, dS^T over dP^T        softmax warps, thread = key row
//       dV += P^T.dO,  dK += dS^T.Q         A from tensor memory, B = dO / Q with hs on the N side
// One launch holds both kinds, the longer dK/dV ones first, so that the dQ ones fill the SMs that a last
// wave of the others leaves idle.
// dQ, dK, dV leave the kernel rounded to TF32: they feed the TF32 projection GEMMs.
//
// No scratch memory, no atomics, no reduction between CTAs: every output row is produced by one
// CTA, so the results are deterministic.  The price is that S and dP are computed twice (7
// products per tile pair instead of 5); this path serves FP32 tensors, whose problems are small.
//
// An FP32 operand that the tensor core reads along M or N must lie in shared memory with the
// 128-byte swizzle in 32-byte units, one that it reads along K with the usual 16-byte units.
// K (dQ) and Q, dO (dK, dV) are needed both ways, so those tiles are loaded twice,
// once per tensor map; the second copy comes from L2.
// Warp 0: TMA producer, warp 1: MMA issuer, warps 2-9: softmax and epilogue, two warps per 32 tensor-memory lanes with half
// of a tile's columns each.
//
// The seven 32 KB tiles that fit shared memory and the tensor-memory columns are dealt out so that the softmax warps and
// the tensor core work at the same time: the scores have two buffers, those of the tile after next are
// computed right behind the product that reads the probabilities (or dS) out of their buffer; dP of
// the next tile is computed under its exponentials; each operand tile is loaded again as soon as its own last product
// is complete, and what is wanted soonest after that has two buffers.  With one buffer of everything, where
// loads, products and exponentials of a tile followed one another, 64 units of 512 x 64 took 79 us with the delta pass, now 52; 128 causal
// units of 1000 307, now 204.
#pragma once
#include "attn_bwd_tc.cuh"

namespace boatcu {
namespace attn_tc {

constexpr int kBwd32Threads = 320;
constexpr int kBwd32Softmax = 256;                 // threads of the softmax warps
constexpr int kBwd32HS = 64;
constexpr int kBwd32Tile = 2 * kBoxBytes;          // one 128 x 64 FP32 tile: two boxes of 128 rows x 128 bytes

struct Bwd32Cfg {
    // Seven tiles + two (lse, delta) buffers + barriers: 231,680 of the 232,448 bytes a CTA may have, so the base has to
    // come 1024-byte aligned from the launch (checked at kernel entry).
    static constexpr int SMEM = 7 * kBwd32Tile + 2048 + 256;
    static constexpr uint32_t COL_S = 0, COL_DP = 256;          // two score buffers, dP
    static constexpr uint32_t COL_DQ = 384;                     // dQ CTAs
    static constexpr uint32_t COL_DV = 384, COL_DK = 448;       // dK, dV CTAs
    static constexpr uint32_t TMEM_COLS = 512;
};

struct Bwd32Params {
    const float* lse;      // [units*S]
    const float* delta;    // [units*S]
    float* dQ;             // dQ CTAs
    float* dK;             // dK, dV CTAs
    float* dV;
    int S, units, causal;
    float scale;
    unsigned int* status;
};

__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t t;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(t) : "f"(x));
    return t;
}

// Loads a 128 x 64 tile; by the elected lane.
__device__ __forceinline__ void bwd32_load(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int row, int unit) {
    mbar_arrive_expect_tx(bar, kBwd32Tile);
    tma_load_4d(dst, map, bar, 0, row, 0, unit);
}

// D[128 x 128] = A . B^T over hs, both tiles read along hs.
__device__ __forceinline__ void bwd32_scores(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc) {
    constexpr uint32_t idesc = make_idesc(kTF32, false, false, kTile, kTile);
#pragma unroll
    for (int kk = 0; kk < kBwd32HS * 4 / 32; ++kk) {
        const uint32_t off = ((kk / 4) * kBoxBytes + (kk % 4) * 32) >> 4;
        mma_ss<true>(d_tmem, a_desc + off, b_desc + off, idesc, kk > 0);
    }
}

// D[128 x hs] += A . B, A [128 x 128] from tensor memory, B read along its 128 rows.
__device__ __forceinline__ void bwd32_accumulate(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, bool more) {
    constexpr uint32_t idesc = make_idesc(kTF32, false, true, kTile, kBwd32HS);
#pragma unroll
    for (int kk = 0; kk < kTile / 8; ++kk) mma_ts<true>(d_tmem, a_tmem + kk * 8, b_desc + (kk * 8 * 128 >> 4), idesc, more || kk > 0);
}

// 32 columns of a finished accumulator, rounded to TF32, to one row of the output.
__device__ __forceinline__ void bwd32_store(float* out, uint32_t taddr, bool live) {
    uint32_t r[32];
    tmem_ld32(taddr, r);
    tmem_wait_ld();
    if (!live) return;
#pragma unroll
    for (int i = 0; i < 32; i += 4)
        *reinterpret_cast<float4*>(out + i) = make_float4(round_to_tf32(__uint_as_float(r[i])), round_to_tf32(__uint_as_float(r[i + 1])),
                                                          round_to_tf32(__uint_as_float(r[i + 2])), round_to_tf32(__uint_as_float(r[i + 3])));
}

// ------------------------------------------------------------------------------------------------
// dQ: one query tile per CTA
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void bwd32_dq(uint8_t* smem, int block, const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_k_mn,
                                         const CUtensorMap& map_v, const CUtensorMap& map_do, const Bwd32Params& p) {
    using C = Bwd32Cfg;
    constexpr int HS = kBwd32HS;
    uint8_t* q_smem = smem;
    uint8_t* do_smem = q_smem + kBwd32Tile;
    uint8_t* k_smem = do_smem + kBwd32Tile;          // K read along hs (scores)
    uint8_t* v_smem = k_smem + kBwd32Tile;           // [2]
    uint8_t* kmn_smem = v_smem + 2 * kBwd32Tile;     // [2] K read along the key rows (dQ)
    uint64_t* bars = (uint64_t*)(smem + 7 * kBwd32Tile + 2048);
    uint64_t* q_full = bars;            // Q landed
    uint64_t* do_full = bars + 1;       // dO landed
    uint64_t* k_full = bars + 2;        // K landed
    uint64_t* k_empty = bars + 3;       // ... and the tile's S is complete
    uint64_t* v_full = bars + 4;        // [2]
    uint64_t* v_empty = bars + 6;       // [2] dP complete
    uint64_t* kmn_full = bars + 8;      // [2]
    uint64_t* kmn_empty = bars + 10;    // [2] dQ of the tile complete
    uint64_t* s_full = bars + 12;       // [2] S complete
    uint64_t* dp_full = bars + 14;      // dP complete
    uint64_t* ds_full = bars + 15;      // dS written over S (256 arrivals)
    uint64_t* dq_done = bars + 16;      // last dQ MMA complete
    uint32_t* tmem_slot = (uint32_t*)(bars + 17);

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int n_tiles = (p.S + kTile - 1) / kTile;
    const int unit = block % p.units;
    const int qt = n_tiles - 1 - block / p.units;       // long (late) rows first when causal
    const int n_kv = p.causal ? qt + 1 : n_tiles;

    if (threadIdx.x == 0) {
        for (int b = 0; b < 17; ++b) mbar_init(&bars[b], &bars[b] == ds_full ? kBwd32Softmax : 1);
        fence_barrier_init();
        tma_prefetch_desc(&map_q);
        tma_prefetch_desc(&map_k);
        tma_prefetch_desc(&map_k_mn);
        tma_prefetch_desc(&map_v);
        tma_prefetch_desc(&map_do);
    }
    if (warp == 1) tmem_alloc(tmem_slot, C::TMEM_COLS);
    griddep_sync();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_s = tmem_base + C::COL_S, tmem_dp = tmem_base + C::COL_DP, tmem_dq = tmem_base + C::COL_DQ;

    if (warp == 0) {
        // the whole warp in step, one elected lane issues, loads and products alike (see the forward kernel)
        const bool leader = elect_one();
        bool ok = true;
        // K, V and K again of tile j
        auto load_k = [&](int j) {
            if (!ok || j >= n_kv) return;
            ok = mbar_wait_warp(k_empty, (j & 1) ^ 1, p.status, kTimeoutProducer);
            if (ok && leader) bwd32_load(k_smem, &map_k, k_full, j * kTile, unit);
        };
        auto load_v = [&](int j) {
            if (!ok || j >= n_kv) return;
            ok = mbar_wait_warp(&v_empty[j & 1], ((j >> 1) & 1) ^ 1, p.status, kTimeoutProducer);
            if (ok && leader) bwd32_load(v_smem + (j & 1) * kBwd32Tile, &map_v, &v_full[j & 1], j * kTile, unit);
        };
        auto load_kmn = [&](int j) {
            if (!ok || j >= n_kv) return;
            ok = mbar_wait_warp(&kmn_empty[j & 1], ((j >> 1) & 1) ^ 1, p.status, kTimeoutProducer);
            if (ok && leader) bwd32_load(kmn_smem + (j & 1) * kBwd32Tile, &map_k_mn, &kmn_full[j & 1], j * kTile, unit);
        };
        // what the first product wants comes first
        if (leader) bwd32_load(q_smem, &map_q, q_full, qt * kTile, unit);
        load_k(0);
        if (leader) bwd32_load(do_smem, &map_do, do_full, qt * kTile, unit);
        load_v(0);
        load_kmn(0);
        load_v(1);
        load_kmn(1);
        load_k(1);
        // in the order in which the buffers come free
        for (int j = 0; j + 2 < n_kv && ok; ++j) {
            load_v(j + 2);
            load_k(j + 2);
            load_kmn(j + 2);
        }
        if (!ok)
            for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    } else if (warp == 1) {
        const uint64_t q_d = smem_desc_sw128(smem_u32(q_smem), 16, 1024), do_d = smem_desc_sw128(smem_u32(do_smem), 16, 1024);
        const uint64_t k_d = smem_desc_sw128(smem_u32(k_smem), 16, 1024), v_d = smem_desc_sw128(smem_u32(v_smem), 16, 1024);
        const uint64_t k_mn = smem_desc_mn(smem_u32(kmn_smem), kBoxBytes, true);
        const bool leader = elect_one();
        bool ok = mbar_wait_warp(q_full, 0, p.status, kTimeoutMma);
        auto issue_s = [&](int j) {
            if (!ok || j >= n_kv) return;
            ok = mbar_wait_warp(k_full, j & 1, p.status, kTimeoutMma);
            if (!ok) return;
            tc_fence_after_sync();
            if (leader) {
                bwd32_scores(tmem_s + (j & 1) * kTile, q_d, k_d);
                mma_commit(&s_full[j & 1]);
                mma_commit(k_empty);
            }
        };
        auto issue_dp = [&](int j) {
            if (!ok || j >= n_kv) return;
            ok = mbar_wait_warp(&v_full[j & 1], (j >> 1) & 1, p.status, kTimeoutMma);
            if (!ok) return;
            tc_fence_after_sync();
            if (leader) {
                bwd32_scores(tmem_dp, do_d, v_d + ((j & 1) * kBwd32Tile >> 4));
                mma_commit(dp_full);
                mma_commit(&v_empty[j & 1]);
            }
        };
        issue_s(0);
        ok = ok && mbar_wait_warp(do_full, 0, p.status, kTimeoutMma);
        issue_dp(0);
        issue_s(1);
        for (int j = 0; j < n_kv && ok; ++j) {
            if (!mbar_wait_warp(ds_full, j & 1, p.status, kTimeoutMma)) { ok = false; break; }
            issue_dp(j + 1);                        // dP(j) has been read, dS(j) is written
            if (!ok || !mbar_wait_warp(&kmn_full[j & 1], (j >> 1) & 1, p.status, kTimeoutMma)) { ok = false; break; }
            tc_fence_after_sync();
            if (leader) {
                bwd32_accumulate(tmem_dq, tmem_s + (j & 1) * kTile, k_mn + ((j & 1) * kBwd32Tile >> 4), j > 0);
                mma_commit(&kmn_empty[j & 1]);
                if (j == n_kv - 1) mma_commit(dq_done);
            }
            issue_s(j + 2);                         // behind dQ(j) on the in-order pipe, which reads its buffer
        }
    } else {
        // softmax warps: thread = query row and half of the tile's key columns
        const int lane_group = warp & 3, half = (warp - 2) >> 2;
        const int r_in_tile = lane_group * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(lane_group * 32) << 16;
        const int64_t grow = (int64_t)unit * p.S + (int64_t)qt * kTile + r_in_tile;
        const bool live = qt * kTile + r_in_tile < p.S;         // a row of the sequence (the last tile may be short)
        const float sl2 = p.scale * 1.4426950408889634f;
        const float neg_lse2 = live ? -p.lse[grow] * 1.4426950408889634f : 0.f;
        const float neg_delta_s = live ? -p.delta[grow] * p.scale : 0.f;
        const int c0 = half * 64;
        bool ok = true;
        for (int j = 0; j < n_kv; ++j) {
            const uint32_t s_cols = tmem_s + (j & 1) * kTile + lane_addr + c0;
            if (!mbar_wait_warp(&s_full[j & 1], (j >> 1) & 1, p.status, kTimeoutSoftmax)) { ok = false; break; }
            tc_fence_after_sync();
            // keys beyond the diagonal, or without a mask beyond the end of the sequence
            const bool masked = p.causal ? j == qt : j == n_tiles - 1;
            const int last = (p.causal ? r_in_tile : p.S - 1 - j * kTile) - c0;
            uint32_t s[64];
            tmem_ld32(s_cols, *reinterpret_cast<uint32_t(*)[32]>(s));
            tmem_ld32(s_cols + 32, *reinterpret_cast<uint32_t(*)[32]>(s + 32));
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 64; ++i) s[i] = __float_as_uint(fast_exp2(fmaf(__uint_as_float(s[i]), sl2, neg_lse2)));
            if (masked) {
#pragma unroll
                for (int i = 0; i < 64; ++i)
                    if (i > last) s[i] = 0u;
            }
            if (!mbar_wait_warp(dp_full, j & 1, p.status, kTimeoutSoftmax)) { ok = false; break; }
            tc_fence_after_sync();
            uint32_t d[64];
            tmem_ld32(tmem_dp + lane_addr + c0, *reinterpret_cast<uint32_t(*)[32]>(d));
            tmem_ld32(tmem_dp + lane_addr + c0 + 32, *reinterpret_cast<uint32_t(*)[32]>(d + 32));
            tmem_wait_ld();
            // P * (dP - delta) / sqrt(hs)
#pragma unroll
            for (int i = 0; i < 64; ++i) s[i] = to_tf32(__uint_as_float(s[i]) * fmaf(__uint_as_float(d[i]), p.scale, neg_delta_s));
            tmem_st32(s_cols, *reinterpret_cast<uint32_t(*)[32]>(s));
            tmem_st32(s_cols + 32, *reinterpret_cast<uint32_t(*)[32]>(s + 32));
            tmem_wait_st();
            tc_fence_before_sync();
            mbar_arrive(ds_full);
        }
        if (ok && mbar_wait_warp(dq_done, 0, p.status, kTimeoutEpilogue)) {
            tc_fence_after_sync();
            bwd32_store(p.dQ + grow * HS + half * 32, tmem_dq + lane_addr + half * 32, live);
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
}

// ------------------------------------------------------------------------------------------------
// dK, dV: one key tile per CTA
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void bwd32_dkv(uint8_t* smem, int block, const CUtensorMap& map_q, const CUtensorMap& map_q_mn, const CUtensorMap& map_k,
                                          const CUtensorMap& map_v, const CUtensorMap& map_do, const CUtensorMap& map_do_mn,
                                          const Bwd32Params& p) {
    using C = Bwd32Cfg;
    constexpr int HS = kBwd32HS;
    uint8_t* k_smem = smem;
    uint8_t* v_smem = k_smem + kBwd32Tile;
    uint8_t* q_smem = v_smem + kBwd32Tile;           // Q read along hs (scores)
    uint8_t* qmn_smem = q_smem + kBwd32Tile;         // Q read along the query rows (dK)
    uint8_t* domn_smem = qmn_smem + kBwd32Tile;      // dO read along the query rows (dV)
    uint8_t* do_smem = domn_smem + kBwd32Tile;       // [2] dO read along hs (dP)
    float* stat_s = (float*)(smem + 7 * kBwd32Tile); // [2][-lse*log2e [128], -delta/sqrt(hs) [128]]
    uint64_t* bars = (uint64_t*)(stat_s + 512);
    uint64_t* k_full = bars;
    uint64_t* v_full = bars + 18;
    uint64_t* q_full = bars + 1;
    uint64_t* q_empty = bars + 2;       // S^T of the tile complete
    uint64_t* qmn_full = bars + 3;
    uint64_t* qmn_empty = bars + 4;     // dK of the tile complete
    uint64_t* domn_full = bars + 5;
    uint64_t* domn_empty = bars + 6;    // dV of the tile complete
    uint64_t* do_full = bars + 7;       // [2]
    uint64_t* do_empty = bars + 9;      // [2] dP^T complete
    uint64_t* s_full = bars + 11;       // [2] S^T complete
    uint64_t* dp_full = bars + 13;      // dP^T complete
    // P^T written over S^T (256 arrivals).  Two barriers in turn: the scores of tile t+1 are issued before the wait for
    // P^T(t), so the softmax warps may be through with P^T(t+1) by the time the MMA issuer gets to that wait.
    uint64_t* p_full = bars + 14;       // [2]
    uint64_t* ds_full = bars + 16;      // dS^T written over dP^T (256 arrivals)
    uint64_t* acc_done = bars + 17;     // last dV, dK MMAs complete
    uint32_t* tmem_slot = (uint32_t*)(bars + 19);

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int n_tiles = (p.S + kTile - 1) / kTile;
    const int unit = block % p.units;
    const int jt = block / p.units;                     // early key tiles have the long walks when causal
    const int i0 = p.causal ? jt : 0;
    const int n_q = n_tiles - i0;

    if (threadIdx.x == 0) {
        for (int b = 0; b < 19; ++b) mbar_init(&bars[b], &bars[b] >= p_full && &bars[b] <= ds_full ? kBwd32Softmax : 1);
        fence_barrier_init();
        tma_prefetch_desc(&map_q);
        tma_prefetch_desc(&map_q_mn);
        tma_prefetch_desc(&map_k);
        tma_prefetch_desc(&map_v);
        tma_prefetch_desc(&map_do);
        tma_prefetch_desc(&map_do_mn);
    }
    if (warp == 1) tmem_alloc(tmem_slot, C::TMEM_COLS);
    griddep_sync();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_st = tmem_base + C::COL_S, tmem_dpt = tmem_base + C::COL_DP;
    const uint32_t tmem_dv = tmem_base + C::COL_DV, tmem_dk = tmem_base + C::COL_DK;

    if (warp == 0) {
        const bool leader = elect_one();
        bool ok = true;
        auto load = [&](int t, uint8_t* dst, const CUtensorMap* map, uint64_t* full, uint64_t* empty, uint32_t parity) {
            if (!ok || t >= n_q) return;
            ok = mbar_wait_warp(empty, parity ^ 1, p.status, kTimeoutProducer);
            if (ok && leader) bwd32_load(dst, map, full, (i0 + t) * kTile, unit);
        };
        auto load_q = [&](int t) { load(t, q_smem, &map_q, q_full, q_empty, t & 1); };
        auto load_qmn = [&](int t) { load(t, qmn_smem, &map_q_mn, qmn_full, qmn_empty, t & 1); };
        auto load_domn = [&](int t) { load(t, domn_smem, &map_do_mn, domn_full, domn_empty, t & 1); };
        auto load_do = [&](int t) { load(t, do_smem + (t & 1) * kBwd32Tile, &map_do, &do_full[t & 1], &do_empty[t & 1], (t >> 1) & 1); };
        // what the first product wants comes first
        if (leader) bwd32_load(k_smem, &map_k, k_full, jt * kTile, unit);
        load_q(0);
        if (leader) bwd32_load(v_smem, &map_v, v_full, jt * kTile, unit);
        load_do(0);
        load_domn(0);
        load_qmn(0);
        load_do(1);
        load_q(1);
        // in the order in which the buffers come free
        for (int t = 0; t + 1 < n_q && ok; ++t) {
            load_q(t + 2);
            load_do(t + 2);
            load_domn(t + 1);
            load_qmn(t + 1);
        }
        if (!ok)
            for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    } else if (warp == 1) {
        const uint64_t k_d = smem_desc_sw128(smem_u32(k_smem), 16, 1024), v_d = smem_desc_sw128(smem_u32(v_smem), 16, 1024);
        const uint64_t q_d = smem_desc_sw128(smem_u32(q_smem), 16, 1024), do_d = smem_desc_sw128(smem_u32(do_smem), 16, 1024);
        const uint64_t q_mn = smem_desc_mn(smem_u32(qmn_smem), kBoxBytes, true), do_mn = smem_desc_mn(smem_u32(domn_smem), kBoxBytes, true);
        const bool leader = elect_one();
        bool ok = mbar_wait_warp(k_full, 0, p.status, kTimeoutMma);
        auto issue_s = [&](int t) {
            if (!ok || t >= n_q) return;
            ok = mbar_wait_warp(q_full, t & 1, p.status, kTimeoutMma);
            if (!ok) return;
            tc_fence_after_sync();
            if (leader) {
                bwd32_scores(tmem_st + (t & 1) * kTile, k_d, q_d);
                mma_commit(&s_full[t & 1]);
                mma_commit(q_empty);
            }
        };
        auto issue_dp = [&](int t) {
            if (!ok || t >= n_q) return;
            ok = mbar_wait_warp(&do_full[t & 1], (t >> 1) & 1, p.status, kTimeoutMma);
            if (!ok) return;
            tc_fence_after_sync();
            if (leader) {
                bwd32_scores(tmem_dpt, v_d, do_d + ((t & 1) * kBwd32Tile >> 4));
                mma_commit(dp_full);
                mma_commit(&do_empty[t & 1]);
            }
        };
        issue_s(0);
        ok = ok && mbar_wait_warp(v_full, 0, p.status, kTimeoutMma);
        issue_dp(0);
        issue_s(1);
        for (int t = 0; t < n_q && ok; ++t) {
            if (!mbar_wait_warp(&p_full[t & 1], (t >> 1) & 1, p.status, kTimeoutMma)) { ok = false; break; }
            if (!mbar_wait_warp(domn_full, t & 1, p.status, kTimeoutMma)) { ok = false; break; }
            tc_fence_after_sync();
            if (leader) {
                bwd32_accumulate(tmem_dv, tmem_st + (t & 1) * kTile, do_mn, t > 0);
                mma_commit(domn_empty);
            }
            issue_s(t + 2);                         // behind dV(t) on the in-order pipe, which reads its buffer
            if (!ok || !mbar_wait_warp(ds_full, t & 1, p.status, kTimeoutMma)) { ok = false; break; }
            if (!mbar_wait_warp(qmn_full, t & 1, p.status, kTimeoutMma)) { ok = false; break; }
            tc_fence_after_sync();
            if (leader) {
                bwd32_accumulate(tmem_dk, tmem_dpt, q_mn, t > 0);
                mma_commit(qmn_empty);
                if (t == n_q - 1) mma_commit(acc_done);
            }
            issue_dp(t + 1);                        // behind dK(t), which reads dS^T out of its columns
        }
    } else {
        // softmax warps: thread = key row and half of the tile's query columns; the statistics belong to the columns
        const int lane_group = warp & 3, half = (warp - 2) >> 2;
        const int r = lane_group * 32 + lane;
        const int tid = (warp - 2) * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(lane_group * 32) << 16;
        const float sl2 = p.scale * 1.4426950408889634f;
        const int c0 = half * 64;
        // One statistic of the tile's 128 queries per thread: -lse (log2 domain) or -delta/sqrt(hs).  Queries beyond the
        // end of the sequence get an offset of -inf: their P is exactly zero.
        const float* const stat = tid < 128 ? p.lse : p.delta;
        const float factor = tid < 128 ? -1.4426950408889634f : -p.scale;
        auto fetch = [&](int t) -> float {
            const int q = (i0 + t) * kTile + (tid & 127);
            if (t < n_q && q < p.S) return stat[(int64_t)unit * p.S + q] * factor;
            return tid < 128 ? -INFINITY : 0.f;
        };
        float mine = fetch(0);
        bool ok = true;
        // A warp whose wait gave up does no more work but stays in the loop, so that nobody is left alone at the barrier.
        for (int t = 0; t < n_q; ++t) {
            // Two buffers by tile parity: nobody gets to tile t+2 before everybody has passed the barrier of t+1, that is,
            // has read the statistics of tile t.
            float* lse_s = stat_s + (t & 1) * 256;
            const float* delta_s = lse_s + 128;
            lse_s[tid] = mine;
            mine = fetch(t + 1);
            named_barrier_sync(1, kBwd32Softmax);
            const uint32_t s_cols = tmem_st + (t & 1) * kTile + lane_addr + c0, d_cols = tmem_dpt + lane_addr + c0;
            ok = ok && mbar_wait_warp(&s_full[t & 1], (t >> 1) & 1, p.status, kTimeoutSoftmax);
            if (!ok) continue;
            tc_fence_after_sync();
            const bool diag = p.causal && i0 + t == jt;
            uint32_t s[64];                         // P, not rounded
            tmem_ld32(s_cols, *reinterpret_cast<uint32_t(*)[32]>(s));
            tmem_ld32(s_cols + 32, *reinterpret_cast<uint32_t(*)[32]>(s + 32));
            tmem_wait_ld();
#pragma unroll
            for (int x = 0; x < 64; x += 4) {
                const float4 l4 = *reinterpret_cast<const float4*>(lse_s + c0 + x);
                const float nl[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) s[x + e] = __float_as_uint(fast_exp2(fmaf(__uint_as_float(s[x + e]), sl2, nl[e])));
            }
            if (diag) {                             // query q sees key r only when q >= r
#pragma unroll
                for (int x = 0; x < 64; ++x)
                    if (c0 + x < r) s[x] = 0u;
            }
#pragma unroll
            for (int c = 0; c < 64; c += 32) {
                uint32_t q[32];
#pragma unroll
                for (int x = 0; x < 32; ++x) q[x] = to_tf32(__uint_as_float(s[c + x]));
                tmem_st32(s_cols + c, q);
            }
            tmem_wait_st();
            tc_fence_before_sync();
            mbar_arrive(&p_full[t & 1]);
            ok = mbar_wait_warp(dp_full, t & 1, p.status, kTimeoutSoftmax);
            if (!ok) continue;
            tc_fence_after_sync();
#pragma unroll
            for (int c = 0; c < 64; c += 32) {
                uint32_t d[32];
                tmem_ld32(d_cols + c, d);
                tmem_wait_ld();
#pragma unroll
                for (int x = 0; x < 32; x += 4) {
                    const float4 d4 = *reinterpret_cast<const float4*>(delta_s + c0 + c + x);
                    const float nd[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) d[x + e] = to_tf32(__uint_as_float(s[c + x + e]) * fmaf(__uint_as_float(d[x + e]), p.scale, nd[e]));
                }
                tmem_st32(d_cols + c, d);
            }
            tmem_wait_st();
            tc_fence_before_sync();
            mbar_arrive(ds_full);
        }
        if (ok && mbar_wait_warp(acc_done, 0, p.status, kTimeoutEpilogue)) {
            tc_fence_after_sync();
            // dV by the first four warps, dK by the others
            const int64_t grow = (int64_t)unit * p.S + (int64_t)jt * kTile + r;
            const bool live = jt * kTile + r < p.S;
            float* out = (half ? p.dK : p.dV) + grow * HS;
            const uint32_t col = (half ? tmem_dk : tmem_dv) + lane_addr;
            bwd32_store(out, col, live);
            bwd32_store(out + 32, col + 32, live);
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
}

struct Bwd32Maps {
    CUtensorMap q, q_mn, k, k_mn, v, dout, dout_mn;      // _mn: read along the rows, 32-byte swizzle units
};

__global__ void __launch_bounds__(kBwd32Threads, 1)
attn_bwd_tf32_kernel(const __grid_constant__ Bwd32Maps m, const __grid_constant__ Bwd32Params p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    if ((smem_u32(smem_raw) & 1023u) != 0) {     // uniform for the whole CTA; nothing to undo yet
        if (threadIdx.x == 0) atomicCAS(p.status, 0u, (unsigned int)kTimeoutOther + 100u);
        return;
    }
    const int n = gridDim.x / 2;
    if (blockIdx.x < n) bwd32_dkv(smem_raw, blockIdx.x, m.q, m.q_mn, m.k, m.v, m.dout, m.dout_mn, p);
    else                bwd32_dq(smem_raw, blockIdx.x - n, m.q, m.k, m.k_mn, m.v, m.dout, p);
}

}  // namespace attn_tc
}  // namespace boatcu
