// attn_bwd_tc.cuh - fused attention backward on tcgen05 (BF16 storage, FP32 accumulation).
//
// Replaces attention_backward (reference src/layers/attention.c:1421-1526), which keeps the
// probabilities of the forward and builds four more [B,nh,S,S] tensors.  Here P is rebuilt
// from the saved log-sum-exp, tile by tile, and nothing of size S x S touches HBM.
//
// A walk: one 128-row key/value tile of one (batch,head) unit against the query tiles that see
// it (all of them, or those at or below the diagonal when causal).  K and V stay in shared
// memory, dK and dV accumulate in tensor memory for the whole walk.  One CTA per SM does one walk after
// the other without a break in the pipeline: loads (with head size 64 also K and V), scores and dP^T of
// the next walk are under way while the last tile of this one is worked on, and dK, dV are stored behind
// the exponentials of the next walk's first tile.  (A CTA per walk or two paid some 10000 cycles for
// start, first loads and end, a quarter of the time at 16-tile walks.)
// Per query tile, with everything transposed so that key rows sit on the TMEM lanes:
//
//   S^T  = K . Q^T                                              SS MMA into region R0
//   P^T  = exp2(S^T*c - lse)        phase A, 8 softmax warps, written over S^T in R0 (BF16)
//   dV  += P^T . dO                 A = P^T in tensor memory
//   dP^T = V . dO^T                 SS MMA into R0 again, behind dV on the in-order tensor pipe
//   dS^T = P^T * (dP^T - delta) / sqrt(hs)    phase B; P^T is kept in registers, dS^T goes to smem
//   dK  += dS^T . Q                 A = dS^T from shared memory (K-major view)
//   dQ_i = dS . K                   A = the same shared-memory tile read along M (MN-major view)
//
// Tensor memory (512 columns): R0 = S^T / P^T (128), dQ (HS), dV (HS), dK (HS); with head size
// 128 that is all of it and dP^T borrows the dQ columns: the dQ warps take a tile's dQ into
// registers and shared memory within a few hundred cycles of its completion, and the next dQ
// product only comes after the softmax warps have consumed dP^T.  With head size 64 dP^T has 128
// columns of its own, and P^T 64.  In both cases dP^T is issued a tile ahead, and S^T of tile t+1 follows dV of
// tile t on the pipe - with head size 64 the softmax warps' taking of tile t's - so that those go from the exponentials
// (A) straight to dS^T (B) without waiting for the tensor pipe.
//
// dQ of a query tile gets one contribution per key tile; CTAs add theirs into an FP32 buffer
// with TMA reduce-add (cp.reduce.async.bulk.tensor), and a cast kernel turns the sum into the
// output type afterwards.  Four dedicated warps move the dQ tile out of tensor memory, through
// a staging area or (head size 128) the tile's dO stage, which is idle once the tile's MMAs are complete.  An SM
// gets reductions out at only about 20 bytes per clock (measured alike for TMA reduce-add and
// for red.global.add.v4.f32, which also stalls the softmax warps' shared memory traffic), so
// the read-out of a tile takes most of a tile period - off the critical path.
// The softmax warps synchronise only through the mbarriers of the pipeline - no barrier among
// themselves inside a walk: the per-row statistics of a query tile (-lse*log2e and
// -delta/sqrt(hs), pre-scaled by a small kernel) are brought in by the producer with two bulk
// copies per tile.
// Warp 0: TMA producer (K, V, Q, dO, statistics), warp 1: MMA issuer, warps 2-9: softmax + final dK/dV store
// (two warps per TMEM lane group, 64 query columns each), warps 10-13: dQ reduction.
#pragma once
#include <type_traits>
#include "attn_fwd_tc.cuh"

namespace boatcu {
namespace attn_tc {

constexpr int kBwdThreads = 448;
constexpr int kBwdAnswers = 4;        // answers to requests for work in flight

template <int HS>
struct BwdCfg {
    static constexpr int ROWB = HS * 2;
    static constexpr int NBOX = ROWB / 128;
    static constexpr int TILE_BYTES = NBOX * kBoxBytes;       // one 128 x HS BF16 tile
    static constexpr int DS_BYTES = 2 * kBoxBytes;             // dS^T: 128 x 128 BF16
    // With head size 64 dQ leaves through a staging area of its own; with 128 through the tile's idle dO stage.
    static constexpr int DQ_BYTES = HS == 64 ? 128 * HS * 4 : 0;
    // Q / dO stages: three when they fit (head size 64), so that the dO tile loaded behind a
    // dQ read-out is not needed before the tile after next
    static constexpr int Q_STAGES = HS == 64 ? 3 : 2;
    static constexpr int KV_BUFS = HS == 64 ? 2 : 1;          // K and V of this walk, and of the next where they fit
    // K,V + Q,dO stages + dS^T + dQ + two (lse, delta) buffers + barriers.  There is no room for manual alignment slack, so the
    // base must come 1024-byte aligned from the launch (checked at kernel entry).
    static constexpr int SMEM = KV_BUFS * 2 * TILE_BYTES + Q_STAGES * 2 * TILE_BYTES + DS_BYTES + DQ_BYTES + 2048 + 448;
    static constexpr int kMaxSmem = 232448;                   // of a CTA
    static_assert(SMEM <= kMaxSmem && SMEM + 1023 > kMaxSmem, "no room for alignment slack, and none needed");
    // tensor memory columns
    // R0 (columns 0..127) holds S^T, then P^T.  With head size 64 dP^T has 128 columns of its
    // own.  With head size 128 nothing is left (R0 + dQ + dV + dK = 512), and dP^T borrows the dQ
    // columns: they are idle from the moment the dQ warps hold a tile's dQ in registers and
    // shared memory until the next tile's dQ product, which needs dS^T and therefore comes after
    // the softmax warps have read dP^T anyway.  Either way dP^T of a tile is issued before the
    // softmax warps ask for it, and they go from the exponentials straight on to dS^T.
    static constexpr bool DP_OWN = 256 + 3 * HS <= 512;
    // With head size 64 P^T has columns of its own too (128 BF16 in 64 columns), so that the scores of the next tile, and
    // likewise its dP^T, follow as soon as the softmax warps have taken this tile's into registers, and are there when
    // those ask for them.
    static constexpr uint32_t COL_S = 0;
    static constexpr uint32_t COL_DQ = DP_OWN ? 256 : 128, COL_DV = COL_DQ + HS, COL_DK = COL_DQ + 2 * HS;
    static constexpr uint32_t COL_DP = DP_OWN ? 128 : COL_DQ;
    static constexpr uint32_t COL_P = DP_OWN ? 256 + 3 * HS : COL_S;
    static constexpr uint32_t P_HALF = DP_OWN ? 32 : 64;      // from the first half of a row of P^T to the second
    static constexpr uint32_t TMEM_COLS = 512;
};

struct BwdParams {
    const float* lse2;     // [units, whole tiles]  -lse * log2(e): the exponent offset in the log2 domain;
                           // -inf beyond the end of the sequence, where P is then exactly zero
    const float* delta2;   // [units, whole tiles]  -delta / sqrt(hs)
    float* dq_accum;       // [units*S, hs] FP32, zeroed before the launch
    void* dK;
    void* dV;
    int S, units, causal;
    int group;             // units scheduled together, see bwd_walk
    float scale;
    unsigned int* status;
};

__device__ __forceinline__ void named_barrier_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}

struct BwdWalk {
    int unit, jt;          // key tile
    int i0, n;             // first query tile, number of them
};

// Walk `index` (n 0: none).  Walk order: units in groups of p.group; inside a group the key tile is the
// slow index, longest walks first when causal.  The CTAs that run at the same time then belong to a few
// (batch, head) units, so the FP32 dQ rows they reduce into (S*HS*4 bytes per unit) and the unit's Q and dO
// stay in L2 - with key tiles as the slow index over all units, the dQ buffer of a large problem (268 MB
// at 64 units x 8192 x 128) no longer fits and every reduction misses to HBM.
__device__ __forceinline__ BwdWalk bwd_walk(const BwdParams& p, int index) {
    BwdWalk w;
    w.unit = w.jt = w.i0 = w.n = 0;
    if (index < 0) return w;
    const int n_tiles = (p.S + kTile - 1) / kTile;
    const int per_group = p.group * n_tiles;
    const int grp = index / per_group, rem = index - grp * per_group;
    const int in_group = min(p.group, p.units - grp * p.group);
    w.jt = rem / in_group;
    w.unit = grp * p.group + rem % in_group;
    w.i0 = p.causal ? w.jt : 0;
    w.n = n_tiles - w.i0;
    return w;
}

template <int HS>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                 const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_do,
                 const __grid_constant__ CUtensorMap map_dq, const BwdParams p) {
    using C = BwdCfg<HS>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw;
    if ((smem_u32(smem) & 1023u) != 0) {         // uniform for the whole CTA; nothing to undo yet
        if (threadIdx.x == 0) atomicCAS(p.status, 0u, (unsigned int)kTimeoutOther + 100u);
        return;
    }
    uint8_t* kv_smem = smem;                                           // [KV_BUFS] K, V
    uint8_t* q_smem = kv_smem + C::KV_BUFS * 2 * C::TILE_BYTES;        // [Q_STAGES]
    uint8_t* do_smem = q_smem + C::Q_STAGES * C::TILE_BYTES;           // [Q_STAGES]
    uint8_t* ds_smem = do_smem + C::Q_STAGES * C::TILE_BYTES;
    uint8_t* dq_smem = ds_smem + C::DS_BYTES;
    float* stat_s = (float*)(dq_smem + C::DQ_BYTES);                   // [2][-lse*log2e[128], -delta/sqrt(hs)[128]]
    uint64_t* bars = (uint64_t*)(stat_s + 512);
    uint64_t* kv_full = bars;                   // [KV_BUFS]
    uint64_t* q_full = bars + 16;               // [Q_STAGES] Q tile landed
    uint64_t* s_full = bars + 5;                // S^T complete
    uint64_t* dq_full = bars + 7;               // all MMAs of the tile complete
    uint64_t* dq_empty = bars + 8;              // dQ is out of its TMEM columns
    uint64_t* all_done = bars + 9;
    uint64_t* dp_full = bars + 10;              // dP^T complete
    uint64_t* do_full = bars + 19;              // [Q_STAGES] dO tile landed
    uint64_t* q_empty = bars + 22;              // [Q_STAGES] S^T and dK of the tile are complete: its Q stage is free
    uint64_t* p_full = bars + 3;                // P^T in TMEM (256 arrivals)
    uint64_t* kv_empty = bars + 26;             // [KV_BUFS] the walk's MMAs are complete: K and V may be replaced
    uint64_t* acc_free = bars + 2;              // dK, dV of the walk are out of tensor memory (256 arrivals)
    uint64_t* stat_full = bars + 11;            // [2] the tile's statistics landed
    uint64_t* stat_empty = bars + 13;           // [2] phase B of the tile is over (256 arrivals)
    uint64_t* s_read = bars + 4;                // the softmax warps hold S^T (256 arrivals; head size 64)
    uint64_t* ds_empty = bars + 6;              // dK of the tile is complete: the dS^T tile may be overwritten (head size 64)
    uint64_t* do_empty = bars + 48;             // [Q_STAGES] the tile's dO is free: dP^T and dV complete, or (head size 128) dQ through it
    uint64_t* dp_read = bars + 15;              // ... and dP^T
    uint64_t* work_full = bars + 28;            // [kBwdAnswers] the answer to a request for work is there
    uint64_t* work_empty = bars + 32;           // [kBwdAnswers] producer, MMA issuer, softmax and dQ warps have read it
    uint8_t* answers = (uint8_t*)(bars + 36);   // [kBwdAnswers] 16 bytes
    uint32_t* tmem_slot = (uint32_t*)(bars + 44);
    // [2] dS^T in smem (256 arrivals).  Two in turn: with head size 64 dP^T of tile t+1 is issued before the wait for dS^T(t), so
    // dS^T(t+1) may be there by the time the MMA issuer gets to that wait.
    uint64_t* ds_full = bars + 46;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int n_tiles = (p.S + kTile - 1) / kTile;

    if (threadIdx.x == 0) {
        for (int b = 0; b < C::KV_BUFS; ++b) {
            mbar_init(&kv_full[b], 1);
            mbar_init(&kv_empty[b], 1);
        }
        for (int s = 0; s < C::Q_STAGES; ++s) {
            mbar_init(&q_full[s], 1);
            mbar_init(&do_full[s], 1);
            mbar_init(&q_empty[s], 1);
            mbar_init(&do_empty[s], C::DQ_BYTES ? 1 : 4);
        }
        mbar_init(s_full, 1);
        mbar_init(&ds_full[0], 256);
        mbar_init(&ds_full[1], 256);
        mbar_init(s_read, 256);
        mbar_init(dp_read, 256);
        mbar_init(p_full, 256);
        mbar_init(dp_full, 1);
        mbar_init(dq_full, 1);
        mbar_init(dq_empty, 4);
        mbar_init(ds_empty, 1);
        mbar_init(all_done, 1);
        mbar_init(acc_free, 256);
        for (int b = 0; b < kBwdAnswers; ++b) {
            mbar_init(&work_full[b], 1);
            mbar_init(&work_empty[b], 14);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&stat_full[b], 1);
            mbar_init(&stat_empty[b], 256);
        }
        fence_barrier_init();
        tma_prefetch_desc(&map_q);
        tma_prefetch_desc(&map_k);
        tma_prefetch_desc(&map_v);
        tma_prefetch_desc(&map_do);
        tma_prefetch_desc(&map_dq);
    }
    if (warp == 1) tmem_alloc(tmem_slot, C::TMEM_COLS);
    griddep_sync();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    // Walk r + 1 of this CTA: the answer to the request made during walk r (whole warps).
    auto next_walk = [&](int r, unsigned int code, bool& ok) -> BwdWalk {
        const int a = r % kBwdAnswers;
        if (!mbar_wait_warp(&work_full[a], (r / kBwdAnswers) & 1, p.status, code)) {
            ok = false;
            return bwd_walk(p, -1);
        }
        const int index = taken_cta(answers + a * 16);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&work_empty[a]);
        return bwd_walk(p, index);
    };

    if (warp == 0) {
        // ---------------- TMA producer, and the one who asks for work ----------------
        // the whole warp in step, one elected lane issues, here as for the MMAs: a lone lane, whose operands cannot live
        // in uniform registers, takes about 100 cycles per load
        const bool leader = elect_one();
        bool ok = true;
        uint32_t t = 0;                                      // tiles so far, of all walks
        BwdWalk w = bwd_walk(p, blockIdx.x);
        for (int r = 0; ok && w.n > 0; ++r) {
            const int a = r % kBwdAnswers;
            if (!mbar_wait_warp(&work_empty[a], ((r / kBwdAnswers) & 1) ^ 1, p.status, kTimeoutProducer)) break;
            if (leader) {
                mbar_arrive_expect_tx(&work_full[a], 16);
                request_next_cta(answers + a * 16, &work_full[a]);
            }
            const int kb = r % C::KV_BUFS;
            uint8_t* k_dst = kv_smem + kb * 2 * C::TILE_BYTES;
            if (!mbar_wait_warp(&kv_empty[kb], ((r / C::KV_BUFS) & 1) ^ 1, p.status, kTimeoutProducer)) break;
            if (leader) {
                mbar_arrive_expect_tx(&kv_full[kb], 2 * C::TILE_BYTES);
                tma_load_4d(k_dst, &map_k, &kv_full[kb], 0, w.jt * kTile, 0, w.unit);
                tma_load_4d(k_dst + C::TILE_BYTES, &map_v, &kv_full[kb], 0, w.jt * kTile, 0, w.unit);
            }
            const int64_t stat_base = (int64_t)w.unit * n_tiles * kTile;    // the statistics are padded to whole tiles
            for (int i = w.i0; i < w.i0 + w.n; ++i, ++t) {
                const int s = t % C::Q_STAGES;
                if (!mbar_wait_warp(&q_empty[s], ((t / C::Q_STAGES) & 1) ^ 1, p.status, kTimeoutProducer)) { ok = false; break; }
                if (leader) {
                    mbar_arrive_expect_tx(&q_full[s], C::TILE_BYTES);
                    tma_load_4d(q_smem + s * C::TILE_BYTES, &map_q, &q_full[s], 0, i * kTile, 0, w.unit);
                }
                // the tile's 128 exponent offsets and 128 deltas, into the buffer of its parity once
                // the tile before last has left it
                if (!mbar_wait_warp(&stat_empty[t & 1], ((t >> 1) & 1) ^ 1, p.status, kTimeoutProducer)) { ok = false; break; }
                if (leader) {
                    mbar_arrive_expect_tx(&stat_full[t & 1], 1024);
                    bulk_load_1d(stat_s + (t & 1) * 256, p.lse2 + stat_base + i * kTile, 512, &stat_full[t & 1]);
                    bulk_load_1d(stat_s + (t & 1) * 256 + 128, p.delta2 + stat_base + i * kTile, 512, &stat_full[t & 1]);
                }
                if (!mbar_wait_warp(&do_empty[s], ((t / C::Q_STAGES) & 1) ^ 1, p.status, kTimeoutProducer)) { ok = false; break; }
                if (leader) {
                    mbar_arrive_expect_tx(&do_full[s], C::TILE_BYTES);
                    tma_load_4d(do_smem + s * C::TILE_BYTES, &map_do, &do_full[s], 0, i * kTile, 0, w.unit);
                }
            }
            if (ok) w = next_walk(r, kTimeoutProducer, ok);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // The whole warp in step, one elected lane issues: operands stay in uniform registers (see the
        // forward kernel; a single lane's issue took about 100 cycles per MMA, 40 MMAs per tile pair).
        {
            constexpr uint32_t idesc_st = make_idesc(kBF16, false, false, kTile, kTile);   // K.Q^T, V.dO^T
            constexpr uint32_t idesc_acc = make_idesc(kBF16, false, true, kTile, HS);      // dV, dK
            constexpr uint32_t idesc_dq = make_idesc(kBF16, true, true, kTile, HS);        // dQ
            const bool leader = elect_one();
            const uint64_t k_desc = smem_desc_sw128(smem_u32(kv_smem), 16, 1024), v_desc = k_desc + (C::TILE_BYTES >> 4);
            const uint64_t q_desc = smem_desc_sw128(smem_u32(q_smem), 16, 1024), do_desc = smem_desc_sw128(smem_u32(do_smem), 16, 1024);
            const uint64_t ds_desc = smem_desc_sw128(smem_u32(ds_smem), 16, 1024);
            // the same tiles read along their rows
            const uint64_t k_mn = smem_desc_mn(smem_u32(kv_smem), kBoxBytes, false), q_mn = smem_desc_mn(smem_u32(q_smem), kBoxBytes, false);
            const uint64_t do_mn = smem_desc_mn(smem_u32(do_smem), kBoxBytes, false), ds_mn = smem_desc_mn(smem_u32(ds_smem), kBoxBytes, false);
            // Issue order on the (in-order) tensor pipe, per tile t:
            //   dV(t) S(t+1) | dQ(t) dK(t) | dP(t+1)          with head size 64: S(t+1) | dV(t) | dP(t+1) | dQ(t) dK(t)
            // dV follows phase A; S^T of the next tile overwrites R0 right behind it (dV, ahead on
            // the pipe, is the only reader of P^T).  dK and dQ need dS^T from phase B.  dP^T of the
            // next tile follows them: into its own columns (head size 64), or into the dQ columns
            // once the dQ warps have taken this tile's dQ out of them (head size 128) - in both
            // cases long before phase B of the next tile asks for it.
            // the last argument is the K/V buffer of the tile's walk
            auto issue_s = [&](uint32_t t, int kb) -> bool {
                const int s = t % C::Q_STAGES;
                if (!mbar_wait_warp(&q_full[s], (t / C::Q_STAGES) & 1, p.status, kTimeoutMma)) return false;
                tc_fence_after_sync();
                const uint64_t qd = q_desc + (s * C::TILE_BYTES >> 4), kd = k_desc + (kb * 2 * C::TILE_BYTES >> 4);
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < C::ROWB / 32; ++kk) {
                        const uint32_t off = ((kk / 4) * kBoxBytes + (kk % 4) * 32) >> 4;
                        mma_ss<false>(tmem_base + C::COL_S, kd + off, qd + off, idesc_st, kk > 0);
                    }
                    mma_commit(s_full);
                }
                return true;
            };
            auto issue_dp = [&](uint32_t t, int kb) -> bool {        // dP^T = V . dO^T
                const int s = t % C::Q_STAGES;
                if (!mbar_wait_warp(&do_full[s], (t / C::Q_STAGES) & 1, p.status, kTimeoutMma)) return false;
                tc_fence_after_sync();
                const uint64_t dod = do_desc + (s * C::TILE_BYTES >> 4), vd = v_desc + (kb * 2 * C::TILE_BYTES >> 4);
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < C::ROWB / 32; ++kk) {
                        const uint32_t off = ((kk / 4) * kBoxBytes + (kk % 4) * 32) >> 4;
                        mma_ss<false>(tmem_base + C::COL_DP, vd + off, dod + off, idesc_st, kk > 0);
                    }
                    mma_commit(dp_full);
                }
                return true;
            };
            bool ok = true;
            uint32_t t = 0;                                  // tiles so far, of all walks
            BwdWalk w = bwd_walk(p, blockIdx.x);
            if (w.n > 0) {
                ok = mbar_wait_warp(&kv_full[0], 0, p.status, kTimeoutMma);
                ok = ok && issue_s(0, 0);
                ok = ok && issue_dp(0, 0);
            }
            for (int r = 0; ok && w.n > 0; ++r) {
                const int kb = r % C::KV_BUFS;
                const BwdWalk next = next_walk(r, kTimeoutMma, ok);
                const uint64_t k_d = k_mn + (kb * 2 * C::TILE_BYTES >> 4);
                for (int i = 0; i < w.n && ok; ++i, ++t) {
                    const int s = t % C::Q_STAGES;
                    const bool first = i == 0;                       // first tile of a walk: dK, dV start over
                    const bool last = i == w.n - 1;
                    const bool more = !last || next.n > 0;           // there is a tile t+1
                    // ... whose scores may be issued now: it uses the same K and V, or K and V have a second buffer
                    const bool early = more && (!last || C::KV_BUFS == 2);
                    const int kb_next = last ? (r + 1) % C::KV_BUFS : kb;
                    const uint64_t q_d = q_mn + (s * C::TILE_BYTES >> 4), do_d = do_mn + (s * C::TILE_BYTES >> 4);
                    auto next_s = [&]() -> bool {                    // S of tile t+1, the K and V of its walk first
                        if (last && !mbar_wait_warp(&kv_full[kb_next], ((r + 1) / C::KV_BUFS) & 1, p.status, kTimeoutMma)) return false;
                        return issue_s(t + 1, kb_next);
                    };
                    if (C::DP_OWN && more) {
                        if (!mbar_wait_warp(s_read, t & 1, p.status, kTimeoutMma)) { ok = false; break; }
                        if (!next_s()) { ok = false; break; }
                    }
                    if (!mbar_wait_warp(p_full, t & 1, p.status, kTimeoutMma)) { ok = false; break; }
                    if (!mbar_wait_warp(&do_full[s], (t / C::Q_STAGES) & 1, p.status, kTimeoutMma)) { ok = false; break; }
                    // the previous walk's dK, dV must have left tensor memory
                    if (first && r > 0 && !mbar_wait_warp(acc_free, (r - 1) & 1, p.status, kTimeoutMma)) { ok = false; break; }
                    tc_fence_after_sync();
                    if (leader) {
#pragma unroll
                        for (int kk = 0; kk < kTile / 16; ++kk)      // dV += P^T . dO      (K = 128 query rows)
                            mma_ts<false>(tmem_base + C::COL_DV, tmem_base + C::COL_P + (kk / 4) * C::P_HALF + (kk % 4) * 8,
                                          do_d + (kk * 2048 >> 4), idesc_acc, !first || kk > 0);
                        if (C::DQ_BYTES) mma_commit(&do_empty[s]);
                    }
                    if (C::DP_OWN && more) {
                        if (!mbar_wait_warp(dp_read, t & 1, p.status, kTimeoutMma)) { ok = false; break; }
                        if (!issue_dp(t + 1, kb_next)) { ok = false; break; }
                    }
                    // R0 is free as soon as dV, ahead on the pipe, has read P^T
                    if (!C::DP_OWN && early && !next_s()) { ok = false; break; }
                    if (!mbar_wait_warp(&ds_full[t & 1], (t >> 1) & 1, p.status, kTimeoutMma)) { ok = false; break; }
                    if (t > 0) {
                        // the previous dQ must have left its TMEM columns
                        if (!mbar_wait_warp(dq_empty, (t - 1) & 1, p.status, kTimeoutMma)) { ok = false; break; }
                    }
                    tc_fence_after_sync();
                    // dQ first: its completion starts the read-out, whose first step (tensor memory ->
                    // registers) gates the next tile's dP^T when that borrows the dQ columns; dK runs
                    // on the pipe meanwhile.  This tile's dO stage was last read by dV and dP^T, which
                    // are ahead of dQ on the pipe, so it is free for the read-out's staging at dq_full.
                    if (leader) {
#pragma unroll
                        for (int kk = 0; kk < kTile / 16; ++kk)      // dQ_i = dS . K        (K = 128 key rows)
                            mma_ss<false>(tmem_base + C::COL_DQ, ds_mn + (kk * 2048 >> 4), k_d + (kk * 2048 >> 4), idesc_dq, kk > 0);
                        mma_commit(dq_full);
#pragma unroll
                        for (int kk = 0; kk < kTile / 16; ++kk) {    // dK += dS^T . Q
                            const uint32_t off = ((kk / 4) * kBoxBytes + (kk % 4) * 32) >> 4;
                            mma_ss<false>(tmem_base + C::COL_DK, ds_desc + off, q_d + (kk * 2048 >> 4), idesc_acc, !first || kk > 0);
                        }
                        if (C::DQ_BYTES) mma_commit(ds_empty);
                        mma_commit(&q_empty[s]);  // also: the dS^T tile is no longer read
                        if (last) {
                            mma_commit(&kv_empty[kb]);              // K and V of the walk are no longer read
                            mma_commit(all_done);                   // and its dK, dV are complete
                        }
                    }
                    if (!C::DP_OWN && more && !early && !next_s()) { ok = false; break; }
                    // dS^T of tile t is in shared memory, so the softmax warps are done with dP^T(t)
                    if (!C::DP_OWN && more) {
                        // borrowed columns: this tile's dQ, just issued, has to complete and leave them first
                        if (!mbar_wait_warp(dq_empty, t & 1, p.status, kTimeoutMma)) { ok = false; break; }
                        if (!issue_dp(t + 1, kb_next)) { ok = false; break; }
                    }
                }
                w = next;
            }
        }
    } else if (warp < 10) {
        // ---------------- softmax / dS: warps 2..9 ----------------
        // thread = (key row r, half h of the 128 query columns); the two warps that share a
        // TMEM lane group each own 64 columns.
        const int lane_group = warp & 3;
        const int half = (warp - 2) >> 2;
        const int r = lane_group * 32 + lane;                       // key row inside the tile
        const uint32_t lane_addr = (uint32_t)(lane_group * 32) << 16;
        const uint32_t col0 = 64u * half;                           // first query column of this thread
        const float sl2 = p.scale * 1.4426950408889634f;
        const uint64_t sl2_2 = pack_f32x2(sl2, sl2), scale_2 = pack_f32x2(p.scale, p.scale);
        uint8_t* ds_row = ds_smem + half * kBoxBytes + r * 128;     // box `half` holds query columns 64h..64h+63
        const int swz = r & 7;
        bool ok = true;
        // Every thread does its own (bounded) waits; there is no barrier among the softmax warps
        // inside the walk, so a thread that is done with a tile moves on at once.  When a wait
        // gives up, the thread leaves the loop; the others see the status word at their next wait
        // and follow.
        // dK, dV of a finished walk: the first four warps store dV, the other four dK.
        auto store_dkdv = [&](int unit, int jt, uint32_t phase) -> bool {
            if (!mbar_wait_warp(all_done, phase, p.status, kTimeoutEpilogue)) return false;
            tc_fence_after_sync();
            const int64_t grow = (int64_t)unit * p.S + (int64_t)jt * kTile + r;
            const bool live = jt * kTile + r < p.S;
            __nv_bfloat16* out = (__nv_bfloat16*)(half ? p.dK : p.dV) + grow * HS;
            const uint32_t col = half ? C::COL_DK : C::COL_DV;
#pragma unroll 1
            for (int c = 0; c < HS / 32; ++c) {
                uint32_t v[32];
                tmem_ld32(tmem_base + col + lane_addr + c * 32, v);
                tmem_wait_ld();
                if (!live) continue;
#pragma unroll
                for (int x = 0; x < 32; x += 8) {
                    uint4 o;
                    o.x = pack_bf16(__uint_as_float(v[x]), __uint_as_float(v[x + 1]));
                    o.y = pack_bf16(__uint_as_float(v[x + 2]), __uint_as_float(v[x + 3]));
                    o.z = pack_bf16(__uint_as_float(v[x + 4]), __uint_as_float(v[x + 5]));
                    o.w = pack_bf16(__uint_as_float(v[x + 6]), __uint_as_float(v[x + 7]));
                    *reinterpret_cast<uint4*>(out + c * 32 + x) = o;
                }
            }
            return true;
        };
        uint32_t t = 0;                                             // tiles so far, of all walks
        int jt_before = -1, unit_before = 0;                        // walk whose dK, dV are still to be stored
        BwdWalk w = bwd_walk(p, blockIdx.x);
        for (int r_walk = 0; ok && w.n > 0; ++r_walk) {
        const bool key_live = w.jt * kTile + r < p.S;
        for (int i = w.i0; i < w.i0 + w.n; ++i, ++t) {
            // -lse*log2e and -delta/sqrt(hs) of this query tile, put into the buffer of this tile's
            // parity by the producer
            const float* lse_s = stat_s + (t & 1) * 256;
            const float* delta_s = lse_s + 128;
            if (!mbar_wait_warp(&stat_full[t & 1], (t >> 1) & 1, p.status, kTimeoutSoftmax)) { ok = false; break; }
            if (!mbar_wait_warp(s_full, t & 1, p.status, kTimeoutSoftmax)) { ok = false; break; }
            tc_fence_after_sync();
            const bool diag = p.causal && i == w.jt;
            // ---- phase A: P^T = exp2(S^T*c - lse) for this thread's 64 columns ----
            uint32_t ph[32];                                        // 64 probabilities as BF16 pairs
            {
                uint32_t s0[32], s1[32];
                tmem_ld32(tmem_base + C::COL_S + lane_addr + col0, s0);
                tmem_ld32(tmem_base + C::COL_S + lane_addr + col0 + 32, s1);
                tmem_wait_ld();
                if (C::DP_OWN) {
                    tc_fence_before_sync();
                    mbar_arrive(s_read);
                }
                // The mask test is a compile-time flag of the loop body: a branch per group of
                // columns would end the compiler's scheduling region there and leave the warp
                // running each group's FMA -> exp2 -> convert chain at its latency.
                auto phase_a = [&](auto diag_c) {
                constexpr bool kDiag = decltype(diag_c)::value;
#pragma unroll
                for (int x = 0; x < 32; x += 4) {
                    // four consecutive query columns from each 32-column chunk; their -lse come
                    // as one 16-byte shared-memory load (a broadcast: all threads ask for the same)
                    const int q0 = col0 + x, q1 = col0 + 32 + x;
                    const float4 la = *reinterpret_cast<const float4*>(lse_s + q0);
                    const float4 lb = *reinterpret_cast<const float4*>(lse_s + q1);
                    float a[4], b[4];
                    // s*c - lse for two columns per FMA-pipe instruction
                    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(s0[x]), __uint_as_float(s0[x + 1])), sl2_2, pack_f32x2(la.x, la.y)), a[0], a[1]);
                    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(s0[x + 2]), __uint_as_float(s0[x + 3])), sl2_2, pack_f32x2(la.z, la.w)), a[2], a[3]);
                    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(s1[x]), __uint_as_float(s1[x + 1])), sl2_2, pack_f32x2(lb.x, lb.y)), b[0], b[1]);
                    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(s1[x + 2]), __uint_as_float(s1[x + 3])), sl2_2, pack_f32x2(lb.z, lb.w)), b[2], b[3]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        a[e] = fast_exp2(a[e]);
                        b[e] = fast_exp2(b[e]);
                    }
                    if (kDiag) {                     // query q sees key r only when q >= r
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            a[e] = q0 + e < r ? 0.f : a[e];
                            b[e] = q1 + e < r ? 0.f : b[e];
                        }
                    }
                    ph[x >> 1] = pack_bf16(a[0], a[1]);
                    ph[(x >> 1) + 1] = pack_bf16(a[2], a[3]);
                    ph[16 + (x >> 1)] = pack_bf16(b[0], b[1]);
                    ph[16 + (x >> 1) + 1] = pack_bf16(b[2], b[3]);
                }
                };
                if (diag) phase_a(std::true_type{});
                else      phase_a(std::false_type{});
                // A key row beyond the end of the sequence has zero scores, whose exp2(-lse) may overflow;
                // its dS^T meets a zero row of K, so it has to be a number.
                if (!key_live) {
#pragma unroll
                    for (int x = 0; x < 32; ++x) ph[x] = 0u;
                }
                // P^T(t-1) has been read: dP^T(t) was issued behind the dV that read it.  (Phase B wants dP^T(t) anyway.)
                if (C::DP_OWN) {
                    if (!mbar_wait_warp(dp_full, t & 1, p.status, kTimeoutSoftmax)) { ok = false; break; }
                    tc_fence_after_sync();
                }
                // 64 BF16 = 32 columns; with head size 128 the first of this thread's own S^T columns
                tmem_st32(tmem_base + C::COL_P + lane_addr + half * C::P_HALF, ph);
            }
            tmem_wait_st();
            tc_fence_before_sync();
            mbar_arrive(p_full);
            if (i == w.i0 && jt_before >= 0) {
                // dK, dV of the previous walk leave tensor memory before this one's first dV and dK start
                // them over; behind its phase A they have been complete for a while
                if (!store_dkdv(unit_before, jt_before, (r_walk - 1) & 1)) { ok = false; break; }
                tc_fence_before_sync();
                mbar_arrive(acc_free);
            }
            // ---- phase B: dS^T = P^T * (dP^T - delta) / sqrt(hs) ----
            if (!C::DP_OWN) {
                if (!mbar_wait_warp(dp_full, t & 1, p.status, kTimeoutSoftmax)) { ok = false; break; }
                tc_fence_after_sync();
            }
            {
                uint32_t d0[32], d1[32];
                tmem_ld32(tmem_base + C::COL_DP + lane_addr + col0, d0);
                tmem_ld32(tmem_base + C::COL_DP + lane_addr + col0 + 32, d1);
                tmem_wait_ld();
                if (C::DP_OWN) {
                    tc_fence_before_sync();
                    mbar_arrive(dp_read);
                    if (t > 0 && !mbar_wait_warp(ds_empty, (t - 1) & 1, p.status, kTimeoutSoftmax)) { ok = false; break; }
                }
#pragma unroll
                for (int half32 = 0; half32 < 2; ++half32) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {            // one 16-byte unit = 8 query columns
                        const int x = u * 8;                                  // index inside the 32-column chunk
                        const int q = col0 + half32 * 32 + x;
                        const float4 da = *reinterpret_cast<const float4*>(delta_s + q);
                        const float4 db = *reinterpret_cast<const float4*>(delta_s + q + 4);
                        const float nd[8] = {da.x, da.y, da.z, da.w, db.x, db.y, db.z, db.w};
                        uint32_t o[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const uint32_t pk = ph[half32 * 16 + (x >> 1) + e];        // two probabilities, BF16
                            const float dp0 = __uint_as_float(half32 ? d1[x + 2 * e] : d0[x + 2 * e]);
                            const float dp1 = __uint_as_float(half32 ? d1[x + 2 * e + 1] : d0[x + 2 * e + 1]);
                            // (dP - delta) / sqrt(hs) for both columns in one FP32 FMA, rounded to BF16 and
                            // multiplied with the BF16 probabilities in one packed BF16 multiply
                            float t0, t1;
                            unpack_f32x2(fma_f32x2(pack_f32x2(dp0, dp1), scale_2, pack_f32x2(nd[2 * e], nd[2 * e + 1])), t0, t1);
                            o[e] = mul_bf16x2(pk, pack_bf16(t0, t1));
                        }
                        const int unit16 = half32 * 4 + u;
                        *reinterpret_cast<uint4*>(ds_row + ((unit16 ^ swz) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
                    }
                }
            }
            fence_proxy_async_smem();
            mbar_arrive(&ds_full[t & 1]);
            mbar_arrive(&stat_empty[t & 1]);                 // this tile's statistics are no longer read
        }
        jt_before = w.jt;
        unit_before = w.unit;
        if (!ok) break;
        w = next_walk(r_walk, kTimeoutSoftmax, ok);
        if (ok && w.n == 0) store_dkdv(unit_before, jt_before, r_walk & 1);
        }
    } else {
        // ---------------- dQ reduction: warps 10..13, thread = query row ----------------
        // Each warp by itself: its 32 rows of the tile, 64 columns at a time, from tensor memory to two boxes of its own (32
        // rows x 128 bytes) and from there, by TMA reduce-add, into the sum.  With head size 64 the boxes are an area of their
        // own; with 128 they are a quarter of the tile's dO stage, which is idle once the tile's MMAs are complete, and the
        // stage is handed back to the producer when the four warps' reductions have read it.  The second 64 columns are
        // taken into registers before anything else, since the next dP^T waits for the dQ columns.
        // (All four warps in step, through 128-row boxes, with a barrier for each move and the dO tiles loaded behind it, took
        // 3300 cycles a tile at head size 64, all of the tile's period: with scores and dP^T ahead 256 units of 2048 rows,
        // causal, with preparation and cast took 541 us before and 519 now, 512 of 1024 518 and 503.  What bounds a tile
        // there now is shared memory (304 KB, 2375 cycles): without exponentials, statistics and reductions it still takes
        // 460.  Tried on this: one half of the softmax warps half a tile behind the other 528; dS^T in tensor memory as dK's
        // operand, in P^T's columns, 608.  Head size 128, 64 units of 4096 rows: 783 and 765.)
        const int lane_group = warp & 3;
        const uint32_t t_dq = tmem_base + C::COL_DQ + ((uint32_t)(lane_group * 32) << 16);
        const int swz = lane & 7;
        const bool leader = elect_one();
        bool ok = true;
        uint32_t t = 0;                                      // tiles so far, of all walks
        BwdWalk w = bwd_walk(p, blockIdx.x);
        for (int r_walk = 0; ok && w.n > 0; ++r_walk) {
            for (int i = w.i0; i < w.i0 + w.n; ++i, ++t) {
                const int s = t % C::Q_STAGES, y = i * kTile + lane_group * 32;
                uint8_t* const boxes = (C::DQ_BYTES ? dq_smem : do_smem + s * C::TILE_BYTES) + lane_group * 8192;
                uint32_t v[2][32];
                auto take = [&](int col) {
#pragma unroll
                    for (int b = 0; b < 2; ++b) tmem_ld32(t_dq + col + b * 32, v[b]);
                    tmem_wait_ld();
                };
                auto stage = [&] {
#pragma unroll
                    for (int b = 0; b < 2; ++b)
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            *reinterpret_cast<uint4*>(boxes + b * 4096 + lane * 128 + ((u ^ swz) << 4)) = make_uint4(v[b][4 * u], v[b][4 * u + 1], v[b][4 * u + 2], v[b][4 * u + 3]);
                };
                auto send = [&](int col) {                   // by the leader
                    if (y < p.S) {
#pragma unroll
                        for (int b = 0; b < 2; ++b) tma_reduce_add_3d(&map_dq, boxes + b * 4096, col + b * 32, y, w.unit);
                    }
                    tma_commit_group();
                };
                if (!mbar_wait_warp(dq_full, t & 1, p.status, kTimeoutOther)) { ok = false; break; }
                tc_fence_after_sync();
                take(0);
                if (C::DQ_BYTES) {
                    tc_fence_before_sync();
                    __syncwarp();
                    if (leader) {
                        mbar_arrive(dq_empty);               // this warp's part of the dQ columns is free
                        tma_wait_group_read0();
                    }
                    __syncwarp();
                    stage();
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (leader) send(0);
                } else {
                    stage();
                    take(64);
                    tc_fence_before_sync();
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (leader) {
                        mbar_arrive(dq_empty);
                        send(0);
                        tma_wait_group_read0();
                    }
                    __syncwarp();
                    stage();
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (leader) {
                        send(64);
                        tma_wait_group_read0();
                        mbar_arrive(&do_empty[s]);
                    }
                }
            }
            if (!ok) break;
            w = next_walk(r_walk, kTimeoutOther, ok);
        }
        // The CTA may end once the reductions have read their shared-memory source; that they have
        // landed in global memory by the time the next kernel runs is the grid's completion.
        if (leader) tma_wait_group_read0();
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
}

}  // namespace attn_tc
}  // namespace boatcu
