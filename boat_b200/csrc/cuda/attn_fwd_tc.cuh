// attn_fwd_tc.cuh - fused attention forward on tcgen05: scaled QK^T, causal mask, online
// softmax and PV in one kernel; the S x S matrix lives only in tensor memory, only the
// log-sum-exp per row is saved for the backward.
//
// Replaces scaled_dot_product_attention_impl (reference src/layers/attention.c:997-1073),
// which materialises scores and probabilities as [B,nh,S,S] FP32 tensors.
//
// One CTA per SM works off (unit, pair of adjacent 128-row query tiles A and B) items and walks the
// key/value tiles of 128 rows.  Per key tile and query tile ("step"):
//     S  = Q . K^T            tcgen05.mma, both operands from shared memory, S in tensor memory
//     P  = exp2(S*c - m*c)    4 softmax warps per query tile, one thread per query row (TMEM lane =
//                             row): the row of 128 scores comes into registers with one
//                             tcgen05.ld wait, running max m and sum l stay in registers, P is
//                             written back over S (BF16 pairs, or TF32-valued FP32)
//     O += P . V              tcgen05.mma, A = P from tensor memory, B = V from shared memory
//                             read along its contiguous head dimension (no transpose)
// The accumulator O is rescaled in tensor memory only when the running max has grown by more
// than 2^8 (the warp votes), the exact correction is folded into the final 1/l.
//
// One lane, elected by a warp that stays in step, issues the MMAs of all steps of all items in one order, steps of A and
// B alternating:
//     S(0) .. S(NB-1) | P.V(0) S(NB) | P.V(1) S(NB+1) | ...
// so that the exponentials of one tile run under the MMAs of the other.  S(i) takes the buffer of
// step i-NB, whose P.V is ahead of it on the in-order tensor pipe.  With head size 64 there is room for
// NB = 3 score buffers: a tile's next scores are complete before its softmax warps come back for them,
// which leaves the special-function unit as the limit.  With head size 128 tensor memory holds two; the
// P.V of a step then starts on the first half of P while the second is being computed.
//
// The items of a launch run through the same pipeline without a break: loads and scores of the next
// item are under way while the last steps and the output of the previous one finish (a CTA per item
// paid about 9000 cycles for start and end, as much as two to three steps).  Measured with ten launches back to back:
// 256 units of 2048 x 64 causal 305 -> 210 us, 64 units of 8192 x 128 causal 1047 -> 961 us = 1144 TFLOP/s.  Items are handed out by
// the hardware in index order (cluster launch control), long rows first.  K and V tiles are loaded
// once for both query tiles; the CTAs at work belong to a few units at a time, whose K and V stay in L2.
//
// Warp 0: TMA producer; warp 1: MMA issuer; warps 4-7: softmax and output of tile A;
// warps 8-11: of tile B.  Registers are shared out by warpgroup: a softmax thread holds a row of 128
// scores and would spill with its even share of 168.
#pragma once
#include "tc_common.cuh"
#include <float.h>

namespace boatcu {
namespace attn_tc {

using namespace tc;

constexpr int kTile = 128;            // query rows per CTA and key rows per step
constexpr int kBoxBytes = kTile * 128;   // one TMA box: 128 rows x 128 bytes
constexpr int kFwdThreads = 384;     // producer, MMA issuer, two idle warps, 2 x 4 softmax warps

template <typename T, int HS>
struct FwdCfg {
    static constexpr int ES = sizeof(T);
    static constexpr bool TF32 = ES == 4;
    static constexpr int ROWB = HS * ES;                 // bytes per row of Q/K/V
    static constexpr int NBOX = ROWB / 128;              // boxes per 128-row tile
    static constexpr int BOXC = 128 / ES;                // elements per box row
    static constexpr int UK = 32 / ES;                   // K extent of one MMA
    static constexpr int TILE_BYTES = NBOX * kBoxBytes;
    static constexpr int KV_STAGES = TILE_BYTES <= 16384 ? 4 : 2;
    static constexpr int Q_BUFS = TILE_BYTES <= 16384 ? 2 : 1;       // query tile pairs in shared memory
    static constexpr int SMEM = TILE_BYTES * (2 * Q_BUFS + 2 * KV_STAGES) + 1024 + 512;
    static constexpr int NB = 2 * HS + 3 * kTile <= 512 ? 3 : 2;     // score buffers
    static constexpr bool HALVES = NB == 2;              // P.V in two halves
    static constexpr uint32_t COL_O = NB * kTile;        // S/P buffers, then O of A, then O of B
    static constexpr uint32_t TMEM_COLS = 512;
    static_assert(NB * kTile + 2 * HS <= 512, "tensor memory budget");
    static_assert(SMEM <= 227 * 1024, "shared memory budget");
    static_assert(ROWB % 128 == 0, "row must be whole 128-byte boxes");
};

struct FwdParams {
    void* O;
    float* lse;
    int S;             // sequence length
    int units;
    int causal;
    float scale;       // 1/sqrt(hs)
    int wide;          // O is 32-byte aligned: a whole sector per store
    int group;         // units whose CTAs are scheduled together (their K and V share L2)
    unsigned int* status;
};

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// COLS scores of a row in registers, columns from `first` on -> probabilities exp2(s*sl2 + neg_m) in
// place (BF16: packed pairs in the first half; TF32: TF32-valued floats); returns their sum.  Columns
// beyond `last` are masked (MASK only).
//
// Written as a software pipeline over column pairs: the multiply-add of pair t+2D, the exponentials of
// pair t+D and the conversion and sum of pair t stand next to each other and depend on nothing close
// by, in an order fixed by volatile asm.  (Left to the compiler each pair's FMA -> exp2 -> convert chain
// ran with little overlap: the special-function unit was busy 50 % of the time, and two warps per
// scheduler do not cover for it.)
template <bool TF32, bool MASK, int COLS>
__device__ __forceinline__ float exp_row(uint32_t* sc, float sl2, float neg_m, int first, int last) {
    constexpr int PAIRS = COLS / 2, D = 4;
    const uint64_t sl2_2 = pack_f32x2(sl2, sl2), neg_m2 = pack_f32x2(neg_m, neg_m);
    uint64_t l2[2] = {0ull, 0ull};                       // chains of (even, odd) partial sums
#pragma unroll
    for (int t = -2 * D; t < PAIRS; ++t) {
        const int f = t + 2 * D, e = t + D, c = t;       // pairs in the three stages
        if (e >= 0 && e < PAIRS) asm volatile("ex2.approx.ftz.f32 %0, %0;" : "+r"(sc[2 * e]));
        if (f < PAIRS) {
            uint64_t v;
            asm volatile("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(sc[2 * f]), "r"(sc[2 * f + 1]));
            asm volatile("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(v) : "l"(sl2_2), "l"(neg_m2));
            asm volatile("mov.b64 {%0, %1}, %2;" : "=r"(sc[2 * f]), "=r"(sc[2 * f + 1]) : "l"(v));
        }
        if (e >= 0 && e < PAIRS) asm volatile("ex2.approx.ftz.f32 %0, %0;" : "+r"(sc[2 * e + 1]));
        if (c >= 0) {
            uint32_t e0 = sc[2 * c], e1 = sc[2 * c + 1];
            if (MASK) {
                e0 = first + 2 * c > last ? 0u : e0;
                e1 = first + 2 * c + 1 > last ? 0u : e1;
            }
            if (TF32) {
                // round to the nearest TF32 value: the MMA would otherwise truncate
                asm volatile("cvt.rna.tf32.f32 %0, %0;" : "+r"(e0));
                asm volatile("cvt.rna.tf32.f32 %0, %0;" : "+r"(e1));
            }
            uint64_t v;
            asm volatile("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(e0), "r"(e1));
            asm volatile("add.rn.f32x2 %0, %0, %1;" : "+l"(l2[c & 1]) : "l"(v));
            if (TF32) {
                sc[2 * c] = e0;
                sc[2 * c + 1] = e1;
            } else {
                asm volatile("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(sc[c]) : "r"(e1), "r"(e0));
            }
        }
    }
    float a0, a1;
    unpack_f32x2(add_f32x2(l2[0], l2[1]), a0, a1);
    return a0 + a1;
}

// A work item: two adjacent query tiles of a unit.
struct FwdItem {
    int unit, qt;          // first query tile; the second is qt + 1
    int n_a, n_b;          // key tiles of each (n_b 0: an odd tile count leaves the last item one tile)
};

// Item order: units in groups of p.group, so that the K and V tiles which the CTAs running at one
// time stream through shared memory (every item of a unit reads all of the unit's K and V) stay
// in L2; inside a group the tile pair is the slow index, long (late) rows first when causal.
// When the units do not divide into whole groups the short group goes first: the launch then ends
// with the short items of a full group, which fill the SMs evenly.
__device__ __forceinline__ FwdItem fwd_item(const FwdParams& p, int index) {
    const int q_tiles = (p.S + kTile - 1) / kTile, n_pairs = (q_tiles + 1) / 2;
    const int short_group = p.units % p.group;             // 0: all groups are whole
    const int short_items = short_group * n_pairs;
    int unit0 = 0, in_group = short_group, rem = index;
    if (index >= short_items) {
        const int per_group = p.group * n_pairs, grp = (index - short_items) / per_group;
        unit0 = short_group + grp * p.group;
        in_group = p.group;
        rem = index - short_items - grp * per_group;
    }
    FwdItem it;
    it.unit = unit0 + rem % in_group;
    it.qt = 2 * (n_pairs - 1 - rem / in_group);
    const bool has_b = it.qt + 1 < q_tiles;
    it.n_a = p.causal ? it.qt + 1 : q_tiles;
    it.n_b = has_b ? (p.causal ? it.qt + 2 : q_tiles) : 0;
    return it;
}

template <typename T, int HS>
__global__ void __launch_bounds__(kFwdThreads, 1)
attn_fwd_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v, const __grid_constant__ FwdParams p) {
    using C = FwdCfg<T, HS>;
    constexpr bool TF32 = C::TF32;
    constexpr int ST = C::KV_STAGES, NB = C::NB, QB = C::Q_BUFS;
    constexpr int WS = 4;                                  // work answers in flight
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* q_smem = smem;                               // [QB] tile A, then tile B
    uint8_t* k_smem = q_smem + QB * 2 * C::TILE_BYTES;
    uint8_t* v_smem = k_smem + ST * C::TILE_BYTES;
    uint8_t* answers = v_smem + ST * C::TILE_BYTES;       // [WS] 16 bytes
    uint64_t* bars = (uint64_t*)(answers + WS * 16);
    uint64_t* q_full = bars;              // [QB]
    uint64_t* q_empty = q_full + QB;      // [QB]: the item's last S is complete
    uint64_t* k_full = q_empty + QB;      // [ST]
    uint64_t* k_empty = k_full + ST;      // [ST]
    uint64_t* v_full = k_empty + ST;      // [ST]
    uint64_t* v_empty = v_full + ST;      // [ST]
    uint64_t* s_full = v_empty + ST;      // [2][NB]: scores of tile A / B complete in tensor memory
    uint64_t* p_half = s_full + 2 * NB;   // [NB]: first half of P written (128 arrivals; HALVES only)
    uint64_t* p_full = p_half + NB;       // [NB]: P written (128 arrivals)
    uint64_t* pv_done = p_full + NB;      // [2][4]: P.V number 4x+r of tile A / B is complete
    uint64_t* work_full = pv_done + 8;    // [WS]: the answer to a request for work is there
    uint64_t* work_empty = work_full + WS;   // [WS]: everybody has read it (producer, MMA issuer, 8 softmax warps)
    uint32_t* tmem_slot = (uint32_t*)(work_empty + WS);

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int q_tiles = (p.S + kTile - 1) / kTile;
    // A last tile that is only partly filled: its missing rows read as zeros (the tensor maps end with
    // the unit), missing query rows are not stored, missing keys are masked.
    const int tail = p.S - (q_tiles - 1) * kTile;          // rows of the last tile

    if (threadIdx.x == 0) {
        for (int b = 0; b < QB; ++b) {
            mbar_init(&q_full[b], 1);
            mbar_init(&q_empty[b], 1);
        }
        for (int s = 0; s < ST; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
        }
        for (int b = 0; b < NB; ++b) {
            mbar_init(&s_full[b], 1);
            mbar_init(&s_full[NB + b], 1);
            mbar_init(&p_half[b], 128);
            mbar_init(&p_full[b], 128);
        }
        for (int b = 0; b < 8; ++b) mbar_init(&pv_done[b], 1);
        for (int w = 0; w < WS; ++w) {
            mbar_init(&work_full[w], 1);
            mbar_init(&work_empty[w], 10);
        }
        fence_barrier_init();
        tma_prefetch_desc(&map_q);
        tma_prefetch_desc(&map_k);
        tma_prefetch_desc(&map_v);
    }
    if (warp == 1) tmem_alloc(tmem_slot, C::TMEM_COLS);
    griddep_sync();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if (warp < 4) {
    regs_release<80>();          // registers per thread from here: 80 + 208 + 208 <= 3 * 168 of the launch
    if (warp == 0) {
        // ---------------- TMA producer, and the one who asks for work ----------------
        // the whole warp in step, one elected lane issues (see the MMA issuer: the same holds for TMA)
        const bool leader = elect_one();
        bool ok = true;
        uint32_t s = 0, par = 1;                          // key/value stage, parity of its next wait
        int index = blockIdx.x;
        for (uint32_t n = 0; index >= 0 && ok; ++n) {
            const FwdItem it = fwd_item(p, index);
            // the next item, long before anybody needs it
            const uint32_t w = n % WS;
            if (!mbar_wait_warp(&work_empty[w], ((n / WS) & 1) ^ 1, p.status, kTimeoutProducer)) { ok = false; break; }
            if (leader) {
                mbar_arrive_expect_tx(&work_full[w], 16);
                request_next_cta(answers + w * 16, &work_full[w]);
            }
            const uint32_t qb = n % QB;
            if (!mbar_wait_warp(&q_empty[qb], ((n / QB) & 1) ^ 1, p.status, kTimeoutProducer)) { ok = false; break; }
            const int tiles = it.n_b > 0 ? 2 : 1, n_kv = it.n_a > it.n_b ? it.n_a : it.n_b;
            if (leader) {
                mbar_arrive_expect_tx(&q_full[qb], tiles * C::TILE_BYTES);
                for (int g = 0; g < tiles; ++g)
                    tma_load_4d(q_smem + (qb * 2 + g) * C::TILE_BYTES, &map_q, &q_full[qb], 0, (it.qt + g) * kTile, 0, it.unit);
            }
            for (int j = 0; j < n_kv; ++j) {
                if (!mbar_wait_warp(&k_empty[s], par, p.status, kTimeoutProducer)) { ok = false; break; }
                if (leader) {
                    mbar_arrive_expect_tx(&k_full[s], C::TILE_BYTES);
                    tma_load_4d(k_smem + s * C::TILE_BYTES, &map_k, &k_full[s], 0, j * kTile, 0, it.unit);
                }
                if (!mbar_wait_warp(&v_empty[s], par, p.status, kTimeoutProducer)) { ok = false; break; }
                if (leader) {
                    mbar_arrive_expect_tx(&v_full[s], C::TILE_BYTES);
                    tma_load_4d(v_smem + s * C::TILE_BYTES, &map_v, &v_full[s], 0, j * kTile, 0, it.unit);
                }
                if (++s == ST) {
                    s = 0;
                    par ^= 1;
                }
            }
            if (!ok || !mbar_wait_warp(&work_full[w], (n / WS) & 1, p.status, kTimeoutProducer)) { ok = false; break; }
            index = taken_cta(answers + w * 16);
            fence_proxy_async_smem();
            __syncwarp();
            if (leader) mbar_arrive(&work_empty[w]);
        }
        if (!ok)
            for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // The whole warp runs this, in step, and one elected lane issues: everything but the instructions
        // themselves is then uniform and lives in uniform registers, where tcgen05.mma wants its
        // operands.  (Run by a single lane, moving four operands per MMA over took about 100 cycles of
        // issue per MMA - more than the tensor core needs for it.)
        {
            constexpr uint32_t fmt = TF32 ? kTF32 : kBF16;
            constexpr uint32_t idesc_s = make_idesc(fmt, false, false, kTile, kTile);   // S = Q K^T
            constexpr uint32_t idesc_o = make_idesc(fmt, false, true, kTile, HS);       // O = P V
            const uint64_t q_desc = smem_desc_sw128(smem_u32(q_smem), 16, 1024);
            const uint64_t k_desc = smem_desc_sw128(smem_u32(k_smem), 16, 1024);
            const uint64_t v_desc = smem_desc_mn(smem_u32(v_smem), kBoxBytes, TF32);
            const bool leader = elect_one();
            bool ok = true;
            // the step whose S comes next
            int index = blockIdx.x, g = 0, j = 0;
            uint32_t n = 0, kv0 = 0;                       // item count, key tiles of earlier items
            FwdItem it = fwd_item(p, index);
            uint32_t i_s = 0, i_pv = 0;                    // steps issued
            uint32_t pv_a = 0, pv_b = 0;                   // P.V issued for each tile
            // steps between their S and their P.V, oldest first: tile, first step of its item, last user of
            // the V tile, V tile
            uint32_t queue[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b) queue[b] = 0;

            // issues S of the next step, if there is one; false when a wait gave up
            auto issue_s = [&]() -> bool {
                if (index < 0) return true;
                const uint32_t kv = kv0 + j, s = kv % ST, qb = n % QB, buf = i_s % NB;
                if (j == 0 && g == 0 && !mbar_wait_warp(&q_full[qb], (n / QB) & 1, p.status, kTimeoutMma)) return false;
                if (!mbar_wait_warp(&k_full[s], (kv / ST) & 1, p.status, kTimeoutMma)) return false;
                tc_fence_after_sync();
                const uint64_t qd = q_desc + ((qb * 2 + g) * C::TILE_BYTES >> 4), kd = k_desc + (s * C::TILE_BYTES >> 4);
                const uint32_t d = tmem_base + buf * kTile;
                const bool last_user = g == 1 || j >= it.n_b;         // of this K (and V) tile
                if (leader) {
#pragma unroll
                    for (int kk = 0; kk < C::ROWB / 32; ++kk) {
                        const uint32_t off = ((kk / 4) * kBoxBytes + (kk % 4) * 32) >> 4;
                        mma_ss<TF32>(d, qd + off, kd + off, idesc_s, kk > 0);
                    }
                    mma_commit(&s_full[g * NB + buf]);
                    if (last_user) mma_commit(&k_empty[s]);
                }
                const uint32_t step = (uint32_t)g | (j == 0 ? 2u : 0u) | (last_user ? 4u : 0u) | (kv << 3);
#pragma unroll
                for (int b = 0; b < NB; ++b)
                    if (b == (int)(i_s - i_pv)) queue[b] = step;
                ++i_s;
                // on to the next step
                if (g == 0 && j < it.n_b) {
                    g = 1;
                    return true;
                }
                ++j;
                g = j < it.n_a ? 0 : 1;
                if (g == 0 || j < it.n_b) return true;
                // ... of the next item
                if (leader) mma_commit(&q_empty[qb]);
                kv0 += (uint32_t)j;
                j = 0;
                g = 0;
                const uint32_t w = n % WS;
                if (!mbar_wait_warp(&work_full[w], (n / WS) & 1, p.status, kTimeoutMma)) return false;
                index = taken_cta(answers + w * 16);
                fence_proxy_async_smem();
                __syncwarp();
                if (leader) mbar_arrive(&work_empty[w]);
                ++n;
                if (index >= 0) it = fwd_item(p, index);
                return true;
            };
            for (int b = 0; b < NB && ok; ++b) ok = issue_s();
            while (ok && i_pv < i_s) {
                const uint32_t step = queue[0], kv = step >> 3, s = kv % ST, buf = i_pv % NB, par = (i_pv / NB) & 1;
                const uint32_t tile = step & 1;
                const bool first = (step & 2) != 0;
#pragma unroll
                for (int b = 0; b + 1 < NB; ++b) queue[b] = queue[b + 1];
                const uint64_t vd = v_desc + (s * C::TILE_BYTES >> 4);
                const uint32_t d = tmem_base + C::COL_O + tile * HS, a = tmem_base + buf * kTile;
                constexpr int KK = kTile / C::UK;
                if (!mbar_wait_warp(&v_full[s], (kv / ST) & 1, p.status, kTimeoutMma)) { ok = false; break; }
                if (C::HALVES) {
                    if (!mbar_wait_warp(&p_half[buf], par, p.status, kTimeoutMma)) { ok = false; break; }
                    tc_fence_after_sync();
                    if (leader) {
#pragma unroll
                        for (int kk = 0; kk < KK / 2; ++kk)
                            mma_ts<TF32>(d, a + kk * 8, vd + (kk * C::UK * 128 >> 4), idesc_o, !first || kk > 0);
                    }
                }
                if (!mbar_wait_warp(&p_full[buf], par, p.status, kTimeoutMma)) { ok = false; break; }
                tc_fence_after_sync();
                const uint32_t done = tile * 4 + ((tile ? pv_b : pv_a) & 3);
                if (leader) {
#pragma unroll
                    for (int kk = C::HALVES ? KK / 2 : 0; kk < KK; ++kk)
                        mma_ts<TF32>(d, a + kk * 8, vd + (kk * C::UK * 128 >> 4), idesc_o, !first || kk > 0);
                    mma_commit(&pv_done[done]);
                    if (step & 4) mma_commit(&v_empty[s]);
                }
                if (tile) ++pv_b;
                else      ++pv_a;
                ++i_pv;
                ok = issue_s();
            }
        }
    }
    } else {
        regs_claim<208>();
        // ---------------- softmax + output: warps 4..7 tile A, 8..11 tile B; thread = query row ----------------
        const int g = (warp - 4) >> 2;
        const int lane_group = warp & 3;
        const int r_in_tile = lane_group * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(lane_group * 32) << 16;
        const uint32_t tmem_o = tmem_base + C::COL_O + g * HS + lane_addr;
        const float sl2 = p.scale * 1.4426950408889634f;      // scores -> log2 domain
        uint32_t i0 = 0;             // steps of earlier items
        uint32_t pv = 0;             // P.V of this tile so far
        uint32_t s_par = 0;          // parity of the next wait on this tile's s_full barriers, by buffer
        // Waits for the latest P.V of this tile.  A thread does not watch every one of them, and up to three
        // may be outstanding, while a parity only tells neighbouring phases apart: four barriers take turns.
        auto wait_pv = [&](unsigned int code) -> bool {
            return mbar_wait_warp(&pv_done[g * 4 + ((pv - 1) & 3)], ((pv - 1) >> 2) & 1, p.status, code);
        };
        bool ok = true;
        int index = blockIdx.x;
        for (uint32_t n = 0; index >= 0 && ok; ++n) {
            const FwdItem it = fwd_item(p, index);
            const int n_g = g ? it.n_b : it.n_a, qt = it.qt + g;
            float m_ref = -FLT_MAX;      // max the exponentials are taken against
            float l = 0.f;               // running sum of exp
            for (int j = 0; j < n_g; ++j) {
                const uint32_t i = i0 + (j < it.n_a ? (it.n_b > 0 ? 2 * j + g : j) : it.n_a + j);
                const uint32_t buf = i % NB;
                const uint32_t tmem_s = tmem_base + buf * kTile + lane_addr;
                if (!mbar_wait_warp(&s_full[g * NB + buf], (s_par >> buf) & 1, p.status, kTimeoutSoftmax)) { ok = false; break; }
                s_par ^= 1u << buf;
                tc_fence_after_sync();
                // Keys this row does not see in this tile: beyond the diagonal, or - without a mask - beyond the
                // end of the sequence (under the mask no stored row reaches that far).
                const bool masked = p.causal ? j == qt : (j == q_tiles - 1 && tail < kTile);
                const int last = p.causal ? r_in_tile : tail - 1;
                // The whole row of scores (128 columns) comes into registers with one wait; the maximum and
                // the exponentials both work from there.
                uint32_t sc[kTile];
#pragma unroll
                for (int c = 0; c < kTile / 32; ++c)
                    tmem_ld32(tmem_s + c * 32, *reinterpret_cast<uint32_t(*)[32]>(sc + c * 32));
                tmem_wait_ld();
                // row maximum of the visible scores (the mask exists in one tile only)
                float tmax;
                {
                    float t8[8];
#pragma unroll
                    for (int x = 0; x < 8; ++x) t8[x] = -FLT_MAX;
                    if (masked) {
#pragma unroll
                        for (int x = 0; x < kTile; ++x)
                            t8[x & 7] = fmaxf(t8[x & 7], x <= last ? __uint_as_float(sc[x]) : -FLT_MAX);
                    } else {
#pragma unroll
                        for (int x = 0; x < kTile; x += 2)
                            t8[(x >> 1) & 7] = max3_f32(t8[(x >> 1) & 7], __uint_as_float(sc[x]), __uint_as_float(sc[x + 1]));
                    }
                    tmax = fmaxf(max3_f32(t8[0], t8[1], t8[2]), max3_f32(t8[3], t8[4], t8[5]));
                    tmax = max3_f32(tmax, t8[6], t8[7]);
                }
                const float m_new = fmaxf(m_ref, tmax);
                const bool need = (j == 0) || (m_new - m_ref) * sl2 > 8.0f;
                if (__any_sync(0xffffffffu, need)) {
                    float alpha = 1.f;
                    if (need) {
                        alpha = (j == 0) ? 0.f : fast_exp2((m_ref - m_new) * sl2);
                        m_ref = m_new;
                        l *= alpha;
                    }
                    if (j > 0) {
                        // the tile's earlier P.V must have left the tensor pipe
                        if (!wait_pv(kTimeoutSoftmax)) { ok = false; break; }
                        tc_fence_after_sync();
#pragma unroll 1
                        for (int c = 0; c < HS / 16; ++c) {
                            uint32_t r[16];
                            tmem_ld16(tmem_o + c * 16, r);
                            tmem_wait_ld();
#pragma unroll
                            for (int x = 0; x < 16; ++x) r[x] = __float_as_uint(__uint_as_float(r[x]) * alpha);
                            tmem_st16(tmem_o + c * 16, r);
                        }
                        tmem_wait_st();
                    }
                }
                // P = exp2(s*sl2 - m*sl2) in place in the registers (BF16: packed pairs), two elements per
                // FMA-pipe instruction, then written over S
                const float neg_m = -m_ref * sl2;
                constexpr int PART = C::HALVES ? kTile / 2 : kTile, PCOLS = TF32 ? PART : PART / 2;
#pragma unroll
                for (int h = 0; h < kTile / PART; ++h) {
                    uint32_t* part = sc + h * PART;
                    l += masked ? exp_row<TF32, true, PART>(part, sl2, neg_m, h * PART, last)
                                : exp_row<TF32, false, PART>(part, sl2, neg_m, h * PART, last);
#pragma unroll
                    for (int c = 0; c < PCOLS / 32; ++c)
                        tmem_st32(tmem_s + h * PCOLS + c * 32, *reinterpret_cast<uint32_t(*)[32]>(part + c * 32));
                    tmem_wait_st();
                    tc_fence_before_sync();
                    mbar_arrive(C::HALVES && h == 0 ? &p_half[buf] : &p_full[buf]);
                }
                ++pv;
            }
            i0 += (uint32_t)(it.n_a + it.n_b);
            // output: O / l -> global, lse = m*scale + ln(l)
            if (n_g > 0 && ok) {
                if (!wait_pv(kTimeoutEpilogue)) { ok = false; break; }
                tc_fence_after_sync();
                const float inv = 1.f / l;
                const int64_t grow = (int64_t)it.unit * p.S + (int64_t)qt * kTile + r_in_tile;
                const bool live = qt * kTile + r_in_tile < p.S;
                T* out = (T*)p.O + grow * HS;
#pragma unroll 1
                for (int c = 0; c < HS / 32; ++c) {
                    uint32_t r[32];
                    tmem_ld32(tmem_o + c * 32, r);
                    tmem_wait_ld();
                    if (!live) continue;
                    constexpr int PER = 32 / C::ES;                 // elements per 32-byte store
#pragma unroll
                    for (int x = 0; x < 32; x += PER) {
                        uint32_t o[8];
                        if (TF32) {
                            // TF32-valued output: it feeds the TF32 output projection
#pragma unroll
                            for (int e = 0; e < 8; ++e) o[e] = __float_as_uint(round_to_tf32(__uint_as_float(r[(x + e) & 31]) * inv));
                        } else {
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                __nv_bfloat162 h2 = __floats2bfloat162_rn(__uint_as_float(r[(x + 2 * e) & 31]) * inv, __uint_as_float(r[(x + 2 * e + 1) & 31]) * inv);
                                o[e] = *reinterpret_cast<uint32_t*>(&h2);
                            }
                        }
                        if (p.wide) {
                            st_global_v8(out + c * 32 + x, o);
                        } else {
                            uint4* dst = reinterpret_cast<uint4*>(out + c * 32 + x);
                            dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
                            dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
                        }
                    }
                }
                // O has been read before the first P of the next item is announced, and that is what its first
                // P.V, which starts O over, waits for
                tc_fence_before_sync();
                if (live) p.lse[grow] = m_ref * p.scale + logf(l);
            }
            if (!ok) break;
            const uint32_t w = n % WS;
            if (!mbar_wait_warp(&work_full[w], (n / WS) & 1, p.status, kTimeoutSoftmax)) { ok = false; break; }
            index = taken_cta(answers + w * 16);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&work_empty[w]);
        }
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
