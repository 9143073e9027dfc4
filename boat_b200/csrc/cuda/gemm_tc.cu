// gemm_tc.cu - the projection GEMMs of the attention layer on Blackwell tensor cores.
//
//   C[M,N] = op(A) . op(B) (+ bias)      BF16 storage (kind::f16) or FP32 storage (kind::tf32),
//                                         FP32 accumulation in tensor memory
//
// Replaces boat_matmul (reference src/ops/linear.c:116-130) inside linear_projection
// (src/layers/attention.c:247-308) and linear_projection_backward (attention.c:1186-1293).
// The three products of a projection differ only in which operand is stored transposed;
// instead of materialising transposes as the reference does (linear.c:306-334), the shared
// memory descriptors tell the tensor core which way each operand lies:
//
//   Y  = X . W      A = X  [M,K] K-major      B = W  [K,N] N-major
//   dX = dY . W^T   A = dY [M,K] K-major      B = W  [N,K] K-major
//   dW = X^T . dY   A = X  [K,M] M-major      B = dY [K,N] N-major
//
// Kernel shape: persistent, 320-thread CTAs, alone or as pairs on one tile (CTAS).  Warp 0 feeds a
// shared-memory ring with TMA (128-byte swizzle, no multicast); warp 1 walks the stages in step and one
// elected lane of it issues tcgen05.mma and commits stages back to the producer; warps 2-9 drain the accumulator from tensor
// memory.  Every warp that issues TMA or MMA does so as a whole, with one elected lane: a lone lane needed 310 to 580
// cycles for the loads of a K-block, as long as its MMAs (32768 x 4096 x 1024 plain 196 -> 180 us, with GELU 266 -> 238, with its
// derivative 332 -> 237; 1332 x 768 x 3072 15.2 -> 11.7).  The accumulator is double-buffered in tensor memory (2 x BN columns) so that the epilogue
// of one tile overlaps the main loop of the next.
//
// CTA pairs (cta_group::2, 256 x BN tiles): each CTA holds its 128 rows of A and half of B; the tensor
// cores of both SMs read both halves of B.  A CTA then brings in and reads 32 KB per 64 of K instead of 48 -
// a single CTA's 128 x 256 tile keeps the SM's shared-memory port 75 % busy with operands alone.  All
// loads of a pair count on a barrier of the first CTA, whose warp 1 issues the MMAs; its commits
// arrive at both CTAs.
//
// Epilogue: two warps per 32 rows of the tile, taking its boxes in turn.  A warp reads 64 BF16 (32 FP32) columns from tensor memory,
// converts them, writes them as 128-byte rows to a swizzled staging box of its own and stores the box
// with TMA.  (Storing from registers, where a lane holds a row, gave every 16-byte store a 32-byte
// sector of its own: 786 TFLOP/s at 32768 x 4096 x 1024.)  The same boxes serve as
// reductions (cp.reduce .add) for split K and for accumulation into the output.
//
// The epilogue can carry on with element-wise work on its tile (Epilogue): GELU beside the
// pre-activation it came from, the product with GELU's derivative, a residual - whose second operand comes
// in through the same kind of boxes.  Each saves a pass over [T, 4d] or [T, d] matrices.
//
// Weight gradients can carry the column sums of dY, the bias gradients (CSUM): four more warps add up what the first
// row of tiles streams, 16 KB per K-block and CTA, behind the products.  As passes of their own the sums read dY again: 15 us
// per 32768 x 1024 BF16 matrix at HBM rate, 5 to 7 us where a launch is the bound; step of 16 x 2048 x 1024 with Adam 1689 -> 1642
// us, encoder block of 4 x 333 x 768 256 -> 239.
//
// A chained launch sums the products of its groups in one accumulator: the three input gradients of
// self-attention are one gradient.
//
// FP32 results (weight gradients) have few tiles and a long K.  Whole waves of tiles are done by one CTA
// (pair) each; the tiles left over, which would keep most SMs idle for one more wave, are split along K
// into pieces that add into a zeroed output.
//
// Up to kMaxGroups problems of one shape and layout (the Q, K and V projections of a layer, their
// weight gradients, their input gradients) run as one launch: the persistent CTAs walk the tiles of
// all groups, group index fastest, so CTAs at work at the same time read the operand the groups
// share (X for self-attention) from L2.
#include "tc_common.cuh"
#include "gelu.cuh"

namespace boatcu {

using namespace tc;

namespace {

constexpr int BM = 128;                          // rows of C per CTA
constexpr int kEpiWarps = 8;
constexpr int kSumWarps = 4;                     // launches with column sums only
constexpr int kThreads = 64 + 32 * kEpiWarps;
constexpr int kMaxGroups = 4;
constexpr int kBoxRows = 32;                     // rows of a staging box: one epilogue warp's rows
constexpr int kStageBox = kBoxRows * 128;        // 32 rows x 128 bytes

template <typename T, int CTAS, int BN, int EPI>
struct Cfg {
    // boxes per epilogue warp: one result, and one of the second result or operand
    static constexpr int BOXES = EPI == BOAT_EPI_NONE ? 1 : 2;
    static constexpr int ES = sizeof(T);
    static constexpr int BK = 128 / ES;             // one 128-byte swizzle row of K (or of M/N)
    static constexpr int UK = 32 / ES;              // K extent of one tcgen05.mma
    static constexpr int BNC = BN / CTAS;           // rows of B held by one CTA
    static constexpr int A_BYTES = BM * 128;
    static constexpr int B_BYTES = BNC * 128;
    static constexpr int STAGE = A_BYTES + B_BYTES;
    static constexpr int CHUNK_BYTES = BK * 128;    // one [BK rows x 128 B] box of an MN-major operand
    static constexpr int OUT_BYTES = kEpiWarps * BOXES * kStageBox;
    static constexpr int FIT = (232448 - 1024 - 512 - OUT_BYTES) / STAGE;
    static constexpr int STAGES = FIT < 8 ? FIT : 8;
    static constexpr int SMEM = STAGES * STAGE + OUT_BYTES + 1024 /*alignment*/ + 512 /*barriers*/;
    static constexpr uint32_t TMEM_COLS = 2 * BN;   // two accumulators
};

struct GroupMaps {
    CUtensorMap a[kMaxGroups], b[kMaxGroups], c[kMaxGroups];
    CUtensorMap aux;         // second result (BOAT_EPI_GELU) or element-wise operand of the epilogue
};

struct Params {
    const float* bias[kMaxGroups];
    float* colsum[kMaxGroups];       // sums over K of B's columns
    int colsum_add;      // ... are added to what is there
    float* part_sums;    // [groups][split][N]: those of the pieces of split tiles
    unsigned int* arrived;           // zeros: pieces whose sums are there, per group, column of tiles, CTA of a pair and warp
    int groups;
    int chain;           // the groups' products are summed into one result
    int M, N, K;
    int out_type;
    int full;            // tiles done in one piece; the rest is split along K
    int split;
    int wide_a, wide_b;  // an operand read along M or N comes as one copy per stage (make_tensor_map_chunks)
    int follow;          // how the launch follows the one before (Follow)
    int add_all;         // every tile adds to the output, not only the pieces of split tiles
    unsigned int* status;
};

struct WorkItem {
    int g, m0, n0, kb0, kb1;
    int part, pieces;    // which piece of its tile; the first adds the bias
    bool add;            // result is added to the output
};

template <typename T, bool A_MN, bool B_MN, int CTAS, int BN, int EPI, bool CSUM>
__global__ void __launch_bounds__(kThreads + (CSUM ? 32 * kSumWarps : 0), 1)
gemm_tc_kernel(const __grid_constant__ GroupMaps maps, const __grid_constant__ Params p) {
    using C = Cfg<T, CTAS, BN, EPI>;
    constexpr bool AUX_IN = EPI == BOAT_EPI_GELU_GRAD || EPI == BOAT_EPI_ADD;
    constexpr bool TF32 = sizeof(T) == 4;
    constexpr int STAGES = C::STAGES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* a_smem = smem;
    uint8_t* b_smem = smem + STAGES * C::A_BYTES;
    uint8_t* out_smem = b_smem + STAGES * C::B_BYTES;
    uint64_t* bars = (uint64_t*)(out_smem + C::OUT_BYTES);
    uint64_t* full = bars;                        // [STAGES] TMA -> MMA (of the first CTA of a pair)
    uint64_t* empty = bars + STAGES;              // [STAGES] MMA -> TMA
    uint64_t* acc_full = bars + 2 * STAGES;       // [2] MMA -> epilogue
    uint64_t* acc_empty = bars + 2 * STAGES + 2;  // [2] epilogue -> MMA (of the first CTA of a pair)
    uint64_t* aux_full = bars + 2 * STAGES + 4;   // [kEpiWarps] an epilogue warp's operand box landed
    uint32_t* tmem_slot = (uint32_t*)(bars + 2 * STAGES + 12);
    uint64_t* summed = bars + 2 * STAGES + 13;    // [STAGES] column sums -> TMA, behind `empty` (CSUM)
    uint64_t* const refill = CSUM ? summed : empty;

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const uint32_t rank = CTAS == 2 ? cluster_rank() : 0;
    const int worker = blockIdx.x / CTAS, workers = gridDim.x / CTAS;
    const int m_tiles = (p.M + BM * CTAS - 1) / (BM * CTAS), n_tiles = (p.N + BN - 1) / BN;
    const int k_one = (p.K + C::BK - 1) / C::BK;                   // K-blocks of one product
    const int k_blocks = p.chain ? k_one * p.groups : k_one;
    const int results = p.chain ? 1 : p.groups;
    const int tiles = m_tiles * n_tiles * results;
    const int work_items = p.full + (tiles - p.full) * p.split;
    auto item = [&](int w) {
        WorkItem it;
        // pieces of one K range are neighbours: the CTAs at work together share the rows they stream
        const int rest = tiles - p.full;
        const int tile = w < p.full ? w : p.full + (w - p.full) % rest;
        it.part = w < p.full ? 0 : (w - p.full) / rest;
        it.pieces = w < p.full ? 1 : p.split;
        const int mn = tile / results;
        it.g = tile % results;
        it.m0 = (mn / n_tiles) * BM * CTAS + (int)rank * BM;
        it.n0 = (mn % n_tiles) * BN;
        it.kb0 = (int)((int64_t)it.part * k_blocks / it.pieces);
        it.kb1 = (int)((int64_t)(it.part + 1) * k_blocks / it.pieces);
        it.add = it.pieces > 1 || p.add_all;
        return it;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
            if (CSUM) mbar_init(&summed[s], kSumWarps);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], kEpiWarps * CTAS);
        }
        for (int b = 0; b < kEpiWarps; ++b) mbar_init(&aux_full[b], 1);
        fence_barrier_init();
        for (int g = 0; g < p.groups; ++g) {
            tma_prefetch_desc(&maps.a[g]);
            tma_prefetch_desc(&maps.b[g]);
            if (g < results) tma_prefetch_desc(&maps.c[g]);
        }
        if (EPI != BOAT_EPI_NONE) tma_prefetch_desc(&maps.aux);
    }
    if (warp == 1) {
        if (CTAS == 2) tmem_alloc_pair(tmem_slot, C::TMEM_COLS);
        else           tmem_alloc(tmem_slot, C::TMEM_COLS);
    }
    griddep_enter(p.follow);
    tc_fence_before_sync();
    __syncthreads();
    if (CTAS == 2) cluster_sync_all();            // the peer's barriers exist before anything arrives there
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        // the whole warp in step, one elected lane issues: with the loop on a lone lane, whose operands cannot live in
        // uniform registers, the three loads of a K-block took 310 cycles to issue (580 beside a GELU epilogue) and
        // the tensor core waited for them half of its time
        const bool leader = elect_one();
        uint32_t s = 0, parity = 1;
        bool ok = true;
        for (int w = worker; w < work_items && ok; w += workers) {
            const WorkItem t = item(w);
            const int nb = t.n0 + (int)rank * C::BNC;                 // this CTA's rows of B
            int g = t.g, k0 = t.kb0 * C::BK, k_end = t.kb1 * C::BK;
            if (p.chain) {
                g = t.kb0 / k_one;
                k0 -= g * k_one * C::BK;
                k_end -= g * k_one * C::BK;
            }
            for (;;) {                                                // one product of a chain, or all
                const CUtensorMap* const map_a = &maps.a[g];
                const CUtensorMap* const map_b = &maps.b[g];
                const int stop = p.chain ? min(k_end, k_one * C::BK) : k_end;
                for (; k0 < stop; k0 += C::BK) {
                    if (!mbar_wait_warp(&refill[s], parity, p.status, kTimeoutProducer)) { ok = false; break; }
                    uint8_t* const a_dst = a_smem + s * C::A_BYTES;
                    uint8_t* const b_dst = b_smem + s * C::B_BYTES;
                    const uint32_t bar = CTAS == 2 ? peer_addr(&full[s], 0) : 0;
                    auto load = [&](uint8_t* dst, const CUtensorMap* map, int x, int y) {
                        if (CTAS == 2) tma_load_2d_pair(dst, map, bar, x, y);
                        else           tma_load_2d(dst, map, &full[s], x, y);
                    };
                    auto load_columns = [&](uint8_t* dst, const CUtensorMap* map, int column) {
                        if (CTAS == 2) tma_load_3d_pair(dst, map, bar, 0, k0, column);
                        else           tma_load_3d(dst, map, &full[s], 0, k0, column);
                    };
                    if (leader) {
                        if (rank == 0) mbar_arrive_expect_tx(&full[s], CTAS * C::STAGE);
                        if (A_MN && p.wide_a) {
                            load_columns(a_dst, map_a, t.m0 / C::BK);
                        } else if (A_MN) {
#pragma unroll
                            for (int c = 0; c < BM / C::BK; ++c) load(a_dst + c * C::CHUNK_BYTES, map_a, t.m0 + c * C::BK, k0);
                        } else {
                            load(a_dst, map_a, k0, t.m0);
                        }
                        if (B_MN && p.wide_b) {
                            load_columns(b_dst, map_b, nb / C::BK);
                        } else if (B_MN) {
#pragma unroll
                            for (int c = 0; c < C::BNC / C::BK; ++c) load(b_dst + c * C::CHUNK_BYTES, map_b, nb + c * C::BK, k0);
                        } else {
                            load(b_dst, map_b, k0, nb);
                        }
                    }
                    if (++s == STAGES) {
                        s = 0;
                        parity ^= 1;
                    }
                }
                if (!ok || k0 >= k_end) break;
                ++g;
                k0 = 0;
                k_end -= k_one * C::BK;
            }
        }
        if (!ok) {
            // give loads already in flight time to land before the CTA's memory goes away
            for (int i = 0; i < 1000; ++i) __nanosleep(1000);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // the whole warp in step, one elected lane issues, so that the operands stay in uniform registers
        if (rank == 0) {
            constexpr uint32_t idesc = make_idesc(TF32 ? kTF32 : kBF16, A_MN, B_MN, BM * CTAS, BN);
            const uint64_t a_desc0 = A_MN ? smem_desc_mn(smem_u32(a_smem), C::CHUNK_BYTES, TF32) : smem_desc_sw128(smem_u32(a_smem), 16, 1024);
            const uint64_t b_desc0 = B_MN ? smem_desc_mn(smem_u32(b_smem), C::CHUNK_BYTES, TF32) : smem_desc_sw128(smem_u32(b_smem), 16, 1024);
            const bool leader = elect_one();
            uint32_t s = 0, parity = 0, acc_it = 0;
            bool ok = true;
            for (int w = worker; w < work_items && ok; w += workers, ++acc_it) {
                const WorkItem t = item(w);
                const int buf = acc_it & 1;
                if (!mbar_wait_warp(&acc_empty[buf], ((acc_it >> 1) & 1) ^ 1, p.status, kTimeoutMma)) { ok = false; break; }
                tc_fence_after_sync();
                const uint32_t d_tmem = tmem_base + buf * BN;
                for (int kb = t.kb0; kb < t.kb1; ++kb) {
                    if (!mbar_wait_warp(&full[s], parity, p.status, kTimeoutMma)) { ok = false; break; }
                    tc_fence_after_sync();
                    const uint64_t a_desc = a_desc0 + (s * C::A_BYTES >> 4), b_desc = b_desc0 + (s * C::B_BYTES >> 4);
                    if (leader) {
#pragma unroll
                        for (int kk = 0; kk < C::BK / C::UK; ++kk) {
                            const uint64_t ad = a_desc + ((A_MN ? kk * C::UK * 128 : kk * 32) >> 4);
                            const uint64_t bd = b_desc + ((B_MN ? kk * C::UK * 128 : kk * 32) >> 4);
                            if (CTAS == 2) mma_ss_pair<TF32>(d_tmem, ad, bd, idesc, kb > t.kb0 || kk > 0);
                            else           mma_ss<TF32>(d_tmem, ad, bd, idesc, kb > t.kb0 || kk > 0);
                        }
                        // stage reusable once these MMAs have read it
                        if (CTAS == 2) mma_commit_pair(&empty[s]);
                        else           mma_commit(&empty[s]);
                    }
                    if (++s == STAGES) {
                        s = 0;
                        parity ^= 1;
                    }
                }
                if (ok && leader) {                   // accumulator complete
                    if (CTAS == 2) mma_commit_pair(&acc_full[buf]);
                    else           mma_commit(&acc_full[buf]);
                }
            }
        }
    } else if (CSUM && warp >= 2 + kEpiWarps) {
        // ---------------- column sums of B: warps 10..13 ----------------
        // A tile of the first row of tiles adds up the rows of B that it streams anyway, once the tensor core is done with
        // them (both CTAs of a pair hear of that; only the first hears of the loads), and hands the stage on to the
        // producer.  A warp has a quarter of the columns, a lane 16 bytes of every RL-th row; the rows are dealt out so
        // that the eight lanes of a shared-memory phase meet eight swizzle positions.  A K-block is summed for itself
        // before it joins the total.  Where the tile is one of several pieces of K the sums wait beside those of the others, and
        // the warp that comes last adds them up in the order of the pieces: the same bits every time.
        constexpr int PER = 16 / C::ES, UW = C::BNC / PER / kSumWarps, RL = 32 / UW, PH = UW < 8 ? 8 / UW : 1;
        constexpr int PERIOD = TF32 ? 4 : 8, H = PERIOD / PH;
        const int unit = (warp - 2 - kEpiWarps) * UW + lane % UW, rl = lane / UW, u8 = unit & 7;
        const int row_first = (rl % PH) * H + (rl / PH) % H + rl / (PH * H) * (PH * H);
        const uint8_t* const column = b_smem + (unit >> 3) * C::CHUNK_BYTES;
        const bool leader = elect_one();
        uint32_t s = 0, parity = 0;
        bool ok = true;
        for (int w = worker; w < work_items && ok; w += workers) {
            const WorkItem t = item(w);
            const bool mine = t.m0 == (int)rank * BM;
            float total[PER];
#pragma unroll
            for (int e = 0; e < PER; ++e) total[e] = 0.f;
            for (int kb = t.kb0; kb < t.kb1; ++kb) {
                if (!mbar_wait_warp(&empty[s], parity, p.status, kTimeoutOther)) { ok = false; break; }
                if (mine) {
                    float sum[PER];
#pragma unroll
                    for (int e = 0; e < PER; ++e) sum[e] = 0.f;
#pragma unroll
                    for (int i = 0; i < C::BK / RL; ++i) {
                        const int row = i * RL + row_first;
                        const int at = TF32 ? ((((u8 >> 1) ^ (row & 3)) << 1) | (u8 & 1)) : (u8 ^ (row & 7));
                        const uint4 q = *reinterpret_cast<const uint4*>(column + s * C::B_BYTES + row * 128 + (at << 4));
                        const uint32_t x[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            if (TF32) {
                                sum[e] += __uint_as_float(x[e]);
                            } else {
                                sum[2 * e % PER] += __uint_as_float(x[e] << 16);
                                sum[(2 * e + 1) % PER] += __uint_as_float(x[e] & 0xffff0000u);
                            }
                        }
                    }
#pragma unroll
                    for (int e = 0; e < PER; ++e) total[e] += sum[e];
                }
                fence_proxy_async_smem();             // the reads are done before the producer's next copy into the stage
                __syncwarp();
                if (leader) mbar_arrive(&summed[s]);
                if (++s == STAGES) {
                    s = 0;
                    parity ^= 1;
                }
            }
            if (!ok || !mine) continue;
#pragma unroll
            for (int e = 0; e < PER; ++e)
#pragma unroll
                for (int d = UW; d < 32; d <<= 1) total[e] += __shfl_xor_sync(0xffffffffu, total[e], d);
            const int col = t.n0 + (int)rank * C::BNC + unit * PER;
            if (t.pieces > 1) {
                float* const parts = p.part_sums + (int64_t)t.g * t.pieces * p.N + col;
                if (rl == 0) {
#pragma unroll
                    for (int e = 0; e < PER; ++e)
                        if (col + e < p.N) parts[(int64_t)t.part * p.N + e] = total[e];
                }
                __threadfence();
                __syncwarp();
                unsigned int before = 0;
                if (lane == 0) before = atomicAdd(p.arrived + ((t.g * n_tiles + t.n0 / BN) * CTAS + (int)rank) * kSumWarps + warp - 2 - kEpiWarps, 1u);
                if (__shfl_sync(0xffffffffu, before, 0) + 1 != (unsigned int)t.pieces) continue;
                __threadfence();
#pragma unroll
                for (int e = 0; e < PER; ++e) total[e] = 0.f;
                for (int i = 0; i < t.pieces; ++i)
#pragma unroll
                    for (int e = 0; e < PER; ++e)
                        if (col + e < p.N) total[e] += __ldcg(parts + (int64_t)i * p.N + e);
            }
            if (rl == 0) {
                float* const out = p.colsum[t.g] + col;
#pragma unroll
                for (int e = 0; e < PER; ++e)
                    if (col + e < p.N) out[e] = p.colsum_add ? out[e] + total[e] : total[e];
            }
        }
    } else {
        // ---------------- epilogue: warps 2..9 ----------------
        // two warps per quarter of the rows, box by box in turn
        const int lane_group = warp & 3;              // TMEM lanes this warp may touch
        const int turn = (warp - 2) >> 2;
        uint8_t* const box = out_smem + (warp - 2) * C::BOXES * kStageBox;    // result, then the second kind
        uint8_t* const row = box + lane * 128;
        uint8_t* const row2 = row + kStageBox;
        uint64_t* const aux_bar = &aux_full[warp - 2];
        uint32_t aux_it = 0;                          // operand boxes used so far
        auto load_aux = [&](int x, int y) {           // by the leader
            mbar_arrive_expect_tx(aux_bar, kStageBox);
            tma_load_2d(box + kStageBox, &maps.aux, aux_bar, x, y);
        };
        const bool leader = elect_one();
        const int swz = lane & 7;
        const bool bf16_out = p.out_type == BOAT_CUDA_BF16;
        const int step = bf16_out ? 64 : 32;          // columns per box
        uint32_t acc_it = 0;
        bool ok = true;
        for (int w = worker; w < work_items && ok; w += workers, ++acc_it) {
            const WorkItem t = item(w);
            const CUtensorMap* map_c = &maps.c[t.g];
            const float* const bias = t.part == 0 ? p.bias[t.g] : nullptr;
            const bool bias16 = ((uintptr_t)bias & 15) == 0;
            const int buf = acc_it & 1;
            const int row0 = t.m0 + lane_group * 32;
            const int cols = min(BN, p.N - t.n0), c_first = turn * step;
            if (AUX_IN && leader && c_first < cols) load_aux(t.n0 + c_first, row0);
            if (!mbar_wait_warp(&acc_full[buf], (acc_it >> 1) & 1, p.status, kTimeoutEpilogue)) { ok = false; break; }
            tc_fence_after_sync();
            const uint32_t t_addr = tmem_base + ((uint32_t)(lane_group * 32) << 16) + buf * BN;
            auto leave_accumulator = [&] {            // this warp's part of the tile is out of tensor memory
                tc_fence_before_sync();
                __syncwarp();
                if (leader) {
                    if (CTAS == 2) mbar_arrive_peer(peer_addr(&acc_empty[buf], 0));
                    else           mbar_arrive(&acc_empty[buf]);
                }
            };
            if (c_first >= cols) leave_accumulator();
#pragma unroll 1
            for (int c = c_first; c < cols; c += 2 * step) {
                const int col0 = t.n0 + c;
                uint4 aux[8];                         // the operand's row of the box
                if (AUX_IN) {
                    if (!mbar_wait_warp(aux_bar, aux_it & 1, p.status, kTimeoutEpilogue)) { ok = false; break; }
                    ++aux_it;
#pragma unroll
                    for (int u = 0; u < 8; ++u) aux[u] = *reinterpret_cast<const uint4*>(row2 + ((u ^ swz) << 4));
                    // The next one comes in under the work on this one, into the same box: not before every lane's reads have been
                    // performed.  Without the fence they may still be queued when the copy lands (16 bytes of a row in
                    // one of a hundred steps).
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (leader && c + 2 * step < cols) load_aux(col0 + 2 * step, row0);
                }
                // one 32-column half of the box (all of an FP32 box) at a time
#pragma unroll
                for (int h = 0; h < 64; h += 32) {
                    if (h == step) break;
                    uint32_t r[32];
                    tmem_ld32(t_addr + c + h, r);
                    tmem_wait_ld();
                    float v[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
                    if (bias) {
                        const float* b = bias + col0 + h;
                        if (bias16 && col0 + h + 32 <= p.N) {
#pragma unroll
                            for (int j = 0; j < 32; j += 4) {
                                const float4 q = __ldg(reinterpret_cast<const float4*>(b + j));
                                v[j] += q.x; v[j + 1] += q.y; v[j + 2] += q.z; v[j + 3] += q.w;
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (col0 + h + j < p.N) v[j] += __ldg(b + j);
                        }
                    }
                    if (AUX_IN) {                     // BF16 only
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const uint32_t x[4] = {aux[h / 8 + u].x, aux[h / 8 + u].y, aux[h / 8 + u].z, aux[h / 8 + u].w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x[e]));
                                if (EPI == BOAT_EPI_ADD) {
                                    v[8 * u + 2 * e] += f.x;
                                    v[8 * u + 2 * e + 1] += f.y;
                                } else {
                                    float& v0 = v[8 * u + 2 * e];
                                    float& v1 = v[8 * u + 2 * e + 1];
                                    GeluPair::unpack(GeluPair::mul(GeluPair::pack(v0, v1), GeluPair(f.x, f.y).grad()), v0, v1);
                                }
                            }
                        }
                    }
                    if (h == 0) {                     // the stores that used this box (and its pair) last have read it
                        if (leader) tma_wait_group_read0();
                        __syncwarp();
                    }
                    if (EPI == BOAT_EPI_GELU) {       // the rounded pre-activation, kept, then GELU of it
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            uint32_t o[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                __nv_bfloat162 q = __floats2bfloat162_rn(v[8 * u + 2 * e], v[8 * u + 2 * e + 1]);
                                o[e] = *reinterpret_cast<uint32_t*>(&q);
                                const float2 f = __bfloat1622float2(q);
                                GeluPair(f.x, f.y).value(v[8 * u + 2 * e], v[8 * u + 2 * e + 1]);
                            }
                            *reinterpret_cast<uint4*>(row2 + (((h / 8 + u) ^ swz) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
                        }
                    }
                    if (bf16_out) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            uint32_t o[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                __nv_bfloat162 q = __floats2bfloat162_rn(v[8 * u + 2 * e], v[8 * u + 2 * e + 1]);
                                o[e] = *reinterpret_cast<uint32_t*>(&q);
                            }
                            *reinterpret_cast<uint4*>(row + (((h / 8 + u) ^ swz) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
                        }
                    } else {
                        if (p.out_type == BOAT_CUDA_F32_TF32) {        // feeds another TF32 contraction
#pragma unroll
                            for (int j = 0; j < 32; ++j) v[j] = round_to_tf32(v[j]);
                        }
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            *reinterpret_cast<float4*>(row + ((u ^ swz) << 4)) = make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
                    }
                }
                if (c + 2 * step >= cols) leave_accumulator();
                fence_proxy_async_smem();
                __syncwarp();
                if (leader) {
                    if (row0 < p.M) {
                        if (t.add) tma_reduce_add_2d(map_c, box, col0, row0);
                        else       tma_store_2d(map_c, box, col0, row0);
                        if (EPI == BOAT_EPI_GELU) tma_store_2d(&maps.aux, box + kStageBox, col0, row0);
                    }
                    tma_commit_group();
                }
            }
        }
        if (leader) tma_wait_group0();
        if (AUX_IN && !ok)                            // an operand box may be in flight
            for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    tc_fence_before_sync();
    __syncthreads();
    if (CTAS == 2) cluster_sync_all();            // the peer may still read this CTA's operands or arrive here
    if (warp == 1) {
        tc_fence_after_sync();
        if (CTAS == 2) tmem_dealloc_pair(tmem_base, C::TMEM_COLS);
        else           tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
    griddep_leave(p.follow);
}

bool g_yielding = false;

struct Problem {
    int groups;
    int64_t M, N, K;
    const void* const* A;
    int64_t lda;
    const void* const* B;
    int64_t ldb;
    void* const* C;
    int64_t ldc;
    int out_type;
    const float* const* bias;
    bool add;            // add to C instead of overwriting it (FP32)
    bool chain;          // one result: the sum of the groups' products
    void* aux;           // second result or operand of the epilogue, laid out like C
    float* const* colsum;    // per group the sums over K of B's columns, written or (add) added to; NULL: none
    int results() const { return chain ? 1 : groups; }           // entries of C
};

// A tile shape and what it costs, measured on B200 with every shape forced on 66 outputs from 128 x 1024 to 8192 x 1024 with K
// of 512 to 3072: microseconds per K-block (128 bytes of K per row, either type) on a full GPU, [1] with A read along M, and
// once per launch more than the narrowest tile, which has about 3.5 (filling the ring, the epilogue that nothing
// overlaps).  A K-block costs what its bytes cost to bring to the SM: 24, 32, 48 KB per CTA.  The choice is within 0.5 % of the
// best shape on average, 7 % at worst (K of 3072 at 8000 x 1024: pairs 36 us, 128 x 256 37, 128 x 128 43, 128 x 64 59;
// 1332 x 768: 20, 18, 12, 11.5).
struct Shape { int ctas, bn; double block_us[2], once_us; };
constexpr Shape kShapes[4] = {{2, 256, {0.29, 0.28}, 2.6},
                              {1, 256, {0.32, 0.38}, 1.0},
                              {1, 128, {0.18, 0.22}, 0.3},
                              {1, 64, {0.156, 0.18}, 0.0}};

struct Plan {
    int64_t tiles, full, split;
    double us;
};

// Which tiles are cut along K, into how many pieces, and how long the launch should take.
Plan make_plan(const Problem& q, const Shape& sh, int bk, bool a_mn) {
    const double block_us = sh.block_us[a_mn];
    const int64_t workers = sm_count() / sh.ctas, k_blocks = ceil_div(q.K, bk) * (q.chain ? q.groups : 1);
    Plan r;
    r.tiles = ceil_div(q.M, BM * sh.ctas) * ceil_div(q.N, sh.bn) * q.results();
    r.full = r.tiles;
    r.split = 1;
    r.us = (double)ceil_div(r.tiles, workers) * (double)k_blocks * block_us + sh.once_us;
    if (q.out_type != BOAT_CUDA_F32) return r;
    // FP32 results: the last, partly filled wave of tiles is cut so that its pieces come out even over
    // all workers; at least 8 K-blocks per piece, and none below K = 2048: there a group of problems gives
    // the bits of single calls, and the pieces hardly pay for clearing the output.  An SM gets its part of a piece out at about 36 KB per
    // microsecond, behind the next piece's main loop but for the last one; the output is cleared first.
    const int64_t rest = r.tiles % workers, whole = r.tiles / workers;
    const double out_us = BM * sh.bn * 4.0 / 36e3;
    const double clear_us = q.add ? 0.0 : 2.0 + (double)q.M * (double)q.N * q.results() * 4.0 / 4e6;
    int64_t most = k_blocks / 8;
    if (q.K < 2048) most = 1;
    if (most > 32) most = 32;
    for (int64_t s = 2; s <= most && rest > 0; ++s) {
        double piece = (double)k_blocks / (double)s * block_us;
        if (piece < out_us) piece = out_us;
        const double t = (double)whole * (double)k_blocks * block_us + (double)ceil_div(rest * s, workers) * piece + out_us +
                         clear_us + sh.once_us;
        if (t < r.us) {
            r.us = t;
            r.split = s;
            r.full = r.tiles - rest;
        }
    }
    return r;
}

// Zeroes every output of a launch that adds pieces to them, and the counters of its column sums: one launch, in order with the
// others.  (A memset per output also keeps the GEMM from being set up behind the kernel before it.)
struct ClearTable {
    float* out[kMaxGroups + 1];      // matrices of `rows` rows, then the counters
    int64_t rows, N, ldc, counters;
    int matrices, follow;
};

__global__ void __launch_bounds__(256) clear_kernel(const ClearTable t) {
    griddep_enter(t.follow);
    float* const out = t.out[blockIdx.y];
    const bool matrix = (int)blockIdx.y < t.matrices;
    const int64_t ld = matrix ? t.ldc : t.counters, row = matrix ? t.N : t.counters, n = matrix ? t.rows * t.N : t.counters;
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    if (ld == row && n % 4 == 0 && ((uintptr_t)out & 15) == 0) {
        for (int64_t i = first; i < n / 4; i += step) reinterpret_cast<float4*>(out)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
        for (int64_t i = first; i < n; i += step) out[i / row * ld + i % row] = 0.f;
    }
    griddep_leave(t.follow);
}

int clear(const Problem& q, unsigned int* arrived, int64_t counters) {
    ClearTable t;
    t.rows = q.M;
    t.N = q.N;
    t.ldc = q.ldc;
    t.matrices = q.add ? 0 : q.results();
    t.counters = counters;
    int count = 0;
    for (int g = 0; g < t.matrices; ++g) t.out[count++] = (float*)q.C[g];
    if (counters) t.out[count++] = (float*)arrived;
    if (count == 0) return 0;
    const int64_t blocks = ceil_div(q.add ? counters : q.M * q.N, 256 * 4 * 4), most = 4 * sm_count();
    LaunchTurn turn;
    for (int g = 0; g < t.matrices; ++g) turn.writes(t.out[g], q.M, q.N, q.ldc, 4);
    turn.writes(arrived, (size_t)counters * 4);
    t.follow = turn.follow();
    BOATCU_CHECK(launch_in_turn(turn, clear_kernel, dim3((unsigned)(blocks < most ? blocks : most), (unsigned)count), dim3(256), 0, 1, t));
    BOATCU_LAUNCH_OK("gemm_tc clear");
    return 0;
}

// Memory of one launch for the column sums of split tiles, counters and then sums.  Given back in the order of the stream.
struct PartSums {
    unsigned int* arrived = nullptr;
    float* sums = nullptr;
    int64_t counters = 0;
    size_t bytes = 0;
    int take(int64_t count, int64_t values) {
        counters = ceil_div(count, 4) * 4;
        bytes = (size_t)(counters + values) * 4;
        void* block = nullptr;
        if (int rc = boat_cuda_malloc(&block, bytes)) return rc;
        arrived = (unsigned int*)block;
        sums = (float*)(arrived + counters);
        return 0;
    }
    ~PartSums() {
        if (arrived) boat_cuda_free(arrived);
    }
};

template <typename T, bool A_MN, bool B_MN, int CTAS, int BN, int EPI, bool CSUM>
int launch(const Problem& q, const Plan& plan) {
    using C = Cfg<T, CTAS, BN, EPI>;
    GroupMaps maps;
    Params p;
    const bool bf16_out = q.out_type == BOAT_CUDA_BF16;
    p.wide_a = q.M % C::BK == 0;
    p.wide_b = q.N % C::BK == 0;
    for (int g = 0; g < q.groups; ++g) {
        // A: K-major -> matrix [M rows, K cols], box [BM, BK].  M-major -> stored [K rows, M cols], boxes [BK, BK], all of them
        // in one copy where the rows are whole 128-byte columns.
        if (int rc = !A_MN      ? make_tensor_map_2d(&maps.a[g], q.A[g], C::ES, (uint64_t)q.M, (uint64_t)q.K, (uint64_t)q.lda, BM, C::BK)
                     : p.wide_a ? make_tensor_map_chunks(&maps.a[g], q.A[g], C::ES, (uint64_t)q.K, (uint64_t)q.M, (uint64_t)q.lda, C::BK, BM / C::BK, C::ES == 4)
                                : make_tensor_map_2d(&maps.a[g], q.A[g], C::ES, (uint64_t)q.K, (uint64_t)q.M, (uint64_t)q.lda, C::BK, C::BK, C::ES == 4))
            return rc;
        if (int rc = !B_MN      ? make_tensor_map_2d(&maps.b[g], q.B[g], C::ES, (uint64_t)q.N, (uint64_t)q.K, (uint64_t)q.ldb, C::BNC, C::BK)
                     : p.wide_b ? make_tensor_map_chunks(&maps.b[g], q.B[g], C::ES, (uint64_t)q.K, (uint64_t)q.N, (uint64_t)q.ldb, C::BK, C::BNC / C::BK, C::ES == 4)
                                : make_tensor_map_2d(&maps.b[g], q.B[g], C::ES, (uint64_t)q.K, (uint64_t)q.N, (uint64_t)q.ldb, C::BK, C::BK, C::ES == 4))
            return rc;
        if (g >= q.results()) continue;
        if (int rc = make_tensor_map_2d(&maps.c[g], q.C[g], bf16_out ? 2 : 4, (uint64_t)q.M, (uint64_t)q.N, (uint64_t)q.ldc, kBoxRows, bf16_out ? 64 : 32))
            return rc;
        p.bias[g] = q.bias ? q.bias[g] : nullptr;
    }
    if (EPI != BOAT_EPI_NONE)
        if (int rc = make_tensor_map_2d(&maps.aux, q.aux, 2, (uint64_t)q.M, (uint64_t)q.N, (uint64_t)q.ldc, kBoxRows, 64)) return rc;
    const int64_t full = plan.full, split = plan.split, tiles = plan.tiles, workers = sm_count() / CTAS;
    // the sums of split tiles: those of the first row of tiles, which come first
    const int64_t n_tiles = ceil_div(q.N, BN), summing = n_tiles * q.groups;
    PartSums parts;
    if (CSUM && split > 1 && full < summing)
        if (int rc = parts.take(summing * CTAS * kSumWarps, q.groups * split * q.N)) return rc;
    if (split > 1)
        if (int rc = clear(q, parts.arrived, parts.counters)) return rc;
    p.part_sums = parts.sums;
    p.arrived = parts.arrived;
    for (int g = 0; g < q.groups; ++g) p.colsum[g] = CSUM ? q.colsum[g] : nullptr;
    p.colsum_add = q.add ? 1 : 0;
    p.groups = q.groups;
    p.chain = q.chain ? 1 : 0;
    p.M = (int)q.M;
    p.N = (int)q.N;
    p.K = (int)q.K;
    p.out_type = q.out_type;
    p.full = (int)full;
    p.split = (int)split;
    p.add_all = q.add ? 1 : 0;
    p.status = kernel_status_ptr();
    auto kern = gemm_tc_kernel<T, A_MN, B_MN, CTAS, BN, EPI, CSUM>;
    static bool configured = false;     // per process = per device: the library binds to one device
    if (!configured) {
        BOATCU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
        configured = true;
    }
    const int64_t work = full + (tiles - full) * split;
    // Persistent by default: one CTA per SM walks the tiles.  A yielding launch has one CTA per tile
    // instead, so that SMs come free all along and the CTAs of a collective started beside it (whose
    // stream has priority) get placed while the GEMM runs, not after it.
    const int64_t grid = (g_yielding || work < workers ? work : workers) * CTAS;
    ProfileScope prof(A_MN ? "gemm_tc_tn" : (B_MN ? "gemm_tc_nn" : "gemm_tc_nt"));
    {
        LaunchTurn turn;
        for (int g = 0; g < q.groups; ++g) {
            turn.reads(q.A[g], A_MN ? q.K : q.M, A_MN ? q.M : q.K, q.lda, C::ES);
            turn.reads(q.B[g], B_MN ? q.K : q.N, B_MN ? q.N : q.K, q.ldb, C::ES);
            if (g >= q.results()) continue;
            turn.writes(q.C[g], q.M, q.N, q.ldc, bf16_out ? 2 : 4);
            turn.reads(p.bias[g], (size_t)q.N * 4);
            turn.writes(p.colsum[g], (size_t)q.N * 4);
        }
        turn.writes(q.aux, q.M, q.N, q.ldc, 2);
        turn.writes(parts.arrived, parts.bytes);
        p.follow = turn.follow();
        BOATCU_CHECK(launch_in_turn(turn, kern, dim3((unsigned)grid), dim3(kThreads + (CSUM ? 32 * kSumWarps : 0)), C::SMEM, CTAS, maps, p));
    }
    BOATCU_LAUNCH_OK("gemm_tc");
    return 0;
}

// The tile shape with the shortest estimate.
template <typename T, bool A_MN, bool B_MN, int EPI = BOAT_EPI_NONE, bool CSUM = false>
int pick_tile(const Problem& q) {
    int best = 0;
    Plan plan;
    for (int i = 0; i < 4; ++i) {
        const Plan t = make_plan(q, kShapes[i], 128 / (int)sizeof(T), A_MN);
        if (i == 0 || t.us < plan.us) {
            plan = t;
            best = i;
        }
    }
    switch (best) {
        case 0: return launch<T, A_MN, B_MN, 2, 256, EPI, CSUM>(q, plan);
        case 1: return launch<T, A_MN, B_MN, 1, 256, EPI, CSUM>(q, plan);
        case 2: return launch<T, A_MN, B_MN, 1, 128, EPI, CSUM>(q, plan);
        default: return launch<T, A_MN, B_MN, 1, 64, EPI, CSUM>(q, plan);
    }
}

template <typename T>
int dispatch_layout(int ta, int tb, const Problem& q) {
    // trans_a: A stored [K,M] (M-major).  trans_b == 0: B stored [K,N] (N-major).
    if (!ta && !tb) return pick_tile<T, false, true>(q);
    if (!ta && tb) return pick_tile<T, false, false>(q);
    if (ta && !tb) return pick_tile<T, true, true>(q);
    return pick_tile<T, true, false>(q);
}

}  // namespace

bool gemm_tc_supported(int mma, int ta, int tb, int64_t M, int64_t N, int64_t K, const void* A, int64_t lda,
                       const void* B, int64_t ldb, int in_type, const void* C, int64_t ldc, int out_type) {
    (void)ta;
    (void)tb;
    if (mma != BOAT_MMA_BF16 && mma != BOAT_MMA_TF32) return false;
    const int es = mma == BOAT_MMA_BF16 ? 2 : 4;
    if ((mma == BOAT_MMA_BF16) != (in_type == BOAT_CUDA_BF16)) return false;
    const int oes = out_type == BOAT_CUDA_BF16 ? 2 : 4;
    if (M < 128 || N < 64 || K < 128 / es) return false;               // small problems: CUDA cores
    if (M > INT32_MAX || N > INT32_MAX || K > INT32_MAX) return false;
    if (((uintptr_t)A | (uintptr_t)B | (uintptr_t)C) & 15) return false;
    if ((lda * es) % 16 || (ldb * es) % 16 || (ldc * oes) % 16) return false;
    if (N % (16 / oes)) return false;
    return true;
}

int gemm_tc_grouped(int mma, int ta, int tb, int groups, int64_t M, int64_t N, int64_t K, const void* const* A,
                    int64_t lda, const void* const* B, int64_t ldb, void* const* C, int64_t ldc, int out_type,
                    const float* const* bias) {
    if (groups < 1 || groups > kMaxGroups) return set_error(11, "gemm_tc_grouped: %d groups (1..%d)", groups, kMaxGroups);
    if (int rc = ensure_init()) return rc;
    const Problem q{groups, M, N, K, A, lda, B, ldb, C, ldc, out_type, bias, false, false, nullptr, nullptr};
    return mma == BOAT_MMA_BF16 ? dispatch_layout<__nv_bfloat16>(ta, tb, q) : dispatch_layout<float>(ta, tb, q);
}

int gemm_tc_weight_grads(int mma, int groups, int64_t I, int64_t O, int64_t T, const void* const* X, const void* const* dY,
                         float* const* dW, float* const* db, bool add) {
    if (int rc = ensure_init()) return rc;
    const Problem q{groups, I, O, T, X, I, dY, O, (void* const*)dW, O, BOAT_CUDA_F32, nullptr, add, false, nullptr, db};
    typedef __nv_bfloat16 bf;
    if (!db) return mma == BOAT_MMA_BF16 ? pick_tile<bf, true, true>(q) : pick_tile<float, true, true>(q);
    return mma == BOAT_MMA_BF16 ? pick_tile<bf, true, true, BOAT_EPI_NONE, true>(q) : pick_tile<float, true, true, BOAT_EPI_NONE, true>(q);
}

int gemm_tc_sum(int mma, int ta, int tb, int groups, int64_t M, int64_t N, int64_t K, const void* const* A, int64_t lda,
                const void* const* B, int64_t ldb, void* C, int64_t ldc, int out_type) {
    if (int rc = ensure_init()) return rc;
    const Problem q{groups, M, N, K, A, lda, B, ldb, &C, ldc, out_type, nullptr, false, true, nullptr, nullptr};
    return mma == BOAT_MMA_BF16 ? dispatch_layout<__nv_bfloat16>(ta, tb, q) : dispatch_layout<float>(ta, tb, q);
}

bool gemm_tc_fused_supported(int epilogue, int ta, int tb) {
    return !ta && (epilogue == BOAT_EPI_GELU_GRAD ? tb != 0 : tb == 0);
}

int gemm_tc_fused(int epilogue, int64_t M, int64_t N, int64_t K, const void* A, int64_t lda, const void* B, int64_t ldb,
                  void* C, int64_t ldc, const float* bias, void* aux) {
    if (int rc = ensure_init()) return rc;
    const Problem q{1, M, N, K, &A, lda, &B, ldb, &C, ldc, BOAT_CUDA_BF16, &bias, false, false, aux, nullptr};
    typedef __nv_bfloat16 bf;
    if (epilogue == BOAT_EPI_GELU) return pick_tile<bf, false, true, BOAT_EPI_GELU>(q);
    if (epilogue == BOAT_EPI_ADD) return pick_tile<bf, false, true, BOAT_EPI_ADD>(q);
    return pick_tile<bf, false, false, BOAT_EPI_GELU_GRAD>(q);
}

void gemm_tc_set_yielding(bool on) { g_yielding = on; }

int gemm_tc(int mma, int ta, int tb, int64_t M, int64_t N, int64_t K, const void* A, int64_t lda, const void* B,
            int64_t ldb, int in_type, void* C, int64_t ldc, int out_type, const float* bias) {
    (void)in_type;
    return gemm_tc_grouped(mma, ta, tb, 1, M, N, K, &A, lda, &B, ldb, &C, ldc, out_type, &bias);
}

}  // namespace boatcu
