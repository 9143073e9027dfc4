// gemm_simt.cu - CUDA-core GEMM with FP32 accumulation: the exact-FP32 mode, and shapes the
// tensor-core kernels do not take.  Stands in for boat_matmul's triple loop (reference
// src/ops/linear.c:116-130).
//
// 256 threads.  A warp computes 64 x 32 outputs, 8 x 8 per lane (lanes as 8 x 4): 64 multiply-adds
// for four 16-byte shared loads, all of them free of bank conflicts, so that the FMA pipe is the bound
// and not the shared memory.  The eight warps of a CTA lie as WM x WN tiles times WK slices of K: one
// 64 x 32 output tile with eight slices keeps every warp at that ratio where a problem has too few
// outputs to give each warp its own.  Operand tiles go to shared memory exactly as they lie in global
// memory (cp.async, stages of 32 along K), whichever way that is: no transposed copy.
//
// The slices' partial tiles are added through shared memory and, where a long K is also split over
// the CTAs of a cluster, through distributed shared memory, each in a fixed order: the result does not
// vary from run to run.  The column sums of B that a bias gradient wants come from the same pass.
//
// 1000 x 256 x 256 takes 8.1 us, 4096 x 512 x 512 63 (34 TFLOP/s), 512 x 512 x 4096 (dW) 65; a register-only loop of these
// multiply-adds reaches 57 TFLOP/s.  Stages of 64 along K where a warp has an eighth of them (8 between two barriers, not 4): 8.7 -> 8.1
// us, three 512 x 512 x 4096 226 -> 198.
#include "common.cuh"
#include <cooperative_groups.h>
#include <type_traits>

namespace boatcu {

namespace {

constexpr int kMaxGroups = 4;
constexpr int kMaxSplit = 8;         // portable cluster size
constexpr int kWarpM = 64, kWarpN = 32, kWarpTile = kWarpM * kWarpN;

struct SimtParams {
    const void* A[kMaxGroups];
    const void* B[kMaxGroups];
    void* C[kMaxGroups];
    const float* bias[kMaxGroups];
    float* colsum[kMaxGroups];       // sum over K of B's columns, or NULL
    int64_t M, N, K, lda, ldb, ldc;
    int n_tiles, split;
    int vec_a, vec_b, vec_c;         // 16-byte accesses possible
    int follow;                      // how the launch follows the one before (Follow)
    int add;                         // add to C and colsum instead of overwriting them (FP32 output)
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}

// 16 bytes of shared memory of CTA `rank` of the cluster, at this CTA's shared address `at`
__device__ __forceinline__ float4 ld_cluster4(uint32_t at, int rank) {
    uint32_t there;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(at), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(there) : "memory");
    return v;
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// The tiles of one operand along K, in shared rows LD floats apart; zeros beyond the matrix.  K_ROWS: the
// operand is stored [K, X] and a tile is kBK rows of XT columns, else it is [X, K] and a tile is XT rows
// of kBK columns.  What does not change along K is worked out once: with 16-byte copies a thread keeps
// one column of every tile, so that a copy inside the matrix costs little more than itself.
template <typename T, int XT, bool K_ROWS, int LD, int kBK>
struct TileLoader {
    static constexpr int ROWS = K_ROWS ? kBK : XT, COLS = K_ROWS ? XT : kBK;
    static constexpr int PER_ROW = COLS / 4, ROW_STEP = 256 / PER_ROW;
    static_assert(ROWS % ROW_STEP == 0 && 256 % PER_ROW == 0, "whole passes");
    const T* p;                      // this thread's first element of tile 0
    uint32_t at;                     // where it goes, in bytes from the start of the shared tile
    int fixed;                       // K_ROWS: bytes of the thread's column; else rows from its first one to the matrix's end
    bool whole;                      // the tile is inside the matrix across K

    __device__ __forceinline__ TileLoader(const T* base, int64_t ld, int64_t x0, int64_t X) {
        const int r = threadIdx.x / PER_ROW, c = (threadIdx.x % PER_ROW) * 4;
        p = base + (K_ROWS ? r * ld + x0 + c : (x0 + r) * ld + c);
        const int64_t left = X - x0 - (K_ROWS ? c : r);
        at = (r * LD + c) * 4;
        whole = X - x0 >= XT;
        fixed = K_ROWS ? (int)(left >= 4 ? 16 : (left > 0 ? left * 4 : 0)) : (int)(left > XT ? XT : left);
    }
    // dst: the tile in shared memory, dst_at: the same as an address of the shared window
    __device__ __forceinline__ void fetch(float* dst, uint32_t dst_at, int step, const T* base, int64_t ld, int64_t x0, int64_t X, int64_t K, int vec) const {
        const int64_t k0 = (int64_t)step * kBK;
        if constexpr (sizeof(T) == 4) {
            if (vec) {
                const int r = threadIdx.x / PER_ROW, c = (threadIdx.x % PER_ROW) * 4;
                const T* q = p + (K_ROWS ? k0 * ld : k0);
                const uint32_t d = dst_at + at;
                if (whole && k0 + kBK <= K) {
#pragma unroll
                    for (int i = 0; i < ROWS / ROW_STEP; ++i, q += ROW_STEP * ld) cp_async16(d + i * ROW_STEP * LD * 4, q);
                    return;
                }
                const int64_t rest = K - k0 - (K_ROWS ? r : c);
                const int left = (int)(rest < kBK ? rest : kBK);
                const int tail = left >= 4 ? 16 : (left > 0 ? left * 4 : 0);
#pragma unroll 1
                for (int i = 0; i < ROWS / ROW_STEP; ++i, q += ROW_STEP * ld) {
                    const int bytes = i * ROW_STEP < (K_ROWS ? left : fixed) ? (K_ROWS ? fixed : tail) : 0;
                    cp_async16(d + i * ROW_STEP * LD * 4, bytes ? q : base, bytes);
                }
                return;
            }
        }
        const int64_t r0 = K_ROWS ? k0 : x0, c0 = K_ROWS ? x0 : k0, rows = K_ROWS ? K : X, cols = K_ROWS ? X : K;
#pragma unroll 1
        for (int e = threadIdx.x; e < ROWS * COLS; e += 256) {
            const int er = e / COLS, ec = e % COLS;
            const int64_t gr = r0 + er, gc = c0 + ec;
            const bool in = gr < rows && gc < cols;
            if constexpr (sizeof(T) == 4) cp_async4(dst + er * LD + ec, in ? base + gr * ld + gc : base, in ? 4 : 0);
            else dst[er * LD + ec] = in ? to_f32(base[gr * ld + gc]) : 0.f;
        }
    }
};

// A_M: A is stored [K, M] (contiguous along M), else [M, K].  B_K: B is stored [N, K], else [K, N].
// WM x WN warp tiles, 8 / (WM * WN) slices of K.
template <bool A_M, bool B_K, int WM, int WN>
struct SimtTile {
    static constexpr int BM = kWarpM * WM, BN = kWarpN * WN, TILES = WM * WN, WK = 8 / TILES;
    static constexpr int kBK = WK == 8 ? 64 : 32;         // K per stage
    static constexpr int LDA = A_M ? BM + 4 : kBK + 4, LDB = B_K ? kBK + 4 : BN + 4;
    static constexpr int A_FLOATS = A_M ? kBK * LDA : BM * LDA, B_FLOATS = B_K ? BN * LDB : kBK * LDB;
    static constexpr int STAGE = A_FLOATS + B_FLOATS;
    static constexpr int STAGES = WK > 1 && WK < 8 ? 4 : 3;
    static constexpr int PARTS = 8 * kWarpTile, SUMS = 8 * kWarpN;      // the partial tiles take the stages' place
    static constexpr int SMEM = (STAGES * STAGE > PARTS + SUMS ? STAGES * STAGE : PARTS + SUMS) * 4;
    static_assert(2 * (SMEM + 1024) <= 228 * 1024, "two CTAs per SM");
};

// `N` neighbouring floats of shared memory
template <int N> __device__ __forceinline__ void load_shared(float (&v)[N], const float* p) {
    if constexpr (N == 4) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
        const float2 t = *reinterpret_cast<const float2*>(p);
        v[0] = t.x; v[1] = t.y;
    }
}

// CTA `block` of problem g.  Where K is split, the blocks of one tile are the CTAs of a cluster.
template <typename TI, typename TO, bool A_M, bool B_K, int WM, int WN>
__device__ __forceinline__ void simt_tile(const SimtParams& p, int block, int g, float* smem) {
    using S = SimtTile<A_M, B_K, WM, WN>;
    constexpr int kBK = S::kBK;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lm = lane >> 2, ln = lane & 3;
    const int wk = warp / S::TILES, wm = warp % S::TILES / WN, wn = warp % WN;
    const int split = p.split;
    const int ks = block % split, tile = block / split;
    const int64_t m0 = (int64_t)(tile / p.n_tiles) * S::BM, n0 = (int64_t)(tile % p.n_tiles) * S::BN;
    const TI* A = (const TI*)p.A[g];
    const TI* B = (const TI*)p.B[g];
    const int steps = (int)((p.K + kBK - 1) / kBK);
    const int s0 = (int)((int64_t)steps * ks / split), s1 = (int)((int64_t)steps * (ks + 1) / split);
    constexpr bool kSums = A_M && !B_K;                   // a weight gradient
    const bool sums = kSums && p.colsum[g] != nullptr && m0 == 0;

    const TileLoader<TI, S::BM, A_M, S::LDA, kBK> load_a(A, p.lda, m0, p.M);
    const TileLoader<TI, S::BN, !B_K, S::LDB, kBK> load_b(B, p.ldb, n0, p.N);

    const uint32_t smem_at = (uint32_t)__cvta_generic_to_shared(smem);
    float acc[8][8], bsum = 0.f;                          // bsum: column `lane` of the warp tile
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i][j] = 0.f;
    // Rows and columns of a lane inside the warp tile: groups of four neighbours where the operand is
    // contiguous that way, strided by the lanes where it is contiguous along K, so that the lanes of a load
    // touch all banks once.
    auto row = [&](int i) { return A_M ? (i / 4) * 32 + lm * 4 + i % 4 : lm + 8 * i; };
    auto col = [&](int j) { return B_K ? ln + 4 * j : (j / 4) * 16 + ln * 4 + j % 4; };

    griddep_enter(p.follow);
    // the first rounds only fetch, so that the code of a fetch is there once
    for (int s = s0 - (S::STAGES - 1); s < s1; ++s) {
        if (s >= s0) {
            asm volatile("cp.async.wait_group %0;" ::"n"(S::STAGES - 2) : "memory");
            __syncthreads();                              // stage s has landed, stage s-1 is no longer read
        }
        const int ahead = s + S::STAGES - 1;
        if (ahead < s1) {
            const int to = ahead % S::STAGES * S::STAGE;
            load_a.fetch(smem + to, smem_at + to * 4, ahead, A, p.lda, m0, p.M, p.K, p.vec_a);
            load_b.fetch(smem + to + S::A_FLOATS, smem_at + (to + S::A_FLOATS) * 4, ahead, B, p.ldb, n0, p.N, p.K, p.vec_b);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (s < s0) continue;
        constexpr int KW = kBK / S::WK;                   // this warp's share of the stage
        const float* a_s = smem + s % S::STAGES * S::STAGE + (A_M ? (wk * KW) * S::LDA + wm * kWarpM : wm * kWarpM * S::LDA + wk * KW);
        const float* b_s = smem + s % S::STAGES * S::STAGE + S::A_FLOATS + (B_K ? wn * kWarpN * S::LDB + wk * KW : (wk * KW) * S::LDB + wn * kWarpN);
#pragma unroll(KW < 8 ? KW / 2 : 4)
        for (int k = 0; k < KW; k += 2) {
            float a[8][2], b[8][2];
            if (A_M) {
#pragma unroll
                for (int kk = 0; kk < 2; ++kk)
#pragma unroll
                    for (int i = 0; i < 8; i += 4) {
                        float t[4];
                        load_shared<4>(t, a_s + (k + kk) * S::LDA + row(i));
#pragma unroll
                        for (int u = 0; u < 4; ++u) a[i + u][kk] = t[u];
                    }
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) load_shared<2>(a[i], a_s + row(i) * S::LDA + k);
            }
            if (B_K) {
#pragma unroll
                for (int j = 0; j < 8; ++j) load_shared<2>(b[j], b_s + col(j) * S::LDB + k);
            } else {
#pragma unroll
                for (int kk = 0; kk < 2; ++kk)
#pragma unroll
                    for (int j = 0; j < 8; j += 4) {
                        float t[4];
                        load_shared<4>(t, b_s + (k + kk) * S::LDB + col(j));
#pragma unroll
                        for (int u = 0; u < 4; ++u) b[j + u][kk] = t[u];
                    }
            }
#pragma unroll
            for (int kk = 0; kk < 2; ++kk)
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i][kk], b[j][kk], acc[i][j]);
        }
        if (sums && wm == 0) {
#pragma unroll
            for (int k = 0; k < KW; ++k) bsum += b_s[k * S::LDB + lane];
        }
    }

    // Partial tiles to shared memory: one block of 64 rows of 32 floats per warp.  The 16-byte units of a
    // row are permuted by the row's lane, so that neither the lanes of a store nor those of a load meet.
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    auto unit = [&](int r, int c4) {
        const int l = A_M ? (r >> 2) & 7 : r & 7;
        return r * kWarpN + ((c4 ^ ((l & 1) << 2 | (l & 2) | l >> 2)) << 2);
    };
    float* part = smem + warp * kWarpTile;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = row(i);
        if constexpr (B_K) {
#pragma unroll
            for (int j = 0; j < 8; ++j) part[unit(r, j) + ln] = acc[i][j];
        } else {
#pragma unroll
            for (int j = 0; j < 8; j += 4)
                *reinterpret_cast<float4*>(part + unit(r, col(j) >> 2)) = make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
        }
    }
    float* sum_s = smem + S::PARTS;
    if (sums && wm == 0) sum_s[(wk * WN + wn) * kWarpN + lane] = bsum;
    __syncthreads();

    TO* C = (TO*)p.C[g];
    const float* bias = p.bias[g];
    auto put = [&](int e, float4 v) {                      // unit e of the CTA's tile, numbered as the sums below do
        const int t = e / (kWarpTile / 4), r = e / 8 % kWarpM, c4 = e % 8;
        const int64_t gm = m0 + (t / WN) * kWarpM + r, gn = n0 + (t % WN) * kWarpN + c4 * 4;
        if (gm >= p.M || gn >= p.N) return;
        TO* dst = C + gm * p.ldc + gn;
        if constexpr (sizeof(TO) == 4) {
            if (p.vec_c) {                                // N is a multiple of 4 here
                if (bias) v = add4(v, *reinterpret_cast<const float4*>(bias + gn));
                if constexpr (std::is_same<TO, float>::value) {
                    if (p.add) v = add4(*reinterpret_cast<const float4*>(dst), v);
                } else {
                    v = make_float4(round_to_tf32(v.x), round_to_tf32(v.y), round_to_tf32(v.z), round_to_tf32(v.w));
                }
                *reinterpret_cast<float4*>(dst) = v;
                return;
            }
        }
        const float out[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (gn + u >= p.N) break;
            float w = out[u] + (bias ? bias[gn + u] : 0.f);
            if constexpr (std::is_same<TO, float>::value) {
                if (p.add) w += dst[u];
            }
            dst[u] = from_f32<TO>(w);
        }
    };
    constexpr int kUnits = S::BM * S::BN / 4;
    auto sliced = [&](int e) {                             // unit e added over the slices of this CTA, where it lies in smem
        const int t = e / (kWarpTile / 4), at = unit(e / 8 % kWarpM, e % 8);
        float4 v = *reinterpret_cast<const float4*>(smem + t * kWarpTile + at);
#pragma unroll
        for (int w = 1; w < S::WK; ++w) v = add4(v, *reinterpret_cast<const float4*>(smem + (w * S::TILES + t) * kWarpTile + at));
        return v;
    };
    if (sums && tid < S::BN) {
        float v = sum_s[tid];
#pragma unroll
        for (int w = 1; w < S::WK; ++w) v += sum_s[w * S::BN + tid];
        if (split > 1) sum_s[tid] = v;
        else if (n0 + tid < p.N) p.colsum[g][n0 + tid] = v + (p.add ? p.colsum[g][n0 + tid] : 0.f);
    }
    if (split == 1) {
#pragma unroll 2
        for (int e = tid; e < kUnits; e += 256) put(e, sliced(e));
        griddep_leave(p.follow);
        return;
    }
    // every CTA of the cluster adds its share of the tile over all of them, lowest K first
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    auto place = [&](int e) { return e / (kWarpTile / 4) * kWarpTile + unit(e / 8 % kWarpM, e % 8); };
    if (S::WK > 1) {
#pragma unroll 2
        for (int e = tid; e < kUnits; e += 256) *reinterpret_cast<float4*>(smem + place(e)) = sliced(e);
    }
    cluster.sync();
    auto over_cluster = [&](int at) {
        float4 t[kMaxSplit];
#pragma unroll
        for (int r = 0; r < kMaxSplit; ++r)
            if (r < split) t[r] = ld_cluster4(smem_at + at * 4, r);
        float4 v = t[0];
#pragma unroll
        for (int r = 1; r < kMaxSplit; ++r)
            if (r < split) v = add4(v, t[r]);
        return v;
    };
    for (int e = ks * 256 + tid; e < kUnits; e += split * 256) put(e, over_cluster(place(e)));
    if (sums && ks == 0 && tid < S::BN / 4) {
        const float4 v = over_cluster(S::PARTS + tid * 4);
        const float out[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t gn = n0 + tid * 4 + u;
            if (gn < p.N) p.colsum[g][gn] = out[u] + (p.add ? p.colsum[g][gn] : 0.f);
        }
    }
    cluster.sync();                                       // nobody leaves while its partial tile is being read
    griddep_leave(p.follow);
}

template <typename TI, typename TO, bool A_M, bool B_K, int WM, int WN>
__global__ void __launch_bounds__(256, 2)
gemm_simt_kernel(const __grid_constant__ SimtParams p) {
    extern __shared__ __align__(16) float smem[];
    simt_tile<TI, TO, A_M, B_K, WM, WN>(p, blockIdx.x, blockIdx.z, smem);
}

// The weight gradients of a few small projections and, behind them, their input gradients, which read the same dY: one
// launch instead of two.  dw_blocks, dx_blocks: CTAs per group.
__global__ void __launch_bounds__(256, 2)
gemm_simt_grads_kernel(const __grid_constant__ SimtParams dw, const __grid_constant__ SimtParams dx, int groups, int dw_blocks, int dx_blocks) {
    extern __shared__ __align__(16) float smem[];
    int b = blockIdx.x;
    if (b < groups * dw_blocks) {
        simt_tile<float, float, true, false, 1, 1>(dw, b % dw_blocks, b / dw_blocks, smem);
        return;
    }
    b -= groups * dw_blocks;
    if (b < groups * dx_blocks) simt_tile<float, float, false, true, 1, 1>(dx, b % dx_blocks, b / dx_blocks, smem);
}

void name_memory(LaunchTurn& turn, const SimtParams& p, int groups, bool a_m, bool b_k, size_t in_size, size_t out_size) {
    for (int g = 0; g < groups; ++g) {
        turn.reads(p.A[g], a_m ? p.K : p.M, a_m ? p.M : p.K, p.lda, in_size);
        turn.reads(p.B[g], b_k ? p.N : p.K, b_k ? p.K : p.N, p.ldb, in_size);
        turn.writes(p.C[g], p.M, p.N, p.ldc, out_size);
        turn.reads(p.bias[g], (size_t)p.N * 4);
        turn.writes(p.colsum[g], (size_t)p.N * 4);
    }
}

template <typename TI, typename TO, bool A_M, bool B_K, int WM, int WN>
int launch_tile(SimtParams& p, int groups, int split) {
    using S = SimtTile<A_M, B_K, WM, WN>;
    auto kern = gemm_simt_kernel<TI, TO, A_M, B_K, WM, WN>;
    static bool configured = false;      // per process = per device: the library binds to one device
    if (!configured) {
        BOATCU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM > kSpreadSmem ? S::SMEM : kSpreadSmem));
        configured = true;
    }
    const int64_t tiles = ceil_div(p.M, S::BM) * ceil_div(p.N, S::BN);
    if (tiles * split > 0x7fffffffLL) return set_error(7, "gemm_simt: %lld x %lld outputs are too many for one launch", (long long)p.M, (long long)p.N);
    p.n_tiles = (int)ceil_div(p.N, S::BN);
    p.split = split;
    const int smem = spread_smem(S::SMEM, tiles * split * groups);
    {
        LaunchTurn turn;
        name_memory(turn, p, groups, A_M, B_K, sizeof(TI), sizeof(TO));
        p.follow = turn.follow();
        BOATCU_CHECK(launch_in_turn(turn, kern, dim3((unsigned)(tiles * split), 1, (unsigned)groups), dim3(256), smem, (unsigned)split, p));
    }
    BOATCU_LAUNCH_OK("gemm_simt");
    return 0;
}

struct Choice { int wm, wn, split; };

// Tile and split of K for an M x N x K problem; fp32: FP32 in and out.
Choice choose(int64_t M, int64_t N, int64_t K, bool fp32) {
    const int64_t sms = sm_count();
    auto tiles = [&](int bm, int bn) { return ceil_div(M, bm) * ceil_div(N, bn); };
    // Larger tiles fetch less per product, smaller ones leave no SM idle.  128 x 128 pays from three quarters of the SMs on (4096 x
    // 512 x 512, 128 of them: 63 us, 64 x 64 74; three such 175 and 202), 128 x 64 from six tenths (3000 x 256 x 256, 96: 19.8 and 21.0;
    // three 34.9 and 40.8; but 1000 x 256 x 256, 32 of them: 20, 64 x 32 8.1).  Where 64 x 64 does not fill the GPU but does so with K cut
    // in up to four, and 512 of it for each CTA of the cluster, that is next (512 x 512 x 4096 65 us, 64 x 32 69).  Else 64 x 32 with K
    // split over a cluster, at least 64 of it per CTA - and into two CTAs per SM where each still has 512: eight warps alone wait for
    // one another's loads.  The order of the sum goes by the size of one problem alone, so that a group gives the bits of single
    // calls.
    if (fp32 && tiles(128, 128) * 4 >= sms * 3) return {2, 4, 1};
    if (fp32 && tiles(128, 64) * 10 >= sms * 6) return {2, 2, 1};
    if (tiles(64, 64) >= sms) return {1, 2, 1};
    const int in = tiles(64, 64) * 2 >= sms ? 2 : 4;
    if (tiles(64, 64) * in >= sms && K / in >= 512) return {1, 2, in};
    int64_t split = sms / tiles(64, 32);
    const int64_t two = 2 * sms / tiles(64, 32) < K / 512 ? 2 * sms / tiles(64, 32) : K / 512;
    if (split < two) split = two;
    if (split > K / 64) split = K / 64;
    if (split > kMaxSplit) split = kMaxSplit;
    if (split < 1) split = 1;
    return {1, 1, (int)split};
}

template <typename TI, typename TO, bool A_M, bool B_K>
int pick_tile(SimtParams& p, int groups) {
    constexpr bool fp32 = std::is_same<TI, float>::value && std::is_same<TO, float>::value;
    const Choice c = choose(p.M, p.N, p.K, fp32);
    if constexpr (fp32) {
        if (c.wm == 2 && c.wn == 4) return launch_tile<TI, TO, A_M, B_K, 2, 4>(p, groups, 1);
        if (c.wm == 2) return launch_tile<TI, TO, A_M, B_K, 2, 2>(p, groups, 1);
    }
    if (c.wn == 2) return launch_tile<TI, TO, A_M, B_K, 1, 2>(p, groups, c.split);
    return launch_tile<TI, TO, A_M, B_K, 1, 1>(p, groups, c.split);
}

template <typename TI, typename TO>
int pick_layout(SimtParams& p, int groups, int ta, int tb) {
    if (!ta && !tb) return pick_tile<TI, TO, false, false>(p, groups);
    if (!ta && tb) return pick_tile<TI, TO, false, true>(p, groups);
    if (ta && !tb) return pick_tile<TI, TO, true, false>(p, groups);
    return pick_tile<TI, TO, true, true>(p, groups);
}

SimtParams make_params(int groups, int64_t M, int64_t N, int64_t K, const void* const* A, int64_t lda, const void* const* B, int64_t ldb,
                       void* const* C, int64_t ldc, const float* const* bias, float* const* colsum, bool add) {
    SimtParams p;
    p.M = M; p.N = N; p.K = K; p.lda = lda; p.ldb = ldb; p.ldc = ldc;
    p.add = add ? 1 : 0;
    p.vec_a = lda % 4 == 0;
    p.vec_b = ldb % 4 == 0;
    p.vec_c = ldc % 4 == 0 && N % 4 == 0;
    for (int g = 0; g < kMaxGroups; ++g) {
        const int s = g < groups ? g : 0;
        p.A[g] = A[s];
        p.B[g] = B[s];
        p.C[g] = C[s];
        p.bias[g] = bias ? bias[s] : nullptr;
        p.colsum[g] = colsum ? colsum[s] : nullptr;
        p.vec_a = p.vec_a && ((uintptr_t)A[s] & 15) == 0;
        p.vec_b = p.vec_b && ((uintptr_t)B[s] & 15) == 0;
        p.vec_c = p.vec_c && (((uintptr_t)C[s] | (uintptr_t)p.bias[g]) & 15) == 0;
    }
    return p;
}

}  // namespace

int gemm_simt_grouped(int ta, int tb, int groups, int64_t M, int64_t N, int64_t K, const void* const* A, int64_t lda,
                      const void* const* B, int64_t ldb, int in_type, void* const* C, int64_t ldc, int out_type,
                      const float* const* bias, float* const* colsum, bool add) {
    if (M <= 0 || N <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    SimtParams p = make_params(groups, M, N, K, A, lda, B, ldb, C, ldc, bias, colsum, add);
    typedef __nv_bfloat16 bf;
    const bool bf_in = in_type == BOAT_CUDA_BF16;
    if (out_type == BOAT_CUDA_F32_TF32)
        return bf_in ? pick_layout<bf, f32_tf32>(p, groups, ta, tb) : pick_layout<float, f32_tf32>(p, groups, ta, tb);
    if (out_type == BOAT_CUDA_F32)
        return bf_in ? pick_layout<bf, float>(p, groups, ta, tb) : pick_layout<float, float>(p, groups, ta, tb);
    return bf_in ? pick_layout<bf, bf>(p, groups, ta, tb) : pick_layout<float, bf>(p, groups, ta, tb);
}

int gemm_simt_grads(int groups, int64_t T, int64_t I, int64_t O, const void* const* X, const void* const* dY, const void* const* W,
                    void* const* dX, float* const* dW, float* const* db) {
    if (int rc = ensure_init()) return rc;
    const Choice cw = choose(I, O, T, true), cx = choose(T, I, O, true);
    const int64_t dw_blocks = ceil_div(I, kWarpM) * ceil_div(O, kWarpN) * cw.split, dx_blocks = ceil_div(T, kWarpM) * ceil_div(I, kWarpN);
    // Both of them small tiles, and an SM for every CTA: what it costs to launch is then most of the cost.  (2 x 64 tokens of width
    // 64, 12 CTAs each: the host's part of a layer's backward 17.9 us, 11.8 with both pairs in one launch; the step 42.3 and 36.5.)
    if (cw.wn != 1 || cx.wn != 1 || cx.split != 1 || groups * (dw_blocks + dx_blocks) > sm_count()) return 13;
    SimtParams w = make_params(groups, I, O, T, X, I, dY, O, (void* const*)dW, O, nullptr, db, false);
    SimtParams x = make_params(groups, T, I, O, dY, O, W, O, dX, I, nullptr, nullptr, false);
    w.n_tiles = (int)ceil_div(O, kWarpN);
    w.split = cw.split;
    x.n_tiles = (int)ceil_div(I, kWarpN);
    x.split = 1;
    using Sw = SimtTile<true, false, 1, 1>;
    using Sx = SimtTile<false, true, 1, 1>;
    constexpr int need = Sw::SMEM > Sx::SMEM ? Sw::SMEM : Sx::SMEM;
    static bool configured = false;      // per process = per device: the library binds to one device
    if (!configured) {
        BOATCU_CHECK(cudaFuncSetAttribute(gemm_simt_grads_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, need > kSpreadSmem ? need : kSpreadSmem));
        configured = true;
    }
    const int64_t grid = ceil_div(groups * (dw_blocks + dx_blocks), cw.split) * cw.split;       // whole clusters
    LaunchTurn turn;
    name_memory(turn, w, groups, true, false, 4, 4);
    name_memory(turn, x, groups, false, true, 4, 4);
    w.follow = x.follow = turn.follow();
    BOATCU_CHECK(launch_in_turn(turn, gemm_simt_grads_kernel, dim3((unsigned)grid), dim3(256), spread_smem(need, grid), (unsigned)cw.split, w, x, groups,
                                (int)dw_blocks, (int)dx_blocks));
    BOATCU_LAUNCH_OK("gemm_simt_grads");
    return 0;
}

}  // namespace boatcu
