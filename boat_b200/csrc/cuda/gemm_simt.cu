// gemm_simt.cu - CUDA-core GEMM with FP32 accumulation: the exact-FP32 mode, and shapes the
// tensor-core kernels do not take.  Stands in for boat_matmul's triple loop (reference
// src/ops/linear.c:116-130).
//
// 256 threads as 16 x 16, TM x TN outputs each.  Operand tiles go to shared memory exactly as they
// lie in global memory (cp.async, three stages of 32 along K), whichever way that is: four steps
// of K are multiplied at a time, an operand that is contiguous along K is read as one 16-byte load
// per row and four steps, one that is contiguous along M or N as one 16-byte load per step and four
// rows.  No transposed copy, no bank conflict either way (K-contiguous rows are 36 floats apart, so
// 8 lanes on 8 rows cover all banks).  Every output is one chain of fused multiply-adds in ascending
// K, as before.
//
// Small outputs with a long K (weight gradients) are split along K over the CTAs of a cluster, which
// add their partial tiles through distributed shared memory in a fixed order: the result does not
// vary from run to run.  The columns sums of B that a bias gradient wants come from the same pass.
#include "common.cuh"
#include <cooperative_groups.h>
#include <type_traits>

namespace boatcu {

namespace {

constexpr int kBK = 32;              // K per stage
constexpr int kStages = 3;
constexpr int kMaxGroups = 4;
constexpr int kMaxSplit = 8;         // portable cluster size

struct SimtParams {
    const void* A[kMaxGroups];
    const void* B[kMaxGroups];
    void* C[kMaxGroups];
    const float* bias[kMaxGroups];
    float* colsum[kMaxGroups];       // sum over K of B's columns, or NULL
    int64_t M, N, K, lda, ldb, ldc;
    int n_tiles, split;
    int vec_a, vec_b, vec_c;         // 16-byte accesses possible
    int add;                         // add to C and colsum instead of overwriting them (FP32 output)
};

__device__ __forceinline__ void cp_async16(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}

// A tile of `ROWS` rows of `COLS` contiguous elements, from row r0 and column c0 of a [rows, cols]
// matrix, to shared rows LD floats apart; zeros beyond the matrix.
template <int ROWS, int COLS, int LD>
__device__ __forceinline__ void load_tile(float* dst, const float* src, int64_t ld, int64_t r0, int64_t c0, int64_t rows,
                                          int64_t cols, int vec) {
    if (vec) {
#pragma unroll
        for (int e = threadIdx.x; e < ROWS * COLS / 4; e += 256) {
            const int r = e / (COLS / 4), c = (e % (COLS / 4)) * 4;
            const int64_t gr = r0 + r, gc = c0 + c, left = gr < rows ? cols - gc : 0;
            const int bytes = left >= 4 ? 16 : (left > 0 ? (int)left * 4 : 0);
            cp_async16(dst + r * LD + c, bytes ? src + gr * ld + gc : src, bytes);
        }
    } else {
#pragma unroll 4
        for (int e = threadIdx.x; e < ROWS * COLS; e += 256) {
            const int r = e / COLS, c = e % COLS;
            const int64_t gr = r0 + r, gc = c0 + c;
            const bool in = gr < rows && gc < cols;
            cp_async4(dst + r * LD + c, in ? src + gr * ld + gc : src, in ? 4 : 0);
        }
    }
}
template <int ROWS, int COLS, int LD>
__device__ __forceinline__ void load_tile(float* dst, const __nv_bfloat16* src, int64_t ld, int64_t r0, int64_t c0,
                                          int64_t rows, int64_t cols, int vec) {
    (void)vec;
#pragma unroll 4
    for (int e = threadIdx.x; e < ROWS * COLS; e += 256) {
        const int r = e / COLS, c = e % COLS;
        const int64_t gr = r0 + r, gc = c0 + c;
        dst[r * LD + c] = gr < rows && gc < cols ? to_f32(src[gr * ld + gc]) : 0.f;
    }
}

// A_M: A is stored [K, M] (contiguous along M), else [M, K].  B_K: B is stored [N, K], else [K, N].
template <bool A_M, bool B_K, int TM, int TN>
struct SimtTile {
    static constexpr int BM = 16 * TM, BN = 16 * TN;
    static constexpr int LDA = A_M ? BM + 4 : kBK + 4, LDB = B_K ? kBK + 4 : BN + 4;
    static constexpr int A_FLOATS = A_M ? kBK * LDA : BM * LDA, B_FLOATS = B_K ? BN * LDB : kBK * LDB;
    static constexpr int STAGE = A_FLOATS + B_FLOATS;
    static constexpr int SMEM = kStages * STAGE * 4;
    static_assert(BM * BN + BN <= kStages * STAGE, "the partial tile must fit the stages");
};

template <typename TI, typename TO, bool A_M, bool B_K, int TM, int TN>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const __grid_constant__ SimtParams p) {
    using S = SimtTile<A_M, B_K, TM, TN>;
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int g = blockIdx.z, split = p.split;
    const int ks = blockIdx.x % split, tile = blockIdx.x / split;
    const int64_t m0 = (int64_t)(tile / p.n_tiles) * S::BM, n0 = (int64_t)(tile % p.n_tiles) * S::BN;
    const TI* A = (const TI*)p.A[g];
    const TI* B = (const TI*)p.B[g];
    const int steps = (int)((p.K + kBK - 1) / kBK);
    const int s0 = (int)((int64_t)steps * ks / split), s1 = (int)((int64_t)steps * (ks + 1) / split);
    const bool sums = p.colsum[g] != nullptr && m0 == 0;

    auto fetch = [&](int s) {
        if (s < s1) {
            float* a = smem + (s % kStages) * S::STAGE;
            const int64_t k0 = (int64_t)s * kBK;
            if (A_M) load_tile<kBK, S::BM, S::LDA>(a, A, p.lda, k0, m0, p.K, p.M, p.vec_a);
            else     load_tile<S::BM, kBK, S::LDA>(a, A, p.lda, m0, k0, p.M, p.K, p.vec_a);
            if (B_K) load_tile<S::BN, kBK, S::LDB>(a + S::A_FLOATS, B, p.ldb, n0, k0, p.N, p.K, p.vec_b);
            else     load_tile<kBK, S::BN, S::LDB>(a + S::A_FLOATS, B, p.ldb, k0, n0, p.K, p.N, p.vec_b);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float acc[TM][TN], bsum[TN];
#pragma unroll
    for (int j = 0; j < TN; ++j) {
        bsum[j] = 0.f;
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = 0.f;
    }
    // Rows of this thread: ty*TM + i.  Columns: with B contiguous along N groups of min(TN,4) neighbours,
    // with B contiguous along K tx + 16*j (neighbouring lanes on neighbouring shared rows).
    constexpr int VN = TN < 4 ? TN : 4, VM = TM < 4 ? TM : 4;
    auto col = [&](int j) { return B_K ? tx + 16 * j : (j / VN) * 16 * VN + tx * VN + j % VN; };
    auto row = [&](int i) { return (i / VM) * 16 * VM + ty * VM + i % VM; };

    griddep_sync();
    fetch(s0);
    fetch(s0 + 1);
    for (int s = s0; s < s1; ++s) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                  // stage s has landed, stage s-1 is no longer read
        fetch(s + 2);
        const float* a_s = smem + (s % kStages) * S::STAGE;
        const float* b_s = a_s + S::A_FLOATS;
#pragma unroll
        for (int k = 0; k < kBK; k += 4) {
            float a[TM][4], b[4][TN];
            if (A_M) {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                    for (int i = 0; i < TM; i += VM) {
                        const float* q = a_s + (k + kk) * S::LDA + row(i);
                        if constexpr (VM == 4) {
                            const float4 v = *reinterpret_cast<const float4*>(q);
                            a[i][kk] = v.x; a[i + 1][kk] = v.y; a[i + 2][kk] = v.z; a[i + 3][kk] = v.w;
                        } else {
#pragma unroll
                            for (int u = 0; u < VM; ++u) a[i + u][kk] = q[u];
                        }
                    }
            } else {
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float4 v = *reinterpret_cast<const float4*>(a_s + row(i) * S::LDA + k);
                    a[i][0] = v.x; a[i][1] = v.y; a[i][2] = v.z; a[i][3] = v.w;
                }
            }
            if (B_K) {
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const float4 v = *reinterpret_cast<const float4*>(b_s + col(j) * S::LDB + k);
                    b[0][j] = v.x; b[1][j] = v.y; b[2][j] = v.z; b[3][j] = v.w;
                }
            } else {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                    for (int j = 0; j < TN; j += VN) {
                        const float* q = b_s + (k + kk) * S::LDB + col(j);
                        if constexpr (VN == 4) {
                            const float4 v = *reinterpret_cast<const float4*>(q);
                            b[kk][j] = v.x; b[kk][j + 1] = v.y; b[kk][j + 2] = v.z; b[kk][j + 3] = v.w;
                        } else {
#pragma unroll
                            for (int u = 0; u < VN; ++u) b[kk][j + u] = q[u];
                        }
                    }
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i][kk], b[kk][j], acc[i][j]);
            if (sums) {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                    for (int j = 0; j < TN; ++j) bsum[j] += b[kk][j];
            }
        }
    }

    TO* C = (TO*)p.C[g];
    const float* bias = p.bias[g];
    auto put = [&](TO* dst, float v) {
        if constexpr (std::is_same<TO, float>::value) {
            if (p.add) v += *dst;
        }
        *dst = from_f32<TO>(v);
    };
    if (split == 1) {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int64_t gm = m0 + row(i);
            if (gm >= p.M) continue;
            if constexpr (!B_K && VN == 4 && sizeof(TO) == 4) {
                if (p.vec_c) {
#pragma unroll
                    for (int j = 0; j < TN; j += 4) {
                        const int64_t gn = n0 + col(j);
                        if (gn >= p.N) continue;              // N is a multiple of 4 here
                        float4 v = make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
                        if (bias) {
                            const float4 t = *reinterpret_cast<const float4*>(bias + gn);
                            v = make_float4(v.x + t.x, v.y + t.y, v.z + t.z, v.w + t.w);
                        }
                        if constexpr (!std::is_same<TO, float>::value)
                            v = make_float4(round_to_tf32(v.x), round_to_tf32(v.y), round_to_tf32(v.z), round_to_tf32(v.w));
                        float4* dst = reinterpret_cast<float4*>(C + gm * p.ldc + gn);
                        if (p.add) {
                            const float4 t = *dst;
                            v = make_float4(t.x + v.x, t.y + v.y, t.z + v.z, t.w + v.w);
                        }
                        *dst = v;
                    }
                    continue;
                }
            }
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int64_t gn = n0 + col(j);
                if (gn < p.N) put(C + gm * p.ldc + gn, acc[i][j] + (bias ? bias[gn] : 0.f));
            }
        }
        if (sums && ty == 0) {
#pragma unroll
            for (int j = 0; j < TN; ++j)
                if (n0 + col(j) < p.N) p.colsum[g][n0 + col(j)] = bsum[j] + (p.add ? p.colsum[g][n0 + col(j)] : 0.f);
        }
        return;
    }
    // Partial tiles to shared memory, then every CTA of the cluster adds its share of the tile over
    // all of them, lowest K first.
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) smem[row(i) * S::BN + col(j)] = acc[i][j];
    if (sums && ty == 0) {
#pragma unroll
        for (int j = 0; j < TN; ++j) smem[S::BM * S::BN + col(j)] = bsum[j];
    }
    cluster.sync();
    const float* part[kMaxSplit];
#pragma unroll
    for (int r = 0; r < kMaxSplit; ++r) part[r] = cluster.map_shared_rank(smem, r < split ? r : 0);
    const int total = S::BM * S::BN + (sums ? S::BN : 0);
    for (int e = ks * 256 + tid; e < total; e += split * 256) {
        float v = part[0][e];
#pragma unroll
        for (int r = 1; r < kMaxSplit; ++r)
            if (r < split) v += part[r][e];
        const int64_t gn = n0 + e % S::BN;
        if (gn >= p.N) continue;
        if (e >= S::BM * S::BN) {
            p.colsum[g][gn] = v + (p.add ? p.colsum[g][gn] : 0.f);
        } else {
            const int64_t gm = m0 + e / S::BN;
            if (gm < p.M) put(C + gm * p.ldc + gn, v + (bias ? bias[gn] : 0.f));
        }
    }
    cluster.sync();                                       // nobody leaves while its partial tile is being read
}

template <typename TI, typename TO, bool A_M, bool B_K, int TM, int TN>
int launch_tile(SimtParams& p, int groups, int split) {
    using S = SimtTile<A_M, B_K, TM, TN>;
    auto kern = gemm_simt_kernel<TI, TO, A_M, B_K, TM, TN>;
    static bool configured = false;      // per process = per device: the library binds to one device
    if (!configured) {
        BOATCU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM));
        configured = true;
    }
    const int64_t tiles = ceil_div(p.M, S::BM) * ceil_div(p.N, S::BN);
    if (tiles * split > 0x7fffffffLL) return set_error(7, "gemm_simt: %lld x %lld outputs are too many for one launch", (long long)p.M, (long long)p.N);
    p.n_tiles = (int)ceil_div(p.N, S::BN);
    p.split = split;
    BOATCU_CHECK(launch_dependent(kern, dim3((unsigned)(tiles * split), 1, (unsigned)groups), dim3(256), S::SMEM, (unsigned)split, p));
    BOATCU_LAUNCH_OK("gemm_simt");
    return 0;
}

template <typename TI, typename TO, bool A_M, bool B_K>
int pick_tile(SimtParams& p, int groups) {
    const int64_t sms = sm_count();
    auto tiles = [&](int bm, int bn) { return ceil_div(p.M, bm) * ceil_div(p.N, bn); };
    // 128 x 128 tiles (64 outputs per thread, bound by the FMA pipe) once they fill the GPU;
    // 64 x 64 (bound by shared memory at about half that rate) with K split over a cluster while
    // SMs would stay idle, at least 64 of K per CTA; 32 x 32 for outputs so small that even so
    // most SMs would have nothing.  The split - the order of the sum - goes by the size of one problem
    // alone, so that a group gives the bits of single calls.
    const int64_t t64 = tiles(64, 64);
    int64_t split = sms / t64;
    if (split > p.K / 64) split = p.K / 64;
    if (split > kMaxSplit) split = kMaxSplit;
    if (split < 1) split = 1;
    if constexpr (std::is_same<TI, float>::value && std::is_same<TO, float>::value)
        if (split == 1 && tiles(128, 128) * groups >= sms) return launch_tile<TI, TO, A_M, B_K, 8, 8>(p, groups, 1);
    if (split == 1 && t64 * groups * 4 <= sms) return launch_tile<TI, TO, A_M, B_K, 2, 2>(p, groups, 1);
    return launch_tile<TI, TO, A_M, B_K, 4, 4>(p, groups, (int)split);
}

template <typename TI, typename TO>
int pick_layout(SimtParams& p, int groups, int ta, int tb) {
    if (!ta && !tb) return pick_tile<TI, TO, false, false>(p, groups);
    if (!ta && tb) return pick_tile<TI, TO, false, true>(p, groups);
    if (ta && !tb) return pick_tile<TI, TO, true, false>(p, groups);
    return pick_tile<TI, TO, true, true>(p, groups);
}

}  // namespace

int gemm_simt_grouped(int ta, int tb, int groups, int64_t M, int64_t N, int64_t K, const void* const* A, int64_t lda,
                      const void* const* B, int64_t ldb, int in_type, void* const* C, int64_t ldc, int out_type,
                      const float* const* bias, float* const* colsum, bool add) {
    if (M <= 0 || N <= 0) return 0;
    if (int rc = ensure_init()) return rc;
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
    typedef __nv_bfloat16 bf;
    const bool bf_in = in_type == BOAT_CUDA_BF16;
    if (out_type == BOAT_CUDA_F32_TF32)
        return bf_in ? pick_layout<bf, f32_tf32>(p, groups, ta, tb) : pick_layout<float, f32_tf32>(p, groups, ta, tb);
    if (out_type == BOAT_CUDA_F32)
        return bf_in ? pick_layout<bf, float>(p, groups, ta, tb) : pick_layout<float, float>(p, groups, ta, tb);
    return bf_in ? pick_layout<bf, bf>(p, groups, ta, tb) : pick_layout<float, bf>(p, groups, ta, tb);
}

}  // namespace boatcu
