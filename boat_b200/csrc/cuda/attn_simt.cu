// attn_simt.cu - CUDA-core attention core, forward and backward, FP32 arithmetic, any sequence
// length and head size up to 128.
//
// Restates scaled_dot_product_attention_impl (reference src/layers/attention.c:997-1073)
// and attention_backward (attention.c:1421-1526) for the exact-FP32 mode and for shapes
// outside the tensor-core kernels.  The S x S matrices are never written to memory:
// probabilities are rebuilt from the saved log-sum-exp.
//
// A CTA of 16 threads per 4 rows owns 64 rows - or 32, with half the threads, where 64 would leave SMs
// without a CTA - and walks the other side in tiles of 64 rows.  A score tile is 4 x 4 per thread, contracted along the head dimension with 16-byte shared loads of four
// elements; rows are HS+4 floats apart, so 8 lanes on 8 rows touch all banks once.  The tile's rows
// stay with the 16 lanes that made them - soft-max statistics are shuffles, and the products with the
// probabilities (P.V, dS.K, P^T.dO, dS^T.Q) read rows which the same half warp wrote: a walk has one CTA
// barrier per tile.  The next tile is fetched (cp.async) while the current one is worked on.
//
// Backward: one launch holds CTAs that own query rows (dQ) and CTAs that own key rows (dK, dV).  Both
// rebuild the scores they need - seven products per tile pair instead of five - and nothing is summed
// between CTAs, so results do not vary from run to run.  The two kinds are the same walk:
//   own = Q, dO, walk = K, V:   S = own0.walk0^T   dP = own1.walk1^T   dQ += dS.walk0
//   own = K, V,  walk = Q, dO:  the same, transposed             dK += dS^T.walk0   dV += P^T.walk1
#include "common.cuh"
#include <float.h>

namespace boatcu {

namespace {

constexpr int kRows = 64;             // rows per walked tile
constexpr int kLdP = kRows + 4;       // shared row pitch of a probability tile

// OWN: rows a CTA owns (64 or 32)
template <int HS, int OWN>
struct Tiles {
    static constexpr int LD = HS + 4;
    static constexpr int THREADS = OWN * 4;
    static constexpr int OWN_FLOATS = OWN * LD;
    static constexpr int FLOATS = kRows * LD;
    static constexpr int CPT = HS / 16;                  // output columns per thread
    static constexpr int BUFS = HS <= 64 ? 2 : 1;        // walked tiles in flight
    static constexpr int FWD_SMEM = (OWN_FLOATS + FLOATS * 2 * BUFS + OWN * kLdP) * 4;
    static constexpr int BWD_SMEM = (OWN_FLOATS * 2 + FLOATS * 2 * BUFS + 2 * OWN * kLdP + 2 * 2 * kRows) * 4;
    static_assert(BWD_SMEM <= 227 * 1024, "shared memory budget");
};

// Rows r0..r0+ROWS-1 of a [S, hs] matrix to shared rows LD apart; zeros beyond S and from hs to HS.
template <int HS, int ROWS, int THREADS>
__device__ __forceinline__ void load_rows(float* dst, const float* src, int r0, int S, int hs, bool vec) {
    if (vec) {
#pragma unroll
        for (int e = threadIdx.x; e < ROWS * HS / 4; e += THREADS) {
            const int r = e / (HS / 4), c = (e % (HS / 4)) * 4;
            const bool in = r0 + r < S && c < hs;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + r * (HS + 4) + c)),
                         "l"(in ? src + (int64_t)(r0 + r) * hs + c : src), "r"(in ? 16 : 0) : "memory");
        }
    } else {
        for (int e = threadIdx.x; e < ROWS * HS; e += THREADS) {
            const int r = e / HS, c = e % HS;
            const bool in = r0 + r < S && c < hs;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + r * (HS + 4) + c)),
                         "l"(in ? src + (int64_t)(r0 + r) * hs + c : src), "r"(in ? 4 : 0) : "memory");
        }
    }
}
template <int HS, int ROWS, int THREADS>
__device__ __forceinline__ void load_rows(float* dst, const __nv_bfloat16* src, int r0, int S, int hs, bool vec) {
    if (vec) {
#pragma unroll 4
        for (int e = threadIdx.x; e < ROWS * HS / 4; e += THREADS) {
            const int r = e / (HS / 4), c = (e % (HS / 4)) * 4;
            uint2 v = make_uint2(0u, 0u);
            if (r0 + r < S && c < hs) v = *reinterpret_cast<const uint2*>(src + (int64_t)(r0 + r) * hs + c);
            const float2 lo = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&v.x));
            const float2 hi = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&v.y));
            *reinterpret_cast<float4*>(dst + r * (HS + 4) + c) = make_float4(lo.x, lo.y, hi.x, hi.y);
        }
    } else {
        for (int e = threadIdx.x; e < ROWS * HS; e += THREADS) {
            const int r = e / HS, c = e % HS;
            dst[r * (HS + 4) + c] = r0 + r < S && c < hs ? to_f32(src[(int64_t)(r0 + r) * hs + c]) : 0.f;
        }
    }
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// s[i][j] = sum_d A[ty*4+i][d] * B[tx+16j][d], ascending d
template <int HS>
__device__ __forceinline__ void scores(const float* A, const float* B, int ty, int tx, float (&s)[4][4]) {
    constexpr int LD = HS + 4;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
    for (int d = 0; d < HS; d += 4) {
        float4 a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(A + (ty * 4 + i) * LD + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(B + (tx + 16 * j) * LD + d);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[i][j] = fmaf(a[i].x, b[j].x, s[i][j]);
                s[i][j] = fmaf(a[i].y, b[j].y, s[i][j]);
                s[i][j] = fmaf(a[i].z, b[j].z, s[i][j]);
                s[i][j] = fmaf(a[i].w, b[j].w, s[i][j]);
            }
    }
}

// First output column of group u (min(CPT,4) columns each) of a thread
template <int HS> __device__ __forceinline__ int out_col(int tx, int u) {
    constexpr int CPT = HS / 16, V = CPT < 4 ? CPT : 4;
    return u * 16 * V + tx * V;
}

// acc[i][:] += sum_k P[ty*4+i][k] * X[k][cols of this thread], ascending k
template <int HS>
__device__ __forceinline__ void accumulate(const float* P, const float* X, int ty, int tx, float (&acc)[4][HS / 16]) {
    constexpr int LD = HS + 4, CPT = HS / 16, V = CPT < 4 ? CPT : 4;
#pragma unroll 4
    for (int k = 0; k < kRows; k += 4) {
        float p[4][4], x[4][CPT];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 t = *reinterpret_cast<const float4*>(P + (ty * 4 + i) * kLdP + k);
            p[i][0] = t.x; p[i][1] = t.y; p[i][2] = t.z; p[i][3] = t.w;
        }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int u = 0; u < CPT / V; ++u) {
                const float* q = X + (k + kk) * LD + out_col<HS>(tx, u);
                if constexpr (V == 4) {
                    const float4 t = *reinterpret_cast<const float4*>(q);
                    x[kk][4 * u] = t.x; x[kk][4 * u + 1] = t.y; x[kk][4 * u + 2] = t.z; x[kk][4 * u + 3] = t.w;
                } else {
#pragma unroll
                    for (int v = 0; v < V; ++v) x[kk][v] = q[v];
                }
            }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int c = 0; c < CPT; ++c) acc[i][c] = fmaf(p[i][kk], x[kk][c], acc[i][c]);
    }
}

template <int HS, typename T>
__device__ __forceinline__ void store_rows(T* dst, int r0, int S, int hs, int ty, int tx, const float (&acc)[4][HS / 16]) {
    constexpr int CPT = HS / 16, V = CPT < 4 ? CPT : 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = r0 + ty * 4 + i;
        if (r >= S) continue;
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
            const int d = out_col<HS>(tx, c / V) + c % V;
            if (d < hs) dst[(int64_t)r * hs + d] = from_f32<T>(acc[i][c]);
        }
    }
}

// reductions over the 16 lanes that share a row
__device__ __forceinline__ float row_max(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---- forward -----------------------------------------------------------------------------------
template <int HS, int OWN, typename T>
__global__ void __launch_bounds__(OWN * 4)
attn_fwd_simt_kernel(int units, int S, int hs, int causal, float scale, int vec, const T* __restrict__ Q,
                     const T* __restrict__ K, const T* __restrict__ V, T* __restrict__ O, float* __restrict__ lse) {
    using C = Tiles<HS, OWN>;
    extern __shared__ __align__(16) float smem[];
    float* q_s = smem;
    float* kv_s = q_s + C::OWN_FLOATS;                        // [BUFS][K, V]
    float* p_s = kv_s + 2 * C::BUFS * C::FLOATS;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const int n_own = (S + OWN - 1) / OWN;
    const int unit = blockIdx.x % units, qt = n_own - 1 - blockIdx.x / units;        // long rows first when causal
    const int64_t base = (int64_t)unit * S * hs;
    const int q0 = qt * OWN, n_kv = ((causal ? min(q0 + OWN, S) : S) + kRows - 1) / kRows;
    auto fetch = [&](int j) {
        float* b = kv_s + (j % C::BUFS) * 2 * C::FLOATS;
        load_rows<HS, kRows, C::THREADS>(b, K + base, j * kRows, S, hs, vec);
        load_rows<HS, kRows, C::THREADS>(b + C::FLOATS, V + base, j * kRows, S, hs, vec);
        commit();
    };
    griddep_sync();
    load_rows<HS, OWN, C::THREADS>(q_s, Q + base, q0, S, hs, vec);
    fetch(0);
    float o[4][C::CPT], m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -FLT_MAX;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < C::CPT; ++c) o[i][c] = 0.f;
    }
    for (int j = 0; j < n_kv; ++j) {
        if (C::BUFS == 1 && j > 0) {
            __syncthreads();
            fetch(j);
        }
        wait_all();
        __syncthreads();
        if (C::BUFS == 2 && j + 1 < n_kv) fetch(j + 1);
        const float* k_s = kv_s + (j % C::BUFS) * 2 * C::FLOATS;
        float s[4][4];
        scores<HS>(q_s, k_s, ty, tx, s);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int limit = min(S - 1, causal ? q0 + ty * 4 + i : S - 1) - j * kRows;      // last visible key of the tile
            float t = -FLT_MAX;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                s[i][c] = tx + 16 * c <= limit ? s[i][c] * scale : -FLT_MAX;
                t = fmaxf(t, s[i][c]);
            }
            const float m_new = fmaxf(m[i], row_max(t));
            const float corr = expf(m[i] - m_new);          // 0 for the first tile: every row sees its key 0
            float sum = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float e = s[i][c] == -FLT_MAX ? 0.f : expf(s[i][c] - m_new);
                sum += e;
                p_s[(ty * 4 + i) * kLdP + tx + 16 * c] = e;
            }
            l[i] = l[i] * corr + row_sum(sum);
            m[i] = m_new;
#pragma unroll
            for (int c = 0; c < C::CPT; ++c) o[i][c] *= corr;
        }
        __syncwarp();
        accumulate<HS>(p_s, k_s + C::FLOATS, ty, tx, o);
        __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float inv = 1.f / l[i];
#pragma unroll
        for (int c = 0; c < C::CPT; ++c) o[i][c] *= inv;
        const int r = q0 + ty * 4 + i;
        if (tx == 0 && r < S) lse[(int64_t)unit * S + r] = m[i] + logf(l[i]);
    }
    store_rows<HS, T>(O + base, q0, S, hs, ty, tx, o);
}

// ---- backward ------------------------------------------------------------------------------------
template <typename T>
struct BwdArgs {
    const T *Q, *K, *V, *dO;
    const float *lse, *delta;
    const T* O;                      // not NULL: delta is not given, the CTAs make it from O and dO
    T *dQ, *dK, *dV;
    int units, S, hs, causal, vec;
    float scale;
};

// KEYS: the CTA owns key rows (dK, dV), otherwise query rows (dQ).
template <int HS, int OWN, typename T, bool KEYS>
__device__ __forceinline__ void bwd_walk(const BwdArgs<T>& a, int unit, int tile, float* smem) {
    using C = Tiles<HS, OWN>;
    float* own0 = smem;
    float* own1 = own0 + C::OWN_FLOATS;
    float* walk = own1 + C::OWN_FLOATS;                       // [BUFS][walk0, walk1]
    float* ds_s = walk + 2 * C::BUFS * C::FLOATS;
    float* p_s = ds_s + OWN * kLdP;
    float* stat = p_s + OWN * kLdP;                     // [2][lse[64], delta[64]] of the query rows
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const int S = a.S, hs = a.hs, n_tiles = (S + kRows - 1) / kRows;
    const int64_t base = (int64_t)unit * S * hs, sbase = (int64_t)unit * S;
    const int r0 = tile * OWN;
    const int first = KEYS && a.causal ? r0 / kRows : 0;
    const int end = !KEYS && a.causal ? min((r0 + OWN + kRows - 1) / kRows, n_tiles) : n_tiles;
    const T* w0 = (KEYS ? a.Q : a.K) + base;
    const T* w1 = (KEYS ? a.dO : a.V) + base;
    auto load_stats = [&](int q0, int buf) {
        if (a.O) {
            // delta of 64 query rows, TPR neighbouring threads per row
            constexpr int TPR = C::THREADS / kRows;
            const int r = threadIdx.x / TPR, part = threadIdx.x % TPR;
            const int64_t at = base + (int64_t)(q0 + r) * hs;
            float sum = 0.f;
            if (q0 + r < S) {
                if (sizeof(T) == 4 && a.vec) {
                    for (int c = part; c < hs / 4; c += TPR) {
                        const float4 x = reinterpret_cast<const float4*>(a.O + at)[c], y = reinterpret_cast<const float4*>(a.dO + at)[c];
                        sum += x.x * y.x + x.y * y.y + x.z * y.z + x.w * y.w;
                    }
                } else {
                    for (int c = part; c < hs; c += TPR) sum += to_f32(a.O[at + c]) * to_f32(a.dO[at + c]);
                }
            }
#pragma unroll
            for (int w = 1; w < TPR; w <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
            float* st = stat + buf * 2 * kRows;
            if (part == 0) {
                st[r] = q0 + r < S ? a.lse[sbase + q0 + r] : 0.f;
                st[kRows + r] = sum;
            }
        } else if (threadIdx.x < 2 * kRows) {
            const int r = threadIdx.x & (kRows - 1);
            const float* src = threadIdx.x < kRows ? a.lse : a.delta;
            stat[buf * 2 * kRows + threadIdx.x] = q0 + r < S ? src[sbase + q0 + r] : 0.f;
        }
    };
    auto fetch = [&](int j) {
        float* b = walk + (j % C::BUFS) * 2 * C::FLOATS;
        load_rows<HS, kRows, C::THREADS>(b, w0, j * kRows, S, hs, a.vec);
        load_rows<HS, kRows, C::THREADS>(b + C::FLOATS, w1, j * kRows, S, hs, a.vec);
        commit();
    };
    griddep_sync();
    load_rows<HS, OWN, C::THREADS>(own0, (KEYS ? a.K : a.Q) + base, r0, S, hs, a.vec);
    load_rows<HS, OWN, C::THREADS>(own1, (KEYS ? a.V : a.dO) + base, r0, S, hs, a.vec);
    fetch(first);
    load_stats(KEYS ? first * kRows : r0, KEYS ? first & 1 : 0);
    float acc0[4][C::CPT], acc1[4][C::CPT];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < C::CPT; ++c) acc0[i][c] = acc1[i][c] = 0.f;
    for (int j = first; j < end; ++j) {
        if (C::BUFS == 1 && j > first) {
            __syncthreads();
            fetch(j);
        }
        wait_all();
        __syncthreads();
        if (C::BUFS == 2 && j + 1 < end) fetch(j + 1);
        if (KEYS && !a.O && j + 1 < end) load_stats((j + 1) * kRows, (j + 1) & 1);
        const float* x0 = walk + (j % C::BUFS) * 2 * C::FLOATS;
        const float* x1 = x0 + C::FLOATS;
        float s[4][4], dp[4][4];
        scores<HS>(own0, x0, ty, tx, s);
        scores<HS>(own1, x1, ty, tx, dp);
        const float* st = stat + (KEYS ? j & 1 : 0) * 2 * kRows;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int mine = r0 + ty * 4 + i, other = j * kRows + tx + 16 * c;
                const int q = KEYS ? other : mine, k = KEYS ? mine : other;
                const int q_in = KEYS ? tx + 16 * c : ty * 4 + i;
                const bool seen = q < S && k < S && (!a.causal || k <= q);
                const float pr = seen ? expf(s[i][c] * a.scale - st[q_in]) : 0.f;
                ds_s[(ty * 4 + i) * kLdP + tx + 16 * c] = pr * (dp[i][c] - st[kRows + q_in]) * a.scale;
                if (KEYS) p_s[(ty * 4 + i) * kLdP + tx + 16 * c] = pr;
            }
        __syncwarp();
        accumulate<HS>(ds_s, x0, ty, tx, acc0);
        if (KEYS) accumulate<HS>(p_s, x1, ty, tx, acc1);
        __syncwarp();
        // behind the tile's products: unlike the loads above, these are waited for
        if (KEYS && a.O && j + 1 < end) load_stats((j + 1) * kRows, (j + 1) & 1);
    }
    if (KEYS) {
        store_rows<HS, T>(a.dK + base, r0, S, hs, ty, tx, acc0);
        store_rows<HS, T>(a.dV + base, r0, S, hs, ty, tx, acc1);
    } else {
        store_rows<HS, T>(a.dQ + base, r0, S, hs, ty, tx, acc0);
    }
}

template <int HS, int OWN, typename T>
__global__ void __launch_bounds__(OWN * 4)
attn_bwd_simt_kernel(const BwdArgs<T> a) {
    extern __shared__ __align__(16) float smem[];
    // the longest walks first when causal: early key tiles, late query tiles
    const int n_own = (a.S + OWN - 1) / OWN;
    const int b = blockIdx.x >> 1, unit = b % a.units, t = b / a.units;
    if (blockIdx.x & 1) bwd_walk<HS, OWN, T, false>(a, unit, n_own - 1 - t, smem);
    else                bwd_walk<HS, OWN, T, true>(a, unit, t, smem);
}

bool rows_aligned(const void* const* ptrs, int n, int64_t hs, int es) {
    bool ok = hs % 4 == 0;
    for (int i = 0; i < n; ++i) ok = ok && ((uintptr_t)ptrs[i] & (4 * es - 1)) == 0;
    return ok;
}

template <int HS, int OWN, typename T>
int launch_fwd_own(int64_t units, int64_t S, int hs, int causal, float scale, const void* Q, const void* K,
               const void* V, void* O, float* lse) {
    auto kern = attn_fwd_simt_kernel<HS, OWN, T>;
    constexpr int smem = Tiles<HS, OWN>::FWD_SMEM;
    static bool configured = false;     // per process = per device: the library binds to one device
    if (!configured) {
        BOATCU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem > kSpreadSmem ? smem : kSpreadSmem));
        configured = true;
    }
    const void* in[3] = {Q, K, V};
    const unsigned grid = (unsigned)(units * ceil_div(S, OWN));
    BOATCU_RUN(kern, grid, OWN * 4, spread_smem(smem, grid), (int)units, (int)S, hs, causal, scale, rows_aligned(in, 3, hs, sizeof(T)),
                                                             (const T*)Q, (const T*)K, (const T*)V, (T*)O, lse);
    BOATCU_LAUNCH_OK("attn_fwd_simt");
    return 0;
}

template <int HS, int OWN, typename T>
int launch_bwd_own(int64_t units, int64_t S, int hs, int causal, float scale, const void* Q, const void* K,
               const void* V, const void* O, const void* dO, const float* lse, const float* delta, void* dQ, void* dK, void* dV) {
    auto kern = attn_bwd_simt_kernel<HS, OWN, T>;
    constexpr int smem = Tiles<HS, OWN>::BWD_SMEM;
    static bool configured = false;
    if (!configured) {
        BOATCU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem > kSpreadSmem ? smem : kSpreadSmem));
        configured = true;
    }
    const void* in[5] = {Q, K, V, dO, O ? O : dO};
    BwdArgs<T> a;
    a.O = (const T*)O;
    a.Q = (const T*)Q; a.K = (const T*)K; a.V = (const T*)V; a.dO = (const T*)dO;
    a.lse = lse; a.delta = delta;
    a.dQ = (T*)dQ; a.dK = (T*)dK; a.dV = (T*)dV;
    a.units = (int)units; a.S = (int)S; a.hs = hs; a.causal = causal;
    a.vec = rows_aligned(in, 5, hs, sizeof(T));
    a.scale = scale;
    const unsigned grid = (unsigned)(2 * units * ceil_div(S, OWN));
    BOATCU_RUN(kern, grid, OWN * 4, spread_smem(smem, grid), a);
    BOATCU_LAUNCH_OK("attn_bwd_simt");
    return 0;
}

// 64 owned rows make half as many fetches of the other side; 32 halve the longest walk of a CTA.  Below
// about four 64-row CTAs per SM the length of the last walks decides, from there on the fetches do.
bool own_half(int64_t ctas64) { return ctas64 < 4 * (int64_t)sm_count(); }

template <int HS, typename T, typename... A>
int launch_fwd(int64_t units, int64_t S, A... args) {
    return own_half(units * ceil_div(S, 64)) ? launch_fwd_own<HS, 32, T>(units, S, args...) : launch_fwd_own<HS, 64, T>(units, S, args...);
}
template <int HS, typename T, typename... A>
int launch_bwd(int64_t units, int64_t S, A... args) {
    return own_half(2 * units * ceil_div(S, 64)) ? launch_bwd_own<HS, 32, T>(units, S, args...) : launch_bwd_own<HS, 64, T>(units, S, args...);
}

#define DISPATCH_HS(FN, ...)                                                                  \
    do {                                                                                      \
        if (io_type == BOAT_CUDA_BF16) {                                                      \
            if (hs <= 16) return FN<16, __nv_bfloat16>(__VA_ARGS__);                          \
            if (hs <= 32) return FN<32, __nv_bfloat16>(__VA_ARGS__);                          \
            if (hs <= 64) return FN<64, __nv_bfloat16>(__VA_ARGS__);                          \
            return FN<128, __nv_bfloat16>(__VA_ARGS__);                                       \
        } else {                                                                              \
            if (hs <= 16) return FN<16, float>(__VA_ARGS__);                                  \
            if (hs <= 32) return FN<32, float>(__VA_ARGS__);                                  \
            if (hs <= 64) return FN<64, float>(__VA_ARGS__);                                  \
            return FN<128, float>(__VA_ARGS__);                                               \
        }                                                                                     \
    } while (0)

int check_shape(int64_t units, int64_t S, int64_t hs) {
    if (hs > 128) return set_error(8, "attention: head size %lld > 128 is not supported", (long long)hs);
    if (S > (1ll << 30) || units * ceil_div(S, 32) > (1ll << 30))
        return set_error(8, "attention: %lld (batch x heads) units of %lld rows are too many for one launch", (long long)units, (long long)S);
    return 0;
}

}  // namespace

int attn_fwd_simt(int64_t units, int64_t S, int64_t hs, int causal, float scale, const void* Q, const void* K,
                  const void* V, int io_type, void* O, float* lse) {
    if (units <= 0 || S <= 0 || hs <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    if (int rc = check_shape(units, S, hs)) return rc;
    DISPATCH_HS(launch_fwd, units, S, (int)hs, causal, scale, Q, K, V, O, lse);
}

// Where the launch of a pass for delta (1.1 to 1.4 us) is more than what each CTA's reading of O and dO costs: up to eight CTAs of 64
// rows per SM, one tile, or two of head size 64 and less.  With the pass and without, us, operands in L2:
//   8 units of 64 x 16       7.1    6.0        64 units of 64 x 64     15.8   14.7      512 units of 64 x 64     81.4   80.8
//   2048 units of 8 x 16    91.6   94.9        2048 units of 64 x 64    310    314      8192 units of 8 x 64     1051   1107
//   64 units of 128 x 16    18.1   17.0        64 units of 100 x 32    21.7   20.8      512 units of 100 x 16    70.0   71.4
//   8 units of 128 x 64     18.6   18.5        64 units of 128 x 64    34.9   35.5      512 units of 128 x 64     215    220
//   8 units of 100 x 128    34.2   34.9        64 units of 128 x 128   83.2   87.6      64 units of 192 x 32     34.8   35.4
bool attn_bwd_simt_makes_delta(int64_t units, int64_t S, int64_t hs, int io_type) {
    const int64_t tiles = ceil_div(S, kRows);
    return io_type == BOAT_CUDA_F32 && 2 * units * tiles < 8 * (int64_t)sm_count() && (tiles == 1 || (tiles == 2 && hs <= 64));
}

int attn_bwd_simt(int64_t units, int64_t S, int64_t hs, int causal, float scale, const void* Q, const void* K,
                  const void* V, const void* O, const void* dO, const float* lse, const float* delta, int io_type, void* dQ,
                  void* dK, void* dV) {
    if (units <= 0 || S <= 0 || hs <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    if (int rc = check_shape(units, S, hs)) return rc;
    DISPATCH_HS(launch_bwd, units, S, (int)hs, causal, scale, Q, K, V, O, dO, lse, delta, dQ, dK, dV);
}

}  // namespace boatcu
