// elementwise.cu - the HBM-bound tail of the attention step: bias/grad element-wise work,
// column sums for bias gradients, FP32<->BF16 casts, the row dot product delta = sum(dO*O)
// and a tiled transpose.  Every kernel moves 128 bits per thread per access when the
// pointers and sizes allow it and falls back to scalar accesses otherwise; reductions use
// warp shuffles.  Reference counterparts are named per function in boat_cuda.h.
#include "common.cuh"
#include <cooperative_groups.h>

namespace boatcu {

static const int kThreads = 256;

// One CTA per 256 work items, no persistent cap: for these streaming kernels the hardware's
// CTA scheduler balances better than a grid-stride loop over 8 CTAs per SM (measured on the
// Adam step: 6.3 TB/s against 5.3 TB/s).  The kernels keep their grid-stride loops, so the
// limit of the grid's x dimension only matters beyond 2^31 * 256 items.
static inline int grid_for(int64_t work_items, int per_block) {
    int64_t blocks = ceil_div(work_items, per_block);
    if (blocks > 0x7fffffffLL) blocks = 0x7fffffffLL;
    if (blocks < 1) blocks = 1;
    return (int)blocks;
}

static inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// Rounded product, then rounded sum - deliberately not an FMA: the reference's SGD step is
// p - fl(g*lr) (boat_mul_scalar then boat_sub_), and with alpha = -lr this reproduces it
// bit for bit.
__device__ __forceinline__ float mul_add(float alpha, float x, float y) { return __fadd_rn(__fmul_rn(alpha, x), y); }

// ---- y = alpha*x (+ y), 4 floats per access -------------------------------------------
template <bool ACCUM>
__global__ void axpy_vec4(float* __restrict__ y, const float* __restrict__ x, float alpha, int64_t n4, int follow) {
    griddep_enter(follow);
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t step = (int64_t)gridDim.x * blockDim.x;
    float4* y4 = reinterpret_cast<float4*>(y);
    const float4* x4 = reinterpret_cast<const float4*>(x);
    for (; i < n4; i += step) {
        float4 a = x4[i];
        float4 r;
        if (ACCUM) {
            float4 b = y4[i];
            r = make_float4(mul_add(alpha, a.x, b.x), mul_add(alpha, a.y, b.y), mul_add(alpha, a.z, b.z), mul_add(alpha, a.w, b.w));
        } else {
            r = make_float4(alpha * a.x, alpha * a.y, alpha * a.z, alpha * a.w);
        }
        y4[i] = r;
    }
    griddep_leave(follow);
}

template <bool ACCUM>
__global__ void axpy_scalar(float* __restrict__ y, const float* __restrict__ x, float alpha, int64_t n, int follow) {
    griddep_enter(follow);
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (; i < n; i += step) y[i] = ACCUM ? mul_add(alpha, x[i], y[i]) : alpha * x[i];
    griddep_leave(follow);
}

template <bool ACCUM>
static int launch_axpy(float* y, const float* x, float alpha, int64_t n) {
    if (n <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    LaunchTurn turn;
    turn.reads(x, (size_t)n * 4);
    turn.writes(y, (size_t)n * 4);
    const int follow = turn.follow();
    if (aligned16(y) && aligned16(x) && (n % 4) == 0) {
        BOATCU_RUN_IN_TURN(turn, axpy_vec4<ACCUM>, grid_for(n / 4, kThreads), kThreads, 0, y, x, alpha, n / 4, follow);
    } else {
        BOATCU_RUN_IN_TURN(turn, axpy_scalar<ACCUM>, grid_for(n, kThreads), kThreads, 0, y, x, alpha, n, follow);
    }
    BOATCU_LAUNCH_OK("axpy");
    return 0;
}

// ---- y[t] = alpha*x[t] + y[t] for several tensors, blockIdx.y = tensor: the SGD step of a layer -------
constexpr int kMaxAxpy = 8;
struct AxpyTable {
    float* y[kMaxAxpy];
    const float* x[kMaxAxpy];
    int64_t n[kMaxAxpy];
};
__global__ void axpy_multi_kernel(const AxpyTable t, float alpha, int vec) {
    griddep_sync();
    float* __restrict__ y = t.y[blockIdx.y];
    const float* __restrict__ x = t.x[blockIdx.y];
    const int64_t n = t.n[blockIdx.y], n4 = vec ? n / 4 : 0;
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = i0; i < n4; i += step) {
        const float4 a = reinterpret_cast<const float4*>(x)[i], b = reinterpret_cast<const float4*>(y)[i];
        reinterpret_cast<float4*>(y)[i] = make_float4(mul_add(alpha, a.x, b.x), mul_add(alpha, a.y, b.y),
                                                      mul_add(alpha, a.z, b.z), mul_add(alpha, a.w, b.w));
    }
    for (int64_t i = n4 * 4 + i0; i < n; i += step) y[i] = mul_add(alpha, x[i], y[i]);
}

// ---- bytes between HBM and page-locked host memory -----------------------------------------------------
// A kernel, not the copy engine, for what a small step sends and fetches: it follows and precedes the step's
// kernels without the stream changing engines, which costs several times what the bytes do: a step of
// 2 x 4 x 32 with six such copies 157 -> 148 us.  From about kStageKernelBytes on the copy engine is as good.
constexpr size_t kStageKernelBytes = 256 * 1024;
__global__ void stage_copy_kernel(uint4* __restrict__ dst, const uint4* __restrict__ src, int64_t n) {
    griddep_sync();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[i];
}

// ---- y += x[0] + x[1] + ..., in that order: the gradient contributions of one variable ---------------
constexpr int kMaxAddN = 4;
struct AddTable {
    const float* x[kMaxAddN];
    int count;
};
__global__ void add_n_kernel(float* __restrict__ y, const AddTable t, int64_t n, int vec) {
    griddep_sync();
    const int64_t n4 = vec ? n / 4 : 0;
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = i0; i < n4; i += step) {
        float4 a[kMaxAddN], v = reinterpret_cast<const float4*>(y)[i];
#pragma unroll
        for (int k = 0; k < kMaxAddN; ++k)
            if (k < t.count) a[k] = reinterpret_cast<const float4*>(t.x[k])[i];
#pragma unroll
        for (int k = 0; k < kMaxAddN; ++k)
            if (k < t.count) v = make_float4(v.x + a[k].x, v.y + a[k].y, v.z + a[k].z, v.w + a[k].w);
        reinterpret_cast<float4*>(y)[i] = v;
    }
    for (int64_t i = n4 * 4 + i0; i < n; i += step) {
        float v = y[i];
        for (int k = 0; k < t.count; ++k) v += t.x[k][i];
        y[i] = v;
    }
}

// ---- the SGD step of a layer that accumulates its gradients: y -= fl(lr*g), then g = 0 ----------------
__global__ void sgd_clear_kernel(const AxpyTable t, float lr, int vec, int follow) {
    griddep_enter(follow);
    float* __restrict__ y = t.y[blockIdx.y];
    float* __restrict__ g = const_cast<float*>(t.x[blockIdx.y]);
    const int64_t n = t.n[blockIdx.y], n4 = vec ? n / 4 : 0;
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = i0; i < n4; i += step) {
        const float4 a = reinterpret_cast<const float4*>(g)[i], b = reinterpret_cast<const float4*>(y)[i];
        reinterpret_cast<float4*>(y)[i] = make_float4(mul_add(-lr, a.x, b.x), mul_add(-lr, a.y, b.y), mul_add(-lr, a.z, b.z), mul_add(-lr, a.w, b.w));
        reinterpret_cast<float4*>(g)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int64_t i = n4 * 4 + i0; i < n; i += step) {
        y[i] = mul_add(-lr, g[i], y[i]);
        g[i] = 0.f;
    }
    griddep_leave(follow);
}

// ---- y = a * b -------------------------------------------------------------------------------
__global__ void mul_kernel(float* __restrict__ y, const float* __restrict__ a, const float* __restrict__ b,
                           int64_t n, int vec) {
    griddep_sync();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t step = (int64_t)gridDim.x * blockDim.x;
    if (vec) {
        int64_t n4 = n / 4;
        for (; i < n4; i += step) {
            float4 p = reinterpret_cast<const float4*>(a)[i];
            float4 q = reinterpret_cast<const float4*>(b)[i];
            reinterpret_cast<float4*>(y)[i] = make_float4(p.x * q.x, p.y * q.y, p.z * q.z, p.w * q.w);
        }
    } else {
        for (; i < n; i += step) y[i] = a[i] * b[i];
    }
}

// ---- y[i,j] = x[i,j] + bias[j] ---------------------------------------------------------------
__global__ void add_bias_kernel(float* __restrict__ y, const float* __restrict__ x,
                                const float* __restrict__ bias, int64_t rows, int64_t cols, int vec) {
    griddep_sync();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t step = (int64_t)gridDim.x * blockDim.x;
    if (vec) {
        int64_t c4 = cols / 4, n4 = rows * c4;
        for (; i < n4; i += step) {
            float4 v = reinterpret_cast<const float4*>(x)[i];
            float4 b = reinterpret_cast<const float4*>(bias)[i % c4];
            reinterpret_cast<float4*>(y)[i] = make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w);
        }
    } else {
        int64_t n = rows * cols;
        for (; i < n; i += step) y[i] = x[i] + bias[i % cols];
    }
}

// ---- y = alpha*a + beta*b on FP32 or BF16 storage (residual adds, differences, MSE gradient) ----
template <typename T>
__global__ void lincomb_kernel(T* __restrict__ y, const T* __restrict__ a, float alpha, const T* __restrict__ b,
                               float beta, int64_t n, int vec, int follow) {
    griddep_enter(follow);
    constexpr int V = 16 / sizeof(T);
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    if (vec) {
        const int64_t nv = n / V;
        for (; i < nv; i += step) {
            uint4 av = reinterpret_cast<const uint4*>(a)[i], bv = reinterpret_cast<const uint4*>(b)[i], ov;
            const T* ae = reinterpret_cast<const T*>(&av);
            const T* be = reinterpret_cast<const T*>(&bv);
            T* oe = reinterpret_cast<T*>(&ov);
#pragma unroll
            for (int k = 0; k < V; ++k) oe[k] = from_f32<T>(alpha * to_f32(ae[k]) + beta * to_f32(be[k]));
            reinterpret_cast<uint4*>(y)[i] = ov;
        }
    } else {
        for (; i < n; i += step) y[i] = from_f32<T>(alpha * to_f32(a[i]) + beta * to_f32(b[i]));
    }
    griddep_leave(follow);
}

// ---- casts -----------------------------------------------------------------------------------
__global__ void cast_f32_to_bf16(__nv_bfloat16* __restrict__ dst, const float* __restrict__ src, int64_t n, int vec, int follow) {
    griddep_enter(follow);
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t step = (int64_t)gridDim.x * blockDim.x;
    if (vec) {   // 8 elements: two 128-bit loads, one 128-bit store
        int64_t n8 = n / 8;
        for (; i < n8; i += step) {
            float4 a = reinterpret_cast<const float4*>(src)[2 * i];
            float4 b = reinterpret_cast<const float4*>(src)[2 * i + 1];
            __nv_bfloat162 p0 = __floats2bfloat162_rn(a.x, a.y), p1 = __floats2bfloat162_rn(a.z, a.w);
            __nv_bfloat162 p2 = __floats2bfloat162_rn(b.x, b.y), p3 = __floats2bfloat162_rn(b.z, b.w);
            uint4 o;
            o.x = *reinterpret_cast<uint32_t*>(&p0); o.y = *reinterpret_cast<uint32_t*>(&p1);
            o.z = *reinterpret_cast<uint32_t*>(&p2); o.w = *reinterpret_cast<uint32_t*>(&p3);
            reinterpret_cast<uint4*>(dst)[i] = o;
        }
    } else {
        for (; i < n; i += step) dst[i] = __float2bfloat16_rn(src[i]);
    }
    griddep_leave(follow);
}

__global__ void cast_bf16_to_f32(float* __restrict__ dst, const __nv_bfloat16* __restrict__ src, int64_t n, int vec, int follow) {
    griddep_enter(follow);
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t step = (int64_t)gridDim.x * blockDim.x;
    if (vec) {
        int64_t n8 = n / 8;
        for (; i < n8; i += step) {
            uint4 v = reinterpret_cast<const uint4*>(src)[i];
            __nv_bfloat162 p0 = *reinterpret_cast<__nv_bfloat162*>(&v.x), p1 = *reinterpret_cast<__nv_bfloat162*>(&v.y);
            __nv_bfloat162 p2 = *reinterpret_cast<__nv_bfloat162*>(&v.z), p3 = *reinterpret_cast<__nv_bfloat162*>(&v.w);
            float2 f0 = __bfloat1622float2(p0), f1 = __bfloat1622float2(p1);
            float2 f2 = __bfloat1622float2(p2), f3 = __bfloat1622float2(p3);
            reinterpret_cast<float4*>(dst)[2 * i] = make_float4(f0.x, f0.y, f1.x, f1.y);
            reinterpret_cast<float4*>(dst)[2 * i + 1] = make_float4(f2.x, f2.y, f3.x, f3.y);
        }
    } else {
        for (; i < n; i += step) dst[i] = __bfloat162float(src[i]);
    }
    griddep_leave(follow);
}

// ---- y = x rounded to the nearest TF32 value (10-bit mantissa), still stored as FP32 -------------
// tcgen05 kind::tf32 drops the low 13 mantissa bits of its operands; a chain of contractions
// then drifts by a systematic ~2^-11 per stage.  Rounding operands to nearest beforehand
// makes the truncation exact and the error unbiased.
__device__ __forceinline__ float round_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

__global__ void round_tf32_kernel(float* __restrict__ y, const float* __restrict__ x, int64_t n, int vec, int follow) {
    griddep_enter(follow);
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t step = (int64_t)gridDim.x * blockDim.x;
    if (vec) {
        int64_t n4 = n / 4;
        for (; i < n4; i += step) {
            float4 v = reinterpret_cast<const float4*>(x)[i];
            reinterpret_cast<float4*>(y)[i] = make_float4(round_tf32(v.x), round_tf32(v.y), round_tf32(v.z), round_tf32(v.w));
        }
    } else {
        for (; i < n; i += step) y[i] = round_tf32(x[i]);
    }
    griddep_leave(follow);
}

// ---- several FP32 tensors to BF16 or to TF32-valued FP32, one launch ----------------------------
constexpr int kMaxConvert = 8;
struct ConvertTable {
    const float* src[kMaxConvert];
    void* dst[kMaxConvert];
    int64_t n[kMaxConvert];
};

// blockIdx.y = tensor; vec: every tensor is 16-byte aligned with a multiple of 8 elements
template <bool TO_BF16>
__global__ void convert_multi_kernel(const ConvertTable t, int vec, int follow) {
    griddep_enter(follow);
    const float* __restrict__ src = t.src[blockIdx.y];
    const int64_t n = t.n[blockIdx.y];
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    if (vec) {
        const int64_t n8 = n / 8;
        for (; i < n8; i += step) {
            const float4 a = reinterpret_cast<const float4*>(src)[2 * i];
            const float4 b = reinterpret_cast<const float4*>(src)[2 * i + 1];
            if (TO_BF16) {
                __nv_bfloat162 p0 = __floats2bfloat162_rn(a.x, a.y), p1 = __floats2bfloat162_rn(a.z, a.w);
                __nv_bfloat162 p2 = __floats2bfloat162_rn(b.x, b.y), p3 = __floats2bfloat162_rn(b.z, b.w);
                uint4 o;
                o.x = *reinterpret_cast<uint32_t*>(&p0); o.y = *reinterpret_cast<uint32_t*>(&p1);
                o.z = *reinterpret_cast<uint32_t*>(&p2); o.w = *reinterpret_cast<uint32_t*>(&p3);
                reinterpret_cast<uint4*>(t.dst[blockIdx.y])[i] = o;
            } else {
                float4* d = reinterpret_cast<float4*>(t.dst[blockIdx.y]);
                d[2 * i] = make_float4(round_tf32(a.x), round_tf32(a.y), round_tf32(a.z), round_tf32(a.w));
                d[2 * i + 1] = make_float4(round_tf32(b.x), round_tf32(b.y), round_tf32(b.z), round_tf32(b.w));
            }
        }
    } else {
        for (; i < n; i += step) {
            if (TO_BF16) ((__nv_bfloat16*)t.dst[blockIdx.y])[i] = __float2bfloat16_rn(src[i]);
            else         ((float*)t.dst[blockIdx.y])[i] = round_tf32(src[i]);
        }
    }
    griddep_leave(follow);
}

// ---- column sums: out[j] = sum_i X[i,j] ------------------------------------------------------
// A CTA's threads are LANES column lanes (16 bytes of a row each) x row lanes, eight rows' loads in flight
// per thread; row lanes fold in shared memory.  Two ways to fold the CTAs of a column group:
//   - a cluster of 8 CTAs, through distributed shared memory in a fixed order: one launch, no cleared
//     output, the same bits every time.  3 x 8000 x 1024 BF16 back to back 14 us from HBM, 11 from L2 (18.5 the
//     other way).  But clusters pack unevenly onto SMs, which costs bandwidth once a matrix is large (32768 x
//     2048: 43 us);
//   - from 32 MB per matrix on, independent CTAs on a full grid that add into a cleared output with
//     atomics (27 us).
// blockIdx.y is the column group, blockIdx.z selects one of several matrices of the same shape; a launch takes as many
// groups as a grid has in y, from `first` on.
constexpr int64_t kMaxGridY = 65535;
constexpr int kMaxColsum = 4;
constexpr int kColsumCluster = 8;
struct ColsumTable {
    const void* x[kMaxColsum];
    float* out[kMaxColsum];
};

template <typename T, int VEC, int LANES, int THREADS, bool CLUSTER>
__global__ void __launch_bounds__(THREADS) colsum_kernel(const __grid_constant__ ColsumTable t, int64_t rows, int64_t cols, int64_t first, int follow) {
    constexpr int ROWS = THREADS / LANES, COLS = LANES * VEC, UNROLL = 8;
    __shared__ float part[ROWS * COLS];
    __shared__ float folded[CLUSTER ? COLS : 1];
    griddep_enter(follow);
    const T* __restrict__ X = (const T*)t.x[blockIdx.z];
    const int tx = threadIdx.x % LANES, ty = threadIdx.x / LANES;
    const int64_t group0 = (first + blockIdx.y) * COLS, col0 = group0 + tx * VEC;
    float acc[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) acc[v] = 0.f;
    if (col0 < cols) {
        const int64_t step = (int64_t)gridDim.x * ROWS;
        int64_t r = (int64_t)blockIdx.x * ROWS + ty;
        if constexpr (VEC == 1) {
            for (; r < rows; r += step) acc[0] += to_f32(X[r * cols + col0]);
        } else {
            auto add = [&](const uint4& v) {
                if constexpr (sizeof(T) == 4) {
                    acc[0] += __uint_as_float(v.x); acc[1] += __uint_as_float(v.y); acc[2] += __uint_as_float(v.z); acc[3] += __uint_as_float(v.w);
                } else {
                    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float2 f = __bfloat1622float2(h[k]);
                        acc[2 * k] += f.x;
                        acc[2 * k + 1] += f.y;
                    }
                }
            };
            for (; r + (UNROLL - 1) * step < rows; r += UNROLL * step) {
                uint4 v[UNROLL];
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) v[u] = __ldg(reinterpret_cast<const uint4*>(X + (r + u * step) * cols + col0));
#pragma unroll
                for (int u = 0; u < UNROLL; ++u) add(v[u]);
            }
            for (; r < rows; r += step) add(__ldg(reinterpret_cast<const uint4*>(X + r * cols + col0)));
        }
    }
#pragma unroll
    for (int v = 0; v < VEC; ++v) part[ty * COLS + tx * VEC + v] = acc[v];
    __syncthreads();
    for (int c = threadIdx.x; c < COLS; c += THREADS) {
        float s = 0.f;
#pragma unroll 8
        for (int k = 0; k < ROWS; ++k) s += part[k * COLS + c];
        if (CLUSTER) folded[c] = s;
        else if (group0 + c < cols) atomicAdd(t.out[blockIdx.z] + group0 + c, s);
    }
    if constexpr (CLUSTER) {
        cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
        cluster.sync();
        if (blockIdx.x == 0) {
            for (int c = threadIdx.x; c < COLS; c += THREADS) {
                float s = 0.f;
#pragma unroll
                for (int r = 0; r < kColsumCluster; ++r) s += cluster.map_shared_rank(folded, r)[c];
                float* o = t.out[blockIdx.z] + group0 + c;
                if (group0 + c < cols) *o = s;
            }
        }
        cluster.sync();
    }
    griddep_leave(follow);
}

template <typename T, int VEC, int LANES>
static int launch_colsum_cluster(const ColsumTable& t, int64_t rows, int64_t cols, int count) {
    const int64_t groups = ceil_div(cols, LANES * VEC);
    for (int64_t first = 0; first < groups; first += kMaxGridY) {
        const int64_t n = groups - first < kMaxGridY ? groups - first : kMaxGridY;
        LaunchTurn turn;
        for (int i = 0; i < count; ++i) {
            turn.reads(t.x[i], (size_t)rows * cols * sizeof(T));
            turn.writes(t.out[i], (size_t)cols * 4);
        }
        BOATCU_CHECK(launch_in_turn(turn, colsum_kernel<T, VEC, LANES, 512, true>, dim3(kColsumCluster, (unsigned)n, (unsigned)count),
                                    dim3(512), 0, kColsumCluster, t, rows, cols, first, turn.follow()));
        BOATCU_LAUNCH_OK("colsum");
    }
    return 0;
}

template <typename T, int VEC>
static int launch_colsum(const ColsumTable& t, int64_t rows, int64_t cols, int count) {
    if (rows * cols * (int64_t)sizeof(T) >= (32ll << 20)) {
        for (int i = 0; i < count; ++i) BOATCU_CHECK(cudaMemsetAsync(t.out[i], 0, (size_t)cols * sizeof(float), stream()));
        const int64_t groups = ceil_div(cols, 32 * VEC);
        int64_t y = (int64_t)sm_count() * 8 / (groups * count);         // eight CTAs per SM
        if (y < 1) y = 1;
        if (y > ceil_div(rows, 8)) y = ceil_div(rows, 8);
        for (int64_t first = 0; first < groups; first += kMaxGridY) {
            const int64_t n = groups - first < kMaxGridY ? groups - first : kMaxGridY;
            BOATCU_CHECK(launch_dependent(colsum_kernel<T, VEC, 32, 256, false>, dim3((unsigned)y, (unsigned)n, (unsigned)count), dim3(256), 0, 1,
                                          t, rows, cols, first, (int)kRelease));
            BOATCU_LAUNCH_OK("colsum");
        }
        return 0;
    }
    // the runs of a row are 512 bytes where that makes enough CTAs for the GPU, else 256 or 128
    auto ctas = [&](int lanes) { return ceil_div(cols, lanes * VEC) * kColsumCluster * count; };
    const int64_t enough = (int64_t)sm_count() * 4 / 5;
    if (ctas(32) >= enough) return launch_colsum_cluster<T, VEC, 32>(t, rows, cols, count);
    if (ctas(16) >= enough) return launch_colsum_cluster<T, VEC, 16>(t, rows, cols, count);
    return launch_colsum_cluster<T, VEC, 8>(t, rows, cols, count);
}

// ---- what the BF16 tensor-core backward starts from, in one pass over dO and O --------------------------
// Per row -delta*scale (delta = sum_d dO*O) and -lse*log2(e), the form its inner loops consume (one FMA each),
// laid out for whole tiles: S rows of a unit take padded_S entries, the surplus ones hold 0 and -inf, with
// which missing query rows contribute exactly nothing; and zeros in the FP32 buffer that dQ is summed in.
// HS/8 lanes per row, 16 bytes each; a thread has the loads of four rows in flight.  HBM-bound: 64 x 8192 x
// 128 (268 MB read, 268 MB cleared) took 80 us + a 40 us memset as two passes with one row in flight.
template <int HS>
__global__ void __launch_bounds__(256) bwd_prepare_kernel(const __nv_bfloat16* __restrict__ dO, const __nv_bfloat16* __restrict__ O,
                                                          const float* __restrict__ lse, int rows, int S, int padded_S, float scale,
                                                          float* __restrict__ delta2, float* __restrict__ lse2, float* __restrict__ dq) {
    constexpr int LANES = HS / 8, ROWS = 256 / LANES, U = 4;
    griddep_sync();
    const int l = threadIdx.x % LANES;
    const int row0 = blockIdx.x * ROWS * U + threadIdx.x / LANES;
    int64_t src[U];
    uint4 a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int row = row0 + u * ROWS;
        src[u] = -1;
        if (row < rows) {
            if (S == padded_S) {
                src[u] = row;
            } else {
                const int unit = row / padded_S, r = row - unit * padded_S;
                if (r < S) src[u] = (int64_t)unit * S + r;
            }
        }
        a[u] = b[u] = make_uint4(0u, 0u, 0u, 0u);
        if (src[u] >= 0) {
            a[u] = __ldg(reinterpret_cast<const uint4*>(dO + src[u] * HS + l * 8));
            b[u] = __ldg(reinterpret_cast<const uint4*>(O + src[u] * HS + l * 8));
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (src[u] >= 0) {
            float4* z = reinterpret_cast<float4*>(dq + src[u] * HS + l * 8);
            z[0] = z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const __nv_bfloat162* ha = reinterpret_cast<const __nv_bfloat162*>(&a[u]);
        const __nv_bfloat162* hb = reinterpret_cast<const __nv_bfloat162*>(&b[u]);
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 x = __bfloat1622float2(ha[k]), y = __bfloat1622float2(hb[k]);
            s += x.x * y.x + x.y * y.y;
        }
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const int row = row0 + u * ROWS;
        if (l == 0 && row < rows) {
            delta2[row] = src[u] < 0 ? 0.f : s * -scale;
            lse2[row] = src[u] < 0 ? -INFINITY : lse[src[u]] * -1.4426950408889634f;
        }
    }
}

int attn_bwd_prepare(const void* dO, const void* O, const float* lse, int64_t units, int64_t S, int64_t padded_S, int64_t hs, float scale,
                     float* delta2, float* lse2, float* dq) {
    const int64_t rows = units * padded_S;
    const int64_t blocks = ceil_div(rows, 256 / (hs / 8) * 4);
    typedef const __nv_bfloat16* bf;
    if (hs == 64)
        BOATCU_RUN(bwd_prepare_kernel<64>, (unsigned)blocks, 256, 0, (bf)dO, (bf)O, lse, (int)rows, (int)S, (int)padded_S, scale, delta2, lse2, dq);
    else
        BOATCU_RUN(bwd_prepare_kernel<128>, (unsigned)blocks, 256, 0, (bf)dO, (bf)O, lse, (int)rows, (int)S, (int)padded_S, scale, delta2, lse2, dq);
    BOATCU_LAUNCH_OK("bwd_prepare");
    return 0;
}

// ---- delta[r] = sum_d dO[r,d] * O[r,d]: one warp per row, shuffle reduction --------------------
template <typename T>
__global__ void rowdot_kernel(const T* __restrict__ A, const T* __restrict__ B, int64_t rows, int cols,
                              float* __restrict__ out) {
    griddep_sync();
    const int lane = threadIdx.x & 31;
    int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t step = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (; row < rows; row += step) {
        const T* a = A + row * cols;
        const T* b = B + row * cols;
        float s = 0.f;
        for (int d = lane; d < cols; d += 32) s += to_f32(a[d]) * to_f32(b[d]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) out[row] = s;
    }
}

// 128-bit variant: 8 bf16 (or 4 floats) per lane per access; cols must divide accordingly.
template <typename T, int VEC>
__global__ void rowdot_vec_kernel(const T* __restrict__ A, const T* __restrict__ B, int64_t rows, int cols,
                                  float* __restrict__ out) {
    griddep_sync();
    const int lanes_per_row = cols / VEC;            // power of two <= 32 checked by the launcher
    const int rows_per_warp = 32 / lanes_per_row;
    const int lane = threadIdx.x & 31;
    const int sub = lane / lanes_per_row, l = lane % lanes_per_row;
    int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = warp * rows_per_warp; base < rows; base += nwarps * rows_per_warp) {
        int64_t row = base + sub;
        float s = 0.f;
        if (row < rows) {
            const uint4 va = *reinterpret_cast<const uint4*>(A + row * cols + l * VEC);
            const uint4 vb = *reinterpret_cast<const uint4*>(B + row * cols + l * VEC);
            if (sizeof(T) == 4) {
                const float* fa = reinterpret_cast<const float*>(&va);
                const float* fb = reinterpret_cast<const float*>(&vb);
#pragma unroll
                for (int k = 0; k < 4; ++k) s += fa[k] * fb[k];
            } else {
                const __nv_bfloat162* ha = reinterpret_cast<const __nv_bfloat162*>(&va);
                const __nv_bfloat162* hb = reinterpret_cast<const __nv_bfloat162*>(&vb);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float2 x = __bfloat1622float2(ha[k]), y = __bfloat1622float2(hb[k]);
                    s += x.x * y.x + x.y * y.y;
                }
            }
        }
        for (int o = lanes_per_row >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (l == 0 && row < rows) out[row] = s;
    }
}

int rowdot(const void* A, const void* B, int type, int64_t rows, int64_t cols, float* out) {
    if (rows <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    const int vec = type == BOAT_CUDA_BF16 ? 8 : 4;
    int64_t lpr = cols / vec;
    bool pow2 = lpr > 0 && (lpr & (lpr - 1)) == 0;
    if (cols % vec == 0 && pow2 && lpr <= 32 && aligned16(A) && aligned16(B)) {
        int rows_per_block = (kThreads / 32) * (int)(32 / lpr);
        int grid = grid_for(rows, rows_per_block);
        if (type == BOAT_CUDA_BF16)
            BOATCU_RUN((rowdot_vec_kernel<__nv_bfloat16, 8>), grid, kThreads, 0, 
                (const __nv_bfloat16*)A, (const __nv_bfloat16*)B, rows, (int)cols, out);
        else
            BOATCU_RUN((rowdot_vec_kernel<float, 4>), grid, kThreads, 0, (const float*)A, (const float*)B, rows, (int)cols, out);
    } else {
        int grid = grid_for(rows, kThreads / 32);
        if (type == BOAT_CUDA_BF16)
            BOATCU_RUN(rowdot_kernel<__nv_bfloat16>, grid, kThreads, 0, 
                (const __nv_bfloat16*)A, (const __nv_bfloat16*)B, rows, (int)cols, out);
        else
            BOATCU_RUN(rowdot_kernel<float>, grid, kThreads, 0, (const float*)A, (const float*)B, rows, (int)cols, out);
    }
    BOATCU_LAUNCH_OK("rowdot");
    return 0;
}

// ---- out[b, j, i] = in[b, i, j], 32x32 shared-memory tiles --------------------------------------
__global__ void transpose_kernel(float* __restrict__ out, const float* __restrict__ in, int64_t rows, int64_t cols) {
    griddep_sync();
    __shared__ float tile[32][33];
    const float* src = in + (int64_t)blockIdx.z * rows * cols;
    float* dst = out + (int64_t)blockIdx.z * rows * cols;
    int64_t c = (int64_t)blockIdx.x * 32 + threadIdx.x;
    for (int k = threadIdx.y; k < 32; k += 8) {
        int64_t r = (int64_t)blockIdx.y * 32 + k;
        if (r < rows && c < cols) tile[k][threadIdx.x] = src[r * cols + c];
    }
    __syncthreads();
    int64_t r2 = (int64_t)blockIdx.y * 32 + threadIdx.x;   // becomes the column of out
    for (int k = threadIdx.y; k < 32; k += 8) {
        int64_t c2 = (int64_t)blockIdx.x * 32 + k;         // becomes the row of out
        if (c2 < cols && r2 < rows) dst[c2 * rows + r2] = tile[threadIdx.x][k];
    }
}

}  // namespace boatcu

using namespace boatcu;

extern "C" {

int boat_cuda_axpy(float* y, const float* x, float alpha, int64_t n) { return launch_axpy<true>(y, x, alpha, n); }
int boat_cuda_scale(float* y, const float* x, float alpha, int64_t n) { return launch_axpy<false>(y, x, alpha, n); }

static int fill_axpy_table(const char* who, float* const* y, const float* const* x, const int64_t* n, int count, AxpyTable& t,
                           int& vec_out, int64_t& longest_out) {
    if (count > kMaxAxpy || !y || !x || !n) return set_error(11, "%s: bad table (%d tensors, 1 to %d)", who, count, kMaxAxpy);
    int vec = 1;
    int64_t longest = 0;
    for (int i = 0; i < kMaxAxpy; ++i) {
        const int s = i < count ? i : 0;
        if (n[s] > 0 && (!y[s] || !x[s])) return set_error(11, "%s: bad entry %d", who, s);
        t.y[i] = y[s];
        t.x[i] = x[s];
        t.n[i] = n[s];
        vec = vec && aligned16(y[s]) && aligned16(x[s]);
        if (n[s] > longest) longest = n[s];
    }
    vec_out = vec;
    longest_out = longest;
    return 0;
}

int boat_cuda_axpy_multi(float* const* y, const float* const* x, float alpha, const int64_t* n, int count) {
    if (count <= 0) return 0;
    AxpyTable t;
    int vec;
    int64_t longest;
    if (int rc = fill_axpy_table("boat_cuda_axpy_multi", y, x, n, count, t, vec, longest)) return rc;
    if (longest <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    BOATCU_RUN(axpy_multi_kernel, dim3((unsigned)grid_for(vec ? ceil_div(longest, 4) : longest, kThreads), (unsigned)count), kThreads, 0, t, alpha, vec);
    BOATCU_LAUNCH_OK("axpy_multi");
    return 0;
}

int boat_cuda_add_n(float* y, const float* const* x, int count, int64_t n) {
    if (count < 1 || count > kMaxAddN) return set_error(11, "boat_cuda_add_n: %d terms (1 to %d)", count, kMaxAddN);
    if (n <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    if (!y || !x) return set_error(11, "boat_cuda_add_n: NULL operand");
    AddTable t = {};
    t.count = count;
    bool vec = aligned16(y);
    for (int k = 0; k < count; ++k) {
        if (!x[k]) return set_error(11, "boat_cuda_add_n: NULL operand");
        t.x[k] = x[k];
        vec = vec && aligned16(x[k]);
    }
    BOATCU_RUN(add_n_kernel, grid_for(vec ? ceil_div(n, 4) : n, kThreads), kThreads, 0, y, t, n, vec ? 1 : 0);
    BOATCU_LAUNCH_OK("add_n");
    return 0;
}

int boat_cuda_stage_copy(void* dst, const void* src, size_t bytes, int down) {
    if (bytes == 0) return 0;
    if (int rc = ensure_init()) return rc;
    if (bytes > kStageKernelBytes || !aligned16(dst) || !aligned16(src) || bytes % 16) {
        ordinary_launch_next();
        BOATCU_CHECK(cudaMemcpyAsync(dst, src, bytes, down ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, stream()));
        return 0;
    }
    const int64_t n = (int64_t)(bytes / 16);
    BOATCU_RUN(stage_copy_kernel, (unsigned)ceil_div(n, kThreads), kThreads, 0, (uint4*)dst, (const uint4*)src, n);
    BOATCU_LAUNCH_OK("stage_copy");
    return 0;
}

int boat_cuda_sgd_clear(float* const* y, float* const* g, float lr, const int64_t* n, int count) {
    if (count <= 0) return 0;
    AxpyTable t;
    int vec;
    int64_t longest;
    if (int rc = fill_axpy_table("boat_cuda_sgd_clear", y, g, n, count, t, vec, longest)) return rc;
    if (longest <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    LaunchTurn turn;
    for (int i = 0; i < count; ++i) {
        turn.writes(y[i], (size_t)n[i] * 4);
        turn.writes(g[i], (size_t)n[i] * 4);
    }
    BOATCU_RUN_IN_TURN(turn, sgd_clear_kernel, dim3((unsigned)grid_for(vec ? ceil_div(longest, 4) : longest, kThreads), (unsigned)count), kThreads, 0, t, lr,
                       vec, turn.follow());
    BOATCU_LAUNCH_OK("sgd_clear");
    return 0;
}

int boat_cuda_mul(float* y, const float* a, const float* b, int64_t n) {
    if (n <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    int vec = aligned16(y) && aligned16(a) && aligned16(b) && (n % 4) == 0;
    BOATCU_RUN(mul_kernel, grid_for(vec ? n / 4 : n, kThreads), kThreads, 0, y, a, b, n, vec);
    BOATCU_LAUNCH_OK("mul");
    return 0;
}

int boat_cuda_add_bias(float* y, const float* x, const float* bias, int64_t rows, int64_t cols) {
    if (rows <= 0 || cols <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    int vec = aligned16(y) && aligned16(x) && aligned16(bias) && (cols % 4) == 0;
    int64_t n = rows * cols;
    BOATCU_RUN(add_bias_kernel, grid_for(vec ? n / 4 : n, kThreads), kThreads, 0, y, x, bias, rows, cols, vec);
    BOATCU_LAUNCH_OK("add_bias");
    return 0;
}

int boat_cuda_cast(void* dst, int dst_type, const void* src, int src_type, int64_t n) {
    if (n <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    if (dst_type == src_type) return boat_cuda_memcpy_d2d(dst, src, (size_t)n * type_size(dst_type));
    int vec = aligned16(dst) && aligned16(src) && (n % 8) == 0;
    int grid = grid_for(vec ? n / 8 : n, kThreads);
    ProfileScope prof("cast");
    LaunchTurn turn;
    turn.reads(src, (size_t)n * type_size(src_type));
    turn.writes(dst, (size_t)n * type_size(dst_type));
    const int follow = turn.follow();
    if (dst_type == BOAT_CUDA_BF16)
        BOATCU_RUN_IN_TURN(turn, cast_f32_to_bf16, grid, kThreads, 0, (__nv_bfloat16*)dst, (const float*)src, n, vec, follow);
    else
        BOATCU_RUN_IN_TURN(turn, cast_bf16_to_f32, grid, kThreads, 0, (float*)dst, (const __nv_bfloat16*)src, n, vec, follow);
    BOATCU_LAUNCH_OK("cast");
    return 0;
}

int boat_cuda_lincomb(void* y, const void* a, float alpha, const void* b, float beta, int type, int64_t n) {
    if (n <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    const int V = type == BOAT_CUDA_BF16 ? 8 : 4;
    int vec = aligned16(y) && aligned16(a) && aligned16(b) && (n % V) == 0;
    int grid = grid_for(vec ? n / V : n, kThreads);
    ProfileScope prof("lincomb");
    LaunchTurn turn;
    turn.reads(a, (size_t)n * type_size(type));
    turn.reads(b, (size_t)n * type_size(type));
    turn.writes(y, (size_t)n * type_size(type));
    const int follow = turn.follow();
    if (type == BOAT_CUDA_BF16)
        BOATCU_RUN_IN_TURN(turn, lincomb_kernel<__nv_bfloat16>, grid, kThreads, 0, (__nv_bfloat16*)y, (const __nv_bfloat16*)a, alpha,
                                                                       (const __nv_bfloat16*)b, beta, n, vec, follow);
    else
        BOATCU_RUN_IN_TURN(turn, lincomb_kernel<float>, grid, kThreads, 0, (float*)y, (const float*)a, alpha, (const float*)b, beta, n, vec, follow);
    BOATCU_LAUNCH_OK("lincomb");
    return 0;
}

int boat_cuda_round_tf32(float* y, const float* x, int64_t n) {
    if (n <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    int vec = aligned16(y) && aligned16(x) && (n % 4) == 0;
    ProfileScope prof("round_tf32");
    LaunchTurn turn;
    turn.reads(x, (size_t)n * 4);
    turn.writes(y, (size_t)n * 4);
    BOATCU_RUN_IN_TURN(turn, round_tf32_kernel, grid_for(vec ? n / 4 : n, kThreads), kThreads, 0, y, x, n, vec, turn.follow());
    BOATCU_LAUNCH_OK("round_tf32");
    return 0;
}

}  // extern "C"

namespace boatcu {
int colsum_multi(const void* const* X, int x_type, int64_t rows, int64_t cols, float* const* out, int count) {
    if (cols <= 0 || count <= 0) return 0;
    if (count > kMaxColsum) return set_error(11, "boat_cuda_colsum_multi: %d matrices (1 to %d)", count, kMaxColsum);
    if (!X || !out) return set_error(11, "boat_cuda_colsum_multi: NULL table");
    if (int rc = ensure_init()) return rc;
    ProfileScope prof("colsum");
    ColsumTable t;
    const int vec = x_type == BOAT_CUDA_BF16 ? 8 : 4;
    bool can_vec = (cols % vec) == 0;
    for (int i = 0; i < kMaxColsum; ++i) {
        const int s = i < count ? i : 0;
        if (!X[s] || !out[s]) return set_error(11, "boat_cuda_colsum_multi: NULL operand");
        t.x[i] = X[s];
        t.out[i] = out[s];
        can_vec = can_vec && aligned16(X[s]);
    }
    if (rows < 0) rows = 0;
    if (x_type == BOAT_CUDA_BF16)
        return can_vec ? launch_colsum<__nv_bfloat16, 8>(t, rows, cols, count) : launch_colsum<__nv_bfloat16, 1>(t, rows, cols, count);
    return can_vec ? launch_colsum<float, 4>(t, rows, cols, count) : launch_colsum<float, 1>(t, rows, cols, count);
}

}  // namespace boatcu

extern "C" {

int boat_cuda_colsum_multi(const void* const* X, int x_type, int64_t rows, int64_t cols, float* const* out, int count) {
    return colsum_multi(X, x_type, rows, cols, out, count);
}

int boat_cuda_colsum(const void* X, int x_type, int64_t rows, int64_t cols, float* out) {
    if (cols <= 0) return 0;
    return boat_cuda_colsum_multi(&X, x_type, rows, cols, &out, 1);
}

int boat_cuda_convert_multi(void* const* dst, int dst_type, const float* const* src, const int64_t* n, int count) {
    if (count <= 0) return 0;
    if (count > kMaxConvert) return set_error(11, "boat_cuda_convert_multi: %d tensors (1 to %d)", count, kMaxConvert);
    if (dst_type != BOAT_CUDA_BF16 && dst_type != BOAT_CUDA_F32_TF32)
        return set_error(10, "boat_cuda_convert_multi: target type %d (BF16 or TF32-valued FP32)", dst_type);
    if (!dst || !src || !n) return set_error(11, "boat_cuda_convert_multi: NULL table");
    if (int rc = ensure_init()) return rc;
    ConvertTable t;
    int vec = 1;
    int64_t longest = 0;
    for (int i = 0; i < kMaxConvert; ++i) {
        const int s = i < count ? i : 0;
        if (n[s] < 0 || (n[s] > 0 && (!dst[s] || !src[s]))) return set_error(11, "boat_cuda_convert_multi: bad entry %d", s);
        t.src[i] = src[s];
        t.dst[i] = dst[s];
        t.n[i] = n[s];
        vec = vec && aligned16(dst[s]) && aligned16(src[s]) && (n[s] % 8) == 0;
        if (n[s] > longest) longest = n[s];
    }
    if (longest == 0) return 0;
    // the blocks of all tensors together fill the GPU a few times over
    int64_t per_tensor = ceil_div(vec ? longest / 8 : longest, kThreads);
    const int64_t cap = ceil_div((int64_t)sm_count() * 16, count);
    if (per_tensor > cap) per_tensor = cap;
    dim3 grid((unsigned)per_tensor, (unsigned)count, 1);
    ProfileScope prof("cast");
    LaunchTurn turn;
    for (int i = 0; i < count; ++i) {
        turn.reads(src[i], (size_t)n[i] * 4);
        turn.writes(dst[i], (size_t)n[i] * type_size(dst_type));
    }
    const int follow = turn.follow();
    if (dst_type == BOAT_CUDA_BF16) BOATCU_RUN_IN_TURN(turn, convert_multi_kernel<true>, grid, kThreads, 0, t, vec, follow);
    else                            BOATCU_RUN_IN_TURN(turn, convert_multi_kernel<false>, grid, kThreads, 0, t, vec, follow);
    BOATCU_LAUNCH_OK("convert_multi");
    return 0;
}

int boat_cuda_transpose(float* out, const float* in, int64_t batch, int64_t rows, int64_t cols) {
    if (batch <= 0 || rows <= 0 || cols <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    if (batch > 65535) return set_error(6, "boat_cuda_transpose: batch %lld exceeds 65535", (long long)batch);
    dim3 grid((unsigned)ceil_div(cols, 32), (unsigned)ceil_div(rows, 32), (unsigned)batch);
    BOATCU_RUN(transpose_kernel, grid, dim3(32, 8, 1), 0, out, in, rows, cols);
    BOATCU_LAUNCH_OK("transpose");
    return 0;
}

}  // extern "C"
