// norm_act.cu - LayerNorm forward/backward and GELU forward/backward: the HBM-bound kernels
// of the pre-LN encoder block around the attention layer.
//
// LayerNorm forward restates boat_layernorm_forward (reference src/layers/norm.c:231-317):
// per row, mean = sum/H, biased variance = sum((x-mean)^2)/H, y = (x-mean)/sqrt(var+eps)*w + b.
// The reference has no LayerNorm backward (norm.c:397-402 is a stub) and no GELU
// (src/ops/activation.c:298-302 is a stub); those follow the textbook formulas, with the
// exact erf form of GELU.  A warp (forward) or a CTA (backward) holds a row in registers, so a row is read from HBM
// once per kernel; rows that are no whole 16-byte vectors, or too long for that, are kept in the shared memory of a
// CTA each.
#include "common.cuh"
#include "gelu.cuh"
#include <initializer_list>

namespace boatcu {

static const int kNormThreads = 256;

__device__ __forceinline__ float block_sum(float v, float* red) {
    // red: 32 floats of shared memory.  Returns the sum over the CTA in every thread.
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();                       // protects `red` against the previous use
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float t = (lane < (int)(blockDim.x >> 5)) ? red[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

// vec: rows are whole 16-byte vectors and start on 16 bytes
template <typename T>
__device__ __forceinline__ void load_row(float* dst, const T* src, int cols, bool vec) {
    if (sizeof(T) == 2 && vec) {
        for (int i = threadIdx.x; i < cols / 8; i += blockDim.x) {
            uint4 v = reinterpret_cast<const uint4*>(src)[i];
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float2 f = __bfloat1622float2(h[k]);
                dst[8 * i + 2 * k] = f.x;
                dst[8 * i + 2 * k + 1] = f.y;
            }
        }
    } else if (sizeof(T) == 4 && vec) {
        for (int i = threadIdx.x; i < cols / 4; i += blockDim.x)
            reinterpret_cast<float4*>(dst)[i] = reinterpret_cast<const float4*>(src)[i];
    } else {
        for (int i = threadIdx.x; i < cols; i += blockDim.x) dst[i] = to_f32(src[i]);
    }
}

template <typename T>
__device__ __forceinline__ void store_row(T* dst, const float* src, int cols, bool vec) {
    if (sizeof(T) == 2 && vec) {
        for (int i = threadIdx.x; i < cols / 8; i += blockDim.x) {
            uint4 o;
            __nv_bfloat162 h0 = __floats2bfloat162_rn(src[8 * i], src[8 * i + 1]);
            __nv_bfloat162 h1 = __floats2bfloat162_rn(src[8 * i + 2], src[8 * i + 3]);
            __nv_bfloat162 h2 = __floats2bfloat162_rn(src[8 * i + 4], src[8 * i + 5]);
            __nv_bfloat162 h3 = __floats2bfloat162_rn(src[8 * i + 6], src[8 * i + 7]);
            o.x = *reinterpret_cast<uint32_t*>(&h0);
            o.y = *reinterpret_cast<uint32_t*>(&h1);
            o.z = *reinterpret_cast<uint32_t*>(&h2);
            o.w = *reinterpret_cast<uint32_t*>(&h3);
            reinterpret_cast<uint4*>(dst)[i] = o;
        }
    } else if (sizeof(T) == 4 && vec) {
        for (int i = threadIdx.x; i < cols / 4; i += blockDim.x)
            reinterpret_cast<float4*>(dst)[i] = reinterpret_cast<const float4*>(src)[i];
    } else {
        for (int i = threadIdx.x; i < cols; i += blockDim.x) dst[i] = from_f32<T>(src[i]);
    }
}

// y = (x - mean) * rstd * gamma + beta, row statistics saved for the backward
template <typename T>
__global__ void __launch_bounds__(kNormThreads)
layernorm_fwd_kernel(const T* __restrict__ x, int cols, const float* __restrict__ gamma, const float* __restrict__ beta,
                     float eps, T* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out, bool vec) {
    griddep_sync();
    extern __shared__ float row[];          // [cols] + 32
    float* red = row + cols;
    const int64_t r = blockIdx.x;
    load_row(row, x + r * cols, cols, vec);
    __syncthreads();
    float s = 0.f;
    for (int i = threadIdx.x; i < cols; i += blockDim.x) s += row[i];
    const float mean = block_sum(s, red) / (float)cols;
    float v = 0.f;
    for (int i = threadIdx.x; i < cols; i += blockDim.x) {
        float d = row[i] - mean;
        v += d * d;
    }
    const float var = block_sum(v, red) / (float)cols;
    const float rstd = 1.0f / sqrtf(var + eps);
    for (int i = threadIdx.x; i < cols; i += blockDim.x) {
        float n = (row[i] - mean) * rstd;
        if (gamma) n = n * gamma[i];
        if (beta) n = n + beta[i];
        row[i] = n;
    }
    __syncthreads();
    store_row(y + r * cols, row, cols, vec);
    if (threadIdx.x == 0) {
        if (mean_out) mean_out[r] = mean;
        if (rstd_out) rstd_out[r] = rstd;
    }
}

// dx = rstd * (g - mean(g) - xhat * mean(g * xhat)),  g = dy * gamma,  xhat = (x - mean) * rstd
template <typename T>
__global__ void __launch_bounds__(kNormThreads)
layernorm_bwd_dx_kernel(const T* __restrict__ dy, const T* __restrict__ x, int cols, const float* __restrict__ gamma,
                        const float* __restrict__ mean, const float* __restrict__ rstd, T* __restrict__ dx, bool vec) {
    griddep_sync();
    extern __shared__ float smem[];         // g[cols], xhat[cols], 32
    float* g = smem;
    float* xh = smem + cols;
    float* red = xh + cols;
    const int64_t r = blockIdx.x;
    load_row(g, dy + r * cols, cols, vec);
    load_row(xh, x + r * cols, cols, vec);
    __syncthreads();
    const float m = mean[r], rs = rstd[r];
    float s1 = 0.f, s2 = 0.f;
    for (int i = threadIdx.x; i < cols; i += blockDim.x) {
        float gi = g[i] * (gamma ? gamma[i] : 1.f);
        float xi = (xh[i] - m) * rs;
        g[i] = gi;
        xh[i] = xi;
        s1 += gi;
        s2 += gi * xi;
    }
    const float mg = block_sum(s1, red) / (float)cols;
    const float mgx = block_sum(s2, red) / (float)cols;
    for (int i = threadIdx.x; i < cols; i += blockDim.x) g[i] = rs * (g[i] - mg - xh[i] * mgx);
    __syncthreads();
    store_row(dx + r * cols, g, cols, vec);
}

// ---- rows of whole 16-byte vectors -------------------------------------------------------------------
// Both kernels are bound by HBM, which wants some 45 KB in flight per SM.
template <typename T> struct Vec16 { static constexpr int N = 16 / sizeof(T); };

template <typename T>
__device__ __forceinline__ void unpack16(const uint4& v, float* f) {
    if (sizeof(T) == 2) {
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float2 t = __bfloat1622float2(h[k]);
            f[2 * k] = t.x;
            f[2 * k + 1] = t.y;
        }
    } else {
        f[0] = __uint_as_float(v.x); f[1] = __uint_as_float(v.y); f[2] = __uint_as_float(v.z); f[3] = __uint_as_float(v.w);
    }
}

template <typename T>
__device__ __forceinline__ uint4 pack16(const float* f) {
    uint4 o;
    if (sizeof(T) == 2) {
        __nv_bfloat162 h0 = __floats2bfloat162_rn(f[0], f[1]), h1 = __floats2bfloat162_rn(f[2], f[3]);
        __nv_bfloat162 h2 = __floats2bfloat162_rn(f[4], f[5]), h3 = __floats2bfloat162_rn(f[6], f[7]);
        o.x = *reinterpret_cast<uint32_t*>(&h0); o.y = *reinterpret_cast<uint32_t*>(&h1);
        o.z = *reinterpret_cast<uint32_t*>(&h2); o.w = *reinterpret_cast<uint32_t*>(&h3);
    } else {
        o.x = __float_as_uint(f[0]); o.y = __float_as_uint(f[1]); o.z = __float_as_uint(f[2]); o.w = __float_as_uint(f[3]);
    }
    return o;
}

// V (4 or 8) consecutive floats of a parameter vector, 16-byte loads
template <int V>
__device__ __forceinline__ void load_param(const float* __restrict__ p, int c0, float* f) {
#pragma unroll
    for (int k = 0; k < V; k += 4) {
        const float4 t = *reinterpret_cast<const float4*>(p + c0 + k);
        f[k] = t.x; f[k + 1] = t.y; f[k + 2] = t.z; f[k + 3] = t.w;
    }
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums of N values over the CTA, one barrier; `red` is one of two buffers used in turn ([32][N] floats).
template <int N>
__device__ __forceinline__ void block_sums(float (&v)[N], float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    const int warps = blockDim.x >> 5;
    if (warps == 1) return;
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int k = 0; k < N; ++k) red[(threadIdx.x >> 5) * N + k] = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = 0.f;
    for (int w = 0; w < warps; ++w)
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] += red[w * N + k];
}

constexpr int kNormMaxRowThreads = 512;      // threads per row; longer rows take the kernels above

// A warp per row: lane l holds vectors l, l+32, ... of it, the statistics are shuffles, gamma and beta come from
// shared memory (in registers they cost as much as the row itself), and the next row is on its way while
// this one is worked on.
template <typename T, int NV>
__global__ void __launch_bounds__(kNormThreads)
layernorm_fwd_rows_kernel(const T* __restrict__ x, int64_t rows, int cols, const float* __restrict__ gamma,
                          const float* __restrict__ beta, float eps, T* __restrict__ y, float* __restrict__ mean_out,
                          float* __restrict__ rstd_out, int follow) {
    constexpr int V = Vec16<T>::N;
    extern __shared__ __align__(16) float params[];          // gamma, beta
    griddep_enter(follow);
    for (int i = threadIdx.x; i < cols; i += kNormThreads) {
        params[i] = gamma ? gamma[i] : 1.f;
        params[cols + i] = beta ? beta[i] : 0.f;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, nvec = cols / V;
    const float inv = 1.0f / (float)cols;
    const int64_t step = (int64_t)gridDim.x * (kNormThreads / 32);
    int64_t r = (int64_t)blockIdx.x * (kNormThreads / 32) + (threadIdx.x >> 5);
    uint4 raw[NV];
    auto fetch = [&](int64_t row) {
        const uint4* src = reinterpret_cast<const uint4*>(x + row * cols);
#pragma unroll
        for (int i = 0; i < NV; ++i)
            raw[i] = row < rows && i * 32 + lane < nvec ? src[i * 32 + lane] : make_uint4(0u, 0u, 0u, 0u);
    };
    fetch(r);
    for (; r < rows; r += step) {
        float f[NV][V];
        float sum[1] = {0.f};
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            unpack16<T>(raw[i], f[i]);
#pragma unroll
            for (int k = 0; k < V; ++k) sum[0] += f[i][k];
        }
        fetch(r + step);
        const float mean = warp_sum(sum[0]) * inv;
        float q = 0.f;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const bool in = i * 32 + lane < nvec;
#pragma unroll
            for (int k = 0; k < V; ++k) {
                f[i][k] = in ? f[i][k] - mean : 0.f;
                q += f[i][k] * f[i][k];
            }
        }
        const float rstd = 1.0f / sqrtf(warp_sum(q) * inv + eps);
        uint4* dst = reinterpret_cast<uint4*>(y + r * cols);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            if (i * 32 + lane < nvec) {
                const int c0 = (i * 32 + lane) * V;
                float gm[V], bt[V];
                load_param<V>(params, c0, gm);
                load_param<V>(params + cols, c0, bt);
#pragma unroll
                for (int k = 0; k < V; ++k) f[i][k] = fmaf(f[i][k] * rstd, gm[k], bt[k]);
                dst[i * 32 + lane] = pack16<T>(f[i]);
            }
        }
        if (lane == 0) {
            if (mean_out) mean_out[r] = mean;
            if (rstd_out) rstd_out[r] = rstd;
        }
    }
    griddep_leave(follow);
}

// dx as in layernorm_bwd_dx_kernel, plus `add` (a residual branch's gradient) if given.  A thread owns one
// 16-byte vector column of every row its CTA walks (8 BF16 or 4 FP32), so gamma and the sums for dgamma and
// dbeta are a few registers; a CTA takes R rows at a time, whose loads are all in flight together, and folds
// their sums with one barrier.  The column sums over a CTA's rows go to its row of `partial` ([2][CTAs, cols]),
// which a column-sum launch folds (a thousand CTAs adding to the same addresses took 100 us).
template <typename T, int R>
__global__ void __launch_bounds__(kNormMaxRowThreads)
layernorm_bwd_rows_kernel(const T* __restrict__ dy, const T* __restrict__ x, int64_t rows, int cols,
                          const float* __restrict__ gamma, const float* __restrict__ mean, const float* __restrict__ rstd,
                          const T* __restrict__ add, T* __restrict__ dx, float* __restrict__ partial) {
    constexpr int V = Vec16<T>::N;
    __shared__ float red[2][16 * 2 * R];
    griddep_sync();
    const int c0 = threadIdx.x * V;
    const bool mine = c0 < cols;
    const float inv = 1.0f / (float)cols;
    float gm[V], ag[V], ab[V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
        gm[k] = 1.f;
        ag[k] = ab[k] = 0.f;
    }
    if (mine && gamma) load_param<V>(gamma, c0, gm);
    int turn = 0;
    for (int64_t r0 = (int64_t)blockIdx.x * R; r0 < rows; r0 += (int64_t)gridDim.x * R, turn ^= 1) {
        uint4 graw[R], xraw[R], araw[R];
        float m[R], rs[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const bool in = mine && r0 + r < rows;
            const int64_t at = (r0 + r) * cols + c0;
            graw[r] = in ? *reinterpret_cast<const uint4*>(dy + at) : make_uint4(0u, 0u, 0u, 0u);
            xraw[r] = in ? *reinterpret_cast<const uint4*>(x + at) : make_uint4(0u, 0u, 0u, 0u);
            if (add) araw[r] = in ? *reinterpret_cast<const uint4*>(add + at) : make_uint4(0u, 0u, 0u, 0u);
            m[r] = r0 + r < rows ? mean[r0 + r] : 0.f;
            rs[r] = r0 + r < rows ? rstd[r0 + r] : 0.f;
        }
        float g[R][V], xh[R][V], s[2 * R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            unpack16<T>(graw[r], g[r]);
            unpack16<T>(xraw[r], xh[r]);
            s[2 * r] = s[2 * r + 1] = 0.f;
#pragma unroll
            for (int k = 0; k < V; ++k) {
                xh[r][k] = (xh[r][k] - m[r]) * rs[r];
                ag[k] = fmaf(g[r][k], xh[r][k], ag[k]);
                ab[k] += g[r][k];
                g[r][k] *= gm[k];
                s[2 * r] += g[r][k];
                s[2 * r + 1] = fmaf(g[r][k], xh[r][k], s[2 * r + 1]);
            }
        }
        block_sums<2 * R>(s, red[turn]);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (!mine || r0 + r >= rows) break;
            const float mg = s[2 * r] * inv, mgx = s[2 * r + 1] * inv;
#pragma unroll
            for (int k = 0; k < V; ++k) g[r][k] = rs[r] * (g[r][k] - mg - xh[r][k] * mgx);
            if (add) {
                float t[V];
                unpack16<T>(araw[r], t);
#pragma unroll
                for (int k = 0; k < V; ++k) g[r][k] += t[k];
            }
            *reinterpret_cast<uint4*>(dx + (r0 + r) * cols + c0) = pack16<T>(g[r]);
        }
    }
    if (!mine || !partial) return;
    float* pg = partial + (int64_t)blockIdx.x * cols + c0;
    float* pb = pg + (int64_t)gridDim.x * cols;
#pragma unroll
    for (int k = 0; k < V; k += 4) {
        *reinterpret_cast<float4*>(pg + k) = make_float4(ag[k], ag[k + 1], ag[k + 2], ag[k + 3]);
        *reinterpret_cast<float4*>(pb + k) = make_float4(ab[k], ab[k + 1], ab[k + 2], ab[k + 3]);
    }
}

// dgamma[j] += sum_r dy[r,j] * xhat[r,j],  dbeta[j] += sum_r dy[r,j]   (outputs zeroed by the caller)
template <typename T>
__global__ void layernorm_bwd_params_kernel(const T* __restrict__ dy, const T* __restrict__ x, int64_t rows, int cols,
                                            const float* __restrict__ mean, const float* __restrict__ rstd,
                                            float* __restrict__ dgamma, float* __restrict__ dbeta) {
    griddep_sync();
    __shared__ float pg[8][33], pb[8][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int col = blockIdx.x * 32 + tx;
    float ag = 0.f, ab = 0.f;
    if (col < cols) {
        for (int64_t r = (int64_t)blockIdx.y * 8 + ty; r < rows; r += (int64_t)gridDim.y * 8) {
            float d = to_f32(dy[r * cols + col]);
            float xh = (to_f32(x[r * cols + col]) - mean[r]) * rstd[r];
            ag += d * xh;
            ab += d;
        }
    }
    pg[ty][tx] = ag;
    pb[ty][tx] = ab;
    __syncthreads();
    if (ty == 0 && col < cols) {
        float sg = 0.f, sb = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            sg += pg[k][tx];
            sb += pb[k][tx];
        }
        if (dgamma) atomicAdd(dgamma + col, sg);
        if (dbeta) atomicAdd(dbeta + col, sb);
    }
}

// ---- GELU (gelu.cuh) ------------------------------------------------------------------------------
template <typename T, bool BWD>
__global__ void gelu_kernel(T* __restrict__ out, const T* __restrict__ x, const T* __restrict__ dy, int64_t n) {
    griddep_sync();
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (; i < n; i += step) {
        float v = to_f32(x[i]);
        out[i] = from_f32<T>(BWD ? to_f32(dy[i]) * gelu_grad_f(v) : gelu_f(v));
    }
}

// 8 BF16 or 4 FP32 per 16-byte access; a thread issues the loads of kGeluUnroll accesses (a CTA
// covers kGeluUnroll consecutive runs of 256 vectors) before it computes, to keep enough bytes in
// flight with one or two input streams.
constexpr int kGeluUnroll = 4;
template <typename T, bool BWD>
__global__ void __launch_bounds__(256)
gelu_vec_kernel(T* __restrict__ out, const T* __restrict__ x, const T* __restrict__ dy, int64_t nvec) {
    griddep_sync();
    constexpr int V = 16 / sizeof(T);
    const int64_t chunk = (int64_t)gridDim.x * 256 * kGeluUnroll;
    for (int64_t base = (int64_t)blockIdx.x * 256 * kGeluUnroll + threadIdx.x; base < nvec; base += chunk) {
        uint4 xv[kGeluUnroll], dv[kGeluUnroll];
#pragma unroll
        for (int u = 0; u < kGeluUnroll; ++u) {
            const int64_t i = base + u * 256;
            if (i < nvec) {
                xv[u] = reinterpret_cast<const uint4*>(x)[i];
                if (BWD) dv[u] = reinterpret_cast<const uint4*>(dy)[i];
            }
        }
#pragma unroll
        for (int u = 0; u < kGeluUnroll; ++u) {
            const int64_t i = base + u * 256;
            if (i >= nvec) break;
            const T* xe = reinterpret_cast<const T*>(&xv[u]);
            const T* de = reinterpret_cast<const T*>(&dv[u]);
            uint4 ov;
            T* oe = reinterpret_cast<T*>(&ov);
#pragma unroll
            for (int k = 0; k < V; ++k) {
                float v = to_f32(xe[k]);
                oe[k] = from_f32<T>(BWD ? to_f32(de[k]) * gelu_grad_f(v) : gelu_f(v));
            }
            reinterpret_cast<uint4*>(out)[i] = ov;
        }
    }
}

static inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

template <typename T, bool BWD>
static int launch_gelu(void* out, const void* x, const void* dy, int64_t n) {
    constexpr int V = 16 / sizeof(T);
    const bool vec = (n % V) == 0 && aligned16(out) && aligned16(x) && (!BWD || aligned16(dy));
    int64_t items = vec ? n / V : n;
    int64_t blocks = ceil_div(items, vec ? 256 * kGeluUnroll : 256);   // the loops are grid-stride
    if (blocks > 0x7fffffffLL) blocks = 0x7fffffffLL;
    ProfileScope prof(BWD ? "gelu_bwd" : "gelu_fwd");
    if (vec)
        BOATCU_RUN((gelu_vec_kernel<T, BWD>), (unsigned)blocks, 256, 0, (T*)out, (const T*)x, (const T*)dy, items);
    else
        BOATCU_RUN((gelu_kernel<T, BWD>), (unsigned)blocks, 256, 0, (T*)out, (const T*)x, (const T*)dy, n);
    BOATCU_LAUNCH_OK("gelu");
    return 0;
}

// Whether rows of this length in these arrays are whole 16-byte vectors at 16-byte addresses.
static bool rows_of_vectors(int type, int64_t cols, std::initializer_list<const void*> ptrs) {
    bool ok = cols % (type == BOAT_CUDA_BF16 ? 8 : 4) == 0;
    for (const void* q : ptrs) ok = ok && aligned16(q);
    return ok;
}
// Whether the kernels for such rows take this length.
static bool rows_kernel_fits(int type, int64_t cols, std::initializer_list<const void*> ptrs) {
    return cols / (type == BOAT_CUDA_BF16 ? 8 : 4) <= kNormMaxRowThreads && rows_of_vectors(type, cols, ptrs);
}

template <typename T, int NV>
static int layernorm_fwd_launch(const void* x, int64_t rows, int64_t cols, const float* gamma, const float* beta, float eps, void* y,
                                float* mean_out, float* rstd_out) {
    const size_t smem = 2 * (size_t)cols * sizeof(float);
    int64_t blocks = ceil_div(rows, kNormThreads / 32);
    if (blocks > (int64_t)sm_count() * 8) blocks = (int64_t)sm_count() * 8;
    LaunchTurn turn;
    turn.reads(x, (size_t)rows * cols * sizeof(T));
    turn.reads(gamma, (size_t)cols * 4);
    turn.reads(beta, (size_t)cols * 4);
    turn.writes(y, (size_t)rows * cols * sizeof(T));
    turn.writes(mean_out, (size_t)rows * 4);
    turn.writes(rstd_out, (size_t)rows * 4);
    BOATCU_RUN_IN_TURN(turn, (layernorm_fwd_rows_kernel<T, NV>), (unsigned)blocks, kNormThreads, smem, (const T*)x, rows, (int)cols, gamma, beta, eps, (T*)y,
                       mean_out, rstd_out, turn.follow());
    BOATCU_LAUNCH_OK("layernorm_fwd_rows");
    return 0;
}

template <typename T>
static int layernorm_fwd_rows(const void* x, int64_t rows, int64_t cols, const float* gamma, const float* beta,
                              float eps, void* y, float* mean_out, float* rstd_out) {
    const int64_t nv = ceil_div(cols, 32 * Vec16<T>::N);
    if (nv <= 1) return layernorm_fwd_launch<T, 1>(x, rows, cols, gamma, beta, eps, y, mean_out, rstd_out);
    if (nv <= 2) return layernorm_fwd_launch<T, 2>(x, rows, cols, gamma, beta, eps, y, mean_out, rstd_out);
    if (nv <= 3) return layernorm_fwd_launch<T, 3>(x, rows, cols, gamma, beta, eps, y, mean_out, rstd_out);
    if (nv <= 4) return layernorm_fwd_launch<T, 4>(x, rows, cols, gamma, beta, eps, y, mean_out, rstd_out);
    return layernorm_fwd_launch<T, 8>(x, rows, cols, gamma, beta, eps, y, mean_out, rstd_out);
}

template <typename T, int R>
static int layernorm_bwd_rows_launch(unsigned blocks, int threads, const void* dy, const void* x, int64_t rows, int64_t cols, const float* gamma,
                                     const float* mean, const float* rstd, const void* add, void* dx, void* partial) {
    BOATCU_RUN((layernorm_bwd_rows_kernel<T, R>), blocks, threads, 0, (const T*)dy, (const T*)x, rows, (int)cols, gamma, mean, rstd,
               (const T*)add, (T*)dx, (float*)partial);
    BOATCU_LAUNCH_OK("layernorm_bwd_rows");
    return 0;
}

template <typename T>
static int layernorm_bwd_rows(const void* dy, const void* x, int64_t rows, int64_t cols, const float* gamma,
                              const float* mean, const float* rstd, const void* add, void* dx, float* dgamma, float* dbeta) {
    const int threads = (int)ceil_div(cols / Vec16<T>::N, 32) * 32;
    const bool four = rows >= 4 * 2 * (int64_t)sm_count();            // every SM gets two CTAs with four rows at least
    int64_t blocks = ceil_div(rows, four ? 4 : 1);
    const int64_t most = (int64_t)sm_count() * (1024 / threads > 8 ? 8 : 1024 / threads);
    if (blocks > most) blocks = most;
    void* partial = nullptr;
    if (dgamma || dbeta)
        if (int rc = boat_cuda_malloc(&partial, 2 * (size_t)blocks * (size_t)cols * sizeof(float))) return rc;
    int rc = four ? layernorm_bwd_rows_launch<T, 4>((unsigned)blocks, threads, dy, x, rows, cols, gamma, mean, rstd, add, dx, partial)
                  : layernorm_bwd_rows_launch<T, 1>((unsigned)blocks, threads, dy, x, rows, cols, gamma, mean, rstd, add, dx, partial);
    if (!partial) return rc;
    const void* from[2] = {partial, (const float*)partial + blocks * cols};
    float* to[2] = {dgamma, dbeta};
    const int first = dgamma ? 0 : 1, count = (dgamma ? 1 : 0) + (dbeta ? 1 : 0);
    if (rc == 0) rc = colsum_multi(from + first, BOAT_CUDA_F32, blocks, cols, to + first, count);
    const int freed = boat_cuda_free(partial);
    return rc ? rc : freed;
}

}  // namespace boatcu

using namespace boatcu;

extern "C" {

int boat_cuda_layernorm_fwd(const void* x, int type, int64_t rows, int64_t cols, const float* gamma, const float* beta,
                            float eps, void* y, float* mean_out, float* rstd_out) {
    if (rows <= 0 || cols <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    if (cols > 12000) return set_error(50, "layernorm: row length %lld exceeds 12000", (long long)cols);
    if (rows > 0x7fffffffLL) return set_error(50, "layernorm: too many rows");
    size_t smem = ((size_t)cols + 32) * sizeof(float);
    ProfileScope prof("layernorm_fwd");
    if (cols <= 8 * 32 * (type == BOAT_CUDA_BF16 ? 8 : 4) && rows_kernel_fits(type, cols, {x, y}))
        return type == BOAT_CUDA_BF16 ? layernorm_fwd_rows<__nv_bfloat16>(x, rows, cols, gamma, beta, eps, y, mean_out, rstd_out)
                                      : layernorm_fwd_rows<float>(x, rows, cols, gamma, beta, eps, y, mean_out, rstd_out);
    const bool vec = rows_of_vectors(type, cols, {x, y});
    if (type == BOAT_CUDA_BF16) {
        auto k = layernorm_fwd_kernel<__nv_bfloat16>;
        BOATCU_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        BOATCU_RUN(k, (unsigned)rows, kNormThreads, smem, (const __nv_bfloat16*)x, (int)cols, gamma, beta, eps,
                                                            (__nv_bfloat16*)y, mean_out, rstd_out, vec);
    } else {
        auto k = layernorm_fwd_kernel<float>;
        BOATCU_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        BOATCU_RUN(k, (unsigned)rows, kNormThreads, smem, (const float*)x, (int)cols, gamma, beta, eps, (float*)y,
                                                            mean_out, rstd_out, vec);
    }
    BOATCU_LAUNCH_OK("layernorm_fwd");
    return 0;
}

int boat_cuda_layernorm_bwd(const void* dy, const void* x, int type, int64_t rows, int64_t cols, const float* gamma,
                            const float* mean, const float* rstd, void* dx, float* dgamma, float* dbeta) {
    return boat_cuda_layernorm_bwd_add(dy, x, type, rows, cols, gamma, mean, rstd, NULL, dx, dgamma, dbeta);
}

int boat_cuda_layernorm_bwd_add(const void* dy, const void* x, int type, int64_t rows, int64_t cols, const float* gamma,
                                const float* mean, const float* rstd, const void* add, void* dx, float* dgamma, float* dbeta) {
    if (rows <= 0 || cols <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    if (cols > 12000) return set_error(50, "layernorm: row length %lld exceeds 12000", (long long)cols);
    size_t smem = (2 * (size_t)cols + 32) * sizeof(float);
    ProfileScope prof("layernorm_bwd");
    if (rows_kernel_fits(type, cols, {dy, x, dx, gamma, add}))
        return type == BOAT_CUDA_BF16 ? layernorm_bwd_rows<__nv_bfloat16>(dy, x, rows, cols, gamma, mean, rstd, add, dx, dgamma, dbeta)
                                      : layernorm_bwd_rows<float>(dy, x, rows, cols, gamma, mean, rstd, add, dx, dgamma, dbeta);
    if (dgamma) BOATCU_CHECK(cudaMemsetAsync(dgamma, 0, (size_t)cols * sizeof(float), stream()));
    if (dbeta) BOATCU_CHECK(cudaMemsetAsync(dbeta, 0, (size_t)cols * sizeof(float), stream()));
    const bool vec = rows_of_vectors(type, cols, {dy, x, dx});
    dim3 pgrid((unsigned)ceil_div(cols, 32), 1);
    int64_t want = (int64_t)sm_count() * 8 / pgrid.x, max_y = ceil_div(rows, 8);
    pgrid.y = (unsigned)(want < 1 ? 1 : (want > max_y ? max_y : want));
    if (type == BOAT_CUDA_BF16) {
        typedef __nv_bfloat16 bf;
        auto k = layernorm_bwd_dx_kernel<bf>;
        BOATCU_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        BOATCU_RUN(k, (unsigned)rows, kNormThreads, smem, (const bf*)dy, (const bf*)x, (int)cols, gamma, mean, rstd, (bf*)dx, vec);
        BOATCU_LAUNCH_OK("layernorm_bwd_dx");
        if (dgamma || dbeta) {
            BOATCU_RUN(layernorm_bwd_params_kernel<bf>, pgrid, 256, 0, (const bf*)dy, (const bf*)x, rows, (int)cols, mean, rstd, dgamma, dbeta);
            BOATCU_LAUNCH_OK("layernorm_bwd_params");
        }
    } else {
        auto k = layernorm_bwd_dx_kernel<float>;
        BOATCU_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        BOATCU_RUN(k, (unsigned)rows, kNormThreads, smem, (const float*)dy, (const float*)x, (int)cols, gamma, mean, rstd, (float*)dx, vec);
        BOATCU_LAUNCH_OK("layernorm_bwd_dx");
        if (dgamma || dbeta) {
            BOATCU_RUN(layernorm_bwd_params_kernel<float>, pgrid, 256, 0, (const float*)dy, (const float*)x, rows, (int)cols, mean, rstd, dgamma, dbeta);
            BOATCU_LAUNCH_OK("layernorm_bwd_params");
        }
    }
    return add ? boat_cuda_lincomb(dx, dx, 1.0f, add, 1.0f, type, rows * cols) : 0;
}

int boat_cuda_gelu_fwd(void* y, const void* x, int type, int64_t n) {
    if (n <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    return type == BOAT_CUDA_BF16 ? launch_gelu<__nv_bfloat16, false>(y, x, nullptr, n) : launch_gelu<float, false>(y, x, nullptr, n);
}

int boat_cuda_gelu_bwd(void* dx, const void* dy, const void* x, int type, int64_t n) {
    if (n <= 0) return 0;
    if (int rc = ensure_init()) return rc;
    return type == BOAT_CUDA_BF16 ? launch_gelu<__nv_bfloat16, true>(dx, x, dy, n) : launch_gelu<float, true>(dx, x, dy, n);
}

}  // extern "C"
