// common.cuh - shared helpers for the sm_100a kernels: status handling, launch accounting,
// storage-type helpers.  Internal to the CUDA backend.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stdio.h>
#include "boat_cuda.h"

namespace boatcu {

// Records a failure text for boat_cuda_last_error() and returns the status to hand back.
int set_error(int status, const char* fmt, ...);
cudaStream_t stream();
void count_launch(int n = 1);
int ensure_init();
bool ready();          // has boat_cuda_init (or a first call) bound the library to a device yet?
int bound_device();    // index of that device, -1 before
int sm_count();        // its number of SMs (grid sizing); 1 before the library is bound
int comm_stream_sync();   // waits for gradient sums still running on the communication stream

// Optional per-kernel timing (boat_cuda_profile_*): while enabled, a scope records a CUDA
// event pair on the library stream around the launches it encloses.
struct ProfileScope {
    explicit ProfileScope(const char* name);
    ~ProfileScope();
    int slot;
};

#define BOATCU_CHECK(expr)                                                          \
    do {                                                                            \
        cudaError_t err__ = (expr);                                                 \
        if (err__ != cudaSuccess)                                                   \
            return boatcu::set_error(1000 + (int)err__, "%s failed: %s (%s:%d)",   \
                                     #expr, cudaGetErrorString(err__), __FILE__, __LINE__); \
    } while (0)

// After a kernel launch: catches bad launch configurations without synchronising.
#define BOATCU_LAUNCH_OK(name)                                                      \
    do {                                                                            \
        cudaError_t err__ = cudaGetLastError();                                     \
        if (err__ != cudaSuccess)                                                   \
            return boatcu::set_error(1000 + (int)err__, "launch of %s failed: %s", \
                                     name, cudaGetErrorString(err__));              \
        boatcu::count_launch();                                                     \
    } while (0)

// Kernels of the library follow one another on one stream, and a launch that only begins when its
// predecessor has drained costs 2-4 us of idle GPU - as much as a small kernel.  So every kernel is
// launched as the programmatic dependent of the one before: its CTAs may be placed as soon as all CTAs
// of the predecessor are running, do what depends on nobody (barriers, tensor memory, descriptors), and
// wait in griddep_sync() until the predecessor is complete and its writes are visible.  EVERY kernel
// calls it before its first access to global memory, in every thread: completion of a kernel then
// implies completion of all kernels before it.
__device__ __forceinline__ void griddep_sync() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// GEMMs, and the passes that prepare their operands and outputs, name the memory they read and write (LaunchTurn).  Such a
// kernel lets its successor's CTAs be placed only once it has passed its own wait (kRelease): what came before it is
// complete when they run.  A successor that also names its memory, and touches none that matters to the kernels which may still
// be running, does not wait for them (kBeside): a weight gradient beside an input gradient, a conversion beside either.  It
// fills the SMs as they come free, without the gap between two launches, and waits for its predecessor at its
// end instead, so that its completion still implies that of all kernels before it.  A weight gradient that is split along K
// and overwrites its output waits behind the launch that clears it, and so for what is before that; what follows it may run
// beside it.
// Only within a sequence (boat_cuda_launches_begin): the first launch of one, and every launch outside one, waits for whatever is
// before it on the stream, a program's own kernels or NCCL's too (launch_order.h).
// The step with every kernel waiting and so: encoder block of 4 x 333 x 768 BF16 225 us and 218, residual attention of 4 x 250 x 256
// FP32 149 and 142, 8 x 512 x 512 TF32 177 and 171, 8 x 1000 x 1024 BF16 350 and 345; a lone forward of 1 x 128 x 1024 23 and 23.
enum Follow { kRelease = 1, kBeside = 2 };
__device__ __forceinline__ void griddep_enter(int follow) {
    if (follow != kBeside) asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void griddep_leave(int follow) {
    if (follow == kBeside) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// One launch on the library stream.  Holds the order of launches still while it lives, so that the kernels
// before are the ones it is compared with.  reads() and writes() name what the kernel touches, all of it; follow() then says
// how it is to be launched.  A turn that names nothing is an ordinary launch, and so is what follows a copy, a memset or a wait for
// an event on the stream.
class LaunchTurn {
public:
    LaunchTurn();
    ~LaunchTurn();
    LaunchTurn(const LaunchTurn&) = delete;
    void reads(const void* p, size_t bytes) { name(p, bytes, false); }
    void writes(const void* p, size_t bytes) { name(p, bytes, true); }
    // rows of `cols` elements of `es` bytes, ld elements apart
    void reads(const void* p, int64_t rows, int64_t cols, int64_t ld, size_t es) { reads(p, span(rows, cols, ld, es)); }
    void writes(const void* p, int64_t rows, int64_t cols, int64_t ld, size_t es) { writes(p, span(rows, cols, ld, es)); }
    int follow();
    cudaError_t launched(cudaError_t err) {      // a turn without a launch that worked leaves nothing to be beside of
        launched_ = err == cudaSuccess;
        return err;
    }

private:
    static size_t span(int64_t rows, int64_t cols, int64_t ld, size_t es) { return rows > 0 && cols > 0 ? (size_t)((rows - 1) * ld + cols) * es : 0; }
    void name(const void* p, size_t bytes, bool written);
    bool launched_ = false;
};

// Something other than a named kernel comes next on the library stream, or the stream changes.
void ordinary_launch_next();

template <typename... P, typename... A>
inline cudaError_t launch_in_turn(LaunchTurn& turn, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, unsigned cluster, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream();
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return turn.launched(cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...));
}
template <typename... P, typename... A>
inline cudaError_t launch_dependent(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, unsigned cluster, A&&... args) {
    LaunchTurn turn;
    return launch_in_turn(turn, kern, grid, block, smem, cluster, static_cast<A&&>(args)...);
}
static inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Dynamic shared memory of a launch of `ctas` CTAs that need `smem` bytes each: so much that no SM takes
// more than its even share.  CTAs that are placed behind a running predecessor go where it leaves room, two
// to an SM while others stay empty: 512 x 512 x 4096 on 128 CTAs of gemm_simt took 146 us, spread 90.
constexpr int kSpreadSmem = 114 * 1024;                   // the most this asks for: no two of them fit an SM's 228 KB
inline int spread_smem(int smem, int64_t ctas) {
    const int64_t share = ceil_div(ctas, sm_count());
    const int least = share <= 3 ? (int)(228 / (share + 1)) * 1024 : 0;
    return smem > least ? smem : least;
}

#define BOATCU_RUN_IN_TURN(turn, kern, grid, block, smem, ...) \
    BOATCU_CHECK(boatcu::launch_in_turn(turn, kern, dim3(grid), dim3(block), smem, 1, __VA_ARGS__))
#define BOATCU_RUN(kern, grid, block, smem, ...) \
    BOATCU_CHECK(boatcu::launch_dependent(kern, dim3(grid), dim3(block), smem, 1, __VA_ARGS__))

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

inline size_t type_size(int t) { return t == BOAT_CUDA_BF16 ? 2 : 4; }

// FP32 value rounded to the nearest TF32 number (ties away from zero), still an FP32 bit pattern.
__device__ __forceinline__ float round_to_tf32(float v) {
    uint32_t t;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(t) : "f"(v));
    return __uint_as_float(t);
}
// Output element of BOAT_CUDA_F32_TF32: stored as float, rounded on conversion.
struct f32_tf32 { float v; };
template <> __device__ __forceinline__ f32_tf32 from_f32<f32_tf32>(float v) { return f32_tf32{round_to_tf32(v)}; }


// out[r] = sum_d A[r,d]*B[r,d] over [rows, cols] row-major buffers of storage type `type`.
int rowdot(const void* A, const void* B, int type, int64_t rows, int64_t cols, float* out);
// What the BF16 tensor-core backward starts from (hs 64 or 128): per row delta2 = -scale * sum_d dO*O and
// lse2 = -lse * log2(e), each unit of S rows padded to padded_S entries (0 and -inf), and zeros in dq
// [units*S, hs].  units * padded_S must fit 31 bits.
int attn_bwd_prepare(const void* dO, const void* O, const float* lse, int64_t units, int64_t S, int64_t padded_S, int64_t hs, float scale,
                     float* delta2, float* lse2, float* dq);

// CUDA-core (exact FP32 accumulate) implementations, any shape.
// gemm_simt_grouped: up to four problems of one shape in one launch; bias may be NULL or hold NULLs; with
// `colsum` (may be NULL or hold NULLs) problem g also writes the sums of B's columns over K.  `add`: both are
// added to what is there (FP32 output).
int gemm_simt_grouped(int trans_a, int trans_b, int groups, int64_t M, int64_t N, int64_t K, const void* const* A,
                      int64_t lda, const void* const* B, int64_t ldb, int in_type, void* const* C, int64_t ldc,
                      int out_type, const float* const* bias, float* const* colsum, bool add = false);
// boat_cuda_linear_grads in FP32 on the CUDA cores, for problems so small that one launch is worth it; 13 for others.
int gemm_simt_grads(int groups, int64_t T, int64_t I, int64_t O, const void* const* X, const void* const* dY, const void* const* W,
                    void* const* dX, float* const* dW, float* const* db);
// boat_cuda_colsum_multi
int colsum_multi(const void* const* X, int x_type, int64_t rows, int64_t cols, float* const* out, int count);
int attn_fwd_simt(int64_t units, int64_t S, int64_t hs, int causal, float scale, const void* Q, const void* K,
                  const void* V, int io_type, void* O, float* lse);
// With O it works delta out from O and dO, for what attn_bwd_simt_makes_delta takes and where no result shares memory with O; without,
// `delta` is given (rowdot).
bool attn_bwd_simt_makes_delta(int64_t units, int64_t S, int64_t hs, int io_type);
int attn_bwd_simt(int64_t units, int64_t S, int64_t hs, int causal, float scale, const void* Q, const void* K,
                  const void* V, const void* O, const void* dO, const float* lse, const float* delta, int io_type,
                  void* dQ, void* dK, void* dV);

// boat_cuda_attn_bwd with a say in the kernels: without `tensor_cores` the CUDA-core ones, whose scratch is
// what boat_cuda_attn_bwd_scratch_bytes gives for FP32 (delta only).
int attn_bwd_core(int mma, bool tensor_cores, int64_t units, int64_t S, int64_t hs, int causal, float scale, const void* Q,
                  const void* K, const void* V, const void* O, const void* dO, const float* lse, int io_type, void* dQ,
                  void* dK, void* dV, void* scratch, size_t scratch_bytes);

// tcgen05 implementations, for what gemm_tc_supported takes.
bool gemm_tc_supported(int mma, int trans_a, int trans_b, int64_t M, int64_t N, int64_t K, const void* A,
                       int64_t lda, const void* B, int64_t ldb, int in_type, const void* C, int64_t ldc,
                       int out_type);
int gemm_tc(int mma, int trans_a, int trans_b, int64_t M, int64_t N, int64_t K, const void* A, int64_t lda,
            const void* B, int64_t ldb, int in_type, void* C, int64_t ldc, int out_type, const float* bias);
// boat_cuda_weight_grads: dW = X^T . dY (FP32) and, unless db is NULL, the column sums of dY, in one pass; with `add`
// both are added to what is there.
int gemm_tc_weight_grads(int mma, int groups, int64_t I, int64_t O, int64_t T, const void* const* X, const void* const* dY,
                         float* const* dW, float* const* db, bool add);
// C = sum over the groups of op(A[g]).op(B[g]), one accumulator.
int gemm_tc_sum(int mma, int trans_a, int trans_b, int groups, int64_t M, int64_t N, int64_t K, const void* const* A,
                int64_t lda, const void* const* B, int64_t ldb, void* C, int64_t ldc, int out_type);
// BF16 products with element-wise work in the epilogue (BOAT_EPI_*); aux is laid out like C.
bool gemm_tc_fused_supported(int epilogue, int trans_a, int trans_b);
int gemm_tc_fused(int epilogue, int64_t M, int64_t N, int64_t K, const void* A, int64_t lda, const void* B, int64_t ldb,
                  void* C, int64_t ldc, const float* bias, void* aux);
void gemm_tc_set_yielding(bool on);
// `groups` (1..4) problems of one shape, layout and type in one launch; bias may be NULL or hold NULLs.
int gemm_tc_grouped(int mma, int trans_a, int trans_b, int groups, int64_t M, int64_t N, int64_t K,
                    const void* const* A, int64_t lda, const void* const* B, int64_t ldb, void* const* C,
                    int64_t ldc, int out_type, const float* const* bias);

}  // namespace boatcu
