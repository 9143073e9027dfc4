/* The attention layer's host code over a CUDA layer that computes nothing: call number `fail_at` of a forward,
 * backward and update returns an error.  Whatever fails, freeing the layer has to bring back every block. */
#include <boat/layers.h>
#include <boat/layers/attention.h>
#include <boat/optimizers.h>
#include <boat/tensor.h>
#include <boat_cuda.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static int calls, fail_at = -1, device_blocks, pinned_blocks;

static int step(void) { return calls++ == fail_at ? 99 : 0; }

int boat_cuda_init(int device) { (void)device; return step(); }
int boat_cuda_device_count(void) { return 1; }
const char* boat_cuda_last_error(void) { return "made up"; }
static int open_sequences;
void boat_cuda_launches_begin(void) { ++open_sequences; }
void boat_cuda_launches_end(void) { --open_sequences; }
int boat_cuda_sync(void) { return step(); }
size_t boat_cuda_bytes_in_use(void) { return 0; }
int boat_cuda_malloc(void** p, size_t n) {
    *p = NULL;
    if (step()) return 99;
    *p = calloc(1, n ? n : 1);
    ++device_blocks;
    return 0;
}
int boat_cuda_free(void* p) {
    if (p) --device_blocks;
    free(p);
    return 0;
}
void* boat_cuda_host_alloc(size_t n) {
    if (step()) return NULL;
    ++pinned_blocks;
    return calloc(1, n);
}
int boat_cuda_host_free(void* p) {
    if (p) --pinned_blocks;
    free(p);
    return 0;
}
static int copy(void* d, const void* s, size_t n) {
    if (step()) return 99;
    memcpy(d, s, n);
    return 0;
}
int boat_cuda_memcpy_h2d(void* d, const void* s, size_t n) { return copy(d, s, n); }
int boat_cuda_memcpy_h2d_async(void* d, const void* s, size_t n) { return copy(d, s, n); }
int boat_cuda_memcpy_d2h(void* d, const void* s, size_t n) { return copy(d, s, n); }
int boat_cuda_memcpy_d2d(void* d, const void* s, size_t n) { return copy(d, s, n); }
int boat_cuda_upload_async(void* d, const void* s, size_t n) { return copy(d, s, n); }
int boat_cuda_download_async(void* d, const void* s, size_t n) { return copy(d, s, n); }
int boat_cuda_stage_copy(void* d, const void* s, size_t n, int down) { (void)down; return copy(d, s, n); }
int boat_cuda_memset(void* d, int v, size_t n) { memset(d, v, n); return step(); }
int boat_cuda_copies_after_compute(void) { return step(); }
int boat_cuda_join_uploads(void) { return step(); }
int boat_cuda_comm_world(void) { return 1; }
int boat_cuda_allreduce_begin(float* const* p, const int64_t* n, int k) { (void)p; (void)n; (void)k; return step(); }
int boat_cuda_allreduce_join(void) { return step(); }
int boat_cuda_allreduce_pending(void) { return 0; }
int boat_cuda_gemm_set_yielding(int on) { (void)on; return 0; }
size_t boat_cuda_attn_bwd_scratch_bytes(int mma, int64_t units, int64_t S, int64_t hs) { (void)mma; return (size_t)(units * S * (hs + 3)) * 4; }
int boat_cuda_axpy_multi(float* const* y, const float* const* x, float a, const int64_t* n, int k) { (void)y; (void)x; (void)a; (void)n; (void)k; return step(); }
int boat_cuda_cast(void* d, int dt, const void* s, int st, int64_t n) { (void)d; (void)dt; (void)s; (void)st; (void)n; return step(); }
int boat_cuda_round_tf32(float* y, const float* x, int64_t n) { (void)y; (void)x; (void)n; return step(); }
int boat_cuda_lincomb(void* y, const void* a, float al, const void* b, float be, int t, int64_t n) { (void)y; (void)a; (void)al; (void)b; (void)be; (void)t; (void)n; return step(); }
int boat_cuda_convert_multi(void* const* d, int t, const float* const* s, const int64_t* n, int k) { (void)d; (void)t; (void)s; (void)n; (void)k; return step(); }
int boat_cuda_gemm(int mma, int ta, int tb, int64_t M, int64_t N, int64_t K, const void* A, int64_t lda, const void* B, int64_t ldb, int it, void* C, int64_t ldc,
                   int ot, const float* bias) {
    (void)mma; (void)ta; (void)tb; (void)M; (void)N; (void)K; (void)A; (void)lda; (void)B; (void)ldb; (void)it; (void)C; (void)ldc; (void)ot; (void)bias;
    return step();
}
int boat_cuda_gemm_grouped(int mma, int ta, int tb, int g, int64_t M, int64_t N, int64_t K, const void* const* A, int64_t lda, const void* const* B, int64_t ldb,
                           int it, void* const* C, int64_t ldc, int ot, const float* const* bias) {
    (void)mma; (void)ta; (void)tb; (void)g; (void)M; (void)N; (void)K; (void)A; (void)lda; (void)B; (void)ldb; (void)it; (void)C; (void)ldc; (void)ot; (void)bias;
    return step();
}
int boat_cuda_gemm_fused(int mma, int e, int ta, int tb, int64_t M, int64_t N, int64_t K, const void* A, int64_t lda, const void* B, int64_t ldb, int t, void* C,
                         int64_t ldc, const float* bias, void* aux) {
    (void)mma; (void)e; (void)ta; (void)tb; (void)M; (void)N; (void)K; (void)A; (void)lda; (void)B; (void)ldb; (void)t; (void)C; (void)ldc; (void)bias; (void)aux;
    return step();
}
int boat_cuda_gemm_sum(int mma, int ta, int tb, int g, int64_t M, int64_t N, int64_t K, const void* const* A, int64_t lda, const void* const* B, int64_t ldb, int it,
                       void* C, int64_t ldc, int ot) {
    (void)mma; (void)ta; (void)tb; (void)g; (void)M; (void)N; (void)K; (void)A; (void)lda; (void)B; (void)ldb; (void)it; (void)C; (void)ldc; (void)ot;
    return step();
}
int boat_cuda_weight_grads(int mma, int g, int64_t I, int64_t O, int64_t T, const void* const* X, const void* const* dY, int it, float* const* dW, float* const* db,
                           int acc) {
    (void)mma; (void)g; (void)I; (void)O; (void)T; (void)X; (void)dY; (void)it; (void)dW; (void)db; (void)acc;
    return step();
}
/* the packed calls have both pairs of products in one launch, the larger ones are told 13: by launches of their own */
int boat_cuda_linear_grads(int mma, int g, int64_t T, int64_t I, int64_t O, const void* const* X, const void* const* dY, const void* const* W, void* const* dX,
                           float* const* dW, float* const* db) {
    (void)mma; (void)g; (void)I; (void)O; (void)X; (void)dY; (void)W; (void)dX; (void)dW; (void)db;
    return T <= 8 ? step() : 13;
}
int boat_cuda_attn_fwd(int mma, int64_t u, int64_t S, int64_t hs, int c, float sc, const void* Q, const void* K, const void* V, int t, void* O, float* lse) {
    (void)mma; (void)u; (void)S; (void)hs; (void)c; (void)sc; (void)Q; (void)K; (void)V; (void)t; (void)O; (void)lse;
    return step();
}
int boat_cuda_attn_bwd(int mma, int64_t u, int64_t S, int64_t hs, int c, float sc, const void* Q, const void* K, const void* V, const void* O, const void* dO,
                       const float* lse, int t, void* dQ, void* dK, void* dV, void* scratch, size_t n) {
    (void)mma; (void)u; (void)S; (void)hs; (void)c; (void)sc; (void)Q; (void)K; (void)V; (void)O; (void)dO; (void)lse; (void)t; (void)dQ; (void)dK; (void)dV;
    (void)scratch; (void)n;
    return step();
}

void boat_optimizer_add_parameter(boat_optimizer_t* o, boat_tensor_t* p, boat_tensor_t* g) { (void)o; (void)p; (void)g; }

/* Forward, backward and update of a host layer on `device` tensors [B, S, H]; the number of calls made. */
static int run(int B, int S, int H, boat_device_t device, int fail) {
    calls = 0;
    fail_at = -1;
    boat_attention_config_t cfg = {(size_t)H, 2, 0, 0.0f, true, true, false, 10000.0f};
    boat_attention_t* a = boat_attention_create(&cfg);
    const int64_t shape[3] = {B, S, H};
    boat_tensor_t* x = boat_tensor_create(shape, 3, BOAT_DTYPE_FLOAT32, device);
    boat_tensor_t* g = boat_tensor_create(shape, 3, BOAT_DTYPE_FLOAT32, device);
    boat_tensor_t *out, *gq = NULL, *gk = NULL, *gv = NULL;
    calls = 0;
    fail_at = fail;
    out = boat_attention_forward(a, x, x, x, NULL);
    if (out && boat_attention_backward(a, g, &gq, &gk, &gv)) {
        boat_tensor_free(gq);
        boat_tensor_free(gk);
        boat_tensor_free(gv);
        boat_attention_update(a, 0.1f);
    }
    const int made = calls;
    fail_at = -1;
    if (out) boat_tensor_free(out);
    boat_attention_free(a);
    boat_tensor_free(x);
    boat_tensor_free(g);
    if (device_blocks || pinned_blocks) {
        printf("%d x %d x %d on device %d, call %d failing: %d device and %d pinned blocks left\n", B, S, H, (int)device, fail, device_blocks, pinned_blocks);
        exit(1);
    }
    if (open_sequences) {
        printf("%d x %d x %d on device %d, call %d failing: %d launch sequences left open\n", B, S, H, (int)device, fail, open_sequences);
        exit(1);
    }
    return made;
}

int main(void) {
    /* packed small tensors, separate larger ones, chunks of a large call, CUDA tensors with a host layer */
    const int sizes[4][4] = {{2, 4, 16, BOAT_DEVICE_CPU}, {2, 80, 128, BOAT_DEVICE_CPU}, {4, 2048, 64, BOAT_DEVICE_CPU}, {2, 30, 32, BOAT_DEVICE_CUDA}};
    for (int i = 0; i < 4; ++i) {
        const int* s = sizes[i];
        const int n = run(s[0], s[1], s[2], (boat_device_t)s[3], -1);
        for (int k = 0; k < n; ++k) run(s[0], s[1], s[2], (boat_device_t)s[3], k);
        printf("%d x %d x %d: %d calls\n", s[0], s[1], s[2], n);
    }
    printf("ok\n");
    return 0;
}
