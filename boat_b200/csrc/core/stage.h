/* stage.h - moving tensors between the caller's memory space/dtype and device buffers in the
 * storage type a kernel wants.  Shared by the layers around attention (LayerNorm, dense). */
#ifndef BOAT_STAGE_H
#define BOAT_STAGE_H

#include "boat_internal.h"

int    boat_storage_of(boat_dtype_t dt);                 /* BOAT_CUDA_F32 / BOAT_CUDA_BF16 */
size_t boat_storage_size(int type);
bool   boat_dtype_supported(boat_dtype_t dt);            /* FLOAT32 or BFLOAT16 */
/* Whether `t` is `n` elements of storage `type` in HBM: an operand that a kernel reads element by element beside
 * another tensor of that size. */
bool   boat_is_device_operand(const boat_tensor_t* t, int type, size_t n);
void*  boat_dev_alloc(size_t bytes);                     /* NULL + message on failure */
void   boat_dev_free(void* p);
/* Device buffer with tensor `t` in storage `type`; *owned: caller must boat_dev_free it. */
void*  boat_stage_in(const boat_tensor_t* t, int type, bool* owned);
/* New tensor shaped `shape`, with dtype/device of `like`, filled from device buffer `src`. */
boat_tensor_t* boat_emit_out(const int64_t* shape, size_t ndim, const boat_tensor_t* like, void* src, int type);
/* Like boat_emit_out for a buffer from boat_dev_alloc that the caller is done with: a CUDA result
 * of the same storage type becomes a tensor around *src itself (no copy) and *src is set to NULL,
 * so that the caller's boat_dev_free(*src) is a no-op; every other case copies as boat_emit_out. */
boat_tensor_t* boat_emit_out_take(const int64_t* shape, size_t ndim, const boat_tensor_t* like, void** src, int type);

/* Host tensors on their way to the GPU for one call.  Every copy has a fixed cost of some 10 us when the
 * host waits for it, which is all that small tensors cost; so those under BOAT_BUNDLE_LIMIT bytes are
 * packed into one page-locked image and go up as one copy, larger ones are sent one by one, and
 * nothing is waited for until the call ends. */
#define BOAT_BUNDLE_LIMIT ((size_t)64 * 1024)          /* from here on tensors are page-locked: memory.c */
#define BOAT_IMAGE_LIMIT ((size_t)256 * 1024)          /* results under this total come down as one copy */
enum { BOAT_BUNDLE_MAX = 16 };
typedef struct {
    void *host, *dev;                                    /* the image and its copy in HBM */
    const boat_tensor_t* tensor[BOAT_BUNDLE_MAX];
    size_t offset[BOAT_BUNDLE_MAX];
    int count;
    bool sent;                                           /* uploads of this call may still be reading host memory */
} boat_bundle_t;
/* Sends the small host tensors among the n given ones (NULL entries are skipped).  false on failure. */
bool   boat_bundle_send(boat_bundle_t* b, const boat_tensor_t* const* tensors, int n);
/* Where tensor `t` lies in HBM, or NULL when it was not packed. */
void*  boat_bundle_find(const boat_bundle_t* b, const boat_tensor_t* t);
/* Ends the call: waits for the uploads unless `synced` (the host has waited for a later copy), and
 * gives the image back.  The HBM copy is the caller's to free (boat_dev_free(b->dev)). */
void   boat_bundle_settle(boat_bundle_t* b, bool synced);
/* The block that a call's results for the host are produced in.  `direct`: the kernels that write it use plain
 * stores and none reads it back; then a small block is page-locked host memory, which they write over
 * the bus, and no copy follows.  *on_host tells which it is; freed with boat_landing_free. */
#define BOAT_DIRECT_LIMIT ((size_t)64 * 1024)
void*  boat_landing_alloc(size_t bytes, bool direct, bool* on_host);
void   boat_landing_free(void* block, bool on_host, bool synced);      /* synced: as for boat_bundle_settle */
/* Copies n pieces of one device block (at `offset`, `bytes` long) to host memory and waits: small totals as
 * one copy through a page-locked image, no copy at all where the block is such an image (`on_host`). */
int    boat_scatter_down(const void* dev, bool on_host, size_t total, void* const* host, const size_t* offset, const size_t* bytes, int n);
static inline size_t boat_align256(size_t n) { return (n + 255) & ~(size_t)255; }

/* Arithmetic for FP32/BF16 inputs outside the attention layer: BF16 storage -> BF16 tensor
 * cores; FP32 storage -> env BOAT_MMA (tf32 | fp32), default exact FP32. */
int    boat_default_mma(boat_dtype_t dt);

#endif
