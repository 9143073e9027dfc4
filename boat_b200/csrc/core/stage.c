/* stage.c - see stage.h. */
#include "stage.h"
#include <stdlib.h>
#include <string.h>
#include <strings.h>

int boat_storage_of(boat_dtype_t dt) { return dt == BOAT_DTYPE_BFLOAT16 ? BOAT_CUDA_BF16 : BOAT_CUDA_F32; }
size_t boat_storage_size(int type) { return type == BOAT_CUDA_BF16 ? 2 : 4; }
bool boat_dtype_supported(boat_dtype_t dt) { return dt == BOAT_DTYPE_FLOAT32 || dt == BOAT_DTYPE_BFLOAT16; }

bool boat_is_device_operand(const boat_tensor_t* t, int type, size_t n) {
    return t->device == BOAT_DEVICE_CUDA && boat_dtype_supported(t->dtype) && boat_storage_of(t->dtype) == type && t->nelements == n;
}

void* boat_dev_alloc(size_t bytes) {
    void* p = NULL;
    if (boat_report("device allocation", boat_cuda_malloc(&p, bytes)) != 0) return NULL;
    return p;
}

void boat_dev_free(void* p) {
    if (p) boat_report("device free", boat_cuda_free(p));
}

void* boat_stage_in(const boat_tensor_t* t, int type, bool* owned) {
    int have = boat_storage_of(t->dtype);
    size_t n = t->nelements;
    *owned = false;
    if (t->device == BOAT_DEVICE_CUDA && have == type) return t->data;
    *owned = true;
    void* raw = t->data;
    void* tmp = NULL;
    if (t->device != BOAT_DEVICE_CUDA) {
        tmp = boat_dev_alloc(n * boat_storage_size(have));
        if (!tmp) return NULL;
        if (boat_report("upload", boat_cuda_memcpy_h2d(tmp, t->data, n * boat_storage_size(have))) != 0) {
            boat_dev_free(tmp);
            return NULL;
        }
        if (have == type) return tmp;
        raw = tmp;
    }
    void* out = boat_dev_alloc(n * boat_storage_size(type));
    if (out && boat_report("cast", boat_cuda_cast(out, type, raw, have, (int64_t)n)) != 0) {
        boat_dev_free(out);
        out = NULL;
    }
    boat_dev_free(tmp);
    return out;
}

boat_tensor_t* boat_emit_out(const int64_t* shape, size_t ndim, const boat_tensor_t* like, void* src, int type) {
    boat_tensor_t* out = boat_tensor_create_uninit(shape, ndim, like->dtype, like->device);
    if (!out) return NULL;
    int want = boat_storage_of(like->dtype);
    size_t n = out->nelements;
    int rc;
    if (like->device == BOAT_DEVICE_CUDA) {
        rc = boat_cuda_cast(out->data, want, src, type, (int64_t)n);
    } else if (want == type) {
        rc = boat_cuda_memcpy_d2h(out->data, src, n * boat_storage_size(type));
    } else {
        void* tmp = boat_dev_alloc(n * boat_storage_size(want));
        rc = tmp ? boat_cuda_cast(tmp, want, src, type, (int64_t)n) : 1;
        if (rc == 0) rc = boat_cuda_memcpy_d2h(out->data, tmp, n * boat_storage_size(want));
        boat_dev_free(tmp);
    }
    if (boat_report("result transfer", rc) != 0) {
        boat_tensor_free(out);
        return NULL;
    }
    return out;
}

boat_tensor_t* boat_emit_out_take(const int64_t* shape, size_t ndim, const boat_tensor_t* like, void** src, int type) {
    if (like->device == BOAT_DEVICE_CUDA && boat_storage_of(like->dtype) == type && *src) {
        boat_tensor_t* out = boat_tensor_adopt_device(shape, ndim, like->dtype, *src);
        if (out) *src = NULL;
        return out;
    }
    return boat_emit_out(shape, ndim, like, *src, type);
}

int boat_default_mma(boat_dtype_t dt) {
    if (dt == BOAT_DTYPE_BFLOAT16) return BOAT_MMA_BF16;
    const char* e = getenv("BOAT_MMA");
    if (e && !strcasecmp(e, "tf32")) return BOAT_MMA_TF32;
    return BOAT_MMA_FP32;
}

bool boat_bundle_send(boat_bundle_t* b, const boat_tensor_t* const* tensors, int n) {
    memset(b, 0, sizeof *b);
    size_t total = 0;
    for (int i = 0; i < n; ++i) {
        const boat_tensor_t* t = tensors[i];
        if (!t || t->device == BOAT_DEVICE_CUDA || t->nbytes >= BOAT_BUNDLE_LIMIT || b->count == BOAT_BUNDLE_MAX) continue;
        bool seen = false;
        for (int j = 0; j < b->count; ++j) seen = seen || b->tensor[j] == t;
        if (seen) continue;
        b->tensor[b->count] = t;
        b->offset[b->count++] = total;
        total += boat_align256(t->nbytes);
    }
    if (b->count == 0) return true;
    b->host = boat_cuda_host_alloc(total);
    b->dev = b->host ? boat_dev_alloc(total) : NULL;
    if (!b->dev) {                                       /* no image: the tensors are sent one by one */
        if (b->host) boat_cuda_host_free(b->host);
        memset(b, 0, sizeof *b);
        return true;
    }
    for (int i = 0; i < b->count; ++i) memcpy((char*)b->host + b->offset[i], b->tensor[i]->data, b->tensor[i]->nbytes);
    b->sent = true;
    return boat_report("upload", boat_cuda_stage_copy(b->dev, b->host, total, 0)) == 0;
}

void* boat_bundle_find(const boat_bundle_t* b, const boat_tensor_t* t) {
    for (int i = 0; i < b->count; ++i)
        if (b->tensor[i] == t) return (char*)b->dev + b->offset[i];
    return NULL;
}

void boat_bundle_settle(boat_bundle_t* b, bool synced) {
    if (b->sent && !synced) boat_report("upload", boat_cuda_sync());
    b->sent = false;
    if (b->host) boat_cuda_host_free(b->host);
    b->host = NULL;
}

void* boat_landing_alloc(size_t bytes, bool direct, bool* on_host) {
    void* p = direct && bytes <= BOAT_DIRECT_LIMIT ? boat_cuda_host_alloc(bytes) : NULL;
    *on_host = p != NULL;
    return p ? p : boat_dev_alloc(bytes);
}

void boat_landing_free(void* block, bool on_host, bool synced) {
    if (on_host && !synced) boat_report("result", boat_cuda_sync());
    if (on_host) boat_cuda_host_free(block);
    else boat_dev_free(block);
}

int boat_scatter_down(const void* dev, bool on_host, size_t total, void* const* host, const size_t* offset, const size_t* bytes, int n) {
    if (on_host) {
        const int done = boat_cuda_sync();
        for (int i = 0; i < n && done == 0; ++i) memcpy(host[i], (const char*)dev + offset[i], bytes[i]);
        return done;
    }
    char* image = total < BOAT_IMAGE_LIMIT ? (char*)boat_cuda_host_alloc(total) : NULL;
    int rc = 0;
    if (image) {
        /* the offsets are multiples of 256 bytes: whole 16-byte units, in the block as in the image */
        rc = boat_cuda_stage_copy(image, dev, total, 1);
        const int done = boat_cuda_sync();
        if (rc == 0) rc = done;
        for (int i = 0; i < n && rc == 0; ++i) memcpy(host[i], image + offset[i], bytes[i]);
        boat_cuda_host_free(image);
        return rc;
    }
    for (int i = 0; i < n && rc == 0; ++i) rc = boat_cuda_download_async(host[i], (const char*)dev + offset[i], bytes[i]);
    const int done = boat_cuda_sync();
    return rc ? rc : done;
}
