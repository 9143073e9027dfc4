// Whether csrc/cuda/comm.cu and selftest.cu tell the launch order (boatcu::ordinary_launch_next) of what they put on the library
// stream without it: NCCL's collectives and a plainly launched kernel.  Linked with those two files as they are; the rest
// of the library is played here, and so is NCCL: the file once more as a library of its own (PLAYED_NCCL).
#include <dlfcn.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <cuda_runtime.h>
#include <nccl.h>
#include <boat_cuda.h>

#ifdef PLAYED_NCCL
extern "C" {
int boat_fake_nccl = 1;
void (*played_on_reduce)(void);
static int comm;
ncclResult_t ncclGetUniqueId(ncclUniqueId*) { return ncclSuccess; }
ncclResult_t ncclCommInitRankConfig(ncclComm_t* c, int, ncclUniqueId, int, ncclConfig_t*) { return *c = (ncclComm_t)&comm, ncclSuccess; }
ncclResult_t ncclCommGetAsyncError(ncclComm_t, ncclResult_t* r) { return *r = ncclSuccess; }
ncclResult_t ncclCommAbort(ncclComm_t) { return ncclSuccess; }
ncclResult_t ncclCommFinalize(ncclComm_t) { return ncclSuccess; }
ncclResult_t ncclCommDestroy(ncclComm_t) { return ncclSuccess; }
ncclResult_t ncclAllReduce(const void*, void*, size_t, ncclDataType_t, ncclRedOp_t, ncclComm_t, cudaStream_t) { return played_on_reduce(), ncclSuccess; }
ncclResult_t ncclGroupStart() { return ncclSuccess; }
ncclResult_t ncclGroupEnd() { return ncclSuccess; }
const char* ncclGetErrorString(ncclResult_t) { return ""; }
}
#else
static int told, reduces, unannounced;

namespace boatcu {
int set_error(int status, const char*, ...) { return status; }
cudaStream_t stream() { return 0; }
void count_launch(int) {}
int ensure_init() { return 0; }
unsigned int* kernel_status_ptr() { return nullptr; }
void ordinary_launch_next() { ++told; }
}  // namespace boatcu

extern "C" {
const char* boat_cuda_last_error(void) { return ""; }
int boat_cuda_malloc(void** p, size_t n) { return (*p = malloc(n)) ? 0 : 1; }
int boat_cuda_free(void* p) { return free(p), 0; }
int boat_cuda_memcpy_h2d(void* d, const void* s, size_t n) { return memcpy(d, s, n), 0; }
int boat_cuda_memcpy_d2h(void* d, const void* s, size_t n) { return memcpy(d, s, n), 0; }
int boat_cuda_sync(void) { return 0; }

}

static void on_reduce(void) {
    ++reduces;
    if (told == 0) ++unannounced;
    told = 0;
}

int main() {
    ncclUniqueId id;
    void* nccl = dlopen(getenv("BOAT_NCCL_LIB"), RTLD_NOW | RTLD_GLOBAL);
    if (!nccl) return printf("%s\n", dlerror()), 1;
    *(void (**)(void))dlsym(nccl, "played_on_reduce") = on_reduce;
    float bucket[4] = {1, 2, 3, 4};
    if (boat_cuda_comm_unique_id(&id) || boat_cuda_comm_init(0, 2, &id)) return printf("no communicator\n"), 1;
    // the agreement on the length and the sum, then sums alone
    for (int i = 0; i < 3; ++i)
        if (boat_cuda_allreduce_sum_f32(bucket, 4)) return printf("sum %d failed\n", i), 1;
    if (reduces != 4 || unannounced) return printf("%d of %d collectives unannounced\n", unannounced, reduces), 1;
    told = 0;
    boat_cuda_selftest_wait_timeout(1000);              // without a GPU the launch itself fails
    if (!told) return printf("the self test's kernel is unannounced\n"), 1;
    printf("ok\n");
    return 0;
}
#endif
