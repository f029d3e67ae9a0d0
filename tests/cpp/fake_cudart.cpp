// The CUDA runtime calls of unit_build_failures.cu: memory is the host's, copies and memsets are done,
// kernels are counted and not run, and the allocation or the call that fake_reset names fails.
#include <cstdlib>
#include <cstring>

extern "C" {

int fake_allocations, fake_fail_allocation, fake_live;
int fake_calls, fake_fail_call, fake_failed;
int fake_launches_after_failure;
static int last_error, reads;

void fake_reset(int fail_allocation, int fail_call) {
    fake_allocations = fake_live = fake_calls = fake_failed = 0;
    fake_launches_after_failure = last_error = reads = 0;
    fake_fail_allocation = fail_allocation;
    fake_fail_call = fail_call;
}

int fake_allocate(void **p, size_t bytes) {
    if (fake_allocations++ == fake_fail_allocation) {
        fake_failed = 1;
        return last_error = 2;  // cudaErrorMemoryAllocation
    }
    *p = calloc(1, bytes ? bytes : 1);
    ++fake_live;
    return 0;
}
void fake_release(void *p) {
    if (p) --fake_live;
    free(p);
}
// One call that may fail, with cudaErrorInvalidValue.
static int call() {
    if (fake_calls++ != fake_fail_call) return 0;
    fake_failed = 1;
    return last_error = 1;
}
static int launch() {
    if (fake_failed) ++fake_launches_after_failure;
    return call();
}

int cudaMalloc(void **p, size_t bytes) { return fake_allocate(p, bytes); }
int cudaFree(void *p) {
    fake_release(p);
    return 0;
}
int cudaMemcpyAsync(void *dst, const void *, size_t bytes, int, void *) {
    // what the build reads back: units, slices, their size, shared stencils
    const long long value[4] = {20000, 700, 9000, 40000};
    memcpy(dst, &value[reads++ % 4], bytes);
    return call();
}
int cudaMemsetAsync(void *p, int v, size_t bytes, void *) {
    memset(p, v, bytes);
    return call();
}
int cudaStreamSynchronize(void *) { return call(); }
int cudaGetLastError() {
    const int e = last_error;
    last_error = 0;
    return e;
}
int cudaPeekAtLastError() { return last_error; }
int cudaGetDevice(int *d) { return *d = 0; }
int cudaSetDevice(int) { return 0; }
int cudaGetDeviceCount(int *n) {
    *n = 1;
    return 0;
}
int cudaDeviceGetAttribute(int *v, int attribute, int) {
    *v = attribute == 75 ? 10 : attribute == 76 ? 3 : 152;  // compute capability; SMs
    return 0;
}
int cudaFuncGetAttributes(void *attributes, const void *) {
    // sharedSizeBytes, constSizeBytes, localSizeBytes (size_t); maxThreadsPerBlock, numRegs,
    // ptxVersion, binaryVersion (int)
    memset(attributes, 0, 3 * sizeof(size_t));
    int *v = (int *)((char *)attributes + 3 * sizeof(size_t));
    v[0] = 1024;
    v[1] = 32;
    v[2] = v[3] = 103;
    return 0;
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t,
                                                           unsigned) {
    *n = 2;
    return 0;
}
int cudaLaunchKernelExC(const void *, const void *, void **) { return launch(); }
int __cudaLaunchKernel(...) { return launch(); }
const char *cudaGetErrorString(int) { return ""; }
unsigned __cudaPushCallConfiguration(...) { return 0; }
int __cudaPopCallConfiguration(...) { return 0; }
int __cudaGetKernel(void **kernel, const void *f) {
    *kernel = const_cast<void *>(f);
    return 0;
}
void **__cudaRegisterFatBinary(void *) {
    static void *handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(...) {}
void __cudaRegisterVar(...) {}
char __cudaInitModule(void **) { return 1; }
}
