// GB300PatchTableEval over a faked CUDA runtime: which source rows its copy of a Loop table's rows
// may read.  A point needs the rows of its own patch; the copy reads every row that the table names,
// so it is made only where the allocation that the source lies in holds them all.  Prints "ok".
#include "../../opensubdiv_gb300/csrc/allocation.cu"
#include "../../opensubdiv_gb300/csrc/objects.cu"

#include <cstdlib>
#include <cstring>

static uintptr_t g_start;  // the allocation that the driver reports
static size_t g_size;
static bool g_known;
static int g_copied, g_evaluated;
static const float *g_source;

#ifndef __CUDA_ARCH__  // the host's runtime
static CUresult fake_attributes(unsigned n, CUpointer_attribute *which, void **out, CUdeviceptr) {
    if (!g_known) return CUDA_ERROR_INVALID_VALUE;
    for (unsigned k = 0; k < n; ++k) {
        if (which[k] == CU_POINTER_ATTRIBUTE_RANGE_START_ADDR) *(CUdeviceptr *)out[k] = g_start;
        if (which[k] == CU_POINTER_ATTRIBUTE_RANGE_SIZE) *(size_t *)out[k] = g_size;
    }
    return CUDA_SUCCESS;
}

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    *p = calloc(1, n);
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char *name, void **fn, unsigned,
                                             unsigned long long,
                                             cudaDriverEntryPointQueryResult *found) {
    const bool known = !strcmp(name, "cuPointerGetAttributes");
    *fn = known ? (void *)fake_attributes : nullptr;
    *found = known ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) {
    static void *handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
char __cudaInitModule(void **) { return 1; }
}
#endif

namespace gb300 {
std::atomic<uint64_t> g_launches{0};
int fail(int code, const char *, ...) { return code; }
int ok() { return GB300_OK; }
int check_cuda(cudaError_t e, const char *) { return e == cudaSuccess ? GB300_OK : GB300_ERR_CUDA; }
int check_launch(const char *) { return GB300_OK; }
int scratch_alloc(void **p, size_t n, cudaStream_t, const char *) {
    return (*p = calloc(1, n)) ? GB300_OK : GB300_ERR_OUT_OF_MEMORY;
}
void scratch_free(void *p, cudaStream_t) { free(p); }
int build_sell(int, const int *, const int *, const int *, const float *const *, cudaStream_t,
               SellTable &, void **, const char *) { return GB300_OK; }
int build_units(int, const int *, const int *, const int *, const float *, cudaStream_t,
                UnitTable &, void **, const char *) { return GB300_OK; }
bool units_take(const float *, int) { return false; }
bool units_collect(const float *, int) { return false; }
int eval_stencils(const float *, float *const *, const int *, const float *const *, int, int,
                  const int *, const int *, const int *, int, int, cudaStream_t,
                  const char *) { return GB300_OK; }
int eval_stencils_sell(const SellTable &, const float *, float *const *, const int *,
                       const float *const *, int, int, cudaStream_t,
                       const char *) { return GB300_OK; }
UnitRows units_rows(const UnitTable &, const float *, int, int, long long, bool) {
    return kUnitNone;
}
int eval_stencils_units(const UnitTable &, UnitRows, const float *, float *, int, int, int,
                        cudaStream_t, const char *) { return GB300_OK; }
int find_patches(const PatchMapDevice &, int, const int *, const float *, const float *, void *,
                 cudaStream_t) { return GB300_OK; }
int tess_factors(const void *, int, const int *, const void *, int, const float *, int,
                 GB300PatchTessOptions const *, float *, float *, float *, float *,
                 cudaStream_t) { return GB300_OK; }
GB300StencilTable *tess_stencils(const void *, const int *, const void *, int, const void *, int,
                                 int64_t, const int *, const int *, const int *, const float *, int,
                                 int, cudaStream_t, const char *) { return nullptr; }
int build_patch_map(int, const int *, int, const int *, int, PatchMapHost &) { return GB300_OK; }
int gather_patch_rows(const float *, int, const int *, int, float *, cudaStream_t) {
    ++g_copied;
    return GB300_OK;
}
int batch::launch_pad_one(const PadJob &, cudaStream_t) {
    ++g_copied;
    return GB300_OK;
}
int eval_patches(const float *src, float *const *, const int *, int, int, int, const void *,
                 const void *, const int *, const void *, cudaStream_t, const char *, int, int,
                 int) {
    ++g_evaluated;
    g_source = src;
    return GB300_OK;
}
}  // namespace gb300

int main() {
    // two Loop patches of 12 points: the second one names rows up to rows - 1, few (a copy of the rows)
    // or many (with derivatives a row per index)
    const int arrays[6] = {5, 5, 2, 0, 12, 0};
    int indices[24], params[6] = {};
    static float buffer[4 * 40000];
    const int n = 1 << 18;
    for (int stride = 3; stride <= 4; ++stride)
        for (int more = 0; more < 4; ++more)  // P alone, and with derivatives; few rows, and many
            for (int offset = 0; offset < 2; ++offset)
                for (int negative = 0; negative < 2; ++negative) {
                    const int rows = more < 2 ? 1000 : 40000;
                    for (int j = 0; j < 24; ++j) indices[j] = j < 12 ? j : rows - 1 - (j - 12);
                    if (negative) indices[23] = -1;
                    GB300PatchTable *t =
                        GB300PatchTableCreate(1, arrays, 24, indices, 2, params, 1, nullptr);
                    if (!t) return printf("no table\n"), 1;
                    const size_t need = ((rows - 1) * (size_t)stride + 3 + offset) * 4;
                    for (int state = 0; state < 4; ++state) {
                        // the whole buffer, a float less, one patch's rows, an unknown pointer
                        g_known = state < 3;
                        g_start = (uintptr_t)buffer;
                        g_size = state == 0 ? need : state == 1 ? need - 4 : 12 * stride * 4;
                        g_copied = g_evaluated = 0;
                        float *du = more & 1 ? buffer : nullptr;
                        const int st = GB300PatchTableEval(t, buffer + offset, buffer, du, nullptr,
                                                           nullptr, nullptr, nullptr, 3, stride, 3,
                                                           3, 3, 3, 3, 3, n, buffer, nullptr);
                        const int want = state == 0 && !negative;
                        if (st != GB300_OK || g_evaluated != 1 || g_copied != want ||
                            (g_source == buffer + offset) == (want == 1))
                            return printf("rows %d stride %d more %d offset %d negative %d state %d: "
                                          "status %d, %d copies\n", rows, stride, more, offset, negative,
                                          state, st, g_copied), 1;
                    }
                    GB300PatchTableDestroy(t);
                }
    printf("ok\n");
    return 0;
}
