// Shared host/device helpers for libosd_gb300.so: status reporting, launch accounting and
// small PTX wrappers.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstdio>
#include <string>

#include "../../include/osd_gb300.h"

namespace gb300 {

// ---- status -------------------------------------------------------------------------------

// Records `msg` as the calling thread's last error and returns `code`.
int fail(int code, const char *fmt, ...);
// Clears the calling thread's last error and returns GB300_OK.
int ok();
// Maps a CUDA error to a status (recording its message); GB300_OK for cudaSuccess.
int check_cuda(cudaError_t e, const char *what);
// Checks the launch that was just queued.
int check_launch(const char *what);

extern std::atomic<uint64_t> g_launches;
inline void count_launch(uint64_t n = 1) { g_launches.fetch_add(n, std::memory_order_relaxed); }

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

// Number of SMs of the current device (cached per device).
int num_sms();

// Stream-ordered scratch from a memory pool the library keeps per device: allocations and
// frees are ordered on `s` like cudaMallocAsync / cudaFreeAsync, but up to kScratchRetainBytes
// of freed memory stay mapped in the pool between calls (the device's default pool returns
// freed memory at every synchronisation, so a per-call scratch paid a fresh mapping, ~0.1 ms,
// on every call).
constexpr size_t kScratchRetainBytes = size_t(512) << 20;
int scratch_alloc(void **p, size_t bytes, cudaStream_t s, const char *who);
void scratch_free(void *p, cudaStream_t s);

// Device address of the library's status word on the current device (the word
// GB300GetDeviceStatus reads and clears; staged kernels record an expired bounded wait there).
int status_word_address(int **out);

// Whether the `bytes` from p on lie in the one allocation that p points into: they can be read then,
// whatever they hold.  False where the driver does not know the pointer.  About 0.1 us.
bool inside_allocation(const void *p, size_t bytes);

// Launches `kern` as the programmatic dependent of the kernel queued before it: it may be started
// while that one still runs (at once if it called launch_dependents, else when it ends), and calls
// wait_for_primary before it touches anything that work queued earlier reads or writes.  What it may
// read before is a table's own layout, whose builder synchronised before it returned the table.
// Anything else is written during the lifetime of such a kernel, as far as the memory model goes,
// so it is read with coherent loads, which the wait orders: the ones below, or C++ loads through
// pointers that are not __restrict__.  The non-coherent path (ld.global.nc, __ldg) is for the
// tables' own arrays.
// A captured launch keeps its plain dependency on whatever node precedes it.
template <class K, class... A>
void launch_kernel(K kern, dim3 grid, int threads, size_t smem, cudaStream_t s, const A &... arg) {
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) {
        cudaGetLastError();
        cs = cudaStreamCaptureStatusActive;
    }
    c.attrs = &attr;
    c.numAttrs = cs == cudaStreamCaptureStatusNone ? 1 : 0;
    cudaLaunchKernelEx(&c, kern, arg...);  // the caller checks the launch
    count_launch();
}

// Runs `fn` (returning a status) once per device for one call site: `done` is that call site's
// bitmask of devices it already succeeded on (devices >= 64 run it every time).
template <class F>
int once_per_device(std::atomic<uint64_t> &done, F fn) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return fn();
    const uint64_t bit = 1ull << dev;
    if (done.load(std::memory_order_acquire) & bit) return GB300_OK;
    const int st = fn();
    if (st == GB300_OK) done.fetch_or(bit, std::memory_order_release);
    return st;
}

// ---- device helpers -----------------------------------------------------------------------

// Programmatic dependent launch (launch_kernel).  launch_dependents lets the next kernel be started
// as soon as every CTA of this one runs; it is then resident, and waits in wait_for_primary until
// this one is done and its writes are visible.  A kernel that calls it before it waits itself lets
// the chain behind it start as well.
__device__ __forceinline__ void launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_for_primary() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// The pointer as it stands behind the wait: a load through it depends on this, and so on the wait.
template <class T>
__device__ __forceinline__ void behind_wait(T *&p) {
    asm volatile("" : "+l"(p) : : "memory");
}

// L2 eviction policies (createpolicy) for the cache-hinted loads below.
__device__ __forceinline__ uint64_t l2_evict_first() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_evict_last() {
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}

// Streaming (read-once) 32-bit loads for the stencil table: no L1 allocation and an
// evict-first L2 policy, so the table stream does not push the source rows out of L2.  Non-coherent:
// for a table's own arrays, or in kernels that are launched behind all earlier work.
__device__ __forceinline__ int ld_stream(const int *p, uint64_t pol) {
    int v;
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.b32 %0, [%1], %2;"
                 : "=r"(v) : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ float ld_stream(const float *p, uint64_t pol) {
    float v;
    asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;"
                 : "=f"(v) : "l"(p), "l"(pol));
    return v;
}

// Coherent loads of the caller's data, which a kernel queued before may write.  Two forms keep them
// behind wait_for_primary: the volatile ones keep their order among themselves and with the wait;
// the others the compiler may move, as far as their address allows, which is to come from
// behind_wait.  (EvalPatches, 4 M points: lanes with volatile rows and indices 374 -> 396 us, their
// loads no longer overlapping as the compiler had them.  Elsewhere the pointer's registers cost more:
// Loop rows through behind_wait 255 -> 261 us, three outputs of 4-wide stencil rows 18.7 -> 20.5.)
//
// Source rows: kept in L1, evict-last in L2 (the control points are re-read by every stencil that
// touches them).
__device__ __forceinline__ float ld_src(const float *p, uint64_t pol) {
    float v;
    asm volatile("ld.global.L1::evict_last.L2::cache_hint.f32 %0, [%1], %2;"
                 : "=f"(v)
                 : "l"(p), "l"(pol));
    return v;
}
__device__ __forceinline__ float4 ld_src4(const float *p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ void ld_src8(const float *p, float (&x)[8]) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]),
                   "=f"(x[6]), "=f"(x[7])
                 : "l"(p));
}
__device__ __forceinline__ float4 ld_row4(const float *p, uint64_t pol) {
    float4 v;
    asm volatile("ld.global.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p), "l"(pol)
                 : "memory");
    return v;
}
// Movable: rows in a unit or a batched slice, elements and indices of patches read by lanes.
__device__ __forceinline__ void ld_point8(const float *p, float (&x)[8]) {
    asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]),
          "=f"(x[7])
        : "l"(p));
}
__device__ __forceinline__ float4 ld_point4(const float *p) {
    float4 v;
    asm("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_point(const float *p, uint64_t pol) {
    float v;
    asm("ld.global.L1::evict_last.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
    return v;
}
template <bool MOVABLE>
__device__ __forceinline__ int ld_index(const int *p, uint64_t pol) {
    int v;
    if constexpr (MOVABLE)
        asm("ld.global.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
    else
        asm volatile("ld.global.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
    return v;
}
template <bool MOVABLE>
__device__ __forceinline__ int4 ld_index4(const int *p, uint64_t pol) {
    int4 v;
    if constexpr (MOVABLE)
        asm("ld.global.L2::cache_hint.v4.b32 {%0, %1, %2, %3}, [%4], %5;"
            : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
            : "l"(p), "l"(pol));
    else
        asm volatile("ld.global.L2::cache_hint.v4.b32 {%0, %1, %2, %3}, [%4], %5;"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "l"(p), "l"(pol));
    return v;
}
// Params of patches, and queries (read once: no L1 allocation).
__device__ __forceinline__ int ld_param(const int *p, uint64_t pol) {
    int v;
    asm volatile("ld.global.L2::cache_hint.b32 %0, [%1], %2;"
                 : "=r"(v)
                 : "l"(p), "l"(pol)
                 : "memory");
    return v;
}
__device__ __forceinline__ int ld_query(const int *p, uint64_t pol) {
    int v;
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.b32 %0, [%1], %2;"
                 : "=r"(v)
                 : "l"(p), "l"(pol)
                 : "memory");
    return v;
}

// Streaming stores for outputs (written once, not re-read by this launch).
__device__ __forceinline__ void st_stream(float *p, float v) {
    asm volatile("st.global.cs.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

}  // namespace gb300
