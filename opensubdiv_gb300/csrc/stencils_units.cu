// EvalStencils over the unit layout of a table with one weight array (units.h).
//
// One persistent CTA of 16 warps per SM; a warp takes slices through its own queue (unit_ring.cuh)
// and evaluates one at a time, one unit per lane or pair or quad of lanes.
#include "common.cuh"
#include "unit_ring.cuh"

namespace gb300 {
namespace units {

struct Args {
    const float *src;
    int srcStride, length, shift;
    const int4 *slice;
    const char *blob;
    int numSlices;
    int *status;
    float *dst[1];
    int dstStride[1];
};

template <bool COLLECT>
__global__ void __launch_bounds__(kThreads, 1) k_stencils_units(const Args arg) {
    Args a = arg;
    launch_dependents();
    extern __shared__ __align__(128) char smem[];
    __shared__ Queue queue[kWarps];
    __shared__ int claimed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) claimed = 0;
    queue_init(queue);
    // this CTA's slices: blockIdx.x, + gridDim.x, ..., which spreads the slices of an irregular
    // region over the SMs; its warps claim them one by one
    const int count = (a.numSlices - 1 - (int)blockIdx.x) / (int)gridDim.x + 1;
    const int4 *own = a.slice + blockIdx.x;
    Queue &q = queue[warp];
    char *bytes = smem + (size_t)warp * kWarpBytes;
    const uint64_t pol_stream = l2_evict_first();
    // the next slice to queue: claimed, and its descriptor requested, a step ahead
    int4 d = make_int4(0, 0, 0, 0);
    bool more = true;
    auto claim = [&]() {
        int k = 0;
        if (lane == 0) k = atomicAdd(&claimed, 1);
        k = __shfl_sync(0xffffffffu, k, 0);
        more = k < count;
        if (more) d = __ldg(own + (size_t)k * gridDim.x);
    };
    claim();
    Feed f;
    Far far = warp_far(bytes, q.far);
    bool wait = true;  // for the kernel before; the table's slices are on their way meanwhile
    for (;; ++f.popped) {
        while (more && f.room(q, d.w)) {
            f.push(q, bytes, a.blob, d, lane, pol_stream);
            claim();
        }
        if (wait) wait_for_primary();
        behind_wait(a.src);
        wait = false;
        if (f.popped == f.pushed) return;
        const int s = f.popped % kAhead;
        if (!ring::wait(&q.full[s], (uint32_t)(f.popped / kAhead) & 1, a.status) ||
            !consume<COLLECT>(a, q, bytes, a.blob, far, s, lane, a.shift, pol_stream, a.status)) {
            drain(q, f, far, a.status);
            return;
        }
        __syncwarp();
    }
}

}  // namespace units

bool units_take(const float *src, int srcStride) {
    return ((uintptr_t)src & 15) == 0 && srcStride % 4 == 0;
}

bool units_collect(const float *dst, int dstStride) {
    return ((uintptr_t)dst & 15) != 0 || dstStride % 4 != 0;
}

int eval_stencils_units(const UnitTable &t, const float *src, float *dst, int dstStride,
                        int length, int srcStride, cudaStream_t s, const char *who) {
    if (t.numSlices == 0) return ok();
    if (!src || length <= 0 || srcStride < length)
        return fail(GB300_ERR_INVALID_ARGUMENT, "%s: bad source", who);
    if (dstStride < length)
        return fail(GB300_ERR_INVALID_ARGUMENT, "%s: output 0 stride / weights", who);
    if (!units_take(src, srcStride))
        return fail(GB300_ERR_INVALID_ARGUMENT, "%s: rows are not 16-byte aligned", who);
    auto kern = units_collect(dst, dstStride) ? units::k_stencils_units<true>
                                              : units::k_stencils_units<false>;
    static std::atomic<uint64_t> attr{0};
    int r = once_per_device(attr, [&] {
        const int st = check_cuda(cudaFuncSetAttribute(units::k_stencils_units<true>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       units::kSmemBytes),
                                  who);
        return st != GB300_OK ? st
                              : check_cuda(cudaFuncSetAttribute(
                                               units::k_stencils_units<false>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               units::kSmemBytes),
                                           who);
    });
    units::Args a{};
    if (r != GB300_OK || (r = status_word_address(&a.status)) != GB300_OK) return r;
    a.src = src;
    a.srcStride = srcStride;
    a.length = length;
    a.shift = units::unit_shift(length);
    a.slice = t.slice;
    a.blob = t.blob;
    a.numSlices = t.numSlices;
    a.dst[0] = dst;
    a.dstStride[0] = dstStride;
    launch_kernel(kern, min(a.numSlices, num_sms()), units::kThreads, units::kSmemBytes, s,
                  a);
    return check_launch(who);
}

}  // namespace gb300
