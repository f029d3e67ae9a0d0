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

// Units write a row's quads by lanes whose other rows lie far apart, so what decides is how they fill the
// 32-byte sectors.  Rows of quads without gaps fill them (8-wide 2.9 M Loop stencils 73 -> 56 us), but
// a tail takes a store per element (3 floats in rows of 4, 2.9 M Loop stencils: 53 us sliced, 69 by
// unit rows), and a sector of which a part is written leaves the L2 as such once the rows outgrow it
// (8.6 M stencils of quads 191 and 245 us, 8.4 M irregular ones 186 and 308).  Tables whose
// slices are mostly uniform (`regular`) are written collected there (167 us of the 191); irregular ones
// wait for their weights as well, and stay with the sliced layout.  Rows of 13 and more floats take the
// sliced layout two passes and more (16-wide, 1.9 M irregular stencils: 98 us, 58 by unit rows).
// us, sliced / by row / collected, "4/8" 4 floats in rows of 8:
//   regular    3/4: 0.3 M 8.4/9.5/10.3, 0.5 M 14.4/13.5/12.6, 4.3 M 89/82/61
//              4/8: 0.9 M 23/16/20, 4.3 M (136 MB) 112/111/118, 8.6 M 224/237/245
//              7/8: 0.3 M 12.2/10.9/12.4, 0.9 M 35/29/25, 4.3 M 151/188/129, 8.6 M 302/406/259
//              8/12: 8.6 M 335/289/304   11/12: 0.9 M 42/32/37, 8.6 M 399/423/357
//   irregular  4/4: 0.5 M 12.7/13.2/17.2, 1.0 M 23/19/25, 4.1 M 83/78/86, 8.0 M 149/158/165
//              5/8: 1.0 M 34/24/29, 1.9 M (62 MB) 54/52/58, 4.1 M 121/140/136
//              7/8: 0.5 M 18.5/21.8/22.1, 1.9 M 58/69/61   8/12: 1.0 M 33/23/32, 8.0 M 297/306/319
//              11/12: 0.3 M 16.5/13.5/18.0, 1.0 M 51/37/44, 1.9 M (93 MB) 80/85/89
//              15/16: 1.9 M (124 MB) 114/105/107, 2.9 M 156/162/147   16/20: 8.0 M 477/435/459
// Rows that are not 16-byte aligned are collected, which costs about a third more instructions: a single
// call takes the layout for them from kUnitAnyRow on, and for regular tables only (5-wide rows: level 3
// of quads, 1.2 M stencils 41.5 and 45.2 us, 2.1 M 59.7 and 71.8; level 4 of triangles split at random,
// 1.2 M 50.1 and 39.7).  In a batch the other jobs hide what an irregular table waits for (3 such
// tables of 1.9 M stencils, 3, 5 and 11 floats: 118, 155 and 229 us, 139, 193 and 230 sliced; but 3
// floats of 6.4 M, 230 MB, 463 and 420; 259 k Loop ones 30 and 27; scenes
// of 8 to 64 meshes 0-4% slower for their part).
UnitRows units_rows(const UnitTable &t, const float *dst, int stride, int length, long long bytes,
                    bool batch) {
    const long long mb = bytes >> 20;
    const int n = t.numStencils, tail = length % 4, gap = stride - length;
    if (n == 0 || (!batch && n < kUnitCall)) return kUnitNone;
    if (units_collect(dst, stride)) {
        if (t.regular) return batch || n >= kUnitAnyRow ? kUnitCollected : kUnitNone;
        return batch && (length > 3 || mb <= 192) ? kUnitCollected : kUnitNone;
    }
    const bool sectors = length % 8 == 0 && stride % 8 == 0 && ((uintptr_t)dst & 31) == 0;
    if (length > 12)
        return length >= 16 || tail <= 1 || t.regular || mb <= 128 ? kUnitByRow : kUnitNone;
    if (length < 4)
        return t.regular && (batch || n >= 2 * kUnitCall) && (gap < 4 || mb <= 64) ? kUnitCollected
                                                                                   : kUnitNone;
    if (length == 4) {
        if (t.regular) return gap == 0 || mb <= 128 ? kUnitByRow : kUnitNone;
        return (batch || n >= 15 << 16) && mb <= (gap ? 64 : batch ? 192 : 96) ? kUnitByRow : kUnitNone;
    }
    if (gap == 0 || sectors) return kUnitByRow;
    if (t.regular)
        return tail && gap < 4 && (mb > 64 || (batch && tail > 1)) ? kUnitCollected
               : mb <= 64 || length >= 8                           ? kUnitByRow
                                                                   : kUnitNone;
    return (tail <= 1 || length > 8) && mb <= (tail ? 64 : 128) ? kUnitByRow : kUnitNone;
}

int eval_stencils_units(const UnitTable &t, UnitRows rows, const float *src, float *dst, int dstStride,
                        int length, int srcStride, cudaStream_t s, const char *who) {
    if (t.numSlices == 0) return ok();
    if (!src || length <= 0 || srcStride < length)
        return fail(GB300_ERR_INVALID_ARGUMENT, "%s: bad source", who);
    if (dstStride < length)
        return fail(GB300_ERR_INVALID_ARGUMENT, "%s: output 0 stride / weights", who);
    if (!units_take(src, srcStride))
        return fail(GB300_ERR_INVALID_ARGUMENT, "%s: rows are not 16-byte aligned", who);
    if (rows == kUnitNone || (rows == kUnitByRow && units_collect(dst, dstStride)))
        return fail(GB300_ERR_INVALID_ARGUMENT, "%s: output rows are not 16-byte aligned", who);
    auto kern = rows == kUnitCollected ? units::k_stencils_units<true>
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
