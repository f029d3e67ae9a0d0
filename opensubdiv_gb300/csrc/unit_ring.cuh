// The shared-memory queue through which a warp takes slices of the unit layout (units.h), for
// the table kernel (stencils_units.cu) and the batched kernel (stencils_batch.cu).
//
// Every warp feeds itself: while it evaluates one slice, the staged parts of the next ones are on
// their way into its own byte ring (slices differ in length), one bulk copy each, and the weights
// of a slice that is not uniform on their way into L2.  One producer warp per CTA, handing slices
// over through barriers, reached about 2 slices per microsecond, half of what 8 warps consume.
#pragma once

#include "stage_ring.cuh"
#include "unit_eval.cuh"
#include "units.h"

namespace gb300 {
namespace units {

constexpr int kWarps = 16;  // one CTA per SM: 128 registers a thread
constexpr int kThreads = kWarps * 32;
constexpr int kAhead = 2;  // slices a warp has in its ring
constexpr int kWarpBytes = kUnitRing * 128 + kFarBlocks * kFarBlock * 16 + kOut * 4;
constexpr int kSmemBytes = kWarps * kWarpBytes;

// A warp's part of the shared memory: its ring, its weights in flight, its output rows.
__device__ __forceinline__ Far warp_far(char *bytes, uint64_t *full) {
    return Far{reinterpret_cast<float4 *>(bytes + (size_t)kUnitRing * 128),
               reinterpret_cast<float *>(bytes + kWarpBytes - kOut * 4), full};
}

struct Queue {
    uint64_t full[kAhead];
    // x: offset / 128 in the ring (kInGlobal: in the blob array), y: n, z: m | uniform << 8,
    // w: offset / 128 of the blob's weights
    int4 desc[kAhead];
    int start[kAhead];  // position of the staged bytes
    uint64_t far[kFarBlocks];
};

constexpr int kInGlobal = 512;  // descriptor bit: the staged part is longer than the ring

__device__ __forceinline__ void queue_init(Queue *q) {
    if (threadIdx.x < kWarps) {
        for (int s = 0; s < kAhead; ++s) ring::init(&q[threadIdx.x].full[s], 1);
        for (int s = 0; s < kFarBlocks; ++s) ring::init(&q[threadIdx.x].far[s], 1);
    }
    ring::fence_init();
    __syncthreads();
}

// The state of a warp's queue, the same in all lanes.  Positions are in units of 128 bytes and
// grow without wrapping; a blob does not wrap around the ring's end.
struct Feed {
    int pushed = 0, popped = 0;
    int pos = 0, at = 0;  // position of the next blob, and the same within the ring

    // Whether a slice with `len` * 128 bytes to stage finds room now.
    __device__ __forceinline__ bool room(const Queue &q, int len) const {
        if (pushed == popped) return true;
        if (pushed - popped == kAhead) return false;
        if (len > kUnitRing) return true;
        const int skip = at + len > kUnitRing ? kUnitRing - at : 0;
        return pos + skip + len - q.start[popped % kAhead] <= kUnitRing;
    }

    // Appends the slice `d` (offset / 128, n, m | uniform << 8, bytes to stage / 128) of `blob`.
    __device__ __forceinline__ void push(Queue &q, char *bytes, const char *blob, int4 d, int lane,
                                         uint64_t policy) {
        const int s = pushed % kAhead;
        const bool fits = d.w <= kUnitRing;
        if (fits && at + d.w > kUnitRing) {
            pos += kUnitRing - at;
            at = 0;
        }
        if (lane == 0) {
            q.start[s] = pos;
            q.desc[s] = make_int4(fits ? at : d.x, d.y, fits ? d.z : d.z | kInGlobal, d.x + d.w);
            if (fits) {
                ring::arrive_expect_tx(&q.full[s], (uint32_t)d.w * 128);
                ring::bulk_g2s(bytes + (size_t)at * 128, blob + (size_t)d.x * 128,
                               (uint32_t)d.w * 128, &q.full[s], policy);
            } else {
                ring::arrive(&q.full[s]);
            }
            if (!(d.z & 256) && d.y > 0)  // at most what kUnitMost lists of kUnitList have
                ring::bulk_prefetch(blob + (size_t)(d.x + d.w) * 128,
                                    (uint32_t)min(((d.y + 3) & ~3) * (d.z & 0xff),
                                                  kUnitMost * kUnitList) * 128);
        }
        if (fits) {
            pos += d.w;
            at += d.w;
        }
        ++pushed;
        __syncwarp();
    }
};

// The slice in slot s, once full.  shift: log2 of the lanes that share a unit.  False when a wait
// for its weights expired.
template <bool COLLECT, class A>
__device__ __forceinline__ bool consume(const A &a, const Queue &q, const char *bytes,
                                        const char *blob, Far &far, int s, int lane, int shift,
                                        uint64_t pol_stream, int *status) {
    const int4 d = q.desc[s];
    const char *p = bytes + (size_t)d.x * 128;
    const float4 *w = reinterpret_cast<const float4 *>(blob + (size_t)d.w * 128);
    const int m = d.z & 0xff;
    const bool uni = (d.z & 256) != 0;
    switch (d.y > kUnitList ? 5 : (d.y + 3) >> 2) {
        case 4:
            return slice<4, COLLECT>(a, p, w, far, d.y, m, uni, lane, shift, pol_stream, status);
        case 3:
            return slice<3, COLLECT>(a, p, w, far, d.y, m, uni, lane, shift, pol_stream, status);
        case 2:
            return slice<2, COLLECT>(a, p, w, far, d.y, m, uni, lane, shift, pol_stream, status);
        case 5:
            long_slice<COLLECT>(a,
                            reinterpret_cast<const int *>(
                                d.z & kInGlobal ? blob + (size_t)d.x * 128 : p),
                            w, d.y, far.out, lane, shift);
            return true;
        default:
            return slice<1, COLLECT>(a, p, w, far, d.y, m, uni, lane, shift, pol_stream, status);
    }
}

// Behind an expired wait: the copies that are still on their way into this warp's shared memory,
// which is another CTA's when this one has left, each waited for with a limit again.
__device__ __forceinline__ void drain(Queue &q, const Feed &f, const Far &far, int *status) {
    for (int k = f.popped; k < f.pushed; ++k)
        ring::wait(&q.full[k % kAhead], (uint32_t)(k / kAhead) & 1, status);
    for (int k = far.used; k < far.issued; ++k)
        ring::wait(&q.far[k % kFarBlocks], (uint32_t)(k / kFarBlocks) & 1, status);
}

// Lanes that share a unit of a primvar `length` floats wide: one per 4 columns, 4 at most.
__host__ __device__ inline int unit_shift(int length) { return length <= 4 ? 0 : length <= 8 ? 1 : 2; }

}  // namespace units
}  // namespace gb300
