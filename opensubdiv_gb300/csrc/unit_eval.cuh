// Evaluation of one slice of the unit layout (units.h) by one warp, shared by the table kernel
// (stencils_units.cu) and the batched kernel (stencils_batch.cu).  `A` is the launch's argument
// view: src (rows 16-byte aligned), srcStride, length, dst[0], dstStride[0].  COLLECT: the rows of
// dst are not 16-byte aligned.
//
// A lane holds 4 columns of the up to 16 source rows of its unit's list in registers and runs
// through the unit's stencils: the rows are gathered once for all of them, 16 loads in flight at
// a time, and each stencil is 64 fused multiply-adds on registers.  2 or 4 neighbouring lanes share
// a unit of 5-8 or more columns, so that they read and write a row together.
//
// Per stencil the sum runs over its entries in table order with one fused multiply-add per
// element, as in every other EvalStencils kernel here, so results do not depend on the layout.
#pragma once

#include "stage_ring.cuh"
#include "units.h"

namespace gb300 {
namespace units {

// Columns [c0, c0 + 4) of source row `id`: rows are 16-byte aligned, their stride a multiple of 4
// floats (columns at or past the length, inside the stride, are read and not used).
template <class A>
__device__ __forceinline__ float4 load_quad(const A &a, int id, int c0) {
    return ld_point4(a.src + (size_t)id * a.srcStride + c0);
}

// Output rows are 16-byte aligned, their stride a multiple of 4 floats.
template <class A>
__device__ __forceinline__ void store_quad(const A &a, int row, int c0, const float4 &v) {
    float *d = a.dst[0] + (size_t)row * a.dstStride[0] + c0;
    const int rem = a.length - c0;
    if (rem >= 4) {
        asm volatile("st.global.cs.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(d), "f"(v.x), "f"(v.y),
                     "f"(v.z), "f"(v.w)
                     : "memory");
        return;
    }
    st_stream(d, v.x);
    if (rem > 1) st_stream(d + 1, v.y);
    if (rem > 2) st_stream(d + 2, v.z);
}

constexpr int kOut = 128;  // floats of one stencil of all units evaluated at a time

// Rows of any other layout (xyz above all): the columns [c, c + width) of one stencil of `units` units,
// collected in `out` and written so that neighbouring lanes write neighbouring elements.  The lanes'
// own stores would take one for every element, each to another row's sector.  magic: 65536 / width + 1.
template <class A>
__device__ __forceinline__ void store_collected(const A &a, float *out, const int *rows, int units,
                                                int shift, int c, int width, unsigned magic,
                                                int lane, const float4 &v) {
    const int at = 4 * (lane & ((1 << shift) - 1));
    float *d = out + (lane >> shift) * width + at;
    if (at < width) d[0] = v.x;
    if (at + 1 < width) d[1] = v.y;
    if (at + 2 < width) d[2] = v.z;
    if (at + 3 < width) d[3] = v.w;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kOut / 32; ++i) {
        const int e = lane + 32 * i, u = (int)((unsigned)e * magic >> 16);
        if (e >= units * width) break;
        const int row = rows[u];
        if (row >= 0)
            st_stream(a.dst[0] + (size_t)row * a.dstStride[0] + c + (e - u * width), out[e]);
    }
    __syncwarp();
}

__device__ __forceinline__ float4 load_far(const float4 *p) {  // weights, read once
    float4 v;
    asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "l"(p));
    return v;
}

// Weights of slices that are not uniform, on their way to a warp: blocks of kFarBlock float4s of
// shared memory, each filled by bulk copies and handed over by its barrier.
constexpr int kFarBlocks = 3;
constexpr int kFarBlock = 128;

struct Far {
    float4 *buf;
    float *out;  // kOut floats, where output rows are collected
    uint64_t *full;
    int issued = 0, used = 0;  // blocks, over all slices
};

__device__ __forceinline__ void add_row(float w, const float4 &x, float4 &acc) {
    acc.x = fmaf(w, x.x, acc.x);
    acc.y = fmaf(w, x.y, acc.y);
    acc.z = fmaf(w, x.z, acc.z);
    acc.w = fmaf(w, x.w, acc.w);
}

// Rows [j0, j0 + 4 NQ) of a unit's list of k entries; zeros past its end (whose weights are 0).
template <int NQ, class A>
__device__ __forceinline__ void gather(const A &a, const int *idx, int j0, int k, int c0,
                                       float4 (&x)[4 * NQ]) {
#pragma unroll
    for (int j = 0; j < 4 * NQ; ++j) {
        x[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (j0 + j < k) x[j] = load_quad(a, idx[32 * (j0 + j)], c0);
    }
}

// A slice whose rows, sizes and indices are in shared memory at p, with a uniform slice's weights
// behind them; the weights of any other slice are in global memory (weights) and pass through
// `far`, a block of 2^shift stencils at a time, as many blocks ahead as there are.  NQ =
// ceil(n / 4).  One loop serves both kinds: with one body per kind the instruction cache did not
// hold the bodies that the warps of an SM run at the same time.
template <int NQ, bool COLLECT, class A>
__device__ __forceinline__ bool slice(const A &a, const char *p, const float4 *weights, Far &far,
                                      int n, int m, bool uni, int lane, int shift,
                                      uint64_t pol_stream, int *status) {
    const int *rows = reinterpret_cast<const int *>(p);
    const int *idx = rows + 32 * m + (uni ? 0 : 32);
    const int units = 32 >> shift;            // evaluated at a time
    const int per = uni ? m : 1 << shift;     // stencils per block
    const int qstep = uni ? 1 : 8;            // float4s between the quads of a stencil
    // where the block after the last requested one starts
    int fu = 0, fc = 0, fs = 0;
    auto fetch = [&]() {
        if (fu >= 32) return;
        const int count = min(per, m - fs);
        if (lane == 0) {
            const int k = far.issued % kFarBlocks;
            ring::arrive_expect_tx(&far.full[k], (uint32_t)(count * NQ * units) * 16);
            for (int o = 0; o < units / 8; ++o)
                ring::bulk_g2s(far.buf + k * kFarBlock + o * per * NQ * 8,
                               weights + (size_t)((fu / 8 + o) * m + fs) * (NQ * 8),
                               (uint32_t)(count * NQ * 8) * 16, &far.full[k], pol_stream);
        }
        ++far.issued;
        fs += per;
        if (fs >= m) {
            fs = 0;
            fc += 4 << shift;
            if (fc >= a.length) {
                fc = 0;
                fu += units;
            }
        }
    };
    if (!uni)
        for (int b = 0; b < kFarBlocks; ++b) fetch();
#pragma unroll 1
    for (int u0 = 0; u0 < 32; u0 += units) {
        const int u = u0 + (lane >> shift);
        const int k = uni ? n : rows[32 * m + u];
#pragma unroll 1
        for (int c = 0; c < a.length; c += 4 << shift) {
            const int c0 = c + 4 * (lane & ((1 << shift) - 1));
            const bool on = c0 < a.length;
            const int width = min(4 << shift, a.length - c);
            const unsigned magic = COLLECT ? 65536u / (unsigned)width + 1 : 0;
            float4 x[4 * NQ];
            gather<NQ>(a, idx + u, 0, on ? k : 0, c0, x);
#pragma unroll 1
            for (int s = 0; s < m;) {
                const float4 *w = reinterpret_cast<const float4 *>(idx + 32 * n);
                if (!uni) {
                    const int b = far.used % kFarBlocks;
                    if (!ring::wait(&far.full[b], (uint32_t)(far.used / kFarBlocks) & 1, status))
                        return false;
                    const int lu = lane >> shift;
                    w = far.buf + b * kFarBlock + (lu >> 3) * per * NQ * 8 + (lu & 7);
                }
                const int end = min(s + per, m);
#pragma unroll 1
                for (; s < end; ++s) {
                    const int row = COLLECT ? 0 : rows[32 * s + u];
                    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                    for (int q = 0; q < NQ; ++q, w += qstep) {
                        const float4 v = *w;
                        add_row(v.x, x[4 * q], acc);
                        add_row(v.y, x[4 * q + 1], acc);
                        add_row(v.z, x[4 * q + 2], acc);
                        add_row(v.w, x[4 * q + 3], acc);
                    }
                    if constexpr (COLLECT)
                        store_collected(a, far.out, rows + 32 * s + u0, units, shift, c, width,
                                        magic, lane, acc);
                    else if (on && row >= 0)
                        store_quad(a, row, c0, acc);
                }
                if (!uni) {
                    __syncwarp();
                    ++far.used;
                    fetch();
                }
            }
        }
    }
    return true;
}

// A slice of single stencils of more than 16 entries, 16 at a time; p may be in global memory.
template <bool COLLECT, class A>
__device__ __forceinline__ void long_slice(const A &a, const int *rows, const float4 *far, int n,
                                           float *out, int lane, int shift) {
    const int nq = (n + 3) / 4;
#pragma unroll 1
    for (int u = lane >> shift; u < 32; u += 32 >> shift) {
        const int row = rows[u], k = rows[32 + u];
        const int *idx = rows + 64 + u;
#pragma unroll 1
        for (int c = 0; c < a.length; c += 4 << shift) {
            const int c0 = c + 4 * (lane & ((1 << shift) - 1));
            const bool on = c0 < a.length && row >= 0;
            float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 1
            for (int j = 0; j < k; j += 16) {
                float4 x[16], v[4];
                gather<4>(a, idx, j, on ? k : 0, c0, x);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    v[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (j + 4 * q < k)
                        v[q] = load_far(far + ((size_t)(u / 8) * nq + j / 4 + q) * 8 + u % 8);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    add_row(v[q].x, x[4 * q], acc);
                    add_row(v[q].y, x[4 * q + 1], acc);
                    add_row(v[q].z, x[4 * q + 2], acc);
                    add_row(v[q].w, x[4 * q + 3], acc);
                }
            }
            if constexpr (COLLECT) {
                const int width = min(4 << shift, a.length - c);
                store_collected(a, out, rows + u - (lane >> shift), 32 >> shift, shift, c, width,
                                65536u / (unsigned)width + 1, lane, acc);
            } else if (on) {
                store_quad(a, row, c0, acc);
            }
        }
    }
}

}  // namespace units
}  // namespace gb300
