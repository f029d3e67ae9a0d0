// Unit evaluation layout of a device stencil table with one weight array: its construction on
// the device (unit_build.cu) and its EvalStencils launch (stencils_units.cu).
//
// Refined vertices come in families.  The stencils of the vertices of one face share their
// control vertices (25 of the 64 level-3 vertices of a regular quad read the same 16 control
// points), and the faces of a neighbourhood repeat the same weights.  The layout stores each of the
// two once:
//   unit   stencils with the same list of control indices (same order), in table order, evaluated
//          by one lane (or 2 or 4) from rows that are gathered once; up to kUnitMost of them, fewer
//          in a small table, 1 when the list is longer than kUnitList;
//   slice  32 units, one warp's work; m = the most stencils, n = the longest list of its units.  A
//          slice whose 32 units have the same weights is uniform and holds them once.
// Units are ordered by the lowest control index of their stencils, cut into windows, and within
// a window by size and weights, so that equal weights fill whole slices.
//
// A slice is one blob, a multiple of 128 bytes:
//   rows     32 * m ints, rows[32 s + lane]: destination stencil (-1: none)
//   sizes    32 ints, the unit's number of entries (not in a uniform slice: all have n)
//   indices  32 * n ints, entry j of lane l at 32 j + l
//   weights  n4 = n rounded up to a multiple of 4, at least 4, zeros past the end; uniform:
//            m * n4 floats, [s][j] (padded to 128 bytes), else 32 * m * n4, by 8 lanes:
//            [lane / 8][s][j / 4][lane % 8][j % 4]
// All but the weights of a slice that is not uniform is staged through shared memory.
// Slices are stored in locality order (by the first of their units), so that the slices of one
// neighbourhood, which read the same source rows, are evaluated together.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace gb300 {

struct UnitTable {
    int numSlices = 0;
    const int4 *slice = nullptr;  // blob offset / 128, n, m | uniform << 8, bytes to stage / 128
    const char *blob = nullptr;
    bool regular = false;  // at least half of the stencils are in uniform slices
    int numStencils = 0;
};

// Tables from kUnitTable stencils on may have the layout beside the sliced one: from kUnitCall on they get
// it when they are made, smaller ones in the first batch that may take it (a table of 69 k stencils was
// made in 2.6 ms before the layout, 3.1 with it).  A single call takes it from kUnitCall on; below, there are too few slices for the SMs' warps (8-wide level-3 rows, against the
// sliced layout: 131 k stencils 10.3 and 10.3 us, 295 k 12.3 and 14.7 us, 524 k 14.8 and 20.7 us, 1.2 M
// 29.1 and 39.0 us).  A batch's jobs fill the SMs together: it takes the layout for all of them when
// they have 2 * kUnitTable stencils between them (one job of 75 k stencils, 3- and 12-wide: 13.8 and
// 12.4 us with it, 12.4 and 10.3 without; of 134 k 13.0 and 12.4, 16.4 and 18.3 without).
constexpr int kUnitTable = 1 << 16, kUnitCall = 1 << 18, kUnitAnyRow = 3 << 19;

constexpr int kUnitMost = 16;  // stencils per unit
constexpr int kUnitList = 16;  // entries held in registers

// Bytes / 128 of a warp's ring; a slice with more to stage is read from global memory.
constexpr int kUnitRing = 60;

// Builds the layout of the device CSR table (sizes, offsets, indices, one weight array) on
// stream `s` and waits for it.  The 2 allocations (slice, blob) go to `owned` for the
// caller to free; `t` points into them.  GB300_ERR_UNSUPPORTED (nothing allocated): the table has
// fewer than 2 stencils per unit, and little to share (level-1 stencils, 12-wide rows: 18.4 us
// against 13.7 us from the sliced layout).
int build_units(int numStencils, const int *sizes, const int *offsets, const int *indices,
                const float *weights, cudaStream_t s, UnitTable &t, void *owned[2],
                const char *who);

// Whether the layout's kernels read these source rows: 16-byte aligned, the stride a multiple of 4
// floats.  Output rows may have any layout; those that are not 16-byte aligned are collected.
bool units_take(const float *src, int srcStride);
bool units_collect(const float *dst, int dstStride);

// How the layout writes `length` floats in rows of `stride` at dst, if it is the better one there: not at
// all, row by row, or collected.  bytes: the rows of the call, or of all jobs of a batch.
enum UnitRows { kUnitNone, kUnitByRow, kUnitCollected };
UnitRows units_rows(const UnitTable &t, const float *dst, int stride, int length, long long bytes,
                    bool batch);

int eval_stencils_units(const UnitTable &t, UnitRows rows, const float *src, float *dst, int dstStride,
                        int length, int srcStride, cudaStream_t s, const char *who);

}  // namespace gb300
