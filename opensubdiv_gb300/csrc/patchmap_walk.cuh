// Device walk of the PatchMap quadtree (far/patchMap.h:192-231), shared by the FindPatches
// kernel and kernels that locate the points they generate.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace gb300 {

// Child slot encoding of a packed quadtree node: set, leaf (a patch handle index) or inner
// node index.
static constexpr uint32_t kSet = 0x80000000u, kLeaf = 0x40000000u, kIndex = 0x3fffffffu;

constexpr int kMapArrays = 4;

struct PatchMapView {
    const uint4 *nodes;
    const int4 *handles;
    int minFace, maxFace, maxDepth, triangular, numPatches;
    // first patch and indices per patch of each patch array, for tables of at most kMapArrays
    // (numArrays 0: loaded): a handle is then computed from the leaf instead of loaded (one random
    // 16-byte read less per query, out of 23 MB for 1.4 M patches; small tables' stay in L1)
    int numArrays = 0;
    int first[kMapArrays] = {}, step[kMapArrays] = {};
};

__device__ __forceinline__ uint32_t child_of(const uint4 &n, int q) {
    return q == 0 ? n.x : q == 1 ? n.y : q == 2 ? n.z : n.w;
}

// The handle of leaf h: patch h of the table, which is the (h - first)-th of its array.
__device__ __forceinline__ int4 patch_map_handle(const PatchMapView &m, int h) {
    if (m.numArrays == 0) return __ldg(m.handles + h);
    int a = 0;
#pragma unroll
    for (int k = 1; k < kMapArrays; ++k)
        if (k < m.numArrays && h >= m.first[k]) a = k;
    int first = m.first[0], step = m.step[0];
#pragma unroll
    for (int k = 1; k < kMapArrays; ++k)
        if (a == k) first = m.first[k], step = m.step[k];
    return make_int4(a, h, (h - first) * step, 0);
}

// u + v >= m for floats 0 <= u, v <= m (m a power of two), as the sum in double compares (a double
// sum of floats below m rounds to m only when it is m), without the FP64 pipe: m - v = t + e
// exactly, t the rounded difference and e its error, |e| at most half the distance from t to its
// neighbour, so u decides unless it is t.
__device__ __forceinline__ bool sum_reaches(float u, float v, float m) {
    const float t = __fsub_rn(m, v);
    const float e = __fsub_rn(__fsub_rn(m, t), v);
    return u > t || (u == t && e <= 0.0f);
}

// Handle {array, patch, vert} of the patch holding (f, fu, fv), or {-1, -1, -1} for a miss.
__device__ __forceinline__ int4 patch_map_find(const PatchMapView &m, int f, float fu,
                                               float fv) {
    int4 h = make_int4(-1, -1, -1, 0);
    const bool in_range = m.numPatches > 0 && f >= m.minFace && f <= m.maxFace && fu >= 0.0f &&
                          fu <= 1.0f && fv >= 0.0f && fv <= 1.0f;
    if (!in_range) return h;
    uint4 node = __ldg(m.nodes + (f - m.minFace));
    if (!(node.x & kSet)) return h;
    if (!m.triangular) {
        float u = fu, v = fv, median = 0.5f;
        for (int d = 0; d <= m.maxDepth; ++d, median *= 0.5f) {
            int q = 0;
            if (u >= median) { u -= median; q |= 1; }
            if (v >= median) { v -= median; q |= 2; }
            const uint32_t c = child_of(node, q);
            if (!(c & kSet)) break;
            if (c & kLeaf) { h = patch_map_handle(m, (int)(c & kIndex)); break; }
            node = __ldg(m.nodes + (c & kIndex));
        }
    } else {
        // every subtraction takes the power-of-two median from a value in [median, 2 * median]
        // (exact in float, Sterbenz), so u and v hold the reference's double values exactly;
        // the sums u + v, which the reference rounds in double, are compared exactly
        float u = fu, v = fv, median = 0.5f;
        bool rot = false;
        for (int d = 0; d <= m.maxDepth; ++d, median *= 0.5f) {
            int q;
            if (!rot) {
                if (u >= median) { u -= median; q = 1; }
                else if (v >= median) { v -= median; q = 2; }
                else if (sum_reaches(u, v, median)) { rot = true; q = 3; }
                else q = 0;
            } else {
                if (u < median) { v -= median; q = 1; }
                else if (v < median) { u -= median; q = 2; }
                else {
                    u -= median;
                    v -= median;
                    if (!sum_reaches(u, v, median)) { rot = false; q = 3; }
                    else q = 0;
                }
            }
            const uint32_t c = child_of(node, q);
            if (!(c & kSet)) break;
            if (c & kLeaf) { h = patch_map_handle(m, (int)(c & kIndex)); break; }
            node = __ldg(m.nodes + (c & kIndex));
        }
    }
    return h;
}

}  // namespace gb300
