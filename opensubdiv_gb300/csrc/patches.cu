// EvalPatches for sm_103a: one thread per patch coordinate; PatchParam decode, basis and the
// gather of up to 20 control points are fused and kept in registers, and all requested
// outputs (P, dPdu, dPdv, dPduu, dPduv, dPdvv) come out of one pass.  Replaces
// computePatches (osd/cudaKernel.cu:244-328), which spills six float[20] weight arrays and
// accumulates each output in global memory.
#include "common.cuh"
#include "patch_basis.cuh"

namespace gb300 {

struct Coord {
    int arrayIndex, patchIndex, vertIndex;
    float s, t;
};
struct Array {
    int regDesc, desc, numPatches, indexBase, stride, primitiveIdBase;
};
struct ParamRec {
    int field0, field1;
    float sharpness;
};

// A query's patch coordinate (read once: evict-first) and its patch's param (evict-last).
__device__ __forceinline__ Coord load_coord(const Coord *p) {
    const int *q = reinterpret_cast<const int *>(p);
    const uint64_t pol = l2_evict_first();
    Coord c;
    c.arrayIndex = ld_query(q, pol);
    c.patchIndex = ld_query(q + 1, pol);
    c.vertIndex = ld_query(q + 2, pol);
    c.s = __int_as_float(ld_query(q + 3, pol));
    c.t = __int_as_float(ld_query(q + 4, pol));
    return c;
}
__device__ __forceinline__ ParamRec load_param(const ParamRec *p) {
    const int *q = reinterpret_cast<const int *>(p);
    const uint64_t pol = l2_evict_last();
    return ParamRec{ld_param(q, pol), ld_param(q + 1, pol), __int_as_float(ld_param(q + 2, pol))};
}

struct PatchArgs {
    const float *src;
    float *dst[6];
    int dstStride[6];
    int active;
    int length;
    int srcStride;
    int numCoords;
    const Coord *coords;
    const Array *arrays;
    const int *indices;
    const ParamRec *params;
    int rows;  // kQuadRows: source rows are padded to quads; kPatchRows: and one per patch index
};

// The arguments with the pointers whose loads may move as they stand behind the wait.
template <int LC, int V4>
__device__ __forceinline__ PatchArgs args_behind_wait(const PatchArgs &arg) {
    PatchArgs a = arg;
    if (LC == 1) {
        behind_wait(a.src);
        behind_wait(a.indices);
    }
    return a;
}

// Highest output index a derivative order needs: 0 P only, 1 P + du + dv, 2 all six.  The
// kernels are instantiated per order so the unused accumulations compile away.
__host__ __device__ constexpr int last_output(int order) { return order == 0 ? 0 : order == 1 ? 2 : 5; }

// Elements [e0, e0 + LC) of all outputs of the point at c, and the outputs' scales.
template <int LC, bool QUAD, int V4>
__device__ __forceinline__ void eval_point(const PatchArgs &a, const Coord &c, int e0,
                                           Acc6<LC> &acc, float (&scale)[6]) {
    acc.zero();
    float d1 = 1.0f, d2 = 1.0f;
    if (c.arrayIndex >= 0) {
        const Array arr = a.arrays[c.arrayIndex];
        const ParamRec pr = load_param(a.params + c.patchIndex);
        const Param p{pr.field0, pr.field1};
        const int type = p.regular() ? arr.regDesc : arr.desc;
        const int first = arr.indexBase + arr.stride * (c.patchIndex - arr.primitiveIdBase);
        const float *src = V4 == kPatchRows ? a.src + (size_t)first * 4 : a.src;
        if (!eval_patch_point<LC, QUAD, V4>(type, p, c.s, c.t, a.indices + first, src,
                                            a.srcStride, e0, a.length, acc, d1, d2))
            acc.zero();
    }
    scale[0] = 1.0f;
    scale[1] = scale[2] = d1;
    scale[3] = scale[4] = scale[5] = d2;
}

// 5 resident blocks per SM where the registers allow it without spills (0.2847 vs 0.2908 ms
// for 4 M Loop points at LC = 3; LC = 4 would spill)
// QUAD: Catmull-Clark tables (REGULAR / GREGORY_BASIS / QUADS only): without the Loop and
// triangle bases the kernel fits 7 blocks per SM for orders 0 and 1 without spills.
// Outputs are stored by their threads: collected through shared memory, whole sectors a store, they
// take the warp a loop of its own and the registers for it (4 M Loop points of xyz, 71 k rows: P 164
// and 173 us, with first derivatives 170 and 181, all six 199 and 211; points in patch order, 2.9 M
// coords of a tessellation, 132 and 154).
// V4: source rows are read as one quad each (patch_basis.cuh; with a row per patch index 4 M Loop
// points of six outputs take 205 us, copy included, with a row per control point 231, in place 293).
template <int LC, int ORDER, bool QUAD = false, int V4 = kAnyRows>
__global__ void __launch_bounds__(128, LC == 4 ? 4 : (ORDER < 2 && !V4 ? (QUAD ? 7 : 6) : 5))
    k_eval_patches(const PatchArgs arg) {
    launch_dependents();
    wait_for_primary();
    const PatchArgs a = args_behind_wait<LC, V4>(arg);
    const int stride = gridDim.x * blockDim.x;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.numCoords; i += stride) {
        const Coord c = load_coord(a.coords + i);
        for (int e0 = 0; e0 < a.length; e0 += LC) {
            Acc6<LC> acc;
            float scale[6];
            eval_point<LC, QUAD, V4>(a, c, e0, acc, scale);
#pragma unroll
            for (int k = 0; k <= last_output(ORDER); ++k) {
                if (!(a.active & (1 << k))) continue;
                float *out = a.dst[k] + (size_t)i * a.dstStride[k] + e0;
#pragma unroll
                for (int m = 0; m < LC; ++m)
                    if (e0 + m < a.length) st_stream(out + m, acc.v[k][m] * scale[k]);
            }
        }
    }
}

// G lanes per point, lane l owning primvar elements l, l + G, ...: one source-row fetch is a
// single coalesced access for the whole group, the accumulators are per element (6 per
// lane) and no cross-lane reduction is needed.  The basis is evaluated by every lane of the
// group (cheap for the separable quad-family bases this kernel is used for).  P and first derivatives
// of 6 and more lanes take a REGULAR patch row by row; else its 16 loads are in flight together (2 M
// points of 5, 8 and 12 floats 1007, 277 and 1012 us so, 944, 266 and 950 row by row; all six outputs
// of 5 floats 1205 and 1257, P of 8 floats 229 and 234).
template <int G, int ORDER>
__global__ void __launch_bounds__(256, 4) k_eval_patches_lanes(const PatchArgs arg) {
    launch_dependents();
    wait_for_primary();
    const PatchArgs a = args_behind_wait<1, kAnyRows>(arg);
    // G need not be a power of two: a warp holds floor(32 / G) groups (3 lanes per point
    // for xyz: 10 points per warp) and its remaining lanes stay idle
    constexpr int kPerWarp = 32 / G;
    const int wl = threadIdx.x & 31;
    const int slot = wl / G;
    if (slot >= kPerWarp) return;
    const int lane = wl - slot * G;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int group = warp * kPerWarp + slot;
    const int ngroups = nwarps * kPerWarp;
    for (int i = group; i < a.numCoords; i += ngroups) {
        const Coord c = load_coord(a.coords + i);
        for (int e0 = 0; e0 < a.length; e0 += G) {
            const int e = e0 + lane;
            Acc6<1> acc;
            acc.zero();
            float d1 = 1.0f, d2 = 1.0f;
            if (c.arrayIndex >= 0) {
                const Array arr = a.arrays[c.arrayIndex];
                const ParamRec pr = load_param(a.params + c.patchIndex);
                const Param p{pr.field0, pr.field1};
                const int type = p.regular() ? arr.regDesc : arr.desc;
                const int *cvs =
                    a.indices + arr.indexBase + arr.stride * (c.patchIndex - arr.primitiveIdBase);
                if (!eval_patch_point<1, true, kAnyRows, (ORDER == 1 && G >= 6)>(
                        type, p, c.s, c.t, cvs, a.src, a.srcStride, e, a.length, acc, d1, d2))
                    acc.zero();
            }
            if (e < a.length) {
                const float scale[6] = {1.0f, d1, d1, d2, d2, d2};
#pragma unroll
                for (int k = 0; k <= last_output(ORDER); ++k)
                    if (a.active & (1 << k))
                        st_stream(a.dst[k] + (size_t)i * a.dstStride[k] + e, acc.v[k][0] * scale[k]);
            }
        }
    }
}

template <int ORDER>
void launch_lanes(int G, int grid, int threads, cudaStream_t s, const PatchArgs &a) {
    switch (G) {
        case 1: launch_kernel(k_eval_patches_lanes<1, ORDER>, grid, threads, 0, s, a); break;
        case 2: launch_kernel(k_eval_patches_lanes<2, ORDER>, grid, threads, 0, s, a); break;
        case 3: launch_kernel(k_eval_patches_lanes<3, ORDER>, grid, threads, 0, s, a); break;
        case 4: launch_kernel(k_eval_patches_lanes<4, ORDER>, grid, threads, 0, s, a); break;
        case 6: launch_kernel(k_eval_patches_lanes<6, ORDER>, grid, threads, 0, s, a); break;
        case 8: launch_kernel(k_eval_patches_lanes<8, ORDER>, grid, threads, 0, s, a); break;
        default: launch_kernel(k_eval_patches_lanes<32, ORDER>, grid, threads, 0, s, a); break;
    }
}

template <int ORDER, bool QUAD>
void launch_points(int length, int grid, int threads, cudaStream_t s, const PatchArgs &a) {
    // whole quads at 16-byte aligned addresses: nothing past a row's elements is read
    const bool v4 = ((uintptr_t)a.src & 15) == 0 && a.srcStride % 4 == 0 &&
                    (a.length % 4 == 0 || a.rows);
    switch (length) {
        case 1: launch_kernel(k_eval_patches<1, ORDER, QUAD>, grid, threads, 0, s, a); break;
        case 2: launch_kernel(k_eval_patches<2, ORDER, QUAD>, grid, threads, 0, s, a); break;
        case 3:
            if constexpr (!QUAD) {
                if (a.rows == kPatchRows) {
                    launch_kernel(k_eval_patches<3, ORDER, false, kPatchRows>, grid, threads, 0, s, a);
                    break;
                }
            }
            if (v4) launch_kernel(k_eval_patches<3, ORDER, QUAD, kQuadRows>, grid, threads, 0, s, a);
            else launch_kernel(k_eval_patches<3, ORDER, QUAD>, grid, threads, 0, s, a);
            break;
        default:
            if (v4) launch_kernel(k_eval_patches<4, ORDER, QUAD, kQuadRows>, grid, threads, 0, s, a);
            else launch_kernel(k_eval_patches<4, ORDER, QUAD>, grid, threads, 0, s, a);
            break;
    }
}

// One quad per patch index: the row of 3 floats that it names.
struct GatherArgs {
    const float *src;
    int srcStride;
    const int *indices;
    int n;
    float4 *rows;
};

__global__ void __launch_bounds__(256) k_gather_patch_rows(const GatherArgs a) {
    launch_dependents();
    wait_for_primary();
    const int stride = gridDim.x * blockDim.x;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < a.n; j += stride) {
        const int cv = a.indices[j];
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (cv >= 0) {
            const float *p = a.src + (size_t)cv * a.srcStride;
            v.x = p[0], v.y = p[1], v.z = p[2];
        }
        a.rows[j] = v;
    }
}

int gather_patch_rows(const float *src, int srcStride, const int *indices, int n, float *rows,
                      cudaStream_t s) {
    const GatherArgs a{src, srcStride, indices, n, reinterpret_cast<float4 *>(rows)};
    const int blocks = (n + 255) / 256, cap = num_sms() * 8;
    launch_kernel(k_gather_patch_rows, blocks < cap ? blocks : cap, 256, 0, s, a);
    return GB300_OK;
}

int eval_patches(const float *src, float *const *dst, const int *strides, int length,
                 int srcStride, int numCoords, const void *coords, const void *arrays,
                 const int *indices, const void *params, cudaStream_t s, const char *who,
                 int quadFamily, int grouped, int rows) {
    if (numCoords <= 0) return ok();
    if (!src || !coords || !arrays || !indices || !params)
        return fail(GB300_ERR_INVALID_ARGUMENT, "%s: null source, coord or table pointer", who);
    if (length <= 0 || srcStride < length)
        return fail(GB300_ERR_INVALID_ARGUMENT, "%s: bad length %d / source stride %d", who,
                    length, srcStride);
    PatchArgs a{};
    a.src = src;
    a.length = length;
    a.srcStride = srcStride;
    a.numCoords = numCoords;
    a.coords = (const Coord *)coords;
    a.arrays = (const Array *)arrays;
    a.indices = indices;
    a.params = (const ParamRec *)params;
    a.rows = rows;
    for (int k = 0; k < 6; ++k) {
        if (!dst[k]) continue;
        if (strides[k] < length)
            return fail(GB300_ERR_INVALID_ARGUMENT, "%s: output %d stride %d < length %d", who, k,
                        strides[k], length);
        a.dst[k] = dst[k];
        a.dstStride[k] = strides[k];
        a.active |= 1 << k;
    }
    if (!a.active) return ok();
    const int order = (a.active & 0x38) ? 2 : (a.active & 0x6) ? 1 : 0;
    if (quadFamily && !grouped) {
        // element-lane kernel: G = length lanes per point for the common widths, else 32
        // lanes looping over element chunks
        const int G = (length <= 4 || length == 6 || length == 8) ? length : 32;
        const int perWarp = 32 / G;
        const int threads = 256;
        long long warps = ((long long)numCoords + perWarp - 1) / perWarp;
        long long blocks = (warps * 32 + threads - 1) / threads;
        long long cap = (long long)num_sms() * 16;
        const int grid = (int)(blocks < cap ? blocks : cap);
        if (order == 0) launch_lanes<0>(G, grid, threads, s, a);
        else if (order == 1) launch_lanes<1>(G, grid, threads, s, a);
        else launch_lanes<2>(G, grid, threads, s, a);
        return check_launch(who);
    }
    // one thread per point: tables with triangle patches, and points grouped by patch (a
    // tessellation's coords), whose row loads are shared by the warp and whose basis each
    // thread then computes once rather than once per element lane
    const int threads = 128;
    long long blocks = ((long long)numCoords + threads - 1) / threads;
    long long cap = (long long)num_sms() * 32;
    const int grid = (int)(blocks < cap ? blocks : cap);
    if (quadFamily) {
        if (order == 0) launch_points<0, true>(length, grid, threads, s, a);
        else if (order == 1) launch_points<1, true>(length, grid, threads, s, a);
        else launch_points<2, true>(length, grid, threads, s, a);
    } else {
        if (order == 0) launch_points<0, false>(length, grid, threads, s, a);
        else if (order == 1) launch_points<1, false>(length, grid, threads, s, a);
        else launch_points<2, false>(length, grid, threads, s, a);
    }
    return check_launch(who);
}

}  // namespace gb300

using namespace gb300;

extern "C" {

int GB300EvalPatches(const float *src, float *dst, int length, int srcStride, int dstStride,
                     int numPatchCoords, const void *patchCoords, const void *patchArrays,
                     const int *patchIndices, const void *patchParams, void *stream) {
    if (!dst) return fail(GB300_ERR_INVALID_ARGUMENT, "GB300EvalPatches: null destination");
    float *d[6] = {dst, 0, 0, 0, 0, 0};
    int st[6] = {dstStride, 0, 0, 0, 0, 0};
    return eval_patches(src, d, st, length, srcStride, numPatchCoords, patchCoords, patchArrays,
                        patchIndices, patchParams, as_stream(stream), "GB300EvalPatches", 0, 0, 0);
}

int GB300EvalPatchesWithDerivatives(
    const float *src, float *dst, float *du, float *dv, float *duu, float *duv, float *dvv,
    int length, int srcStride, int dstStride, int duStride, int dvStride, int duuStride,
    int duvStride, int dvvStride, int numPatchCoords, const void *patchCoords,
    const void *patchArrays, const int *patchIndices, const void *patchParams, void *stream) {
    float *d[6] = {dst, du, dv, duu, duv, dvv};
    int st[6] = {dstStride, duStride, dvStride, duuStride, duvStride, dvvStride};
    return eval_patches(src, d, st, length, srcStride, numPatchCoords, patchCoords, patchArrays,
                        patchIndices, patchParams, as_stream(stream),
                        "GB300EvalPatchesWithDerivatives", 0, 0, 0);
}

}  // extern "C"
