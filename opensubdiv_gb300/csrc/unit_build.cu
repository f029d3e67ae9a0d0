// Device construction of the unit layout (units.h) of a stencil table:
//   1. one key per stencil (lowest control index, hash of its index list) and a hash of its
//      weights; a radix sort brings stencils with equal lists together, in locality order, table
//      order within a list;
//   2. neighbours whose lists are equal (compared entry by entry) form groups, cut into units;
//   3. one key per unit (window, class, size, hash of its weights): a sort brings units with
//      equal weights together inside each window; every full 32 of a run become a candidate
//      uniform slice, the rest of the window's class follows in order of size;
//   4. slices: their size, the uniform ones verified bit for bit (a hash collision only costs
//      the sharing), a scan of the blob sizes, then one warp per slice writes its blob.
#include <climits>

#include <cub/cub.cuh>

#include "common.cuh"
#include "units.h"

namespace gb300 {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWindow = 16384;  // units per window
constexpr int kPartBits = 1;    // 2^kPartBits parts of a window
constexpr int kMaxSize = 1023;  // longest list told apart by the units' keys

int grid_of(long long items, int perBlock) {
    const long long b = (items + perBlock - 1) / perBlock;
    return (int)std::max<long long>(1, std::min<long long>(b, (long long)num_sms() * 16));
}

// Stencils per unit of a group of `count` stencils with a list of n entries: equal parts of at
// most `most`.
__device__ __forceinline__ int unit_stencils(int n, int count, int most) {
    if (n > kUnitList) return 1;
    const int parts = (count + most - 1) / most;
    return (count + parts - 1) / parts;
}

__device__ __forceinline__ unsigned long long mix(unsigned long long h, unsigned v) {
    h = (h ^ v) * 0x9e3779b97f4a7c15ull;
    return h ^ (h >> 29);
}

struct Csr {
    const int *sizes, *offsets, *indices;
    const float *weights;
};

__global__ void __launch_bounds__(256) k_unit_keys(const Csr c, int n, unsigned long long *key,
                                                   unsigned long long *hashW, int *iota) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int m = c.sizes[i];
        const int *idx = c.indices + c.offsets[i];
        const float *w = c.weights + c.offsets[i];
        unsigned long long hs = 0x1234567u + (unsigned)m, hw = hs;
        unsigned lo = m > 0 ? 0xffffffffu : 0u;
        for (int j = 0; j < m; ++j) {
            const unsigned v = (unsigned)idx[j];
            hs = mix(hs, v);
            hw = mix(hw, __float_as_uint(w[j]));
            lo = min(lo, v);
        }
        key[i] = ((unsigned long long)lo << 32) | (hs >> 32);
        hashW[i] = hw;
        iota[i] = i;
    }
}

// flag[i] = 1 where position i starts a group: its list differs from the one before (flag[n] = 0
// closes the scan).
__global__ void __launch_bounds__(256) k_unit_heads(const Csr c, int n,
                                                    const unsigned long long *key,
                                                    const int *order, int *flag) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
        bool same = i == n || (i > 0 && key[i] == key[i - 1]);
        if (same && i < n) {
            const int a = order[i - 1], b = order[i], m = c.sizes[a];
            same = m == c.sizes[b];
            const int *x = c.indices + c.offsets[a], *y = c.indices + c.offsets[b];
            for (int j = 0; same && j < m; ++j) same = x[j] == y[j];
        }
        flag[i] = !same;
    }
}

// firstOf[g] = first position of item g (id: exclusive scan of the items' start flags), firstOf
// of the number of items = n.
__global__ void __launch_bounds__(256) k_unit_firsts(const int *id, int n, int *firstOf) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x)
        if (id[p + 1] != id[p]) firstOf[id[p]] = p;
    if (blockIdx.x == 0 && threadIdx.x == 0) firstOf[id[n]] = n;
}

// flag[i] = 1 where position i starts a unit of its group (flag[n] = 0 closes the scan).
__global__ void __launch_bounds__(256) k_unit_flags(const Csr c, int n, int most,
                                                    const int *order, const int *group,
                                                    const int *groupAt, int *flag) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
        bool start = false;
        if (i < n) {
            const int g = group[i + 1] - 1, at = groupAt[g];
            start = (i - at) % unit_stencils(c.sizes[order[i]], groupAt[g + 1] - at, most) == 0;
        }
        flag[i] = start;
    }
}

// Per unit its first position and number of stencils, and its key: window, more stencils first,
// longer lists first, hash of the weights of its stencils.
__global__ void __launch_bounds__(256) k_unit_units(const Csr c, int n, int windowBits,
                                                    const int *order, const int *id,
                                                    const int *unitAt,
                                                    const unsigned long long *hashW, int *count,
                                                    unsigned long long *key, int *iota) {
    const int nu = id[n];
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < nu; u += gridDim.x * blockDim.x) {
        const int i = unitAt[u], m = unitAt[u + 1] - i, size = c.sizes[order[i]];
        unsigned long long h = 0x51ed27u + m;
        for (int k = 0; k < m; ++k) {
            const unsigned long long w = hashW[order[i + k]];
            h = mix(mix(h, (unsigned)w), (unsigned)(w >> 32));
        }
        h *= 0xbf58476d1ce4e5b9ull;
        const unsigned long long top =
            ((unsigned long long)(u / kWindow) << 5 | (kUnitMost - m)) << 10 |
            (kMaxSize - min(size, kMaxSize));
        count[u] = m;
        key[u] = top << (49 - windowBits) | h >> (15 + windowBits);
        iota[u] = u;
    }
}

template <class K>
__device__ __forceinline__ int lower_bound(const K *a, int n, K v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1; else hi = mid;
    }
    return lo;
}
template <class K>
__device__ __forceinline__ int upper_bound(const K *a, int n, K v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a[mid] <= v) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Per unit in key order its segment -- the window, and 0: one of the full 32s of its run of equal
// keys, 1: left over, 2: a list longer than kUnitList -- and for the last two the part of the
// window it comes from.
__global__ void __launch_bounds__(256) k_unit_segments(const unsigned long long *key,
                                                       const int *unit, int nu, int windowBits,
                                                       unsigned *segment) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < nu; p += gridDim.x * blockDim.x) {
        const unsigned long long k = key[p];
        const int lo = lower_bound(key, nu, k), run = upper_bound(key, nu, k) - lo;
        const unsigned window = (unsigned)(k >> (63 - windowBits) >> 1);
        const int size = kMaxSize - (int)(k >> (49 - windowBits) & kMaxSize);
        const unsigned kind = size > kUnitList ? 2 : p - lo >= run / 32 * 32;
        const unsigned part = kind ? unit[p] % kWindow / (kWindow >> kPartBits) : 0;
        segment[p] = (window << 2 | kind) << kPartBits | part;
    }
}

// flag[p] = 1 where a slice starts: every 32 units of a segment.
__global__ void __launch_bounds__(256) k_unit_slices(const unsigned *segment, int nu, int *flag) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p <= nu; p += gridDim.x * blockDim.x)
        flag[p] = p < nu &&
                  (p - lower_bound(segment, nu, segment[p] >> kPartBits << kPartBits)) % 32 == 0;
}

// One warp per slice: the first of its units, which gives its place in the order of slices.  In
// the last fifth the slices that hold their weights once stand behind the others: they take the
// least time, and what is claimed last should.
__global__ void __launch_bounds__(256) k_unit_places(const int *firstOf, const int *unit,
                                                     const unsigned *segment, int ns, int nu,
                                                     unsigned *key, int *iota) {
    const int lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < ns; s += warps) {
        const int p = firstOf[s] + lane;
        unsigned k =
            __reduce_min_sync(kFull, p < firstOf[s + 1] ? (unsigned)unit[p] : 0xffffffffu);
        const bool uniform = (segment[firstOf[s]] >> kPartBits & 3) == 0;
        if (uniform && k >= (unsigned)(nu - nu / 5)) k += (unsigned)nu;
        if (lane == 0) key[s] = k, iota[s] = s;
    }
}

struct Slices {
    Csr c;
    int numSlices;
    const int *at;            // slice in the order of positions that stands here
    const int *firstOf;       // first unit position of each of those (+ end)
    const unsigned *segment;  // per position
    const int *unit;          // per position
    const int *pos, *count;   // per unit
    const int *order;
    const long long *start;   // blob offset / 128 (fill)
    long long *bytes;         // blob size / 128 (size)
    unsigned long long *shared;  // stencils of uniform slices
    int4 *slice;
    char *blob;
};

// The lane's unit of slice s: its stencils (0: none), its entries and its first position.
struct Unit {
    int m = 0, n = 0, i = 0;
    bool on;
    __device__ __forceinline__ Unit(const Slices &a, int s, int lane) {
        const int p = a.firstOf[a.at[s]] + lane;
        on = p < a.firstOf[a.at[s] + 1];
        if (on) {
            const int u = a.unit[p];
            m = a.count[u];
            i = a.pos[u];
            n = a.c.sizes[a.order[i]];
        }
    }
};

__device__ __forceinline__ int padded(int n) { return n > 4 ? (n + 3) & ~3 : 4; }

// One warp per slice: n, m, whether its 32 units really have the same weights, its size.
__global__ void __launch_bounds__(256) k_unit_sizes(const Slices a, int4 *meta) {
    const int lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < a.numSlices; s += warps) {
        const Unit u(a, s, lane);
        const int m = (int)__reduce_max_sync(kFull, (unsigned)u.m);
        const int n = (int)__reduce_max_sync(kFull, (unsigned)u.n);
        const unsigned kind = a.segment[a.firstOf[a.at[s]]] >> kPartBits & 3;
        bool same = __all_sync(kFull, kind == 0 && u.m == m && u.n == n);
        for (int k = 0; same && k < m; ++k) {  // the same for all lanes: uniform loops
            const float *w = a.c.weights + a.c.offsets[a.order[u.i + k]];
            bool equal = true;
            for (int j = 0; j < n; ++j) {
                const int v = __float_as_int(w[j]);
                equal = equal && v == __shfl_sync(kFull, v, 0);
            }
            same = __all_sync(kFull, equal);
        }
        if (lane == 0) {
            const long long w = (long long)m * padded(n), head = m + (long long)n;
            meta[s] = make_int4(0, n, m | (same ? 256 : 0), 0);
            a.bytes[s] = same ? head + (w + 31) / 32 : head + 1 + w;
            if (same) atomicAdd(a.shared, 32ull * m);
        }
    }
}

// One warp per slice: its blob and its descriptor.
__global__ void __launch_bounds__(256) k_unit_fill(const Slices a, const int4 *meta) {
    const int lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < a.numSlices; s += warps) {
        const int4 d = meta[s];
        const int m = d.z & 0xff, n = d.y, n4 = padded(n);
        const bool uni = (d.z & 256) != 0;
        const int o = (int)a.start[s];
        if (lane == 0)
            a.slice[s] = make_int4(o, n, d.z, uni ? (int)a.bytes[s] : m + 1 + n);
        const Unit u(a, s, lane);
        int *rows = reinterpret_cast<int *>(a.blob + (size_t)o * 128);
        for (int k = 0; k < m; ++k) rows[32 * k + lane] = k < u.m ? a.order[u.i + k] : -1;
        int *idx = rows + 32 * m;
        if (!uni) {
            idx[lane] = u.n;
            idx += 32;
        }
        const int *src = u.on ? a.c.indices + a.c.offsets[a.order[u.i]] : nullptr;
        for (int j = 0; j < n; ++j) idx[32 * (size_t)j + lane] = j < u.n ? src[j] : 0;
        float *w = reinterpret_cast<float *>(idx + 32 * (size_t)n);
        if (uni) {
            const int i = __shfl_sync(kFull, u.i, 0);
            for (int k = lane; k < (m * n4 + 31) / 32 * 32; k += 32) {
                const int st = k / n4, j = k % n4;
                w[k] = st < m && j < n ? a.c.weights[a.c.offsets[a.order[i + st]] + j] : 0.0f;
            }
        } else {
            for (int k = 0; k < m; ++k) {
                const float *x = k < u.m ? a.c.weights + a.c.offsets[a.order[u.i + k]] : nullptr;
                float *to = w + (size_t)(lane / 8 * m + k) * n4 * 8 + lane % 8 * 4;
                for (int j = 0; j < n4; ++j)
                    to[(size_t)(j / 4) * 32 + j % 4] = x && j < u.n ? x[j] : 0.0f;
            }
        }
    }
}

// Stream-ordered temporaries, released when the build returns, and the first failure: what comes
// behind one works on nothing, so the steps that write by what an earlier one computed are not
// queued any more.
struct Temps {
    cudaStream_t s;
    const char *who;
    void *p[32] = {};
    int status = GB300_OK;
    bool failed() const { return status != GB300_OK; }
    bool check(cudaError_t e) {
        if (!failed()) status = check_cuda(e, who);
        return !failed();
    }
    template <class T>
    T *get(size_t count) {
        void **slot = p;
        while (slot < p + 32 && *slot) ++slot;
        if (!failed() && slot == p + 32) status = fail(GB300_ERR_CUDA, "%s: temporaries", who);
        if (failed()) return nullptr;
        status = scratch_alloc(slot, std::max<size_t>(count * sizeof(T), 16), s, who);
        if (failed()) *slot = nullptr;
        return (T *)*slot;
    }
    void drop(void *q) {
        for (void *&x : p)
            if (x && x == q) scratch_free(q, s), x = nullptr;
    }
    ~Temps() {
        for (void *x : p) scratch_free(x, s);
    }
};

}  // namespace

int build_units(int n, const int *sizes, const int *offsets, const int *indices,
                const float *weights, cudaStream_t s, UnitTable &t, void *owned[2],
                const char *who) {
    t = UnitTable{};
    for (int k = 0; k < 2; ++k) owned[k] = nullptr;
    if (n <= 0 || n == INT_MAX) return n <= 0 ? ok() : GB300_ERR_UNSUPPORTED;
    typedef unsigned long long u64;
    const Csr c{sizes, offsets, indices, weights};
    Temps tmp{s, who};
    auto launched = [&] {
        count_launch();
        tmp.check(cudaGetLastError());
    };
    auto read = [&](auto *host, const auto *dev) {
        if (!tmp.failed() &&
            tmp.check(cudaMemcpyAsync(host, dev, sizeof(*host), cudaMemcpyDeviceToHost, s)))
            tmp.check(cudaStreamSynchronize(s));
        return tmp.status;
    };
    auto sort = [&](auto *kin, auto *kout, int *vin, int *vout, int count, int bits) {
        size_t bytes = 0;
        if (tmp.failed() || !tmp.check(cub::DeviceRadixSort::SortPairs(
                                nullptr, bytes, kin, kout, vin, vout, count, 0, bits, s)))
            return;
        void *q = tmp.get<char>(bytes);
        if (!q) return;
        tmp.check(cub::DeviceRadixSort::SortPairs(q, bytes, kin, kout, vin, vout, count, 0, bits,
                                                  s));
        count_launch();
        tmp.drop(q);
    };
    auto scan = [&](auto *in, auto *out, int count) {  // exclusive sum
        size_t bytes = 0;
        if (tmp.failed() ||
            !tmp.check(cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, count, s)))
            return;
        void *q = tmp.get<char>(bytes);
        if (!q) return;
        tmp.check(cub::DeviceScan::ExclusiveSum(q, bytes, in, out, count, s));
        count_launch();
        tmp.drop(q);
    };
    // Larger units read fewer source rows and hold fewer index lists; smaller ones make more
    // slices, which a small table lacks, and wait for fewer weights where slices are not uniform.
    // us with 8 and 16: level 3 of quads, 8-wide rows, 0.3 M stencils 8.8 and 11.8, 2.1 M 34.9
    // and 33.0, 4.3 M 62 and 57, 5.2 M 76 and 68, 8.6 M 120 and 104 (12-wide 227 and 240, xyz 122 and
    // 132); level 4, 8.6 M 123 and 120; irregular tables, 8-wide, 0.65 M 17.7 and 14.7, 1.9 M 42.8
    // and 46.1, 4.1 M 81 and 87, 8.5 M 156 and 169; Loop, level 3, 1.3 M 27.6 and 33.2, 8.0 M 139 and 136.
    const int most = n >= (4 << 20) ? kUnitMost : kUnitMost / 2;

    // stencils in locality order, equal lists together
    u64 *hashW = tmp.get<u64>(n), *key = tmp.get<u64>(n), *key2 = tmp.get<u64>(n);
    int *iota = tmp.get<int>(n), *order = tmp.get<int>(n);
    if (tmp.failed()) return tmp.status;
    k_unit_keys<<<grid_of(n, 256), 256, 0, s>>>(c, n, key, hashW, iota);
    launched();
    sort(key, key2, iota, order, n, 64);
    int *flag = tmp.get<int>((size_t)n + 1), *group = tmp.get<int>((size_t)n + 1);
    int *groupAt = tmp.get<int>((size_t)n + 1);
    if (tmp.failed()) return tmp.status;
    k_unit_heads<<<grid_of(n + 1LL, 256), 256, 0, s>>>(c, n, key2, order, flag);
    launched();
    scan(flag, group, n + 1);
    if (tmp.failed()) return tmp.status;
    k_unit_firsts<<<grid_of(n, 256), 256, 0, s>>>(group, n, groupAt);
    launched();
    tmp.drop(key);
    tmp.drop(key2);
    tmp.drop(iota);
    // units
    int *id = tmp.get<int>((size_t)n + 1);
    if (tmp.failed()) return tmp.status;
    k_unit_flags<<<grid_of(n + 1LL, 256), 256, 0, s>>>(c, n, most, order, group, groupAt, flag);
    launched();
    scan(flag, id, n + 1);
    if (tmp.failed()) return tmp.status;
    int *pos = groupAt;  // the groups are done with
    k_unit_firsts<<<grid_of(n, 256), 256, 0, s>>>(id, n, pos);
    launched();
    int nu = 0;
    int st = read(&nu, id + n);
    if (st != GB300_OK) return st;
    if (nu > n / 2) return GB300_ERR_UNSUPPORTED;
    int windowBits = 0;
    while (windowBits < 20 && (nu - 1) / kWindow >> windowBits) ++windowBits;
    int *count = tmp.get<int>(nu);
    u64 *ukey = tmp.get<u64>(nu), *ukey2 = tmp.get<u64>(nu);
    int *uiota = tmp.get<int>(nu), *unit = tmp.get<int>(nu);
    unsigned *seg = tmp.get<unsigned>(nu), *seg2 = tmp.get<unsigned>(nu);
    if (tmp.failed()) return tmp.status;
    k_unit_units<<<grid_of(nu, 256), 256, 0, s>>>(c, n, windowBits, order, id, pos, hashW, count,
                                                  ukey, uiota);
    launched();
    sort(ukey, ukey2, uiota, unit, nu, 64);
    if (tmp.failed()) return tmp.status;
    k_unit_segments<<<grid_of(nu, 256), 256, 0, s>>>(ukey2, unit, nu, windowBits, seg);
    launched();
    sort(seg, seg2, unit, uiota, nu, windowBits + 2 + kPartBits);  // stable: key order kept
    unit = uiota;
    // slices
    int *sflag = tmp.get<int>((size_t)nu + 1), *sid = tmp.get<int>((size_t)nu + 1);
    if (tmp.failed()) return tmp.status;
    k_unit_slices<<<grid_of(nu + 1LL, 256), 256, 0, s>>>(seg2, nu, sflag);
    launched();
    scan(sflag, sid, nu + 1);
    if (tmp.failed()) return tmp.status;
    int ns = 0;
    if ((st = read(&ns, sid + nu)) != GB300_OK) return st;
    int *firstOf = tmp.get<int>((size_t)ns + 1);
    long long *bytes = tmp.get<long long>((size_t)ns + 1), *start = tmp.get<long long>((size_t)ns + 1);
    int4 *meta = tmp.get<int4>(ns);
    if (tmp.failed()) return tmp.status;
    k_unit_firsts<<<grid_of(nu, 256), 256, 0, s>>>(sid, nu, firstOf);
    launched();
    unsigned *skey = tmp.get<unsigned>(ns), *skey2 = tmp.get<unsigned>(ns);
    int *siota = tmp.get<int>(ns), *at = tmp.get<int>(ns);
    if (tmp.failed()) return tmp.status;
    k_unit_places<<<grid_of((long long)ns * 32, 256), 256, 0, s>>>(firstOf, unit, seg2, ns, nu, skey,
                                                                     siota);
    launched();
    sort(skey, skey2, siota, at, ns, 32);
    if (tmp.failed()) return tmp.status;
    u64 *shared = tmp.get<u64>(1);
    if (tmp.failed()) return tmp.status;
    Slices a{c,     ns,    at,      firstOf, seg2,    unit, pos, count,
             order, start, bytes, shared,  nullptr, nullptr};
    if (!tmp.check(cudaMemsetAsync(bytes + ns, 0, 8, s)) ||
        !tmp.check(cudaMemsetAsync(shared, 0, 8, s)))
        return tmp.status;
    k_unit_sizes<<<grid_of((long long)ns * 32, 256), 256, 0, s>>>(a, meta);
    launched();
    scan(bytes, start, ns + 1);
    if (tmp.failed()) return tmp.status;
    long long total = 0;
    u64 sharing = 0;
    if ((st = read(&total, start + ns)) != GB300_OK || (st = read(&sharing, shared)) != GB300_OK)
        return st;
    if (total > INT_MAX) return GB300_ERR_UNSUPPORTED;
    auto fail_all = [&](int code) {
        for (int k = 0; k < 2; ++k)
            if (owned[k]) cudaFree(owned[k]), owned[k] = nullptr;
        return code;
    };
    if (!tmp.check(cudaMalloc(&owned[0], (size_t)ns * sizeof(int4))) ||
        !tmp.check(cudaMalloc(&owned[1], (size_t)total * 128))) {
        cudaGetLastError();
        return fail_all(tmp.status);
    }
    a.slice = (int4 *)owned[0];
    a.blob = (char *)owned[1];
    k_unit_fill<<<grid_of((long long)ns * 32, 256), 256, 0, s>>>(a, meta);
    launched();
    if (tmp.failed() || !tmp.check(cudaStreamSynchronize(s))) return fail_all(tmp.status);
    t.numSlices = ns;
    t.regular = sharing >= (u64)n / 2;
    t.numStencils = n;
    t.slice = a.slice;
    t.blob = a.blob;
    return ok();
}

}  // namespace gb300
