// Mean squared distance to the 3 nearest neighbours of every point: the initial scale of a point
// cloud without scales (classes/point_cloud.py:374-378 -> distCUDA2 of the simple-knn extension,
// submodules/simple-knn/spatial.cu:14-25 and simple_knn.cu:126-221).
//
// The extension's result is exact: for point i, (d0 + d1 + d2) / 3 with d0 <= d1 <= d2 the three
// smallest squared distances |p_j - p_i|^2 (j != i), each evaluated as dx*dx + dy*dy + dz*dz with
// the multiply-adds contracted, the sum left to right; fewer than three other points leave FLT_MAX
// entries (two neighbours: about FLT_MAX / 3; one or none: +inf).  Its Morton boxes only prune the
// search.
//
// This engine's search: points sorted by a 48-bit Morton code (k_knn_bounds, k_knn_morton, CUB radix
// sort) and copied in that order, boxes of kBox consecutive points and groups of kGroup boxes
// (k_knn_boxes), then one warp per 32 consecutive points (k_knn_query): the warp's own box and its
// neighbours first, then groups and their boxes, nearest first, as long as their distance to the warp's
// query box is at most the warp's largest third-best distance; a box that some lane's own point is
// near enough to is staged in shared memory and read by all 32 queries.
//
// Bound by instruction issue in dense regions and by the warps of sparse ones, whose 32 points lie far
// apart: they decide when the launch ends, and prune the sooner the nearer boxes come first.  200k
// points (80 % in a ball, 20 % out to 50 times its radius): 1.11 ms before the finer code (ten bits an
// axis left hundreds of points of a dense core in one cell), the nearest-first order, the groups and the
// points in sorted order, 0.50 ms now; a million 5.85 and 1.47 ms.
#include <cfloat>
#include <cstdint>
#include <type_traits>

#include <cub/device/device_radix_sort.cuh>

#include "rg_common.cuh"

namespace {

using rg::f2ord;
using rg::ord2f;

constexpr int kBox = 32;          // sorted points per box: one per lane, and a warp's queries
constexpr int kGroup = 32;        // boxes per group: one per lane
constexpr int kNear = 2;          // boxes on each side of the warp's own box scanned first
constexpr int kMortonBits = 16;   // per axis

struct KnnWs {
    int* bounds;                  // 6 ordered ints: scene min, max
    unsigned long long* keys_in;
    unsigned long long* keys_out;
    int* vals_in;
    int* vals_out;                // sorted point ids
    float4* pts;                  // points in sorted order
    float4* box_lo;
    float4* box_hi;
    float4* group_lo;
    float4* group_hi;
    void* sort_temp;
    size_t sort_bytes;
};

size_t a256(size_t x) { return (x + 255) & ~size_t(255); }

size_t sort_bytes(long long n) {
    size_t b = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, b, (const unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                    (const int*)nullptr, (int*)nullptr, (int)n, 0, 3 * kMortonBits);
    return b;
}

long long n_boxes(long long n) { return (n + kBox - 1) / kBox; }
long long n_groups(long long n) { return (n_boxes(n) + kGroup - 1) / kGroup; }

KnnWs carve(void* base, long long n, size_t* end = nullptr) {
    uintptr_t p = (reinterpret_cast<uintptr_t>(base) + 255) & ~uintptr_t(255);
    auto take = [&](auto*& q, size_t count) {
        q = reinterpret_cast<std::remove_reference_t<decltype(q)>>(p);
        p += a256(sizeof(*q) * count);
    };
    KnnWs w;
    take(w.bounds, 6);
    take(w.keys_in, n);
    take(w.keys_out, n);
    take(w.vals_in, n);
    take(w.vals_out, n);
    take(w.pts, n);
    take(w.box_lo, n_boxes(n));
    take(w.box_hi, n_boxes(n));
    take(w.group_lo, n_groups(n));
    take(w.group_hi, n_groups(n));
    w.sort_temp = reinterpret_cast<void*>(p);
    w.sort_bytes = sort_bytes(n);
    if (end) *end = p + a256(w.sort_bytes);
    return w;
}

size_t ws_bytes(long long n) {
    size_t end = 0;
    carve(nullptr, n, &end);
    return end + 256;             // the base is rounded up to 256 bytes
}

__global__ void k_knn_init_bounds(int* b) {
    if (threadIdx.x < 3) b[threadIdx.x] = f2ord(INFINITY);
    else if (threadIdx.x < 6) b[threadIdx.x] = f2ord(-INFINITY);
}

__device__ __forceinline__ float warp_min(float v) {
    for (int o = 16; o; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
    for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Grid-stride, a handful of blocks per SM: the six atomics of a block are on the same addresses.
__global__ void __launch_bounds__(256) k_knn_bounds(long long n, const float* __restrict__ p, int* __restrict__ b) {
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += 256ll * gridDim.x) {
        for (int a = 0; a < 3; ++a) {
            const float v = p[3 * i + a];
            lo[a] = fminf(lo[a], v);
            hi[a] = fmaxf(hi[a], v);
        }
    }
    __shared__ float red[6][8];
    for (int a = 0; a < 3; ++a) {
        const float l = warp_min(lo[a]), h = warp_max(hi[a]);
        if ((threadIdx.x & 31) == 0) {
            red[a][threadIdx.x >> 5] = l;
            red[3 + a][threadIdx.x >> 5] = h;
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        float v = red[threadIdx.x][0];
        for (int w = 1; w < 8; ++w)
            v = threadIdx.x < 3 ? fminf(v, red[threadIdx.x][w]) : fmaxf(v, red[threadIdx.x][w]);
        if (threadIdx.x < 3) atomicMin(b + threadIdx.x, f2ord(v));
        else atomicMax(b + threadIdx.x, f2ord(v));
    }
}

// Spread the low 16 bits of v so that bit i lands at bit 3i.
__device__ __forceinline__ unsigned long long spread16(unsigned long long v) {
    v = (v | (v << 32)) & 0x1f00000000ffffull;
    v = (v | (v << 16)) & 0x1f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

__global__ void __launch_bounds__(256) k_knn_morton(long long n, const float* __restrict__ p,
                                                    const int* __restrict__ b, unsigned long long* __restrict__ keys,
                                                    int* __restrict__ vals) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    constexpr float top = (float)((1 << kMortonBits) - 1);
    unsigned q[3];
    for (int a = 0; a < 3; ++a) {
        const float lo = ord2f(b[a]), hi = ord2f(b[3 + a]);
        const float u = hi > lo ? (p[3 * i + a] - lo) / (hi - lo) : 0.f;
        q[a] = (unsigned)fminf(fmaxf(u * top, 0.f), top);
    }
    keys[i] = spread16(q[0]) | (spread16(q[1]) << 1) | (spread16(q[2]) << 2);
    vals[i] = (int)i;
}

// A block per group: its points in sorted order, its boxes (a warp per box, four in turn) and their union.
__global__ void __launch_bounds__(256) k_knn_boxes(long long n, const float* __restrict__ p,
                                                   const int* __restrict__ sorted, float4* __restrict__ pts,
                                                   float4* __restrict__ blo, float4* __restrict__ bhi,
                                                   float4* __restrict__ glo, float4* __restrict__ ghi) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float g[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
    for (int j = warp; j < kGroup; j += 8) {
        const long long bx = (long long)blockIdx.x * kGroup + j;
        if (bx * kBox >= n) break;
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        const long long i = bx * kBox + lane;
        if (i < n) {
            const long long s = sorted[i];
            const float x[3] = {p[3 * s], p[3 * s + 1], p[3 * s + 2]};
            pts[i] = make_float4(x[0], x[1], x[2], 0.f);
            for (int a = 0; a < 3; ++a) {
                lo[a] = fminf(lo[a], x[a]);
                hi[a] = fmaxf(hi[a], x[a]);
            }
        }
        for (int a = 0; a < 3; ++a) {
            lo[a] = warp_min(lo[a]);
            hi[a] = warp_max(hi[a]);
            g[a] = fminf(g[a], lo[a]);
            g[3 + a] = fmaxf(g[3 + a], hi[a]);
        }
        if (lane == 0) {
            blo[bx] = make_float4(lo[0], lo[1], lo[2], 0.f);
            bhi[bx] = make_float4(hi[0], hi[1], hi[2], 0.f);
        }
    }
    __shared__ float red[6][8];
    if (lane == 0)
        for (int a = 0; a < 6; ++a) red[a][warp] = g[a];
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w)
            for (int a = 0; a < 6; ++a) g[a] = a < 3 ? fminf(g[a], red[a][w]) : fmaxf(g[a], red[a][w]);
        glo[blockIdx.x] = make_float4(g[0], g[1], g[2], 0.f);
        ghi[blockIdx.x] = make_float4(g[3], g[4], g[5], 0.f);
    }
}

__device__ __forceinline__ void insert3(float d, float (&best)[3]) {
    // updateKBest<3>: keep the three smallest in ascending order
    for (int j = 0; j < 3; ++j) {
        if (best[j] > d) {
            const float t = best[j];
            best[j] = d;
            d = t;
        }
    }
}

// The distances from this lane's query to the kBox points of box `bx`, staged in `stage` (the end of
// the last box at infinity).
__device__ __forceinline__ void scan_box(long long n, const float4* __restrict__ pts, float4* stage, long long bx,
                                         long long me, float3 q, float (&best)[3], int lane) {
    __syncwarp();
    const long long i = bx * kBox + lane;
    stage[lane] = i < n ? pts[i] : make_float4(INFINITY, INFINITY, INFINITY, 0.f);
    __syncwarp();
    const long long self = me - bx * kBox;            // this lane's own point, when it is in the box
#pragma unroll 8
    for (int j = 0; j < kBox; ++j) {
        const float4 v = stage[j];
        const float dx = v.x - q.x, dy = v.y - q.y, dz = v.z - q.z;
        const float d = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
        if (d < best[2] && j != self) insert3(d, best);
    }
}

// Squared gap between two boxes, a little less than it is (a relative margin keeps its rounding from
// dropping a point at the tie distance).
__device__ __forceinline__ float gap2(float4 l, float4 h, const float (&ql)[3], const float (&qh)[3]) {
    const float gx = fmaxf(0.f, fmaxf(l.x - qh[0], ql[0] - h.x));
    const float gy = fmaxf(0.f, fmaxf(l.y - qh[1], ql[1] - h.y));
    const float gz = fmaxf(0.f, fmaxf(l.z - qh[2], ql[2] - h.z));
    return __fmul_rn(gx * gx + gy * gy + gz * gz, 0.999999f);
}

__global__ void __launch_bounds__(128) k_knn_query(long long n, const float4* __restrict__ pts,
                                                   const int* __restrict__ sorted, const float4* __restrict__ blo,
                                                   const float4* __restrict__ bhi, const float4* __restrict__ glo,
                                                   const float4* __restrict__ ghi, float* __restrict__ out) {
    __shared__ float4 stage_all[4][kBox];
    float4* const stage = stage_all[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long me = warp * 32 + lane;
    if (warp * 32 >= n) return;                       // whole warp past the end
    const bool active = me < n;
    const long long nb = (n + kBox - 1) / kBox, ng = (nb + kGroup - 1) / kGroup;
    float3 q = make_float3(0.f, 0.f, 0.f);
    if (active) {
        const float4 v = pts[me];
        q = make_float3(v.x, v.y, v.z);
    }
    // the warp's query box
    float ql[3] = {active ? q.x : INFINITY, active ? q.y : INFINITY, active ? q.z : INFINITY};
    float qh[3] = {active ? q.x : -INFINITY, active ? q.y : -INFINITY, active ? q.z : -INFINITY};
    const float own_lo[3] = {q.x, q.y, q.z};
    for (int a = 0; a < 3; ++a) {
        ql[a] = warp_min(ql[a]);
        qh[a] = warp_max(qh[a]);
    }
    float best[3] = {FLT_MAX, FLT_MAX, FLT_MAX};
    const long long own = warp;
    const long long n0 = own - kNear > 0 ? own - kNear : 0;
    const long long n1 = own + kNear < nb - 1 ? own + kNear : nb - 1;
    for (long long bx = n0; bx <= n1; ++bx) scan_box(n, pts, stage, bx, me, q, best, lane);
    // Every other box within the warp's largest third-best distance of the query box, nearest first: a
    // box (or a group) is left out only when clearly farther than every lane's third best.
    auto reach = [&]() {
        return __uint_as_float(__reduce_max_sync(0xffffffffu, active ? __float_as_uint(best[2]) : 0u));
    };
    // calls visit(lane) for the lanes' candidates by increasing gap, as far as the reach of the moment goes
    auto nearest_first = [&](bool in, float gap, auto visit) {
        unsigned key = in ? __float_as_uint(gap) : 0xffffffffu;
        while (true) {
            const unsigned k = __reduce_min_sync(0xffffffffu, key);
            if (k == 0xffffffffu || __uint_as_float(k) > reach()) break;
            const int j = __ffs(__ballot_sync(0xffffffffu, key == k)) - 1;
            if (lane == j) key = 0xffffffffu;
            visit(j);
        }
    };
    // whether some lane's own point is close enough to a box: the query box of a warp whose points straddle
    // a jump of the Morton curve can hold half the scene
    auto wanted = [&](float4 l, float4 h) {
        return __any_sync(0xffffffffu, active && !(gap2(l, h, own_lo, own_lo) > best[2]));
    };
    auto visit_group = [&](long long g) {
        if (!wanted(glo[g], ghi[g])) return;
        const long long b0 = g * kGroup, bx = b0 + lane;
        const bool in = bx < nb && (bx < n0 || bx > n1);
        const float4 l = in ? blo[bx] : make_float4(0.f, 0.f, 0.f, 0.f), h = in ? bhi[bx] : l;
        nearest_first(in, gap2(l, h, ql, qh), [&](int j) {
            if (wanted(blo[b0 + j], bhi[b0 + j])) scan_box(n, pts, stage, b0 + j, me, q, best, lane);
        });
    };
    // the warp's own group, then 32 groups at a time outwards from it
    const long long own_g = own / kGroup, nc = (ng + 31) / 32, own_c = own_g / 32;
    const long long far_c = own_c > nc - 1 - own_c ? own_c : nc - 1 - own_c;
    visit_group(own_g);
    for (long long k = 0; k <= 2 * far_c; ++k) {
        const long long c = k & 1 ? own_c + (k + 1) / 2 : own_c - k / 2;
        if (c < 0 || c >= nc) continue;
        const long long g = c * 32 + lane;
        const bool in = g < ng && g != own_g;
        const float4 l = in ? glo[g] : make_float4(0.f, 0.f, 0.f, 0.f), h = in ? ghi[g] : l;
        nearest_first(in, gap2(l, h, ql, qh), [&](int j) { visit_group(c * 32 + j); });
    }
    if (active) out[sorted[me]] = __fdiv_rn(__fadd_rn(__fadd_rn(best[0], best[1]), best[2]), 3.0f);
}

}  // namespace

extern "C" {

int rg_knn_workspace_bytes(int64_t n, uint64_t* bytes) {
    if (!bytes || n < 0 || n > INT32_MAX) return RG_ERR_INVALID_ARG;
    *bytes = ws_bytes(n);
    return RG_OK;
}

int rg_knn_mean_dist(const float* points, int64_t n, float* mean_dist, void* workspace, void* stream) {
    if (n < 0 || n > INT32_MAX || (n > 0 && (!points || !mean_dist || !workspace))) return RG_ERR_INVALID_ARG;
    if (n == 0) return RG_OK;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    KnnWs w = carve(workspace, n);
    const unsigned blocks = (unsigned)((n + 255) / 256);
    k_knn_init_bounds<<<1, 32, 0, s>>>(w.bounds);
    k_knn_bounds<<<blocks < 592u ? blocks : 592u, 256, 0, s>>>(n, points, w.bounds);
    k_knn_morton<<<blocks, 256, 0, s>>>(n, points, w.bounds, w.keys_in, w.vals_in);
    size_t bytes = w.sort_bytes;
    if (cub::DeviceRadixSort::SortPairs(w.sort_temp, bytes, w.keys_in, w.keys_out, w.vals_in, w.vals_out, (int)n, 0,
                                        3 * kMortonBits, s) != cudaSuccess)
        return RG_ERR_CUDA;
    k_knn_boxes<<<(unsigned)n_groups(n), 256, 0, s>>>(n, points, w.vals_out, w.pts, w.box_lo, w.box_hi, w.group_lo,
                                                      w.group_hi);
    const long long warps = (n + 31) / 32;
    k_knn_query<<<(unsigned)((warps + 3) / 4), 128, 0, s>>>(n, w.pts, w.vals_out, w.box_lo, w.box_hi, w.group_lo,
                                                            w.group_hi, mean_dist);
    return cudaGetLastError() == cudaSuccess ? RG_OK : RG_ERR_CUDA;
}

}  // extern "C"
