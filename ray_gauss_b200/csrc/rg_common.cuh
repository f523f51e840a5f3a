// Shared device definitions of the B200 ray-caster engine.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "raygauss_b200.h"

namespace rg {

// Reference constants (optix_raycasting/cuda_train/forward/gaussians_aabb.h:2-5).
constexpr int kBuf = 8;                 // samples per slab
constexpr float kDt = 0.0025f;          // sample spacing
constexpr float kSlab = kDt * kBuf;     // slab length (0.02)
constexpr float kTeps = 0.003f;         // early-exit transmittance
constexpr float kSigThr = 0.1f;         // per-sample density threshold

constexpr int kWarp = 32;
constexpr int kTileW = 8;               // a warp renders an 8x4 pixel tile
constexpr int kTileH = 4;
// ... or, with two or four slabs of a ray side by side (split; parity arithmetic), a 4x4 or 4x2 one
__host__ __device__ constexpr int tile_w(int split) { return split == 1 ? kTileW : 4; }
__host__ __device__ constexpr int tile_h(int split) { return split == 4 ? 2 : 4; }
// The splits of a launch, for scenes whose box is short and long (render_split).
struct SplitPair {
    int near, far;
};
constexpr float kFarBox = 20.f;         // diagonal of a long box: 1000 slabs
constexpr int kMaxChunk = 255;          // slabs per traversal chunk (slab ranges are bytes)
constexpr int kStack = 256;             // warp traversal stack depth (up to 31 pushes per wide node on the path)

// Device status block (mirrors rg_status) + work counters.
struct DevStatus {
    unsigned long long hit_pairs;
    unsigned long long slabs;
    unsigned long long slab_cap_exceeded;
    unsigned long long list_passes;
    unsigned long long chunk_splits;
    unsigned long long stack_overflows;
    unsigned long long watchdog_trips;
    unsigned long long nonfinite_inputs;
    unsigned long long traversals;        // warp-level BVH traversals
    unsigned long long node_visits;       // warp-level internal-node visits
    unsigned long long leaf_tests;        // warp-level leaf (ellipsoid) tests
    unsigned long long list_entries;      // hit-list entries appended
    unsigned long long slab_steps;        // warp-level slab iterations with at least one entry
    unsigned long long entry_slabs;       // warp-level (entry, slab) evaluations
    unsigned long long replayed_chunks;   // backward chunks whose list came from the forward record
    unsigned long long record_overflows;  // tiles whose record did not fit the arena
};

// Per-launch view table computed on the device from the camera array (no host sync).
struct ViewTable {
    int n_views;
    int split;              // slabs side by side (1, 2 or 4): the kernels of another split return at once
    int total_tiles;
    long long total_rays;
    int tile_prefix[65];
    long long ray_prefix[65];
};
constexpr int kMaxViews = 64;

// ---- small float3 helpers (own definitions) -------------------------------------------------
__host__ __device__ __forceinline__ float3 f3(float x, float y, float z) { return make_float3(x, y, z); }
__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator*(float3 a, float s) { return f3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float dot3(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

// Ordered-int encoding so that float min/max can use integer atomics.
__device__ __forceinline__ int f2ord(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__host__ __device__ __forceinline__ float ord2f(int i) {
#ifdef __CUDA_ARCH__
    return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff);
#else
    union { int i; float f; } u;
    u.i = i >= 0 ? i : i ^ 0x7fffffff;
    return u.f;
#endif
}

__device__ __forceinline__ float load_param(const void* p, long long i, int storage) {
    if (storage == RG_STORAGE_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
    return reinterpret_cast<const float*>(p)[i];
}

// 2^x with the SFU (one MUFU.EX2); inputs here are <= 0 and the result may flush to zero.
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Three-input min / max (one instruction on sm_100)
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// SFU base-2 logarithm (x <= 0 gives -inf / NaN, which fail every threshold comparison)
__device__ __forceinline__ float sqrt_approx(float x) {
    float y;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_approx(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two FP32 values in one 64-bit register pair: the packed instructions (f32x2, sm_100) do two IEEE
// round-to-nearest operations per issue slot, and each half rounds like the scalar operation.
using f2 = unsigned long long;
__device__ __forceinline__ f2 pk(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ f2 dup2(float a) { return pk(a, a); }
__device__ __forceinline__ float lo2(f2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi2(f2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// The product as a fused multiply-add of `nz`, a pair of -0 that the assembler cannot see through (a
// kernel argument): the same value, and never contracted with a following addition, which a packed
// multiplication is even with its rounding given.
__device__ __forceinline__ f2 mul2_rn(f2 a, f2 b, f2 nz) { return fma2(a, b, nz); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// Half h (0 or 1, a constant after unrolling) of a pair, read and replaced.
__device__ __forceinline__ float half2(f2 v, int h) { return h ? hi2(v) : lo2(v); }
__device__ __forceinline__ f2 with_half2(f2 v, int h, float x) { return h ? pk(lo2(v), x) : pk(x, hi2(v)); }

// tea<4>(v0, v1) seeding and LCG draws of the reference RNG (forward/gaussians_aabb.h:63-94).
__device__ __forceinline__ unsigned tea4(unsigned v0, unsigned v1) {
    unsigned s0 = 0;
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        s0 += 0x9e3779b9u;
        v0 += ((v1 << 4) + 0xa341316cu) ^ (v1 + s0) ^ ((v1 >> 5) + 0xc8013ea4u);
        v1 += ((v0 << 4) + 0xad90777du) ^ (v0 + s0) ^ ((v0 >> 5) + 0x7e95761eu);
    }
    return v0;
}
__device__ __forceinline__ float lcg_rnd(unsigned& prev) {
    prev = 1664525u * prev + 1013904223u;
    return (float)(prev & 0x00FFFFFFu) / (float)0x01000000;
}

// Leaf record (leaf order), 64 bytes: {mu.xyz, density}, {M row 0, k}, {M row 1, log2(density)},
// {M row 2, 1 / density} where m = M (x - mu) = S^-1 R^T (x - mu) and k = 1/sqrt(log((density/0.1)^2))
// scales M to the threshold ellipsoid (forward/gaussians_aabb.cu:341-357); the log and reciprocal
// (SFU approximations) serve the fast sample arithmetic.
struct __align__(16) LeafRec {
    float4 a, r0, r1, r2;
};

// Threshold-ellipsoid conic of a leaf in the reference's arithmetic, 48 bytes: the rotation columns
// scaled by 1/(s_j sqrt(log((density/0.1)^2))) (forward/gaussians_aabb.cu:341-357), used by the
// exact ray/ellipsoid interval test of the parity arithmetic; u.w holds sqrt(log((density/0.1)^2)),
// the factor the inference programs scale their sample conic back with.
struct __align__(16) LeafIS {
    float4 u, v, w;
};

// Per-Gaussian pre-pass output in Gaussian order (gathered into leaf order by the BVH build).
struct __align__(16) GaussRec {
    LeafRec s;
    LeafIS is;
};

// Wide traversal nodes of up to kWideSlots children (one per lane), collapsed from the binary tree
// (k_refit decides which binary nodes they are), stored as consecutive slots in leaf order.  A slot
// holds the child's box, its id and the last leaf of its subtree (the multi-pass cursor test).  The id
// of a leaf child is ~leaf (< 0); that of a wide child holds the child's own slots, first slot |
// (count - 1) << kWideCountShift (>= 0), so a visit needs no other load.  32 bytes, one 256-bit load
// per lane.  A leaf or a wide node but the root is one slot: at most 2n.
constexpr int kWideSlots = 32;
constexpr int kWideCountShift = 26;                       // first slot < 2^26: at most 2^25 Gaussians
constexpr long long kMaxGaussians = 1ll << 25;
__host__ __device__ __forceinline__ int wide_pack(int first, int count) {
    return first | ((count - 1) << kWideCountShift);
}
struct __align__(32) WideSlot {
    float lo[3], hi[3];
    int id;
    int range_hi;
};

// BVH internal node, 64 bytes: child boxes, child ids (>= 0 internal, < 0 leaf ~id),
// split position and last leaf of the node's range.
struct __align__(32) Node {   // 32-byte aligned for 256-bit loads
    float4 n0;  // lbox lo.xyz, lbox hi.x
    float4 n1;  // lbox hi.yz, rbox lo.xy
    float4 n2;  // rbox lo.z, rbox hi.xyz
    int4 n3;    // left, right, split, range_hi
};

}  // namespace rg
