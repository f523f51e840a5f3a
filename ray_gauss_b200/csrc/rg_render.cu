// Persistent, warp-cooperative ray-casting kernels: forward (density/colour sampling, alpha
// compositing, early termination) and the recompute-based adjoint.
//
// Reference semantics (paths inside the reference project):
//   ray generation            optix_raycasting/cuda_train/forward/gaussians_aabb.cu:405-434
//   scene-box clip, slab loop :521-612 (slab = 8 samples x 0.0025 starting at the box entry,
//                             per-slab early-exit test T > 0.003, samples past the box exit in the
//                             last slab are still evaluated)
//   exact ellipsoid test      :324-402 (including its root-order behaviour for b <= 0)
//   sample buffers            :437-498, compositing :500-519
//   adjoint                   optix_raycasting/cuda_train/backward/gaussians_aabb.cu:505-775
//
// Design.  A warp owns an 8x4 pixel tile, or a part of one where it takes several slabs of a ray at a time
// (TileShape; in the fast arithmetic the warps of a tile then share its list); tiles of all views are pulled
// from one atomic work counter.  Each ray marches with the reference's slab sequence (tb += 0.02 in FP32);
// the warp advances in chunks of K slabs per ray (K adapts between 1 and 255: it grows while hits are sparse
// and shrinks in place when the hit list overflows).  For a chunk the warp traverses the wide BVH once for the packet of its rays' segments (one child slot per lane,
// tested with interval arithmetic over the rays' directions) with a warp-uniform stack.  Leaves wait until
// there are 32, are culled one per lane against the tile's ray cone, and the candidates take the exact
// ellipsoid test, all rays at a time.  A leaf that any ray hits is appended to a shared hit list with, per
// ray, the range of the chunk's slabs its interval covers (settled with the exact test where it decides).
// The list is consumed slab by slab: each lane evaluates only entries whose range holds its slab, reading the
// leaf record with a warp-uniform (broadcast) load.  A full list for a single slab is consumed in several
// passes (a leaf-index cursor skips the leaves already taken; DFS order visits leaves in increasing index),
// so no hit is dropped.
// The adjoint recomputes each slab's sample buffers, folds the compositing adjoint into three
// scalars per sample, evaluates each Gaussian's gradient per lane, reduces it across the warp with
// a transposed shuffle reduction (16 shuffles for 14 values) and issues one atomic per value.
//
// Sample arithmetic.  RG_MODE_PARITY evaluates samples, ray generation and compositing in the
// reference's operation order with IEEE round-to-nearest operations (no FMA contraction); when a
// sample's density*weight lies within a few ulps of the 0.1 threshold the weight is re-evaluated
// with a correctly rounded exponential so the threshold decision matches the FP32 reference
// arithmetic.  RG_MODE_FAST evaluates the 8 samples of a slab from the quadratic form of the
// Mahalanobis distance along the ray with the SFU exponential and accumulates the adjoint in
// moment form.
#include <algorithm>
#include <cstddef>

#include "rg_common.cuh"
#include "rg_exp.cuh"
#include "rg_kernels.h"

namespace rg {

constexpr int kWarpsPerBlock = 4;
constexpr unsigned kFull = 0xffffffffu;
constexpr int kMaxRounds = 1 << 20;        // chunk rounds per tile before the watchdog trips
constexpr float kNegHalfLog2e = -0.72134752044448170f;
constexpr float kLog2SigThr = -3.3219280948873623f;   // log2(0.1): per-sample density threshold
constexpr float kInvSlab = 50.0f;          // 1 / 0.02
constexpr int kExactChunk = 8;             // chunks up to this length use exact slab ranges
constexpr int kCounters = 9;               // per-warp counters: the WarpStats fields, hit pairs, slabs
#ifndef RG_DIRECT_ATOMIC_LANES
#define RG_DIRECT_ATOMIC_LANES 24  // up to this many contributing lanes add with float4 atomics directly
#endif
#ifndef RG_SPLIT_DIRECT_ATOMIC_LANES
// ... and on split tiles, whose lanes are few rays' slabs: a Gaussian near the camera gets 10^5 and more of
// them, and what is added alone to its large sum is lost below the sum's last bit (24 here: 3e-3 off on 4
// views at 1920x1080; 4: as exact as whole tiles at the sizes that are split)
#define RG_SPLIT_DIRECT_ATOMIC_LANES 4
#endif
constexpr unsigned kNoRecord = 0xffffffffu;     // hit-list record: no (next) chunk record
constexpr unsigned kRecordMulti = 0x80000000u;  // chunk consumed in several traversal passes
constexpr unsigned kRecordFailed = 0xfffffffeu; // the tile's last chunk did not fit the arena

// Rays and slabs of a warp.  SUB == 1: 32 rays (8x4 pixels), a slab at a time.  SUB == 2 or 4: 16 (4x4) or 8
// (4x2) rays, the lanes SUB r .. SUB r + SUB - 1 holding ray r's slabs k .. k + SUB - 1.  Their sums are
// independent; only transmittance and colour (in the adjoint: g . R) run through them in turn, by the same
// operations as slab after slab.  A Gaussian spans a few slabs, so a list entry is evaluated once for them
// all, for fewer rays: not many more evaluations in all, but a fraction of them in one tile's chain, and a
// launch of few tiles lasts as long as its slowest one.  render_split has the lines between them.
//   Parity arithmetic: a list holds each ray's exact slabs, so it does not matter which rays share it.  A warp
// is by itself, with a smaller tile; leaves are tested SUB at a time.
//   Fast arithmetic: a ray evaluates the slabs that any ray of its list covers, up to the chunk's end, and at
// a slab's edge a sample can round above the threshold outside the ray's own interval.  So the rays that
// share a list and a chunk stay those of the 8x4 tile: SUB warps are a team, which builds the tile's list
// together (TeamSmem) and then marches a part of its rays each.
template <int SUB>
struct TileShape {
    static constexpr int rays = 32 / SUB;
    static constexpr int w = tile_w(SUB), h = tile_h(SUB);
    static_assert(w * h == rays, "a ray per pixel");
};

// Warp hit-list layout.  Parity arithmetic keeps, per entry and ray, the exact range of the chunk's
// slabs the ray's interval covers (2 B per entry and ray); the fast arithmetic keeps only the mask of
// rays whose interval overlaps the chunk (4 B per entry) and lets those rays evaluate every slab of the
// entry's union range (samples outside the ray's interval fall outside the threshold ellipsoid and
// are masked out), which allows longer lists and so longer chunks in dense regions.
template <bool FAST, int SUB, int CAP>
struct WarpSmem {
    using Store = WarpSmem;                              // what lies in shared memory: one per warp
    static constexpr int kStores = kWarpsPerBlock;
    __device__ static WarpSmem& of(Store* s, int warp, int) { return s[warp]; }
    static constexpr int MB = FAST || SUB > 1 ? 4 : 2;   // slabs per entry-mask block (a multiple of SUB)
    static constexpr int NB = 64;                        // entry-mask blocks
    static constexpr int KM = MB == 4 ? 255 : 128;       // longest chunk (MB * NB, slab ranges are bytes)
    int ids[CAP];
    unsigned urng[CAP];                              // union of the lanes' slab ranges: lo | hi << 16
    unsigned lmask[FAST ? CAP : 1];                  // fast: rays whose interval overlaps the chunk
    unsigned short lrng[FAST ? 1 : CAP][32 / SUB];   // parity: per ray lo | hi << 8 (lo > hi: no hit)
    unsigned smask[NB][CAP / 32];                    // entries whose union range meets block k / MB
    unsigned long long occ[4];                       // slabs holding any entry (union occupancy)
    __align__(16) float packet[24];                  // the chunk's ray packet (set_packet), read as float4
    __align__(16) float cone[12];                    // the tile's ray directions (set_cone), read as float4
    int stack[kStack];
    // hit-list record of the warp's current tile (written by lane 0)
    unsigned rec_first, rec_prev;                    // forward: first / last chunk record
    unsigned rec_cur;                                // backward: next chunk record to replay
    unsigned long long cnt[kCounters];               // activity counters of the warp (lane 0)
};

// A team's part of shared memory: the list of its 8x4 tile and, per warp, the entry masks of the warp's rays.
template <int SUB, int CAP>
struct TeamSmem {
    struct Warp {
        unsigned smask[64][CAP / 32];
        unsigned long long occ[4], cnt[kCounters];
    };
    int ids[CAP];
    unsigned urng[CAP], lmask[CAP];                  // over the tile's 32 rays
    unsigned leaves[2 * CAP], cand[2 * CAP];         // leaves of the walk, and those that pass the cone test
    __align__(16) float packet[24];
    __align__(16) float cone[12];
    int stack[kStack];
    unsigned rec_first, rec_prev;
    int tile[2];
    unsigned hits[2][SUB];                           // leaves that each warp found hit
    unsigned walked;                                 // leaves of the walk | tree not through << 31
    unsigned char live[32];                          // rays that go on
    Warp warp[SUB];
};
// A warp of a team: names of what it uses in the team's part.
template <int SUB, int CAP>
struct TeamWarp {
    using Store = TeamSmem<SUB, CAP>;
    static constexpr int kStores = kWarpsPerBlock / SUB;
    static constexpr int MB = 4, NB = 64, KM = 255;
    Store& t;
    const int w;                                     // the warp's number in the team; 0 leads
    const int slot;                                  // the list lane (pixel of the 8x4 tile) of this lane's ray
    const unsigned own;                              // the list lanes of the warp's rays
    int flip = 0, tile_flip = 0;                     // which of the two buffers is next
    int (&ids)[CAP];
    unsigned (&urng)[CAP], (&lmask)[CAP];
    unsigned (&smask)[64][CAP / 32];
    unsigned long long (&occ)[4], (&cnt)[kCounters];
    float (&packet)[24], (&cone)[12];
    int (&stack)[kStack];
    // the warp's rays: the tile's left or right half (SUB == 2), or one of its quarters
    __device__ static int first(int w) { return SUB == 2 ? 4 * w : 4 * (w & 1) + 16 * (w >> 1); }
    __device__ TeamWarp(Store& s, int w_, int lane)
        : t(s), w(w_), slot(first(w_) + lane / SUB % 4 + 8 * (lane / SUB / 4)),
          own((SUB == 2 ? 0x0f0f0f0fu : 0x00000f0fu) << first(w_)), ids(s.ids), urng(s.urng), lmask(s.lmask),
          smask(s.warp[w_].smask), occ(s.warp[w_].occ), cnt(s.warp[w_].cnt), packet(s.packet), cone(s.cone),
          stack(s.stack) {}
    // Waits for the team's warps (what they wrote to shared memory is then visible).
    __device__ void sync() const {
        __syncwarp();
        asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)(threadIdx.x >> 5) / SUB), "n"(32 * SUB) : "memory");
    }
};
template <int CAP>
struct WarpSmem<true, 2, CAP> : TeamWarp<2, CAP> {
    using TeamWarp<2, CAP>::TeamWarp;
    __device__ static WarpSmem of(TeamSmem<2, CAP>* s, int warp, int lane) { return WarpSmem(s[warp / 2], warp % 2, lane); }
};
template <int CAP>
struct WarpSmem<true, 4, CAP> : TeamWarp<4, CAP> {
    using TeamWarp<4, CAP>::TeamWarp;
    __device__ static WarpSmem of(TeamSmem<4, CAP>* s, int warp, int lane) { return WarpSmem(s[warp / 4], warp % 4, lane); }
};

// Warp-uniform activity counters of one tile (32-bit; added to the warp's shared-memory totals at
// the end of the tile so that few registers stay live through the traversal and slab loops).
struct WarpStats {
    unsigned traversals = 0, node_visits = 0, leaf_tests = 0, entries = 0, slab_steps = 0, entry_slabs = 0,
             replays = 0;
};

struct RayState {
    float3 o, d;
    float tenter, texit;
    float tb;
    float T;
    float3 C;     // forward: accumulated colour
    float3 g;     // backward: dL/dcolour of the ray
    float gR;     // backward: g . R, R the colour still to come (the adjoint needs only this product)
    unsigned seed;
    bool alive;
};

// ---- IEEE-ordered helpers (no contraction) for the parity arithmetic ----------------------------
__device__ __forceinline__ float dot_rn(float3 a, float3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ float3 rows_rn(float3 r0, float3 r1, float3 r2, float3 v) {
    return f3(dot_rn(r0, v), dot_rn(r1, v), dot_rn(r2, v));
}

// One wide-node child slot (32 bytes) in one 256-bit read-only load.
__device__ __forceinline__ void load_slot(const WideSlot* p, float3& lo, float3& hi, int& id, int& range_hi) {
    float f[6];
    int u[2];
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]), "=r"(u[0]), "=r"(u[1])
        : "l"(p));
    lo = f3(f[0], f[1], f[2]);
    hi = f3(f[3], f[4], f[5]);
    id = u[0];
    range_hi = u[1];
}

// The chunk's ray packet for the wide-node test (interval arithmetic).  All rays start at the eye;
// over the active lanes, per axis the direction component lies in [dmin, dmax] and the ray
// parameter of the chunk segments in [tmin, tmax].  For a box, a ray's entry and exit parameters
// along axis a are the smaller and larger of (lo_a - o_a) / d_a and (hi_a - o_a) / d_a, linear in
// 1 / d_a: over the packet they lie between the products at the ends of the 1 / d interval, so the
// box can meet a segment only if the largest of the smallest entries (and tmin) does not exceed
// the smallest of the largest exits (and tmax).  Exact for one ray, conservative for a packet, tight
// for the nearly parallel rays of a tile.  An axis whose direction interval holds 0 gives no bound
// there; the box of the packet's segments (o + t d over the t and d intervals) bounds every axis.
// Stored per axis {1/dmax, 1/dmin, -o/dmax, -o/dmin}, then {tmin - slack, tmax + slack}, then the
// segments' box {lo.xyz, -}, {hi.xyz, -} widened by a position slack.  The
// products round like the per-ray slab test's t = b/d - o/d: a few ulps of |o| in position, far
// inside the leaf boxes' 1e-5 inflation, so the bound needs no slack of its own; a small one in t
// covers the ends of the segments.  (A slack that grows with 1/|d| would stretch the packets of
// rays nearly parallel to a coordinate plane over most of their length.)
template <bool FAST, int SUB, int CAP>
__device__ __forceinline__ void set_packet(WarpSmem<FAST, SUB, CAP>& sm, const RayState& r, bool on, float seg_hi,
                                           int lane) {
    float dmin[3], dmax[3];
    const float dv[3] = {r.d.x, r.d.y, r.d.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        dmin[a] = ord2f(__reduce_min_sync(kFull, on ? f2ord(dv[a]) : 0x7fffffff));
        dmax[a] = ord2f(__reduce_max_sync(kFull, on ? f2ord(dv[a]) : (int)0x80000000));
    }
    const float tmin = __uint_as_float(__reduce_min_sync(kFull, on ? __float_as_uint(fmaxf(r.tb, 0.f)) : 0x7f800000u));
    const float tmax = __uint_as_float(__reduce_max_sync(kFull, on ? __float_as_uint(fmaxf(seg_hi, 0.f)) : 0u));
    if (lane == 0) {
        const float ov[3] = {r.o.x, r.o.y, r.o.z};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            float4 q;
            if (!(dmin[a] > 0.f) && !(dmax[a] < 0.f)) {
                q = make_float4(0.f, 0.f, -INFINITY, INFINITY);   // the interval holds 0: no bound
            } else {
                const float rA = 1.f / dmax[a], rB = 1.f / dmin[a];
                q = make_float4(rA, rB, -ov[a] * rA, -ov[a] * rB);
            }
            *reinterpret_cast<float4*>(sm.packet + 4 * a) = q;
        }
        const float slack = 1e-6f * (tmax + 1.f);
        *reinterpret_cast<float4*>(sm.packet + 12) = make_float4(tmin - slack, tmax + slack, 0.f, 0.f);
        const float pslack = 1e-6f * (fabsf(ov[0]) + fabsf(ov[1]) + fabsf(ov[2]) + tmax + 1.f);
        float bl[3], bh[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float e0 = tmin * dmin[a], e1 = tmin * dmax[a], e2 = tmax * dmin[a], e3 = tmax * dmax[a];
            bl[a] = ov[a] + fminf(fminf(e0, e1), fminf(e2, e3)) - pslack;
            bh[a] = ov[a] + fmaxf(fmaxf(e0, e1), fmaxf(e2, e3)) + pslack;
        }
        *reinterpret_cast<float4*>(sm.packet + 16) = make_float4(bl[0], bl[1], bl[2], 0.f);
        *reinterpret_cast<float4*>(sm.packet + 20) = make_float4(bh[0], bh[1], bh[2], 0.f);
    }
    __syncwarp();
}

__device__ __forceinline__ void packet_axis(float4 q, float lo, float hi, float& tin, float& tout) {
    const float p1 = fmaf(lo, q.x, q.z), p2 = fmaf(lo, q.y, q.w), p3 = fmaf(hi, q.x, q.z), p4 = fmaf(hi, q.y, q.w);
    tin = fminf(fminf(p1, p2), fminf(p3, p4));
    tout = fmaxf(fmaxf(p1, p2), fmaxf(p3, p4));
}

// Whether a box may meet a segment of the packet (see set_packet).
__device__ __forceinline__ bool packet_hit(const float* F, float3 lo, float3 hi) {
    const float4 qx = *reinterpret_cast<const float4*>(F), qy = *reinterpret_cast<const float4*>(F + 4),
                 qz = *reinterpret_cast<const float4*>(F + 8), qt = *reinterpret_cast<const float4*>(F + 12);
    const float4 bl = *reinterpret_cast<const float4*>(F + 16), bh = *reinterpret_cast<const float4*>(F + 20);
    float ix, ox, iy, oy, iz, oz;
    packet_axis(qx, lo.x, hi.x, ix, ox);
    packet_axis(qy, lo.y, hi.y, iy, oy);
    packet_axis(qz, lo.z, hi.z, iz, oz);
    const bool in_box = lo.x <= bh.x && hi.x >= bl.x && lo.y <= bh.y && hi.y >= bl.y && lo.z <= bh.z && hi.z >= bl.z;
    return in_box && fmaxf(max3f(ix, iy, iz), qt.x) <= fminf(min3f(ox, oy, oz), qt.y);
}

// The tile's ray directions before normalisation, w + u dx + v dy, as centre + s * cone_u + t * cone_v
// with s and t in [-1, 1]: {centre.xyz, cone_u.x}, {cone_u.yz, cone_v.xy}, {cone_v.z,
// smallest and largest length, -}.
template <bool FAST, int SUB, int CAP>
__device__ __forceinline__ void set_cone(WarpSmem<FAST, SUB, CAP>& sm, const rg_camera& cam, float dx, float dy, bool valid,
                                         int lane) {
    const float x0 = ord2f(__reduce_min_sync(kFull, valid ? f2ord(dx) : 0x7fffffff));
    const float x1 = ord2f(__reduce_max_sync(kFull, valid ? f2ord(dx) : (int)0x80000000));
    const float y0 = ord2f(__reduce_min_sync(kFull, valid ? f2ord(dy) : 0x7fffffff));
    const float y1 = ord2f(__reduce_max_sync(kFull, valid ? f2ord(dy) : (int)0x80000000));
    if (lane == 0) {
        const float xc = 0.5f * (x0 + x1), yc = 0.5f * (y0 + y1), hx = 0.5f * (x1 - x0), hy = 0.5f * (y1 - y0);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            sm.cone[c] = fmaf(cam.u[c], xc, fmaf(cam.v[c], yc, cam.w[c]));
            sm.cone[3 + c] = cam.u[c] * hx;
            sm.cone[6 + c] = cam.v[c] * hy;
        }
        // bounds of |D| over the tile
        const float dc = sqrtf(dot3(f3(sm.cone[0], sm.cone[1], sm.cone[2]), f3(sm.cone[0], sm.cone[1], sm.cone[2])));
        const float dh = sqrtf(dot3(f3(sm.cone[3], sm.cone[4], sm.cone[5]), f3(sm.cone[3], sm.cone[4], sm.cone[5]))) +
                         sqrtf(dot3(f3(sm.cone[6], sm.cone[7], sm.cone[8]), f3(sm.cone[6], sm.cone[7], sm.cone[8])));
        sm.cone[9] = fmaxf(dc - dh, 0.f);
        sm.cone[10] = dc + dh;
    }
}

// Whether a ray of the tile may meet the leaf's threshold ellipsoid at ray parameters in [t0, t1] (one
// leaf per lane), and a lower bound of the parameter where it does.  In the space of m = M (x - mu) the
// ellipsoid is a sphere of radius R = 1 / k around 0 and the rays leave O = M (o - mu) along C + s U +
// t V (the images of the cone).  With e the unit vector along C, b = -O.e and p the unit vector from
// the central ray towards the sphere's centre, rho away, take the plane through O that is p tilted
// towards the rays until all of them lie under it: the tilt's tangent is tau = (|p.U| + |p.V|) /
// (|C| - |e.U| - |e.V|), and the centre's height over the plane is (rho - b tau) / sqrt(1 + tau^2).
// No ray reaches a sphere that lies over the plane.  Along e the sphere spans b -+ R and a ray moves
// by (|C| -+ |e.U| -+ |e.V|) / |D| per unit of its parameter.
//   Rounding.  O, C, U, V and the exact test's images of the ray are products with M: each is off by up to
// 2e-7 |M| times the vector that went in, which for a flat Gaussian is far more than 2e-7 times the result.
// Carried to the sphere each moves a ray by 2e-7 |M| |mu - o|, all of them by less than 1e-6 of it (|M| the
// Frobenius norm); the steps after the products add 1e-5 |O| at most: both widen R, with a thousandth of it.
// What is left of b e in P would be multiplied by the long U and V: they enter the tilt without their parts
// along e, with 4e-7 of their lengths for what that rounds off.  NaN (a Gaussian that is never hit, an
// overflow) keeps the leaf: the exact test decides.
template <bool FAST, int SUB, int CAP>
__device__ __forceinline__ bool may_hit(const WarpSmem<FAST, SUB, CAP>& sm, const LeafRec& rec, float3 o, float t0, float t1,
                                        float& t_first) {
    const float4 q0 = *reinterpret_cast<const float4*>(sm.cone), q1 = *reinterpret_cast<const float4*>(sm.cone + 4),
                 q2 = *reinterpret_cast<const float4*>(sm.cone + 8);
    const float3 dc = f3(q0.x, q0.y, q0.z), du = f3(q0.w, q1.x, q1.y), dv = f3(q1.z, q1.w, q2.x);
    const float3 r0 = f3(rec.r0.x, rec.r0.y, rec.r0.z), r1 = f3(rec.r1.x, rec.r1.y, rec.r1.z),
                 r2 = f3(rec.r2.x, rec.r2.y, rec.r2.z);
    const float3 v = f3(rec.a.x, rec.a.y, rec.a.z) - o;
    const float3 O = f3(dot3(r0, v), dot3(r1, v), dot3(r2, v));   // -O: from the eye to the centre
    const float3 C = f3(dot3(r0, dc), dot3(r1, dc), dot3(r2, dc));
    const float3 U = f3(dot3(r0, du), dot3(r1, du), dot3(r2, du));
    const float3 V = f3(dot3(r0, dv), dot3(r1, dv), dot3(r2, dv));
    const float c2 = dot3(C, C), ic = rsqrtf(c2), c1 = c2 * ic;
    const float3 e = C * ic;
    const float b = dot3(O, e);
    const float3 P = O - e * b;
    const float rho2 = dot3(P, P), ir = rsqrtf(rho2);
    const float rho = rho2 * ir;
    const float eu = dot3(e, U), ev = dot3(e, V);
    const float width = (fabsf(dot3(P, U - e * eu)) + fabsf(dot3(P, V - e * ev))) * ir +
                        4e-7f * (sqrt_approx(dot3(U, U)) + sqrt_approx(dot3(V, V)));
    const float spread = fabsf(eu) + fabsf(ev);
    const float along = c1 * 0.99999f - spread;
    const float m2 = dot3(r0, r0) + dot3(r1, r1) + dot3(r2, r2);
    const float R = __fdividef(1.f, rec.r0.w) * 1.001f + 1e-5f * (rho + fabsf(b)) + 1e-6f * sqrt_approx(m2 * dot3(v, v));
    const bool miss = along > 0.f && rho * along - b * width > R * sqrtf(along * along + width * width);
    t_first = __fdividef(fmaxf(b - R, 0.f) * q2.y, c1 + spread) * 0.99999f;
    const bool before = along > 0.f && (b + R) * q2.z * 1.00001f < t0 * along, after = t_first > t1;
    return !(miss || before || after);
}

__device__ __forceinline__ LeafRec load_rec(const LeafRec* p, int i) {
    const float4* q = reinterpret_cast<const float4*>(p + i);
    LeafRec r;
    r.a = __ldg(q);
    r.r0 = __ldg(q + 1);
    r.r1 = __ldg(q + 2);
    r.r2 = __ldg(q + 3);
    return r;
}

// Ray/ellipsoid interval in the reference intersection program's arithmetic
// (forward/gaussians_aabb.cu:359-381): IEEE operations in source order on the precomputed
// threshold-scaled conic.  Returns false when disc <= 1e-7 (no report).
__device__ __forceinline__ bool roots_exact(const LeafIS& s, float3 mu, const RayState& r, float& root1,
                                            float& root2) {
    float3 U = f3(s.u.x, s.u.y, s.u.z), V = f3(s.v.x, s.v.y, s.v.z), W = f3(s.w.x, s.w.y, s.w.z);
    float3 O = f3(__fsub_rn(r.o.x, mu.x), __fsub_rn(r.o.y, mu.y), __fsub_rn(r.o.z, mu.z));
    float3 Oe = f3(dot_rn(U, O), dot_rn(V, O), dot_rn(W, O));
    float3 De = f3(dot_rn(U, r.d), dot_rn(V, r.d), dot_rn(W, r.d));
    float l = __fdiv_rn(1.f, __fsqrt_rn(dot_rn(De, De)));
    float3 D = f3(__fmul_rn(De.x, l), __fmul_rn(De.y, l), __fmul_rn(De.z, l));
    float b = -dot_rn(Oe, D);
    float c = __fsub_rn(dot_rn(Oe, Oe), 1.f);
    float3 p = f3(__fadd_rn(Oe.x, __fmul_rn(D.x, b)), __fadd_rn(Oe.y, __fmul_rn(D.y, b)),
                  __fadd_rn(Oe.z, __fmul_rn(D.z, b)));
    float disc = __fsub_rn(1.f, dot_rn(p, p));
    if (!(disc > 1e-7f)) return false;
    float sd = __fsqrt_rn(disc);
    float q = __fadd_rn(b, b > 0.f ? sd : -sd);
    root1 = __fmul_rn(__fdiv_rn(c, q), l);
    root2 = __fmul_rn(q, l);
    return true;
}

// The same interval from the sampling conic scaled by the threshold factor k (fast arithmetic).
__device__ __forceinline__ bool roots_fast(const LeafRec& rec, const RayState& r, float& root1, float& root2) {
    float3 O = r.o - f3(rec.a.x, rec.a.y, rec.a.z);
    float k = rec.r0.w;
    float3 r0 = f3(rec.r0.x, rec.r0.y, rec.r0.z), r1 = f3(rec.r1.x, rec.r1.y, rec.r1.z),
           r2 = f3(rec.r2.x, rec.r2.y, rec.r2.z);
    float3 Oe = f3(dot3(r0, O) * k, dot3(r1, O) * k, dot3(r2, O) * k);
    float3 De = f3(dot3(r0, r.d) * k, dot3(r1, r.d) * k, dot3(r2, r.d) * k);
    // SFU reciprocal square roots and a fast division (the fast arithmetic's interval ends move by
    // ulps; the forward and the backward's replay run this same test)
    float l = rsqrtf(dot3(De, De));
    float3 Dn = De * l;
    float b = -dot3(Oe, Dn);
    float c = dot3(Oe, Oe) - 1.f;
    float3 p = Oe + Dn * b;
    float disc = 1.f - dot3(p, p);
    if (!(disc > 1e-7f)) return false;
    float sd = disc * rsqrtf(disc);
    float q = b + (b > 0.f ? sd : -sd);   // |q| >= sd > 3e-4
    root1 = __fdividef(c, q) * l;
    root2 = q * l;
    return true;
}

__device__ __forceinline__ LeafIS load_is(const LeafIS* p, int i) {
    const float4* q = reinterpret_cast<const float4*>(p + i);
    LeafIS s;
    s.u = __ldg(q);
    s.v = __ldg(q + 1);
    s.w = __ldg(q + 2);
    return s;
}

// Slab range [lo, hi] of the chunk (K slabs from r.tb) hit by the interval [root1, root2].
// Slab k of the chunk against the interval, in slab units from tb (a, b: interval ends, e: box
// exit) with tb_k = k up to the margin m: 1 certain hit, -1 certain miss, 0 undecided.  Slab k is
// hit iff root1 <= min(texit, tb_k + 0.02), tb_k <= root2 and root1 <= root2.
__device__ __forceinline__ int classify_slab(int k, float a, float b, float e, float m) {
    const float kf = (float)k;
    if (a > b || a > kf + 1.f + m || a > e + m || kf - m > b) return -1;
    if (a <= kf + 1.f - m && a <= e - m && kf + m <= b) return 1;
    return 0;
}

// The reference's test for slab k of the chunk, tb_k by k repeated FP32 additions from tb.
__device__ __noinline__ bool slab_k_hit(float tb, float tenter, float texit, int k, float root1, float root2) {
    float t = tb;
    for (int j = 0; j < k; ++j) t = t + kSlab;
    const float th = fminf(texit, t + kSlab);
    return th > tenter && fmaxf(t, root1) <= fminf(th, root2);
}

// The interval's slabs, mapped arithmetically.  Slab k starts at tb_k, tb plus k slabs by repeated FP32
// addition, and is hit iff root1 <= tb_k + 0.02 and tb_k <= root2.  The range keeps a margin that
// covers the drift of the repeated addition, so it holds every hit slab and at most one extra slab at
// each end.  Chunks up to kExactChunk and the parity arithmetic settle the ends exactly here; in
// longer chunks the fast arithmetic evaluates them (their samples fall outside the threshold
// ellipsoid).
template <bool FAST>
__device__ __forceinline__ void slab_range(const RayState& r, int K, int nv, float seg_hi, float tclip, float root1,
                                           float root2, int& lo, int& hi) {
    lo = 255;
    hi = -1;
    if (fmaxf(r.tb, root1) <= fminf(seg_hi, root2)) {
        // (the eight tests of a short chunk one after the other took twice the instructions)
        float a = fmaxf((root1 - r.tb) * kInvSlab, -1.f);
        float b = fminf((root2 - r.tb) * kInvSlab, 4096.f);
        // drift of tb_k in slab units: (K + 1) ulps of |tb| + K slabs, 2^-23 relative each (four
        // times the bound of round-to-nearest additions)
        const float m = (float)(K + 1) * (fabsf(r.tb) + (float)K * kSlab) * (kInvSlab * 2.4e-7f) + 1e-4f;
        lo = max(0, (int)ceilf(a - 1.f - m));
        hi = min(nv - 1, (int)floorf(b + m));
        if (!FAST || K <= kExactChunk) {
            // Settle both ends exactly.  A slab whose hit or miss the margins cannot decide gets the
            // reference's per-slab test (rare: its interval end lies within the margin of a slab
            // edge or of the box exit).
            const float e = fminf((tclip - r.tb) * kInvSlab, 4096.f);
            while (lo <= hi) {
                const int c = classify_slab(lo, a, b, e, m);
                if (c > 0 || (c == 0 && slab_k_hit(r.tb, r.tenter, tclip, lo, root1, root2))) break;
                ++lo;
            }
            while (hi >= lo) {
                const int c = classify_slab(hi, a, b, e, m);
                if (c > 0 || (c == 0 && slab_k_hit(r.tb, r.tenter, tclip, hi, root1, root2))) break;
                --hi;
            }
        }
        if (lo > hi) { lo = 255; hi = -1; }
    }
}

// 32-entry mask words holding `count` list entries.
__device__ __forceinline__ int nwords(int count) { return (count + 31) >> 5; }

// Union occupancy of the chunk's slabs (256 bits): bit k set when some lane has a hit in slab k.
__device__ __forceinline__ bool occ_test(const unsigned long long* occ, int k) {
    return (occ[k >> 6] >> (k & 63)) & 1ull;
}
// whether any of the slabs k .. k + n - 1 is occupied (n <= 4, k a multiple of n: one word)
__device__ __forceinline__ bool occ_any(const unsigned long long* occ, int k, int n) {
    return (occ[k >> 6] >> (k & 63)) & ((1ull << n) - 1ull);
}
// first occupied slab >= k (K when none)
__device__ __forceinline__ int occ_next(const unsigned long long* occ, int k, int K) {
    for (int w = k >> 6; w < 4 && 64 * w < K; ++w) {
        unsigned long long m = occ[w];
        if (w == (k >> 6)) m &= (~0ull) << (k & 63);
        if (m) return min(K, 64 * w + __ffsll((long long)m) - 1);
    }
    return K;
}

// Where the chunk records of a tile are kept: with the warp, or with the team.
template <bool FAST, int SUB, int CAP>
__device__ __forceinline__ auto& record_of(WarpSmem<FAST, SUB, CAP>& sm) {
    if constexpr (FAST && SUB > 1) return sm.t;
    else return sm;
}

// Adds the tile's counters to the warp's totals and resets them.
template <bool FAST, int SUB, int CAP, bool DIAG>
__device__ __forceinline__ void flush_stats(WarpSmem<FAST, SUB, CAP>& sm, WarpStats& ws, unsigned hits, unsigned slabs,
                                            int lane) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        hits += __shfl_xor_sync(kFull, hits, o);
        slabs += __shfl_xor_sync(kFull, slabs, o);
    }
    if (lane == 0) {
        sm.cnt[0] += ws.traversals;
        if (DIAG) {
            sm.cnt[1] += ws.node_visits;
            sm.cnt[2] += ws.leaf_tests;
            sm.cnt[3] += ws.entries;
            sm.cnt[4] += ws.slab_steps;
            sm.cnt[5] += ws.entry_slabs;
        }
        sm.cnt[6] += ws.replays;
        sm.cnt[7] += hits;
        sm.cnt[8] += slabs;
    }
    ws = WarpStats();
}

// The slabs [lo, hi] of the chunk in which a ray meets a leaf (exact test; lo > hi: none).
template <bool FAST>
__device__ __forceinline__ void leaf_slabs(const RenderArgs& a, const RayState& r, float seg_hi, int K, int nv, int leaf,
                                           bool infer, int& lo, int& hi) {
    float root1, root2;
    bool ok;
    if (FAST) {
        ok = roots_fast(load_rec(a.rec, leaf), r, root1, root2);
    } else {
        float4 m4 = __ldg(reinterpret_cast<const float4*>(a.rec + leaf));
        ok = roots_exact(load_is(a.is_rec, leaf), f3(m4.x, m4.y, m4.z), r, root1, root2);
    }
    // the slab query ends at the box exit in training launches and at the slab end in
    // inference launches (cuda_test/gaussians_aabb.cu:408-409)
    const float tclip = infer ? INFINITY : r.texit;
    if (ok) slab_range<FAST>(r, K, nv, seg_hi, tclip, root1, root2, lo, hi);
}

// Exact test of SUB leaves at a time, each by the 32 / SUB rays of the tile (`leaf`: the one of the
// lane's sub-slab, < 0 for none).  Leaves that any ray hits are appended to the list, in order.  Returns
// how many leaves were dealt with: SUB, or the number of those before the one that found the list full.
template <bool FAST, int SUB, int CAP, bool DIAG>
__device__ __forceinline__ int leaf_batch(WarpSmem<FAST, SUB, CAP>& sm, const RenderArgs& a, const RayState& r, bool on,
                                          float seg_hi, int K, int nv, int leaf, int& count, int lane,
                                          WarpStats& ws, bool infer) {
    if (DIAG) ws.leaf_tests += __popc(__ballot_sync(kFull, lane < SUB && leaf >= 0));
    int lo = 255, hi = -1;
    if (on && (SUB == 1 || leaf >= 0)) leaf_slabs<FAST>(a, r, seg_hi, K, nv, leaf, infer, lo, hi);
    const unsigned any = __ballot_sync(kFull, lo <= hi);
    if (!any) return SUB;
    if constexpr (SUB == 1) {
        if (count == CAP) return 0;
        int ulo = (int)__reduce_min_sync(kFull, (unsigned)lo);
        int uhi = (int)__reduce_max_sync(kFull, (unsigned)(hi + 1)) - 1;
        if (FAST) {
            if (lane == 0) sm.lmask[count] = any;
        } else {
            sm.lrng[count][lane] = (unsigned short)((lo & 0xff) | ((hi & 0xff) << 8));
        }
        if (lane == 0) {
            sm.ids[count] = leaf;
            sm.urng[count] = (unsigned)ulo | ((unsigned)uhi << 16);
        }
        ++count;
        return 1;
    } else {
        static_assert(!FAST, "teams test their leaves with team_batch");
        const int sub = lane % SUB;
        int ulo = lo, uhi = hi;
        unsigned hit = any;          // bit q: some ray hits the leaf of sub-slab q
#pragma unroll
        for (int o = SUB; o < 32; o <<= 1) {
            ulo = min(ulo, __shfl_xor_sync(kFull, ulo, o));
            uhi = max(uhi, __shfl_xor_sync(kFull, uhi, o));
            hit |= hit >> o;
        }
        hit &= (1u << SUB) - 1u;
        const int at = count + __popc(hit & ((1u << sub) - 1u)), n = __popc(hit);
        if (((hit >> sub) & 1u) && at < CAP) {
            sm.lrng[at][lane / SUB] = (unsigned short)((lo & 0xff) | ((hi & 0xff) << 8));
            if (lane < SUB) {
                sm.ids[at] = leaf;
                sm.urng[at] = (unsigned)ulo | ((unsigned)uhi << 16);
            }
        }
        const int room = CAP - count;
        count += min(n, room);
        if (n <= room) return SUB;
        // the first leaf without room: bit number `room` of the hits
        for (int i = 0; i < room; ++i) hit &= hit - 1u;
        return __ffs(hit) - 1;
    }
}

// The lane's leaf of the next SUB in `todo` (bits of lanes whose `mine` holds a leaf): its sub-slab's, or -1.
template <int SUB>
__device__ __forceinline__ int next_leaf(unsigned todo, unsigned mine, int lane) {
    unsigned t = todo;
#pragma unroll
    for (int i = 0; i < SUB - 1; ++i)
        if (i < lane % SUB) t &= t - 1u;
    const int leaf = (int)__shfl_sync(kFull, mine, __ffs(t) - 1);
    return SUB == 1 || t ? leaf : -1;
}

// Bits lo..hi of 64-slab word w (none where the range does not meet it).
__device__ __forceinline__ unsigned long long range_bits(int lo, int hi, int w) {
    const int a0 = max(lo - 64 * w, 0), b0 = min(hi - 64 * w, 63);
    return a0 <= b0 ? ((~0ull) >> (63 - (b0 - a0))) << a0 : 0ull;
}

// Publishes the chunk list: occupancy bits and the entry masks per block of MB slabs.  One lane per
// entry: a word of 32 entries costs a ballot per block and an OR-reduction per 32 slabs, against a
// serial walk of all entries per block and, for the occupancy, by lane 0 as entries were appended.
template <bool FAST, int SUB, int CAP, bool DIAG>
__device__ __forceinline__ void finish_list(WarpSmem<FAST, SUB, CAP>& sm, int count, int K, int lane, WarpStats& ws) {
    constexpr bool TEAM = FAST && SUB > 1;   // a team's warp takes the entries that its rays hit
    __syncwarp();
    if constexpr (TEAM) {
        if (DIAG && sm.w == 0) ws.entries += count;
    } else {
        if (DIAG) ws.entries += count;
    }
    constexpr int MB = WarpSmem<FAST, SUB, CAP>::MB;
    const int nblk = (K + MB - 1) / MB, nocc = (K + 63) >> 6;
    const int nw = nwords(count);
    if (lane < 4) sm.occ[lane] = 0ull;
    __syncwarp();
#pragma unroll 1
    for (int w = 0; w < nw; ++w) {
        const int e = 32 * w + lane;
        bool in = e < count;
        if constexpr (TEAM) in = in && (sm.lmask[e] & sm.own);
        const unsigned u = in ? sm.urng[e] : 0xffffu;   // no entry: lo 65535 > hi 0
        const int lo = (int)(u & 0xffffu), hi = (int)(u >> 16);
        // entry e meets block bk iff b0 <= bk <= b1
        const int b0 = lo / MB, b1 = hi / MB;
#pragma unroll 1
        for (int bk = 0; bk < nblk; bk += 32) {
            const int m = min(32, nblk - bk);
            unsigned mine = 0u;
#pragma unroll 4
            for (int j = 0; j < m; ++j) {
                const unsigned mw = __ballot_sync(kFull, b0 <= bk + j && bk + j <= b1);
                if (lane == j) mine = mw;
            }
            if (lane < m) sm.smask[bk + lane][w] = mine;
        }
#pragma unroll 1
        for (int o = 0; o < nocc; ++o) {
            const unsigned long long v = range_bits(lo, hi, o);
            const unsigned vl = __reduce_or_sync(kFull, (unsigned)v), vh = __reduce_or_sync(kFull, (unsigned)(v >> 32));
            if (lane == 0) sm.occ[o] |= ((unsigned long long)vh << 32) | vl;
        }
    }
    __syncwarp();
}

// Slabs of the chunk a lane marches (nv: slab k is marched iff tb_k < texit, tb_k by repeated
// addition) and the end of its searched segment.
__device__ __forceinline__ void chunk_extent(const RayState& r, bool on, int K, float t_end, int& nv, float& seg_hi) {
    nv = 0;
    seg_hi = r.tb;
    if (!on) return;
    if (K <= kExactChunk) {
        float t = r.tb;
        for (int kk = 0; kk < K; ++kk) {
            if (t < r.texit) { nv = kk + 1; t = t + kSlab; } else break;
        }
        seg_hi = fminf(t_end, t);
    } else {
        nv = K;
        seg_hi = fminf(t_end, r.tb + (float)(K + 1) * kSlab);
    }
}

// A walk through the wide tree (warp-uniform).  Candidates [0, nc), then leaves still waiting for may_hit
// [nc, nc + nr).  A candidate is leaf | (first slab / 2) << 25.
struct Walk {
    int nc = 0, nr = 0;
    int sp = 0, cur = ~0;    // one Gaussian: the root is a leaf
    bool more = true;        // cur is still to be visited
    unsigned guard = 0, visits = 0;
};
constexpr unsigned kLeafMask = (1u << 25) - 1u;
static_assert(kMaxGaussians == 1ll << 25, "25 bits of a candidate hold the leaf");

__device__ __forceinline__ Walk walk_start(const RenderArgs& a) {
    Walk s;
    if (a.n_leaves > 1) {
        const int2 root = __ldg(a.wide_tab);
        s.cur = wide_pack(root.x, root.y);
    }
    return s;
}

// may_hit for a leaf of the lane's own.  A ray of the tile may meet it in the chunk: `first` is the first slab
// where.  [t0, t1]: where the tile's chunks start; t_last: where they end.
struct ChunkSpan {
    float t0, t1, t_last;
};
__device__ __forceinline__ ChunkSpan chunk_span(const RayState& r, bool on, float seg_hi) {
    return {__uint_as_float(__reduce_min_sync(kFull, on ? __float_as_uint(r.tb) : 0x7f800000u)),
            __uint_as_float(__reduce_max_sync(kFull, on ? __float_as_uint(r.tb) : 0u)),
            __uint_as_float(__reduce_max_sync(kFull, on ? __float_as_uint(seg_hi) : 0u))};
}
template <bool FAST, int SUB, int CAP>
__device__ __forceinline__ bool cull(const WarpSmem<FAST, SUB, CAP>& sm, const RenderArgs& a, float3 o, const ChunkSpan& c,
                                     int K, int leaf, int& first) {
    float t;
    const bool may = may_hit<FAST, SUB, CAP>(sm, load_rec(a.rec, leaf), o, c.t0 * 0.99999f, c.t_last * 1.00001f, t);
    // slab s of a lane starts at tb + 0.02 s up to the drift of the repeated addition
    const float drift = (float)(K + 1) * (c.t1 + (float)K * kSlab) * (kInvSlab * 2.4e-7f);
    first = min(255, max(0, (int)((t - c.t1) * kInvSlab - 1.f - drift)));
    return may && first < K;
}

// Goes on until the buffer (2 CAP words) is nearly full or the tree is through.  CULL: the leaves take may_hit
// on the way; else every leaf is a candidate.
template <bool CULL, bool FAST, int SUB, int CAP, bool DIAG>
__device__ __forceinline__ void walk_tree(WarpSmem<FAST, SUB, CAP>& sm, unsigned* cand, const RenderArgs& a,
                                          const RayState& r, bool on, float seg_hi, int K, int cursor, Walk& s,
                                          int lane) {
    constexpr int NC = 2 * CAP;
    const unsigned guard_max = 2u * (unsigned)a.n_leaves + 64u;
    while (true) {
        if constexpr (!CULL) {
            s.nc += s.nr;
            s.nr = 0;
        }
        if (CULL && (s.nr >= 32 || (s.nr > 0 && !s.more))) {
            // may_hit for up to 32 waiting leaves; the rest moves up behind the candidates
            const int m = min(s.nr, 32);
            const unsigned leaf = lane < m ? cand[s.nc + lane] : 0u;
            const unsigned next = 32 + lane < s.nr ? cand[s.nc + 32 + lane] : 0u;
            const ChunkSpan c = chunk_span(r, on, seg_hi);
            int first = 0;
            const bool may = lane < m && (int)leaf > cursor && cull<FAST, SUB, CAP>(sm, a, r.o, c, K, (int)leaf, first);
            const unsigned mm = __ballot_sync(kFull, may);
            if (may) cand[s.nc + __popc(mm & ((1u << lane) - 1u))] = leaf | ((unsigned)(first >> 1) << 25);
            s.nc += __popc(mm);
            s.nr -= m;
            __syncwarp();
            if (lane < s.nr) cand[s.nc + lane] = next;
            __syncwarp();
        } else if (s.more && s.nc <= NC - 64) {
            if (++s.guard > guard_max) {
                if (lane == 0) atomicAdd(&a.st->watchdog_trips, 1ull);
                s.more = false;
                continue;
            }
            if (s.cur >= 0) {
                if (DIAG) ++s.visits;
                const int first = s.cur & ((1 << kWideCountShift) - 1), n = (s.cur >> kWideCountShift) + 1;
                bool hit = false;
                int cid = 0;
                if (lane < n) {
                    float3 lo, hi;
                    int range_hi;
                    load_slot(a.slots + first + lane, lo, hi, cid, range_hi);
                    hit = (range_hi > cursor) && packet_hit(sm.packet, lo, hi);
                }
                const unsigned hm = __ballot_sync(kFull, hit), im = __ballot_sync(kFull, hit && cid >= 0);
                const unsigned lead = hm & ((im & (0u - im)) - 1u);   // leaves before the first node (all: no node)
                if ((lead >> lane) & 1u) cand[s.nc + s.nr + __popc(lead & ((1u << lane) - 1u))] = (unsigned)~cid;
                s.nr += __popc(lead);
                unsigned rest = hm & ~lead;
                if (rest) {
                    // a hit lane's place on the stack is the number of hit children above it
                    const int f = __ffs(rest) - 1;
                    rest &= rest - 1u;
                    const int more = __popc(rest);
                    if (s.sp + more <= kStack) {
                        if ((rest >> lane) & 1u) sm.stack[s.sp + __popc(rest >> lane) - 1] = cid;
                        s.sp += more;
                    } else if (lane == 0) {
                        atomicAdd(&a.st->stack_overflows, 1ull);
                    }
                    s.cur = __shfl_sync(kFull, cid, f);
                    __syncwarp();
                    continue;
                }
            } else {
                if (lane == 0) cand[s.nc + s.nr] = (unsigned)~s.cur;
                ++s.nr;
            }
            __syncwarp();
            if (s.sp == 0) s.more = false;
            else s.cur = sm.stack[--s.sp];
        } else {
            break;
        }
    }
}

// Marches up to n slabs by repeated addition; returns how many.  Its variables are its own: an empty far field is
// nothing but this loop, and a ray's state that is spilled around it would be loaded and stored in every turn
// (5000 Gaussians in a ball, two views at 610x442, forward / backward: 2.39 / 2.10 ms so, 2.12 / 1.77 now).
__device__ __forceinline__ unsigned march(float& tb, float texit, int n) {
    float t = tb;
    int j = 0;
    for (; j < n && t < texit; ++j) t = t + kSlab;
    tb = t;
    return (unsigned)j;
}

// Warp-cooperative traversal for the chunk [tb, seg_hi] of every active lane (the packet set by
// set_packet).  At a wide node lane k tests child slot k against the packet.  Hit leaves wait in a
// buffer (the leading ones of a node are taken all at once); the first hit child that is a node is
// visited next and the children after it wait on the stack, the lowest index on top, so leaves are
// reached in increasing index (the multi-pass cursor relies on it).  Thirty-two waiting leaves at a
// time, one per lane, may_hit drops those that no ray of the tile meets; the candidates that remain
// keep the first slab that they can reach.  When the tree is through, the candidates get the exact
// test per ray, and those that any ray hits are appended to the warp list, whose entry count is
// returned.  A leaf costs a visit's warp 1/32 of may_hit instead of a whole exact test: on 1M
// Gaussians x 16 views 364M exact tests instead of 633M (128M entries), forward 251 -> 225 ms; 3M x 4 x
// 1080p: 243 -> 198 ms.
//
// A chunk with too many Gaussians is shortened in place (K, nv and seg_hi): when the list fills up, K is
// halved, entries that start at slab K or later are dropped, those that stay get the exact test again,
// and the traversal goes on from its stack with the smaller packet.  The list is the one that a
// traversal started with the shorter chunk builds, and nothing is visited twice.  Only entries count: a
// chunk's length decides which samples at slab edges the fast arithmetic evaluates, so it must not depend
// on how many leaves pass may_hit.  When these fill their buffer they get the exact test at once and the
// walk goes on.  `ovf` is set when the list filled up for a single slab before the traversal finished.
template <bool FAST, int SUB, int CAP, bool DIAG>
__device__ int traverse(WarpSmem<FAST, SUB, CAP>& sm, const RenderArgs& a, const RayState& r, bool on, float t_end,
                        float& seg_hi, int& K, int& nv, int cursor, bool& ovf, int lane, WarpStats& ws, bool infer) {
    int count = 0;
    ++ws.traversals;
    ovf = false;
    // the candidates lie in the entry masks' space, which finish_list writes only afterwards
    unsigned* const cand = &sm.smask[0][0];
    static_assert(sizeof(sm.smask) >= 2 * CAP * sizeof(unsigned) && 2 * CAP >= 256, "candidate buffer");
    int done = 0;            // candidates that had the exact test
    int rt = 0, rn = 0;      // entries of the shortened chunk's old list still to test again: [rt, rn)
    Walk s = walk_start(a);
    while (true) {
        if (rt >= rn && done == 0) walk_tree<true, FAST, SUB, CAP, DIAG>(sm, cand, a, r, on, seg_hi, K, cursor, s, lane);
        // exact tests, in order: the list's entries again after a chunk was shortened, else candidates
        const bool again = rt < rn;
        unsigned todo;
        unsigned mine = 0u;
        if (again) {
            // in registers before its places are written again (an entry never moves up)
            const bool in = rt + lane < rn;
            if (in) mine = (unsigned)sm.ids[rt + lane];
            todo = __ballot_sync(kFull, in && (int)(sm.urng[rt + lane] & 0xffffu) < K);
            rt += 32;
        } else {
            if (done >= s.nc) {
                if (!s.more) break;
                // the candidates were many: they are in the list, the tree goes on (under 32 leaves wait)
                const unsigned w = lane < s.nr ? cand[s.nc + lane] : 0u;
                __syncwarp();
                if (lane < s.nr) cand[lane] = w;
                s.nc = done = 0;
                __syncwarp();
                continue;
            }
            const bool in = done + lane < s.nc;
            const unsigned c = in ? cand[done + lane] : 0u;
            mine = c & kLeafMask;
            todo = __ballot_sync(kFull, in && 2 * (int)(c >> 25) < K);
        }
        while (todo) {
            const int leaf = next_leaf<SUB>(todo, mine, lane);
            const int n = leaf_batch<FAST, SUB, CAP, DIAG>(sm, a, r, on, seg_hi, K, nv, leaf, count, lane, ws, infer);
#pragma unroll
            for (int i = 0; i < SUB; ++i)
                if (i < n) todo &= todo - 1u;
            if (n < SUB) break;
        }
        if (!again) done = min(s.nc, done + (todo ? __ffs(todo) - 1 : 32));
        if (todo) {
            if (K == 1) {
                ovf = true;
                break;
            }
            // the list is full: shorten the chunk, test its entries again, then come back to this leaf
            __syncwarp();
            K >>= 1;
            if (lane == 0) atomicAdd(&a.st->chunk_splits, 1ull);
            chunk_extent(r, on, K, t_end, nv, seg_hi);
            set_packet<FAST, SUB, CAP>(sm, r, on, seg_hi, lane);
            rt = 0;
            rn = count;
            count = 0;
        }
        __syncwarp();
    }
    if (DIAG) ws.node_visits += s.visits;
    finish_list<FAST, SUB, CAP, DIAG>(sm, count, K, lane, ws);
    return count;
}

// Exact tests of a team: the leaves of `todo` (bits of lanes whose `mine` holds a leaf, the same in every warp)
// are dealt out to its warps, a lane per ray of the tile (r: the list lane's ray), and those that any ray
// hits are appended to the list, in order.  Returns what is left of `todo` when the list is full, else 0.
// One barrier: the buffers alternate, and an entry's place is at or before the one its leaf was read from.
template <int SUB, int CAP, bool DIAG>
__device__ __forceinline__ unsigned team_batch(WarpSmem<true, SUB, CAP>& sm, const RenderArgs& a, const RayState& r,
                                               bool on, float seg_hi, int K, int nv, unsigned todo, unsigned mine,
                                               int& count, int lane, WarpStats& ws, bool infer) {
    constexpr int kShare = 32 / SUB;
    unsigned hits = 0u, rays = 0u, range = 0u;   // lane i keeps the warp's i-th leaf
#pragma unroll 2
    for (int i = 0; i < kShare; ++i) {
        const int b = i * SUB + sm.w;
        const int leaf = (int)__shfl_sync(kFull, mine, b);
        if (!((todo >> b) & 1u)) continue;
        int lo = 255, hi = -1;
        if (on) leaf_slabs<true>(a, r, seg_hi, K, nv, leaf, infer, lo, hi);
        const unsigned any = __ballot_sync(kFull, lo <= hi);
        if (!any) continue;
        const unsigned ulo = __reduce_min_sync(kFull, (unsigned)lo);
        const unsigned uhi = __reduce_max_sync(kFull, (unsigned)(hi + 1)) - 1u;
        hits |= 1u << b;
        if (lane == i) {
            rays = any;
            range = ulo | (uhi << 16);
        }
    }
    if (DIAG) ws.leaf_tests += sm.w == 0 ? __popc(todo) : 0;
    if (lane == 0) sm.t.hits[sm.flip][sm.w] = hits;
    sm.sync();
    unsigned all = 0u;
#pragma unroll
    for (int q = 0; q < SUB; ++q) all |= sm.t.hits[sm.flip][q];
    sm.flip ^= 1;
    const int b = lane % kShare * SUB + sm.w;
    const int leaf = (int)__shfl_sync(kFull, mine, b);
    const int at = count + __popc(all & ((1u << b) - 1u)), n = __popc(all), room = CAP - count;
    if (rays && at < CAP) {
        sm.ids[at] = leaf;
        sm.urng[at] = range;
        sm.lmask[at] = rays;
    }
    count += min(n, room);
    if (n <= room) return 0u;
    for (int i = 0; i < room; ++i) all &= all - 1u;   // the first leaf without room
    return todo & ~((all & (0u - all)) - 1u);
}

// traverse by a team: the same list, from the rays of its 8x4 tile.  The team's first warp walks, all of them
// cull and test.  Every warp takes the same way through here.
template <int SUB, int CAP, bool DIAG>
__device__ int team_traverse(WarpSmem<true, SUB, CAP>& sm, const RenderArgs& a, const RayState& r, bool on, float t_end,
                             float& seg_hi, int& K, int& nv, int cursor, bool& ovf, int lane, WarpStats& ws, bool infer) {
    unsigned* const cand = sm.t.cand;
    int count = 0;
    ovf = false;
    Walk s = walk_start(a);
    if (sm.w == 0) {
        ++ws.traversals;
        set_packet<true, SUB, CAP>(sm, r, on, seg_hi, lane);
    }
    sm.sync();               // the last chunk's list has been read
    while (true) {
        if (sm.w == 0) {
            walk_tree<false, true, SUB, CAP, DIAG>(sm, sm.t.leaves, a, r, on, seg_hi, K, cursor, s, lane);
            if (lane == 0) sm.t.walked = (unsigned)s.nc | (s.more ? 1u << 31 : 0u);
        }
        sm.sync();
        const int nl = (int)(sm.t.walked & 0xffffu);
        const bool more = sm.t.walked >> 31;
        // the cone test, 32 leaves per warp
        const ChunkSpan span = chunk_span(r, on, seg_hi);
        int nc = 0;
        for (int base = 0; base < nl; base += 32 * SUB) {
            const int l = base + 32 * sm.w + lane;
            const unsigned leaf = l < nl ? sm.t.leaves[l] : 0u;
            int first = 0;
            const bool may = l < nl && (int)leaf > cursor && cull<true, SUB, CAP>(sm, a, r.o, span, K, (int)leaf, first);
            const unsigned mm = __ballot_sync(kFull, may);
            if (lane == 0) sm.t.hits[sm.flip][sm.w] = mm;
            sm.sync();
            int at = nc;
#pragma unroll
            for (int q = 0; q < SUB; ++q) {
                const int n = __popc(sm.t.hits[sm.flip][q]);
                if (q < sm.w) at += n;
                nc += n;
            }
            sm.flip ^= 1;
            if (may) cand[at + __popc(mm & ((1u << lane) - 1u))] = leaf | ((unsigned)(first >> 1) << 25);
        }
        sm.sync();
        for (int done = 0; done < nc;) {
            const bool in = done + lane < nc;
            const unsigned c = in ? cand[done + lane] : 0u;
            const unsigned todo = __ballot_sync(kFull, in && 2 * (int)(c >> 25) < K);
            const unsigned left = team_batch<SUB, CAP, DIAG>(sm, a, r, on, seg_hi, K, nv, todo, c & kLeafMask, count, lane,
                                                             ws, infer);
            done += left ? __ffs(left) - 1 : 32;
            if (!left) continue;
            if (K == 1) {
                ovf = true;
                break;
            }
            // the list is full: shorten the chunk, test its entries again, then come back to this leaf
            K >>= 1;
            chunk_extent(r, on, K, t_end, nv, seg_hi);
            if (sm.w == 0) {
                if (lane == 0) atomicAdd(&a.st->chunk_splits, 1ull);
                set_packet<true, SUB, CAP>(sm, r, on, seg_hi, lane);
            }
            sm.sync();
            const int n = count;
            count = 0;
            for (int e = 0; e < n; e += 32) {
                const bool old = e + lane < n;
                const unsigned leaf = old ? (unsigned)sm.ids[e + lane] : 0u;
                const unsigned stay = __ballot_sync(kFull, old && (int)(sm.urng[e + lane] & 0xffffu) < K);
                team_batch<SUB, CAP, DIAG>(sm, a, r, on, seg_hi, K, nv, stay, leaf, count, lane, ws, infer);
            }
        }
        if (ovf || !more) break;
        // the leaves were many: those hit are in the list, the tree goes on
        s.nc = 0;
    }
    sm.sync();
    if (DIAG) ws.node_visits += s.visits;
    finish_list<true, SUB, CAP, DIAG>(sm, count, K, lane, ws);
    return count;
}

// The chunk list from the forward's record: the recorded leaves (at most the list capacity) get
// the same exact leaf test as in a traversal, without the traversal.
template <bool FAST, int SUB, int CAP, bool DIAG>
__device__ int replay_list(WarpSmem<FAST, SUB, CAP>& sm, const RenderArgs& a, const RayState& r, bool on, float seg_hi,
                           int K, int nv, const unsigned* ids, int n, int lane, WarpStats& ws) {
    int count = 0;
    n = min(n, CAP);
    for (int base = 0; base < n; base += 32) {
        const int mine = base + lane < n ? (int)ids[base + lane] : -1;
        unsigned todo = __ballot_sync(kFull, mine >= 0 && mine < a.n_leaves);
        while (todo) {
            const int leaf = next_leaf<SUB>(todo, (unsigned)mine, lane);
            leaf_batch<FAST, SUB, CAP, DIAG>(sm, a, r, on, seg_hi, K, nv, leaf, count, lane, ws, false);
#pragma unroll
            for (int i = 0; i < SUB; ++i) todo &= todo - 1u;
        }
    }
    finish_list<FAST, SUB, CAP, DIAG>(sm, count, K, lane, ws);
    return count;
}

// replay_list by a team.
template <int SUB, int CAP, bool DIAG>
__device__ int team_replay(WarpSmem<true, SUB, CAP>& sm, const RenderArgs& a, const RayState& r, bool on, float seg_hi,
                           int K, int nv, const unsigned* ids, int n, int lane, WarpStats& ws) {
    int count = 0;
    n = min(n, CAP);
    sm.sync();               // the last chunk's list has been read
    for (int base = 0; base < n; base += 32) {
        const int mine = base + lane < n ? (int)ids[base + lane] : -1;
        const unsigned todo = __ballot_sync(kFull, mine >= 0 && mine < a.n_leaves);
        team_batch<SUB, CAP, DIAG>(sm, a, r, on, seg_hi, K, nv, todo, (unsigned)mine, count, lane, ws, false);
    }
    sm.sync();
    finish_list<true, SUB, CAP, DIAG>(sm, count, K, lane, ws);
    return count;
}

// Per-slab sample offsets beyond i*dt (rnd_sample 1: random; 2+: half step).  Returns the seed
// after the slab's draws (used only when the slab had hits).
__device__ __forceinline__ unsigned slab_offsets(int rnd_sample, unsigned seed, float* roff) {
    if (rnd_sample == 1) {
#pragma unroll
        for (int i = 0; i < kBuf; ++i) roff[i] = lcg_rnd(seed) * kDt;
    } else {
#pragma unroll
        for (int i = 0; i < kBuf; ++i) roff[i] = (rnd_sample == 0) ? 0.f : 0.5f * kDt;
    }
    return seed;
}

// Parity arithmetic: the eight samples of a slab in four pairs (samples 2p and 2p + 1), each operation
// a packed one with the reference's rounding and order.  The unfused multiplies and adds are what the
// parity kernels spend their issue slots on, and a packed instruction does two of them.

// Sample times of a slab (the reference's order: tb + i dt, then the offset).
__device__ __forceinline__ void parity_times(float tb, int rnd_sample, const float* roff, f2* t) {
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
        t[p] = add2(dup2(tb), pk((float)(2 * p) * kDt, (float)(2 * p + 1) * kDt));
        if (rnd_sample) t[p] = add2(t[p], pk(roff[2 * p], roff[2 * p + 1]));
    }
}

// Sample positions o + t d of a slab, the same for all its Gaussians.
struct SlabPoints {
    f2 x[kPairs], y[kPairs], z[kPairs];
    __device__ __forceinline__ void set(const RayState& r, const f2* t, f2 nz) {
#pragma unroll
        for (int p = 0; p < kPairs; ++p) {
            x[p] = add2(dup2(r.o.x), mul2_rn(dup2(r.d.x), t[p], nz));
            y[p] = add2(dup2(r.o.y), mul2_rn(dup2(r.d.y), t[p], nz));
            z[p] = add2(dup2(r.o.z), mul2_rn(dup2(r.d.z), t[p], nz));
        }
    }
};

__device__ __forceinline__ f2 dot2_rn(f2 ax, f2 ay, f2 az, f2 bx, f2 by, f2 bz, f2 nz) {
    return add2(add2(mul2_rn(ax, bx, nz), mul2_rn(ay, by, nz)), mul2_rn(az, bz, nz));
}

// Reference-order weights exp(-|M (x - mu)|^2 / 2) of the slab's samples, zero for the samples whose
// density * weight does not exceed 0.1.  A sample whose density * weight lies within the
// exponential's error of 0.1 is decided with a correctly rounded weight, so that the decision is the
// one of the FP32 reference arithmetic.
__device__ __forceinline__ void parity_weights(const SlabPoints& sp, const LeafRec& rec, f2* w, f2 nz) {
    const f2 mx = dup2(-rec.a.x), my = dup2(-rec.a.y), mz = dup2(-rec.a.z), dn = dup2(rec.a.w);
    const f2 r0x = dup2(rec.r0.x), r0y = dup2(rec.r0.y), r0z = dup2(rec.r0.z);
    const f2 r1x = dup2(rec.r1.x), r1y = dup2(rec.r1.y), r1z = dup2(rec.r1.z);
    const f2 r2x = dup2(rec.r2.x), r2y = dup2(rec.r2.y), r2z = dup2(rec.r2.z);
    f2 q[kPairs], d[kPairs];
    float near = INFINITY;
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
        const f2 vx = add2(sp.x[p], mx), vy = add2(sp.y[p], my), vz = add2(sp.z[p], mz);
        const f2 m0 = dot2_rn(r0x, r0y, r0z, vx, vy, vz, nz), m1 = dot2_rn(r1x, r1y, r1z, vx, vy, vz, nz),
                 m2 = dot2_rn(r2x, r2y, r2z, vx, vy, vz, nz);
        q[p] = mul2(dup2(-0.5f), dot2_rn(m0, m1, m2, m0, m1, m2, nz));
        w[p] = pk(expf(lo2(q[p])), expf(hi2(q[p])));
        d[p] = mul2_rn(dn, w[p], nz);
        const f2 off = add2(d[p], dup2(-kSigThr));
        near = fminf(near, fminf(fabsf(lo2(off)), fabsf(hi2(off))));
    }
    if (near < 4e-8f) {
#pragma unroll
        for (int p = 0; p < kPairs; ++p) {
            if (fabsf(lo2(d[p]) - kSigThr) < 4e-8f) w[p] = pk(exp_exact(lo2(q[p])), hi2(w[p]));
            if (fabsf(hi2(d[p]) - kSigThr) < 4e-8f) w[p] = pk(lo2(w[p]), exp_exact(hi2(q[p])));
            d[p] = mul2_rn(dn, w[p], nz);
        }
    }
#pragma unroll
    for (int p = 0; p < kPairs; ++p)
        w[p] = pk(lo2(d[p]) > kSigThr ? lo2(w[p]) : 0.f, hi2(d[p]) > kSigThr ? hi2(w[p]) : 0.f);
}

__device__ __forceinline__ bool in_urange(unsigned u, int k) {
    return k >= (int)(u & 0xffff) && k <= (int)(u >> 16);
}

// Whether the lane's ray holds list entry e in its slab kl: the fast lists keep the rays whose interval
// meets the chunk, the parity lists each ray's exact slab range.
template <bool FAST, int SUB, int CAP>
__device__ __forceinline__ bool lane_has_entry(const WarpSmem<FAST, SUB, CAP>& sm, int e, int kl, int lane) {
    if constexpr (FAST) {
        if constexpr (SUB == 1) return (sm.lmask[e] >> lane) & 1u;
        else return ((sm.lmask[e] >> sm.slot) & 1u) && in_urange(sm.urng[e], kl);
    } else {
        const unsigned short rg = sm.lrng[e][lane / SUB];
        return kl >= (int)(rg & 0xff) && kl <= (int)(rg >> 8);
    }
}
// Whether an entry's union range meets the slabs k .. k + SUB - 1.
template <int SUB>
__device__ __forceinline__ bool meets_group(unsigned u, int k) {
    return k + SUB - 1 >= (int)(u & 0xffff) && k <= (int)(u >> 16);
}

// Sample buffers of a slab: density sums and, in the forward, the density-weighted colours; in the
// backward (GDOT), which needs the colour only through g . C, the sums of -(g . colour) * density (parity
// arithmetic) or of (g . colour) * density (fast).
template <bool FAST, bool GDOT>
struct SlabBuf {
    float sig[kBuf];
    float3 C[GDOT ? 1 : kBuf];
    float gC[GDOT ? kBuf : 1];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < kBuf; ++i) {
            sig[i] = 0.f;
            if constexpr (GDOT) gC[i] = 0.f;
            else C[i] = f3(0.f, 0.f, 0.f);
        }
    }
    __device__ __forceinline__ bool any_density() const {
        bool any = false;
#pragma unroll
        for (int i = 0; i < kBuf; ++i) any |= sig[i] > 0.f;
        return any;
    }
};
template <bool GDOT>
struct SlabBuf<false, GDOT> {
    f2 sig[kPairs];
    f2 cx[GDOT ? 1 : kPairs], cy[GDOT ? 1 : kPairs], cz[GDOT ? 1 : kPairs];
    f2 ng[GDOT ? kPairs : 1];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int p = 0; p < kPairs; ++p) {
            sig[p] = 0ull;
            if constexpr (GDOT) ng[p] = 0ull;
            else cx[p] = cy[p] = cz[p] = 0ull;
        }
    }
    // sums of densities are zero or positive: their bits are zero exactly where nothing was added
    __device__ __forceinline__ bool any_density() const { return (sig[0] | sig[1] | sig[2] | sig[3]) != 0ull; }
};
static_assert(kPairs == 4, "four sample pairs per slab");

// Sample buffers of slab k: the sums over the lane's hits.
template <bool FAST, int SUB, int CAP, bool GDOT, bool DIAG>
__device__ __forceinline__ int slab_buffers(const WarpSmem<FAST, SUB, CAP>& sm, int k, int K, bool has, const RayState& r,
                                            const RenderArgs& a, int rgb_base, const float* roff,
                                            SlabBuf<FAST, GDOT>& sb, int nw, int lane, WarpStats& ws) {
    int nh = 0;
    SlabPoints sp;
    if constexpr (!FAST) {
        f2 t[kPairs];
        parity_times(r.tb, a.rnd_sample, roff, t);
        sp.set(r, t, a.neg_zero);
    }
#pragma unroll 1
    for (int w = 0; w < nw; ++w) {
        unsigned mw = sm.smask[k / WarpSmem<FAST, SUB, CAP>::MB][w];
        while (mw) {
            const int e = 32 * w + __ffs(mw) - 1;
            mw &= mw - 1u;
            if (!meets_group<SUB>(sm.urng[e], k)) continue;
            if (DIAG) ++ws.entry_slabs;
            if (!has) continue;
            const int leaf = sm.ids[e];
            if (!lane_has_entry<FAST, SUB, CAP>(sm, e, k + lane % SUB, lane)) continue;
            LeafRec rec = load_rec(a.rec, leaf);
            float4 col4 = __ldg(a.rgb + rgb_base + leaf);
            float3 mu = f3(rec.a.x, rec.a.y, rec.a.z);
            float dn = rec.a.w;
            float3 r0 = f3(rec.r0.x, rec.r0.y, rec.r0.z), r1 = f3(rec.r1.x, rec.r1.y, rec.r1.z),
                   r2 = f3(rec.r2.x, rec.r2.y, rec.r2.z);
            ++nh;
            if constexpr (FAST) {
                // log2(dens * w_i) = log2(dens) - q_i log2(e) / 2, q_i quadratic in the sample index
                float3 v0 = (r.o + r.d * r.tb) - mu;
                float3 vb = r.d * kDt;
                float3 m0 = f3(dot3(r0, v0), dot3(r1, v0), dot3(r2, v0));
                float3 mb = f3(dot3(r0, vb), dot3(r1, vb), dot3(r2, vb));
                float A = fmaf(kNegHalfLog2e, dot3(m0, m0), rec.r1.w);   // r1.w = log2(dens)
                float B2 = (2.f * kNegHalfLog2e) * dot3(m0, mb), Cq = kNegHalfLog2e * dot3(mb, mb);
                float3 col = f3(col4.x, col4.y, col4.z);
                const float gcol = GDOT ? dot3(r.g, col) : 0.f;
#pragma unroll
                for (int i = 0; i < kBuf; ++i) {
                    float fi = (float)i;
                    float e = fmaf(fi, fmaf(fi, Cq, B2), A);
                    if (e > kLog2SigThr) {
                        float dw = ex2_approx(e);
                        sb.sig[i] += dw;
                        if constexpr (GDOT) sb.gC[i] = fmaf(gcol, dw, sb.gC[i]);
                        else sb.C[i] = sb.C[i] + col * dw;
                    }
                }
            } else {
                f2 w[kPairs];                  // weights, or density * weight (inference)
                const f2 dn2 = dup2(dn);
                const bool infer = !GDOT && a.infer;
                if (infer) {
                    // Inference programs (cuda_test/gaussians_aabb.cu:282-295, :501-515): the samples step
                    // through the scaled conic space from the slab start, m_{i+1} = m_i + dt * M d, and
                    // weight * density multiplies the colour.  Reference operation order.
                    const LeafIS is = load_is(a.is_rec, leaf);
                    const float kf = is.u.w;   // sqrt(log(ratio^2)) of the Gaussian
                    const float3 U = f3(is.u.x, is.u.y, is.u.z), V = f3(is.v.x, is.v.y, is.v.z),
                                 W = f3(is.w.x, is.w.y, is.w.z);
                    const float3 xg = f3(__fsub_rn(__fadd_rn(r.o.x, __fmul_rn(r.tb, r.d.x)), mu.x),
                                         __fsub_rn(__fadd_rn(r.o.y, __fmul_rn(r.tb, r.d.y)), mu.y),
                                         __fsub_rn(__fadd_rn(r.o.z, __fmul_rn(r.tb, r.d.z)), mu.z));
                    float3 m = f3(__fmul_rn(dot_rn(U, xg), kf), __fmul_rn(dot_rn(V, xg), kf),
                                  __fmul_rn(dot_rn(W, xg), kf));
                    const float3 mdt = f3(__fmul_rn(__fmul_rn(dot_rn(U, r.d), kf), kDt),
                                          __fmul_rn(__fmul_rn(dot_rn(V, r.d), kf), kDt),
                                          __fmul_rn(__fmul_rn(dot_rn(W, r.d), kf), kDt));
                    float near = INFINITY;
                    f2 q[kPairs];
#pragma unroll
                    for (int p = 0; p < kPairs; ++p) {
                        const float3 n = f3(__fadd_rn(m.x, mdt.x), __fadd_rn(m.y, mdt.y), __fadd_rn(m.z, mdt.z));
                        const f2 mx = pk(m.x, n.x), my = pk(m.y, n.y), mz = pk(m.z, n.z);
                        q[p] = mul2(dup2(-0.5f), dot2_rn(mx, my, mz, mx, my, mz, a.neg_zero));
                        w[p] = mul2_rn(pk(expf(lo2(q[p])), expf(hi2(q[p]))), dn2, a.neg_zero);
                        const f2 off = add2(w[p], dup2(-kSigThr));
                        near = fminf(near, fminf(fabsf(lo2(off)), fabsf(hi2(off))));
                        m = f3(__fadd_rn(n.x, mdt.x), __fadd_rn(n.y, mdt.y), __fadd_rn(n.z, mdt.z));
                    }
                    if (near < 4e-8f) {
#pragma unroll
                        for (int p = 0; p < kPairs; ++p) {
                            if (fabsf(lo2(w[p]) - kSigThr) < 4e-8f)
                                w[p] = pk(__fmul_rn(exp_exact(lo2(q[p])), dn), hi2(w[p]));
                            if (fabsf(hi2(w[p]) - kSigThr) < 4e-8f)
                                w[p] = pk(lo2(w[p]), __fmul_rn(exp_exact(hi2(q[p])), dn));
                        }
                    }
#pragma unroll
                    for (int p = 0; p < kPairs; ++p)
                        w[p] = pk(lo2(w[p]) > kSigThr ? lo2(w[p]) : 0.f, hi2(w[p]) > kSigThr ? hi2(w[p]) : 0.f);
                } else {
                    parity_weights(sp, rec, w, a.neg_zero);
                }
                if constexpr (GDOT) {
                    const float ngcol = -(r.g.x * col4.x + r.g.y * col4.y + r.g.z * col4.z);
                    if (fabsf(ngcol) < INFINITY) {
#pragma unroll
                        for (int p = 0; p < kPairs; ++p) {
                            sb.sig[p] = add2(sb.sig[p], mul2_rn(dn2, w[p], a.neg_zero));
                            sb.ng[p] = fma2(dup2(ngcol), mul2(w[p], dn2), sb.ng[p]);
                        }
                    } else {
                        // not finite: 0 * inf must not reach the samples under the threshold
#pragma unroll
                        for (int p = 0; p < kPairs; ++p) {
                            const f2 dw = mul2_rn(dn2, w[p], a.neg_zero);
                            sb.sig[p] = add2(sb.sig[p], dw);
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                                if (half2(dw, h) > 0.f)
                                    sb.ng[p] = with_half2(sb.ng[p], h, fmaf(ngcol, half2(dw, h), half2(sb.ng[p], h)));
                        }
                    }
                } else {
#pragma unroll
                    for (int p = 0; p < kPairs; ++p) {
                        // inference: colour * (weight * density); training: (colour * weight) * density
                        const f2 dw = infer ? w[p] : mul2_rn(dn2, w[p], a.neg_zero);
                        const f2 one = infer ? dup2(1.f) : dn2;
                        sb.sig[p] = add2(sb.sig[p], dw);
                        const f2 cx = mul2_rn(mul2(dup2(col4.x), w[p]), one, a.neg_zero),
                                 cy = mul2_rn(mul2(dup2(col4.y), w[p]), one, a.neg_zero),
                                 cz = mul2_rn(mul2(dup2(col4.z), w[p]), one, a.neg_zero);
                        if (col4.w == 0.f) {
                            sb.cx[p] = add2(sb.cx[p], cx);
                            sb.cy[p] = add2(sb.cy[p], cy);
                            sb.cz[p] = add2(sb.cz[p], cz);
                        } else {
                            // a colour that is not finite
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                                if (half2(dw, h) > 0.f) {
                                    sb.cx[p] = with_half2(sb.cx[p], h, __fadd_rn(half2(sb.cx[p], h), half2(cx, h)));
                                    sb.cy[p] = with_half2(sb.cy[p], h, __fadd_rn(half2(sb.cy[p], h), half2(cy, h)));
                                    sb.cz[p] = with_half2(sb.cz[p], h, __fadd_rn(half2(sb.cz[p], h), half2(cz, h)));
                                }
                        }
                    }
                }
            }
        }
    }
    return nh;
}

__device__ __forceinline__ float exp_neg_fast(float x) { return ex2_approx(-x * 1.4426950408889634f); }

// Opacities 1 - exp(-sig dt) of a slab's samples, in pairs.
template <bool FAST, bool GDOT>
__device__ __forceinline__ void slab_alpha(const SlabBuf<FAST, GDOT>& sb, f2* alpha, f2 nz) {
    if constexpr (FAST) {
#pragma unroll
        for (int p = 0; p < kPairs; ++p)
            alpha[p] = pk(1.f - exp_neg_fast(sb.sig[2 * p] * kDt), 1.f - exp_neg_fast(sb.sig[2 * p + 1] * kDt));
    } else {
        f2 ex[kPairs];
        exp_neg_slab(sb.sig, ex, nz);
#pragma unroll
        for (int p = 0; p < kPairs; ++p) alpha[p] = fma2(ex[p], dup2(-1.f), dup2(1.f));
    }
}

// Alpha compositing of one slab's 8 samples (forward/gaussians_aabb.cu:500-519).  A slab whose
// samples all fell under the threshold composites to exactly nothing (alpha = 1 - exp(0) = 0).
template <bool FAST>
__device__ __forceinline__ void composite(RayState& r, const SlabBuf<FAST, false>& sb, const f2* alpha, f2 nz) {
    if (!sb.any_density()) return;
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
        const f2 om = fma2(alpha[p], dup2(-1.f), dup2(1.f));
        if constexpr (FAST) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                // C[i] is zero wherever sig[i] is (both sum the same above-threshold samples)
                const int i = 2 * p + h;
                const float s = sb.sig[i] > 0.f ? __fdividef(r.T * half2(alpha[p], h), sb.sig[i]) : 0.f;
                r.C = r.C + sb.C[i] * s;
                r.T *= half2(om, h);
            }
        } else {
            const float s0 = lo2(sb.sig[p]), s1 = hi2(sb.sig[p]);
            const f2 inv = pk(s0 > 0.f ? __frcp_rn(s0) : 0.f, s1 > 0.f ? __frcp_rn(s1) : 0.f);   // colours are 0 there
            const float T1 = __fmul_rn(r.T, lo2(om));
            const f2 ta = mul2_rn(pk(r.T, T1), alpha[p], nz);
            const f2 cx = mul2_rn(mul2(sb.cx[p], inv), ta, nz), cy = mul2_rn(mul2(sb.cy[p], inv), ta, nz),
                     cz = mul2_rn(mul2(sb.cz[p], inv), ta, nz);
            r.C = f3(__fadd_rn(__fadd_rn(r.C.x, lo2(cx)), hi2(cx)), __fadd_rn(__fadd_rn(r.C.y, lo2(cy)), hi2(cy)),
                     __fadd_rn(__fadd_rn(r.C.z, lo2(cz)), hi2(cz)));
            r.T = __fmul_rn(T1, hi2(om));
        }
    }
}

__device__ __forceinline__ float4 quat_grad(float4 q, float3 d1, float3 d2, float3 d3) {
    // derivative of the (not normalised) polynomial rotation columns w.r.t. (r, i, j, k)
    float r = q.x, i = q.y, j = q.z, k = q.w;
    float4 o;
    o.x = 2.f * (k * d1.y - j * d1.z - k * d2.x + i * d2.z + j * d3.x - i * d3.y);
    o.y = 2.f * (j * d1.y + k * d1.z + j * d2.x - 2.f * i * d2.y + r * d2.z + k * d3.x - r * d3.y - 2.f * i * d3.z);
    o.z = 2.f * (-2.f * j * d1.x + i * d1.y - r * d1.z + i * d2.x + k * d2.z + r * d3.x + k * d3.y - 2.f * j * d3.z);
    o.w = 2.f * (-2.f * k * d1.x + r * d1.y + i * d1.z - r * d2.x - 2.f * k * d2.y + j * d2.z + i * d3.x + j * d3.y);
    return o;
}

// Transposed warp reduction of 16 values: afterwards lane l holds the warp sum of value
// 8*b4 + 4*b3 + 2*b2 + b1 (b_i = bit i of l); lanes l and l^1 hold the same value.
__device__ __forceinline__ float transpose_reduce16(float* v, int lane) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        bool up = lane & 16;
        float send = up ? v[i] : v[i + 8];
        float keep = up ? v[i + 8] : v[i];
        v[i] = keep + __shfl_xor_sync(kFull, send, 16);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        bool up = lane & 8;
        float send = up ? v[i] : v[i + 4];
        float keep = up ? v[i + 4] : v[i];
        v[i] = keep + __shfl_xor_sync(kFull, send, 8);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        bool up = lane & 4;
        float send = up ? v[i] : v[i + 2];
        float keep = up ? v[i + 2] : v[i];
        v[i] = keep + __shfl_xor_sync(kFull, send, 4);
    }
    {
        bool up = lane & 2;
        float send = up ? v[0] : v[1];
        float keep = up ? v[1] : v[0];
        v[0] = keep + __shfl_xor_sync(kFull, send, 2);
    }
    v[0] += __shfl_xor_sync(kFull, v[0], 1);
    return v[0];
}

// Compositing adjoint scalars of a slab's samples (slab_adjoint_scalars).
template <bool FAST>
struct AdjBuf {
    float H[kBuf], F[kBuf];
};
template <>
struct AdjBuf<false> {
    f2 H[kPairs], F[kPairs];
};

// Adjoint of slab k for all list entries: per-lane gradient of each hit Gaussian, warp reduction,
// one atomic per value.  Value order: ddens, S1.xyz, M2 (xx yy zz xy xz yz), 0, drgb.xyz.
template <bool FAST, int SUB, int CAP, bool DIAG>
__device__ __forceinline__ void slab_adjoint(const WarpSmem<FAST, SUB, CAP>& sm, int k, int K, bool has, const RayState& r,
                                             const RenderArgs& a, int rgb_base, const float* roff,
                                             const AdjBuf<FAST>& ad, int nw, int lane,
                                             WarpStats& ws, int view) {
    SlabPoints sp;
    f2 xt[kPairs];   // parity: sample times from the slab's start
    if constexpr (!FAST) {
        parity_times(r.tb, a.rnd_sample, roff, xt);
        sp.set(r, xt, a.neg_zero);
#pragma unroll
        for (int p = 0; p < kPairs; ++p) xt[p] = add2(xt[p], dup2(-r.tb));
    }
    const int vid = ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
#pragma unroll 1
    for (int w = 0; w < nw; ++w) {
      unsigned mw = sm.smask[k / WarpSmem<FAST, SUB, CAP>::MB][w];
      while (mw) {
        const int e = 32 * w + __ffs(mw) - 1;
        mw &= mw - 1u;
        if (!meets_group<SUB>(sm.urng[e], k)) continue;
        const int leaf = sm.ids[e];
        if (DIAG) ++ws.entry_slabs;
        bool act = has && lane_has_entry<FAST, SUB, CAP>(sm, e, k + lane % SUB, lane);
        unsigned am = __ballot_sync(kFull, act);
        if (am == 0u) continue;
        float v[16];
#pragma unroll
        for (int z = 0; z < 16; ++z) v[z] = 0.f;
        if (act) {
            LeafRec rec = load_rec(a.rec, leaf);
            float4 col4 = __ldg(a.rgb + rgb_base + leaf);
            float3 mu = f3(rec.a.x, rec.a.y, rec.a.z);
            float dn = rec.a.w;
            float3 r0 = f3(rec.r0.x, rec.r0.y, rec.r0.z), r1 = f3(rec.r1.x, rec.r1.y, rec.r1.z),
                   r2 = f3(rec.r2.x, rec.r2.y, rec.r2.z);
            float gcol = r.g.x * col4.x + r.g.y * col4.y + r.g.z * col4.z;
            float gc = 0.f, dd = 0.f;
            // Moment form.  With the sample offsets from the Gaussian v_i = v0 + x_i vb, every
            // geometric gradient of this (ray, Gaussian, slab) is linear in the ray-independent
            // moments S1 = sum_i u_i v_i and M2 = sum_i u_i v_i v_i^T (u_i = dens * h_i * w_i), which
            // follow from U_k = sum_i u_i x_i^k (k = 0, 1, 2).  The moments of all rays and slabs are
            // summed per Gaussian and turned into position/scale/rotation gradients once per
            // Gaussian afterwards (k_moment_grads).  Fast arithmetic: x_i = i, vb = dt * dir.  Parity:
            // x_i = t_i - tb, vb = dir (random sample offsets included), the reference's weights and
            // threshold decisions.
            const float3 v0 = (r.o + r.d * r.tb) - mu;
            const float3 vb = FAST ? r.d * kDt : r.d;
            float U0 = 0.f, U1 = 0.f, U2 = 0.f;
            if constexpr (FAST) {
                // dw_i = dens * w_i in the exponent domain (as in the forward); accumulates
                // sum dw F, sum dw h and the moments of u = dw h, then divides by dens once
                const float3 m0 = f3(dot3(r0, v0), dot3(r1, v0), dot3(r2, v0));
                const float3 mb = f3(dot3(r0, vb), dot3(r1, vb), dot3(r2, vb));
                float A = fmaf(kNegHalfLog2e, dot3(m0, m0), rec.r1.w);   // r1.w = log2(dens)
                float B2 = (2.f * kNegHalfLog2e) * dot3(m0, mb), Cq = kNegHalfLog2e * dot3(mb, mb);
#pragma unroll
                for (int i = 0; i < kBuf; ++i) {
                    float fi = (float)i;
                    float e = fmaf(fi, fmaf(fi, Cq, B2), A);
                    if (e > kLog2SigThr) {
                        float dw = ex2_approx(e);
                        float u = fmaf(ad.F[i], gcol, ad.H[i]) * dw;
                        gc = fmaf(dw, ad.F[i], gc);
                        U0 += u;
                        U1 = fmaf(fi, u, U1);
                        U2 = fmaf(fi * fi, u, U2);
                    }
                }
                dd = (U0 != 0.f) ? U0 * rec.r2.w : 0.f;                   // r2.w = 1 / dens
            } else {
                f2 w[kPairs];
                parity_weights(sp, rec, w, a.neg_zero);
                f2 gc2 = 0ull, s0 = 0ull, s1 = 0ull, s2 = 0ull;
#pragma unroll
                for (int p = 0; p < kPairs; ++p) {
                    const f2 u = mul2(fma2(ad.F[p], dup2(gcol), ad.H[p]), w[p]);
                    gc2 = fma2(w[p], ad.F[p], gc2);
                    s0 = add2(s0, u);
                    s1 = fma2(xt[p], u, s1);
                    s2 = fma2(mul2(xt[p], xt[p]), u, s2);
                }
                gc = lo2(gc2) + hi2(gc2);
                U0 = lo2(s0) + hi2(s0);
                U1 = lo2(s1) + hi2(s1);
                U2 = lo2(s2) + hi2(s2);
                if (!(fabsf(U0) + fabsf(U1) + fabsf(U2) + fabsf(gc) < INFINITY)) {
                    // not finite: take in only the samples above the threshold
                    gc = U0 = U1 = U2 = 0.f;
#pragma unroll
                    for (int i = 0; i < kBuf; ++i) {
                        const float wt = half2(w[i >> 1], i & 1), x = half2(xt[i >> 1], i & 1);
                        if (wt > 0.f) {
                            const float Fi = half2(ad.F[i >> 1], i & 1);
                            const float u = fmaf(Fi, gcol, half2(ad.H[i >> 1], i & 1)) * wt;
                            gc += wt * Fi;
                            U0 += u;
                            U1 += x * u;
                            U2 += x * x * u;
                        }
                    }
                }
                dd = U0;
                gc *= dn;
                U0 *= dn; U1 *= dn; U2 *= dn;
            }
            // S1 = v0 U0 + vb U1; M2 = v0 v0^T U0 + (v0 vb^T + vb v0^T) U1 + vb vb^T U2
            const float3 p = v0 * U0 + vb * U1;     // sum u v
            const float3 q = v0 * U1 + vb * U2;     // sum u x v
            v[0] = dd;
            v[1] = p.x; v[2] = p.y; v[3] = p.z;
            v[4] = v0.x * p.x + vb.x * q.x;         // xx
            v[5] = v0.y * p.y + vb.y * q.y;         // yy
            v[6] = v0.z * p.z + vb.z * q.z;         // zz
            v[7] = v0.x * p.y + vb.x * q.y;         // xy
            v[8] = v0.x * p.z + vb.x * q.z;         // xz
            v[9] = v0.y * p.z + vb.y * q.z;         // yz
            v[11] = r.g.x * gc; v[12] = r.g.y * gc; v[13] = r.g.z * gc;
        }
        float* gg = reinterpret_cast<float*>(a.gacc_geo + 3 * (long long)leaf);
        float* gr = reinterpret_cast<float*>(a.gacc_rgb + (long long)leaf * a.n_views + view);
        // lanes whose samples all fell under the threshold contribute nothing
        const bool nz = act && (v[0] != 0.f || v[1] != 0.f || v[2] != 0.f || v[3] != 0.f || v[11] != 0.f ||
                                v[12] != 0.f || v[13] != 0.f);
        const unsigned zm = __ballot_sync(kFull, nz);
        if (zm == 0u) continue;
        if (__popc(zm) <= (SUB == 1 ? RG_DIRECT_ATOMIC_LANES : RG_SPLIT_DIRECT_ATOMIC_LANES)) {
            if (nz) {
                float4* g4 = reinterpret_cast<float4*>(gg);
                atomicAdd(g4, make_float4(v[0], v[1], v[2], v[3]));
                atomicAdd(g4 + 1, make_float4(v[4], v[5], v[6], v[7]));
                atomicAdd(g4 + 2, make_float4(v[8], v[9], v[10], 0.f));
                atomicAdd(reinterpret_cast<float4*>(gr), make_float4(v[11], v[12], v[13], 0.f));
            }
        } else {
            float s = transpose_reduce16(v, lane);
            if (!(lane & 1) && vid < 14) {
                if (vid < 11) atomicAdd(gg + vid, s);
                else atomicAdd(gr + (vid - 11), s);
            }
        }
      }
    }
}

// Per-sample compositing adjoint scalars of one slab (reference backward :675-730): with
// E = g.((T c - R) dt), F = T alpha / sigma and G = g.c, a Gaussian of colour col and weight w
// at the sample has dL/d(sigma-share) h = E + F (g.col - G) = F g.col + H, H = E - F G.  Only
// g.C (gC, C the colour sum of the sample) and g.R (r.gR) enter: with gc = g.C / sigma,
// E = dt (T gc - g.R), H = E - F gc, and g.R drops by gc T alpha per sample.
// Returns H and F; advances T and g.R over the slab.
template <bool FAST>
__device__ __forceinline__ void slab_adjoint_scalars(const RayState& r, const SlabBuf<FAST, true>& sb, const f2* alpha,
                                                     AdjBuf<FAST>& ad, float& Ta, float& gRa, f2 nz) {
    Ta = r.T;
    gRa = r.gR;
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
        const f2 om = fma2(alpha[p], dup2(-1.f), dup2(1.f));
        if constexpr (FAST) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = 2 * p + h;
                const float cd = sb.sig[i];
                float inv = 0.f;
                if (cd > 0.f) inv = __fdividef(1.f, cd);
                const float gc = sb.gC[i] * inv;
                const float ta = Ta * half2(alpha[p], h);
                ad.F[i] = ta * inv;
                ad.H[i] = kDt * (Ta * gc - gRa) - ad.F[i] * gc;
                gRa -= gc * ta;
                Ta = Ta * half2(om, h);
            }
        } else {
            const float s0 = lo2(sb.sig[p]), s1 = hi2(sb.sig[p]);
            const f2 inv = pk(s0 > 0.f ? __frcp_rn(s0) : 0.f, s1 > 0.f ? __frcp_rn(s1) : 0.f);
            const float T1 = __fmul_rn(Ta, lo2(om));
            const f2 T2 = pk(Ta, T1), ngc = mul2(sb.ng[p], inv), ta = mul2(T2, alpha[p]);   // ngc = -g.C / sigma
            ad.F[p] = mul2(ta, inv);
            const float gR1 = fmaf(lo2(ngc), lo2(ta), gRa);
            ad.H[p] = fma2(ad.F[p], ngc, mul2(fma2(T2, ngc, pk(gRa, gR1)), dup2(-kDt)));
            gRa = fmaf(hi2(ngc), hi2(ta), gR1);
            Ta = __fmul_rn(T1, hi2(om));
        }
    }
}

// The slabs of a group (SUB > 1) in turn: the transmittance runs through them lane by lane, by the same
// multiplications in the same order as slab after slab.  `has` (the lane marches its slab, as far as
// its place on the ray goes) loses the lanes whose ray ended before (T <= 0.003); returns the
// transmittance at the lane's start and leaves the group's end in r.T.
template <int SUB>
__device__ __forceinline__ float group_transmittance(RayState& r, const f2* alpha, bool dense, bool& has, int lane) {
    float T = r.T, mine = r.T;
#pragma unroll
    for (int q = 0; q < SUB; ++q) {
        if (lane % SUB == q) {
            mine = T;
            has = has && T > kTeps;
            if (has && dense) {
#pragma unroll
                for (int p = 0; p < kPairs; ++p) {
                    const f2 om = fma2(alpha[p], dup2(-1.f), dup2(1.f));
                    T = __fmul_rn(__fmul_rn(T, lo2(om)), hi2(om));
                }
            }
        }
        T = __shfl_sync(kFull, T, lane / SUB * SUB + q);
    }
    r.T = T;
    return mine;
}

// composite for the slabs of a group: the terms of a lane's samples side by side, then added to the ray's
// colour in turn.  `act`: the lane's slab counts; r.T is the transmittance at its start.
template <bool FAST, int SUB>
__device__ __forceinline__ void group_colour(RayState& r, const SlabBuf<FAST, false>& sb, const f2* alpha, bool act, int lane,
                                             f2 nz) {
    float w[kBuf];                       // fast: weight of a sample's colour sum
    f2 cx[kPairs], cy[kPairs], cz[kPairs];   // parity: the terms
    float T = r.T;
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
        const f2 om = fma2(alpha[p], dup2(-1.f), dup2(1.f));
        if constexpr (FAST) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = 2 * p + h;
                w[i] = sb.sig[i] > 0.f ? __fdividef(T * half2(alpha[p], h), sb.sig[i]) : 0.f;
                T *= half2(om, h);
            }
        } else {
            const float s0 = lo2(sb.sig[p]), s1 = hi2(sb.sig[p]);
            const f2 inv = pk(s0 > 0.f ? __frcp_rn(s0) : 0.f, s1 > 0.f ? __frcp_rn(s1) : 0.f);
            const float T1 = __fmul_rn(T, lo2(om));
            const f2 ta = mul2_rn(pk(T, T1), alpha[p], nz);
            cx[p] = mul2_rn(mul2(sb.cx[p], inv), ta, nz);
            cy[p] = mul2_rn(mul2(sb.cy[p], inv), ta, nz);
            cz[p] = mul2_rn(mul2(sb.cz[p], inv), ta, nz);
            T = __fmul_rn(T1, hi2(om));
        }
    }
#pragma unroll
    for (int q = 0; q < SUB; ++q) {
        if (lane % SUB == q && act) {
            if constexpr (FAST) {
#pragma unroll
                for (int i = 0; i < kBuf; ++i)
                    r.C = f3(fmaf(sb.C[i].x, w[i], r.C.x), fmaf(sb.C[i].y, w[i], r.C.y), fmaf(sb.C[i].z, w[i], r.C.z));
            } else {
#pragma unroll
                for (int p = 0; p < kPairs; ++p)
                    r.C = f3(__fadd_rn(__fadd_rn(r.C.x, lo2(cx[p])), hi2(cx[p])),
                             __fadd_rn(__fadd_rn(r.C.y, lo2(cy[p])), hi2(cy[p])),
                             __fadd_rn(__fadd_rn(r.C.z, lo2(cz[p])), hi2(cz[p])));
            }
        }
        const int from = lane / SUB * SUB + q;
        r.C = f3(__shfl_sync(kFull, r.C.x, from), __shfl_sync(kFull, r.C.y, from), __shfl_sync(kFull, r.C.z, from));
    }
}

// slab_adjoint_scalars for the slabs of a group: what does not hold g . R side by side, then g . R through
// them in turn.  Returns it at the group's end.
template <bool FAST, int SUB>
__device__ __forceinline__ float group_adjoint_scalars(const RayState& r, const SlabBuf<FAST, true>& sb, const f2* alpha,
                                                       bool act, AdjBuf<FAST>& ad, int lane) {
    float g[kBuf], x[kBuf];             // -g.C / sigma; T alpha, then g . R at the sample
    float T = r.T;
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
        const f2 om = fma2(alpha[p], dup2(-1.f), dup2(1.f));
        if constexpr (FAST) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = 2 * p + h;
                const float cd = sb.sig[i];
                float inv = 0.f;
                if (cd > 0.f) inv = __fdividef(1.f, cd);
                g[i] = -(sb.gC[i] * inv);
                x[i] = T * half2(alpha[p], h);
                ad.F[i] = x[i] * inv;
                T = T * half2(om, h);
            }
        } else {
            const float s0 = lo2(sb.sig[p]), s1 = hi2(sb.sig[p]);
            const f2 inv = pk(s0 > 0.f ? __frcp_rn(s0) : 0.f, s1 > 0.f ? __frcp_rn(s1) : 0.f);
            const float T1 = __fmul_rn(T, lo2(om));
            const f2 ngc = mul2(sb.ng[p], inv), ta = mul2(pk(T, T1), alpha[p]);
            ad.F[p] = mul2(ta, inv);
            g[2 * p] = lo2(ngc);
            g[2 * p + 1] = hi2(ngc);
            x[2 * p] = lo2(ta);
            x[2 * p + 1] = hi2(ta);
            T = __fmul_rn(T1, hi2(om));
        }
    }
    float run = r.gR;
#pragma unroll
    for (int q = 0; q < SUB; ++q) {
        if (lane % SUB == q && act) {
#pragma unroll
            for (int i = 0; i < kBuf; ++i) {
                const float at = run;
                run = fmaf(g[i], x[i], run);
                x[i] = at;
            }
        }
        run = __shfl_sync(kFull, run, lane / SUB * SUB + q);
    }
    T = r.T;
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
        const f2 om = fma2(alpha[p], dup2(-1.f), dup2(1.f));
        if constexpr (FAST) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = 2 * p + h;
                ad.H[i] = ad.F[i] * g[i] - kDt * (T * g[i] + x[i]);
                T = T * half2(om, h);
            }
        } else {
            const float T1 = __fmul_rn(T, lo2(om));
            const f2 ngc = pk(g[2 * p], g[2 * p + 1]), gR = pk(x[2 * p], x[2 * p + 1]);
            ad.H[p] = fma2(ad.F[p], ngc, mul2(fma2(pk(T, T1), ngc, gR), dup2(-kDt)));
            T = __fmul_rn(T1, hi2(om));
        }
    }
    return run;
}

// Resident blocks per SM each kernel is compiled for (0: the compiler's choice).  The fast defaults
// fit the shared memory of the 64-entry tuning (256-entry fast lists) and were measured best on
// 1M Gaussians x 16 views.  The parity kernels want registers for the slab's points and sums rather
// than warps (300k-Gaussian object, forward / backward: 12.8 / 24.7 ms at 4 blocks, 128 registers and
// 400 B of spills; 12.3 / 22.5 at 3; 13.4 / 22.2 at 2, without spills).  Split tiles come in launches whose
// warps do not fill the chip, so registers cost nothing (three views of 60k Gaussians on whole tiles, fast,
// per step: 8.9 ms at 7 blocks, 7.8 at 4, 7.7 at 3).
#ifndef RG_FAST_FWD_MIN_BLOCKS
#define RG_FAST_FWD_MIN_BLOCKS 7
#endif
#ifndef RG_FAST_BWD_MIN_BLOCKS
#define RG_FAST_BWD_MIN_BLOCKS 7
#endif
#ifndef RG_PAR_FWD_MIN_BLOCKS
#define RG_PAR_FWD_MIN_BLOCKS 3
#endif
#ifndef RG_PAR_BWD_MIN_BLOCKS
#define RG_PAR_BWD_MIN_BLOCKS 2
#endif
#ifndef RG_FAST_SPLIT_FWD_MIN_BLOCKS
#define RG_FAST_SPLIT_FWD_MIN_BLOCKS 4
#endif
#ifndef RG_FAST_SPLIT_BWD_MIN_BLOCKS
#define RG_FAST_SPLIT_BWD_MIN_BLOCKS 4
#endif
#ifndef RG_PAR_SPLIT_FWD_MIN_BLOCKS
#define RG_PAR_SPLIT_FWD_MIN_BLOCKS 3
#endif
#ifndef RG_PAR_SPLIT_BWD_MIN_BLOCKS
#define RG_PAR_SPLIT_BWD_MIN_BLOCKS 3
#endif
template <bool BWD, bool FAST, int SUB>
constexpr int min_blocks() {
    if (SUB > 1)
        return FAST ? (BWD ? RG_FAST_SPLIT_BWD_MIN_BLOCKS : RG_FAST_SPLIT_FWD_MIN_BLOCKS)
                    : (BWD ? RG_PAR_SPLIT_BWD_MIN_BLOCKS : RG_PAR_SPLIT_FWD_MIN_BLOCKS);
    return FAST ? (BWD ? RG_FAST_BWD_MIN_BLOCKS : RG_FAST_FWD_MIN_BLOCKS)
                : (BWD ? RG_PAR_BWD_MIN_BLOCKS : RG_PAR_FWD_MIN_BLOCKS);
}

// DIAG: also count node visits, leaf tests, list entries, slab steps and entry-slabs (rg_status);
// without it those counters compile away and the kernel holds fewer live registers.
template <bool BWD, bool FAST, int SUB, int CAP, bool DIAG>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, min_blocks<BWD, FAST, SUB>()) k_render(RenderArgs a) {
    using SM = WarpSmem<FAST, SUB, CAP>;
    constexpr bool TEAM = FAST && SUB > 1;   // the list is the one of a whole tile's rays, shared by SUB warps
    __shared__ typename SM::Store smem[SM::kStores];
    const int lane = threadIdx.x & 31;
    decltype(auto) sm = SM::of(smem, threadIdx.x >> 5, lane);
    const ViewTable* vt = a.views;
    if (vt->split != SUB) return;
    const float bg = a.white_bg ? 1.f : 0.f;
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < kCounters; ++c) sm.cnt[c] = 0ull;
    }
    const int kmax =
        min((a.rnd_sample == 1) ? min(a.chunk_slabs, kExactChunk) : a.chunk_slabs, WarpSmem<FAST, SUB, CAP>::KM);

    while (true) {
        int tile = 0;
        if constexpr (TEAM) {
            // (a team may pass a tile without a barrier: the two places alternate)
            if (sm.w == 0 && lane == 0) sm.t.tile[sm.tile_flip] = atomicAdd(a.work_counter, 1);
            sm.sync();
            tile = sm.t.tile[sm.tile_flip];
            sm.tile_flip ^= 1;
        } else {
            if (lane == 0) tile = atomicAdd(a.work_counter, 1);
            tile = __shfl_sync(kFull, tile, 0);
        }
        if (tile >= vt->total_tiles) break;
        // view of this tile (binary search over the tile prefix)
        int lo = 0, hi = vt->n_views - 1;
        while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (vt->tile_prefix[mid] <= tile) lo = mid; else hi = mid - 1;
        }
        const int view = lo;
        const rg_camera cam = a.cams[view];
        const int W = cam.width, H = cam.height;
        using TS = TileShape<TEAM ? 1 : SUB>;
        const int tiles_x = (W + TS::w - 1) / TS::w;
        const int local = tile - vt->tile_prefix[view];
        const int ray = lane / SUB, sub = lane % SUB;
        const int pixel = TEAM ? lane : ray;
        const int px = (local % tiles_x) * TS::w + pixel % TS::w;
        const int py = (local / tiles_x) * TS::h + pixel / TS::w;
        bool valid = px < W && py < H;
        unsigned ray_l = (unsigned)(py * W + px);
        const int rgb_base = view * a.n_leaves;   // views x leaves < 2^31 (checked by the host)

        RayState r;
        WarpStats ws;
        unsigned hits_acc = 0, slabs_acc = 0;   // this lane's (slab, Gaussian) pairs and slabs
        r.seed = tea4(a.iteration, ray_l);
        {
            // computeRay (forward/gaussians_aabb.cu:405-434) in IEEE operation order
            float ix, iy;
            if (a.jitter == 1) {
                float jx = lcg_rnd(r.seed) * 0.333333f;
                float jy = lcg_rnd(r.seed) * 0.333333f;
                ix = __fdiv_rn(__fadd_rn(__fadd_rn((float)(ray_l % (unsigned)W), 0.333333f), jx), (float)W);
                iy = __fdiv_rn(__fadd_rn(__fadd_rn((float)(ray_l / (unsigned)W), 0.333333f), jy), (float)H);
            } else {
                ix = __fdiv_rn(__fadd_rn((float)(ray_l % (unsigned)W), 0.5f), (float)W);
                iy = __fdiv_rn(__fadd_rn((float)(ray_l / (unsigned)W), 0.5f), (float)H);
            }
            float dx = __fmul_rn(__fsub_rn(__fmul_rn(2.f, ix), 1.f), cam.tan_half_fovx);
            float dy = __fmul_rn(__fsub_rn(__fmul_rn(2.f, iy), 1.f), cam.tan_half_fovy);
            float3 dir = f3(__fadd_rn(__fadd_rn(__fmul_rn(cam.u[0], dx), __fmul_rn(cam.v[0], dy)), cam.w[0]),
                            __fadd_rn(__fadd_rn(__fmul_rn(cam.u[1], dx), __fmul_rn(cam.v[1], dy)), cam.w[1]),
                            __fadd_rn(__fadd_rn(__fmul_rn(cam.u[2], dx), __fmul_rn(cam.v[2], dy)), cam.w[2]));
            float inv = __fdiv_rn(1.f, __fsqrt_rn(dot_rn(dir, dir)));
            r.d = f3(__fmul_rn(dir.x, inv), __fmul_rn(dir.y, inv), __fmul_rn(dir.z, inv));
            r.o = f3(cam.eye[0], cam.eye[1], cam.eye[2]);
            set_cone<FAST, SUB, CAP>(sm, cam, dx, dy, valid, lane);
        }
        {
            float scene[6];   // scene box, read per tile (not kept live through the tile's loops)
#pragma unroll
            for (int z = 0; z < 6; ++z) scene[z] = ord2f(__ldg(a.scene_ord + z));
            float t0x = __fdiv_rn(scene[0] - r.o.x, r.d.x), t1x = __fdiv_rn(scene[3] - r.o.x, r.d.x);
            float t0y = __fdiv_rn(scene[1] - r.o.y, r.d.y), t1y = __fdiv_rn(scene[4] - r.o.y, r.d.y);
            float t0z = __fdiv_rn(scene[2] - r.o.z, r.d.z), t1z = __fdiv_rn(scene[5] - r.o.z, r.d.z);
            r.tenter = fmaxf(0.f, fmaxf(fminf(t0x, t1x), fmaxf(fminf(t0y, t1y), fminf(t0z, t1z))));
            r.texit = fminf(fmaxf(t0x, t1x), fminf(fmaxf(t0y, t1y), fmaxf(t0z, t1z)));
        }
        r.alive = valid && (r.tenter < r.texit);
        r.tb = r.tenter;
        // a team's warp: the list lane's ray of the whole tile, whose lists all warps build, and the ray it marches
        RayState lr = r;
        unsigned live = 0u;
        if constexpr (TEAM) {
            live = __ballot_sync(kFull, r.alive);
            r.d = f3(__shfl_sync(kFull, lr.d.x, sm.slot), __shfl_sync(kFull, lr.d.y, sm.slot),
                     __shfl_sync(kFull, lr.d.z, sm.slot));
            r.texit = __shfl_sync(kFull, lr.texit, sm.slot);
            valid = __shfl_sync(kFull, (int)valid, sm.slot);
            ray_l = __shfl_sync(kFull, ray_l, sm.slot);
        }
        r.T = 1.f;
        r.C = f3(0.f, 0.f, 0.f);
        r.g = f3(0.f, 0.f, 0.f);
        r.gR = 0.f;
        if (BWD && valid) {
            const long long ray_g = vt->ray_prefix[view] + (long long)ray_l;
            r.g = f3(a.dL[3 * ray_g], a.dL[3 * ray_g + 1], a.dL[3 * ray_g + 2]);
            r.gR = r.g.x * a.ray_colors_in[3 * ray_g] + r.g.y * a.ray_colors_in[3 * ray_g + 1] +
                   r.g.z * a.ray_colors_in[3 * ray_g + 2];
        }

        int K = min(kExactChunk, kmax);
        int rounds = 0;
        // end of the searched range: an inference launch queries the last slab in full
        const bool infer = !BWD && a.infer;
        const float l_texit = TEAM ? lr.texit : r.texit;
        const float t_end = infer ? l_texit + kSlab : l_texit;
        // hit-list record of this tile: the forward appends chunk records, the backward replays them
        const bool rec_here = a.rec_arena != nullptr && tile < a.rec_tiles;
        const bool leads = TEAM ? threadIdx.x / 32 % SUB == 0 : true;
        unsigned team_rec = kNoRecord;   // backward: a team's next chunk record to replay
        if constexpr (TEAM) {
            if (BWD && rec_here && a.replay) team_rec = a.rec_tile[tile];
            if (leads && lane == 0) sm.t.rec_first = sm.t.rec_prev = kNoRecord;
        } else if (lane == 0) {
            sm.rec_first = kNoRecord;
            sm.rec_prev = kNoRecord;
            sm.rec_cur = (BWD && rec_here && a.replay) ? a.rec_tile[tile] : kNoRecord;
        }
        __syncwarp();
        while (true) {
            bool on = TEAM ? live != 0u : r.alive;
            if (!__any_sync(kFull, on)) break;
            if (++rounds > kMaxRounds) {
                if (leads && lane == 0) atomicAdd(&a.st->watchdog_trips, 1ull);
                break;
            }
            unsigned rec_hdr = 0u;
            unsigned rec_cur = kNoRecord;
            if constexpr (TEAM) rec_cur = team_rec;
            else if (BWD) rec_cur = sm.rec_cur;
            if (BWD && rec_cur != kNoRecord) {
                if (rec_cur + 2u > a.rec_cap) {
                    rec_cur = kNoRecord;   // malformed link: traverse from here on
                } else {
                    rec_hdr = a.rec_arena[rec_cur];
                    K = max(1, min(kmax, (int)((rec_hdr >> 16) & 0xffu)));
                }
            }
            int nv;
            float seg_hi;
            // a slab step that no longer changes tb (|t| beyond ~2^19) would march forever
            bool l_on = false;   // a team: the list lane's ray
            if constexpr (TEAM) {
                l_on = ((live >> lane) & 1u) && lr.tb < lr.texit && lr.tb + kSlab != lr.tb;
                live = __ballot_sync(kFull, l_on);
                on = (live >> sm.slot) & 1u;
                r.tb = __shfl_sync(kFull, lr.tb, sm.slot);
                chunk_extent(lr, l_on, K, t_end, nv, seg_hi);
            } else {
                if (on && (!(r.tb < r.texit) || r.tb + kSlab == r.tb)) r.alive = on = false;
                chunk_extent(r, on, K, t_end, nv, seg_hi);
            }
            bool ovf = false;
            int count;
            const bool replayed = BWD && rec_cur != kNoRecord && !(rec_hdr & kRecordMulti);
            // the hits after leaf `cursor`: entries (over: more than the list holds)
            auto search = [&](int cursor, bool& over) {
                if constexpr (TEAM)
                    return team_traverse<SUB, CAP, DIAG>(sm, a, lr, l_on, t_end, seg_hi, K, nv, cursor, over, lane, ws,
                                                         infer);
                else
                    return traverse<FAST, SUB, CAP, DIAG>(sm, a, r, on, t_end, seg_hi, K, nv, cursor, over, lane, ws,
                                                          infer);
            };
            if (replayed) {
                const unsigned n_ids = min(rec_hdr & 0xffffu, a.rec_cap - rec_cur - 2u);
                const unsigned* ids = a.rec_arena + rec_cur + 2;
                if constexpr (TEAM)
                    count = team_replay<SUB, CAP, DIAG>(sm, a, lr, l_on, seg_hi, K, nv, ids, (int)n_ids, lane, ws);
                else
                    count = replay_list<FAST, SUB, CAP, DIAG>(sm, a, r, on, seg_hi, K, nv, ids, (int)n_ids, lane, ws);
                if (leads) ++ws.replays;
            } else {
                if constexpr (!TEAM) set_packet<FAST, SUB, CAP>(sm, r, on, seg_hi, lane);
                count = search(-1, ovf);
            }
            const int K_now = K;
            const unsigned long long* occ = sm.occ;
            auto& rec = record_of(sm);
            if (!BWD && rec_here && leads && rec.rec_prev != kRecordFailed) {
                // chunk record: header (multi-pass flag | K << 16 | id count), next record, ids
                const unsigned n_ids = ovf ? 0u : (unsigned)count;
                const unsigned words = 2u + n_ids;
                unsigned off = kNoRecord;
                if (lane == 0) {
                    unsigned long long o = atomicAdd(a.rec_top, (unsigned long long)words);
                    if (o + words <= (unsigned long long)a.rec_cap) {
                        off = (unsigned)o;
                        a.rec_arena[off] = (ovf ? kRecordMulti : 0u) | ((unsigned)K << 16) | n_ids;
                        a.rec_arena[off + 1] = kNoRecord;
                        if (rec.rec_prev != kNoRecord) a.rec_arena[rec.rec_prev + 1] = off;
                        if (rec.rec_first == kNoRecord) rec.rec_first = off;
                        rec.rec_prev = off;
                    } else {
                        rec.rec_prev = kRecordFailed;   // the chunks so far stay: the backward traverses after them
                        atomicAdd(&a.st->record_overflows, 1ull);
                    }
                }
                off = __shfl_sync(kFull, off, 0);
                if (off != kNoRecord)
                    for (unsigned e = lane; e < n_ids; e += 32) a.rec_arena[off + 2 + e] = (unsigned)sm.ids[e];
                __syncwarp();
            }
            if (!ovf) {
                if constexpr (SUB == 1) {
                    for (int k = 0; k < K; ++k) {
                        bool has = on && r.tb < r.texit && r.T > kTeps;
                        if (!__any_sync(kFull, has)) break;
                        if (!occ_test(occ, k)) {
                            // no lane has a hit in slabs [k, k2): march them (tb only; T is unchanged)
                            int k2 = occ_next(occ, k, K);
                            if (has) slabs_acc += march(r.tb, r.texit, k2 - k);
                            k = k2 - 1;
                            continue;
                        }
                        if (DIAG) ++ws.slab_steps;
                        float roff[kBuf];
                        unsigned seed_next = slab_offsets(a.rnd_sample, r.seed, roff);
                        SlabBuf<FAST, BWD> sb;
                        sb.clear();
                        int nh = slab_buffers<FAST, SUB, CAP, BWD, DIAG>(sm, k, K, has, r, a, rgb_base, roff, sb, nwords(count),
                                                                    lane, ws);
                        if (has) {
                            ++slabs_acc;
                            hits_acc += (!BWD && a.counts) ? min(nh, a.max_prim_slice) : nh;
                            if (nh > a.max_prim_slice) atomicAdd(&a.st->slab_cap_exceeded, 1ull);
                        }
                        if constexpr (!BWD) {
                            if (has && nh > 0) {
                                f2 alpha[kPairs];
                                slab_alpha(sb, alpha, a.neg_zero);
                                composite<FAST>(r, sb, alpha, a.neg_zero);
                                r.seed = seed_next;
                            }
                        } else {
                            AdjBuf<FAST> ad;
                            float Ta, gRa;
                            f2 alpha[kPairs];
                            slab_alpha(sb, alpha, a.neg_zero);
                            slab_adjoint_scalars<FAST>(r, sb, alpha, ad, Ta, gRa, a.neg_zero);
                            bool act = has && nh > 0 && sb.any_density();
                            slab_adjoint<FAST, SUB, CAP, DIAG>(sm, k, K, act, r, a, rgb_base, roff, ad, nwords(count), lane, ws,
                                                          view);
                            if (has && nh > 0) {
                                r.T = Ta;
                                r.gR = gRa;
                                r.seed = seed_next;
                            }
                        }
                        if (has) r.tb = r.tb + kSlab;
                    }
                } else {
                    for (int k = 0; k < K; k += SUB) {
                        const bool base = on && r.tb < r.texit && r.T > kTeps;
                        if (!__any_sync(kFull, base)) break;
                        const int n = min(SUB, K - k);   // slabs of the group inside the chunk
                        if (!occ_any(occ, k, n)) {
                            // march the groups without a hit (tb only; T is unchanged)
                            const int k2 = occ_next(occ, k, K), stop = k2 < K ? k2 / SUB * SUB : K;
                            if (base) {
                                const unsigned n_slabs = march(r.tb, r.texit, stop - k);
                                if (sub == 0) slabs_acc += n_slabs;
                            }
                            k = stop - SUB;
                            if (stop == K) break;
                            continue;
                        }
                        if (DIAG) ++ws.slab_steps;
                        // the lane's slab starts sub slabs on, by repeated addition; r.tb while it is marched
                        const float tb0 = r.tb;
#pragma unroll
                        for (int j = 0; j < SUB - 1; ++j)
                            if (j < sub) r.tb = r.tb + kSlab;
                        const float tb_end = r.tb + kSlab;
                        bool has = base && sub < n && r.tb < r.texit;
                        float roff[kBuf];
                        slab_offsets(a.rnd_sample, r.seed, roff);
                        SlabBuf<FAST, BWD> sb;
                        sb.clear();
                        const int nh = slab_buffers<FAST, SUB, CAP, BWD, DIAG>(sm, k, K, has, r, a, rgb_base, roff, sb,
                                                                               nwords(count), lane, ws);
                        const bool dense = nh > 0 && sb.any_density();
                        f2 alpha[kPairs];
                        slab_alpha(sb, alpha, a.neg_zero);
                        const float T0 = group_transmittance<SUB>(r, alpha, dense, has, lane);
                        const float T_end = r.T;
                        r.T = T0;
                        if (has) {
                            ++slabs_acc;
                            hits_acc += (!BWD && a.counts) ? min(nh, a.max_prim_slice) : nh;
                            if (nh > a.max_prim_slice) atomicAdd(&a.st->slab_cap_exceeded, 1ull);
                        }
                        if constexpr (!BWD) {
                            group_colour<FAST, SUB>(r, sb, alpha, has && dense, lane, a.neg_zero);
                        } else {
                            AdjBuf<FAST> ad;
                            const float gR_end = group_adjoint_scalars<FAST, SUB>(r, sb, alpha, has && dense, ad, lane);
                            slab_adjoint<FAST, SUB, CAP, DIAG>(sm, k, K, has && dense, r, a, rgb_base, roff, ad,
                                                               nwords(count), lane, ws, view);
                            r.gR = gR_end;
                        }
                        r.T = T_end;
                        // on to the next group (or the end of the chunk)
                        const float t_next = __shfl_sync(kFull, tb_end, ray * SUB + n - 1);
                        r.tb = base ? t_next : tb0;
                    }
                }
                // next chunk length: aim at half a list, grow at most 2x per chunk
                {
                    int target = count > 0 ? (K * (CAP / 2)) / count : kmax;
                    K = max(1, min(kmax, min(2 * K, target)));
                }
            } else {
                // K == 1 and more hits than the list holds: consume the slab in several passes
                const bool has_ray = on && r.tb < r.texit && r.T > kTeps, has = has_ray && sub == 0;
                float roff[kBuf];
                unsigned seed_next = slab_offsets(a.rnd_sample, r.seed, roff);
                SlabBuf<FAST, BWD> sb;
                sb.clear();
                int nh = slab_buffers<FAST, SUB, CAP, BWD, DIAG>(sm, 0, 1, has, r, a, rgb_base, roff, sb, nwords(count), lane,
                                                            ws);
                bool more = ovf;
                while (more) {
                    int cursor = sm.ids[count - 1];
                    __syncwarp();
                    if (leads && lane == 0) atomicAdd(&a.st->list_passes, 1ull);
                    count = search(cursor, more);
                    nh += slab_buffers<FAST, SUB, CAP, BWD, DIAG>(sm, 0, 1, has, r, a, rgb_base, roff, sb, nwords(count), lane,
                                                             ws);
                }
                if (has) {
                    ++slabs_acc;
                    hits_acc += (!BWD && a.counts) ? min(nh, a.max_prim_slice) : nh;
                    if (nh > a.max_prim_slice) atomicAdd(&a.st->slab_cap_exceeded, 1ull);
                }
                if constexpr (!BWD) {
                    if (has && nh > 0) {
                        f2 alpha[kPairs];
                        slab_alpha(sb, alpha, a.neg_zero);
                        composite<FAST>(r, sb, alpha, a.neg_zero);
                        r.seed = seed_next;
                    }
                } else {
                    AdjBuf<FAST> ad;
                    float Ta, gRa;
                    f2 alpha[kPairs];
                    slab_alpha(sb, alpha, a.neg_zero);
                    slab_adjoint_scalars<FAST>(r, sb, alpha, ad, Ta, gRa, a.neg_zero);
                    bool act = has && nh > 0 && sb.any_density();
                    int cursor = -1;
                    bool more2 = true;
                    while (more2) {
                        count = search(cursor, more2);
                        slab_adjoint<FAST, SUB, CAP, DIAG>(sm, 0, 1, act, r, a, rgb_base, roff, ad, nwords(count), lane, ws,
                                                      view);
                        if (more2) cursor = sm.ids[count - 1];
                        __syncwarp();
                    }
                    if (has && nh > 0) {
                        r.T = Ta;
                        r.gR = gRa;
                        r.seed = seed_next;
                    }
                }
                if constexpr (SUB > 1) {
                    r.T = __shfl_sync(kFull, r.T, ray * SUB);
                    r.gR = __shfl_sync(kFull, r.gR, ray * SUB);
                    r.C = f3(__shfl_sync(kFull, r.C.x, ray * SUB), __shfl_sync(kFull, r.C.y, ray * SUB),
                             __shfl_sync(kFull, r.C.z, ray * SUB));
                }
                if (has_ray) r.tb = r.tb + kSlab;
            }
            if constexpr (TEAM) {
                if (l_on) march(lr.tb, lr.texit, K_now);
                if (sub == 0) sm.t.live[sm.slot] = on && r.T > kTeps && r.tb < r.texit;
                if (BWD) team_rec = (rec_cur != kNoRecord) ? a.rec_arena[rec_cur + 1] : kNoRecord;
                sm.sync();
                live = __ballot_sync(kFull, sm.t.live[lane] != 0);
            } else {
                if (on) r.alive = r.alive && (r.T > kTeps) && (r.tb < r.texit);
                if (BWD && lane == 0) sm.rec_cur = (rec_cur != kNoRecord) ? a.rec_arena[rec_cur + 1] : kNoRecord;
                __syncwarp();
            }
        }
        if (!BWD && rec_here && leads && lane == 0)
            a.rec_tile[tile] = record_of(sm).rec_first;
        flush_stats<FAST, SUB, CAP, DIAG>(sm, ws, hits_acc, slabs_acc, lane);
        if constexpr (!BWD && SUB > 1) {
#pragma unroll
            for (int o = 1; o < SUB; o <<= 1) hits_acc += __shfl_xor_sync(kFull, hits_acc, o);
        }
        if (!BWD && valid && sub == 0) {
            const long long ray_g = vt->ray_prefix[view] + (long long)ray_l;
            a.ray_colors[3 * ray_g] = __fadd_rn(r.C.x, __fmul_rn(r.T, bg));
            a.ray_colors[3 * ray_g + 1] = __fadd_rn(r.C.y, __fmul_rn(r.T, bg));
            a.ray_colors[3 * ray_g + 2] = __fadd_rn(r.C.z, __fmul_rn(r.T, bg));
            if (a.final_T) a.final_T[ray_g] = r.T;
            // Gaussians per ray (inference launches): the per-slab hit counts, each capped at
            // max_prim_slice like the reference any-hit program (cuda_test/gaussians_aabb.cu:438)
            if (a.counts) a.counts[ray_g] = (int)hits_acc;
        }
    }
    // counters: one atomic per warp and counter
    __syncwarp();
    if (lane == 0) {
        atomicAdd(&a.st->traversals, sm.cnt[0]);
        atomicAdd(&a.st->node_visits, sm.cnt[1]);
        atomicAdd(&a.st->leaf_tests, sm.cnt[2]);
        atomicAdd(&a.st->list_entries, sm.cnt[3]);
        atomicAdd(&a.st->slab_steps, sm.cnt[4]);
        atomicAdd(&a.st->entry_slabs, sm.cnt[5]);
        if (BWD) atomicAdd(&a.st->replayed_chunks, sm.cnt[6]);
        atomicAdd(&a.st->hit_pairs, sm.cnt[7]);
        atomicAdd(&a.st->slabs, sm.cnt[8]);
    }
}

// Per-leaf conversion of the summed adjoint moments into gradients (one thread per leaf):
//   in  [dens grad, S1.xyz, M2 xx yy zz xy xz yz, 0, 0]
//   out [dens grad, dpos.xyz, dscale.xyz, dquat.xyzw, 0]
// with m = M v (rows of M = R^T / s): dpos = M^T M S1, dscale_j = r_j^T M2 r_j / s_j and, for the
// rotation, P_j = M2 r_j enters the quaternion derivative as -P_j / s_j.
__global__ void k_moment_grads(int n, const LeafRec* __restrict__ rec, const float4* __restrict__ ext,
                               float4* __restrict__ acc) {
    int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= n) return;
    const float4 a0 = acc[3 * (long long)l], a1 = acc[3 * (long long)l + 1], a2 = acc[3 * (long long)l + 2];
    const LeafRec rr = rec[l];
    const float4 s4 = ext[2 * (long long)l], q4 = ext[2 * (long long)l + 1];
    const float3 r0 = f3(rr.r0.x, rr.r0.y, rr.r0.z), r1 = f3(rr.r1.x, rr.r1.y, rr.r1.z),
                 r2 = f3(rr.r2.x, rr.r2.y, rr.r2.z);
    const float3 S1 = f3(a0.y, a0.z, a0.w);
    const float xx = a1.x, yy = a1.y, zz = a1.z, xy = a1.w, xz = a2.x, yz = a2.y;
    auto m2 = [&](float3 w) {
        return f3(xx * w.x + xy * w.y + xz * w.z, xy * w.x + yy * w.y + yz * w.z, xz * w.x + yz * w.y + zz * w.z);
    };
    const float3 Sm = f3(dot3(r0, S1), dot3(r1, S1), dot3(r2, S1));
    const float3 dp = r0 * Sm.x + r1 * Sm.y + r2 * Sm.z;
    const float3 P0 = m2(r0), P1 = m2(r1), P2 = m2(r2);
    const float3 is = f3(1.f / s4.x, 1.f / s4.y, 1.f / s4.z);
    const float3 dsc = f3(dot3(r0, P0) * is.x, dot3(r1, P1) * is.y, dot3(r2, P2) * is.z);
    const float4 dq = quat_grad(q4, P0 * (-is.x), P1 * (-is.y), P2 * (-is.z));
    acc[3 * (long long)l] = make_float4(a0.x, dp.x, dp.y, dp.z);
    acc[3 * (long long)l + 1] = make_float4(dsc.x, dsc.y, dsc.z, dq.x);
    acc[3 * (long long)l + 2] = make_float4(dq.y, dq.z, dq.w, 0.f);
}

cudaError_t launch_moment_grads(int n, const LeafRec* rec, const float4* ext, float4* acc, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_moment_grads<<<(n + 255) / 256, 256, 0, s>>>(n, rec, ext, acc);
    return cudaGetLastError();
}

// List capacity per arithmetic: 4x the tuning value (64 or 128) for the fast lists; 128 for the
// parity lists of whole tiles at either value (their slab ranges make an entry 72 B; shorter lists turn
// dense slabs into multi-pass traversals, which the backward cannot replay).  The parity lists of split tiles
// hold 192 or 256 entries; a team's list has the length of the whole tile's, for the same chunks.
using ParitySmem = WarpSmem<false, 1, 128>;
using FastSmem256 = WarpSmem<true, 1, 256>;
using FastSmem512 = WarpSmem<true, 1, 512>;
using ParitySplit2Smem = WarpSmem<false, 2, 192>;
using ParitySplitSmem = WarpSmem<false, 4, 256>;
using FastTeam2Smem = TeamSmem<2, 256>;
using FastTeamSmem = TeamSmem<4, 256>;
// packet and cone are read as float4: 16-byte aligned in every warp's slice of the block's array
template <typename S, int WARPS = 1>
constexpr bool smem_fits() {
    return offsetof(S, packet) % 16 == 0 && offsetof(S, cone) % 16 == 0 && sizeof(S) % 16 == 0 &&
           sizeof(S) * kWarpsPerBlock / WARPS <= 48 * 1024;
}
static_assert(smem_fits<ParitySmem>() && smem_fits<FastSmem256>() && smem_fits<FastSmem512>() &&
                  smem_fits<ParitySplit2Smem>() && smem_fits<FastTeam2Smem, 2>() && smem_fits<ParitySplitSmem>() &&
                  smem_fits<FastTeamSmem, 4>(),
              "alignment, static shared memory limit");

// The kernel of a launch: calls f(kernel).
template <bool BWD, bool FAST, bool DIAG, typename F>
static void with_kernel(int cap, int split, F f) {
    if (split == 4) f(k_render<BWD, FAST, 4, 256, DIAG>);
    else if (split == 2) f(k_render<BWD, FAST, 2, FAST ? 256 : 192, DIAG>);
    else if constexpr (!FAST) f(k_render<BWD, FAST, 1, 128, DIAG>);
    else if (cap <= 64) f(k_render<BWD, FAST, 1, 256, DIAG>);
    else f(k_render<BWD, FAST, 1, 512, DIAG>);
}
template <bool DIAG, typename F>
static void with_kernel(bool backward, bool fast, int cap, int split, F f) {
    if (backward) fast ? with_kernel<true, true, DIAG>(cap, split, f) : with_kernel<true, false, DIAG>(cap, split, f);
    else fast ? with_kernel<false, true, DIAG>(cap, split, f) : with_kernel<false, false, DIAG>(cap, split, f);
}

int render_occupancy(bool backward, int mode, int cap, int split) {
    int nb = 0;
    with_kernel<false>(backward, mode == RG_MODE_FAST, cap, split, [&](auto kernel) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, kWarpsPerBlock * 32, 0);
    });
    return nb;
}

// Slabs side by side.  Few tiles wait for the slowest one, which the split shortens, the more the more
// Gaussians a tile sees; many share the traversal better when they are whole, above all where rays are
// long (an unbounded scene's far field: chunk after chunk with few Gaussians).  The results are the same.
// With T the launch's 8x4-pixel tiles and x = Gaussians * views / T / (T / 1000), the lines below are where
// forward + backward cross: fast over 122 launches of 300 to 147,000 tiles, 1 to 8 views and 5k to 600k
// Gaussians in boxes, on shells (3 to 5 units across) and in a ball with a far field (200), where they lose
// 1 to 2 % on the best choice for each; parity over 30 such launches of one view.  In ms with 4 / 2 / 1 slabs:
//   fast, short    200k, 1500 tiles, 2 views  63.3 / 94.0 / 181    20k, 34187, 4 views    4.8 /  3.3 /  2.7
//                  200k, 17048, 4 views       19.8 / 24.6 / 43.0   600k, 34187, 4 views  77.5 / 74.1 / 86.0
//   fast, long     200k, 1500, 2 views        14.3 / 22.7 / 43.3   200k, 17048, 4 views  46.9 / 35.7 / 26.7
//   parity, short  200k, 15000                20.2 / 17.0 / 22.8   600k, 15000           47.1 / 53.2 / 84.6
SplitPair render_split(int mode, int rnd_sample, int cap, long long n, int n_views, long long n_rays) {
    const bool fast = mode == RG_MODE_FAST && rnd_sample == 0;
    // random offsets draw slab after slab; long lists are whole tiles' (the autotuner's choice)
    if (rnd_sample == 1 || cap > 64 || n_rays <= 0) return {1, 1};
    const double t = (double)std::max(1ll, n_rays / (kTileW * kTileH));
    const double x = 1000.0 * (double)n * n_views / (t * t);
    auto pick = [&](double four, double two) { return x >= four ? 4 : x >= two ? 2 : 1; };
    return fast ? SplitPair{pick(2.7, 0.6), pick(45.0, 4.0)} : SplitPair{pick(1.5, 0.2), pick(32.0, 6.0)};
}

cudaError_t launch_render(bool backward, int mode, int cap, int split, int grid, const RenderArgs& args, cudaStream_t s) {
    RenderArgs a = args;
    a.neg_zero = 0x8000000080000000ull;
    const bool fast = (mode == RG_MODE_FAST) && a.rnd_sample == 0;
    auto launch = [&](auto kernel) { kernel<<<grid, kWarpsPerBlock * 32, 0, s>>>(a); };
    if (a.diag) with_kernel<true>(backward, fast, cap, split, launch);
    else with_kernel<false>(backward, fast, cap, split, launch);
    return cudaGetLastError();
}

}  // namespace rg
