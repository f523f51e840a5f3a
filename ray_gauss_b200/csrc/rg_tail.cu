// Fused training-step tail: Adam on every parameter tensor of the Gaussians, the densification
// statistics and the parameter clamps in one launch.
//
// Reference semantics (paths inside the reference project):
//   statistics   scripts/train.py:121-123 -> classes/point_cloud.py:633-640 (accumulate_gradient,
//                accumulate_gradient_gaussians_not_visible: |dL/dposition| summed, visible counts)
//   Adam         classes/optimizer.py:13-21, 203-218 (one torch.optim.Adam per tensor, eps 1e-15,
//                default betas; learning rates and step counts come from the host)
//   clamps       scripts/train.py:166-181 (densities < 0 -> 0, quaternion and lobe-axis
//                normalisation, log scales clamped to [filter_3D, max_scale]) with
//                classes/point_cloud.py:703-727 (zero-norm quaternion -> (1,0,0,0), zero-norm
//                axis -> (0,0,1))
// Adam per element, as torch.optim.Adam:  m += (1 - beta1) (g - m);  v = beta2 v + (1 - beta2) g^2;
// p -= (lr / (1 - beta1^t)) * m / (sqrt(v) / sqrt(1 - beta2^t) + eps).
//
// Layout: k_tail_stream gives every tensor blocks of its own.  A thread takes whole rows with float4
// accesses: a quaternion, four positions or lobe axes (12 floats), or four elements of a tensor whose
// clamp is elementwise, so the clamp and the statistics work on the values in registers.  Every byte is
// read and written once: HBM-bound at 28 bytes per parameter float (param, m, v read and written, grad
// read).  1M Gaussians, 115 floats each, 3.25 GB: 553 us (90 % of a copy's rate), against 805 us when a block took 256
// Gaussians through all tensors in turn (few loads in flight at a time, threads idle at the narrow
// tensors, the clamps on parameters read again behind a barrier).  That form, k_train_tail, still does
// what has no 16-byte alignment, tensors that are not separate, and what l2_resident names.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "rg_common.cuh"

namespace {

constexpr int kTailMaxTensors = RG_TAIL_MAX_TENSORS;
constexpr int kTailThreads = 256;
constexpr int kTailGaussians = 256;

struct TailArgs {
    rg_train_tail d;
};

struct AdamStep {
    float w1, w2, beta2, eps, step_size, bias2_sqrt;
};

__device__ __forceinline__ void adam1(float& p, float g, float& m, float& v, const AdamStep& s) {
    m = m + s.w1 * (g - m);
    v = s.beta2 * v + s.w2 * g * g;
    p -= s.step_size * (m / (sqrtf(v) / s.bias2_sqrt + s.eps));
}

__device__ void adam_range(const rg_adam_tensor& t, const AdamStep& s, long long e0, long long e1) {
    const bool vec = (((uintptr_t)t.param | (uintptr_t)t.grad | (uintptr_t)t.exp_avg | (uintptr_t)t.exp_avg_sq) &
                      15) == 0 && (e0 & 3) == 0;
    long long e = e0;
    if (vec) {
        const long long nv = (e1 - e0) >> 2;
        float4* P = reinterpret_cast<float4*>(t.param + e0);
        const float4* G = reinterpret_cast<const float4*>(t.grad + e0);
        float4* M = reinterpret_cast<float4*>(t.exp_avg + e0);
        float4* V = reinterpret_cast<float4*>(t.exp_avg_sq + e0);
        for (long long j = threadIdx.x; j < nv; j += kTailThreads) {
            float4 p = P[j], m = M[j], v = V[j];
            const float4 g = __ldcs(G + j);
            adam1(p.x, g.x, m.x, v.x, s);
            adam1(p.y, g.y, m.y, v.y, s);
            adam1(p.z, g.z, m.z, v.z, s);
            adam1(p.w, g.w, m.w, v.w, s);
            P[j] = p;
            M[j] = m;
            V[j] = v;
        }
        e = e0 + 4 * nv;
    }
    for (long long j = e + threadIdx.x; j < e1; j += kTailThreads) {
        float p = t.param[j], m = t.exp_avg[j], v = t.exp_avg_sq[j];
        adam1(p, t.grad[j], m, v, s);
        t.param[j] = p;
        t.exp_avg[j] = m;
        t.exp_avg_sq[j] = v;
    }
}

// The step of tensor i (false: it does not step).
__device__ __forceinline__ bool adam_step(const rg_train_tail& d, int i, AdamStep& s) {
    const rg_adam_tensor& t = d.tensors[i];
    if (!t.active || !t.grad || !t.param || t.width <= 0) return false;
    float lr = t.lr, bias1 = t.bias1, bias2_sqrt = t.bias2_sqrt;
    if (d.step_scalars) {
        const float* sc = d.step_scalars + 4 * i;
        if (sc[0] == 0.f) return false;
        lr = sc[1];
        bias1 = sc[2];
        bias2_sqrt = sc[3];
    }
    s = AdamStep{t.one_minus_beta1, t.one_minus_beta2, t.beta2, t.eps, lr / bias1, bias2_sqrt};
    return true;
}

// Densification statistics of Gaussian g from its position gradient.
__device__ __forceinline__ void tail_stats(const rg_train_tail& d, long long g, float gx, float gy, float gz) {
    const float gn = sqrtf(gx * gx + gy * gy + gz * gz);
    if (d.grad_norm_accum) d.grad_norm_accum[g] += gn;
    if (d.num_accum && gn > 0.f) d.num_accum[g] += 1.f;
    if (d.num_accum_gnv && gn > 0.f) d.num_accum_gnv[g] += 1.f;
}
__device__ __forceinline__ float4 unit_quaternion(float4 q) {
    float nn = sqrtf(q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w);
    if (nn == 0.f) { q = make_float4(1.f, 0.f, 0.f, 0.f); nn = 1.f; }
    return make_float4(q.x / nn, q.y / nn, q.z / nn, q.w / nn);
}
__device__ __forceinline__ void unit_axis(float* ax) {
    float nn = sqrtf(ax[0] * ax[0] + ax[1] * ax[1] + ax[2] * ax[2]);
    if (nn == 0.f) { ax[0] = 0.f; ax[1] = 0.f; ax[2] = 1.f; nn = 1.f; }
    for (int k = 0; k < 3; ++k) ax[k] /= nn;
}
__device__ __forceinline__ float clamp_scale(const rg_train_tail& d, float v, long long g) {
    const float lo = d.min_scale ? d.min_scale[g] : -INFINITY;
    if (v < lo) v = lo;
    if (v > d.max_scale) v = d.max_scale;
    return v;
}

// The statistics or the clamp of tensor i for Gaussian g, from memory.
__device__ void tail_row(const rg_train_tail& d, int i, long long g) {
    const rg_adam_tensor& t = d.tensors[i];
    if (i == d.idx_positions && t.grad && (d.grad_norm_accum || d.num_accum || d.num_accum_gnv)) {
        const float* gp = t.grad + 3 * g;
        tail_stats(d, g, gp[0], gp[1], gp[2]);
    }
    if (i == d.idx_densities && t.param[g] < 0.f) t.param[g] = 0.f;
    if (i == d.idx_quaternions && d.normalize_quaternions) {
        float4* qp = reinterpret_cast<float4*>(t.param) + g;
        *qp = unit_quaternion(*qp);
    }
    if (i == d.idx_lobe_axis && d.normalize_lobe_axis)
        for (int l = 0; l < t.width / 3; ++l) unit_axis(t.param + g * t.width + 3 * l);
    if (i == d.idx_scales)
        for (int k = 0; k < 3; ++k) t.param[3 * g + k] = clamp_scale(d, t.param[3 * g + k], g);
}

// Blocks of the tensors: those of segment k end at block_end[k].
struct TailSegments {
    int count, iters;
    int tensor[kTailMaxTensors];
    unsigned block_end[kTailMaxTensors];
};
// float4 units of a thread at a time (loads first), and at most so many such steps of a block: 598 us with
// 2 x 4, 564 with 2 x 8, 548 with 4 x 4, 949 with 1 x 1 (short blocks), 1M Gaussians.  Fewer steps where
// they would leave the chip without four blocks per SM.
constexpr int kTailUnroll = 4, kTailMaxIters = 4;

// NV float4 of a tensor, `stride` float4 apart from number `first` on, those before `end`: stepped when
// `steps`, then clamped by f(values of one, its number).  All loads come first.
template <int NV, typename F>
__device__ __forceinline__ void tail_unit(const rg_adam_tensor& t, const AdamStep& s, bool steps, long long first, int stride,
                                          long long end, F f) {
    float4 p[NV], g[NV], m[NV], v[NV];
    float4* const P = reinterpret_cast<float4*>(t.param) + first;
    const float4* const G = reinterpret_cast<const float4*>(t.grad) + first;
    float4* const M = reinterpret_cast<float4*>(t.exp_avg) + first;
    float4* const V = reinterpret_cast<float4*>(t.exp_avg_sq) + first;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        if (first + k * stride >= end) continue;
        p[k] = P[k * stride];
        if (steps) {
            g[k] = __ldcs(G + k * stride);
            m[k] = M[k * stride];
            v[k] = V[k * stride];
        }
    }
    if (steps) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            if (first + k * stride >= end) continue;
            adam1(p[k].x, g[k].x, m[k].x, v[k].x, s);
            adam1(p[k].y, g[k].y, m[k].y, v[k].y, s);
            adam1(p[k].z, g[k].z, m[k].z, v[k].z, s);
            adam1(p[k].w, g[k].w, m[k].w, v[k].w, s);
            M[k * stride] = m[k];
            V[k * stride] = v[k];
        }
    }
    f(p);
#pragma unroll
    for (int k = 0; k < NV; ++k)
        if (first + k * stride < end) P[k * stride] = p[k];
}

// Gaussians [0, n4), n4 a multiple of 4; every tensor 16-byte aligned.  Where n4 < n a last block per tensor
// takes the rest (10k Gaussians: 41 us a call with a launch of its own for them, 33 without).
__global__ void __launch_bounds__(kTailThreads, 2) k_tail_stream(const TailArgs args, const TailSegments seg, long long n4) {
    const rg_train_tail& d = args.d;
    const unsigned whole = seg.block_end[seg.count - 1];
    if (blockIdx.x >= whole) {
        const int i = seg.tensor[blockIdx.x - whole];
        const rg_adam_tensor& t = d.tensors[i];
        AdamStep s;
        if (adam_step(d, i, s)) adam_range(t, s, n4 * t.width, d.n * t.width);
        __syncthreads();  // the clamp reads parameters that other threads stepped
        if (n4 + threadIdx.x < d.n) tail_row(d, i, n4 + threadIdx.x);
        return;
    }
    int k = 0;
    while (blockIdx.x >= seg.block_end[k]) ++k;
    const int i = seg.tensor[k];
    const rg_adam_tensor& t = d.tensors[i];
    const long long block = blockIdx.x - (k ? seg.block_end[k - 1] : 0u);
    AdamStep s;
    const bool steps = adam_step(d, i, s);
    const bool stats = i == d.idx_positions && t.grad && (d.grad_norm_accum || d.num_accum || d.num_accum_gnv);
    const bool axis = i == d.idx_lobe_axis && d.normalize_lobe_axis;
    if (stats || axis) {
#pragma unroll 1
        for (int it = 0; it < seg.iters; ++it) {
            const long long u = (block * seg.iters + it) * kTailThreads + threadIdx.x;
            if (u >= n4 * t.width / 12) return;
            if (stats) {
                const float4* G = reinterpret_cast<const float4*>(t.grad) + 3 * u;
                const float4 a = G[0], b = G[1], c = G[2];
                tail_stats(d, 4 * u, a.x, a.y, a.z);
                tail_stats(d, 4 * u + 1, a.w, b.x, b.y);
                tail_stats(d, 4 * u + 2, b.z, b.w, c.x);
                tail_stats(d, 4 * u + 3, c.y, c.z, c.w);
            }
            if (steps || axis)
                tail_unit<3>(t, s, steps, 3 * u, 1, 3 * u + 3, [&](float4* p) {
                    if (axis)
                        for (int j = 0; j < 4; ++j) unit_axis(reinterpret_cast<float*>(p) + 3 * j);
                });
        }
        return;
    }
    const bool dens = i == d.idx_densities, quat = i == d.idx_quaternions && d.normalize_quaternions,
               scale = i == d.idx_scales;
    if (!steps && !dens && !quat && !scale) return;
    const long long units = n4 * t.width / 4;
#pragma unroll 1
    for (int it = 0; it < seg.iters; ++it) {
        const long long first = (block * seg.iters + it) * kTailUnroll * kTailThreads + threadIdx.x;
        if (first >= units) return;
        tail_unit<kTailUnroll>(t, s, steps, first, kTailThreads, units, [&](float4* p) {
#pragma unroll
            for (int k = 0; k < kTailUnroll; ++k) {
                float* const e = reinterpret_cast<float*>(p + k);
                const long long at = 4 * (first + k * kTailThreads);
                if (at >= 4 * units) continue;
                if (dens) {
                    for (int c = 0; c < 4; ++c)
                        if (e[c] < 0.f) e[c] = 0.f;
                } else if (quat) {
                    p[k] = unit_quaternion(p[k]);
                } else if (scale) {
                    const long long g = at / 3;
                    const int r = (int)(at - 3 * g);
                    for (int c = 0; c < 4; ++c) e[c] = clamp_scale(d, e[c], g + (r + c >= 3));
                }
            }
        });
    }
}

// The clamps are written out: through tail_row they take registers that cost a block per SM (160k x 44
// floats 43 -> 60 us).
__global__ void __launch_bounds__(kTailThreads) k_train_tail(const TailArgs args) {
    const rg_train_tail& d = args.d;
    const long long g0 = (long long)blockIdx.x * kTailGaussians;
    const long long g1 = g0 + kTailGaussians < d.n ? g0 + kTailGaussians : d.n;
    for (int i = 0; i < d.n_tensors; ++i) {
        AdamStep s;
        if (adam_step(d, i, s)) adam_range(d.tensors[i], s, g0 * d.tensors[i].width, g1 * d.tensors[i].width);
    }
    __syncthreads();  // the clamps below read parameters that other threads of the block stepped
    const long long g = g0 + threadIdx.x;
    if (g >= g1) return;
    // densification statistics from the position gradient
    if (d.idx_positions >= 0 && d.tensors[d.idx_positions].grad &&
        (d.grad_norm_accum || d.num_accum || d.num_accum_gnv)) {
        const float* gp = d.tensors[d.idx_positions].grad + 3 * g;
        tail_stats(d, g, gp[0], gp[1], gp[2]);
    }
    // clamps after the step
    if (d.idx_densities >= 0) {
        float* p = d.tensors[d.idx_densities].param + g;
        if (*p < 0.f) *p = 0.f;
    }
    if (d.normalize_quaternions && d.idx_quaternions >= 0) {
        float4* qp = reinterpret_cast<float4*>(d.tensors[d.idx_quaternions].param) + g;
        *qp = unit_quaternion(*qp);
    }
    if (d.normalize_lobe_axis && d.idx_lobe_axis >= 0 && d.tensors[d.idx_lobe_axis].width > 0) {
        const rg_adam_tensor& t = d.tensors[d.idx_lobe_axis];
        for (int l = 0; l < t.width / 3; ++l) unit_axis(t.param + g * t.width + 3 * l);
    }
    if (d.idx_scales >= 0) {
        float* s = d.tensors[d.idx_scales].param + 3 * g;
        for (int k = 0; k < 3; ++k) s[k] = clamp_scale(d, s[k], g);
    }
}

int check_tail(const rg_train_tail* d) {
    if (!d || d->n < 0 || d->n_tensors < 0 || d->n_tensors > kTailMaxTensors) return RG_ERR_INVALID_ARG;
    const int idx[5] = {d->idx_positions, d->idx_densities, d->idx_scales, d->idx_quaternions, d->idx_lobe_axis};
    const int width[5] = {3, 1, 3, 4, -1};
    for (int j = 0; j < 5; ++j) {
        if (idx[j] < -1 || idx[j] >= d->n_tensors) return RG_ERR_INVALID_ARG;
        if (idx[j] >= 0) {
            const rg_adam_tensor& t = d->tensors[idx[j]];
            // a lobe-axis tensor may have zero width (no SG lobes unlocked yet)
            if ((!t.param && t.width != 0) || (width[j] > 0 && t.width != width[j]) ||
                (width[j] < 0 && t.width % 3 != 0))
                return RG_ERR_INVALID_ARG;
        }
    }
    // the quaternion clamp reads and writes float4 rows
    if (d->normalize_quaternions && d->idx_quaternions >= 0 &&
        ((uintptr_t)d->tensors[d->idx_quaternions].param & 15) != 0)
        return RG_ERR_INVALID_ARG;
    for (int i = 0; i < d->n_tensors; ++i) {
        const rg_adam_tensor& t = d->tensors[i];
        if (!t.active) continue;
        if (!t.param || !t.exp_avg || !t.exp_avg_sq || t.width <= 0) return RG_ERR_INVALID_ARG;
        if (!d->step_scalars && (!(t.bias1 > 0.f) || !(t.bias2_sqrt > 0.f))) return RG_ERR_INVALID_ARG;
    }
    return RG_OK;
}

// Clouds of narrow rows whose tensors (with the gradients) about fit L2 go to k_train_tail: most of what it
// reads hits there, and its blocks, with half the registers, are all resident at once, while k_tail_stream's
// come in waves.  k_train_tail / k_tail_stream, us: 23 floats per Gaussian: 14 / 14 at 40k, 16 / 21 at 80k, 35 / 41
// at 250k, 62 / 62 at 400k; 44 floats: 23 / 21 at 40k, 27 / 35 at 80k, 43 / 51 at 160k, 80 / 71 at 250k; 59
// floats: 23 / 21 at 40k, 25 / 29 at 60k, 53 / 58 at 160k; 79 floats: 51 / 45 at 60k, 92 / 61 at 120k; 115
// floats: 52 / 43 at 40k, 113 / 84 at 120k (it takes the tensors in turn: long chains).
bool l2_resident(const rg_train_tail& d) {
    long long width = 0;
    for (int i = 0; i < d.n_tensors; ++i) width += d.tensors[i].width;
    return width <= 64 && d.n >= 50000 && 16 * d.n * width <= 150000000;
}

// Whether the tensors can be taken side by side: none is in two roles, and what one writes no other uses.
bool separate(const rg_train_tail& d) {
    const int role[5] = {d.idx_positions, d.idx_densities, d.idx_scales, d.idx_quaternions, d.idx_lobe_axis};
    for (int i = 0; i < 5; ++i)
        for (int j = 0; j < i; ++j)
            if (role[i] >= 0 && role[i] == role[j]) return false;
    for (int i = 0; i < d.n_tensors; ++i) {
        const rg_adam_tensor& t = d.tensors[i];
        const uintptr_t at[4] = {(uintptr_t)t.param, (uintptr_t)t.exp_avg, (uintptr_t)t.exp_avg_sq, (uintptr_t)t.grad};
        const uintptr_t size = t.width > 0 ? (uintptr_t)d.n * t.width * sizeof(float) : 0;
        for (int j = 0; j < d.n_tensors; ++j) {
            const rg_adam_tensor& u = d.tensors[j];
            const uintptr_t other[3] = {(uintptr_t)u.param, (uintptr_t)u.exp_avg, (uintptr_t)u.exp_avg_sq};
            const uintptr_t u_size = u.width > 0 ? (uintptr_t)d.n * u.width * sizeof(float) : 0;
            if (i == j) continue;
            for (uintptr_t p : at)
                for (uintptr_t q : other)
                    if (p && q && p < q + u_size && q < p + size) return false;
        }
    }
    return true;
}

}  // namespace

extern "C" {

int rg_train_tail_step(const rg_train_tail* d, void* stream) {
    int rc = check_tail(d);
    if (rc) return rc;
    if (d->n == 0) return RG_OK;
    TailArgs a;
    std::memcpy(&a.d, d, sizeof(rg_train_tail));
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // the streaming form takes every tensor that steps, is clamped or gives the statistics
    TailSegments seg{};
    long long n4 = d->n & ~3ll, blocks = 0, floats_all = 0;
    for (int i = 0; i < d->n_tensors; ++i) floats_all += n4 * d->tensors[i].width;
    seg.iters = (int)std::min<long long>(kTailMaxIters, std::max(1ll, floats_all / (4ll * kTailThreads * kTailUnroll * 592)));
    for (int i = 0; i < d->n_tensors && n4; ++i) {
        const rg_adam_tensor& t = d->tensors[i];
        if (!t.param || t.width <= 0) continue;
        if (((uintptr_t)t.param | (uintptr_t)t.grad | (uintptr_t)t.exp_avg | (uintptr_t)t.exp_avg_sq) & 15) n4 = 0;
        // a thread takes 12 floats where k_tail_stream works on rows of 3, else kTailUnroll float4
        const bool rows = (i == d->idx_positions && t.grad && (d->grad_norm_accum || d->num_accum || d->num_accum_gnv)) ||
                          (i == d->idx_lobe_axis && d->normalize_lobe_axis);
        const long long per_block = kTailThreads * seg.iters * (rows ? 12ll : 4ll * kTailUnroll);
        const long long floats = n4 * t.width;
        blocks += (floats + per_block - 1) / per_block;
        seg.tensor[seg.count] = i;
        seg.block_end[seg.count++] = (unsigned)blocks;
    }
    if (n4 < d->n) blocks += seg.count;
    if (blocks > 0x7fffffffll || !seg.count || l2_resident(*d) || !separate(*d)) n4 = 0;
    if (n4)
        k_tail_stream<<<(unsigned)blocks, kTailThreads, 0, st>>>(a, seg, n4);
    else
        k_train_tail<<<(unsigned)((d->n + kTailGaussians - 1) / kTailGaussians), kTailThreads, 0, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? RG_OK : RG_ERR_CUDA;
}

}  // extern "C"
