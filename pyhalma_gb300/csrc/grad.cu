// Adjoint of the softened potential  phi_i = sum_j m_j (|s_j - t_i|^2 + eps2)^-1/2.
//
// For an upstream gradient g_i = dL/dphi_i the derivatives are two all-pairs sums of the same
// shape, so one kernel serves both:
//   over targets a = t_i, partners b = s_j, weights w_b = m_j:
//       V_a = sum_b w_b (p_b - p_a) r^-3            -> dL/dt_i = g_i * V_a
//   over sources a = s_j, partners b = t_i, weights w_b = g_i:
//       S_a = sum_b w_b r^-1,  V_a = sum_b w_b (p_b - p_a) r^-3
//                                                   -> dL/dm_j = S_a, dL/ds_j = m_j * V_a
// with r^2 = |p_b - p_a|^2 + eps2.  FP32 pair terms (rsqrt) as f32x2 instructions (two partners
// per instruction), per-chunk FP32 partials folded into TwoSum-compensated accumulators.  The
// self pair (b == a + self_offset) is skipped when the mask asks for it.
#include <math.h>
#include <string.h>

#include <algorithm>

#include "common.cuh"
#include "pair_math.cuh"

namespace halma {
namespace {

constexpr int kGWarps = 4;
constexpr float kFarG = 3.0e30f;

__device__ __forceinline__ float4 load_b(const float *__restrict__ x, const float *__restrict__ y,
                                         const float *__restrict__ z, const float *__restrict__ w, int64_t j,
                                         int64_t n) {
    if (j < n) return make_float4(x[j], y[j], z[j], w[j]);
    return make_float4(kFarG, kFarG, kFarG, 0.f);
}

// 32 partners of the staged chunk against the lane's T particles, two partners per f32x2
// instruction: sa[kp] = {x_2kp, x_2kp+1, y_2kp, y_2kp+1}, sb[kp] = {z.., z.., w.., w..}.  Per
// pair: r^-1 and w r^-3 (p_b - p_a); the chunk's partials are {even, odd} pairs.  SELF: the
// pair whose partner index (j0 + slot) equals self[t] is skipped.
template <int T, bool WANT_S, bool SELF>
__device__ __forceinline__ void adjoint_chunk(const float4 *sa, const float4 *sb, const f2x (&px)[T],
                                              const f2x (&py)[T], const f2x (&pz)[T], f2x e2, int64_t j0,
                                              const int64_t (&self)[T], f2x (&ps)[T], f2x (&pvx)[T],
                                              f2x (&pvy)[T], f2x (&pvz)[T]) {
#pragma unroll 4
    for (int kp = 0; kp < 16; ++kp) {
        const float4 qa = sa[kp], qb = sb[kp];
        const f2x X = pack2(qa.x, qa.y), Y = pack2(qa.z, qa.w), Z = pack2(qb.x, qb.y), W = pack2(qb.z, qb.w);
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const f2x dx = sub2(X, px[t]), dy = sub2(Y, py[t]), dz = sub2(Z, pz[t]);
            f2x r2 = fma2(dz, dz, e2);
            r2 = fma2(dy, dy, r2);
            r2 = fma2(dx, dx, r2);
            float r0, r1;
            unpack2(r2, r0, r1);
            float i0 = rsqrt_ftz(r0), i1 = rsqrt_ftz(r1);
            if (SELF) {
                if (j0 + 2 * kp == self[t]) i0 = 0.f;
                if (j0 + 2 * kp + 1 == self[t]) i1 = 0.f;
            }
            const f2x ri = pack2(i0, i1);
            const f2x wr = mul2(W, ri);
            const f2x wr3 = mul2(mul2(wr, ri), ri);
            if (WANT_S) ps[t] = add2(ps[t], wr);
            pvx[t] = fma2(wr3, dx, pvx[t]);
            pvy[t] = fma2(wr3, dy, pvy[t]);
            pvz[t] = fma2(wr3, dz, pvz[t]);
        }
    }
}

__device__ __forceinline__ void fold2(float &s, float &c, f2x v) {
    float lo, hi;
    unpack2(v, lo, hi);
    two_sum_acc(s, c, lo + hi);
}

// One end of the pairs: na particles a, their sums over nb partners b with weights bw, in n_split slices of the partners.
struct AdjointSide {
    const float *bx, *by, *bz, *bw;
    int64_t nb;
    const float *ax, *ay, *az;
    int64_t na, self_off;
    int n_split;
    int64_t split_len;
    const float *vscale;
    float *out_s, *out_v;
    double *part;
};

// One warp per item: a tile of 32*T particles a against one slice of the partners b, streamed in
// chunks of 32 through a per-warp shared buffer; chunk partials folded into TwoSum-compensated sums.
// A slice's sums go to part[(slice * na + a) * NV + v] (v: the scalar sum if wanted, then the vector), added
// in slice order by adjoint_reduce_kernel; with one slice they are the result.
//
// Bound: the FP32 pipe (12 or 13 lane-operations a pair, 10 pairs per SM-cycle).  The partners are sliced so
// that several items wait for every warp slot (choose_slices): one item per tile left 94 warps for 3,000
// cells (150 us a sweep, now 11) and 2.06 blocks an SM, the third round nearly empty, for 160,000
// (19.6 ms, now 12.7).
template <int T, bool WANT_S>
__device__ __forceinline__ void adjoint_items(const AdjointSide &S, float eps2, int self_mask, int64_t block,
                                              float4 (*buf)[32]) {
    const float *__restrict__ bx = S.bx, *__restrict__ by = S.by, *__restrict__ bz = S.bz, *__restrict__ bw = S.bw;
    const float *__restrict__ ax = S.ax, *__restrict__ ay = S.ay, *__restrict__ az = S.az;
    const float *__restrict__ vscale = S.vscale;
    float *__restrict__ out_s = S.out_s, *__restrict__ out_v = S.out_v;
    double *__restrict__ part = S.part;
    const int64_t nb = S.nb, na = S.na, self_off = S.self_off, split_len = S.split_len;
    const int n_split = S.n_split;
    constexpr int NV = WANT_S ? 4 : 3;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float *sa = reinterpret_cast<float *>(buf[w]);        // 16 float4: x/y pairs
    float *sb = reinterpret_cast<float *>(buf[w] + 16);   // 16 float4: z/w pairs
    const int kp = lane >> 1, hf = lane & 1;
    const f2x e2 = pack2(eps2, eps2);
    const int64_t ntiles = (na + 32 * T - 1) / (32 * T);
    const int64_t item = block * kGWarps + w;
    if (item >= ntiles * n_split) return;
    const int64_t tile = item % ntiles;
    const int64_t slice = item / ntiles;
    const int64_t jb = slice * split_len, je = jb + split_len < nb ? jb + split_len : nb;
    f2x px[T], py[T], pz[T];
    float ss[T], sc[T], vxs[T], vxc[T], vys[T], vyc[T], vzs[T], vzc[T];
    int64_t self[T];
#pragma unroll
    for (int t = 0; t < T; ++t) {
        const int64_t a = tile * 32 * T + t * 32 + lane;
        const bool v = a < na;
        const float x = v ? ax[a] : kFarG, y = v ? ay[a] : kFarG, z = v ? az[a] : kFarG;
        px[t] = pack2(x, x);
        py[t] = pack2(y, y);
        pz[t] = pack2(z, z);
        self[t] = (v && self_mask) ? a + self_off : -1;
        ss[t] = sc[t] = vxs[t] = vxc[t] = vys[t] = vyc[t] = vzs[t] = vzc[t] = 0.f;
    }
    // partner indices self[t] lie in [lo_self, lo_self + 32 * T) for this tile
    const int64_t lo_self = tile * 32 * T + self_off;
    float4 nxt = load_b(bx, by, bz, bw, jb + lane, je);
    for (int64_t j0 = jb; j0 < je; j0 += 32) {
        __syncwarp();
        sa[kp * 4 + hf] = nxt.x;
        sa[kp * 4 + 2 + hf] = nxt.y;
        sb[kp * 4 + hf] = nxt.z;
        sb[kp * 4 + 2 + hf] = nxt.w;
        __syncwarp();
        nxt = load_b(bx, by, bz, bw, j0 + 32 + lane, je);
        f2x ps[T], pvx[T], pvy[T], pvz[T];
#pragma unroll
        for (int t = 0; t < T; ++t) ps[t] = pvx[t] = pvy[t] = pvz[t] = pack2(0.f, 0.f);
        const bool self_chunk = self_mask && j0 + 32 > lo_self && j0 < lo_self + 32 * T;
        if (self_chunk)
            adjoint_chunk<T, WANT_S, true>(buf[w], buf[w] + 16, px, py, pz, e2, j0, self, ps, pvx, pvy, pvz);
        else
            adjoint_chunk<T, WANT_S, false>(buf[w], buf[w] + 16, px, py, pz, e2, j0, self, ps, pvx, pvy, pvz);
#pragma unroll
        for (int t = 0; t < T; ++t) {
            if (WANT_S) fold2(ss[t], sc[t], ps[t]);
            fold2(vxs[t], vxc[t], pvx[t]);
            fold2(vys[t], vyc[t], pvy[t]);
            fold2(vzs[t], vzc[t], pvz[t]);
        }
    }
#pragma unroll
    for (int t = 0; t < T; ++t) {
        const int64_t a = tile * 32 * T + t * 32 + lane;
        if (a >= na) continue;
        if (n_split > 1) {
            double *p = part + (slice * na + a) * NV;
            if (WANT_S) p[0] = (double)ss[t] + (double)sc[t];
            p[NV - 3] = (double)vxs[t] + (double)vxc[t];
            p[NV - 2] = (double)vys[t] + (double)vyc[t];
            p[NV - 1] = (double)vzs[t] + (double)vzc[t];
            continue;
        }
        if (WANT_S && out_s) out_s[a] = ss[t] + sc[t];
        if (out_v) {
            const float sc_ = vscale[a];
            out_v[3 * a + 0] = sc_ * (vxs[t] + vxc[t]);
            out_v[3 * a + 1] = sc_ * (vys[t] + vyc[t]);
            out_v[3 * a + 2] = sc_ * (vzs[t] + vzc[t]);
        }
    }
}

template <int T, bool WANT_S>
__global__ void __launch_bounds__(32 * kGWarps) adjoint_kernel(AdjointSide side, float eps2, int self_mask) {
    __shared__ float4 buf[kGWarps][32];
    adjoint_items<T, WANT_S>(side, eps2, self_mask, blockIdx.x, buf);
}

// Both ends, one after the other's blocks: two sweeps too short for a launch each (a gradient of 3,000 cells is bound by the
// host's launches).
__global__ void __launch_bounds__(32 * kGWarps) adjoint_ends_kernel(AdjointSide t, AdjointSide s, unsigned t_blocks,
                                                                    float eps2, int self_mask) {
    __shared__ float4 buf[kGWarps][32];
    if (blockIdx.x < t_blocks) adjoint_items<2, false>(t, eps2, self_mask, blockIdx.x, buf);
    else adjoint_items<2, true>(s, eps2, self_mask, blockIdx.x - t_blocks, buf);
}

// The slices' sums in slice order (FP64), rounded to FP32 as a single slice's are, and scaled.
template <bool WANT_S>
__device__ __forceinline__ void adjoint_reduce(const AdjointSide &S, int64_t k) {
    constexpr int NV = WANT_S ? 4 : 3;
    const int64_t a = k / NV;
    const int v = (int)(k - a * NV) - (NV - 3);   // -1: the scalar sum
    double acc = 0.0;
#pragma unroll 8
    for (int s = 0; s < S.n_split; ++s) acc += S.part[(int64_t)s * S.na * NV + k];
    if (v < 0) {
        if (S.out_s) S.out_s[a] = (float)acc;
    } else if (S.out_v) {
        S.out_v[3 * a + v] = S.vscale[a] * (float)acc;
    }
}

// Of the ends that have several slices (the other's na is 0).
__global__ void __launch_bounds__(256) adjoint_reduce_kernel(AdjointSide t, AdjointSide s) {
    const int64_t nt = 3 * t.na, ns = 4 * s.na;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nt + ns; k += (int64_t)gridDim.x * blockDim.x) {
        if (k < nt) adjoint_reduce<false>(t, k);
        else adjoint_reduce<true>(s, k - nt);
    }
}

// Slices of the partners: about eight items per warp slot (16 warps an SM), at least 128 partners each, at most kMaxSlices,
// which one thread adds up, and at most 2^23 partial sums (64 MB) in all.  (100 targets x 2e6 sources, 9,728 slices:
// 1,470 us; 2,048 513, 1,024 383, 512 322, but 1,024 are 5 to 15 % faster for 5 to 20 sources x 10^7 targets.)
constexpr int64_t kMaxSlices = 1024;

void choose_slices(int64_t na, int64_t nb, int T, int nv, int *n_split, int64_t *split_len) {
    const int64_t ntiles = (na + 32 * T - 1) / (32 * T);
    int64_t s = ((int64_t)device_sm_count() * 16 * 8 + ntiles - 1) / ntiles;
    s = std::min(std::min(s, kMaxSlices), std::min<int64_t>(nb / 128, (1ll << 23) / (na * nv)));
    s = std::max<int64_t>(s, 1);
    const int64_t len = ((nb + s - 1) / s + 31) / 32 * 32;
    *n_split = (int)((nb + len - 1) / len);
    *split_len = len;
}

// ---- both sides of a pair at once -----------------------------------------------------------
// When the gradients of targets and sources are both wanted and there are enough pairs, one sweep gives them: distance,
// rsqrt and r^-3 of a pair are formed once, 17 lane-operations instead of 12 + 13, and the sources' four
// sums (r^-1 and the vector) are reduced over the warp's lanes (half a lane-operation a pair).
// A block of four warps holds 2,304 targets, eighteen a lane, and stages 288 sources; an item is one block of sources
// against `tblocks` blocks of targets, the sources' sums kept in shared memory (compensated) over them, the
// targets' too, a column a thread, as they are touched once in 32 sources.  Per item and target, or source, one
// partial sum is written; they are added in order.
// Bound: the FP32 pipe (17.5 lane-operations, the reduction with them, and a rsqrt a pair; 77 % busy).
// 160,000 x 200,000: 27.5 ms in two sweeps, 19.7 in one.  Fewer reductions and more independent pairs a warp gain more than warps: eight targets with their
// sums in registers and three blocks an SM 22.0 (512 sources), with the sums in shared memory 21.2 (256), sixteen
// and two blocks 20.5, eighteen with 192 to 320 sources 19.7 to 20.3; four targets, two sources an instruction 23.5.
constexpr int kBothT = 18, kBothTargets = 128 * kBothT, kBothSources = 288, kBothChunks = kBothSources / 32;

struct BothShared {
    float4 src[kBothSources][2];            // {x, x, y, y}, {z, z, m, m}
    float part[4][kBothSources][4];         // per warp: the sources' sums over the warp's targets of one block
    float sum[kBothSources][4], comp[kBothSources][4];
    float2 vec[3 * kBothT][128];            // a thread's targets' vectors: compensated sums
};

// 32 sources against the lane's targets, two targets a two-lane instruction.  r^-3 is formed once for both ends of a pair;
// with WIDE each end multiplies its weight in between, where r^-3 by itself could leave the range of normal
// numbers: softenings outside 2^-40 .. 2^40 or coordinates from 2^40 on.
constexpr float kBothReach = 0x1p40f;

template <bool SELF, bool WIDE>
__device__ __forceinline__ void both_chunk(const float4 (*src)[2], const f2x (&px)[kBothT / 2],
                                           const f2x (&py)[kBothT / 2], const f2x (&pz)[kBothT / 2],
                                           const f2x (&g)[kBothT / 2], f2x e2, int self0,
                                           f2x (&vx)[kBothT / 2], f2x (&vy)[kBothT / 2], f2x (&vz)[kBothT / 2],
                                           float *out, int lane) {
#pragma unroll 1
    for (int k0 = 0; k0 < 32; k0 += 4) {
        float v[16];   // sums of 4 sources: s, x, y, z of each
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float4 a = src[k0 + k][0], b = src[k0 + k][1];
            const f2x X = pack2(a.x, a.y), Y = pack2(a.z, a.w), Z = pack2(b.x, b.y), W = pack2(b.z, b.w);
            f2x s0 = pack2(0.f, 0.f), s1 = s0, s2 = s0, s3 = s0;
#pragma unroll
            for (int t = 0; t < kBothT / 2; ++t) {
                const f2x dx = sub2(X, px[t]), dy = sub2(Y, py[t]), dz = sub2(Z, pz[t]);
                f2x r2 = fma2(dz, dz, e2);
                r2 = fma2(dy, dy, r2);
                r2 = fma2(dx, dx, r2);
                float r0, r1;
                unpack2(r2, r0, r1);
                float i0 = rsqrt_ftz(r0), i1 = rsqrt_ftz(r1);
                if (SELF) {
                    if (k0 + k == self0 + 64 * t) i0 = 0.f;
                    if (k0 + k == self0 + 64 * t + 32) i1 = 0.f;
                }
                const f2x ri = pack2(i0, i1);
                const f2x ri2 = mul2(ri, ri);
                const f2x ri3 = mul2(ri, ri2);
                const f2x wr = WIDE ? mul2(mul2(W, ri), ri2) : mul2(W, ri3);
                const f2x gr3 = WIDE ? mul2(mul2(g[t], ri), ri2) : mul2(g[t], ri3);
                vx[t] = fma2(wr, dx, vx[t]);
                vy[t] = fma2(wr, dy, vy[t]);
                vz[t] = fma2(wr, dz, vz[t]);
                s0 = fma2(g[t], ri, s0);
                s1 = fma2(gr3, dx, s1);
                s2 = fma2(gr3, dy, s2);
                s3 = fma2(gr3, dz, s3);
            }
            float lo, hi;
            unpack2(s0, lo, hi);
            v[4 * k + 0] = lo + hi;
            unpack2(s1, lo, hi);
            v[4 * k + 1] = lo + hi;
            unpack2(s2, lo, hi);
            v[4 * k + 2] = lo + hi;
            unpack2(s3, lo, hi);
            v[4 * k + 3] = lo + hi;
        }
        // lane l and l ^ 1 get value l >> 1: source (l >> 3) of the four, component (l >> 1) & 3
        const float r = warp_reduce_scatter16(v, lane);
        if ((lane & 1) == 0) out[k0 * 4 + (lane >> 1)] = r;
    }
}

// part_t[(sb - sb0) * nt + i][3]: target i's vector over source block sb; part_s[tsb * nsrc + j - j0][4]: source j's sums
// over the targets of item column tsb (nsrc sources from j0 = sb0 * kBothSources on).
__global__ void __launch_bounds__(128, 2) adjoint_both_kernel(
    const float *__restrict__ sx, const float *__restrict__ sy, const float *__restrict__ sz,
    const float *__restrict__ sm, int64_t ns, const float *__restrict__ tx, const float *__restrict__ ty,
    const float *__restrict__ tz, const float *__restrict__ tg, int64_t nt, float eps2, int self_mask, int64_t self_off,
    int sb0, int nsb, int tblocks, float2 *__restrict__ part_t, float2 *__restrict__ part_s) {
    extern __shared__ __align__(16) unsigned char both_raw[];
    BothShared &sh = *reinterpret_cast<BothShared *>(both_raw);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int sbl = blockIdx.x % nsb;   // consecutive items share their targets
    const int tsb = blockIdx.x / nsb;
    const int64_t j0 = (int64_t)(sb0 + sbl) * kBothSources;
    const f2x e2 = pack2(eps2, eps2);
    auto beyond = [](const float4 &q) {
        return !(fmaxf(fabsf(q.x), fmaxf(fabsf(q.y), fabsf(q.z))) < kBothReach);
    };
    bool far = !(eps2 >= 0x1p-80f && eps2 <= 0x1p80f);
    for (int k = threadIdx.x; k < kBothSources; k += 128) {
        const float4 q = load_b(sx, sy, sz, sm, j0 + k, ns);
        far |= j0 + k < ns && beyond(q);
        sh.src[k][0] = make_float4(q.x, q.x, q.y, q.y);
        sh.src[k][1] = make_float4(q.z, q.z, q.w, q.w);
#pragma unroll
        for (int v = 0; v < 4; ++v) sh.sum[k][v] = sh.comp[k][v] = 0.f;
    }
    const bool far_sources = __syncthreads_or(far);
    for (int tb = 0; tb < tblocks; ++tb) {
        const int64_t i0 = ((int64_t)tsb * tblocks + tb) * kBothTargets;
        if (i0 >= nt) break;   // the same for the block
        const int64_t iw = i0 + w * 32 * kBothT;
        f2x px[kBothT / 2], py[kBothT / 2], pz[kBothT / 2], g[kBothT / 2];
        bool far_target = false;
#pragma unroll
        for (int t = 0; t < kBothT / 2; ++t) {
            float4 p[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int64_t i = iw + (2 * t + u) * 32 + lane;   // far and with zero weight past the end
                p[u] = i < nt ? make_float4(tx[i], ty[i], tz[i], tg[i]) : make_float4(-kFarG, -kFarG, -kFarG, 0.f);
                far_target |= i < nt && beyond(p[u]);
            }
            px[t] = pack2(p[0].x, p[1].x);
            py[t] = pack2(p[0].y, p[1].y);
            pz[t] = pack2(p[0].z, p[1].z);
            g[t] = pack2(p[0].w, p[1].w);
        }
#pragma unroll
        for (int v = 0; v < 3 * kBothT; ++v) sh.vec[v][threadIdx.x] = make_float2(0.f, 0.f);
        const bool wide = far_sources || __any_sync(0xffffffffu, far_target);
        const int64_t lo = iw + self_off - j0;   // self pairs: sources lo .. lo + 32 T - 1 of the block
        // the lane's first target's own source in the block; its t-th's is 32 t further (never, without self pairs)
        const int self0 = self_mask ? (int)std::max<int64_t>(std::min<int64_t>(lo + lane, 1 << 29), -(1 << 29)) : 1 << 29;
        for (int c = 0; c < kBothChunks; ++c) {
            f2x vx[kBothT / 2], vy[kBothT / 2], vz[kBothT / 2];
#pragma unroll
            for (int t = 0; t < kBothT / 2; ++t) vx[t] = vy[t] = vz[t] = pack2(0.f, 0.f);
            const float4 (*buf)[2] = sh.src + c * 32;
            float *out = &sh.part[w][c * 32][0];
            const bool own = self_mask && lo < c * 32 + 32 && lo + 32 * kBothT > c * 32;
            if (wide)
                both_chunk<true, true>(buf, px, py, pz, g, e2, self0 - c * 32, vx, vy, vz, out, lane);
            else if (own)
                both_chunk<true, false>(buf, px, py, pz, g, e2, self0 - c * 32, vx, vy, vz, out, lane);
            else
                both_chunk<false, false>(buf, px, py, pz, g, e2, self0 - c * 32, vx, vy, vz, out, lane);
#pragma unroll
            for (int t = 0; t < kBothT; t += 2) {
                const f2x q[3] = {vx[t / 2], vy[t / 2], vz[t / 2]};
#pragma unroll
                for (int v = 0; v < 3; ++v) {
                    float a, b;
                    unpack2(q[v], a, b);
                    float2 &s0 = sh.vec[3 * t + v][threadIdx.x], &s1 = sh.vec[3 * t + 3 + v][threadIdx.x];
                    float2 u = s0, w2 = s1;
                    two_sum_acc(u.x, u.y, a);
                    two_sum_acc(w2.x, w2.y, b);
                    s0 = u;
                    s1 = w2;
                }
            }
        }
#pragma unroll
        for (int t = 0; t < kBothT; ++t) {
            const int64_t i = iw + t * 32 + lane;
            if (i >= nt) continue;
            float2 *p = part_t + ((int64_t)sbl * nt + i) * 3;
#pragma unroll
            for (int v = 0; v < 3; ++v) p[v] = sh.vec[3 * t + v][threadIdx.x];
        }
        __syncthreads();
        for (int k = threadIdx.x; k < kBothSources * 4; k += 128) {   // the warps in order, compensated
            float *sum = &sh.sum[0][0] + k, *comp = &sh.comp[0][0] + k;
            float s = *sum, e = *comp;
#pragma unroll
            for (int q = 0; q < 4; ++q) two_sum_acc(s, e, (&sh.part[q][0][0])[k]);
            *sum = s;
            *comp = e;
        }
        __syncthreads();
    }
    for (int k = threadIdx.x; k < kBothSources * 4; k += 128)
        part_s[((int64_t)tsb * nsb + sbl) * kBothSources * 4 + k] =
            make_float2((&sh.sum[0][0])[k], (&sh.comp[0][0])[k]);
}

// After a band of source blocks: the targets' vectors over the band added to tot (first: set), and, after the last
// band, the gradients; the band's sources' sums over the item columns in order, and their gradients.  A partial sum is a
// compensated FP32 sum and its errors; they are added up the same way (in FP64 that pipe was the bound: 452 and
// 140 us of 160,000 targets x 200,000 sources, now, with more partial sums, 528 and 94).
__global__ void __launch_bounds__(256) both_targets_kernel(const float2 *__restrict__ part_t, int nsb, int64_t nt,
                                                           int first, int last, float2 *__restrict__ tot,
                                                           const float *__restrict__ scale, float *__restrict__ out) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < 3 * nt; k += (int64_t)gridDim.x * blockDim.x) {
        float2 acc = first ? make_float2(0.f, 0.f) : tot[k];
#pragma unroll 8
        for (int s = 0; s < nsb; ++s) {
            const float2 v = part_t[(int64_t)s * 3 * nt + k];
            two_sum_acc(acc.x, acc.y, v.x);
            acc.y += v.y;
        }
        if (last) out[k] = scale[k / 3] * (acc.x + acc.y);
        else tot[k] = acc;
    }
}

__global__ void __launch_bounds__(256) both_sources_kernel(const float2 *__restrict__ part_s, int ntsb, int64_t nsrc,
                                                           int64_t j0, int64_t ns, const float *__restrict__ m,
                                                           float *__restrict__ gm, float *__restrict__ gs) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < 4 * nsrc; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = j0 + k / 4;
        const int v = (int)(k & 3);
        if (j >= ns) continue;
        float2 acc = make_float2(0.f, 0.f);
#pragma unroll 8
        for (int s = 0; s < ntsb; ++s) {
            const float2 q = part_s[(int64_t)s * nsrc * 4 + k];
            two_sum_acc(acc.x, acc.y, q.x);
            acc.y += q.y;
        }
        const float sum = acc.x + acc.y;
        // the vector was summed as (source - target): the source's gradient points the other way
        if (v == 0) {
            if (gm) gm[j] = sum;
        } else if (gs) {
            gs[3 * j + v - 1] = m[j] * -sum;
        }
    }
}

// Scratch: the targets' partial sums of one band within kBothBand bytes (one source block at least).
constexpr int64_t kBothBand = 512ll << 20;
// Below kBothPairs pairs its blocks, 2,304 x 288 pairs for an item of four warps, are too few for the GPU: 1.2e8
// pairs take 144 us against 138 with an end's sums each on its own, 5e8 383 against 474.  Whole blocks are computed, so
// neither end may be much short of one: 3,700 targets (4,608 computed) x 10^6 sources 3,278 and 3,307 us, 3,400 3,277 and
// 3,078, 1,800 x 200,000 397 and 444, 1,000 x 200,000 393 and 361; 145 sources (288) x 1.4e6 targets 332 and 421, 100 x
// 2e6 504 and 428, 100 targets x 2e6 sources 3,458 and 383.
constexpr double kBothPairs = 1.5e8, kBothTargetPadding = 4.0 / 3.0, kBothSourcePadding = 2.0;

bool both_at_once(int64_t ns, int64_t nt) {
    auto padding = [](int64_t n, int64_t block) { return (double)((n + block - 1) / block * block) / (double)n; };
    return (double)ns * (double)nt >= kBothPairs && padding(nt, kBothTargets) <= kBothTargetPadding &&
           padding(ns, kBothSources) <= kBothSourcePadding;
}

struct BothPlan {
    int64_t nsb = 0, band = 0, ntsb = 0;   // source blocks, source blocks of a band, item columns
    int tblocks = 0;
    BothPlan(int64_t ns, int64_t nt) {
        nsb = (ns + kBothSources - 1) / kBothSources;
        band = std::min(nsb, std::max<int64_t>(1, kBothBand / (24 * nt)));
        const int64_t tb = (nt + kBothTargets - 1) / kBothTargets;
        // about 32 items for every block that fits on the GPU (two an SM), so that the last ones are short
        const int64_t columns = std::min(tb, std::max<int64_t>(1, ((int64_t)device_sm_count() * 64 + band - 1) / band));
        tblocks = (int)((tb + columns - 1) / columns);
        ntsb = (tb + tblocks - 1) / tblocks;
    }
    size_t bytes(int64_t nt) const {
        return sizeof(float2) * (size_t)(3 * nt * (band + 1) + ntsb * band * kBothSources * 4);
    }
};

int launch_both(const BothPlan &P, const float *sx, const float *sy, const float *sz, const float *m, int64_t ns,
                const float *tx, const float *ty, const float *tz, const float *g, int64_t nt, float eps2, int self,
                int64_t self_off, float *gm, float *gs, float *gt, float2 *scratch, cudaStream_t st) {
    float2 *part_t = scratch, *tot = part_t + 3 * nt * P.band, *part_s = tot + 3 * nt;
    const int smem = (int)sizeof(BothShared), cap = device_sm_count() * 8;
    HALMA_CUDA(cudaFuncSetAttribute(adjoint_both_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    for (int64_t sb0 = 0; sb0 < P.nsb; sb0 += P.band) {
        const int nsb = (int)std::min(P.band, P.nsb - sb0);
        const int64_t j0 = sb0 * kBothSources, nsrc = (int64_t)nsb * kBothSources;
        HALMA_LAUNCH(adjoint_both_kernel, (unsigned)(nsb * P.ntsb), 128, smem, st, sx, sy, sz, m, ns, tx, ty, tz, g, nt,
                     eps2, self, self_off, (int)sb0, nsb, P.tblocks, part_t, part_s);
        HALMA_LAUNCH(both_targets_kernel, grid_for(3 * nt, 256, cap), 256, 0, st, part_t, nsb, nt, sb0 == 0,
                     sb0 + nsb >= P.nsb, tot, g, gt);
        if (gm || gs)
            HALMA_LAUNCH(both_sources_kernel, grid_for(4 * nsrc, 256, cap), 256, 0, st, part_s, (int)P.ntsb, nsrc, j0, ns,
                         m, gm, gs);
    }
    return HALMA_OK;
}

// Targets a lane: four share the loads of a partner, but leave fewer items and, with the scalar sum, fewer warps an SM.
// Vectors alone: 3,000 against 4,000 20 us with two and 23 with four, 20,000 x 25,000 233 and 232, 160,000 x 200,000 13.4 ms
// and 12.7, 10^6 x 4e5 167 and 159; with the scalar two at every size (160,000 x 200,000: 14.2 and 14.5).
template <bool WANT_S>
int adjoint_targets(int64_t na) {
    return !WANT_S && na >= 16384 ? 4 : 2;
}

template <int T>
unsigned adjoint_blocks(const AdjointSide &S) {
    const int64_t items = (S.na + 32 * T - 1) / (32 * T) * S.n_split;
    return (unsigned)((items + kGWarps - 1) / kGWarps);
}

// The wanted ends (na > 0) in a sweep each, or in one launch where two lanes' targets suit both.
int launch_adjoint(AdjointSide t, AdjointSide s, float eps2, int self_mask, cudaStream_t st) {
    const bool wide = adjoint_targets<false>(t.na) == 4;
    if (t.na > 0 && s.na > 0 && !wide) {
        const unsigned tb = adjoint_blocks<2>(t), sb = adjoint_blocks<2>(s);
        HALMA_LAUNCH(adjoint_ends_kernel, tb + sb, 32 * kGWarps, 0, st, t, s, tb, eps2, self_mask);
    } else {
        if (t.na > 0 && wide)
            HALMA_LAUNCH((adjoint_kernel<4, false>), adjoint_blocks<4>(t), 32 * kGWarps, 0, st, t, eps2, self_mask);
        else if (t.na > 0)
            HALMA_LAUNCH((adjoint_kernel<2, false>), adjoint_blocks<2>(t), 32 * kGWarps, 0, st, t, eps2, self_mask);
        if (s.na > 0)
            HALMA_LAUNCH((adjoint_kernel<2, true>), adjoint_blocks<2>(s), 32 * kGWarps, 0, st, s, eps2, self_mask);
    }
    if (t.n_split == 1) t.na = 0;
    if (s.n_split == 1) s.na = 0;
    if (t.na + s.na > 0)
        HALMA_LAUNCH(adjoint_reduce_kernel, grid_for(3 * t.na + 4 * s.na, 256, device_sm_count() * 8), 256, 0, st, t, s);
    return HALMA_OK;
}

}  // namespace
}  // namespace halma

using namespace halma;

extern "C" int halma_potential_grad_f32(int64_t ns, const float *m_, const float *sx_, const float *sy_,
                                        const float *sz_, int64_t nt, const float *tx_, const float *ty_,
                                        const float *tz_, const float *g_, double eps2, int32_t mask,
                                        int64_t self_offset, float *grad_m, float *grad_src, float *grad_tgt,
                                        halma_stream_t stream) {
    if (ns < 0 || nt < 0) return fail(HALMA_ERR_INVALID, "negative size");
    if (mask != HALMA_MASK_SELF && mask != HALMA_MASK_NONE)
        return fail(HALMA_ERR_INVALID, "gradient supports the SELF and NONE masks only");
    if (!(eps2 >= 0.0) || !isfinite(eps2)) return fail(HALMA_ERR_INVALID, "eps2 must be finite and >= 0");
    if ((ns > 0 && (!m_ || !sx_ || !sy_ || !sz_)) || (nt > 0 && (!tx_ || !ty_ || !tz_ || !g_)))
        return fail(HALMA_ERR_INVALID, "null pointer");
    if (ns == 0 || nt == 0) {
        // empty sums: every requested gradient is zero
        std::lock_guard<std::mutex> guard(api_mutex());
        cudaStream_t st = (cudaStream_t)stream;
        float *outs[3] = {grad_m, grad_src, grad_tgt};
        const int64_t cnt[3] = {ns, 3 * ns, 3 * nt};
        for (int q = 0; q < 3; ++q) {
            if (!outs[q] || cnt[q] == 0) continue;
            if (is_device_pointer(outs[q])) HALMA_CUDA(cudaMemsetAsync(outs[q], 0, 4 * cnt[q], st));
            else memset(outs[q], 0, 4 * cnt[q]);
        }
        return HALMA_OK;
    }
    std::lock_guard<std::mutex> guard(api_mutex());
    cudaStream_t st = (cudaStream_t)stream;
    Stager sg;
    const float *m = nullptr, *sx = nullptr, *sy = nullptr, *sz = nullptr, *tx = nullptr, *ty = nullptr,
                *tz = nullptr, *g = nullptr;
    float *gm = nullptr, *gs = nullptr, *gt = nullptr;
    sg.add(m_, ns, true, false, &m);
    sg.add(sx_, ns, true, false, &sx);
    sg.add(sy_, ns, true, false, &sy);
    sg.add(sz_, ns, true, false, &sz);
    sg.add(tx_, nt, true, false, &tx);
    sg.add(ty_, nt, true, false, &ty);
    sg.add(tz_, nt, true, false, &tz);
    sg.add(g_, nt, true, false, &g);
    sg.add((const float *)grad_m, grad_m ? ns : 0, false, true, &gm);
    sg.add((const float *)grad_src, grad_src ? 3 * ns : 0, false, true, &gs);
    sg.add((const float *)grad_tgt, grad_tgt ? 3 * nt : 0, false, true, &gt);
    int split_t = 1, split_s = 1;
    int64_t len_t = ns, len_s = nt;
    if (grad_tgt) choose_slices(nt, ns, adjoint_targets<false>(nt), 3, &split_t, &len_t);
    if (grad_m || grad_src) choose_slices(ns, nt, adjoint_targets<true>(ns), 4, &split_s, &len_s);
    // both sides in one sweep where that suits the sizes, and with a softening that keeps r^-2 finite
    bool both = grad_tgt && (grad_m || grad_src) && both_at_once(ns, nt) && (float)eps2 >= 0x1p-126f;
    const BothPlan plan(ns, nt);
    // where the partial sums do not fit in what is left of the memory: in slices, then without any (slower)
    size_t o_part = 0, o_part_s = 0;
    void *base = nullptr;
    for (;;) {
        Layout L;
        sg.plan(L);
        o_part = L.add(both ? plan.bytes(nt) : split_t > 1 ? 8 * (size_t)(3 * nt * split_t) : 0);
        o_part_s = L.add(!both && split_s > 1 ? 8 * (size_t)(4 * ns * split_s) : 0);
        const int s = workspace(L.total, &base, st);
        if (s == HALMA_OK) break;
        if (s != HALMA_ERR_NOMEM || (!both && split_t == 1 && split_s == 1)) return s;
        if (!both) {
            split_t = split_s = 1;
            len_t = ns;
            len_s = nt;
        }
        both = false;
    }
    HALMA_TRY(sg.bind_and_upload(base, st));
    double *part = at<double>(base, o_part);
    const int self = mask == HALMA_MASK_SELF;
    if (both) {
        HALMA_TRY(launch_both(plan, sx, sy, sz, m, ns, tx, ty, tz, g, nt, (float)eps2, self, self_offset, gm, gs, gt,
                              reinterpret_cast<float2 *>(part), st));
        return sg.download(st);
    }
    HALMA_TRY(launch_adjoint({sx, sy, sz, m, ns, tx, ty, tz, gt ? nt : 0, self_offset, split_t, len_t, g, nullptr, gt, part},
                             {tx, ty, tz, g, nt, sx, sy, sz, gm || gs ? ns : 0, -self_offset, split_s, len_s, m, gm, gs,
                              at<double>(base, o_part_s)},
                             (float)eps2, self, st));
    return sg.download(st);
}
