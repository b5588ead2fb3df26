// Brute-force potential kernels and the C ABI that replaces the f2py symbol
// particle.particle.brute_force_binding_energy (particle_subroutines.f90:466-514).
//
// Layout: sources are read as float32 SoA (m, x, y, z) and staged per warp in shared memory
// as float4 chunks of 32; each lane owns T targets, so one shared-memory broadcast feeds T
// pair terms.  Work items are (target tile of 32*T, source slice); warps stride over items.
#include <math.h>

#include "common.cuh"
#include "pair_math.cuh"
#include "unbind.cuh"

namespace halma {

constexpr int kWarpsPerBlock = 8;
constexpr float kPadCoord = 3.0e30f;   // pad sources: m = 0 at a far point -> exact +0 term

__device__ __forceinline__ float4 load_source(const float *__restrict__ m, const float *__restrict__ x,
                                              const float *__restrict__ y, const float *__restrict__ z,
                                              int64_t j, int64_t end) {
    if (j < end) return make_float4(__ldg(x + j), __ldg(y + j), __ldg(z + j), __ldg(m + j));
    return make_float4(kPadCoord, kPadCoord, kPadCoord, 0.0f);
}

// ---- HALMA_POT_REFERENCE ------------------------------------------------------------------
// The Fortran loop body (f90:497-510) bit for bit: per target a float32 sum over the sources
// in order, every operation rounded on its own, a term m / sqrt(s) only where the source's x, y
// and z all differ from the target's.
//
// Only the additions have to follow one another; the terms do not depend on them.  So a block
// takes TL targets: eight warps compute the terms of 256 sources at a time into shared memory
// and a ninth adds the previous 256 in order (double buffered, one barrier a stage).  One
// warp doing both in turn left the GPU waiting on single dependent chains: 2,000 targets x
// 20,000 sources took 2.20 ms, 40,000 x 100,000 12.2 ms (2.2 warps on an SM's scheduler).
//
// So: 0.065 ms and 3.7 ms.
//
// The terms take 18 two-lane instructions for two, 3.5 terms per SM-cycle at 40,000 x 100,000, where no unit is full: FMA
// pipe 56 % busy, issue slots 54 %, shared memory 44 %.  Of 11 warp-cycles an issue 3.2 are spent at the barrier of a
// stage, 1.6 each on waits for shared memory and for the operation before, 1.5 on the pipe.
// Square root and quotient come from one rsqrt y of s by Markstein's correction steps (P. Markstein, Computation
// of elementary functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990):
// g = s y, r = g + (s - g g) y / 2;  z = y + y (1 - r y);  q = m z, t = q + (m - r q) z.  r is the
// rounded square root for every mantissa (checked over all 2^24 of two binades, in five
// scalings), z the rounded reciprocal of r -- where the theorem makes t the rounded quotient --
// except for four mantissas of s; of those, checked over all 2^23 mantissas of m, t is wrong
// for one m, a power of two, when r's mantissa is all ones.  Those pairs (looked for when a mass is a
// power of two), squared distances under 2^-90, coordinates or masses outside the ranges below
// and values that are not finite take the plain operations instead.
constexpr float kRefFar = 1.0e15f;                // sources past the end: m = 0 here gives +0 terms
constexpr float kRefMaxCoord = 0x1p48f, kRefMinMass = 0x1p-40f, kRefMaxMass = 0x1p80f, kRefMinS = 0x1p-90f;
enum { kRefPlain = 1, kRefPow2 = 2 };             // bits of the flags word

struct __align__(16) Src4 {   // four consecutive sources
    float4 x, y, z, m;
};

// The sources four by four, padded to whole stages, and the flags: kRefPlain when a coordinate or a
// mass is outside the ranges of the correction steps, kRefPow2 when a mass is a power of two.
__global__ void __launch_bounds__(256) ref_pack_kernel(
    const float *__restrict__ m, const float *__restrict__ x, const float *__restrict__ y,
    const float *__restrict__ z, int64_t ns, int64_t nquads, const float *__restrict__ tx,
    const float *__restrict__ ty, const float *__restrict__ tz, int64_t nt, Src4 *__restrict__ src,
    int *__restrict__ flags) {
    int f = 0;
    auto coord = [&](float v) {
        if (!(fabsf(v) < kRefMaxCoord)) f |= kRefPlain;
        return v;
    };
    const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t q = i0; q < nquads; q += step) {
        float v[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int64_t j = 4 * q + k;
            const bool in = j < ns;
            v[0][k] = in ? coord(x[j]) : kRefFar;
            v[1][k] = in ? coord(y[j]) : kRefFar;
            v[2][k] = in ? coord(z[j]) : kRefFar;
            const float mj = in ? m[j] : 0.f;
            v[3][k] = mj;
            if (mj != 0.f) {   // true for NaN
                if (!(fabsf(mj) >= kRefMinMass && fabsf(mj) <= kRefMaxMass)) f |= kRefPlain;
                if ((__float_as_int(mj) & 0x7fffff) == 0) f |= kRefPow2;
            }
        }
        Src4 o;
        o.x = make_float4(v[0][0], v[0][1], v[0][2], v[0][3]);
        o.y = make_float4(v[1][0], v[1][1], v[1][2], v[1][3]);
        o.z = make_float4(v[2][0], v[2][1], v[2][2], v[2][3]);
        o.m = make_float4(v[3][0], v[3][1], v[3][2], v[3][3]);
        src[q] = o;
    }
    for (int64_t i = i0; i < nt; i += step) {
        coord(tx[i]);
        coord(ty[i]);
        coord(tz[i]);
    }
    f = __reduce_or_sync(0xffffffffu, f);
    if (f && (threadIdx.x & 31) == 0) atomicOr(flags, f);
}

// Two terms by the correction steps (+0 where the mask drops the pair); smin follows the smallest
// s met, ones is set when a square root's mantissa is all ones (ONES).  The squares are
// multiply-adds of nz = -0, a kernel argument: the compiler contracts a two-lane product and the
// sum that takes it (also with .rn, and when it knows the -0), which would leave the product unrounded.
template <bool ONES>
__device__ __forceinline__ f2x ref_terms2(f2x X, f2x Y, f2x Z, float m0, float m1, f2x tx, f2x ty, f2x tz, f2x nz,
                                          float &smin, bool &ones) {
    const f2x dx = sub2(X, tx), dy = sub2(Y, ty), dz = sub2(Z, tz);
    const f2x s = add2(add2(fma2(dx, dx, nz), fma2(dy, dy, nz)), fma2(dz, dz, nz));
    float a0, a1, b0, b1, c0, c1, s0, s1;
    unpack2(dx, a0, a1);
    unpack2(dy, b0, b1);
    unpack2(dz, c0, c1);
    unpack2(s, s0, s1);
    // x, y and z all differ <=> no difference is zero (subnormals are kept)
    const bool k0 = fminf(fminf(fabsf(a0), fabsf(b0)), fabsf(c0)) > 0.f;
    const bool k1 = fminf(fminf(fabsf(a1), fabsf(b1)), fabsf(c1)) > 0.f;
    smin = fminf(fminf(smin, s0), s1);
    const f2x M = pack2(k0 ? m0 : 0.f, k1 ? m1 : 0.f);
    const f2x y = pack2(rsqrt_ftz(s0), rsqrt_ftz(s1));
    const f2x g = mul2(s, y), ng = mul2(g, pack2(-1.f, -1.f));
    const f2x nr = fma2(fma2(ng, g, s), mul2(y, pack2(-0.5f, -0.5f)), ng);   // minus the square root
    if (ONES) {
        float r0, r1;
        unpack2(nr, r0, r1);
        ones |= ((~__float_as_int(r0) & 0x7fffff) == 0) | ((~__float_as_int(r1) & 0x7fffff) == 0);
    }
    const f2x iz = fma2(y, fma2(nr, y, pack2(1.f, 1.f)), y);
    const f2x q = mul2(M, iz);
    return fma2(fma2(nr, q, M), iz, q);
}

// The lane's quads q0, q0 + step, .. (N of them) of its warp's sources against its target, terms to
// out[quad][TL].
template <int TL, int N, bool ONES>
__device__ __forceinline__ bool ref_quads(const Src4 *src, int q0, float px, float py, float pz, float nzero,
                                          float4 *__restrict__ out, int t) {
    const f2x tx = pack2(px, px), ty = pack2(py, py), tz = pack2(pz, pz), nz = pack2(nzero, nzero);
    float smin = kRefMaxCoord;
    bool ones = false;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int q = q0 + i * (32 / TL);
        const float4 X = src[q].x, Y = src[q].y, Z = src[q].z, M = src[q].m;
        const f2x lo = ref_terms2<ONES>(pack2(X.x, X.y), pack2(Y.x, Y.y), pack2(Z.x, Z.y), M.x, M.y, tx, ty, tz,
                                        nz, smin, ones);
        const f2x hi = ref_terms2<ONES>(pack2(X.z, X.w), pack2(Y.z, Y.w), pack2(Z.z, Z.w), M.z, M.w, tx, ty, tz,
                                        nz, smin, ones);
        float4 v;
        unpack2(lo, v.x, v.y);
        unpack2(hi, v.z, v.w);
        out[q * TL + t] = v;
    }
    return smin < kRefMinS || ones;
}

// The same with the plain operations.
template <int TL, int N>
__device__ __noinline__ void ref_quads_plain(const Src4 *src, int q0, float px, float py, float pz,
                                             float4 *__restrict__ out, int t) {
    for (int i = 0; i < N; ++i) {
        const int q = q0 + i * (32 / TL);
        const float4 X = src[q].x, Y = src[q].y, Z = src[q].z, M = src[q].m;
        float4 v;
        v.x = pair_term_reference(make_float4(X.x, Y.x, Z.x, M.x), px, py, pz);
        v.y = pair_term_reference(make_float4(X.y, Y.y, Z.y, M.y), px, py, pz);
        v.z = pair_term_reference(make_float4(X.z, Y.z, Z.z, M.z), px, py, pz);
        v.w = pair_term_reference(make_float4(X.w, Y.w, Z.w, M.w), px, py, pz);
        out[q * TL + t] = v;
    }
}

// TL targets a block.  Wide (32): eight warps compute, the ninth adds, for target counts that keep
// the SMs busy; there the terms are the bound (at most three such blocks fit an SM).  Narrow (8):
// for fewer targets the additions are, 4.1 cycles each at best; six warps compute, and the adding
// warp has a scheduler (every fourth warp) to itself: it shares it only with the adding warps of
// the SM's other blocks (sharing it with computing warps: 7 us more of 65 at 2,000 x 20,000).
template <int TL>
struct RefShape {
    static constexpr bool wide = TL == 32;
    static constexpr int computing = wide ? 8 : 6, warps = wide ? 9 : 8;
    static constexpr int take = wide ? 8 : 16;       // quads of a warp in one stage
    static constexpr int quads = computing * take;   // of all
    __device__ static int computes(int w) { return wide ? w : (w % 4 == 3 ? -1 : w - w / 4); }   // its share, or -1
    __device__ static bool adds(int w) { return w == (wide ? 8 : 3); }
};

template <int TL>
__global__ void __launch_bounds__(RefShape<TL>::warps * 32) ref_potential_kernel(
    const Src4 *__restrict__ src, int64_t nstages, const float *__restrict__ tx, const float *__restrict__ ty,
    const float *__restrict__ tz, int64_t nt, const int *__restrict__ flags, float nzero, int first, int leave_plain,
    float *__restrict__ out) {
    using S = RefShape<TL>;
    constexpr int N = S::take * TL / 32;    // quads of a lane in one stage
    extern __shared__ float4 ref_terms[];    // [2][S::quads][TL]
    __shared__ Src4 quads[S::computing][2][S::take];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int share = w < S::warps - (S::wide ? 1 : 0) ? S::computes(w) : -1;
    const int t = lane % TL;
    const int64_t i = (int64_t)blockIdx.x * TL + t;
    const int64_t it = i < nt ? i : nt - 1;
    const float px = tx[it], py = ty[it], pz = tz[it];
    const int fl = *flags;
    if (leave_plain && (fl & kRefPlain)) return;   // ref_direct_kernel's
    // every warp copies its own next sources while it computes
    auto fetch = [&](int64_t st) {
        if (st < nstages) {
            const float4 *from = reinterpret_cast<const float4 *>(src + st * S::quads + share * S::take);
            float4 *to = reinterpret_cast<float4 *>(quads[share][st & 1]);
#pragma unroll
            for (int k = lane; k < S::take * 4; k += 32)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 (unsigned)__cvta_generic_to_shared(to + k)),
                             "l"(from + k)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (share >= 0) fetch(0);
    float acc = first ? 0.f : out[it];   // the sources before these
    for (int64_t st = 0; st <= nstages; ++st) {
        if (share >= 0 && st < nstages) {
            fetch(st + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            float4 *buf = ref_terms + ((st & 1) * S::quads + share * S::take) * TL;
            const Src4 *s = quads[share][st & 1];
            bool again = (fl & kRefPlain) != 0;
            if (!again)
                again = (fl & kRefPow2) ? ref_quads<TL, N, true>(s, lane / TL, px, py, pz, nzero, buf, t)
                                        : ref_quads<TL, N, false>(s, lane / TL, px, py, pz, nzero, buf, t);
            if (again) ref_quads_plain<TL, N>(s, lane / TL, px, py, pz, buf, t);
        } else if (S::adds(w) && st > 0 && lane < TL) {
            const float4 *buf = ref_terms + ((st - 1) & 1) * S::quads * TL;
            // the next eight loads are in flight during the 32 additions of the last eight
            float4 v[8], u[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = buf[k * TL + t];
#pragma unroll
            for (int q = 0; q < S::quads; q += 8) {
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (q + 8 < S::quads) u[k] = buf[(q + 8 + k) * TL + t];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, v[k].x), v[k].y), v[k].z), v[k].w);
                    v[k] = u[k];
                }
            }
        }
        __syncthreads();
    }
    if (S::adds(w) && lane < TL && i < nt) out[i] = acc;
}

// The same with a target a thread and the plain operations, for few sources or many targets with values that need them: no
// stage to fill, and every thread computes.  With kRefDirect sources or fewer it is the one launch: 40 sources x 300,000
// targets 49 us, 113 through the stages; from kRefManyTargets targets on with kRefDirectMany (300 x 300,000 151 and 173,
// 300 x 30,000 77 and 59).  Of those many targets it also takes the pieces whose values need the plain operations throughout
// (only_plain: the flag says so, else it leaves): 3,000 x 300,000 1,328 us through the stages, 1,099 so; fewer targets are
// better off with eight warps for the terms of 32 (3,000 x 30,000 374 us here, 207 there).
constexpr int64_t kRefDirect = 64, kRefDirectMany = 320, kRefManyTargets = 100000;

__global__ void __launch_bounds__(256) ref_direct_kernel(const float *__restrict__ m, const float *__restrict__ x,
                                                         const float *__restrict__ y, const float *__restrict__ z,
                                                         int64_t ns, const float *__restrict__ tx,
                                                         const float *__restrict__ ty, const float *__restrict__ tz,
                                                         int64_t nt, const int *__restrict__ only_plain, int first,
                                                         float *__restrict__ out) {
    if (only_plain && !(*only_plain & kRefPlain)) return;
    __shared__ float4 buf[256];
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool in = i < nt;
    const float px = in ? tx[i] : 0.f, py = in ? ty[i] : 0.f, pz = in ? tz[i] : 0.f;
    float acc = first || !in ? 0.f : out[i];
    for (int64_t j0 = 0; j0 < ns; j0 += 256) {
        const int cnt = (int)min((int64_t)256, ns - j0);
        __syncthreads();
        if ((int)threadIdx.x < cnt) {
            const int64_t j = j0 + threadIdx.x;
            buf[threadIdx.x] = make_float4(x[j], y[j], z[j], m[j]);
        }
        __syncthreads();
        for (int k = 0; k < cnt; ++k) acc = __fadd_rn(acc, pair_term_reference(buf[k], px, py, pz));
    }
    if (in) out[i] = acc;
}

// Packs the sources and runs the kernel, kRefPiece sources at a time (64 MB of packed ones); src holds the quads of a piece.
constexpr int64_t kRefPiece = 1ll << 22;

template <int TL>
static int64_t ref_quads_of(int64_t ns) {
    const int64_t q = RefShape<TL>::quads;
    return ((std::min(ns, kRefPiece) + 3) / 4 + q - 1) / q * q;
}

template <int TL>
static int launch_reference(const float *m, const float *x, const float *y, const float *z, int64_t ns, const float *tx,
                            const float *ty, const float *tz, int64_t nt, Src4 *src, int *flags, float *out,
                            cudaStream_t st) {
    using S = RefShape<TL>;
    constexpr int smem = 2 * S::quads * TL * (int)sizeof(float4);
    HALMA_CUDA(cudaFuncSetAttribute(ref_potential_kernel<TL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    for (int64_t j = 0; j < ns; j += kRefPiece) {
        const int64_t n = std::min(kRefPiece, ns - j), nquads = ref_quads_of<TL>(n);
        HALMA_CUDA(cudaMemsetAsync(flags, 0, sizeof(int), st));
        HALMA_LAUNCH(ref_pack_kernel, grid_for(std::max(nquads, nt), 256, device_sm_count() * 8), 256, 0, st, m + j, x + j,
                     y + j, z + j, n, nquads, tx, ty, tz, nt, src, flags);
        HALMA_LAUNCH(ref_potential_kernel<TL>, (unsigned)((nt + TL - 1) / TL), S::warps * 32, smem, st, src,
                     nquads / S::quads, tx, ty, tz, nt, flags, -0.0f, j == 0, nt >= kRefManyTargets, out);
        if (nt >= kRefManyTargets)
            HALMA_LAUNCH(ref_direct_kernel, grid_for(nt, 256), 256, 0, st, m + j, x + j, y + j, z + j, n, tx, ty, tz, nt,
                         flags, j == 0, out);
    }
    return HALMA_OK;
}

// HALMA_POT_FAST and the softened potential: T targets per lane, FP32 rsqrt pair terms, each 32-source
// chunk summed in FP32 and folded into a TwoSum-compensated accumulator.
// MASK: HALMA_MASK_COORD (reference mask), HALMA_MASK_SELF (skip j == i + self_offset) or
// HALMA_MASK_NONE.  FTZ: eps2 is a normal float, so that no r^2 is subnormal and the rsqrt that
// flushes subnormal arguments gives the same values (one instruction instead of five).
//
// Bound: the special-function unit (one rsqrt a term) and the FP32 pipe (7 lane-operations) together, as
// the unbinding's tile kernel: two sources per two-lane instruction.  With one-lane instructions the
// star terms of a 160,000-cell gas halo (6.4e9) took 2.29 ms, now 1.69.
template <bool FTZ>
__device__ __forceinline__ float pot_rsqrt(float v) {
    return FTZ ? rsqrt_ftz(v) : rsqrtf(v);
}

// The chunk's 32 sources (sa[kp] = {x, x, y, y} of sources 2 kp and 2 kp + 1, sb[kp] = {z, z, m, m}) against
// the lane's T targets.  SELF: source number self[t] of the chunk is skipped.
template <int T, int MASK, bool FTZ, bool SELF>
__device__ __forceinline__ void pot_chunk(const float4 *sa, const float4 *sb, const f2x (&px)[T], const f2x (&py)[T],
                                          const f2x (&pz)[T], f2x e2, const int (&self)[T], f2x (&acc)[T]) {
#pragma unroll 4
    for (int kp = 0; kp < 16; ++kp) {
        const float4 a = sa[kp], b = sb[kp];
        const f2x X = pack2(a.x, a.y), Y = pack2(a.z, a.w), Z = pack2(b.x, b.y), M = pack2(b.z, b.w);
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const f2x dx = sub2(X, px[t]), dy = sub2(Y, py[t]), dz = sub2(Z, pz[t]);
            f2x r2 = fma2(dz, dz, e2);
            r2 = fma2(dy, dy, r2);
            r2 = fma2(dx, dx, r2);
            float r0, r1;
            unpack2(r2, r0, r1);
            float i0 = pot_rsqrt<FTZ>(r0), i1 = pot_rsqrt<FTZ>(r1);
            if (MASK == HALMA_MASK_COORD) {   // the coordinates themselves: equal infinities drop the pair too
                float qx, qy, qz, hi;
                unpack2(px[t], qx, hi);
                unpack2(py[t], qy, hi);
                unpack2(pz[t], qz, hi);
                if (!((a.x != qx) & (a.z != qy) & (b.x != qz))) i0 = 0.f;
                if (!((a.y != qx) & (a.w != qy) & (b.y != qz))) i1 = 0.f;
            }
            if (SELF) {   // the term, not its factor: the mass may be infinite
                const bool skip0 = 2 * kp == self[t], skip1 = 2 * kp + 1 == self[t];
                acc[t] = fma2(pack2(skip0 ? 0.f : b.z, skip1 ? 0.f : b.w), pack2(skip0 ? 0.f : i0, skip1 ? 0.f : i1), acc[t]);
            } else {
                acc[t] = fma2(M, pack2(i0, i1), acc[t]);
            }
        }
    }
}

// One item by a warp: 32 T targets from t0 on against the sources jb .. je; their compensated sums.
template <int T, int MASK, bool FTZ>
__device__ __forceinline__ void pot_item(const float *__restrict__ m, const float *__restrict__ x,
                                         const float *__restrict__ y, const float *__restrict__ z, int64_t jb, int64_t je,
                                         const float *__restrict__ tx, const float *__restrict__ ty,
                                         const float *__restrict__ tz, int64_t t0, int64_t nt, float eps2,
                                         int64_t self_offset, float4 *buf, int lane, float (&sum)[T], float (&comp)[T]) {
    float *sa = reinterpret_cast<float *>(buf);        // 16 float4: x and y pairs
    float *sb = reinterpret_cast<float *>(buf + 16);   // 16 float4: z and m pairs
    const int kp = lane >> 1, hf = lane & 1;
    const f2x e2 = pack2(eps2, eps2);
    f2x px[T], py[T], pz[T];
#pragma unroll
    for (int t = 0; t < T; ++t) {
        const int64_t i = t0 + t * 32 + lane;
        const bool v = i < nt;
        const float cx = v ? tx[i] : kPadCoord, cy = v ? ty[i] : kPadCoord, cz = v ? tz[i] : kPadCoord;
        px[t] = pack2(cx, cx);
        py[t] = pack2(cy, cy);
        pz[t] = pack2(cz, cz);
        sum[t] = 0.f;
        comp[t] = 0.f;
    }
    // the tile's self pairs are with the sources lo_self .. lo_self + 32 T - 1
    const int64_t lo_self = t0 + self_offset;
    float4 nxt = load_source(m, x, y, z, jb + lane, je);
    for (int64_t j0 = jb; j0 < je; j0 += 32) {
        __syncwarp();
        sa[kp * 4 + hf] = nxt.x;
        sa[kp * 4 + 2 + hf] = nxt.y;
        sb[kp * 4 + hf] = nxt.z;
        sb[kp * 4 + 2 + hf] = nxt.w;
        __syncwarp();
        nxt = load_source(m, x, y, z, j0 + 32 + lane, je);
        f2x acc[T];
        int self[T];
#pragma unroll
        for (int t = 0; t < T; ++t) {
            acc[t] = pack2(0.f, 0.f);
            self[t] = -1;
        }
        if (MASK == HALMA_MASK_SELF && j0 + 32 > lo_self && j0 < lo_self + 32 * T) {
#pragma unroll
            for (int t = 0; t < T; ++t) self[t] = (int)(lo_self + t * 32 + lane - j0);
            pot_chunk<T, MASK, FTZ, true>(buf, buf + 16, px, py, pz, e2, self, acc);
        } else {
            pot_chunk<T, MASK, FTZ, false>(buf, buf + 16, px, py, pz, e2, self, acc);
        }
#pragma unroll
        for (int t = 0; t < T; ++t) {
            float a0, a1;
            unpack2(acc[t], a0, a1);
            two_sum_acc(sum[t], comp[t], a0 + a1);
        }
    }
}

template <int T, int MASK, bool FTZ>
__global__ void __launch_bounds__(256) bf_potential_fast_kernel(
    const float *__restrict__ m, const float *__restrict__ x, const float *__restrict__ y,
    const float *__restrict__ z, int64_t ns, const float *__restrict__ tx,
    const float *__restrict__ ty, const float *__restrict__ tz, int64_t nt, float eps2,
    int n_split, int64_t split_len, int64_t self_offset, float *__restrict__ out,
    double *__restrict__ partial) {
    __shared__ float4 buf[kWarpsPerBlock][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t gwarp = (int64_t)blockIdx.x * kWarpsPerBlock + w;
    const int64_t nwarps = (int64_t)gridDim.x * kWarpsPerBlock;
    const int64_t ntiles = (nt + 32 * T - 1) / (32 * T);
    const int64_t nitems = ntiles * n_split;
    for (int64_t item = gwarp; item < nitems; item += nwarps) {
        const int64_t tile = item / n_split;
        const int s = (int)(item - tile * n_split);
        const int64_t jb = (int64_t)s * split_len;
        float sum[T], comp[T];
        pot_item<T, MASK, FTZ>(m, x, y, z, jb, min(ns, jb + split_len), tx, ty, tz, tile * 32 * T, nt, eps2, self_offset,
                               buf[w], lane, sum, comp);
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int64_t i = tile * 32 * T + t * 32 + lane;
            if (i < nt) {
                if (n_split == 1) out[i] = sum[t] + comp[t];
                else partial[(int64_t)s * nt + i] = (double)sum[t] + (double)comp[t];
            }
        }
    }
}

// The slices of 32 targets by one block, their sums added there in the same order: for up to kBlockSlices slices, without
// memory for the partial sums (the allocation-free entry point).
constexpr int kBlockSlices = 32;

template <bool FTZ>
__global__ void __launch_bounds__(256) bf_potential_block_kernel(
    const float *__restrict__ m, const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
    int64_t ns, const float *__restrict__ tx, const float *__restrict__ ty, const float *__restrict__ tz, int64_t nt,
    float eps2, int n_split, int64_t split_len, float *__restrict__ out) {
    __shared__ float4 buf[kWarpsPerBlock][32];
    __shared__ double part[kBlockSlices][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t t0 = (int64_t)blockIdx.x * 32;
    for (int s = w; s < n_split; s += kWarpsPerBlock) {
        const int64_t jb = (int64_t)s * split_len;
        float sum[1], comp[1];
        pot_item<1, HALMA_MASK_COORD, FTZ>(m, x, y, z, jb, min(ns, jb + split_len), tx, ty, tz, t0, nt, eps2, 0, buf[w],
                                           lane, sum, comp);
        part[s][lane] = (double)sum[0] + (double)comp[0];
    }
    __syncthreads();
    if (w == 0 && t0 + lane < nt) {
        double acc = 0.0;
        for (int s = 0; s < n_split; ++s) acc += part[s][lane];
        out[t0 + lane] = (float)acc;
    }
}

// Deterministic combine of the per-slice partial sums (fixed slice order, FP64).
__global__ void reduce_partials_kernel(const double *__restrict__ partial, int n_split, int64_t nt,
                                       float *__restrict__ out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nt;
         i += (int64_t)gridDim.x * blockDim.x) {
        double acc = 0.0;
#pragma unroll 8
        for (int s = 0; s < n_split; ++s) acc += partial[(int64_t)s * nt + i];
        out[i] = (float)acc;
    }
}

// Plain FP64 path: one target per thread, FP64 pair terms and FP64 sum.
__global__ void __launch_bounds__(256) potential_f64_kernel(
    const double *__restrict__ m, const double *__restrict__ sx, const double *__restrict__ sy,
    const double *__restrict__ sz, int64_t ns, const double *__restrict__ tx,
    const double *__restrict__ ty, const double *__restrict__ tz, int64_t nt, double eps2,
    int mask, int64_t self_offset, double *__restrict__ phi) {
    __shared__ double4 buf[256];
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const bool valid = i < nt;
    const double px = valid ? tx[i] : 0.0, py = valid ? ty[i] : 0.0, pz = valid ? tz[i] : 0.0;
    const int64_t self = valid ? i + self_offset : -1;
    double acc = 0.0;
    for (int64_t j0 = 0; j0 < ns; j0 += 256) {
        const int64_t j = j0 + threadIdx.x;
        __syncthreads();
        buf[threadIdx.x] = (j < ns) ? make_double4(sx[j], sy[j], sz[j], m[j]) : make_double4(0, 0, 0, 0);
        __syncthreads();
        const int cnt = (int)min((int64_t)256, ns - j0);
        for (int k = 0; k < cnt; ++k) {
            const double4 q = buf[k];
            const double dx = q.x - px, dy = q.y - py, dz = q.z - pz;
            bool keep = true;
            if (mask == HALMA_MASK_COORD) keep = (q.x != px) && (q.y != py) && (q.z != pz);
            else if (mask == HALMA_MASK_SELF) keep = (j0 + k) != self;
            const double r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
            if (keep) acc = fma(q.w, rsqrt(r2), acc);
        }
    }
    if (valid) phi[i] = acc;
}

constexpr int64_t kMaxPartials = 1ll << 21;   // partial sums of one call, from the finer slices below
constexpr int64_t kCoarseSlice = 2048, kFineSlice = 128;   // sources of a slice at least
static_assert(2 * kCoarseSlice <= kBlockSlices * kFineSlice, "fewer sources have at most kBlockSlices slices");

// Number of source slices so that (target tiles x slices) keeps every SM busy.  Slices have at least
// 2048 sources, or 128 while the partial sums stay within kMaxPartials: 3,000 targets x 4,000
// sources took 248 us in one slice (24 warps), 12 us in 32.
static void choose_split(int64_t ns, int64_t nt, int T, int *n_split, int64_t *split_len) {
    const int sms = device_sm_count();
    const int64_t ntiles = (nt + 32 * T - 1) / (32 * T);
    const int64_t want_items = (int64_t)sms * 64;   // ~2 waves of resident warps
    int64_t s = 1;
    if (ntiles < want_items) s = (want_items + ntiles - 1) / ntiles;
    s = std::min<int64_t>(s, 1024);
    const int64_t coarse = std::min(s, std::max<int64_t>(1, ns / kCoarseSlice));
    const int64_t fine = std::min(s, std::min(ns / kFineSlice, kMaxPartials / nt));
    s = std::max(coarse, fine);
    int64_t len = (ns + s - 1) / s;
    len = (len + 31) / 32 * 32;
    s = std::max<int64_t>(1, (ns + len - 1) / len);
    *n_split = (int)s;
    *split_len = std::max<int64_t>(len, 32);
}

template <int T, bool FTZ>
static int launch_fast_mask(const float *m, const float *x, const float *y, const float *z, int64_t ns,
                            const float *tx, const float *ty, const float *tz, int64_t nt, float eps2,
                            int n_split, int64_t split_len, int mask, int64_t self_offset, float *out,
                            double *partial, cudaStream_t st) {
    const int64_t ntiles = (nt + 32 * T - 1) / (32 * T);
    const int64_t nitems = ntiles * n_split;
    const int sms = device_sm_count();
    const int grid = (int)std::min<int64_t>((nitems + kWarpsPerBlock - 1) / kWarpsPerBlock, (int64_t)sms * 8);
    if (mask == HALMA_MASK_COORD)
        HALMA_LAUNCH((bf_potential_fast_kernel<T, HALMA_MASK_COORD, FTZ>), grid, 256, 0, st, m, x, y, z, ns, tx, ty,
                     tz, nt, eps2, n_split, split_len, self_offset, out, partial);
    else if (mask == HALMA_MASK_SELF)
        HALMA_LAUNCH((bf_potential_fast_kernel<T, HALMA_MASK_SELF, FTZ>), grid, 256, 0, st, m, x, y, z, ns, tx, ty, tz,
                     nt, eps2, n_split, split_len, self_offset, out, partial);
    else
        HALMA_LAUNCH((bf_potential_fast_kernel<T, HALMA_MASK_NONE, FTZ>), grid, 256, 0, st, m, x, y, z, ns, tx, ty, tz,
                     nt, eps2, n_split, split_len, self_offset, out, partial);
    return HALMA_OK;
}

template <int T>
static int launch_fast(const float *m, const float *x, const float *y, const float *z, int64_t ns,
                       const float *tx, const float *ty, const float *tz, int64_t nt, float eps2,
                       int n_split, int64_t split_len, int mask, int64_t self_offset, float *out,
                       double *partial, cudaStream_t st) {
    return eps2 >= 0x1p-126f ? launch_fast_mask<T, true>(m, x, y, z, ns, tx, ty, tz, nt, eps2, n_split, split_len,
                                                         mask, self_offset, out, partial, st)
                             : launch_fast_mask<T, false>(m, x, y, z, ns, tx, ty, tz, nt, eps2, n_split, split_len,
                                                          mask, self_offset, out, partial, st);
}

// Stages the caller's arrays and runs the FP32-compensated kernel with the given mask.
static int potential_fast_api(int64_t ns, const float *mm, const float *sx_, const float *sy_, const float *sz_,
                              int64_t nt, const float *tx_, const float *ty_, const float *tz_, double eps2,
                              int mask, int64_t self_offset, float *out_, cudaStream_t st) {
    constexpr int T = 4;
    int n_split = 1;
    int64_t split_len = ns;
    if (ns > 0) choose_split(ns, nt, T, &n_split, &split_len);
    Stager sg;
    const float *m = nullptr, *x = nullptr, *y = nullptr, *z = nullptr, *tx = nullptr, *ty = nullptr, *tz = nullptr;
    float *out = nullptr;
    sg.add(mm, ns, true, false, &m);
    sg.add(sx_, ns, true, false, &x);
    sg.add(sy_, ns, true, false, &y);
    sg.add(sz_, ns, true, false, &z);
    sg.add(tx_, nt, true, false, &tx);
    sg.add(ty_, nt, true, false, &ty);
    sg.add(tz_, nt, true, false, &tz);
    sg.add((const float *)out_, nt, false, true, &out);
    Layout L;
    sg.plan(L);
    const size_t off_part = (n_split > 1) ? L.add(sizeof(double) * (size_t)n_split * nt) : 0;
    void *base = nullptr;
    HALMA_TRY(workspace(L.total, &base, st));
    HALMA_TRY(sg.bind_and_upload(base, st));
    if (ns == 0) {
        HALMA_CUDA(cudaMemsetAsync(out, 0, sizeof(float) * nt, st));
    } else {
        double *partial = n_split > 1 ? at<double>(base, off_part) : nullptr;
        HALMA_TRY(launch_fast<T>(m, x, y, z, ns, tx, ty, tz, nt, (float)eps2, n_split, split_len, mask, self_offset,
                                 out, partial, st));
        if (n_split > 1)
            HALMA_LAUNCH(reduce_partials_kernel, grid_for(nt, 256, 4096), 256, 0, st, partial, n_split, nt, out);
    }
    return sg.download(st);
}

// ---------------------------------------------------------------------------------------
// Targets that are the first nt sources (self-potential of a set, plus other sources): the
// pairs inside the set go through the symmetric block kernel of the unbinding, each pair
// evaluated once for both particles; the remaining sources through the tile kernel.
constexpr int64_t kSymMinTargets = 8192;

__global__ void pack_sources_kernel(int64_t n, const float *__restrict__ m, const float *__restrict__ x,
                                    const float *__restrict__ y, const float *__restrict__ z, float4 *__restrict__ pk) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        pk[i] = make_float4(x[i], y[i], z[i], m[i]);
}

// phi_i = the set's slices in block order + the other sources (float32 or per-slice FP64
// partials) + the self term m_i eps^-1 when the self pair is counted (mask NONE); FP64 sum, which bounds it (232 us of
// the 160,000-cell gas halo's forward, with one load in flight or eight).
__global__ void sym_finish_kernel(int64_t nt, int nblk, int64_t npad, const float2 *__restrict__ part,
                                  const float *__restrict__ tail, const double *__restrict__ tail_part, int n_tail,
                                  const float *__restrict__ m, double self_scale, float *__restrict__ out) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nt; i += (int64_t)gridDim.x * blockDim.x) {
        double acc = 0.0;
#pragma unroll 8
        for (int b = 0; b < nblk; ++b) {
            const float2 v = part[(int64_t)b * npad + i];
            acc += (double)v.x + (double)v.y;
        }
        if (tail) acc += (double)tail[i];
        for (int s = 0; s < n_tail; ++s) acc += tail_part[(int64_t)s * nt + i];
        acc += self_scale * (double)m[i];
        out[i] = (float)acc;
    }
}

static int potential_sym_api(int64_t ns, const float *m, const float *x, const float *y, const float *z, int64_t nt,
                             double eps2, int mask, float *out, cudaStream_t st) {
    constexpr int T = 4;
    const int nblk = sym_block_count((int)nt);
    const int64_t npad = (nt + 31) / 32 * 32;
    const int64_t nrest = ns - nt;
    int n_split = 1;
    int64_t split_len = nrest;
    if (nrest > 0) choose_split(nrest, nt, T, &n_split, &split_len);
    Layout L;
    const size_t o_pk = L.add(sizeof(float4) * npad), o_part = L.add(sizeof(float2) * (size_t)nblk * npad);
    const size_t o_desc = L.add(512);
    const size_t o_tail = L.add(sizeof(float) * (nrest > 0 && n_split == 1 ? nt : 1));
    const size_t o_tp = L.add(sizeof(double) * (nrest > 0 && n_split > 1 ? (size_t)n_split * nt : 1));
    void *base = nullptr;
    HALMA_TRY(workspace(L.total, &base, st, 9));
    float4 *pk = at<float4>(base, o_pk);
    float2 *part = at<float2>(base, o_part);
    const int g = std::min(device_sm_count() * 8, grid_for(nt, 256));
    HALMA_LAUNCH(pack_sources_kernel, g, 256, 0, st, nt, m, x, y, z, pk);
    HALMA_TRY(sym_self_potential_device(pk, (int)nt, (float)eps2, part, at<void>(base, o_desc), st));
    float *tail = nullptr;
    double *tail_part = nullptr;
    if (nrest > 0) {
        if (n_split > 1) tail_part = at<double>(base, o_tp);
        else tail = at<float>(base, o_tail);
        HALMA_TRY(launch_fast<T>(m + nt, x + nt, y + nt, z + nt, nrest, x, y, z, nt, (float)eps2, n_split, split_len,
                                 HALMA_MASK_NONE, 0, tail, tail_part, st));
    }
    const double self_scale = (mask == HALMA_MASK_NONE && eps2 > 0.0) ? 1.0 / sqrt(eps2) : 0.0;
    HALMA_LAUNCH(sym_finish_kernel, g, 256, 0, st, nt, nblk, npad, part, tail, tail_part, tail_part ? n_split : 0, m,
                 self_scale, out);
    return HALMA_OK;
}

}  // namespace halma

using namespace halma;

extern "C" int halma_bf_potential_f32(int64_t ntotal, const float *total_mass, const float *total_x,
                                      const float *total_y, const float *total_z, int64_t ntest,
                                      const float *test_x, const float *test_y, const float *test_z,
                                      float *binding_energy, int32_t mode, double eps2,
                                      halma_stream_t stream) {
    if (ntotal < 0 || ntest < 0) return fail(HALMA_ERR_INVALID, "negative size (ntotal=%lld ntest=%lld)", (long long)ntotal, (long long)ntest);
    if (ntest == 0) return HALMA_OK;
    if (!binding_energy || !test_x || !test_y || !test_z) return fail(HALMA_ERR_INVALID, "null target/output pointer");
    if (ntotal > 0 && (!total_mass || !total_x || !total_y || !total_z)) return fail(HALMA_ERR_INVALID, "null source pointer");
    if (mode != HALMA_POT_REFERENCE && mode != HALMA_POT_FAST) return fail(HALMA_ERR_INVALID, "unknown mode %d", mode);
    if (!(eps2 >= 0.0) || !isfinite(eps2)) return fail(HALMA_ERR_INVALID, "eps2 must be finite and >= 0");
    if (mode == HALMA_POT_REFERENCE && eps2 != 0.0) return fail(HALMA_ERR_INVALID, "reference mode has no softening (eps2 must be 0)");
    std::lock_guard<std::mutex> guard(api_mutex());
    cudaStream_t st = (cudaStream_t)stream;
    if (mode == HALMA_POT_FAST)
        return potential_fast_api(ntotal, total_mass, total_x, total_y, total_z, ntest, test_x, test_y, test_z, eps2,
                                  HALMA_MASK_COORD, 0, binding_energy, st);
    Stager sg;
    const float *m = nullptr, *x = nullptr, *y = nullptr, *z = nullptr, *tx = nullptr, *ty = nullptr, *tz = nullptr;
    float *out = nullptr;
    sg.add(total_mass, ntotal, true, false, &m);
    sg.add(total_x, ntotal, true, false, &x);
    sg.add(total_y, ntotal, true, false, &y);
    sg.add(total_z, ntotal, true, false, &z);
    sg.add(test_x, ntest, true, false, &tx);
    sg.add(test_y, ntest, true, false, &ty);
    sg.add(test_z, ntest, true, false, &tz);
    sg.add((const float *)binding_energy, ntest, false, true, &out);
    // narrow blocks while three of them an SM hold all targets: 2,000 x 20,000 takes 75 us so and 115 us
    // in wide ones, 4,500 x 20,000 128 and 115 us
    const bool narrow = ntest <= (int64_t)8 * 3 * device_sm_count();
    Layout L;
    sg.plan(L);
    const size_t o_src = L.add(sizeof(Src4) * (size_t)(narrow ? ref_quads_of<8>(ntotal) : ref_quads_of<32>(ntotal)));
    const size_t o_flags = L.add(sizeof(int));
    void *base = nullptr;
    HALMA_TRY(workspace(L.total, &base, st));
    HALMA_TRY(sg.bind_and_upload(base, st));
    if (ntotal == 0) {
        HALMA_CUDA(cudaMemsetAsync(out, 0, sizeof(float) * ntest, st));
    } else if (ntotal <= (ntest < kRefManyTargets ? kRefDirect : kRefDirectMany)) {
        HALMA_LAUNCH(ref_direct_kernel, grid_for(ntest, 256), 256, 0, st, m, x, y, z, ntotal, tx, ty, tz, ntest,
                     (const int *)nullptr, 1, out);
    } else {
        Src4 *src = at<Src4>(base, o_src);
        int *flags = at<int>(base, o_flags);
        HALMA_TRY(narrow ? launch_reference<8>(m, x, y, z, ntotal, tx, ty, tz, ntest, src, flags, out, st)
                         : launch_reference<32>(m, x, y, z, ntotal, tx, ty, tz, ntest, src, flags, out, st));
    }
    return sg.download(st);
}

extern "C" int halma_potential_f32(int64_t ns, const float *m, const float *sx, const float *sy, const float *sz,
                                   int64_t nt, const float *tx, const float *ty, const float *tz, double eps2,
                                   int32_t mask, int64_t self_offset, float *phi, halma_stream_t stream) {
    if (ns < 0 || nt < 0) return fail(HALMA_ERR_INVALID, "negative size");
    if (nt == 0) return HALMA_OK;
    if (!phi || !tx || !ty || !tz) return fail(HALMA_ERR_INVALID, "null target/output pointer");
    if (ns > 0 && (!m || !sx || !sy || !sz)) return fail(HALMA_ERR_INVALID, "null source pointer");
    if (mask < HALMA_MASK_COORD || mask > HALMA_MASK_NONE) return fail(HALMA_ERR_INVALID, "unknown mask %d", mask);
    if (!(eps2 >= 0.0) || !isfinite(eps2)) return fail(HALMA_ERR_INVALID, "eps2 must be finite and >= 0");
    std::lock_guard<std::mutex> guard(api_mutex());
    // targets that are the first sources (device arrays): the set's pairs once for both
    // particles; eps2 > 0 with mask NONE (the self pair is then a finite term), or mask SELF
    // skipping exactly the self pair
    const bool self_set = tx == sx && ty == sy && tz == sz && nt >= kSymMinTargets && nt <= ns &&
                          nt <= 65535ll * 1024 && ((mask == HALMA_MASK_NONE && eps2 > 0.0) ||
                                                   (mask == HALMA_MASK_SELF && self_offset == 0));
    if (self_set && is_device_pointer(m) && is_device_pointer(sx) && is_device_pointer(sy) && is_device_pointer(sz) &&
        is_device_pointer(phi))
        return potential_sym_api(ns, m, sx, sy, sz, nt, eps2, mask, phi, (cudaStream_t)stream);
    return potential_fast_api(ns, m, sx, sy, sz, nt, tx, ty, tz, eps2, mask, self_offset, phi, (cudaStream_t)stream);
}

extern "C" int halma_potential_f64(int64_t ns, const double *mm, const double *sx_, const double *sy_,
                                   const double *sz_, int64_t nt, const double *tx_, const double *ty_,
                                   const double *tz_, double eps2, int32_t mask, int64_t self_offset,
                                   double *phi, halma_stream_t stream) {
    if (ns < 0 || nt < 0) return fail(HALMA_ERR_INVALID, "negative size");
    if (nt == 0) return HALMA_OK;
    if (!phi || !tx_ || !ty_ || !tz_) return fail(HALMA_ERR_INVALID, "null target/output pointer");
    if (ns > 0 && (!mm || !sx_ || !sy_ || !sz_)) return fail(HALMA_ERR_INVALID, "null source pointer");
    if (mask < HALMA_MASK_COORD || mask > HALMA_MASK_NONE) return fail(HALMA_ERR_INVALID, "unknown mask %d", mask);
    if (!(eps2 >= 0.0) || !isfinite(eps2)) return fail(HALMA_ERR_INVALID, "eps2 must be finite and >= 0");
    std::lock_guard<std::mutex> guard(api_mutex());
    cudaStream_t st = (cudaStream_t)stream;
    Stager sg;
    const double *m = nullptr, *sx = nullptr, *sy = nullptr, *sz = nullptr, *tx = nullptr, *ty = nullptr, *tz = nullptr;
    double *out = nullptr;
    sg.add(mm, ns, true, false, &m);
    sg.add(sx_, ns, true, false, &sx);
    sg.add(sy_, ns, true, false, &sy);
    sg.add(sz_, ns, true, false, &sz);
    sg.add(tx_, nt, true, false, &tx);
    sg.add(ty_, nt, true, false, &ty);
    sg.add(tz_, nt, true, false, &tz);
    sg.add((const double *)phi, nt, false, true, &out);
    Layout L;
    sg.plan(L);
    void *base = nullptr;
    HALMA_TRY(workspace(L.total, &base, st));
    HALMA_TRY(sg.bind_and_upload(base, st));
    HALMA_LAUNCH(potential_f64_kernel, grid_for(nt, 256), 256, 0, st, m, sx, sy, sz, ns, tx, ty, tz, nt,
                 eps2, (int)mask, self_offset, out);
    return sg.download(st);
}

// ---------------------------------------------------------------------------------------
// Allocation-free variant of the fast (compensated FP32) potential.
//
// Some callers cannot let a library allocate device memory.  Simulation codes that embed the
// halo finder (an AMR code calling it between time steps, say) usually reserve almost all of
// the GPU's memory up front for their own pool and hand out pieces themselves, so a
// cudaMalloc from the library either fails or breaks the host's accounting; and a cudaFree
// synchronises the whole device, which stalls every other stream of a caller that keeps
// several streams busy.  This entry point serves such callers: it takes device arrays only
// and keeps its scratch -- the per-slice partial sums of the source-split kernel -- in the
// fixed array below instead of the library's cached workspace.  It calls no cudaMalloc,
// cudaFree or allocating library routine.
//
// Limit: the scratch holds kNoAllocScratchDoubles = 2,097,152 partial sums (16 MiB).  The call
// splits the sources exactly as halma_bf_potential_f32 does in HALMA_POT_FAST mode and runs
// the same kernels, so the two return identical values; when that split needs more than
// 2,097,152 partial sums (source slices x targets) the call is rejected with
// HALMA_ERR_CAPACITY.
//
// Every GPU that loads this library holds the 16 MiB array until the process exits.  All calls with 4,096 sources or more
// share it (the slices of fewer are added up inside a block) and it keeps the previous call's contents; each partial sum a call reads is written
// by the same call first, so nothing needs clearing.  Calls that overlap on the GPU (two
// streams, or two host threads without ordering) race on the array and give wrong results.
// The first call on each device looks up the array's device address (cudaGetSymbolAddress with
// that device current); make that first call before any stream capture begins.
constexpr int64_t kNoAllocScratchDoubles = kMaxPartials;   // what the finer slices of any call take
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocScratchDoubles];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
double *g_noalloc_ptr[kMaxDevices] = {};

// Memory the current device's kernels can use in place: device memory of this device, or
// managed memory.  Another GPU's device memory is refused rather than read over the peer link.
bool is_local_device_pointer(const void *p) {
    if (!p) return false;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (a.type == cudaMemoryTypeManaged) return true;
    return a.type == cudaMemoryTypeDevice && a.device == current_device();
}

// Device address of g_noalloc_scratch on the current device (looked up once per device).
int noalloc_scratch(double **out) {
    const int dev = current_device();
    if (dev < 0 || dev >= kMaxDevices) return fail(HALMA_ERR_CAPACITY, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> g(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        HALMA_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
        g_noalloc_ptr[dev] = static_cast<double *>(p);
    }
    *out = g_noalloc_ptr[dev];
    return HALMA_OK;
}
}  // namespace

extern "C" int halma_bf_potential_f32_noalloc(int64_t ntotal, const float *total_mass, const float *total_x,
                                              const float *total_y, const float *total_z, int64_t ntest,
                                              const float *test_x, const float *test_y, const float *test_z,
                                              float *binding_energy, double eps2, halma_stream_t stream) {
    if (ntotal < 0 || ntest < 0) return fail(HALMA_ERR_INVALID, "negative size");
    if (ntest == 0) return HALMA_OK;
    if (!binding_energy || !test_x || !test_y || !test_z) return fail(HALMA_ERR_INVALID, "null target/output pointer");
    if (ntotal > 0 && (!total_mass || !total_x || !total_y || !total_z)) return fail(HALMA_ERR_INVALID, "null source pointer");
    if (!(eps2 >= 0.0) || !isfinite(eps2)) return fail(HALMA_ERR_INVALID, "eps2 must be finite and >= 0");
    const void *arrays[8] = {test_x, test_y, test_z, binding_energy, total_mass, total_x, total_y, total_z};
    for (int k = 0; k < (ntotal > 0 ? 8 : 4); ++k)
        if (!is_local_device_pointer(arrays[k]))
            return fail(HALMA_ERR_INVALID,
                        "the allocation-free entry point takes arrays in the current device's memory only");
    cudaStream_t st = (cudaStream_t)stream;
    if (ntotal == 0) {
        HALMA_CUDA(cudaMemsetAsync(binding_energy, 0, sizeof(float) * ntest, st));
        return HALMA_OK;
    }
    constexpr int T = 4;
    int n_split = 1;
    int64_t split_len = ntotal;
    choose_split(ntotal, ntest, T, &n_split, &split_len);
    if (n_split > 1 && ntotal < 2 * kCoarseSlice) {   // few enough slices for a block, with nothing that calls share
        const unsigned blocks = (unsigned)((ntest + 31) / 32);
        if ((float)eps2 >= 0x1p-126f)
            HALMA_LAUNCH(bf_potential_block_kernel<true>, blocks, 256, 0, st, total_mass, total_x, total_y, total_z, ntotal,
                         test_x, test_y, test_z, ntest, (float)eps2, n_split, split_len, binding_energy);
        else
            HALMA_LAUNCH(bf_potential_block_kernel<false>, blocks, 256, 0, st, total_mass, total_x, total_y, total_z, ntotal,
                         test_x, test_y, test_z, ntest, (float)eps2, n_split, split_len, binding_energy);
        return HALMA_OK;
    }
    if (n_split > 1 && (int64_t)n_split * ntest > kNoAllocScratchDoubles)
        return fail(HALMA_ERR_CAPACITY,
                    "this call needs %lld partial sums (%d source slices x %lld targets); the allocation-free "
                    "scratch holds %lld — use halma_bf_potential_f32",
                    (long long)n_split * ntest, n_split, (long long)ntest, (long long)kNoAllocScratchDoubles);
    double *scratch = nullptr;
    HALMA_TRY(noalloc_scratch(&scratch));
    double *partial = n_split > 1 ? scratch : nullptr;
    HALMA_TRY(launch_fast<T>(total_mass, total_x, total_y, total_z, ntotal, test_x, test_y, test_z, ntest,
                             (float)eps2, n_split, split_len, HALMA_MASK_COORD, 0, binding_energy, partial, st));
    if (n_split > 1)
        HALMA_LAUNCH(reduce_partials_kernel, grid_for(ntest, 256, 4096), 256, 0, st, partial, n_split, ntest,
                     binding_energy);
    return HALMA_OK;
}
