// Batched iterative unbinding of thousands of haloes, and the plain FP64 per-halo path.
//
// The single pass is pyHALMA's escape cut (python_scripts/halo_properties.py:282-361):
//     E_i = 1/2 |v_i - v_bulk|^2 - G * factor_v^2 * phi_i,   bound iff E_i <= 0
// repeated until a pass removes nothing.  Before the first pass:
//   reduce  - per halo, FP64 mass, centre of mass and bulk velocity;
//   pack    - members re-centred on their halo's centre, float4 (x, y, z, m), padded to a
//             multiple of 32 with zero-mass far points (halo-contiguous slots).
// Haloes of up to kSmallMax members run all their passes in one block each (ub_small_kernel).  Every pass over the
// other active haloes is four kernels, the first of these lists being written beside the last kernel of the pass before:
//   items   - the implicit work list: per halo, (target tile of 32*T) x (source slice) items,
//             biggest haloes first, and the energy segments of the pass;
//   pairs   - persistent kernel: warps take items from an atomic counter, stream the slice's
//             sources through a per-warp shared-memory chunk, two sources per f32x2
//             instruction, 32-term FP32 partials folded into a TwoSum-compensated
//             accumulator; the self pair is skipped by slot index;
//   energy / finalize / compact - energy and sign test, the next pass's FP64 mass, centre and bulk
//             velocity, survivors compacted into the other packed buffer; a halo whose pass
//             removed nothing becomes inactive and costs nothing later.
// Passes are launched as they are or as captured graphs (see kPassChunk).
#include <math.h>
#include <string.h>

#include <algorithm>
#include <numeric>
#include <vector>

#include "common.cuh"
#include "pair_math.cuh"
#include "sort.cuh"
#include "unbind.cuh"

namespace halma {

namespace {

constexpr int kUbWarps = 8;
constexpr float kFar = 3.0e30f;

struct HaloState {   // per halo, FP64 unless stated
    double M, cx, cy, cz, vx, vy, vz, ekin, epot;
    // FP32 path: sums of m x and m v over the bound set, kept up to date by subtracting each
    // pass's removed particles; the bulk velocity at packing (packed velocities are relative
    // to it) and the current bulk velocity relative to it in FP32
    double sx, sy, sz, px, py, pz, v0x, v0y, v0z;
    float wx, wy, wz;
    int nb, active, iter, removed, nrem;   // nrem: removed by the last pass (next pass's sources)
    int nprev;                             // slots the last pass examined (nb before its cut)
};

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Block-wide FP64 sums of NV values written to out[0..NV) (fixed association: warp tree,
// then the warps in order).
template <int NV>
__device__ __forceinline__ void block_sum_store(const double (&v)[NV], double (*sh)[32], double *out) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        double s = warp_sum(v[q]);
        if (lane == 0) sh[q][w] = s;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            double s = lane < nw ? sh[q][lane] : 0.0;
            s = warp_sum(s);
            if (lane == 0) out[q] = s;
        }
    }
}

__global__ void ub_init_kernel(int64_t n, unsigned char *bound, int nh, HaloState *hs) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        bound[i] = 1;
    for (int64_t h = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; h < nh; h += (int64_t)gridDim.x * blockDim.x) {
        HaloState s{};
        s.active = 1;
        hs[h] = s;
    }
}

// Member chunks: every halo's CSR range is cut into chunks of kSeg members, chunk c covering
// members off[h] + (c - cstart[h]) * kSeg onward of halo h = chunk_h[c] (laid out on the host),
// so a large halo is spread over many blocks.
constexpr int kSeg = 1024;
constexpr int kSegThreads = 256;
constexpr int kSegPer = kSeg / kSegThreads;
constexpr int kRedSums = 8;   // M, Mx, My, Mz, Mvx, Mvy, Mvz, count

// Per member chunk of an active halo (or of every halo with force): FP64 sums over its bound
// members.  FP64 is slow on this GPU, so the block's partials are combined by a few threads
// in shared memory rather than by warp trees (fixed association: per thread in member order,
// then per value four runs of 64 threads, then the four runs in order).  PART selects the
// sums written: 0 all, 1 mass, mass-weighted positions and count (the velocities are not
// read), 2 the mass-weighted velocities; each sum is formed the same way in every mode, so
// modes 1 then 2 write exactly what mode 0 writes.
__host__ __device__ constexpr bool red_wants(int part, int k) { return part == 0 || (part == 1 ? (k < 4 || k == 7) : (k >= 4 && k < 7)); }

template <int PART>
__global__ void __launch_bounds__(kSegThreads) ub_reduce_seg_kernel(
    const int64_t *__restrict__ off, const int *__restrict__ cstart, const int *__restrict__ chunk_h,
    const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ z,
    const double *__restrict__ vx, const double *__restrict__ vy, const double *__restrict__ vz,
    const double *__restrict__ m, const unsigned char *__restrict__ bound, const HaloState *__restrict__ hs,
    int force, double *__restrict__ part) {
    const int c = blockIdx.x;
    const int h = chunk_h[c];
    if (!force && !hs[h].active) return;
    __shared__ double sh[kRedSums - 1][kSegThreads];
    __shared__ double q4[kRedSums - 1][4];
    const int64_t b = off[h] + (int64_t)(c - cstart[h]) * kSeg;
    const int64_t e = min(off[h + 1], b + kSeg);
    double v[kRedSums - 1] = {0, 0, 0, 0, 0, 0, 0};
    int count = 0;
    // all loads of the thread's members are issued before any is used; members outside the
    // chunk read member b and are skipped
    bool use[kSegPer];
    double f[kSegPer][7];
#pragma unroll
    for (int j = 0; j < kSegPer; ++j) {
        const int64_t i = b + j * kSegThreads + threadIdx.x;
        const bool in = i < e;
        const int64_t s = in ? i : b;
        use[j] = in && bound[s];
        f[j][0] = m[s];
        f[j][1] = red_wants(PART, 1) ? x[s] : 0.0;
        f[j][2] = red_wants(PART, 2) ? y[s] : 0.0;
        f[j][3] = red_wants(PART, 3) ? z[s] : 0.0;
        f[j][4] = red_wants(PART, 4) ? vx[s] : 0.0;
        f[j][5] = red_wants(PART, 5) ? vy[s] : 0.0;
        f[j][6] = red_wants(PART, 6) ? vz[s] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < kSegPer; ++j) {
        if (!use[j]) continue;
        const double mi = f[j][0];
        v[0] += mi;
#pragma unroll
        for (int k = 1; k < 7; ++k)
            if (red_wants(PART, k)) v[k] += mi * f[j][k];
        ++count;
    }
#pragma unroll
    for (int k = 0; k < kRedSums - 1; ++k) sh[k][threadIdx.x] = v[k];
    __shared__ int wcount[kSegThreads / 32];
    int wc = count;
    for (int o = 16; o > 0; o >>= 1) wc += __shfl_down_sync(0xffffffffu, wc, o);
    if ((threadIdx.x & 31) == 0) wcount[threadIdx.x >> 5] = wc;
    __syncthreads();
    if (threadIdx.x < 4 * (kRedSums - 1)) {
        const int k = threadIdx.x % (kRedSums - 1), run = threadIdx.x / (kRedSums - 1);
        double t = 0.0;
        for (int u = run * (kSegThreads / 4); u < (run + 1) * (kSegThreads / 4); ++u) t += sh[k][u];
        q4[k][run] = t;
    }
    __syncthreads();
    if (threadIdx.x < kRedSums - 1) {
        const int k = threadIdx.x;
        if (red_wants(PART, k)) part[(int64_t)c * kRedSums + k] = ((q4[k][0] + q4[k][1]) + q4[k][2]) + q4[k][3];
    } else if (threadIdx.x == kRedSums - 1 && red_wants(PART, 7)) {
        int tot = 0;
        for (int w = 0; w < kSegThreads / 32; ++w) tot += wcount[w];
        part[(int64_t)c * kRedSums + kRedSums - 1] = (double)tot;
    }
}

// One warp per ordered halo: chunk sums added in a fixed order (lane-strided, then the warp tree);
// sets the bound mass, centre of mass, bulk velocity and bound count.
__global__ void ub_reduce_fin_kernel(int nh, const int *__restrict__ order, const int *__restrict__ cstart,
                                     const double *__restrict__ part, int force, HaloState *hs) {
    const int q = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (q >= nh) return;
    const int h = order[q];
    if (!force && !hs[h].active) return;
    double v[kRedSums] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int c = cstart[h] + lane; c < cstart[h + 1]; c += 32)
#pragma unroll
        for (int k = 0; k < kRedSums; ++k) v[k] += part[(int64_t)c * kRedSums + k];
#pragma unroll
    for (int k = 0; k < kRedSums; ++k) v[k] = warp_sum(v[k]);
    if (lane == 0) {
        HaloState &s = hs[h];
        const double M = v[0];
        s.M = M;
        s.nb = (int)v[7];
        s.sx = v[1]; s.sy = v[2]; s.sz = v[3];
        s.px = v[4]; s.py = v[5]; s.pz = v[6];
        if (M > 0) {
            s.cx = v[1] / M; s.cy = v[2] / M; s.cz = v[3] / M;
            s.vx = v[4] / M; s.vy = v[5] / M; s.vz = v[6] / M;
        } else {
            s.cx = s.cy = s.cz = s.vx = s.vy = s.vz = 0.0;
        }
        if (!force) {   // before the first pass: the reference velocity of the packed velocities
            s.v0x = s.vx; s.v0y = s.vy; s.v0z = s.vz;
            s.wx = s.wy = s.wz = 0.f;
        }
    }
}

// First packing, per member chunk: every member is bound before the first pass, so member
// i of halo h goes to slot i - off[h] of the halo's padded range, re-centred on the halo's
// centre of mass; the chunk holding the halo's end also writes the padding (zero-mass far
// points up to the next multiple of 32).  pk == nullptr writes the velocities alone, pv ==
// nullptr the positions and indices alone.
template <class V>
__global__ void __launch_bounds__(kSegThreads) ub_pack_kernel(
    const int64_t *__restrict__ off, const int64_t *__restrict__ poff, const int *__restrict__ cstart,
    const int *__restrict__ chunk_h, const double *__restrict__ x, const double *__restrict__ y,
    const double *__restrict__ z, const double *__restrict__ m, const double *__restrict__ vx,
    const double *__restrict__ vy, const double *__restrict__ vz, const HaloState *__restrict__ hs,
    V *__restrict__ pk, float4 *__restrict__ pv, int *__restrict__ pidx) {
    const int c = blockIdx.x;
    const int h = chunk_h[c];
    const double cx = hs[h].cx, cy = hs[h].cy, cz = hs[h].cz;
    const double v0x = hs[h].v0x, v0y = hs[h].v0y, v0z = hs[h].v0z;
    const int64_t hb = off[h], he = off[h + 1], pb = poff[h];
    const int64_t b = hb + (int64_t)(c - cstart[h]) * kSeg;
    const int64_t e = min(he, b + kSeg);
    for (int64_t i = b + threadIdx.x; i < e; i += kSegThreads) {
        if (pk) {
            V r;
            r.x = x[i] - cx; r.y = y[i] - cy; r.z = z[i] - cz; r.w = m[i];
            pk[pb + (i - hb)] = r;
            pidx[pb + (i - hb)] = (int)i;
        }
        // FP32 path: velocity relative to the bulk velocity at packing, and the mass
        if (pv) pv[pb + (i - hb)] = make_float4((float)(vx[i] - v0x), (float)(vy[i] - v0y), (float)(vz[i] - v0z),
                                                 (float)m[i]);
    }
    if (e == he) {
        const int64_t nb = he - hb, npad = (nb + 31) & ~31ll;
        for (int64_t r = nb + threadIdx.x; r < npad; r += kSegThreads) {
            if (pk) {
                V f;
                f.x = f.y = f.z = kFar; f.w = 0;
                pk[pb + r] = f;
                pidx[pb + r] = -1;
            }
            if (pv) pv[pb + r] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
}

// Work list for the pair kernel: haloes in decreasing initial size, tiles of 32*T targets.
// Also records the pass's pair count (sum of nb^2 over active haloes) in pairs_out.
__device__ __forceinline__ int tile_t_for(const TileTable &tab, int nb) {
    for (int c = 0; c < tab.n; ++c)
        if (nb <= tab.upper[c]) return tab.t[c];
    return 4;
}

// The work list is implicit: ordered halo q owns items istart[q] .. istart[q+1]-1, described
// by idesc[q] = (halo, T, slices, unused); item i of that halo is (tile i / slices,
// slice i % slices).  Only nh+1 prefix counts are written per pass.
// The same pass also lays out the energy segments: active ordered halo q owns segments
// sstart[q] .. sstart[q+1]-1 of kSeg slots each; sown[seg] names the segment's ordered halo.

__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

// Full passes over a halo of more than kSymBlock bound particles use the symmetric block
// kernel instead: blocks of kSymBlock slots, one item per block pair (tb <= sb), B(B+1)/2
// items for B blocks, listed from ystart[q]; the partial sums are then kept per block
// (B slices of kSymBlock).  idesc[q].w is the number of partial slices the energy kernel adds.
constexpr int kSymWarps = 4, kSymT = 8;
constexpr int kSymBlock = kSymWarps * 32 * kSymT;   // 1024 slots

// The pass's work list over the haloes in size order (q):
//   count - per halo q: its halo h, tile shape, source slices, and three counts: warp items
//           (tiles x slices), energy segments, symmetric block-pair items (0 unless active);
//   scan  - exclusive prefix sums of the three counts;
//   fill  - the prefix sums become istart / sstart / ystart, every segment records its owner
//           (sown), and the totals go to cnt[] (warp items, energy segments, block-pair items,
//           their counters reset) and to the last entries of the start arrays.
// With pairs_out (profiling), the pass's pair terms (nb x sources, all haloes) and those of the
// haloes on the symmetric block kernel are summed into pairs_out[0..1] (zeroed beforehand).
// For up to kItemsBlock haloes one block does all three (items_block), for the next pass beside the last one's
// compaction.  As a count, a scan and a fill, four launches with nothing beside them, it took 8.7 us of every pass.
// A block takes 6.9 us for 260 haloes and 32 for 2,000, most of it hidden: haloes of 1,100 to 1,500 members, all
// passes, 260 of them 977 -> 871 us, 1,000 1,974 -> 1,808, 2,000 3,012 -> 2,966.  More haloes take the three steps,
// spread over the GPU.
constexpr int kItemsBlock = 2048;

struct WorkList {
    int4 *idesc;
    int *istart, *ystart, *sstart, *sown, *cnt;
};

struct ItemRule {
    TileTable tab;
    int slice_len, inc, sym_ok;
};

// Counts of halo h (x warp items, y energy segments, z block pairs), its description and its pair terms.
__device__ __forceinline__ int3 halo_items(const HaloState &s, int h, const ItemRule &rule, int4 &desc,
                                           unsigned long long &pairs, unsigned long long &spairs) {
    int n = 0, T = 4, nsl = 1, nseg = 0, ny = 0, nsl_e = 0;
    if (s.active) {
        const int nb = s.nb;
        const int ns = rule.inc ? s.nrem : nb;   // sources: removed particles or the halo itself
        T = tile_t_for(rule.tab, nb);
        nsl = (int)(((int64_t)ns + rule.slice_len - 1) / rule.slice_len);
        if (!rule.inc && rule.sym_ok && nb > kSymBlock && nb <= 65535 * kSymBlock) {
            const int B = (nb + kSymBlock - 1) / kSymBlock;   // B <= 65535: B(B+1)/2 < 2^31
            ny = (int)((int64_t)B * (B + 1) / 2);
            nsl_e = B;
            spairs = (unsigned long long)nb * (unsigned long long)nb;
        } else {
            n = ns > 0 ? ((nb + 32 * T - 1) / (32 * T)) * nsl : 0;
            nsl_e = nsl;
        }
        nseg = max(1, (nb + kSeg - 1) / kSeg);
        pairs = (unsigned long long)nb * (unsigned long long)ns;
    }
    desc = make_int4(h, T, max(nsl, 1), nsl_e);
    return make_int3(n, nseg, ny);
}

__device__ __forceinline__ void add_pairs(unsigned long long *pairs_out, unsigned long long pairs,
                                          unsigned long long spairs, int lane) {
    if (!pairs_out) return;
    for (int o = 16; o > 0; o >>= 1) {
        pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
        spairs += __shfl_xor_sync(0xffffffffu, spairs, o);
    }
    if (lane == 0 && (pairs | spairs)) {   // one atomic per warp
        atomicAdd(pairs_out, pairs);
        atomicAdd(pairs_out + 1, spairs);
    }
}

__device__ __forceinline__ void items_total(const WorkList &wl, int nh, int3 t) {
    wl.istart[nh] = t.x;
    wl.sstart[nh] = t.y;
    wl.ystart[nh] = t.z;
    wl.cnt[0] = t.x;   // warp items
    wl.cnt[1] = 0;     // their counter
    wl.cnt[2] = t.y;   // energy segments
    wl.cnt[3] = t.z;   // symmetric block items
    wl.cnt[4] = 0;     // their counter
}

// The whole list by one block of kSegThreads threads.
__device__ __forceinline__ void items_block(int nh, const int *__restrict__ order, const HaloState *hs,
                                            const ItemRule &rule, const WorkList &wl, unsigned long long *pairs_out) {
    constexpr int kWarps = kSegThreads / 32;
    __shared__ int3 tot[2][kWarps];   // of two rounds in turn: one barrier a round
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int3 run = make_int3(0, 0, 0);
    int par = 0;
    for (int q0 = 0; q0 < nh; q0 += kSegThreads, par ^= 1) {
        const int q = q0 + threadIdx.x;
        int3 c = make_int3(0, 0, 0);
        unsigned long long pairs = 0, spairs = 0;
        if (q < nh) {
            int4 desc;
            const int h = order[q];
            c = halo_items(hs[h], h, rule, desc, pairs, spairs);
            wl.idesc[q] = desc;
        }
        add_pairs(pairs_out, pairs, spairs, lane);
        const int3 i = make_int3(warp_incl_scan(c.x, lane), warp_incl_scan(c.y, lane), warp_incl_scan(c.z, lane));
        if (lane == 31) tot[par][w] = i;
        __syncthreads();
        int3 p = make_int3(run.x + i.x - c.x, run.y + i.y - c.y, run.z + i.z - c.z);
#pragma unroll
        for (int k = 0; k < kWarps; ++k) {
            const int3 t = tot[par][k];
            if (k < w) {
                p.x += t.x;
                p.y += t.y;
                p.z += t.z;
            }
            run.x += t.x;
            run.y += t.y;
            run.z += t.z;
        }
        if (q < nh) {
            wl.istart[q] = p.x;
            wl.sstart[q] = p.y;
            wl.ystart[q] = p.z;
        }
        // a halo's segments: a few by its thread, many by the warp
        const bool many = c.y > 4;
        if (!many)
            for (int sg = 0; sg < c.y; ++sg) wl.sown[p.y + sg] = q;
        for (unsigned todo = __ballot_sync(0xffffffffu, many); todo; todo &= todo - 1) {
            const int l = __ffs(todo) - 1;
            const int first = __shfl_sync(0xffffffffu, p.y, l), count = __shfl_sync(0xffffffffu, c.y, l);
            for (int sg = lane; sg < count; sg += 32) wl.sown[first + sg] = q0 + w * 32 + l;
        }
    }
    if (threadIdx.x == 0) items_total(wl, nh, run);
}

__global__ void __launch_bounds__(kSegThreads) ub_items_kernel(int nh, const int *__restrict__ order,
                                                               const HaloState *hs, ItemRule rule, WorkList wl,
                                                               unsigned long long *__restrict__ pairs_out) {
    items_block(nh, order, hs, rule, wl, pairs_out);
}

__global__ void __launch_bounds__(256) ub_items_count_kernel(int nh, const int *__restrict__ order,
                                                             const HaloState *hs, ItemRule rule,
                                                             int4 *__restrict__ counts, int4 *__restrict__ idesc,
                                                             unsigned long long *__restrict__ pairs_out) {
    for (int q0 = blockIdx.x * blockDim.x; q0 < nh; q0 += gridDim.x * blockDim.x) {
        const int q = q0 + threadIdx.x;
        unsigned long long pairs = 0, spairs = 0;
        if (q < nh) {
            int4 desc;
            const int h = order[q];
            const int3 c = halo_items(hs[h], h, rule, desc, pairs, spairs);
            counts[q] = make_int4(c.x, c.y, c.z, 0);
            idesc[q] = desc;
        }
        add_pairs(pairs_out, pairs, spairs, threadIdx.x & 31);
    }
}

__global__ void __launch_bounds__(256) ub_items_fill_kernel(int nh, const int4 *__restrict__ counts,
                                                            const int4 *__restrict__ pre, WorkList wl) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nh; q += gridDim.x * blockDim.x) {
        const int4 c = counts[q], p = pre[q];
        wl.istart[q] = p.x;
        wl.sstart[q] = p.y;
        wl.ystart[q] = p.z;
        for (int sg = 0; sg < c.y; ++sg) wl.sown[p.y + sg] = q;
        if (q == nh - 1) items_total(wl, nh, make_int3(p.x + c.x, p.y + c.y, p.z + c.z));
    }
}

// 32 sources of the staged chunk against T targets, two sources per f32x2 instruction.
// sa[kp] = {x_2kp, x_2kp+1, y_2kp, y_2kp+1}, sb[kp] = {z.., z.., m.., m..}.  Each target keeps
// an {even, odd} pair of partial sums.  SELF: target ts skips the source in its own lane slot.
template <int T, bool SELF>
__device__ __forceinline__ void chunk_pairs(const float4 *sa, const float4 *sb, const f2x (&tx)[T], const f2x (&ty)[T],
                                            const f2x (&tz)[T], f2x e2, f2x (&acc)[T], int ts, int lane) {
#pragma unroll 4
    for (int kp = 0; kp < 16; ++kp) {
        const float4 a = sa[kp], b = sb[kp];
        const f2x X = pack2(a.x, a.y), Y = pack2(a.z, a.w), Z = pack2(b.x, b.y), M = pack2(b.z, b.w);
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const f2x dx = sub2(X, tx[t]), dy = sub2(Y, ty[t]), dz = sub2(Z, tz[t]);
            f2x r2 = fma2(dz, dz, e2);
            r2 = fma2(dy, dy, r2);
            r2 = fma2(dx, dx, r2);
            float r0, r1;
            unpack2(r2, r0, r1);
            float i0 = rsqrt_ftz(r0), i1 = rsqrt_ftz(r1);
            if (SELF && t == ts && kp == (lane >> 1)) {
                if (lane & 1) i1 = 0.f;
                else i0 = 0.f;
            }
            acc[t] = fma2(M, pack2(i0, i1), acc[t]);
        }
    }
}

// One work item: 32*T target slots of one halo (tpk) against source chunks [c_begin, c_end)
// of spk.  self_ok: targets and sources are the same slots, so the self pair is skipped.
template <int T>
__device__ __forceinline__ void pair_item(const float4 *__restrict__ tpk, const float4 *__restrict__ pk, int64_t base,
                                          int nb, int tile, float eps2, int c_begin, int c_end, bool self_ok,
                                          float2 *__restrict__ out, float4 *buf, int lane) {
    {
        f2x tx[T], ty[T], tz[T];
        float sum[T], comp[T];
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int r = tile * 32 * T + t * 32 + lane;
            const float4 p = r < nb ? tpk[base + r] : make_float4(kFar, kFar, kFar, 0.f);
            tx[t] = pack2(p.x, p.x);
            ty[t] = pack2(p.y, p.y);
            tz[t] = pack2(p.z, p.z);
            sum[t] = 0.f;
            comp[t] = 0.f;
        }
        const f2x e2 = pack2(eps2, eps2);
        float *sa = reinterpret_cast<float *>(buf);        // 16 float4: x/y pairs
        float *sb = reinterpret_cast<float *>(buf + 16);   // 16 float4: z/m pairs
        const int kp = lane >> 1, hf = lane & 1;
        const int self0 = tile * T;   // chunk c holds the self slot of target t = c - self0
        float4 nxt = pk[base + (int64_t)c_begin * 32 + lane];
        for (int c = c_begin; c < c_end; ++c) {
            __syncwarp();
            sa[kp * 4 + hf] = nxt.x;
            sa[kp * 4 + 2 + hf] = nxt.y;
            sb[kp * 4 + hf] = nxt.z;
            sb[kp * 4 + 2 + hf] = nxt.w;
            __syncwarp();
            if (c + 1 < c_end) nxt = pk[base + (int64_t)(c + 1) * 32 + lane];
            f2x acc[T];
#pragma unroll
            for (int t = 0; t < T; ++t) acc[t] = pack2(0.f, 0.f);
            const int ts = c - self0;
            if (self_ok && ts >= 0 && ts < T)
                chunk_pairs<T, true>(buf, buf + 16, tx, ty, tz, e2, acc, ts, lane);
            else
                chunk_pairs<T, false>(buf, buf + 16, tx, ty, tz, e2, acc, ts, lane);
#pragma unroll
            for (int t = 0; t < T; ++t) {
                float a0, a1;
                unpack2(acc[t], a0, a1);
                two_sum_acc(sum[t], comp[t], a0 + a1);
            }
        }
#pragma unroll
        for (int t = 0; t < T; ++t) {
            const int r = tile * 32 * T + t * 32 + lane;
            if (r < nb) out[r] = df_from_acc(sum[t], comp[t]);
        }
    }
}

// Persistent all-pairs kernel over the work list (FP32 pair terms, compensated sums).  An
// item is (halo, target tile, tile shape T, source slice): 32*T targets against one slice of
// slice_chunks*32 source slots.  Each slice writes its own partial sums
// (part[qoff[h] + slice * npad_h + r]); the energy kernel adds the slices in order, so the
// result does not depend on which warp ran which item.  Full passes take the sources from the
// targets' own slots (self pair skipped); incremental passes (inc) take them from the slots of
// the particles removed by the previous pass (spk, hs.nrem of them), whose contribution the
// energy kernel then subtracts from the previous potential.
__global__ void __launch_bounds__(256) ub_pair_kernel(const float4 *__restrict__ pk, const float4 *__restrict__ spk,
                                                      int inc, const int64_t *__restrict__ poff,
                                                      const int64_t *__restrict__ qoff, const HaloState *__restrict__ hs,
                                                      int nh, const int *__restrict__ istart,
                                                      const int4 *__restrict__ idesc, const int *__restrict__ nitems_p,
                                                      int *counter, float eps2, int slice_chunks,
                                                      float2 *__restrict__ part) {
    __shared__ float4 buf[kUbWarps][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nitems = *nitems_p;
    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(counter, 1);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= nitems) break;
        // ordered halo owning the item: last q with istart[q] <= item
        int lo = 0, hi = nh - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (istart[mid] <= item) lo = mid;
            else hi = mid - 1;
        }
        const int4 d = idesc[lo];
        const int local = item - istart[lo];
        const int4 it = make_int4(d.x, local / d.z, d.y, local % d.z);
        const int h = it.x, tile = it.y, slice = it.w;
        const int64_t base = poff[h];
        const int64_t npad = poff[h + 1] - base;
        const int nb = hs[h].nb;
        const int ns = inc ? hs[h].nrem : nb;
        const float4 *src = inc ? spk : pk;
        const int c0 = slice * slice_chunks;
        const int c1 = min((ns + 31) >> 5, c0 + slice_chunks);
        float2 *out = part + qoff[h] + (int64_t)slice * npad;
        switch (it.z) {
            case 1: pair_item<1>(pk, src, base, nb, tile, eps2, c0, c1, !inc, out, buf[w], lane); break;
            case 2: pair_item<2>(pk, src, base, nb, tile, eps2, c0, c1, !inc, out, buf[w], lane); break;
            default: pair_item<4>(pk, src, base, nb, tile, eps2, c0, c1, !inc, out, buf[w], lane); break;
        }
    }
}

// Symmetric form of chunk_pairs: every pair term 1/r is used twice, m_source / r for the
// lane's targets (acc, as in chunk_pairs) and m_target / r for the chunk's sources.  The
// source side is summed over the lane's T targets, then over the warp (reduce-scatter), and
// the warp's 32 * T-target sums of the chunk's 32 sources go to sout[0..32).
template <int T>
__device__ __forceinline__ void chunk_pairs_sym(const float4 *sa, const float4 *sb, const f2x (&tx)[T],
                                                const f2x (&ty)[T], const f2x (&tz)[T], const f2x (&tm)[T], f2x e2,
                                                f2x (&acc)[T], float *sout, int lane) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        f2x sacc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) sacc[k] = pack2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float4 a = sa[half * 8 + k], b = sb[half * 8 + k];
            const f2x X = pack2(a.x, a.y), Y = pack2(a.z, a.w), Z = pack2(b.x, b.y), M = pack2(b.z, b.w);
#pragma unroll
            for (int t = 0; t < T; ++t) {
                const f2x dx = sub2(X, tx[t]), dy = sub2(Y, ty[t]), dz = sub2(Z, tz[t]);
                f2x r2 = fma2(dz, dz, e2);
                r2 = fma2(dy, dy, r2);
                r2 = fma2(dx, dx, r2);
                float r0, r1;
                unpack2(r2, r0, r1);
                const f2x ri = pack2(rsqrt_ftz(r0), rsqrt_ftz(r1));
                acc[t] = fma2(M, ri, acc[t]);
                sacc[k] = fma2(tm[t], ri, sacc[k]);
            }
        }
        float v[16];
#pragma unroll
        for (int k = 0; k < 8; ++k) unpack2(sacc[k], v[2 * k], v[2 * k + 1]);
        const float s = warp_reduce_scatter16(v, lane);
        if ((lane & 1) == 0) sout[half * 16 + (lane >> 1)] = s;
    }
}

// Full passes over the haloes of more than kSymBlock bound particles.  The halo's slots are
// cut into blocks of kSymBlock; an item is a block pair (tb, sb), tb <= sb, taken by one CTA
// from an atomic counter.  The CTA (4 warps of 8 targets per lane, so that the source-side
// reduce-scatter serves 8 targets) stages the source block in shared memory; warp w holds
// targets tb*kSymBlock + w*256 + t*32 + lane.  Diagonal items (tb == sb) are plain (self pair
// skipped) and write the targets' partial for slice sb.  Off-diagonal items compute each pair
// once: the targets' partial goes to slice sb (part[qoff + sb*npad + r]) and the sources'
// partial -- per source, the 4 warps' sums added in warp order, compensated -- to slice tb.  So
// slot r of block b receives slice k from item (b, k) for k >= b and from item (k, b) for
// k < b: every slice exactly once, and the energy kernel adds slices 0..B-1 in order.
__global__ void __launch_bounds__(128) ub_pair_sym_kernel(const float4 *__restrict__ pk,
                                                          const int64_t *__restrict__ poff,
                                                          const int64_t *__restrict__ qoff,
                                                          const HaloState *__restrict__ hs, int nh,
                                                          const int *__restrict__ ystart,
                                                          const int4 *__restrict__ idesc, const int *__restrict__ cnt,
                                                          int *counter, float eps2, float2 *__restrict__ part) {
    extern __shared__ float4 sym_smem[];
    float4 *ssrc = sym_smem;                                            // 32 chunks x (16 + 16) float4
    float *spart = reinterpret_cast<float *>(sym_smem + kSymBlock);     // [kSymWarps][kSymBlock]
    __shared__ int4 job;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nitems = cnt[3];
    const f2x e2 = pack2(eps2, eps2);
    for (;;) {
        if (threadIdx.x == 0) {
            const int item = atomicAdd(counter, 1);
            int4 jb = make_int4(-1, 0, 0, 0);
            if (item < nitems) {
                int lo = 0, hi = nh - 1;   // ordered halo owning the item: last q with ystart[q] <= item
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (ystart[mid] <= item) lo = mid;
                    else hi = mid - 1;
                }
                const int h = idesc[lo].x;
                const int64_t u = item - ystart[lo];
                const int64_t B = (hs[h].nb + kSymBlock - 1) / kSymBlock;
                // row tb of the upper triangle starts at tb*B - tb*(tb-1)/2
                int64_t tb = (int64_t)(((double)(2 * B + 1) - sqrt((double)(2 * B + 1) * (double)(2 * B + 1) -
                                                                     8.0 * (double)u)) * 0.5);
                tb = tb < 0 ? 0 : (tb > B - 1 ? B - 1 : tb);
                while (tb + 1 < B && (tb + 1) * B - (tb + 1) * tb / 2 <= u) ++tb;
                while (tb > 0 && tb * B - tb * (tb - 1) / 2 > u) --tb;
                const int64_t sb = tb + (u - (tb * B - tb * (tb - 1) / 2));
                jb = make_int4(h, (int)tb, (int)sb, 0);
            }
            job = jb;
        }
        __syncthreads();
        const int4 jb = job;
        if (jb.x < 0) break;
        const int h = jb.x, tb = jb.y, sb = jb.z;
        const bool sym = tb != sb;
        const int64_t base = poff[h], npad = poff[h + 1] - base;
        const int nb = hs[h].nb;
        const int s0 = sb * kSymBlock;
        const int nch = min(kSymBlock / 32, (nb - s0 + 31) >> 5);   // chunks holding sources
        // stage the source block (slots past nb: zero mass, far away)
        for (int k = threadIdx.x; k < nch * 32; k += blockDim.x) {
            const int s = s0 + k;
            const float4 p = s < nb ? pk[base + s] : make_float4(kFar, kFar, kFar, 0.f);
            float *ca = reinterpret_cast<float *>(ssrc + (k >> 5) * 32);
            const int li = k & 31, kp = li >> 1, hf = li & 1;
            ca[kp * 4 + hf] = p.x;
            ca[kp * 4 + 2 + hf] = p.y;
            ca[64 + kp * 4 + hf] = p.z;
            ca[64 + kp * 4 + 2 + hf] = p.w;
        }
        __syncthreads();
        const int t0 = tb * kSymBlock + w * 32 * kSymT;   // the warp's first target slot
        float *sp = spart + w * kSymBlock;
        if (t0 < nb) {
            f2x tx[kSymT], ty[kSymT], tz[kSymT], tm[kSymT];
            float sum[kSymT], comp[kSymT];
#pragma unroll
            for (int t = 0; t < kSymT; ++t) {
                const int r = t0 + t * 32 + lane;
                const float4 p = r < nb ? pk[base + r] : make_float4(kFar, kFar, kFar, 0.f);
                tx[t] = pack2(p.x, p.x);
                ty[t] = pack2(p.y, p.y);
                tz[t] = pack2(p.z, p.z);
                tm[t] = pack2(p.w, p.w);
                sum[t] = 0.f;
                comp[t] = 0.f;
            }
            for (int c = 0; c < nch; ++c) {
                const float4 *ca = ssrc + c * 32;
                f2x acc[kSymT];
#pragma unroll
                for (int t = 0; t < kSymT; ++t) acc[t] = pack2(0.f, 0.f);
                if (sym) {
                    chunk_pairs_sym<kSymT>(ca, ca + 16, tx, ty, tz, tm, e2, acc, sp + c * 32, lane);
                } else {
                    const int ts = c - w * kSymT;   // chunk c holds the self slot of target ts
                    if (ts >= 0 && ts < kSymT)
                        chunk_pairs<kSymT, true>(ca, ca + 16, tx, ty, tz, e2, acc, ts, lane);
                    else
                        chunk_pairs<kSymT, false>(ca, ca + 16, tx, ty, tz, e2, acc, ts, lane);
                }
#pragma unroll
                for (int t = 0; t < kSymT; ++t) {
                    float a0, a1;
                    unpack2(acc[t], a0, a1);
                    two_sum_acc(sum[t], comp[t], a0 + a1);
                }
            }
            float2 *out = part + qoff[h] + (int64_t)sb * npad;
#pragma unroll
            for (int t = 0; t < kSymT; ++t) {
                const int r = t0 + t * 32 + lane;
                if (r < nb) out[r] = df_from_acc(sum[t], comp[t]);
            }
        } else if (sym) {
            for (int k = lane; k < nch * 32; k += 32) sp[k] = 0.f;   // no targets here: no terms
        }
        if (sym) {
            __syncthreads();
            float2 *out = part + qoff[h] + (int64_t)tb * npad;
            for (int k = threadIdx.x; k < nch * 32; k += blockDim.x) {
                const int s = s0 + k;
                if (s < nb) {
                    float sum = 0.f, comp = 0.f;   // the warps' sums in warp order, compensated
#pragma unroll
                    for (int ww = 0; ww < kSymWarps; ++ww) two_sum_acc(sum, comp, spart[ww * kSymBlock + k]);
                    out[s] = df_from_acc(sum, comp);
                }
            }
        }
        __syncthreads();   // shared memory is restaged by the next item
    }
}

// The end of a pass runs in three kernels:
//   energy  - per energy segment (kSeg packed slots of one halo, so a big halo is spread over
//             many blocks): FP64 energy and sign test of every slot; removed particles are
//             marked; per-segment FP64 sums of the survivors (count, mass, mass-weighted
//             velocity) and of the pass's kinetic / potential energy.  The centre of mass is
//             not needed between passes (positions stay re-centred on the first pass's
//             centre) and is recomputed over the final bound set after the last pass;
//   finalize- one warp per halo: segment sums added in a fixed order (deterministic):
//             removals, pass count, energies, the next pass's mass and bulk velocity, and the
//             survivors / removed particles before each segment.  A halo whose pass removed
//             nothing becomes inactive;
//   compact - per segment of a halo still active: survivors copied, in order, into the other
//             packed buffer, removed particles into the next pass's source list.
constexpr int kSegSums = 8;   // removed, kept, ekin, epot, M, Mvx, Mvy, Mvz

template <class V>
__global__ void __launch_bounds__(kSegThreads) ub_energy_seg_kernel(
    const int *__restrict__ sstart, const int *__restrict__ sown, const int4 *__restrict__ idesc,
    const int *__restrict__ nsegs, const int64_t *__restrict__ poff, const int64_t *__restrict__ qoff,
    int inc, const int *__restrict__ pidx, const double *__restrict__ part,
    const double *__restrict__ phi_prev, double *__restrict__ phi_cur, const double *__restrict__ vx,
    const double *__restrict__ vy, const double *__restrict__ vz, const double *__restrict__ m, double gfac,
    const HaloState *__restrict__ hs, unsigned char *__restrict__ bound, double *__restrict__ phi_out,
    unsigned char *__restrict__ keepf, double *__restrict__ seg_sums) {
    const int seg = blockIdx.x;
    if (seg >= *nsegs) return;
    __shared__ double sh[kSegSums][32];
    const int q = sown[seg];
    const int h = idesc[q].x;
    const int sl = seg - sstart[q];
    const HaloState s = hs[h];
    const int64_t pb = poff[h], npad = poff[h + 1] - pb, qb = qoff[h];
    const int nsl = idesc[q].w;   // partial-sum slices written by this pass's pair kernels
    const int rend = min(s.nb, (sl + 1) * kSeg);
    // the segment's kSegPer slots per thread are loaded together (independent gathers in
    // flight), then evaluated in slot order
    int r[kSegPer], ii[kSegPer];
    double d[kSegPer];
#pragma unroll
    for (int j = 0; j < kSegPer; ++j) {
        r[j] = sl * kSeg + j * kSegThreads + threadIdx.x;
        ii[j] = r[j] < rend ? pidx[pb + r[j]] : -1;
        d[j] = 0.0;
    }
    for (int k = 0; k < nsl; ++k)   // slices in order
#pragma unroll
        for (int j = 0; j < kSegPer; ++j)
            if (ii[j] >= 0) d[j] += part[qb + (int64_t)k * npad + r[j]];
    // gathers of all the thread's slots issued together (predicated, no branch between them)
    double gv[kSegPer][4], pprev[kSegPer];
#pragma unroll
    for (int j = 0; j < kSegPer; ++j) {
        const int i = ii[j];
        const bool ok = i >= 0;
        gv[j][0] = ok ? vx[i] : 0.0;
        gv[j][1] = ok ? vy[i] : 0.0;
        gv[j][2] = ok ? vz[i] : 0.0;
        gv[j][3] = ok ? m[i] : 0.0;
        pprev[j] = (ok && inc) ? phi_prev[pb + r[j]] : 0.0;
    }
    double v[kSegSums] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < kSegPer; ++j) {
        const int i = ii[j];
        if (i < 0) continue;
        const double dvx = gv[j][0] - s.vx, dvy = gv[j][1] - s.vy, dvz = gv[j][2] - s.vz;
        const double ek = 0.5 * (dvx * dvx + dvy * dvy + dvz * dvz);
        // full pass: the sum itself; incremental pass: previous potential minus the removed
        // particles' contribution
        const double p = inc ? pprev[j] - d[j] : d[j];
        phi_cur[pb + r[j]] = p;
        const double e = ek - gfac * p;
        const bool keep = !(e > 0.0);
        keepf[pb + r[j]] = keep ? 1 : 0;
        if (!keep) {
            bound[i] = 0;
            v[0] += 1.0;
            if (phi_out) phi_out[i] = 0.0;
        } else {
            const double mi = gv[j][3];
            v[1] += 1.0;
            v[2] += mi * ek;
            v[3] += mi * p;
            v[4] += mi;
            v[5] += mi * gv[j][0];
            v[6] += mi * gv[j][1];
            v[7] += mi * gv[j][2];
            if (phi_out) phi_out[i] = p;
        }
    }
    block_sum_store<kSegSums>(v, sh, seg_sums + (int64_t)seg * kSegSums);
}

// One warp per active ordered halo, after the energy pass: the halo's segment sums added in a
// fixed order (lane-strided, then the warp tree), so the result does not depend on timing;
// removals, pass count, energies and the next pass's mass, centre and bulk velocity.  A halo
// whose pass removed nothing becomes inactive.  Also writes, per segment, the survivors and
// removed particles of the halo's earlier segments (seg_pre), where compaction starts writing.
__global__ void ub_finalize_kernel(int nh, const int *__restrict__ order, const int *__restrict__ sstart,
                                   const double *__restrict__ seg_sums, double gfac, HaloState *hs,
                                   int2 *__restrict__ seg_pre) {
    const int q = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (q >= nh) return;
    const int h = order[q];
    if (!hs[h].active) return;
    const int s0 = sstart[q], s1 = sstart[q + 1];
    double v[kSegSums] = {0, 0, 0, 0, 0, 0, 0, 0};
    int keep_run = 0, rem_run = 0;
    for (int b0 = s0; b0 < s1; b0 += 32) {
        const int sg = b0 + lane;
        const bool ok = sg < s1;
        const int nrem = ok ? (int)seg_sums[(int64_t)sg * kSegSums + 0] : 0;
        const int nkeep = ok ? (int)seg_sums[(int64_t)sg * kSegSums + 1] : 0;
        const int ri = warp_incl_scan(nrem, lane), ki = warp_incl_scan(nkeep, lane);
        if (ok) seg_pre[sg] = make_int2(keep_run + ki - nkeep, rem_run + ri - nrem);
        keep_run += __shfl_sync(0xffffffffu, ki, 31);
        rem_run += __shfl_sync(0xffffffffu, ri, 31);
        if (ok)
#pragma unroll
            for (int k = 0; k < kSegSums; ++k) v[k] += seg_sums[(int64_t)sg * kSegSums + k];
    }
#pragma unroll
    for (int k = 0; k < kSegSums; ++k) v[k] = warp_sum(v[k]);
    if (lane == 0) {
        HaloState &o = hs[h];
        o.nprev = o.nb;
        o.removed = (int)v[0];
        o.nrem = (int)v[0];
        o.iter += 1;
        o.ekin = v[2];
        o.epot = -0.5 * gfac * v[3];
        if (v[0] == 0.0) {
            o.active = 0;
        } else {
            const double M = v[4];
            o.M = M;
            o.nb = (int)v[1];
            if (M > 0) {
                o.vx = v[5] / M; o.vy = v[6] / M; o.vz = v[7] / M;
            } else {
                o.vx = o.vy = o.vz = 0.0;
            }
        }
    }
}

// Per segment of a halo that stays active: survivors copied in order into the other packed
// buffer (with their potential, the next incremental pass's starting point), removed
// particles into the removed list (the next pass's sources); the halo's last segment pads
// both to a multiple of 32 with zero-mass far points.
template <class V>
__global__ void __launch_bounds__(kSegThreads) ub_compact_seg_kernel(
    const int *__restrict__ sstart, const int *__restrict__ sown, const int4 *__restrict__ idesc,
    const int *__restrict__ nsegs, const int64_t *__restrict__ poff, const HaloState *__restrict__ hs,
    const unsigned char *__restrict__ keepf, const int2 *__restrict__ seg_pre, const V *__restrict__ pk_in,
    const int *__restrict__ pidx_in, const double *__restrict__ phi_cur, V *__restrict__ pk_out,
    int *__restrict__ pidx_out, double *__restrict__ phi_next, V *__restrict__ removed) {
    const int seg = blockIdx.x;
    if (seg >= *nsegs) return;
    __shared__ int wcount[kSegThreads / 32], wrem[kSegThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int q = sown[seg];
    const int h = idesc[q].x;
    if (!hs[h].active) return;   // converged this pass: its packed slots are not read again
    const int s0 = sstart[q], sl = seg - s0, nseg = sstart[q + 1] - s0;
    const int nb = hs[h].nprev;
    const int64_t pb = poff[h];
    const int2 pre = seg_pre[seg];
    int running = pre.x, rrunning = pre.y;
    const int rend = min(nb, (sl + 1) * kSeg);
    for (int r0 = sl * kSeg; r0 < rend; r0 += kSegThreads) {
        const int r = r0 + threadIdx.x;
        const bool valid = r < rend;
        const bool keep = valid && keepf[pb + r];
        const bool gone = valid && !keep;
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        const unsigned bgone = __ballot_sync(0xffffffffu, gone);
        if (lane == 0) {
            wcount[w] = __popc(bal);
            wrem[w] = __popc(bgone);
        }
        __syncthreads();
        int rank = running, rrank = rrunning, tot = 0, trem = 0;
#pragma unroll
        for (int k = 0; k < kSegThreads / 32; ++k) {
            if (k < w) {
                rank += wcount[k];
                rrank += wrem[k];
            }
            tot += wcount[k];
            trem += wrem[k];
        }
        rank += __popc(bal & ((1u << lane) - 1u));
        rrank += __popc(bgone & ((1u << lane) - 1u));
        if (keep) {
            pk_out[pb + rank] = pk_in[pb + r];
            pidx_out[pb + rank] = pidx_in[pb + r];
            phi_next[pb + rank] = phi_cur[pb + r];
        } else if (gone) {
            removed[pb + rrank] = pk_in[pb + r];
        }
        running += tot;
        rrunning += trem;
        __syncthreads();
    }
    if (sl == nseg - 1) {   // the halo's last segment pads after the survivors and the removed
        V f;
        f.x = f.y = f.z = kFar;
        f.w = 0;
        const int nkeep = running, nrem = rrunning;
        for (int r = nkeep + threadIdx.x; r < ((nkeep + 31) & ~31); r += kSegThreads) {
            pk_out[pb + r] = f;
            pidx_out[pb + r] = -1;
        }
        for (int r = nrem + threadIdx.x; r < ((nrem + 31) & ~31); r += kSegThreads) removed[pb + r] = f;
    }
}

// ---- end of a pass, FP32 path: per-particle work in FP32 and double-float only ----
// This GPU's FP64 rate is a small fraction of its FP32 rate, so the per-particle work of the
// FP32 path runs without FP64: the potential is a double-float (about 48 bits) carried from
// pass to pass, the energy and its sign test are FP32 (relative error ~1e-7, far inside the
// 1e-5 band where FP32 pair sums already leave the cut undecided), and the packed velocities
// are FP32 offsets from the bulk velocity at packing.  The halo's FP64 mass and sums of m x
// and m v are not re-summed over the survivors: each pass subtracts the FP64 sums over the
// particles it removed (gathered from the caller's FP64 arrays), usually a few per cent.
struct SegDF {
    int removed, kept;
    float2 ekin, epot;                            // double-float sums over the survivors: m ek, m phi
    double rm, rmx, rmy, rmz, rmvx, rmvy, rmvz;   // FP64 sums over the removed particles
};

// One slot's potential of the pass (full pass: the sum itself; incremental pass: the previous potential minus the
// removed particles' contribution), kinetic energy per unit mass and cut: u is the packed velocity
// offset and mass, w the halo's bulk-velocity offset.  True when the particle is kept.
struct SlotEnergy {
    float2 p;
    float pf, ek;
    bool keep;
};

__device__ __forceinline__ SlotEnergy slot_energy(float2 p, float4 u, float wx, float wy, float wz, float gfac) {
    SlotEnergy s;
    s.p = p;
    s.pf = p.x + p.y;
    const float dx = u.x - wx, dy = u.y - wy, dz = u.z - wz;
    s.ek = 0.5f * (dx * dx + dy * dy + dz * dz);
    const float e = s.ek - gfac * s.pf;
    s.keep = !(e > 0.f);
    return s;
}

__device__ __forceinline__ float2 df_warp_sum(float2 v) {
    for (int o = 16; o > 0; o >>= 1)
        v = df_add(v, make_float2(__shfl_down_sync(0xffffffffu, v.x, o), __shfl_down_sync(0xffffffffu, v.y, o)));
    return v;
}

// Per energy segment: potential phi (double-float: the slices' partials added in order, or,
// in an incremental pass, the previous potential minus them), FP32 energy
// E = 1/2 |u - w|^2 - G factor_v^2 phi with u the packed velocity offset and w the halo's
// current bulk-velocity offset, sign test; survivors' sums of m ek and m phi in double-float;
// the removed particles are listed in slot order and their FP64 mass, m x and m v summed from
// the caller's arrays, one of the seven sums a warp, while the eighth adds up the energies.
// Bound: latency, three blocks an SM.  With the list, the seven sums and the energies all in warp 0 the other
// seven waited at the barrier: 2.0 million members in haloes of 1,025 to 200,000, 526 us over 16 passes, now 419.
__global__ void __launch_bounds__(kSegThreads) ub_energy_df_kernel(
    const int *__restrict__ sstart, const int *__restrict__ sown, const int4 *__restrict__ idesc,
    const int *__restrict__ nsegs, const int64_t *__restrict__ poff, const int64_t *__restrict__ qoff, int inc,
    const int *__restrict__ pidx, const float4 *__restrict__ pv, const float2 *__restrict__ part,
    const float2 *__restrict__ phi_prev, float2 *__restrict__ phi_cur, const double *__restrict__ x,
    const double *__restrict__ y, const double *__restrict__ z, const double *__restrict__ vx,
    const double *__restrict__ vy, const double *__restrict__ vz, const double *__restrict__ m, float gfac,
    const HaloState *__restrict__ hs, unsigned char *__restrict__ bound, double *__restrict__ phi_out,
    unsigned char *__restrict__ keepf, SegDF *__restrict__ seg_sums) {
    constexpr int kWarps = kSegThreads / 32;
    static_assert(kSeg == 32 * 32 && kWarps == 8, "32 runs of 32 slots, seven sums and the energies");
    __shared__ int rlist[kSeg];
    // of two segments in turn, so that one barrier a segment is enough
    __shared__ float2 se[2][2][kWarps];
    __shared__ int gone[2][kSeg / 32];   // removed among 32 slots
    const int nseg_all = *nsegs;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double *const mine = w == 1 ? x : w == 2 ? y : w == 3 ? z : w == 4 ? vx : w == 5 ? vy : vz;
    int par = 0;
    for (int seg = blockIdx.x; seg < nseg_all; seg += gridDim.x, par ^= 1) {
        const int q = sown[seg];
        const int h = idesc[q].x;
        const int nsl = idesc[q].w;   // partial-sum slices written by this pass's pair kernels
        const int sl = seg - sstart[q];
        const int nb = hs[h].nb;
        const float wx = hs[h].wx, wy = hs[h].wy, wz = hs[h].wz;
        const int64_t pb = poff[h], npad = poff[h + 1] - pb, qb = qoff[h];
        const int rend = min(nb, (sl + 1) * kSeg);
        int r[kSegPer];
        bool ok[kSegPer];
        float4 u[kSegPer];
        float2 d[kSegPer];
#pragma unroll
        for (int j = 0; j < kSegPer; ++j) {
            r[j] = sl * kSeg + j * kSegThreads + threadIdx.x;
            ok[j] = r[j] < rend;
            u[j] = ok[j] ? pv[pb + r[j]] : make_float4(0.f, 0.f, 0.f, 0.f);
            d[j] = make_float2(0.f, 0.f);
        }
        // slices in order, four at a time with all their loads issued before the additions
        const float2 *pr[kSegPer];
#pragma unroll
        for (int j = 0; j < kSegPer; ++j) pr[j] = part + qb + (ok[j] ? r[j] : 0);
        int k = 0;
        for (; k + 4 <= nsl; k += 4) {
            float2 t[4][kSegPer];
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int j = 0; j < kSegPer; ++j) t[kk][j] = pr[j][(int64_t)(k + kk) * npad];
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int j = 0; j < kSegPer; ++j)
                    if (ok[j]) d[j] = df_add(d[j], t[kk][j]);
        }
        for (; k < nsl; ++k)
#pragma unroll
            for (int j = 0; j < kSegPer; ++j)
                if (ok[j]) d[j] = df_add(d[j], pr[j][(int64_t)k * npad]);
        float ek_s = 0.f, ek_c = 0.f, ep_s = 0.f, ep_c = 0.f;
        unsigned out[kSegPer];   // the warp's removed slots of each run
        int idx[kSegPer];
#pragma unroll
        for (int j = 0; j < kSegPer; ++j) {
            bool keep = true;
            idx[j] = 0;
            if (ok[j]) {
                const SlotEnergy s = slot_energy(inc ? df_sub(phi_prev[pb + r[j]], d[j]) : d[j], u[j], wx, wy, wz, gfac);
                keep = s.keep;
                phi_cur[pb + r[j]] = s.p;
                keepf[pb + r[j]] = keep ? 1 : 0;
                if (!keep || phi_out) idx[j] = pidx[pb + r[j]];
                if (keep) {
                    two_sum_acc(ek_s, ek_c, u[j].w * s.ek);
                    two_sum_acc(ep_s, ep_c, u[j].w * s.pf);
                } else {
                    bound[idx[j]] = 0;
                }
                if (phi_out) phi_out[idx[j]] = keep ? df_to_double(s.p) : 0.0;
            }
            out[j] = __ballot_sync(0xffffffffu, !keep);
            if (lane == 0) gone[par][j * kWarps + w] = __popc(out[j]);
        }
        const float2 ekv = df_warp_sum(df_from_acc(ek_s, ek_c));
        const float2 epv = df_warp_sum(df_from_acc(ep_s, ep_c));
        if (lane == 0) {
            se[par][0][w] = ekv;
            se[par][1][w] = epv;
        }
        __syncthreads();
        const int here = gone[par][lane];
        const int incl = warp_incl_scan(here, lane), nrem = __shfl_sync(0xffffffffu, incl, 31);
        if (nrem > 0) {   // the removed particles in slot order
#pragma unroll
            for (int j = 0; j < kSegPer; ++j) {
                const int first = __shfl_sync(0xffffffffu, incl - here, j * kWarps + w);
                if (out[j] >> lane & 1u) rlist[first + __popc(out[j] & ((1u << lane) - 1u))] = idx[j];
            }
            __syncthreads();
        }
        SegDF &o = seg_sums[seg];
        if (w < kWarps - 1) {   // sum w: lane-strided, then the warp tree
            double a = 0.0;
            for (int k = lane; k < nrem; k += 32) {
                const int i = rlist[k];
                a += m[i] * (w == 0 ? 1.0 : mine[i]);
            }
            for (int t = 16; t > 0; t >>= 1)
                if (t < nrem) a += __shfl_down_sync(0xffffffffu, a, t);
            if (lane == 0) (&o.rm)[w] = a;
        } else if (lane < 2) {   // the warps' energies in order
            float2 e = make_float2(0.f, 0.f);
            for (int k = 0; k < kWarps; ++k) e = df_add(e, se[par][lane][k]);
            (&o.ekin)[lane] = e;
            if (lane == 0) {
                o.removed = nrem;
                o.kept = max(rend - sl * kSeg, 0) - nrem;
            }
        }
    }
}

// One warp per active ordered halo after the energy pass (FP32 path): segment sums in a fixed
// order; survivors / removed before each segment (seg_pre); removals, pass count, energies;
// the halo's FP64 mass and sums of m x, m v less the removed particles' (a halo left empty
// is set to zero exactly), its centre, bulk velocity and the FP32 bulk-velocity offset for
// the next pass.  A halo whose pass removed nothing becomes inactive.
// Bound: latency of one warp per halo.  The next 32 segments are read ahead, both running counts are one scan,
// and the six quotients are a lane each: 11.6 us a pass for haloes of up to 200,000 members, now 7.6.
__global__ void ub_finalize_df_kernel(int nh, const int *__restrict__ order, const int *__restrict__ sstart,
                                      const SegDF *__restrict__ seg_sums, double gfac, HaloState *hs,
                                      int2 *__restrict__ seg_pre) {
    const int q = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (q >= nh) return;
    const int h = order[q];
    HaloState &o = hs[h];
    if (!o.active) return;
    const int s0 = sstart[q], s1 = sstart[q + 1];
    // lane 0: the mass; lanes 1 to 6: the sums of m x and m v, the centre and bulk velocity
    double *const sum = lane == 0 ? &o.M : &o.sx + (lane - 1);
    const double old = lane < 7 ? *sum : 0.0;
    const double v0 = lane >= 4 && lane < 7 ? (&o.v0x)[lane - 4] : 0.0;
    const int nb = o.nb, iter = o.iter;
    float2 ek = make_float2(0.f, 0.f), ep = make_float2(0.f, 0.f);
    double a[7] = {0, 0, 0, 0, 0, 0, 0};
    int keep_run = 0, rem_run = 0;
    SegDF next{};
    if (s0 + lane < s1) next = seg_sums[s0 + lane];
    for (int b0 = s0; b0 < s1; b0 += 32) {
        const int sg = b0 + lane;
        const SegDF g = next;
        next = SegDF{};
        if (sg + 32 < s1) next = seg_sums[sg + 32];
        // at most 32 x 1,024 of each: two 16-bit halves
        const unsigned own = (unsigned)g.removed << 16 | (unsigned)g.kept;
        const unsigned incl = (unsigned)warp_incl_scan((int)own, lane), before = incl - own;
        const unsigned all = __shfl_sync(0xffffffffu, incl, 31);
        if (sg < s1) {
            seg_pre[sg] = make_int2(keep_run + (int)(before & 0xffffu), rem_run + (int)(before >> 16));
            ek = df_add(ek, g.ekin);
            ep = df_add(ep, g.epot);
            if (g.removed > 0) {
                a[0] += g.rm; a[1] += g.rmx; a[2] += g.rmy; a[3] += g.rmz;
                a[4] += g.rmvx; a[5] += g.rmvy; a[6] += g.rmvz;
            }
        }
        keep_run += (int)(all & 0xffffu);
        rem_run += (int)(all >> 16);
    }
    ek = df_warp_sum(ek);
    ep = df_warp_sum(ep);
    if (lane == 0) {
        o.nprev = nb;
        o.removed = rem_run;
        o.nrem = rem_run;
        o.iter = iter + 1;
        o.ekin = df_to_double(ek);
        o.epot = -0.5 * gfac * df_to_double(ep);
        if (rem_run == 0) o.active = 0;
        else o.nb = keep_run;
    }
    if (rem_run == 0) return;
    // the halo's sums less the removed particles' (a halo left empty has none), and the means
    double own = 0.0;
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        for (int t = 16; t > 0; t >>= 1)
            if (t < s1 - s0) a[k] += __shfl_down_sync(0xffffffffu, a[k], t);
        const double total = __shfl_sync(0xffffffffu, a[k], 0);
        if (lane == k) own = total;
    }
    const double left = keep_run == 0 ? 0.0 : old - own;
    const double M = __shfl_sync(0xffffffffu, left, 0);
    if (lane >= 7) return;
    *sum = left;
    if (lane == 0) return;
    const double mean = M > 0 ? left / M : 0.0;
    (&o.cx)[lane - 1] = mean;
    if (lane >= 4) (&o.wx)[lane - 4] = (float)(mean - v0);
}

// Per segment of a halo that stays active (FP32 path): survivors' packed position, velocity
// offset, index and potential copied in order into the other buffers, removed particles'
// packed positions into the next pass's source list; the halo's last segment pads both.
// With next.idesc, block 0 writes the next pass's work list meanwhile (another one than this pass's).
// Bound: memory traffic (90 bytes a slot) for large catalogues.
__global__ void __launch_bounds__(kSegThreads) ub_compact_df_kernel(
    const int *__restrict__ sstart, const int *__restrict__ sown, const int4 *__restrict__ idesc,
    const int *__restrict__ nsegs, const int64_t *__restrict__ poff, const HaloState *__restrict__ hs,
    const unsigned char *__restrict__ keepf, const int2 *__restrict__ seg_pre, const float4 *__restrict__ pk_in,
    const float4 *__restrict__ pv_in, const int *__restrict__ pidx_in, const float2 *__restrict__ phi_cur,
    float4 *__restrict__ pk_out, float4 *__restrict__ pv_out, int *__restrict__ pidx_out,
    float2 *__restrict__ phi_next, float4 *__restrict__ removed, int nh, const int *__restrict__ order, ItemRule rule,
    WorkList next, unsigned long long *__restrict__ next_pairs) {
    __shared__ int wcount[kSegThreads / 32], wrem[kSegThreads / 32];
    const int lists = next.idesc ? 1 : 0;
    if ((int)blockIdx.x < lists) {
        items_block(nh, order, hs, rule, next, next_pairs);
        return;
    }
    const int nseg_all = *nsegs;
    for (int seg = blockIdx.x - lists; seg < nseg_all; seg += gridDim.x - lists) {
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        const int q = sown[seg];
        const int h = idesc[q].x;
        if (!hs[h].active) continue;   // converged this pass: its packed slots are not read again
        const int s0 = sstart[q], sl = seg - s0, nseg = sstart[q + 1] - s0;
        const int nb = hs[h].nprev;
        const int64_t pb = poff[h];
        const int2 pre = seg_pre[seg];
        int running = pre.x, rrunning = pre.y;
        const int rend = min(nb, (sl + 1) * kSeg);
        for (int r0 = sl * kSeg; r0 < rend; r0 += kSegThreads) {
            const int r = r0 + threadIdx.x;
            const bool valid = r < rend;
            const bool keep = valid && keepf[pb + r];
            const bool gone = valid && !keep;
            const unsigned bal = __ballot_sync(0xffffffffu, keep);
            const unsigned bgone = __ballot_sync(0xffffffffu, gone);
            if (lane == 0) {
                wcount[w] = __popc(bal);
                wrem[w] = __popc(bgone);
            }
            __syncthreads();
            int rank = running, rrank = rrunning, tot = 0, trem = 0;
#pragma unroll
            for (int k = 0; k < kSegThreads / 32; ++k) {
                if (k < w) {
                    rank += wcount[k];
                    rrank += wrem[k];
                }
                tot += wcount[k];
                trem += wrem[k];
            }
            rank += __popc(bal & ((1u << lane) - 1u));
            rrank += __popc(bgone & ((1u << lane) - 1u));
            if (keep) {
                pk_out[pb + rank] = pk_in[pb + r];
                pv_out[pb + rank] = pv_in[pb + r];
                pidx_out[pb + rank] = pidx_in[pb + r];
                phi_next[pb + rank] = phi_cur[pb + r];
            } else if (gone) {
                removed[pb + rrank] = pk_in[pb + r];
            }
            running += tot;
            rrunning += trem;
            __syncthreads();
        }
        if (sl == nseg - 1) {   // the halo's last segment pads after the survivors and the removed
            const float4 f = make_float4(kFar, kFar, kFar, 0.f);
            const int nkeep = running, nrem = rrunning;
            for (int r = nkeep + threadIdx.x; r < ((nkeep + 31) & ~31); r += kSegThreads) {
                pk_out[pb + r] = f;
                pv_out[pb + r] = make_float4(0.f, 0.f, 0.f, 0.f);
                pidx_out[pb + r] = -1;
            }
            for (int r = nrem + threadIdx.x; r < ((nrem + 31) & ~31); r += kSegThreads) removed[pb + r] = f;
        }
        __syncthreads();   // the shared arrays are reused by the next segment
    }
}

// Haloes of at most kSmallMax members, all passes in one block each: the halo's packed slots, its removed
// particles and its state stay in shared memory, and the passes follow one another without a launch.  Every sum is
// formed in the order of the pass kernels above (reduction, pack, tile kernel with one slice, energy, finalize), so
// the result is theirs bit for bit.
// Bound: latency -- of a pass's barriers and FP64 steps for a single small catalogue, hidden by the other blocks of
// an SM for large ones.  24 haloes of 50 to 1,000 took 16 passes x 9 launches; of 10,000 haloes of which 9,500 are
// this small, a block of 256 threads per halo and kernel was mostly empty.
// P slots, THREADS threads (slot = j * THREADS + thread, as the energy kernel has it: P <= THREADS, or 256 threads).
constexpr int kSmallMax = kSymBlock;

template <int P, int THREADS>
struct SmallShared {
    float4 src[P];       // 32-slot chunks as pairs: 16 x {x, x, y, y}, 16 x {z, z, m, m}
    float4 pv[P];        // velocity offsets and masses
    int idx[P];
    union {
        double red[kRedSums - 1][THREADS];   // before the first pass
        struct {
            float4 rem[P];   // the last pass's removed particles, as src
            float2 phi[P];
            int rlist[P];
        };
    };
    double q4[kRedSums][4];
    double centre[6];    // centre of mass and bulk velocity before the first pass
    float w[3];          // current bulk velocity relative to that
    float2 se[2][THREADS / 32];
    int cnt[2][(P + THREADS - 1) / THREADS][THREADS / 32];
};

template <int P>
__device__ __forceinline__ void put_pair_slot(float4 *chunks, int r, float x, float y, float z, float m) {
    float *c = reinterpret_cast<float *>(chunks + (r >> 5) * 32);
    const int kp = (r & 31) >> 1, hf = r & 1;
    c[kp * 4 + hf] = x;
    c[kp * 4 + 2 + hf] = y;
    c[64 + kp * 4 + hf] = z;
    c[64 + kp * 4 + 2 + hf] = m;
}

__device__ __forceinline__ float4 get_pair_slot(const float4 *chunks, int r) {
    const float *c = reinterpret_cast<const float *>(chunks + (r >> 5) * 32);
    const int kp = (r & 31) >> 1, hf = r & 1;
    return make_float4(c[kp * 4 + hf], c[kp * 4 + 2 + hf], c[64 + kp * 4 + hf], c[64 + kp * 4 + 2 + hf]);
}

// ---- a halo's blocks as a cluster (see kTeam)
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// p of the block of the given rank.
__device__ __forceinline__ void cluster_store(float2 *p, int rank, float2 v) {
    unsigned at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(at), "f"(v.x), "f"(v.y) : "memory");
}

// 32 * T targets from group g0 on against the sources' chunks; the potentials go to phi (minus them when inc), of every
// block of a team of several.  All warps call it, those without a group too: the blocks' phi must be free to
// write first (cluster_wait), which the pair terms hide.
template <int T>
__device__ __forceinline__ void small_pairs(const float4 *tgt, const float4 *src, int nb, int ns, int g0, bool inc,
                                            float eps2, float2 *phi, int team, int lane) {
    if (g0 * 32 >= nb) {
        if (team > 1) cluster_wait();
        return;
    }
    f2x tx[T], ty[T], tz[T];
    float sum[T], comp[T];
#pragma unroll
    for (int t = 0; t < T; ++t) {
        const int r = (g0 + t) * 32 + lane;
        const float4 p = r < nb ? get_pair_slot(tgt, r) : make_float4(kFar, kFar, kFar, 0.f);
        tx[t] = pack2(p.x, p.x);
        ty[t] = pack2(p.y, p.y);
        tz[t] = pack2(p.z, p.z);
        sum[t] = 0.f;
        comp[t] = 0.f;
    }
    const f2x e2 = pack2(eps2, eps2);
    for (int c = 0; c < (ns + 31) >> 5; ++c) {
        const float4 *buf = src + c * 32;
        f2x acc[T];
#pragma unroll
        for (int t = 0; t < T; ++t) acc[t] = pack2(0.f, 0.f);
        const int ts = c - g0;
        if (!inc && ts >= 0 && ts < T) chunk_pairs<T, true>(buf, buf + 16, tx, ty, tz, e2, acc, ts, lane);
        else chunk_pairs<T, false>(buf, buf + 16, tx, ty, tz, e2, acc, ts, lane);
#pragma unroll
        for (int t = 0; t < T; ++t) {
            float a0, a1;
            unpack2(acc[t], a0, a1);
            two_sum_acc(sum[t], comp[t], a0 + a1);
        }
    }
    if (team > 1) cluster_wait();
#pragma unroll
    for (int t = 0; t < T; ++t) {
        const int r = (g0 + t) * 32 + lane;
        if (r >= nb) continue;
        const float2 d = df_add(make_float2(0.f, 0.f), df_from_acc(sum[t], comp[t]));   // as one slice is added
        const float2 q = inc ? df_sub(phi[r], d) : d;
        if (team == 1) phi[r] = q;
        for (int k = 0; team > 1 && k < team; ++k) cluster_store(phi + r, k, q);
    }
}

// A few large haloes leave most SMs idle and wait for one block's pairs (939 members: 41 % of the block's time in the first
// pass, 12 % in the second).  Clusters of kTeam blocks, or of two, then share a halo: every block keeps all of its
// state and does every step, with the same bits, but only its share of the pair terms, and writes the potentials
// to all of them; from the first pass of less than kTeamWork tiles of 32 x 32 pairs on the first goes on alone.  Taken while
// all teams fit on the GPU at once.  24 haloes of 50 to 1,000: 97 us with a block each, 62 with four, 72 with two.
// Where there are many haloes, the blocks that share an SM hide one another's latency: with two instead of one
// (128 registers a thread) 10,000 haloes' largest class takes 352 us instead of 515.
constexpr int kTeam = 4, kTeamWork = 64;

template <int P, int THREADS>
__global__ void __launch_bounds__(THREADS, P == kSmallMax ? 2 : P == 256 ? 3 : 8) ub_small_kernel(
    const int *__restrict__ list, int blocks, const int64_t *__restrict__ off, const double *__restrict__ x,
    const double *__restrict__ y, const double *__restrict__ z, const double *__restrict__ vx,
    const double *__restrict__ vy, const double *__restrict__ vz, const double *__restrict__ m, float eps2, double gfac,
    int max_iter, unsigned char *__restrict__ bound, double *__restrict__ phi_out, HaloState *__restrict__ hs) {
    constexpr int J = (P + THREADS - 1) / THREADS, W = THREADS / 32;
    static_assert(J == 1 || THREADS == kSegThreads, "slots are laid out as in the energy kernel");
    extern __shared__ __align__(16) unsigned char small_raw[];
    auto &sh = *reinterpret_cast<SmallShared<P, THREADS> *>(small_raw);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // the size classes' launches are independent: the next may start as soon as this one's blocks all run, and
    // ends after it (the wait below), so that what follows in the stream follows all of them
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    constexpr bool kTeams = P == kSmallMax;
    const int rank = kTeams ? blockIdx.x % blocks : 0;   // of the halo's blocks, a cluster when there are several
    int team = kTeams ? blocks : 1;
    const int h = list[kTeams ? blockIdx.x / blocks : blockIdx.x];
    const int64_t b = off[h];
    const int n = (int)(off[h + 1] - b);
    const float gfac_f = (float)gfac;
    // ---- FP64 mass, centre and bulk velocity (ub_reduce_seg_kernel, ub_reduce_fin_kernel)
    double f[J][7];
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const int r = j * THREADS + threadIdx.x;
        const int64_t i = b + (r < n ? r : 0);
        const bool in = r < n;
        f[j][0] = in ? m[i] : 0.0;
        f[j][1] = in ? x[i] : 0.0;
        f[j][2] = in ? y[i] : 0.0;
        f[j][3] = in ? z[i] : 0.0;
        f[j][4] = in ? vx[i] : 0.0;
        f[j][5] = in ? vy[i] : 0.0;
        f[j][6] = in ? vz[i] : 0.0;
    }
    {
        double v[kRedSums - 1] = {0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < J; ++j) {
            if (j * THREADS + (int)threadIdx.x >= n) continue;
            const double mi = f[j][0];
            v[0] += mi;
#pragma unroll
            for (int k = 1; k < 7; ++k) v[k] += mi * f[j][k];
        }
#pragma unroll
        for (int k = 0; k < kRedSums - 1; ++k) sh.red[k][threadIdx.x] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < 4 * (kRedSums - 1)) {
        const int k = threadIdx.x % (kRedSums - 1), run = threadIdx.x / (kRedSums - 1);
        double t = 0.0;
        const int u1 = min(min(THREADS, n), (run + 1) * (kSegThreads / 4));   // threads past n hold zeros
        for (int u = run * (kSegThreads / 4); u < u1; ++u) t += sh.red[k][u];
        sh.q4[k][run] = t;
    }
    __syncthreads();
    // Warp 0 keeps the halo's sums, one a lane (0: M, 1..3: m x, 4..6: m v), so that a division or a subtraction is one
    // FP64 instruction for all of them: this GPU's FP64 pipe takes 16 cycles an instruction, and seven lanes cost
    // what one does.
    double val = 0.0, v0 = 0.0;
    auto per_mass = [&](double M) { return M > 0 ? val / M : 0.0; };
    if (w == 0) {
        if (lane < kRedSums - 1) val = ((sh.q4[lane][0] + sh.q4[lane][1]) + sh.q4[lane][2]) + sh.q4[lane][3];
        v0 = per_mass(__shfl_sync(0xffffffffu, val, 0));
        if (lane >= 1 && lane < 7) sh.centre[lane - 1] = v0;
        if (lane < 3) sh.w[lane] = 0.f;
    }
    __syncthreads();
    // ---- packing (ub_pack_kernel)
    {
        const double cx = sh.centre[0], cy = sh.centre[1], cz = sh.centre[2];
        const double v0x = sh.centre[3], v0y = sh.centre[4], v0z = sh.centre[5];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int r = j * THREADS + threadIdx.x;
            if (r < n) {
                put_pair_slot<P>(sh.src, r, (float)(f[j][1] - cx), (float)(f[j][2] - cy), (float)(f[j][3] - cz),
                                 (float)f[j][0]);
                sh.pv[r] = make_float4((float)(f[j][4] - v0x), (float)(f[j][5] - v0y), (float)(f[j][6] - v0z),
                                       (float)f[j][0]);
                sh.idx[r] = (int)(b + r);
            } else if (r < ((n + 31) & ~31)) {
                put_pair_slot<P>(sh.src, r, kFar, kFar, kFar, 0.f);
            }
        }
    }
    __syncthreads();
    int nb = n, nrem = 0, iter = 0;
    double ekin = 0.0, epot = 0.0;   // lane 0 of warp 0
    for (int it = 0; it < max_iter; ++it) {
        // ---- pair terms
        const bool inc = it > 0;
        const int groups = (nb + 31) >> 5, ns = inc ? nrem : nb;
        const float4 *src = inc ? sh.rem : sh.src;
        if (team > 1 && groups * ((ns + 31) >> 5) < kTeamWork) {   // the same in all blocks
            team = 1;
            if (rank > 0) break;
        }
        if (team > 1) cluster_arrive();   // this block's phi is complete and may be written
        const int item = w * team + (team > 1 ? rank : 0), items = W * team;
        if (groups <= items) small_pairs<1>(sh.src, src, nb, ns, item, inc, eps2, sh.phi, team, lane);
        else if (groups <= 2 * items) small_pairs<2>(sh.src, src, nb, ns, 2 * item, inc, eps2, sh.phi, team, lane);
        else small_pairs<4>(sh.src, src, nb, ns, 4 * item, inc, eps2, sh.phi, team, lane);
        if (team > 1) {
            cluster_arrive();
            cluster_wait();
        } else {
            __syncthreads();
        }
        // ---- energies and the cut (ub_energy_df_kernel)
        const float wx = sh.w[0], wy = sh.w[1], wz = sh.w[2];
        float ek_s = 0.f, ek_c = 0.f, ep_s = 0.f, ep_c = 0.f;
        float4 u[J], pos[J];
        float2 ph[J];
        int id[J];
        unsigned kb[J], gb[J];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int r = j * THREADS + threadIdx.x;
            const bool ok = r < nb;
            bool keep = false;
            if (ok) {
                u[j] = sh.pv[r];
                pos[j] = get_pair_slot(sh.src, r);
                id[j] = sh.idx[r];
                const SlotEnergy e = slot_energy(sh.phi[r], u[j], wx, wy, wz, gfac_f);
                ph[j] = e.p;
                keep = e.keep;
                if (keep) {
                    two_sum_acc(ek_s, ek_c, u[j].w * e.ek);
                    two_sum_acc(ep_s, ep_c, u[j].w * e.pf);
                } else if (rank == 0) {
                    bound[id[j]] = 0;
                }
            }
            kb[j] = __ballot_sync(0xffffffffu, keep);
            gb[j] = __ballot_sync(0xffffffffu, ok && !keep);
            if (lane == 0) {
                sh.cnt[0][j][w] = __popc(kb[j]);
                sh.cnt[1][j][w] = __popc(gb[j]);
            }
        }
        const float2 ekv = df_warp_sum(df_from_acc(ek_s, ek_c));
        const float2 epv = df_warp_sum(df_from_acc(ep_s, ep_c));
        if (lane == 0) {
            sh.se[0][w] = ekv;
            sh.se[1][w] = epv;
        }
        __syncthreads();
        // ---- survivors and removed particles in slot order (ub_compact_df_kernel)
        int kept = 0, gone = 0;
        const unsigned lt = (1u << lane) - 1u;
#pragma unroll
        for (int j = 0; j < J; ++j) {
            int kr = kept, gr = gone;
#pragma unroll
            for (int k = 0; k < W; ++k) {
                if (k < w) {
                    kr += sh.cnt[0][j][k];
                    gr += sh.cnt[1][j][k];
                }
                kept += sh.cnt[0][j][k];
                gone += sh.cnt[1][j][k];
            }
            if (kb[j] >> lane & 1) {
                kr += __popc(kb[j] & lt);
                put_pair_slot<P>(sh.src, kr, pos[j].x, pos[j].y, pos[j].z, pos[j].w);   // every slot was read before the barrier
                sh.pv[kr] = u[j];
                sh.idx[kr] = id[j];
                sh.phi[kr] = ph[j];
            } else if (gb[j] >> lane & 1) {
                gr += __popc(gb[j] & lt);
                put_pair_slot<P>(sh.rem, gr, pos[j].x, pos[j].y, pos[j].z, pos[j].w);
                sh.rlist[gr] = id[j];
            }
        }
        if (threadIdx.x < 32) {   // padding of both lists to whole chunks
            const int rk = kept + threadIdx.x, rg = gone + threadIdx.x;
            if (rk < ((kept + 31) & ~31)) put_pair_slot<P>(sh.src, rk, kFar, kFar, kFar, 0.f);
            if (rg < ((gone + 31) & ~31)) put_pair_slot<P>(sh.rem, rg, kFar, kFar, kFar, 0.f);
        }
        __syncthreads();
        // ---- energies of the pass, and the next pass's mass and bulk velocity (ub_finalize_df_kernel)
        ++iter;
        const bool last = gone == 0 || it + 1 == max_iter;
        if (gone > 0) {   // the removed particles' sums, in the order of the energy kernel, spread over the warps
            for (int k = w; k < kRedSums - 1; k += W) {
                const double *const of = k == 1 ? x : k == 2 ? y : k == 3 ? z : k == 4 ? vx : k == 5 ? vy : vz;
                double a = 0.0;
                for (int q = lane; q < gone; q += 32) {
                    const int i = sh.rlist[q];
                    a += m[i] * (k == 0 ? 1.0 : of[i]);
                }
                for (int t = 16; t > 0; t >>= 1)
                    if (t < gone) a += __shfl_down_sync(0xffffffffu, a, t);
                if (lane == 0) sh.q4[k][0] = a;
            }
            __syncthreads();
        }
        if (w == 0) {
            if (gone > 0) {   // the halo's sums, one a lane; the centre is formed after the last pass
                val = kept == 0 || lane >= kRedSums - 1 ? 0.0 : val - sh.q4[lane][0];
                const double v = per_mass(__shfl_sync(0xffffffffu, val, 0));
                if (lane >= 4 && lane < 7) sh.w[lane - 4] = (float)(v - v0);
            }
            if (last && lane == 0) {   // the energies of the last pass are the halo's
                float2 e0 = make_float2(0.f, 0.f), e1 = make_float2(0.f, 0.f);
                for (int k = 0; k < W; ++k) {
                    e0 = df_add(e0, sh.se[0][k]);
                    e1 = df_add(e1, sh.se[1][k]);
                }
                ekin = df_to_double(df_add(make_float2(0.f, 0.f), e0));
                epot = -0.5 * gfac * df_to_double(df_add(make_float2(0.f, 0.f), e1));
            }
        }
        nb = kept;
        nrem = gone;
        if (gone == 0) break;   // the same for all threads
        __syncthreads();
    }
    __syncthreads();
    if (phi_out && rank == 0)
        for (int r = threadIdx.x; r < nb; r += THREADS) phi_out[sh.idx[r]] = df_to_double(sh.phi[r]);
    if (w == 0 && rank == 0) {
        const double v = per_mass(__shfl_sync(0xffffffffu, val, 0));
        HaloState o{};   // what ub_output_kernel reads
        o.M = __shfl_sync(0xffffffffu, val, 0);
        o.cx = __shfl_sync(0xffffffffu, v, 1); o.cy = __shfl_sync(0xffffffffu, v, 2); o.cz = __shfl_sync(0xffffffffu, v, 3);
        o.vx = __shfl_sync(0xffffffffu, v, 4); o.vy = __shfl_sync(0xffffffffu, v, 5); o.vz = __shfl_sync(0xffffffffu, v, 6);
        o.nb = nb;
        o.iter = iter;
        o.ekin = ekin;
        o.epot = epot;
        if (lane == 0) hs[h] = o;
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Plain FP64 pair kernel for one halo (targets = sources = its packed slots).
__global__ void __launch_bounds__(256) ub_pair_f64_kernel(const double4 *__restrict__ pk, int nb, double eps2,
                                                          double *__restrict__ phi) {
    __shared__ double4 sb[256];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const double4 p = i < nb ? pk[i] : make_double4(0, 0, 0, 0);
    double acc = 0.0;
    for (int j0 = 0; j0 < nb; j0 += 256) {
        __syncthreads();
        if (j0 + threadIdx.x < nb) sb[threadIdx.x] = pk[j0 + threadIdx.x];
        __syncthreads();
        const int cnt = min(256, nb - j0);
        for (int k = 0; k < cnt; ++k) {
            if (j0 + k == i) continue;
            const double4 q = sb[k];
            const double dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
            acc = fma(q.w, rsqrt(fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)))), acc);
        }
    }
    if (i < nb) phi[i] = acc;
}

__global__ void ub_output_kernel(int nh, const HaloState *__restrict__ hs, double *__restrict__ out) {
    for (int h = blockIdx.x * blockDim.x + threadIdx.x; h < nh; h += gridDim.x * blockDim.x) {
        const HaloState s = hs[h];
        double *o = out + (int64_t)h * HALMA_UB_NFIELDS;
        o[HALMA_UB_MASS] = s.M;
        o[HALMA_UB_CX] = s.cx; o[HALMA_UB_CY] = s.cy; o[HALMA_UB_CZ] = s.cz;
        o[HALMA_UB_VX] = s.vx; o[HALMA_UB_VY] = s.vy; o[HALMA_UB_VZ] = s.vz;
        o[HALMA_UB_NBOUND] = (double)s.nb;
        o[HALMA_UB_ITER] = (double)s.iter;
        o[HALMA_UB_EKIN] = s.ekin;
        o[HALMA_UB_EPOT] = s.epot;
    }
}

// The passes run in chunks: the first pass (with the reduction and packing) alone, then kPassChunk at a time, after
// which the host asks whether any halo is left.  A call with the buffers, sizes and options of the one before replays
// one graph per chunk, the first two in one.  Another call launches the first pass as it is and captures the others
// while it runs, if its pairs keep the GPU busy for longer than a capture takes (100 us; kCapturePairs take 140);
// otherwise all its passes are launched as they are.  500 haloes of 50 to 200,000 members, other buffers on each
// call: 8,815 us with every chunk captured before its launch, 8,738 so; five of 1,500 to 5,000: 866 and 715.
constexpr int kPassChunk = 8;
constexpr double kCapturePairs = 1e9;
struct GraphCache {
    struct Entry {
        cudaGraphExec_t exec = nullptr;
        int64_t nodes = 0;
    };
    std::vector<Entry> chunks;
    std::vector<cudaGraphExec_t> old;   // of the key before, destroyed once the first chunk has been launched
    std::vector<uintptr_t> key;
    cudaStream_t capture_stream = nullptr;
    int capture_device = -1;
};
GraphCache &graph_cache() {
    static GraphCache g;
    return g;
}

// Number of haloes still active after a chunk of passes (the host stops replaying at 0).
__global__ void ub_active_kernel(int nh, const int *__restrict__ order, const HaloState *__restrict__ hs,
                                 int *__restrict__ count) {
    int a = 0;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nh; q += gridDim.x * blockDim.x) a += hs[order[q]].active;
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31) == 0 && a) atomicAdd(count, a);
}

}  // namespace

Profile &profile() {
    static Profile p;
    return p;
}

static TileTable &tile_table_ref() {
    // default until the autotuner's table is loaded: 1 chunk of targets for haloes of up to
    // 32 bound particles, 2 up to 64, 4 above
    static TileTable t = {3, {32, 64, 0x7fffffff}, {1, 2, 4}, 4096};
    return t;
}

TileTable tile_table() { return tile_table_ref(); }

int Profile::fof_mark(int stage, cudaStream_t st) {
    if (!enabled) return HALMA_OK;
    if (!fev[stage]) HALMA_CUDA(cudaEventCreate(&fev[stage]));
    HALMA_CUDA(cudaEventRecord(fev[stage], st));
    return HALMA_OK;
}

int Profile::ensure_events(int k) {
    while ((int)ev0.size() < k) {
        cudaEvent_t a, b, c;
        HALMA_CUDA(cudaEventCreate(&a));
        HALMA_CUDA(cudaEventCreate(&b));
        HALMA_CUDA(cudaEventCreate(&c));
        ev0.push_back(a);
        ev1.push_back(b);
        evm.push_back(c);
    }
    return HALMA_OK;
}

int sym_block_count(int nb) { return (nb + kSymBlock - 1) / kSymBlock; }

// Self-potential of nb particles packed as float4 (x, y, z, m), every pair evaluated once for
// both particles by the symmetric block kernel: part[b * npad + r] (npad = nb rounded up to
// 32) receives the double-float sum over the sources of block b of m_j (r^2 + eps2)^-1/2,
// j != r, for b < sym_block_count(nb).  scratch: 512 bytes of device memory for the
// description of the single work list.
int sym_self_potential_device(const float4 *pk, int nb, float eps2, float2 *part, void *scratch, cudaStream_t st) {
    if (nb <= 0) return HALMA_OK;
    if (nb > 65535 * kSymBlock) return fail(HALMA_ERR_CAPACITY, "at most %d particles", 65535 * kSymBlock);
    const int64_t B = sym_block_count(nb);
    struct Desc {
        HaloState hs;
        int64_t poff[2], qoff[2];
        int4 idesc;
        int ystart[2];
        int cnt[8];
    } d{};
    static_assert(sizeof(Desc) <= 512, "work description exceeds its scratch");
    d.hs.nb = nb;
    d.hs.active = 1;
    d.poff[1] = ((int64_t)nb + 31) / 32 * 32;
    d.idesc = make_int4(0, kSymT, 1, (int)B);
    d.ystart[1] = (int)(B * (B + 1) / 2);
    d.cnt[3] = d.ystart[1];
    HALMA_CUDA(cudaMemcpyAsync(scratch, &d, sizeof(Desc), cudaMemcpyHostToDevice, st));
    Desc *dd = static_cast<Desc *>(scratch);
    constexpr int kSymSmem = kSymBlock * (int)sizeof(float4) + kSymWarps * kSymBlock * (int)sizeof(float);
    HALMA_CUDA(cudaFuncSetAttribute(ub_pair_sym_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSymSmem));
    int bps = 0;
    HALMA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, ub_pair_sym_kernel, 128, kSymSmem));
    const int grid = (int)std::min<int64_t>((int64_t)device_sm_count() * std::max(bps, 1), d.cnt[3]);
    HALMA_LAUNCH(ub_pair_sym_kernel, grid, 128, kSymSmem, st, pk, dd->poff, dd->qoff, &dd->hs, 1, dd->ystart,
                 &dd->idesc, dd->cnt, dd->cnt + 4, eps2, part);
    return HALMA_OK;
}

template <int P, int THREADS>
static int launch_small(const int *list, int count, const int64_t *off, const double *x, const double *y,
                        const double *z, const double *vx, const double *vy, const double *vz, const double *m,
                        const halma_unbind_params &p, double gfac, unsigned char *bound, double *phi_out, HaloState *hs,
                        bool beside_last, cudaStream_t st) {
    if (count <= 0) return HALMA_OK;
    constexpr int smem = (int)sizeof(SmallShared<P, THREADS>);
    HALMA_CUDA(cudaFuncSetAttribute(ub_small_kernel<P, THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    int per_sm = 1;
    HALMA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ub_small_kernel<P, THREADS>, THREADS, smem));
    int blocks = P == kSmallMax ? kTeam : 1;
    while ((int64_t)count * blocks > (int64_t)device_sm_count() * per_sm && blocks > 1) blocks /= 2;
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = beside_last ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)blocks;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(count * blocks));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    HALMA_CUDA(cudaLaunchKernelEx(&cfg, ub_small_kernel<P, THREADS>, list, blocks, off, x, y, z, vx, vy, vz, m,
                                  (float)(p.eps * p.eps), gfac, p.max_iter, bound, phi_out, hs));
    count_launch();
    return HALMA_OK;
}

// Device-array implementation shared by halma_unbind_batched and the pipeline.
int unbind_device(int64_t n, int nh, const int64_t *d_off, const int64_t *h_off, const double *x, const double *y,
                  const double *z, const double *vx, const double *vy, const double *vz, const double *m,
                  const halma_unbind_params &p, unsigned char *bound, double *phi_out, double *halo_out,
                  cudaStream_t st, cudaEvent_t vel_ready) {
    const TileTable tab = tile_table();
    const bool f64 = p.precision == HALMA_UNBIND_FP64;
    // source slice length (a multiple of 32); the FP64 path sums a halo in one piece
    const int slice_len = f64 ? (1 << 30) : tab.slice;
    // incremental passes subtract the removed particles' potential instead of recomputing
    const bool incremental = !(p.flags & HALMA_UNBIND_FULL_RECOMPUTE);
    // Haloes of at most kSmallMax members run all their passes in one block (ub_small_kernel), which forms the
    // sums as the pass kernels do with one slice; the pass kernels take the others, nb_ of them.
    const bool use_small = !f64 && incremental && slice_len >= kSmallMax;
    auto is_small = [&](int h) { return use_small && h_off[h + 1] - h_off[h] <= kSmallMax; };
    // host-side plan: padded slot offsets, per-slice partial-sum offsets, size order
    std::vector<int64_t> poff(nh + 1), qoff(nh + 1);
    std::vector<int> order;
    order.reserve(nh);
    poff[0] = 0;
    qoff[0] = 0;
    int64_t segcap = 0;   // energy segments at most (initial sizes)
    std::vector<int> cstart(nh + 1), chunk_h;   // member chunks of kSeg (reduce and first pack)
    std::vector<int> by_size(use_small ? kSmallMax + 2 : 0, 0);   // small haloes by size
    for (int h = 0; h < nh; ++h) {
        const int64_t c = h_off[h + 1] - h_off[h];
        cstart[h] = (int)chunk_h.size();
        if (is_small(h)) {
            poff[h + 1] = poff[h];
            qoff[h + 1] = qoff[h];
            ++by_size[kSmallMax - c + 1];
            continue;
        }
        order.push_back(h);
        for (int64_t k = 0; k < (c + kSeg - 1) / kSeg; ++k) chunk_h.push_back(h);
        const int64_t npad = ((c + 31) / 32) * 32;
        int64_t nsl = std::max<int64_t>(1, (c + slice_len - 1) / slice_len);
        if (!f64 && c > kSymBlock) nsl = std::max<int64_t>(nsl, (c + kSymBlock - 1) / kSymBlock);   // symmetric
        poff[h + 1] = poff[h] + npad;
        qoff[h + 1] = qoff[h] + npad * nsl;
        segcap += std::max<int64_t>(1, (c + kSeg - 1) / kSeg);
    }
    cstart[nh] = (int)chunk_h.size();
    const int nchunks = (int)chunk_h.size();
    if (segcap >= (1ll << 31)) return fail(HALMA_ERR_CAPACITY, "too many energy segments");
    const int nb_ = (int)order.size();
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return (h_off[a + 1] - h_off[a]) > (h_off[b + 1] - h_off[b]);
    });
    // the small haloes follow in the same order (counting sort); their size classes are runs of it
    constexpr int kClass[3] = {128, 256, kSmallMax};
    int first[4] = {nb_, nb_, nb_, nb_};   // first[c]: first small halo of at most kClass[c] members
    if (use_small) {
        for (int k = 1; k <= kSmallMax + 1; ++k) by_size[k] += by_size[k - 1];
        order.resize(nh);
        for (int c = 0; c < 3; ++c) first[c] = nb_ + by_size[kSmallMax - kClass[c]];
        first[3] = nb_;
        for (int h = 0; h < nh; ++h)
            if (is_small(h)) order[nb_ + by_size[kSmallMax - (h_off[h + 1] - h_off[h])]++] = h;
    }
    const int64_t P = std::max<int64_t>(poff[nh], 32);
    const int64_t Q = std::max<int64_t>(qoff[nh], 32);
    Layout L;
    const size_t o_hs = L.add(sizeof(HaloState) * (size_t)std::max(nh, 1));
    // the plan's arrays in one piece, uploaded by one copy
    const size_t pl_poff = 0, pl_qoff = sizeof(int64_t) * (nh + 1), pl_cst = 2 * pl_qoff,
                 pl_order = pl_cst + sizeof(int) * (nh + 1), pl_chh = pl_order + sizeof(int) * nh,
                 pl_bytes = pl_chh + sizeof(int) * nchunks;
    const size_t o_plan = L.add(pl_bytes);
    const size_t vsz = f64 ? sizeof(double4) : sizeof(float4);
    const size_t o_pk = L.add(vsz * P), o_pk2 = L.add(vsz * P);       // packed slots, double-buffered
    const size_t o_pidx = L.add(sizeof(int) * P), o_pidx2 = L.add(sizeof(int) * P);
    const size_t o_keep = L.add(P);
    const size_t o_rk = L.add(vsz * P);                               // removed particles' slots
    const size_t o_phic = L.add(sizeof(double) * P), o_phin = L.add(sizeof(double) * P);
    const size_t o_phi = L.add(sizeof(double) * Q);
    const size_t o_ssum = L.add(std::max(sizeof(double) * kSegSums, sizeof(SegDF)) * segcap);
    const size_t o_pv = L.add(f64 ? 0 : sizeof(float4) * P), o_pv2 = L.add(f64 ? 0 : sizeof(float4) * P);
    const size_t o_spre = L.add(sizeof(int2) * segcap);
    const size_t o_rpart = L.add(sizeof(double) * kRedSums * std::max(nchunks, 1));
    const size_t o_cnt = L.add(64);
    // the work lists of a pass and of the next one
    size_t o_list[2][6];
    for (auto &o : o_list) {
        o[0] = L.add(sizeof(int4) * std::max(nh, 1));
        for (int k = 1; k < 4; ++k) o[k] = L.add(sizeof(int) * (nh + 1));
        o[4] = L.add(sizeof(int) * segcap);
        o[5] = L.add(64);
    }
    const size_t o_pairs = L.add(sizeof(unsigned long long) * 2 * p.max_iter);
    const size_t o_off = d_off ? 0 : L.add(sizeof(int64_t) * (nh + 1));
    const size_t o_icnt = L.add(sizeof(int4) * std::max(nh, 1)), o_ipre = L.add(sizeof(int4) * std::max(nh, 1));
    const size_t iscan_bytes = exclusive_sum_int3_bytes(std::max(nb_, 1));
    const size_t o_iscan = L.add(iscan_bytes);
    void *base = nullptr;
    HALMA_TRY(workspace(L.total, &base, st));
    auto *hs = at<HaloState>(base, o_hs);
    auto *dpoff = at<int64_t>(base, o_plan + pl_poff);
    auto *dqoff = at<int64_t>(base, o_plan + pl_qoff);
    auto *dorder = at<int>(base, o_plan + pl_order);
    int *pidxb[2] = {at<int>(base, o_pidx), at<int>(base, o_pidx2)};
    auto *keepf = at<unsigned char>(base, o_keep);
    auto *phic = at<double>(base, o_phic), *phin = at<double>(base, o_phin);
    auto *phi = at<double>(base, o_phi);
    auto *ssum = at<double>(base, o_ssum);
    auto *segpre = at<int2>(base, o_spre);
    auto *dcst = at<int>(base, o_plan + pl_cst);
    auto *dchh = at<int>(base, o_plan + pl_chh);
    auto *rpart = at<double>(base, o_rpart);
    int *nactive = at<int>(base, o_cnt);   // haloes left after a chunk of passes
    WorkList list[2];
    for (int k = 0; k < 2; ++k)
        list[k] = {at<int4>(base, o_list[k][0]), at<int>(base, o_list[k][1]), at<int>(base, o_list[k][2]),
                   at<int>(base, o_list[k][3]),  at<int>(base, o_list[k][4]), at<int>(base, o_list[k][5])};
    const int sgrid = (int)segcap;
    auto *dpairs = at<unsigned long long>(base, o_pairs);
    Profile &prof = profile();
    const bool profiling = prof.enabled;
    if (profiling) {
        HALMA_TRY(prof.ensure_events(p.max_iter));
        HALMA_CUDA(cudaMemsetAsync(dpairs, 0, sizeof(unsigned long long) * 2 * p.max_iter, st));
    }
    const int64_t *off = d_off;
    if (!d_off) {
        int64_t *o = at<int64_t>(base, o_off);
        HALMA_CUDA(cudaMemcpyAsync(o, h_off, sizeof(int64_t) * (nh + 1), cudaMemcpyHostToDevice, st));
        off = o;
    }
    {
        std::vector<unsigned char> plan(pl_bytes);
        memcpy(plan.data() + pl_poff, poff.data(), sizeof(int64_t) * (nh + 1));
        memcpy(plan.data() + pl_qoff, qoff.data(), sizeof(int64_t) * (nh + 1));
        memcpy(plan.data() + pl_cst, cstart.data(), sizeof(int) * (nh + 1));
        memcpy(plan.data() + pl_order, order.data(), sizeof(int) * nh);
        memcpy(plan.data() + pl_chh, chunk_h.data(), sizeof(int) * nchunks);
        HALMA_CUDA(cudaMemcpyAsync(dpoff, plan.data(), pl_bytes, cudaMemcpyHostToDevice, st));
    }
    const int fgrid = grid_for((int64_t)nb_ * 32, 256);   // one warp per halo
    // the pass's work list (see kItemsBlock)
    auto *icount = at<int4>(base, o_icnt), *ipre = at<int4>(base, o_ipre);
    void *iscan_tmp = at<void>(base, o_iscan);
    const int igrid = std::min(grid_for(nb_, 256), device_sm_count() * 4);
    const bool one_block = nb_ <= kItemsBlock;
    auto items = [&](cudaStream_t rs, const WorkList &wl, int inc, int sym_ok, unsigned long long *pairs) -> int {
        const ItemRule rule{tab, slice_len, inc, sym_ok};
        if (pairs) HALMA_CUDA(cudaMemsetAsync(pairs, 0, 2 * sizeof(unsigned long long), rs));
        if (one_block) {
            HALMA_LAUNCH(ub_items_kernel, 1, kSegThreads, 0, rs, nb_, dorder, hs, rule, wl, pairs);
            return HALMA_OK;
        }
        HALMA_LAUNCH(ub_items_count_kernel, igrid, 256, 0, rs, nb_, dorder, hs, rule, icount, wl.idesc, pairs);
        HALMA_TRY(exclusive_sum_int3(iscan_tmp, iscan_bytes, icount, ipre, nb_, rs));
        HALMA_LAUNCH(ub_items_fill_kernel, igrid, 256, 0, rs, nb_, icount, ipre, wl);
        return HALMA_OK;
    };
    // FP64 bound mass, centre and bulk velocity per halo (active ones, or all with force);
    // part as in ub_reduce_seg_kernel (the halo state is final after parts 1 and 2 in turn)
    auto reduce = [&](cudaStream_t rs, int force, int part = 0) -> int {
        if (nchunks > 0) {
            if (part == 1)
                HALMA_LAUNCH(ub_reduce_seg_kernel<1>, nchunks, kSegThreads, 0, rs, off, dcst, dchh, x, y, z, vx, vy,
                             vz, m, bound, hs, force, rpart);
            else if (part == 2)
                HALMA_LAUNCH(ub_reduce_seg_kernel<2>, nchunks, kSegThreads, 0, rs, off, dcst, dchh, x, y, z, vx, vy,
                             vz, m, bound, hs, force, rpart);
            else
                HALMA_LAUNCH(ub_reduce_seg_kernel<0>, nchunks, kSegThreads, 0, rs, off, dcst, dchh, x, y, z, vx, vy,
                             vz, m, bound, hs, force, rpart);
        }
        HALMA_LAUNCH(ub_reduce_fin_kernel, fgrid, 256, 0, rs, nb_, dorder, dcst, rpart, force, hs);
        return HALMA_OK;
    };
    const double gfac = p.G * p.factor_v * p.factor_v;
    const float eps2 = (float)(p.eps * p.eps);
    HALMA_LAUNCH(ub_init_kernel, std::min(device_sm_count() * 8, grid_for(std::max<int64_t>(n, nh), 256)), 256, 0, st,
                 n, bound, nh, hs);
    if (phi_out) HALMA_CUDA(cudaMemsetAsync(phi_out, 0, sizeof(double) * n, st));

    // the longest blocks first; each class may start beside the one launched before it
    auto small = [&]() -> int {
        HALMA_TRY((launch_small<kSmallMax, 256>(dorder + first[2], first[1] - first[2], off, x, y, z, vx, vy, vz, m, p,
                                                gfac, bound, phi_out, hs, false, st)));
        HALMA_TRY((launch_small<256, 256>(dorder + first[1], first[0] - first[1], off, x, y, z, vx, vy, vz, m, p, gfac,
                                          bound, phi_out, hs, first[1] > first[2], st)));
        return launch_small<128, 128>(dorder + first[0], nh - first[0], off, x, y, z, vx, vy, vz, m, p, gfac, bound,
                                      phi_out, hs, first[0] > first[2], st);
    };
    // velocities that may still be arriving: after the big haloes' first pass has waited for them
    if (use_small && !vel_ready) HALMA_TRY(small());
    if (!f64 && nb_ > 0) {
        float4 *pkb[2] = {at<float4>(base, o_pk), at<float4>(base, o_pk2)};
        float4 *pvb[2] = {at<float4>(base, o_pv), at<float4>(base, o_pv2)};
        auto *part2 = reinterpret_cast<float2 *>(phi);   // double-float partials and potentials
        auto *phic2 = reinterpret_cast<float2 *>(phic), *phin2 = reinterpret_cast<float2 *>(phin);
        auto *sdf = reinterpret_cast<SegDF *>(ssum);
        const float gfac_f = (float)gfac;
        int bps = 0;
        HALMA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, ub_pair_kernel, 256, 0));
        const int pgrid = device_sm_count() * std::max(bps, 1);
        constexpr int kSymSmem = kSymBlock * (int)sizeof(float4) + kSymWarps * kSymBlock * (int)sizeof(float);
        HALMA_CUDA(cudaFuncSetAttribute(ub_pair_sym_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSymSmem));
        HALMA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, ub_pair_sym_kernel, 128, kSymSmem));
        const int ygrid = device_sm_count() * std::max(bps, 1);
        // the end-of-pass kernels loop over the pass's energy segments with one wave of blocks
        // (a launch of one block per possible segment cost ~30 us even when few were active)
        HALMA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, ub_energy_df_kernel, kSegThreads, 0));
        const int egrid = std::min(sgrid, device_sm_count() * std::max(bps, 1));
        HALMA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, ub_compact_df_kernel, kSegThreads, 0));
        const int cgrid = std::min(sgrid, device_sm_count() * std::max(bps, 1));
        auto record = [&](cudaStream_t rs, int it0, int it1, bool capturing) -> int {
            // external: captured as event nodes, so that the replay records and waits for them
            const unsigned rec = capturing ? cudaEventRecordExternal : cudaEventRecordDefault;
            // first pass: centre of mass and packing into buffer 0; every pass then compacts
            // its survivors into the other buffer and sets the next pass's halo state
            // With vel_ready, the velocities may still be arriving: the first pass's pair
            // kernels start from the positions and masses, and the velocity sums and packed
            // velocities follow once vel_ready has fired, before the first energy kernel.
            if (it0 == 0) {
                HALMA_TRY(reduce(rs, 0, vel_ready ? 1 : 0));
                if (nchunks > 0)
                    HALMA_LAUNCH(ub_pack_kernel<float4>, nchunks, kSegThreads, 0, rs, off, dpoff, dcst, dchh, x, y, z,
                                 m, vx, vy, vz, hs, pkb[0], vel_ready ? nullptr : pvb[0], pidxb[0]);
            }
            float4 *rk = at<float4>(base, o_rk);
            for (int it = it0; it < it1; ++it) {
                const int a = it & 1, b = a ^ 1;
                const int inc = (it > 0 && incremental) ? 1 : 0;
                const WorkList &wl = list[a];
                // from the second pass on the last compaction may have written it
                if (it == 0 || !one_block) HALMA_TRY(items(rs, wl, inc, 1, profiling ? dpairs + 2 * it : nullptr));
                if (profiling) HALMA_CUDA(cudaEventRecordWithFlags(prof.ev0[it], rs, rec));
                // full passes: the big haloes' block pairs first (the longest items), then the
                // tiles of the small ones; incremental passes have only tiles
                if (!inc)
                    HALMA_LAUNCH(ub_pair_sym_kernel, ygrid, 128, kSymSmem, rs, pkb[a], dpoff, dqoff, hs, nb_,
                                 wl.ystart, wl.idesc, wl.cnt, wl.cnt + 4, eps2, part2);
                if (profiling) HALMA_CUDA(cudaEventRecordWithFlags(prof.evm[it], rs, rec));
                HALMA_LAUNCH(ub_pair_kernel, pgrid, 256, 0, rs, pkb[a], rk, inc, dpoff, dqoff, hs, nb_, wl.istart,
                             wl.idesc, wl.cnt, wl.cnt + 1, eps2, slice_len / 32, part2);
                if (profiling) HALMA_CUDA(cudaEventRecordWithFlags(prof.ev1[it], rs, rec));
                if (it == 0 && vel_ready) {
                    HALMA_CUDA(cudaStreamWaitEvent(rs, vel_ready, capturing ? cudaEventWaitExternal : cudaEventWaitDefault));
                    HALMA_TRY(reduce(rs, 0, 2));
                    if (nchunks > 0)
                        HALMA_LAUNCH(ub_pack_kernel<float4>, nchunks, kSegThreads, 0, rs, off, dpoff, dcst, dchh, x, y,
                                     z, m, vx, vy, vz, hs, (float4 *)nullptr, pvb[0], (int *)nullptr);
                }
                HALMA_LAUNCH(ub_energy_df_kernel, egrid, kSegThreads, 0, rs, wl.sstart, wl.sown, wl.idesc, wl.cnt + 2,
                             dpoff, dqoff, inc, pidxb[a], pvb[a], part2, phin2, phic2, x, y, z, vx, vy, vz, m, gfac_f,
                             hs, bound, phi_out, keepf, sdf);
                HALMA_LAUNCH(ub_finalize_df_kernel, fgrid, 256, 0, rs, nb_, dorder, wl.sstart, sdf, gfac, hs, segpre);
                HALMA_LAUNCH(ub_compact_df_kernel, cgrid + one_block, kSegThreads, 0, rs, wl.sstart, wl.sown, wl.idesc,
                             wl.cnt + 2, dpoff, hs, keepf, segpre, pkb[a], pvb[a], pidxb[a], phic2, pkb[b], pvb[b],
                             pidxb[b], phin2, rk, nb_, dorder, ItemRule{tab, slice_len, incremental ? 1 : 0, 1},
                             one_block ? list[b] : WorkList{},
                             profiling && it + 1 < p.max_iter ? dpairs + 2 * (it + 1) : nullptr);
            }
            if (it1 == 1) return HALMA_OK;
            HALMA_CUDA(cudaMemsetAsync(nactive, 0, sizeof(int), rs));
            HALMA_LAUNCH(ub_active_kernel, std::min(grid_for(nb_, 256), 64), 256, 0, rs, nb_, dorder, hs, nactive);
            return HALMA_OK;
        };
        int passes_run = p.max_iter;
        if (p.use_graph) {
            std::vector<uintptr_t> key = {(uintptr_t)base, (uintptr_t)off, (uintptr_t)x, (uintptr_t)y, (uintptr_t)z,
                                          (uintptr_t)vx, (uintptr_t)vy, (uintptr_t)vz, (uintptr_t)m,
                                          (uintptr_t)bound, (uintptr_t)phi_out, (uintptr_t)n, (uintptr_t)nh,
                                          (uintptr_t)p.max_iter, (uintptr_t)st};
            uint64_t eb = 0, gb = 0;
            memcpy(&eb, &eps2, sizeof(float));
            memcpy(&gb, &gfac, sizeof(double));
            key.push_back((uintptr_t)eb);
            key.push_back((uintptr_t)gb);
            key.insert(key.end(), poff.begin(), poff.end());
            key.push_back((uintptr_t)current_device());
            key.push_back((uintptr_t)profiling);
            key.push_back((uintptr_t)dpairs);
            key.push_back((uintptr_t)tab.n);
            key.push_back((uintptr_t)slice_len);
            key.push_back((uintptr_t)incremental);
            key.push_back((uintptr_t)nchunks);
            key.push_back((uintptr_t)nb_);
            key.push_back((uintptr_t)vel_ready);
            for (int c = 0; c < tab.n; ++c) {
                key.push_back((uintptr_t)tab.upper[c]);
                key.push_back((uintptr_t)tab.t[c]);
            }
            GraphCache &gc = graph_cache();
            const bool again = gc.key == key;
            if (!again) {
                for (auto &e : gc.chunks)
                    if (e.exec) gc.old.push_back(e.exec);
                gc.chunks.clear();
                gc.key = key;
            }
            // capture on a private stream (the legacy default stream cannot be captured)
            if (!gc.capture_stream || gc.capture_device != current_device()) {
                HALMA_CUDA(cudaStreamCreateWithFlags(&gc.capture_stream, cudaStreamNonBlocking));
                gc.capture_device = current_device();
            }
            const int nchunk = 1 + (p.max_iter - 1 + kPassChunk - 1) / kPassChunk;
            auto chunk_start = [&](int ci) { return ci == 0 ? 0 : std::min(p.max_iter, 1 + (ci - 1) * kPassChunk); };
            // replayed, the first chunk is one graph with the second
            auto next_chunk = [&](int ci) { return again && ci == 0 ? 2 : ci + 1; };
            gc.chunks.resize(nchunk);
            double pairs = 0.0;
            for (int q = 0; q < nb_; ++q) {
                const double c = (double)(h_off[order[q] + 1] - h_off[order[q]]);
                pairs += c * c;
            }
            // chunks from here on are graphs, those before are launched one by one
            const int first_graph = again ? 0 : pairs >= kCapturePairs ? 1 : nchunk;
            auto capture = [&](int ci) -> int {
                if (ci < first_graph || ci >= nchunk || gc.chunks[ci].exec) return HALMA_OK;
                GraphCache::Entry &ge = gc.chunks[ci];
                cudaGraph_t graph = nullptr;
                HALMA_CUDA(cudaStreamBeginCapture(gc.capture_stream, cudaStreamCaptureModeThreadLocal));
                const int64_t before = halma_kernel_launch_count();
                int s = record(gc.capture_stream, chunk_start(ci), chunk_start(next_chunk(ci)), true);
                cudaError_t ce = cudaStreamEndCapture(gc.capture_stream, &graph);
                if (s != HALMA_OK) {
                    if (graph) cudaGraphDestroy(graph);
                    return s;
                }
                HALMA_CUDA(ce);
                cudaError_t ie = cudaGraphInstantiate(&ge.exec, graph, 0);
                cudaGraphDestroy(graph);
                HALMA_CUDA(ie);
                ge.nodes = halma_kernel_launch_count() - before;
                add_launches(-ge.nodes);   // counted again at every replay below
                return HALMA_OK;
            };
            passes_run = 0;
            for (int ci = 0; ci < nchunk; ci = next_chunk(ci)) {
                HALMA_TRY(capture(ci));
                if (ci >= first_graph) {
                    HALMA_CUDA(cudaGraphLaunch(gc.chunks[ci].exec, st));
                    add_launches(gc.chunks[ci].nodes);
                } else {
                    HALMA_TRY(record(st, chunk_start(ci), chunk_start(next_chunk(ci)), false));
                }
                for (cudaGraphExec_t e : gc.old) cudaGraphExecDestroy(e);   // 100 us of the host's time
                gc.old.clear();
                passes_run = chunk_start(next_chunk(ci));
                if (passes_run >= p.max_iter) break;
                HALMA_TRY(capture(next_chunk(ci)));   // while this one runs
                if (passes_run == 1) continue;
                int active = 0;
                HALMA_CUDA(cudaMemcpyAsync(&active, nactive, sizeof(int), cudaMemcpyDeviceToHost, st));
                HALMA_CUDA(cudaStreamSynchronize(st));
                if (active == 0) break;
            }
        } else {
            HALMA_TRY(record(st, 0, p.max_iter, false));
        }
        // the halo state already holds the final bound set's mass, centre and bulk velocity
        if (profiling) {
            std::vector<unsigned long long> hp(2 * p.max_iter);
            HALMA_CUDA(cudaMemcpyAsync(hp.data(), dpairs, sizeof(unsigned long long) * 2 * p.max_iter,
                                       cudaMemcpyDeviceToHost, st));
            HALMA_CUDA(cudaStreamSynchronize(st));
            prof.passes.clear();
            for (int it = 0; it < passes_run; ++it) {
                float ms = 0.f, sms = 0.f;
                HALMA_CUDA(cudaEventElapsedTime(&ms, prof.ev0[it], prof.ev1[it]));
                HALMA_CUDA(cudaEventElapsedTime(&sms, prof.ev0[it], prof.evm[it]));
                prof.passes.push_back({(double)hp[2 * it], (double)ms, (double)hp[2 * it + 1], (double)sms});
            }
        }
    } else if (!f64) {
        if (profiling) prof.passes.clear();
    } else {
        // plain FP64 path: per pass, one pair launch per active halo, host checks convergence
        double4 *pkb[2] = {at<double4>(base, o_pk), at<double4>(base, o_pk2)};
        std::vector<HaloState> hh(nh);
        HALMA_TRY(reduce(st, 0));
        if (nchunks > 0)
            HALMA_LAUNCH(ub_pack_kernel<double4>, nchunks, kSegThreads, 0, st, off, dpoff, dcst, dchh, x, y, z, m, vx,
                         vy, vz, hs, pkb[0], nullptr, pidxb[0]);
        double4 *rk = at<double4>(base, o_rk);
        for (int it = 0; it < p.max_iter; ++it) {
            const int a = it & 1, b = a ^ 1;
            const WorkList &wl = list[0];
            HALMA_TRY(items(st, wl, 0, 0, nullptr));
            HALMA_CUDA(cudaMemcpyAsync(hh.data(), hs, sizeof(HaloState) * nh, cudaMemcpyDeviceToHost, st));
            HALMA_CUDA(cudaStreamSynchronize(st));
            int any = 0;
            for (int h = 0; h < nh; ++h) {
                if (!hh[h].active || hh[h].nb == 0) continue;
                any = 1;
                HALMA_LAUNCH(ub_pair_f64_kernel, grid_for(hh[h].nb, 256), 256, 0, st, pkb[a] + poff[h], hh[h].nb,
                             p.eps * p.eps, phi + poff[h]);
            }
            if (!any) break;
            HALMA_LAUNCH(ub_energy_seg_kernel<double4>, sgrid, kSegThreads, 0, st, wl.sstart, wl.sown, wl.idesc,
                         wl.cnt + 2, dpoff, dqoff, 0, pidxb[a], phi, phin, phic, vx, vy, vz, m, gfac, hs, bound, phi_out, keepf,
                         ssum);
            HALMA_LAUNCH(ub_finalize_kernel, fgrid, 256, 0, st, nh, dorder, wl.sstart, ssum, gfac, hs, segpre);
            HALMA_LAUNCH(ub_compact_seg_kernel<double4>, sgrid, kSegThreads, 0, st, wl.sstart, wl.sown, wl.idesc,
                         wl.cnt + 2, dpoff, hs, keepf, segpre, pkb[a], pidxb[a], phic, pkb[b], pidxb[b], phin, rk);
        }
        HALMA_TRY(reduce(st, 1));
    }
    if (use_small && vel_ready) {
        HALMA_CUDA(cudaStreamWaitEvent(st, vel_ready, 0));
        HALMA_TRY(small());
    }
    if (halo_out) HALMA_LAUNCH(ub_output_kernel, grid_for(nh, 256), 256, 0, st, nh, hs, halo_out);
    return HALMA_OK;
}

}  // namespace halma

using namespace halma;

extern "C" int halma_unbind_batched(int64_t n, int64_t n_haloes, const int64_t *offsets, const double *x,
                                    const double *y, const double *z, const double *vx, const double *vy,
                                    const double *vz, const double *m, const halma_unbind_params *params,
                                    uint8_t *bound, double *phi, double *halo_out, halma_stream_t stream) {
    if (!params) return fail(HALMA_ERR_INVALID, "params is NULL");
    const halma_unbind_params p = *params;
    if (n < 0 || n_haloes < 0) return fail(HALMA_ERR_INVALID, "negative size");
    if (n >= (1ll << 31) - 64) return fail(HALMA_ERR_CAPACITY, "at most 2^31-65 particles per call");
    if (n_haloes >= (1ll << 31) - 1) return fail(HALMA_ERR_CAPACITY, "too many haloes");
    if (!(p.eps > 0.0) || !isfinite(p.eps)) return fail(HALMA_ERR_INVALID, "eps must be finite and > 0");
    if (!isfinite(p.G) || !isfinite(p.factor_v)) return fail(HALMA_ERR_INVALID, "G and factor_v must be finite");
    if (p.max_iter < 1 || p.max_iter > 1000) return fail(HALMA_ERR_INVALID, "max_iter must be in [1, 1000]");
    if (p.precision != HALMA_UNBIND_FP32C && p.precision != HALMA_UNBIND_FP64)
        return fail(HALMA_ERR_INVALID, "unknown precision %d", p.precision);
    if (!offsets || (n > 0 && (!x || !y || !z || !vx || !vy || !vz || !m || !bound)))
        return fail(HALMA_ERR_INVALID, "null pointer");
    if (n_haloes == 0) return HALMA_OK;
    std::lock_guard<std::mutex> guard(api_mutex());
    cudaStream_t st = (cudaStream_t)stream;
    // the plan needs the offsets on the host
    std::vector<int64_t> h_off(n_haloes + 1);
    const bool dev_off = is_device_pointer(offsets);
    if (dev_off) {
        HALMA_CUDA(cudaMemcpyAsync(h_off.data(), offsets, sizeof(int64_t) * (n_haloes + 1), cudaMemcpyDeviceToHost, st));
        HALMA_CUDA(cudaStreamSynchronize(st));
    } else {
        memcpy(h_off.data(), offsets, sizeof(int64_t) * (n_haloes + 1));
    }
    if (h_off[0] != 0 || h_off[n_haloes] != n) return fail(HALMA_ERR_INVALID, "offsets must start at 0 and end at n");
    for (int64_t h = 0; h < n_haloes; ++h)
        if (h_off[h + 1] < h_off[h]) return fail(HALMA_ERR_INVALID, "offsets must be non-decreasing");
    Stager sg;
    const double *dx = nullptr, *dy = nullptr, *dz = nullptr, *dvx = nullptr, *dvy = nullptr, *dvz = nullptr,
                 *dm = nullptr;
    unsigned char *db = nullptr;
    double *dphi = nullptr, *dout = nullptr;
    sg.add(x, n, true, false, &dx);
    sg.add(y, n, true, false, &dy);
    sg.add(z, n, true, false, &dz);
    sg.add(vx, n, true, false, &dvx);
    sg.add(vy, n, true, false, &dvy);
    sg.add(vz, n, true, false, &dvz);
    sg.add(m, n, true, false, &dm);
    sg.add((const unsigned char *)bound, n, false, true, &db);
    sg.add((const double *)phi, phi ? n : 0, false, true, &dphi);
    sg.add((const double *)halo_out, halo_out ? n_haloes * HALMA_UB_NFIELDS : 0, false, true, &dout);
    void *stage = nullptr;
    if (sg.any_host) {
        Layout L;
        sg.plan(L);
        HALMA_CUDA(cudaMallocAsync(&stage, L.total, st));
    }
    int s = sg.bind_and_upload(stage, st);
    if (s == HALMA_OK)
        s = unbind_device(n, (int)n_haloes, dev_off ? offsets : nullptr, h_off.data(), dx, dy, dz, dvx, dvy, dvz, dm,
                          p, db, dphi, dout, st);
    if (s == HALMA_OK) s = sg.download(st);
    if (stage) {
        cudaFreeAsync(stage, st);
        cudaStreamSynchronize(st);
    }
    return s;
}

extern "C" int halma_set_tile_table(int32_t n_classes, const int32_t *upper, const int32_t *t_per_class,
                                    int32_t slice_len) {
    if (n_classes < 1 || n_classes > kMaxTileClasses || !upper || !t_per_class)
        return fail(HALMA_ERR_INVALID, "tile table needs 1..%d classes", kMaxTileClasses);
    if (slice_len < 32 || slice_len % 32 != 0 || slice_len > (1 << 26))
        return fail(HALMA_ERR_INVALID, "source slice must be a positive multiple of 32 (at most 2^26)");
    TileTable t{};
    t.n = n_classes;
    t.slice = slice_len;
    for (int c = 0; c < n_classes; ++c) {
        const int v = t_per_class[c];
        if (v != 1 && v != 2 && v != 4) return fail(HALMA_ERR_INVALID, "tile shape must be 1, 2 or 4");
        if (upper[c] < 1 || (c > 0 && upper[c] <= upper[c - 1]))
            return fail(HALMA_ERR_INVALID, "class bounds must be positive and increasing");
        t.upper[c] = upper[c];
        t.t[c] = v;
    }
    std::lock_guard<std::mutex> guard(api_mutex());
    tile_table_ref() = t;
    return HALMA_OK;
}

extern "C" int halma_get_tile_table(int32_t *n_classes, int32_t *upper, int32_t *t_per_class,
                                    int32_t *slice_len) {
    if (!n_classes || !upper || !t_per_class || !slice_len) return fail(HALMA_ERR_INVALID, "null pointer");
    std::lock_guard<std::mutex> guard(api_mutex());
    const TileTable &t = tile_table_ref();
    *n_classes = t.n;
    *slice_len = t.slice;
    for (int c = 0; c < t.n; ++c) {
        upper[c] = t.upper[c];
        t_per_class[c] = t.t[c];
    }
    return HALMA_OK;
}
