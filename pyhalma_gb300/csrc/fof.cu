// Friends-of-friends on the GPU: the C ABI that replaces python_scripts/fof.py:18-79.
//
// Pipeline (all on one stream):
//   1. bounding box (FP64) -> host picks the cell geometry (cell side = ll * (1 + 2^-20));
//   2. each particle gets a row-major cell key with its half-cell (2 x 2 x 2) below it; keys are
//      radix-sorted with their indices;
//   3. the particles of one half-cell lie within sqrt(3)/2 of the linking length of each other, so they
//      are one component whatever their positions: a node.  One pass over the sorted keys numbers
//      cells and nodes and gathers the particles' records (position inside the cell in units of ll,
//      original index);
//   4. per cell, its occupied forward neighbours among 13, found by lower bounds in the sorted cell
//      keys (the key grid is padded so that a neighbour key is a constant offset), in one list of
//      cell pairs;
//   5. links in a lock-free union-find over nodes (atomicCAS, randomised linking, path halving): every node joins
//      the first two nodes ahead of it that it is linked to, which leaves about one in a hundred pairs of
//      neighbouring nodes in different sets; those are listed by a sweep over the nodes and each is tested
//      particle by particle up to its first link.
//      A pair of particles whose float32 distance is clearly inside (outside) the linking length is accepted
//      (rejected); pairs in a +-1e-5 band are re-tested with the exact FP64 predicate
//      ((dx*dx + dy*dy) + dz*dz) <= ll*ll, every operation rounded on its own.  Pairs of crowded nodes without
//      a link among their first tests go to lists that warps, and for the largest blocks, work off;
//   6. each component's label = the smallest ORIGINAL index among its members (atomicMin over nodes), -1
//      for particles alone.
// Inputs of up to kSmallFof particles take all pairs instead (fof_small).
// The result is the reference's partition exactly: same components, same canonical labels.
#include <math.h>
#include <limits.h>
#include <string.h>

#include <map>

#include "common.cuh"
#include "sort.cuh"
#include "unbind.cuh"

namespace halma {

namespace {

constexpr int kUfCapDefault = 1 << 26;   // bound on any union-find loop (never reached in practice)
// The bound the kernels use: halma_set_union_find_cap changes it (a debug knob, so that tests
// can make the loops run out); pushed to each device before its next FoF.
__constant__ int c_uf_cap = kUfCapDefault;

struct FofGeom {
    double xmin, ymin, zmin;
    double cell, inv_cell, inv_scale, r2;
    float cs, lo, hi;
    long long ncx, ncy, ncz;
    // key dimensions: ncy + 1 and ncz + 1.  Every y-row and z-column of the key grid ends in an
    // empty pad cell, so that a neighbour's key is the cell's key plus a constant that never
    // wraps onto an occupied cell (a wrap lands on a pad cell or past the last slab)
    long long ky, kz;
    int sb;   // low key bits holding the half-cell (x, y, z) within the cell: 3, or 0 when nodes are particles
};

// Segmented FoF (links only inside a segment): every segment gets its own origin (the
// minimum corner of its bounding box) and its own run of x columns of one virtual cell grid,
// followed by an empty column, so that a cell's forward neighbours are either cells of the
// same segment or empty.  All pointers are null for a plain FoF.
struct SegGeom {
    const int *seg_of = nullptr;       // segment of each particle
    const double *smin = nullptr;      // [3 * nseg] origin of each segment
    const long long *scol = nullptr;   // [4 * nseg] first virtual x column, columns in x, y, z
};

// SHARED: the parents lie in shared memory.
template <bool SHARED>
__device__ __forceinline__ int uf_load(const int *p) {
    return SHARED ? *(const volatile int *)p : __ldcg(p);
}
template <bool SHARED>
__device__ __forceinline__ void uf_store(int *p, int v) {
    if (SHARED) *(volatile int *)p = v;
    else __stcg(p, v);
}

template <bool SHARED = false>
__device__ __forceinline__ int uf_find(int *parent, int v, int *err) {
    int p = uf_load<SHARED>(parent + v);
    int guard = 0;
    const int cap = c_uf_cap;
    while (p != v) {
        const int gp = uf_load<SHARED>(parent + p);
        if (gp != p) uf_store<SHARED>(parent + v, gp);   // path halving: gp is an ancestor of v
        v = p;
        p = gp;
        if (++guard > cap) {
            atomicOr(err, 1);
            break;
        }
    }
    return v;
}

// A scattered order of the nodes: a bijection of 32-bit integers, multiplicative hashing by the golden ratio (D. E. Knuth,
// The Art of Computer Programming 3, 6.4) twice, with the upper half folded in between.  Neighbouring nodes have neighbouring
// numbers: hooked in the order of their numbers they make chains as long as a group, and a walk is one dependent memory
// access a step; hooked in random order, trees are logarithmically deep (A. Goel, S. Khanna, D. Larkin, R. E. Tarjan,
// Disjoint set union with randomized linking, SODA 2014).
__device__ __forceinline__ unsigned uf_rank(int v) {
    constexpr unsigned kGolden = 2654435769u;   // 2^32 / 1.618.., odd
    const unsigned h = (unsigned)v * kGolden;
    return (h ^ (h >> 16)) * kGolden;
}

// Joins the sets of two ancestors a and b (roots or not): hooks the root of the larger rank under that of
// the smaller, retrying from the current roots when the CAS finds that a is no longer a root.
// Returns the node hooked under (or the common root when the two are one set already): an ancestor
// of every member of both sets, which the caller may use in place of a fresh find.
__device__ __forceinline__ int uf_union(int *parent, int a, int b, int *err) {
    int guard = 0;
    const int cap = c_uf_cap;
    while (a != b) {
        if (uf_rank(a) < uf_rank(b)) {
            const int t = a;
            a = b;
            b = t;
        }
        const int old = atomicCAS(parent + a, a, b);
        if (old == a) return b;
        a = uf_find(parent, old, err);
        b = uf_find(parent, b, err);
        if (++guard > cap) {
            atomicOr(err, 1);
            return b;
        }
    }
    return a;
}

// The same for a whole warp: every lane with need joins its a and b, all lanes one step at a time (one step of
// both walks, or the hook).  In nested loops of their own the lanes ran one after another (3.7 of 32
// active).  Returns each lane's node as above.
template <bool SHARED = false>
__device__ __forceinline__ int uf_union_warp(int *parent, int a, int b, bool need, int *err) {
    const int cap = c_uf_cap;
    int guard = 0, xa = -1, xb = -1;   // the nodes before a and b on their walks
    while (__any_sync(0xffffffffu, need)) {
        if (need) {
            const int pa = uf_load<SHARED>(parent + a), pb = uf_load<SHARED>(parent + b);
            if (pa == a && pb == b) {
                if (a != b) {
                    const bool swap = uf_rank(a) < uf_rank(b);
                    const int hi = swap ? b : a, lo = swap ? a : b;
                    const int old = atomicCAS(parent + hi, hi, lo);
                    a = old == hi ? lo : old;
                    b = lo;
                    xa = xb = -1;
                    need = old != hi;
                } else {
                    need = false;
                }
            } else {   // path halving: pa and pb are ancestors of xa and xb
                if (pa != a && xa >= 0) uf_store<SHARED>(parent + xa, pa);
                if (pb != b && xb >= 0) uf_store<SHARED>(parent + xb, pb);
                xa = a;
                xb = b;
                a = pa;
                b = pb;
                if (a == b) need = false;
            }
            if (need && ++guard > cap) {
                atomicOr(err, 1);
                need = false;
            }
        }
    }
    return b;
}

// Doubles as order-preserving signed 64-bit integers (sign-magnitude turned into two's
// complement), so that a bounding box is integer min / max: GB300 issues FP64 instructions at
// a small fraction of its integer rate.  -0.0 orders just below +0.0; NaN and infinities are
// flagged separately.
__device__ __forceinline__ long long ord_of(double v) {
    const long long u = __double_as_longlong(v);
    return u ^ ((u >> 63) & 0x7fffffffffffffffll);
}

__device__ __forceinline__ double val_of(long long k) {
    return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll));
}

__device__ __forceinline__ bool nonfinite(double v) {
    return (__double_as_longlong(v) & 0x7ff0000000000000ll) == 0x7ff0000000000000ll;
}

// part[7 * block + q]: the block's min x, y, z and max x, y, z as order keys, and a non-finite flag.
__global__ void bbox_partial_kernel(const double *__restrict__ x, const double *__restrict__ y,
                                    const double *__restrict__ z, int n, long long *__restrict__ part) {
    long long mn[3] = {LLONG_MAX, LLONG_MAX, LLONG_MAX}, mx[3] = {LLONG_MIN, LLONG_MIN, LLONG_MIN};
    bool bad = false;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double v[3] = {x[i], y[i], z[i]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            bad |= nonfinite(v[d]);
            const long long k = ord_of(v[d]);
            mn[d] = min(mn[d], k);
            mx[d] = max(mx[d], k);
        }
    }
    __shared__ long long sh[7][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long vals[7] = {mn[0], mn[1], mn[2], mx[0], mx[1], mx[2], __any_sync(0xffffffffu, bad) ? 1ll : 0ll};
#pragma unroll
    for (int q = 0; q < 7; ++q) {
        long long v = vals[q];
        for (int o = 16; o > 0; o >>= 1) {
            const long long u = __shfl_down_sync(0xffffffffu, v, o);
            v = (q < 3) ? min(v, u) : max(v, u);
        }
        if (lane == 0) sh[q][w] = v;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        const int q = threadIdx.x;
        long long v = sh[q][0];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) v = (q < 3) ? min(v, sh[q][k]) : max(v, sh[q][k]);
        part[blockIdx.x * 7 + q] = v;
    }
}

// One block of 256 threads: the g partial boxes strided over the threads, then a tree; out =
// min x, y, z, max x, y, z as doubles and 1.0 if any coordinate is not finite.
__global__ void __launch_bounds__(256) bbox_final_kernel(const long long *__restrict__ part, int g,
                                                         double *__restrict__ out) {
    __shared__ long long sh[7][8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long v[7];
#pragma unroll
    for (int q = 0; q < 7; ++q) v[q] = q < 3 ? LLONG_MAX : LLONG_MIN;
    for (int k = threadIdx.x; k < g; k += blockDim.x)
#pragma unroll
        for (int q = 0; q < 7; ++q) v[q] = q < 3 ? min(v[q], part[k * 7 + q]) : max(v[q], part[k * 7 + q]);
#pragma unroll
    for (int q = 0; q < 7; ++q) {
        for (int o = 16; o > 0; o >>= 1) {
            const long long u = __shfl_down_sync(0xffffffffu, v[q], o);
            v[q] = q < 3 ? min(v[q], u) : max(v[q], u);
        }
        if (lane == 0) sh[q][w] = v[q];
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        const int q = threadIdx.x;
        long long r = sh[q][0];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) r = q < 3 ? min(r, sh[q][k]) : max(r, sh[q][k]);
        out[q] = q < 6 ? val_of(r) : (r ? 1.0 : 0.0);
    }
}

// floor(t) and the value t - 4 * floor(t / 4) of a double t, clamped to [0, qmax], from the
// double's bits with integer operations only: a particle's cell and sub-cell come from one FMA
// per axis, and the rest of the conversion (double to integer, the remainder, the float in-cell
// coordinate) would otherwise be half a dozen more FP64-pipe instructions per axis -- the
// kernel's bound on GB300, whose FP64 rate is a small fraction of its integer rate.  The
// remainder w (quarter cells, in [0, 4) away from the grid's edges) is truncated to 24
// significant bits, an error below 1e-7 of a cell: far inside the +-1e-5 band whose pairs are
// re-tested in FP64.
__device__ __forceinline__ void quarter_split(double t, long long qmax, long long &q, float &w) {
    const long long bits = __double_as_longlong(t);
    if (bits <= 0) {   // +0.0 or negative (the sign bit makes the pattern negative)
        q = 0;
        w = 0.f;
        return;
    }
    const int e = (int)((bits >> 52) & 0x7ff) - 1023;
    const unsigned long long m = (unsigned long long)(bits & 0xfffffffffffffll) | (1ull << 52);
    if (e < 0) {   // t < 1: the float with the double's exponent and top mantissa bits
        q = 0;
        w = e + 127 > 0 ? __int_as_float(((e + 127) << 23) | (int)((m >> 29) & 0x7fffff)) : 0.f;
        return;
    }
    if (e > 52) {   // no fraction bits (cell grids beyond 2^51 quarter cells on an axis)
        const long long qq = e - 52 < 10 ? (long long)(m << (e - 52)) : LLONG_MAX;
        q = min(qq, qmax);
        w = (float)(qq - ((q >> 2) << 2));
        return;
    }
    const int sh = 52 - e;
    const long long qq = (long long)(m >> sh);
    q = min(qq, qmax);
    // remainder as a fixed-point number with sh fraction bits, then its top 24 bits as a float
    const unsigned long long v = ((unsigned long long)(qq - ((q >> 2) << 2)) << sh) | (m & ((1ull << sh) - 1));
    if (v == 0) {
        w = 0.f;
        return;
    }
    const int lz = __clzll((long long)v);
    const int fe = (63 - lz) - sh + 127;   // biased exponent of v * 2^-sh
    w = fe > 0 ? __int_as_float((fe << 23) | (int)(((v << lz) >> 40) & 0x7fffff)) : 0.f;
}

// floor(x * s4 * 2^24) + B exactly, with integer operations only (s4 = S * 2^(es - 52) a
// positive double with 53-bit mantissa S): the product of the two 53-bit mantissas as a 128-bit
// integer, shifted to 24 fraction bits and floored (towards -inf for negative x).  A map that
// is exact to 2^-24 quarter cells and monotone in x, for callers that keep |x * s4| and |B|
// below 2^37 quarter cells.
__device__ __forceinline__ long long fixed_quarter(double x, unsigned long long S, int es, long long B) {
    const long long bits = __double_as_longlong(x);
    int ex = (int)((bits >> 52) & 0x7ff);
    unsigned long long X = (unsigned long long)(bits & 0xfffffffffffffll);
    if (ex == 0)
        ex = 1;   // zero or subnormal: no implicit bit
    else
        X |= 1ull << 52;
    const unsigned long long lo = X * S, hi = __umul64hi(X, S);
    const int sh = 80 - (ex - 1023) - es;   // (X * S) * 2^-sh = x * s4 * 2^24
    unsigned long long mag;
    bool rem;
    if (sh <= 0) {   // outside the callers' range: saturate
        mag = 1ull << 62;
        rem = false;
    } else if (sh < 64) {
        mag = (hi << (64 - sh)) | (lo >> sh);
        rem = (lo & ((1ull << sh) - 1)) != 0;
    } else if (sh < 128) {
        mag = hi >> (sh - 64);
        rem = lo != 0 || (hi & ((1ull << (sh - 64)) - 1)) != 0;
    } else {
        mag = 0;
        rem = (hi | lo) != 0;
    }
    const long long p = bits < 0 ? -(long long)mag - (rem ? 1 : 0) : (long long)mag;
    return p + B;
}

// quarter_split for a fixed-point t (24 fraction bits): floor(t) clamped to [0, qmax] and the
// remainder t - 4 * floor(t / 4) as a float truncated to 24 significant bits.
__device__ __forceinline__ void quarter_split_fixed(long long t, long long qmax, long long &q, float &w) {
    if (t < 0) {
        q = 0;
        w = 0.f;
        return;
    }
    q = min(t >> 24, qmax);
    const unsigned long long v = (unsigned long long)(t - ((q >> 2) << 26));
    if (v == 0) {
        w = 0.f;
        return;
    }
    const int lz = __clzll((long long)v);
    const int fe = (63 - lz) - 24 + 127;   // biased exponent of v * 2^-24
    w = __int_as_float((fe << 23) | (int)(((v << lz) >> 40) & 0x7fffff));
}

// Sort key: row-major cell index, then (with g.sb) the particle's half-cell per axis.  The
// order of particles inside a cell does not change the partition.  The kernel also writes the
// particle's position inside its cell in units of the linking length (pre[i], in input order,
// with the index in .w), so that the sorted records are one 16-byte gather.
//
// Cell coordinates: t = 4 * (x - origin) / cell is evaluated as one FMA, x * (4 / cell) -
// origin * (4 / cell); the cell is floor(t) >> 2 and the sub-cell floor(t) & 3.  Any rounding
// here is harmless as long as it is the same for every particle: the cell side is
// ll * (1 + 2^-20), so two points within ll of each other stay in the same or adjacent cells
// whenever the cell coordinate's error is below 2^-21 cells (it is ~1e-12 cells).
//
// FIXED (plain FoF on coordinates and grids within 2^37 quarter cells): the quarter-cell
// coordinate is the exact integer map fixed_quarter instead of the FP64 FMA, so that the
// kernel issues no FP64 instruction at all (with three FMAs a particle it was FP64-bound:
// ncu showed the FP64 pipe 78 % busy).  Both maps are consistent over all particles, which is
// all the cell assignment needs; B = floor(-origin * (4 / cell) * 2^24) per axis.
template <bool FIXED>
__global__ void keys_kernel(const double *__restrict__ x, const double *__restrict__ y,
                            const double *__restrict__ z, int n, FofGeom g, SegGeom sg, long long Bx, long long By,
                            long long Bz, uint64_t *__restrict__ keys, int *__restrict__ vals,
                            float4 *__restrict__ pre) {
    const double s4 = 4.0 * g.inv_cell;   // exact: a power-of-two scaling
    const float cs4 = 0.25f * g.cs;
    const double bx0 = -g.xmin * s4, by0 = -g.ymin * s4, bz0 = -g.zmin * s4;
    const long long s4bits = __double_as_longlong(s4);
    const unsigned long long S4 = (unsigned long long)(s4bits & 0xfffffffffffffll) | (1ull << 52);
    const int es4 = (int)((s4bits >> 52) & 0x7ff) - 1023;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double bx = bx0, by = by0, bz = bz0;   // -origin * (4 / cell)
        long long x0 = 0, nx = g.ncx, ny = g.ncy, nz = g.ncz;
        if (sg.seg_of) {
            const int s = sg.seg_of[i];
            bx = -sg.smin[3 * s] * s4;
            by = -sg.smin[3 * s + 1] * s4;
            bz = -sg.smin[3 * s + 2] * s4;
            x0 = sg.scol[4 * s];
            nx = sg.scol[4 * s + 1];
            ny = sg.scol[4 * s + 2];
            nz = sg.scol[4 * s + 3];
        }
        // quarter-cell coordinates, clamped to the grid (rounding can put a point on the
        // grid's edge a hair outside it), and the position inside the cell in quarter cells
        long long qx, qy, qz;
        float wx, wy, wz;
        if (FIXED) {
            quarter_split_fixed(fixed_quarter(x[i], S4, es4, Bx), 4 * nx - 1, qx, wx);
            quarter_split_fixed(fixed_quarter(y[i], S4, es4, By), 4 * ny - 1, qy, wy);
            quarter_split_fixed(fixed_quarter(z[i], S4, es4, Bz), 4 * nz - 1, qz, wz);
        } else {
            quarter_split(fma(x[i], s4, bx), 4 * nx - 1, qx, wx);
            quarter_split(fma(y[i], s4, by), 4 * ny - 1, qy, wy);
            quarter_split(fma(z[i], s4, bz), 4 * nz - 1, qz, wz);
        }
        const long long cx = qx >> 2, cy = qy >> 2, cz = qz >> 2;
        uint64_t key = ((uint64_t)(x0 + cx) * (uint64_t)g.ky + (uint64_t)cy) * (uint64_t)g.kz + (uint64_t)cz;
        if (g.sb)
            key = (key << 3) | (uint64_t)(((qx >> 1) & 1) << 2 | ((qy >> 1) & 1) << 1 | ((qz >> 1) & 1));
        keys[i] = key;
        vals[i] = i;
        pre[i] = make_float4(wx * cs4, wy * cs4, wz * cs4, __int_as_float(i));
    }
}

// ---- cells and nodes -----------------------------------------------------------------------
// Sorted position k starts a cell when its cell key differs from its predecessor's, and a node when its
// full key does (without half-cells in the key, every particle is a node).  A warp numbers kScanRun
// consecutive positions with ballots; head_count_kernel leaves cells << 32 | nodes per warp, whose
// exclusive scan is where head_apply_kernel's warp starts.  Together with the scan they take 0.50 ms at 2e7 particles,
// where eight passes (records and run heads, two scans, run joins, cell table, one-component flags) took 0.83.
constexpr int kScanRun = 512;

struct Heads {
    bool cell, node;
};

__device__ __forceinline__ Heads heads_at(const uint64_t *__restrict__ keys, int sb, int k, int n) {
    Heads h{false, false};
    if (k < n) {
        const uint64_t full = keys[k], prev = k > 0 ? keys[k - 1] : ~full;
        h.cell = (prev >> sb) != (full >> sb);
        h.node = sb == 0 || prev != full;
    }
    return h;
}

__global__ void __launch_bounds__(256) head_count_kernel(int n, int sb, const uint64_t *__restrict__ keys,
                                                         int64_t *__restrict__ counts, int nruns,
                                                         int *__restrict__ all_cells) {
    __shared__ int block_cells;
    if (threadIdx.x == 0) block_cells = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int run = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (run < nruns) {
        int cells = 0, nodes = 0;
#pragma unroll 4
        for (int r = 0; r < kScanRun; r += 32) {
            const Heads h = heads_at(keys, sb, run * kScanRun + r + lane, n);
            cells += __popc(__ballot_sync(0xffffffffu, h.cell));
            nodes += __popc(__ballot_sync(0xffffffffu, h.node));
        }
        if (lane == 0) {
            counts[run] = (int64_t)cells << 32 | nodes;
            atomicAdd(&block_cells, cells);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(all_cells, block_cells);
}

// Node m: first sorted position node_start[m], cell node_cell[m], first particle's record
// node_rec[m], half-cell node_sub[m], union-find parent and smallest original
// index (the sort is stable, so the first particle's).  Cell c: first node cell_node[c], key cell_key[c].
// The entries past the last node and cell close the ranges; cnt[0] = cells, cnt[1] = nodes.
__global__ void __launch_bounds__(256) head_apply_kernel(
    int n, int sb, const uint64_t *__restrict__ keys, const int *__restrict__ idx, const float4 *__restrict__ pre,
    const int64_t *__restrict__ base, int nruns, float4 *__restrict__ rec, int *__restrict__ node_of,
    int *__restrict__ node_start, int *__restrict__ node_cell, unsigned char *__restrict__ node_sub,
    float4 *__restrict__ node_rec, int *__restrict__ parent, int *__restrict__ minidx,
    unsigned char *__restrict__ multi, int *__restrict__ cell_node, uint64_t *__restrict__ cell_key,
    int *__restrict__ cnt) {
    const int lane = threadIdx.x & 31;
    const unsigned upto = 0xffffffffu >> (31 - lane);
    const int run = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (run >= nruns) return;
    int cells = (int)(base[run] >> 32), nodes = (int)(base[run] & 0xffffffffll);
#pragma unroll 2
    for (int r = 0; r < kScanRun; r += 32) {
        const int k = run * kScanRun + r + lane;
        const Heads h = heads_at(keys, sb, k, n);
        const unsigned cb = __ballot_sync(0xffffffffu, h.cell), nb = __ballot_sync(0xffffffffu, h.node);
        if (k < n) {
            const int i = idx[k];
            const int m = nodes + __popc(nb & upto) - 1;
            const float4 r = pre[i];
            rec[k] = r;
            node_of[k] = m;
            if (h.node) {
                node_rec[m] = r;
                node_start[m] = k;
                node_cell[m] = cells + __popc(cb & upto) - 1;
                node_sub[m] = sb ? (unsigned char)(keys[k] & 7) : 0;
                parent[m] = m;
                minidx[m] = i;
                multi[m] = 0;
            }
            if (h.cell) {
                const int c = cells + __popc(cb & upto) - 1;
                cell_node[c] = m;
                cell_key[c] = keys[k] >> sb;
            }
        }
        cells += __popc(cb);
        nodes += __popc(nb);
    }
    if (run == nruns - 1 && lane == 0) {
        cnt[0] = cells;
        cnt[1] = nodes;
        cell_node[cells] = nodes;
        node_start[nodes] = n;
    }
}

// scipy's p = 2 distance: ((dx*dx + dy*dy) + dz*dz) <= r*r, each operation rounded
__device__ __forceinline__ bool exact_pair(double xi, double yi, double zi, double xj, double yj, double zj, double r2) {
    const double dx = __dsub_rn(xi, xj);
    const double dy = __dsub_rn(yi, yj);
    const double dz = __dsub_rn(zi, zj);
    double s = __dmul_rn(dx, dx);
    s = __dadd_rn(s, __dmul_rn(dy, dy));
    s = __dadd_rn(s, __dmul_rn(dz, dz));
    return s <= r2;
}

__device__ __forceinline__ bool exact_link(const double *__restrict__ x, const double *__restrict__ y,
                                           const double *__restrict__ z, int i, int j, double r2) {
    return exact_pair(x[i], y[i], z[i], x[j], y[j], z[j], r2);
}

// Lower bound of q in the sorted keys[lo, n), searched forward from lo: doubling steps, then
// bisection of the last step.
__device__ __forceinline__ int gallop_lower_bound(const uint64_t *__restrict__ keys, int lo, int n, uint64_t q) {
    if (lo >= n || keys[lo] >= q) return lo;
    int prev = lo;   // keys[prev] < q
    long long cur = (long long)lo + 1, step = 1;
    while (cur < n && keys[cur] < q) {
        prev = (int)cur;
        step <<= 1;
        cur = prev + step;
    }
    int a = prev + 1, b = (int)(cur < n ? cur : n);
    while (a < b) {
        const int mid = (a + b) >> 1;
        if (keys[mid] < q) a = mid + 1;
        else b = mid;
    }
    return a;
}

// The pairs of cells, listed per cell: the cell itself when it holds more than one node, and its occupied forward
// neighbours, one thread per cell.  On the padded key grid a neighbour's key is the cell's key plus
// a constant, so (0, 0, +1) is the next cell or none, and for each of the stencil's four columns (0, 1),
// (1, -1), (1, 0), (1, 1), whose bases increase, one lower bound of the column's z - 1 key -- galloping
// forward from the cell itself, then from the previous column's bound -- gives its three z
// neighbours in order.  A cell's entries are together, in key order: cell_list[c] = first << 4 | count; the
// order of the cells in the list does not matter.  (A table row of 13 entries per cell,
// mostly empty, took 0.68 ms at 2e7 particles.)
// With half-cells an entry is the second cell's nodes as the linking kernels read them: first node, and nodes - 1
// (at most 7) in bits 0-2, the cell's offset in bits 3-7 (see entry_offset), bit 8 for the cell itself.  Without,
// it is the two cells.
template <bool NODES>
__global__ void __launch_bounds__(256) cell_pair_kernel(const int *__restrict__ cnt, const int *__restrict__ cell_node,
                                                        const uint64_t *__restrict__ cell_key, long long ky, long long kz,
                                                        int2 *__restrict__ pairs, long long *__restrict__ cell_list,
                                                        unsigned long long *__restrict__ npairs) {
    const int nc = cnt[0];
    const int lane = threadIdx.x & 31;
    const uint64_t zrow = (uint64_t)kz, slab = (uint64_t)ky * (uint64_t)kz;
    for (int64_t c0 = blockIdx.x * (int64_t)blockDim.x; c0 < nc; c0 += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(c0 + threadIdx.x);
        int at[4] = {0, 0, 0, 0}, occ = 0;   // first cell of each column, occupied neighbours as a mask
        if (c < nc) {
            const uint64_t key = cell_key[c];
            if (cell_node[c + 1] - cell_node[c] > 1) occ = 1;
            if (c + 1 < nc && cell_key[c + 1] == key + 1) occ |= 2;
            const uint64_t base[4] = {key + zrow, key + slab - zrow, key + slab, key + slab + zrow};
            int lb = c + 1;
#pragma unroll
            for (int col = 0; col < 4; ++col) {
                lb = gallop_lower_bound(cell_key, lb, nc, base[col] - 1);
                at[col] = lb;
                int q = lb;
#pragma unroll
                for (int dz = 0; dz < 3; ++dz)
                    if (q < nc && cell_key[q] == base[col] - 1 + (uint64_t)dz) {
                        occ |= 4 << (3 * col + dz);
                        ++q;
                    }
            }
        }
        const int mine = __popc(occ);
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        unsigned long long w = 0;
        if (lane == 31 && incl > 0) w = atomicAdd(npairs, (unsigned long long)incl);
        w = __shfl_sync(0xffffffffu, w, 31) + (unsigned long long)(incl - mine);
        auto put = [&](int d, int ox, int oy, int oz) {
            if (NODES) {
                const int t0 = cell_node[d];
                pairs[w++] = make_int2(t0, (cell_node[d + 1] - t0 - 1) | ox << 3 | (oy + 1) << 4 | (oz + 1) << 6 |
                                               (d == c ? 1 << 8 : 0));
            } else {
                pairs[w++] = make_int2(c, d);
            }
        };
        if (c < nc) cell_list[c] = (long long)w << 4 | mine;
        if (occ & 1) put(c, 0, 0, 0);
        if (occ & 2) put(c + 1, 0, 0, 1);
#pragma unroll
        for (int col = 0; col < 4; ++col) {
            int q = at[col];
#pragma unroll
            for (int dz = 0; dz < 3; ++dz)
                if (occ & (4 << (3 * col + dz))) put(q++, col > 0 ? 1 : 0, col == 0 ? 1 : col - 2, dz - 1);
        }
    }
}

__device__ __forceinline__ int3 entry_offset(int e) {
    return make_int3((e >> 3) & 1, ((e >> 4) & 3) - 1, ((e >> 6) & 3) - 1);
}

// Offset of cell d (key kd) from cell c (key kc <= kd), per axis; d is c or one of its forward neighbours.
__device__ __forceinline__ int3 cell_offset(uint64_t kc, uint64_t kd, long long ky, long long kz) {
    const long long d = (long long)(kd - kc), slab = ky * kz;
    int3 o;
    o.x = d >= slab - kz - 1 && slab > 1 ? 1 : 0;
    long long r = d - (o.x ? slab : 0);             // dy * kz + dz
    o.y = r > 1 ? 1 : (r < -1 ? -1 : 0);
    o.z = (int)(r - (long long)o.y * kz);
    return o;
}

// A list entry for the blocks: sorted positions [a, a + na) against [b, b + nb), cell b shifted by off (2 bits
// an axis, offset + 1); without shift and with a == b, pairs j > i of one range.
struct __align__(8) HeavyPair {
    int a, na, b, nb, off, pad;
};

// Tests that one pair of nodes gets from a lane: all when they are at most kLaneTests, else a glance, and a warp goes on with
// what is open (up to kWarpTests; kWarpPairs pairs of particles, when they are the nodes, as each may be a union), and
// a block with the rest.  With 1,024 from a lane and the others from a block, crowded nodes kept one lane of a warp at
// work: 2e5 particles in clumps of 200 a twentieth of the linking length wide took 1.99 ms, now 0.34.
constexpr int kLaneTests = 64, kLaneGlance = 8, kWarpTests = 1 << 15, kWarpPairs = 1 << 12;
constexpr int kHookLinks = 2, kHookTests = 16;   // links and candidates of a node in hook_kernel

struct LinkArgs {
    const int *cnt;                 // [0] cells [1] nodes
    const int2 *pairs;
    const unsigned long long *npairs;
    const long long *cell_list;
    const int *cell_node, *node_start, *node_cell;
    const unsigned char *node_sub;
    const uint64_t *cell_key;
    const float4 *rec, *node_rec;
    const double *x, *y, *z;
    int *parent, *err;
    unsigned long long *crowd;      // pairs left to a warp each: nodes h << 32 | t, or the place of a pair of cells
    unsigned long long *ncrowd;
    int crowd_cap;
    HeavyPair *heavy;
    int *nheavy;
    int heavy_cap;
};

// The half-cells of a cell at offset o that can hold a friend of half-cell hs: half-cell offsets reach 3 only
// between the far halves of neighbouring cells, which are more than ll apart.  near(ts) below.
struct NearHalves {
    int up, dn;
    __device__ __forceinline__ NearHalves(int3 o, int hs) {
        const int plus = (o.x > 0 ? 4 : 0) | (o.y > 0 ? 2 : 0) | (o.z > 0 ? 1 : 0);
        const int minus = (o.x < 0 ? 4 : 0) | (o.y < 0 ? 2 : 0) | (o.z < 0 ? 1 : 0);
        up = plus & ~hs;
        dn = minus & hs;
    }
    __device__ __forceinline__ bool near(int ts) const { return !((ts & up) | (~ts & dn)); }
};

// First link between the particles of two nodes (q shifted into p's frame): 1, 0 for none, -1 when the budget
// of tests (left, lowered by those made) ran out before it was decided.
__device__ __forceinline__ int node_link(const LinkArgs &A, const FofGeom &g, int p0, int p1, int q0, int q1, float sx,
                                         float sy, float sz, int &left) {
    for (int p = p0; p < p1; ++p) {
        const float4 a = A.rec[p];
        for (int q = q0; q < q1; ++q) {
            if (left == 0) return -1;
            --left;
            const float4 b = A.rec[q];
            const float dx = (b.x + sx) - a.x, dy = (b.y + sy) - a.y, dz = (b.z + sz) - a.z;
            const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            if (d2 <= g.hi &&
                (d2 < g.lo || exact_link(A.x, A.y, A.z, __float_as_int(a.w), __float_as_int(b.w), g.r2)))
                return 1;
        }
    }
    return 0;
}

// A warp's pairs (of the lanes with one) to the list for warps; false for those that find it full.
__device__ __forceinline__ bool push_crowd_warp(const LinkArgs &A, bool mine, unsigned long long pr, int lane) {
    const unsigned who = __ballot_sync(0xffffffffu, mine);
    if (!who) return false;
    unsigned long long first = 0;
    if (lane == __ffs(who) - 1) first = atomicAdd(A.ncrowd, (unsigned long long)__popc(who));
    const unsigned long long k = __shfl_sync(0xffffffffu, first, __ffs(who) - 1) + __popc(who & ((1u << lane) - 1u));
    if (!mine || k >= (unsigned long long)A.crowd_cap) return false;
    A.crowd[k] = pr;
    return true;
}

__device__ __forceinline__ bool push_heavy(const LinkArgs &A, int a, int na, int b, int nb, int3 o) {
    const int k = atomicAdd(A.nheavy, 1);
    if (k >= A.heavy_cap) return false;
    A.heavy[k] = HeavyPair{a, na, b, nb, (o.x + 1) | (o.y + 1) << 2 | (o.z + 1) << 4, 0};
    return true;
}

// One thread per node: joins it with the first kHookLinks nodes ahead of it (its cell's, then the forward
// neighbours' in key order) whose first particle is a friend of its own first particle, of at most
// kHookTests nodes looked at.
// Bound, as the whole linking: the latency of dependent loads, hidden by many threads, as long as a warp's lanes
// stay in step.  So a candidate is one 16-byte record, and the joins come after the search, one step of all
// lanes' walks at a time: 0.077 ms at 2e6 and 0.58 ms at 2e7 particles.  With the joins made where they were
// found it took 0.23 and 2.4 ms; all pairs of a cell pair in one thread, find by find, 4.3 and 37 ms.
__global__ void __launch_bounds__(256) hook_kernel(LinkArgs A, FofGeom g) {
    const int nn = A.cnt[1];
    for (int64_t v0 = blockIdx.x * (int64_t)blockDim.x; v0 < nn; v0 += (int64_t)gridDim.x * blockDim.x) {
        const bool in = v0 + threadIdx.x < nn;
        const int h = (int)(in ? v0 + threadIdx.x : nn - 1);
        const long long range = in ? A.cell_list[A.node_cell[h]] : 0;
        const int2 *list = A.pairs + (range >> 4), *end = list + (range & 15);
        const float4 a = A.node_rec[h];
        int found[kHookLinks] = {0, 0}, links = 0, looked = 0;
        bool more = list != end;
        while (__any_sync(0xffffffffu, more)) {
            if (!more) continue;
            const int2 e = *list++;
            const int3 o = entry_offset(e.y);
            const int t0 = e.y >> 8 ? h + 1 : e.x, t1 = e.x + (e.y & 7) + 1;
            const float sx = (float)o.x * g.cs - a.x, sy = (float)o.y * g.cs - a.y, sz = (float)o.z * g.cs - a.z;
            for (int t = t0; t < t1 && links < kHookLinks; ++t) {
                const float4 b = A.node_rec[t];
                const float dx = b.x + sx, dy = b.y + sy, dz = b.z + sz;
                if (fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < g.lo) {   // the band is left to the sweep
                    if (links == 0) found[0] = t;
                    else found[1] = t;
                    ++links;
                }
            }
            looked += t1 - t0;
            more = list != end && links < kHookLinks && looked < kHookTests;
        }
        const int r = uf_union_warp(A.parent, h, links > 0 ? found[0] : h, links > 0, A.err);
        uf_union_warp(A.parent, links > 1 ? r : h, links > 1 ? found[1] : h, links > 1, A.err);
    }
}

// Roots as they are after hook_kernel, for the sweep (in an array of their own, see root_kernel).
__global__ void __launch_bounds__(256) flatten_kernel(const int *__restrict__ cnt, int *parent, int *__restrict__ root,
                                                      int *err) {
    const int nn = cnt[1];
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nn; k += (int64_t)gridDim.x * blockDim.x)
        root[k] = uf_find(parent, (int)k, err);
}

// Whether two nodes are in different sets (of roots rh and rt) and linked, by one lane: 1, 0, or -1 when there are too many
// tests for it.
__device__ __forceinline__ int nodes_linked(const LinkArgs &A, const FofGeom &g, int h, int t, int3 o, int &rh, int &rt) {
    rh = uf_find(A.parent, h, A.err);
    rt = uf_find(A.parent, t, A.err);
    if (rh == rt) return 0;
    const int p0 = A.node_start[h], p1 = A.node_start[h + 1], q0 = A.node_start[t], q1 = A.node_start[t + 1];
    int left = (long long)(p1 - p0) * (q1 - q0) <= kLaneTests ? kLaneTests : kLaneGlance;
    return node_link(A, g, p0, p1, q0, q1, (float)o.x * g.cs, (float)o.y * g.cs, (float)o.z * g.cs, left);
}

// The same where no warp is at hand: what a lane leaves open goes to the list for warps, or is decided row by row when that
// is full.
__device__ __forceinline__ void link_nodes(const LinkArgs &A, const FofGeom &g, int h, int t, int3 o) {
    int rh, rt;
    int hit = nodes_linked(A, g, h, t, o, rh, rt);
    if (hit < 0) {
        const int p0 = A.node_start[h], p1 = A.node_start[h + 1], q0 = A.node_start[t], q1 = A.node_start[t + 1];
        const unsigned long long k = atomicAdd(A.ncrowd, 1ull);
        if (k < (unsigned long long)A.crowd_cap) {
            A.crowd[k] = (unsigned long long)h << 32 | (unsigned)t;
            return;
        }
        for (int p = p0; p < p1 && hit <= 0; ++p) {
            int left = q1 - q0;
            hit = node_link(A, g, p, p + 1, q0, q1, (float)o.x * g.cs, (float)o.y * g.cs, (float)o.z * g.cs, left);
        }
    }
    if (hit > 0) uf_union(A.parent, rh, rt, A.err);
}

// A box in a cell's coordinates, and the squared distance of a point from it.
struct Box {
    float lo[3], hi[3];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            lo[d] = INFINITY;
            hi[d] = -INFINITY;
        }
    }
    __device__ __forceinline__ void add(float x, float y, float z) {
        const float v[3] = {x, y, z};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            lo[d] = fminf(lo[d], v[d]);
            hi[d] = fmaxf(hi[d], v[d]);
        }
    }
    __device__ __forceinline__ void join(const Box &b) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            lo[d] = fminf(lo[d], b.lo[d]);
            hi[d] = fmaxf(hi[d], b.hi[d]);
        }
    }
    __device__ __forceinline__ void warp_join() {
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int k = 16; k > 0; k >>= 1) {
                lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], k));
                hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], k));
            }
    }
    __device__ __forceinline__ float d2(float x, float y, float z) const {
        const float v[3] = {x, y, z};
        float s = 0.f;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float e = fmaxf(fmaxf(lo[d] - v[d], v[d] - hi[d]), 0.f);
            s = fmaf(e, e, s);
        }
        return s;
    }
};

// Whether two nodes are linked, by a warp: the particles of the larger a lane each, 32 at a time, against those of the smaller,
// one after another; of many, only those near the smaller's box.
__device__ __forceinline__ bool warp_nodes_linked(const LinkArgs &A, const FofGeom &g, int h, int t, int3 o, int lane) {
    int a0 = A.node_start[h], na = A.node_start[h + 1] - a0, b0 = A.node_start[t], nb = A.node_start[t + 1] - b0;
    float sx = (float)o.x * g.cs, sy = (float)o.y * g.cs, sz = (float)o.z * g.cs;   // added to b's coordinates
    if (nb > na) {
        const int s0 = a0, sn = na;
        a0 = b0;
        na = nb;
        b0 = s0;
        nb = sn;
        sx = -sx;
        sy = -sy;
        sz = -sz;
    }
    const bool boxed = (long long)na * nb > 1024;
    Box box;
    box.clear();
    if (boxed) {
        for (int k = lane; k < nb; k += 32) {
            const float4 b = A.rec[b0 + k];
            box.add(b.x + sx, b.y + sy, b.z + sz);
        }
        box.warp_join();
    }
    for (int k0 = 0; k0 < na; k0 += 32) {
        bool in = k0 + lane < na, known = false;
        const float4 a = A.rec[a0 + min(k0 + lane, na - 1)];
        if (boxed) in = in && box.d2(a.x, a.y, a.z) <= g.hi;
        if (!__any_sync(0xffffffffu, in)) continue;
        const float ax = a.x - sx, ay = a.y - sy, az = a.z - sz;
        double ex = 0.0, ey = 0.0, ez = 0.0;   // the position for exact tests, read at the first of them
        for (int q0 = 0; q0 < nb; q0 += 4) {
            bool hit = false;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float4 b = A.rec[b0 + min(q0 + u, nb - 1)];
                const float dx = b.x - ax, dy = b.y - ay, dz = b.z - az;
                const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                if (!(in && d2 <= g.hi)) continue;
                if (d2 < g.lo) {
                    hit = true;
                    continue;
                }
                if (!known) {
                    const int i = __float_as_int(a.w);
                    ex = A.x[i];
                    ey = A.y[i];
                    ez = A.z[i];
                    known = true;
                }
                const int j = __float_as_int(b.w);
                hit |= exact_pair(ex, ey, ez, A.x[j], A.y[j], A.z[j], g.r2);
            }
            if (__any_sync(0xffffffffu, hit)) return true;
        }
    }
    return false;
}

// One thread per node: the pairs with nodes ahead of it that are near enough and whose roots differ, to the list
// as h << 32 | t (tested in place when the list is full).  The block's pairs are gathered in shared memory, so
// that it takes its place in the list with one atomic.
constexpr int kSweepBuf = 1024;

__global__ void __launch_bounds__(256) sweep_kernel(LinkArgs A, FofGeom g, const int *__restrict__ root,
                                                    unsigned long long *__restrict__ list, long long cap,
                                                    unsigned long long *__restrict__ nlist) {
    __shared__ unsigned long long buf[kSweepBuf], place;
    __shared__ int nbuf;
    const int nn = A.cnt[1];
    for (int64_t v0 = blockIdx.x * (int64_t)blockDim.x; v0 < nn; v0 += (int64_t)gridDim.x * blockDim.x) {
        if (threadIdx.x == 0) nbuf = 0;
        __syncthreads();
        const int64_t v = v0 + threadIdx.x;
        if (v < nn) {
            const int h = (int)v;
            const long long range = A.cell_list[A.node_cell[h]];
            const int2 *ent = A.pairs + (range >> 4), *end = ent + (range & 15);
            const int rh = root[h], hs = A.node_sub[h];
            for (; ent != end; ++ent) {
                const int2 e = *ent;
                const int t0 = e.y >> 8 ? h + 1 : e.x, t1 = e.x + (e.y & 7) + 1;
                unsigned other = 0;   // nodes of the entry in another set
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (t0 + j < t1 && root[t0 + j] != rh) other |= 1u << j;
                if (!other) continue;
                const int3 o = entry_offset(e.y);
                const NearHalves halves(o, hs);
                for (; other; other &= other - 1) {
                    const int t = t0 + __ffs(other) - 1;
                    if (!halves.near(A.node_sub[t])) continue;
                    const unsigned long long pr = (unsigned long long)h << 32 | (unsigned)t;
                    const int k = atomicAdd(&nbuf, 1);
                    if (k < kSweepBuf) {
                        buf[k] = pr;
                    } else {
                        const unsigned long long q = atomicAdd(nlist, 1ull);
                        if ((long long)q < cap) list[q] = pr;
                        else link_nodes(A, g, h, t, o);
                    }
                }
            }
        }
        __syncthreads();
        const int m = min(nbuf, kSweepBuf);
        if (threadIdx.x == 0 && m > 0) place = atomicAdd(nlist, (unsigned long long)m);
        __syncthreads();
        for (int k = threadIdx.x; k < m; k += blockDim.x) {
            const unsigned long long q = place + k;
            if ((long long)q < cap) {
                list[q] = buf[k];
            } else {
                const int h = (int)(buf[k] >> 32), t = (int)(buf[k] & 0xffffffffu);
                link_nodes(A, g, h, t, cell_offset(A.cell_key[A.node_cell[h]], A.cell_key[A.node_cell[t]], g.ky, g.kz));
            }
        }
        __syncthreads();   // the buffer is reused
    }
}

// A pair of nodes by a warp, or the largest listed for a block: whether they are linked.
__device__ __forceinline__ bool warp_decides(const LinkArgs &A, const FofGeom &g, int h, int t, int lane) {
    const int3 o = cell_offset(A.cell_key[A.node_cell[h]], A.cell_key[A.node_cell[t]], g.ky, g.kz);
    const int p0 = A.node_start[h], np = A.node_start[h + 1] - p0, q0 = A.node_start[t], nq = A.node_start[t + 1] - q0;
    if ((long long)np * nq > kWarpTests) {
        bool listed = false;
        if (lane == 0) listed = push_heavy(A, p0, np, q0, nq, o);
        if (__shfl_sync(0xffffffffu, listed, 0)) return false;
    }
    return warp_nodes_linked(A, g, h, t, o, lane);
}

// One lane per listed pair of nodes; the pairs that it leaves open go to the list for warps (its own, when that is full).
__global__ void __launch_bounds__(256) link_kernel(LinkArgs A, FofGeom g, const unsigned long long *__restrict__ list,
                                                   long long cap, const unsigned long long *__restrict__ nlist) {
    const int lane = threadIdx.x & 31;
    const long long nl = (long long)*nlist < cap ? (long long)*nlist : cap;
    for (long long k0 = blockIdx.x * (long long)blockDim.x; k0 < nl; k0 += (long long)gridDim.x * blockDim.x) {
        const long long k = k0 + threadIdx.x;
        const unsigned long long pr = k < nl ? list[k] : 0;
        const int h = (int)(pr >> 32), t = (int)(pr & 0xffffffffu);
        int rh = 0, rt = 0, hit = 0;
        if (k < nl) {
            const int3 o = cell_offset(A.cell_key[A.node_cell[h]], A.cell_key[A.node_cell[t]], g.ky, g.kz);
            hit = nodes_linked(A, g, h, t, o, rh, rt);
        }
        if (push_crowd_warp(A, hit < 0, pr, lane)) hit = 0;
        for (unsigned todo = __ballot_sync(0xffffffffu, hit < 0); todo; todo &= todo - 1) {
            const int l = __ffs(todo) - 1;
            const bool linked = warp_decides(A, g, __shfl_sync(0xffffffffu, h, l), __shfl_sync(0xffffffffu, t, l), lane);
            if (lane == l) hit = linked;
        }
        uf_union_warp(A.parent, rh, rt, hit > 0, A.err);
    }
}

// Particles as nodes: the pairs of two cells' particles (of one, when they are the same) by a warp, a first particle a lane.
__device__ __forceinline__ void warp_join_particles(const LinkArgs &A, const FofGeom &g, int h0, int h1, int t0, int t1,
                                                    int3 o, bool same, int lane) {
    const float sx = (float)o.x * g.cs, sy = (float)o.y * g.cs, sz = (float)o.z * g.cs;
    for (int k0 = h0; k0 < h1; k0 += 32) {
        const int p = min(k0 + lane, h1 - 1);
        const float4 a = A.rec[p];
        int rp = uf_find(A.parent, p, A.err);
        for (int q = same ? k0 + 1 : t0; q < t1; ++q) {
            const float4 b = A.rec[q];
            const float dx = (b.x + sx) - a.x, dy = (b.y + sy) - a.y, dz = (b.z + sz) - a.z;
            const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            bool join = k0 + lane < h1 && (!same || q > p) && d2 <= g.hi;
            if (!__any_sync(0xffffffffu, join)) continue;
            const int rq = uf_find(A.parent, q, A.err);
            join = join && rq != rp &&
                   (d2 < g.lo || exact_link(A.x, A.y, A.z, __float_as_int(a.w), __float_as_int(b.w), g.r2));
            const int r = uf_union_warp(A.parent, rp, rq, join, A.err);
            if (join) rp = r;
        }
    }
}

// Particles as nodes: each joined with the first of the next kHookTests particles of its cell that it is linked to, which
// leaves most of a crowded cell in one set (1e5 particles in some 30 cells of such a grid: 8 to 11 ms without, 1 to 2 so).
__global__ void __launch_bounds__(256) hook_particles_kernel(LinkArgs A, FofGeom g) {
    const int nn = A.cnt[1];
    for (int64_t v0 = blockIdx.x * (int64_t)blockDim.x; v0 < nn; v0 += (int64_t)gridDim.x * blockDim.x) {
        const bool in = v0 + threadIdx.x < nn;
        const int h = (int)(in ? v0 + threadIdx.x : nn - 1);
        const int end = min(A.cell_node[A.node_cell[h] + 1], h + 1 + kHookTests);
        int found = -1;
        if (in && end > h + 1) {
            const float4 a = A.rec[h];
            for (int t = h + 1; t < end && found < 0; ++t) {
                const float4 b = A.rec[t];
                const float dx = b.x - a.x, dy = b.y - a.y, dz = b.z - a.z;
                const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                if (d2 <= g.hi &&
                    (d2 < g.lo || exact_link(A.x, A.y, A.z, __float_as_int(a.w), __float_as_int(b.w), g.r2)))
                    found = t;
            }
        }
        uf_union_warp(A.parent, h, found >= 0 ? found : h, found >= 0, A.err);
    }
}

// A pair of cells' particles by a warp, or listed for a block.
__device__ __forceinline__ void warp_joins_cells(const LinkArgs &A, const FofGeom &g, int2 pr, int lane) {
    const int h0 = A.cell_node[pr.x], h1 = A.cell_node[pr.x + 1], t0 = A.cell_node[pr.y], t1 = A.cell_node[pr.y + 1];
    const int3 o = pr.x == pr.y ? make_int3(0, 0, 0) : cell_offset(A.cell_key[pr.x], A.cell_key[pr.y], g.ky, g.kz);
    if ((long long)(h1 - h0) * (t1 - t0) > kWarpPairs) {
        bool listed = false;
        if (lane == 0) listed = push_heavy(A, h0, h1 - h0, t0, t1 - t0, o);
        if (__shfl_sync(0xffffffffu, listed, 0)) return;
    }
    warp_join_particles(A, g, h0, h1, t0, t1, o, pr.x == pr.y, lane);
}

// Particles as nodes (coincident points only, or no room for half-cells in the key): one lane per cell pair
// tests all its particles; pairs with more than kLaneTests go to the list for warps.
__global__ void __launch_bounds__(256) link_particles_kernel(LinkArgs A, FofGeom g) {
    const int lane = threadIdx.x & 31;
    const long long np = (long long)*A.npairs;
    for (long long w0 = blockIdx.x * (long long)blockDim.x; w0 < np; w0 += (long long)gridDim.x * blockDim.x) {
        const long long w = w0 + threadIdx.x;
        const int2 pr = w < np ? A.pairs[w] : make_int2(0, 0);
        bool many = false;
        if (w < np) {
            const bool same = pr.x == pr.y;
            const int h0 = A.cell_node[pr.x], h1 = A.cell_node[pr.x + 1], t0 = A.cell_node[pr.y], t1 = A.cell_node[pr.y + 1];
            many = (long long)(h1 - h0) * (t1 - t0) > kLaneTests;
            if (!many) {
                int3 o = make_int3(0, 0, 0);
                if (!same) o = cell_offset(A.cell_key[pr.x], A.cell_key[pr.y], g.ky, g.kz);
                for (int h = h0; h < h1; ++h)
                    for (int t = same ? h + 1 : t0; t < t1; ++t) link_nodes(A, g, h, t, o);
            }
        }
        __syncwarp();
        if (push_crowd_warp(A, many, (unsigned long long)w, lane)) many = false;
        for (unsigned todo = __ballot_sync(0xffffffffu, many); todo; todo &= todo - 1) {
            const int l = __ffs(todo) - 1;
            warp_joins_cells(A, g, make_int2(__shfl_sync(0xffffffffu, pr.x, l), __shfl_sync(0xffffffffu, pr.y, l)), lane);
        }
    }
}

// One warp per pair on the list for warps.
__global__ void __launch_bounds__(256) crowd_kernel(LinkArgs A, FofGeom g, int nodes) {
    const int lane = threadIdx.x & 31;
    const int n = (int)min(*A.ncrowd, (unsigned long long)A.crowd_cap);
    for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < n; k += (gridDim.x * blockDim.x) >> 5) {
        const unsigned long long pr = A.crowd[k];
        if (nodes) {
            const int h = (int)(pr >> 32), t = (int)(pr & 0xffffffffu);
            const int rh = uf_find(A.parent, h, A.err), rt = uf_find(A.parent, t, A.err);
            // the lanes may have walked to different ancestors: one lane's word decides
            if (__shfl_sync(0xffffffffu, rh == rt, 0)) continue;
            const bool linked = warp_decides(A, g, h, t, lane);
            if (lane == 0 && linked) uf_union(A.parent, rh, rt, A.err);
            __syncwarp();
        } else {
            warp_joins_cells(A, g, A.pairs[pr], lane);
        }
    }
}

// The list's entries: tiles of 256 x 256 particles, an entry of more than kHuge tiles spread over all blocks, the
// others one block each.  A thread holds one particle of the first range; those of the second range that lie near the first
// one's box are staged in shared memory with their roots, and a thread looks at them when its particle lies near
// theirs.  Two nodes (nodes) are done with their first link: a tile of theirs starts with a look at their roots, and the
// block stops when one of its threads finds a link.  Particles as nodes are joined one by one; candidates already in the thread's
// set need no test.
// Two sheets of 5e5 particles 1.3 linking lengths apart, one pair of nodes: 285 ms with every pair of particles tested, now 22.
constexpr int kHuge = 64;

__device__ __forceinline__ Box block_box(Box box, Box *sh, int lane, int w) {
    box.warp_join();
    if (lane == 0) sh[w] = box;
    __syncthreads();
    Box all = sh[0];
    for (int k = 1; k < 8; ++k) all.join(sh[k]);
    __syncthreads();   // sh is reused
    return all;
}

__global__ void __launch_bounds__(256) heavy_kernel(LinkArgs A, FofGeom g, const int *__restrict__ node_of, int nodes) {
    __shared__ float4 qrec[256];
    __shared__ int qroot[256], qat[256], wcnt[8];
    __shared__ Box boxes[8];
    __shared__ volatile int done;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int ne = min(*A.nheavy, A.heavy_cap);
    for (int e = 0; e < ne; ++e) {
        const HeavyPair hp = A.heavy[e];
        const long long ta = (hp.na + 255) / 256, tb = (hp.nb + 255) / 256, tiles = ta * tb;
        const bool huge = tiles > kHuge;
        if (!huge && e % (int)gridDim.x != (int)blockIdx.x) continue;
        const bool same = hp.a == hp.b;
        const float sx = (float)((hp.off & 3) - 1) * g.cs, sy = (float)(((hp.off >> 2) & 3) - 1) * g.cs,
                    sz = (float)(((hp.off >> 4) & 3) - 1) * g.cs;
        const int node_a = node_of[hp.a], node_b = node_of[hp.b];
        for (long long tile = huge ? blockIdx.x : 0; tile < tiles; tile += huge ? gridDim.x : 1) {
            const int p = hp.a + (int)(tile / tb) * 256 + threadIdx.x;
            const int q = hp.b + (int)(tile % tb) * 256 + threadIdx.x;
            const bool pv = p < hp.a + hp.na, qv = q < hp.b + hp.nb;
            if (nodes) {
                if (threadIdx.x == 0)
                    done = uf_find(A.parent, node_a, A.err) == uf_find(A.parent, node_b, A.err);
                __syncthreads();
                const bool joined = done != 0;
                __syncthreads();   // every thread has read it before it is written again
                if (joined) break;
            }
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
            Box box;
            box.clear();
            if (pv) {
                a = A.rec[p];
                box.add(a.x, a.y, a.z);
            }
            const Box abox = block_box(box, boxes, lane, w);
            bool keep = false;
            if (qv) {
                b = A.rec[q];
                b.x += sx;
                b.y += sy;
                b.z += sz;
                keep = abox.d2(b.x, b.y, b.z) <= g.hi;
            }
            const unsigned kept = __ballot_sync(0xffffffffu, keep);
            if (lane == 0) wcnt[w] = __popc(kept);
            box.clear();
            if (keep) box.add(b.x, b.y, b.z);
            const Box bbox = block_box(box, boxes, lane, w);   // its barriers publish wcnt
            int at = __popc(kept & ((1u << lane) - 1u)), cnt = 0;
            for (int k = 0; k < 8; ++k) {
                if (k < w) at += wcnt[k];
                cnt += wcnt[k];
            }
            if (keep) {
                qrec[at] = b;
                qat[at] = q;
                qroot[at] = nodes ? node_b : uf_find(A.parent, node_of[q], A.err);
            }
            __syncthreads();
            const bool near = pv && bbox.d2(a.x, a.y, a.z) <= g.hi;
            auto linked = [&](int k) {
                const float4 c = qrec[k];
                const float dx = c.x - a.x, dy = c.y - a.y, dz = c.z - a.z;
                const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                return d2 <= g.hi &&
                       (d2 < g.lo || exact_link(A.x, A.y, A.z, __float_as_int(a.w), __float_as_int(c.w), g.r2));
            };
            if (nodes) {
                for (int k0 = 0; k0 < cnt; k0 += 32) {
                    if (!__any_sync(0xffffffffu, near && !done)) break;   // the same for the warp
                    const int k1 = min(k0 + 32, cnt);
                    for (int k = k0; near && k < k1; ++k)
                        if (linked(k)) {
                            uf_union(A.parent, node_a, node_b, A.err);
                            done = 1;
                            break;
                        }
                    __syncwarp();
                }
            } else {
                // every thread starts at another candidate, the next particle in a pair of the same cell: coincident ones
                // are one set after the first step, and known to be after the roots have been looked up again
                int rp = near ? uf_find(A.parent, node_of[p], A.err) : 0;
                // one set already: the tile's usual case
                const bool one = (!near || rp == qroot[0]) && ((int)threadIdx.x >= cnt || qroot[threadIdx.x] == qroot[0]);
                if (__syncthreads_and(one)) continue;
                int k = cnt > 0 ? (threadIdx.x + 1) % cnt : 0;
                for (int j = 0; j < cnt; ++j) {
                    if (near && qroot[k] != rp && !(same && qat[k] <= p) && linked(k))
                        rp = uf_union(A.parent, rp, qroot[k], A.err);
                    k = k + 1 < cnt ? k + 1 : 0;
                    if ((j & (j + 1)) == 0) {
                        __syncthreads();
                        if ((int)threadIdx.x < cnt) qroot[threadIdx.x] = uf_find(A.parent, qroot[threadIdx.x], A.err);
                        if (near) rp = uf_find(A.parent, rp, A.err);
                        __syncthreads();
                    }
                }
            }
            __syncthreads();   // the staging and `done` are written again
        }
    }
}

// Root of every node (in an array of its own: another thread's path halving may still write an older ancestor
// into parent), and per root the smallest original index and whether the component has
// more than one particle.  Consecutive nodes mostly share a root, so the lanes of a warp first take the
// minimum per distinct root and issue one atomicMin each.
__global__ void __launch_bounds__(256) root_kernel(const int *__restrict__ cnt, const int *__restrict__ node_start,
                                                   int *parent, int *__restrict__ root, int *minidx,
                                                   unsigned char *__restrict__ multi, int *err) {
    const int nn = cnt[1];
    const int lane = threadIdx.x & 31;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k - lane < nn; k += (int64_t)gridDim.x * blockDim.x) {
        int r = -1, v = INT_MAX;
        bool many = false;
        if (k < nn) {
            const int m = (int)k;
            r = uf_find(parent, m, err);
            root[m] = r;
            if (r != m) v = minidx[m];   // only roots' entries are lowered
            many = r != m || node_start[m + 1] - node_start[m] > 1;
        }
        unsigned todo = __ballot_sync(0xffffffffu, many);
        while (todo) {
            const int rl = __shfl_sync(0xffffffffu, r, __ffs(todo) - 1);
            const bool mine = many && r == rl;
            const int lo = __reduce_min_sync(0xffffffffu, mine ? v : INT_MAX);
            const unsigned grp = __ballot_sync(0xffffffffu, mine);
            if (lane == __ffs(grp) - 1) {
                if (lo != INT_MAX) atomicMin(minidx + rl, lo);
                multi[rl] = 1;
            }
            todo &= ~grp;
        }
    }
}

__global__ void __launch_bounds__(256) label_kernel(int n, const int *__restrict__ idx, const int *__restrict__ node_of,
                                                    const int *__restrict__ root, const int *__restrict__ minidx,
                                                    const unsigned char *__restrict__ multi, int *__restrict__ labels,
                                                    int *__restrict__ ngroups) {
    const int lane = threadIdx.x & 31;
    int groups = 0;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const int i = idx[k];
        const int r = root[node_of[k]];
        const int l = multi[r] ? minidx[r] : -1;
        labels[i] = l;
        groups += l == i ? 1 : 0;   // one particle a group carries its own index
    }
    for (int o = 16; o > 0; o >>= 1) groups += __shfl_xor_sync(0xffffffffu, groups, o);
    if (lane == 0 && groups) atomicAdd(ngroups, groups);
}

// ---- small inputs ---------------------------------------------------------------------------
// Up to kSmallFof particles, all pairs: no bounding box on the host, no sort, no cells -- five launches and one
// round trip instead of thirty and two.  A call takes 92 us at 5,000 particles (on cells 245), 113 at
// 8,192 (243) and 214 at 16,384 (250).
// A particle is its position relative to particle 0 in linking lengths as two floats an axis (error below 2^-46 of
// the largest); where some lie farther apart than 2^24 linking lengths (or the linking length is subnormal),
// pairs that the floats leave open are tested in FP64 (flags[1]).
constexpr int kSmallFof = 16384;
constexpr float kSmallReach = 16777216.f;

struct SmallArgs {
    int n;
    const double *x, *y, *z;
    float4 *pos_hi, *pos_lo;   // pos_hi[i].w: the particle's root for the sweep
    // [0] non-finite coordinate, [1] coordinates for FP64 tests, [4] the largest |coordinate| (float bits)
    int *flags;
    int *parent, *first, *err;
    float lo, hi;
    double r2;
};

__global__ void __launch_bounds__(256) small_prep_kernel(SmallArgs A, double scale) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int bad = 0, far = 0, reach = 0;
    if (i < A.n) {
        const double v[3] = {A.x[i], A.y[i], A.z[i]}, o[3] = {A.x[0], A.y[0], A.z[0]};
        float hi[3], lo[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (nonfinite(v[d])) bad = 1;
            const double r = (v[d] - o[d]) * scale;
            hi[d] = (float)r;
            lo[d] = (float)(r - (double)hi[d]);
            if (!(fabsf(hi[d]) < kSmallReach)) far = 1;
            reach = max(reach, __float_as_int(fabsf(hi[d])));
        }
        A.pos_hi[i] = make_float4(hi[0], hi[1], hi[2], 0.f);
        A.pos_lo[i] = make_float4(lo[0], lo[1], lo[2], 0.f);
        A.parent[i] = i;
        A.first[i] = A.n;
    }
    bad = __any_sync(0xffffffffu, bad);
    far = __any_sync(0xffffffffu, far);
    reach = __reduce_max_sync(0xffffffffu, reach);
    if ((threadIdx.x & 31) == 0) {
        if (bad) atomicOr(A.flags, 1);
        if (far) atomicOr(A.flags + 1, 1);
        atomicMax(A.flags + 4, reach);
    }
}

// Where the FP64 test's squares overflow or underflow at the linking length, it decides every pair.
__device__ __forceinline__ bool small_in_fp64(const SmallArgs &A) {
    return A.flags[1] != 0 || (A.lo >= 0.f && !(A.r2 > 1e-280 && A.r2 < 1e300));   // (A.lo < 0: linking length 0)
}

// How the kernels below look at a pair: by the first floats, or (low) by both; below `in` their squared distance says that
// the pair is linked, above `out` that it is not.  The second floats are at most 2^-24 of the largest coordinate, two of them an
// axis, so the bounds are 2^-22 of it apart from the linking length, or 2^-45 with both.  Coordinates beyond 2^20 linking
// lengths of particle 0 take both: bounds a quarter of the linking length off would leave too many friends to small_friends
// and a union each, and beyond 2^22 all of them.  With linking length 0 friends have the same floats.
struct SmallRule {
    float in, out;
    bool low;
    __device__ __forceinline__ SmallRule(const SmallArgs &A) {
        const float reach = __int_as_float(A.flags[4]);
        low = !(reach <= 0x1p20f);
        if (A.lo < 0.f) {
            in = -1.f;
            out = 0.f;
        } else if (!(A.r2 > 1e-280 && A.r2 < 1e300)) {
            in = -1.f;
            out = INFINITY;
        } else {
            const float e = reach * (low ? 0x1p-45f : 0x1p-22f) + 1e-5f;
            const float near = sqrtf(A.lo) - e, far = sqrtf(A.hi) + e;
            in = near > 0.f ? near * near * (1.f - 1e-6f) : -1.f;
            out = far * far * (1.f + 1e-6f);   // NaN and infinity: every pair
        }
    }
};

// Squared distance of two particles by both floats.
__device__ __forceinline__ float small_d2(const float4 &ph, const float4 &pl, const float4 &qh, const float4 &ql) {
    const float dx = (qh.x - ph.x) + (ql.x - pl.x), dy = (qh.y - ph.y) + (ql.y - pl.y), dz = (qh.z - ph.z) + (ql.z - pl.z);
    return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

// Whether particles i and j are friends.
__device__ __forceinline__ bool small_friends(const SmallArgs &A, bool fp64, int i, int j) {
    if (fp64) return exact_link(A.x, A.y, A.z, i, j, A.r2);
    const float d2 = small_d2(A.pos_hi[i], A.pos_lo[i], A.pos_hi[j], A.pos_lo[j]);
    if (d2 < A.lo) return true;
    return d2 <= A.hi && exact_link(A.x, A.y, A.z, i, j, A.r2);
}

// All pairs, a particle a lane against a run of kNearLen later ones: the first and the last that are linked beyond doubt.
// The last becomes the particle's parent: the indices rise along every path, so this forest needs no union.
// Each lane remembers two, so no lane waits for another one's search (a warp per particle that stopped at two
// friends took 25 us at 5,000 particles, as lonely ones scan to the end; 10 so).
constexpr int kNearLen = 128, kSweepLen = 512, kSweepT = 8;

__global__ void __launch_bounds__(256) small_near_kernel(SmallArgs A) {
    __shared__ float4 run[kNearLen], tail[kNearLen];
    const int i = blockIdx.x * 256 + threadIdx.x, j0 = blockIdx.y * kNearLen;
    const int len = min(kNearLen, A.n - j0);
    if (j0 + len <= (int)blockIdx.x * 256 + 1) return;   // nothing after any of the block's particles
    const SmallRule rule(A);
    if (threadIdx.x < len) {
        run[threadIdx.x] = A.pos_hi[j0 + threadIdx.x];
        if (rule.low) tail[threadIdx.x] = A.pos_lo[j0 + threadIdx.x];
    }
    __syncthreads();
    if (i >= A.n) return;
    const float4 p = A.pos_hi[i];
    int first = A.n, last = -1;
    auto take = [&](int k, float d2) {
        if (d2 < rule.in) {
            first = min(first, j0 + k);
            last = j0 + k;
        }
    };
    if (!rule.low) {
#pragma unroll 8
        for (int k = max(0, i + 1 - j0); k < len; ++k) {
            const float dx = run[k].x - p.x, dy = run[k].y - p.y, dz = run[k].z - p.z;
            take(k, fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
        }
    } else {
        const float4 pl = A.pos_lo[i];
        for (int k = max(0, i + 1 - j0); k < len; ++k) take(k, small_d2(p, pl, run[k], tail[k]));
    }
    if (last >= 0) {
        atomicMin(A.first + i, first);
        atomicMax(A.parent + i, last);
    }
}

// One block, the parents in shared memory: every particle joined with its first friend, and the roots, for the sweep.
// (In global memory, every step of a path a trip to L2, the unions took 31 us at 5,000 particles; 10 so, roots included.)
__global__ void __launch_bounds__(1024) small_union_kernel(SmallArgs A) {
    extern __shared__ int su_parent[];
    for (int i = threadIdx.x; i < A.n; i += 1024) su_parent[i] = A.parent[i];
    __syncthreads();
    for (int b = 0; b < A.n; b += 1024) {   // whole warps
        const int i = b + threadIdx.x;
        const int first = i < A.n ? A.first[i] : A.n;
        uf_union_warp<true>(su_parent, min(first, A.n - 1), min(i, A.n - 1), first < A.n, A.err);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < A.n; i += 1024) {
        const int r = uf_find<true>(su_parent, i, A.err);
        A.parent[i] = r;
        A.pos_hi[i].w = __int_as_float(r);
    }
}

// All pairs again, eight particles a warp against runs of kSweepLen, one of them a lane: those that may be friends and
// whose roots differ are looked at closely and joined.  A pair costs nine instructions (eight particles share a
// load; the roots come with the positions); with both floats of every position and a particle a warp
// 5,000 particles took 30 us, 11 so (four particles 11, and 223 us for a call on 16,384 instead of 204).
__global__ void __launch_bounds__(256) small_sweep_kernel(SmallArgs A) {
    const int lane = threadIdx.x & 31;
    const int i0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kSweepT;
    const int j1 = min(A.n, (int)(blockIdx.y + 1) * kSweepLen);
    if (i0 >= A.n || i0 + 1 >= j1) return;
    const bool fp64 = small_in_fp64(A);
    const SmallRule rule(A);
    float4 p[kSweepT];
#pragma unroll
    for (int t = 0; t < kSweepT; ++t) p[t] = A.pos_hi[min(i0 + t, A.n - 1)];   // the last one's pairs again past the end
#pragma unroll 2
    for (int j0 = max(i0 & ~31, (int)blockIdx.y * kSweepLen); j0 < j1; j0 += 32) {
        const int j = j0 + lane;
        const float4 q = A.pos_hi[min(j, A.n - 1)];
        unsigned may = 0;
        if (!rule.low) {
#pragma unroll
            for (int t = 0; t < kSweepT; ++t) {
                const float dx = q.x - p[t].x, dy = q.y - p[t].y, dz = q.z - p[t].z;
                const bool near = !(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > rule.out);   // NaN where the floats overflow
                if (near && __float_as_int(q.w) != __float_as_int(p[t].w)) may |= 1u << t;
            }
        } else {
            const float4 ql = A.pos_lo[min(j, A.n - 1)];
#pragma unroll 1
            for (int t = 0; t < kSweepT; ++t) {   // read again: the registers are the other loop's
                const int i = min(i0 + t, A.n - 1);
                const float4 ph = A.pos_hi[i];
                const bool near = !(small_d2(ph, A.pos_lo[i], q, ql) > rule.out);
                if (near && __float_as_int(q.w) != __float_as_int(ph.w)) may |= 1u << t;
            }
        }
        if (!__any_sync(0xffffffffu, may)) continue;
#pragma unroll 1
        for (int t = 0; t < kSweepT; ++t) {
            const int i = min(i0 + t, A.n - 1), jj = min(j, A.n - 1);
            const bool link = (may >> t & 1u) && small_friends(A, fp64, i, jj);
            uf_union_warp(A.parent, i, link ? jj : i, link, A.err);
        }
    }
}

// One block, in shared memory: roots, smallest members and labels (-1 alone), and the number of groups.  No labels where a
// coordinate was not finite (*bad): the call is refused.
__global__ void __launch_bounds__(1024) small_label_kernel(int n, const int *__restrict__ parent,
                                                           const int *__restrict__ bad, int *__restrict__ labels,
                                                           int *__restrict__ ngroups, int *err) {
    if (*bad) return;
    extern __shared__ int sl_smem[];
    int *up = sl_smem, *least = sl_smem + n;   // least[r]: r's smallest member, n + that while r is alone
    __shared__ int groups;
    if (threadIdx.x == 0) groups = 0;
    for (int i = threadIdx.x; i < n; i += 1024) {
        up[i] = parent[i];
        least[i] = n + i;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += 1024) {
        const int r = uf_find<true>(up, i, err);
        if (r != i) atomicMin(least + r, min(i, r));
    }
    __syncthreads();
    int mine = 0;
    for (int i = threadIdx.x; i < n; i += 1024) {
        const int l = least[uf_find<true>(up, i, err)];
        labels[i] = l < n ? l : -1;
        mine += l == i;
    }
    mine = __reduce_add_sync(0xffffffffu, mine);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&groups, mine);
    __syncthreads();
    if (threadIdx.x == 0) *ngroups = groups;
}

int bits_for(uint64_t v) {
    int b = 0;
    while (b < 64 && (v >> b) != 0) ++b;
    return b < 1 ? 1 : b;
}

// --- segmented FoF: per-segment origin and columns -------------------------------------
__global__ void seg_fill_kernel(int nseg, const int64_t *__restrict__ off, int *__restrict__ seg_of) {
    for (int s = blockIdx.x; s < nseg; s += gridDim.x)
        for (int64_t i = off[s] + threadIdx.x; i < off[s + 1]; i += blockDim.x) seg_of[i] = s;
}

// One block per segment: its bounding box (sbox[6s..6s+5] = min xyz, max xyz), the largest
// extent over all segments (as the bits of a non-negative double) and a non-finite flag.
__global__ void __launch_bounds__(256) seg_bbox_kernel(int nseg, const int64_t *__restrict__ off,
                                                       const double *__restrict__ x, const double *__restrict__ y,
                                                       const double *__restrict__ z, double *__restrict__ sbox,
                                                       unsigned long long *__restrict__ ext_bits, int *__restrict__ bad) {
    __shared__ long long sh[6][8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int s = blockIdx.x; s < nseg; s += gridDim.x) {
        long long mn[3] = {LLONG_MAX, LLONG_MAX, LLONG_MAX}, mx[3] = {LLONG_MIN, LLONG_MIN, LLONG_MIN};
        bool nf = false;
        for (int64_t i = off[s] + threadIdx.x; i < off[s + 1]; i += blockDim.x) {
            const double v[3] = {x[i], y[i], z[i]};
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                nf |= nonfinite(v[d]);
                const long long k = ord_of(v[d]);
                mn[d] = min(mn[d], k);
                mx[d] = max(mx[d], k);
            }
        }
        if (__any_sync(0xffffffffu, nf) && lane == 0) atomicOr(bad, 1);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            for (int o = 16; o > 0; o >>= 1) {
                mn[d] = min(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
                mx[d] = max(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
            }
            if (lane == 0) {
                sh[d][w] = mn[d];
                sh[3 + d][w] = mx[d];
            }
        }
        __syncthreads();
        if (threadIdx.x < 6) {
            const int q = threadIdx.x;
            long long v = sh[q][0];
            for (int k = 1; k < (int)(blockDim.x >> 5); ++k) v = q < 3 ? min(v, sh[q][k]) : max(v, sh[q][k]);
            sh[q][0] = v;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const bool empty = off[s + 1] <= off[s];
            double b[6];
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                b[q] = empty ? (q < 3 ? INFINITY : -INFINITY) : val_of(sh[q][0]);
                sbox[6 * (int64_t)s + q] = b[q];
            }
            const double e = empty ? 0.0 : fmax(b[3] - b[0], fmax(b[4] - b[1], b[5] - b[2]));
            if (isfinite(e) && e > 0.0) atomicMax(ext_bits, (unsigned long long)__double_as_longlong(e));
        }
        __syncthreads();
    }
}

// One block: columns of every segment at cell side 1/inv_cell, the first virtual x column of
// each (exclusive prefix of columns + 1 gap), and out = {total columns, max y columns, max z
// columns}.  An empty segment takes one column.
__global__ void __launch_bounds__(1024) seg_cols_kernel(int nseg, const double *__restrict__ sbox, double inv_cell,
                                                        double *__restrict__ smin, long long *__restrict__ scol,
                                                        long long *__restrict__ out) {
    __shared__ long long part[1024];
    __shared__ long long my[1024], mz[1024];
    const int t = threadIdx.x, nt = blockDim.x;
    const int per = (nseg + nt - 1) / nt;
    const int s0 = min(nseg, t * per), s1 = min(nseg, s0 + per);
    long long sum = 0, ay = 1, az = 1;
    for (int s = s0; s < s1; ++s) {
        const double *b = sbox + 6 * (int64_t)s;
        long long cx = 1, cy = 1, cz = 1;
        if (b[3] >= b[0]) {   // non-empty
            cx = (long long)floor((b[3] - b[0]) * inv_cell) + 1;
            cy = (long long)floor((b[4] - b[1]) * inv_cell) + 1;
            cz = (long long)floor((b[5] - b[2]) * inv_cell) + 1;
            smin[3 * (int64_t)s] = b[0];
            smin[3 * (int64_t)s + 1] = b[1];
            smin[3 * (int64_t)s + 2] = b[2];
        } else {
            smin[3 * (int64_t)s] = smin[3 * (int64_t)s + 1] = smin[3 * (int64_t)s + 2] = 0.0;
        }
        scol[4 * (int64_t)s + 1] = cx;
        scol[4 * (int64_t)s + 2] = cy;
        scol[4 * (int64_t)s + 3] = cz;
        sum += cx + 1;
        ay = max(ay, cy);
        az = max(az, cz);
    }
    part[t] = sum;
    my[t] = ay;
    mz[t] = az;
    __syncthreads();
    if (t == 0) {   // 1024 partial sums: a serial pass is cheap next to the per-segment work
        long long run = 0, by = 1, bz = 1;
        for (int k = 0; k < nt; ++k) {
            const long long v = part[k];
            part[k] = run;
            run += v;
            by = max(by, my[k]);
            bz = max(bz, mz[k]);
        }
        out[0] = run;
        out[1] = by;
        out[2] = bz;
    }
    __syncthreads();
    long long run = part[t];
    for (int s = s0; s < s1; ++s) {
        scol[4 * (int64_t)s] = run;
        run += scol[4 * (int64_t)s + 1] + 1;
    }
}

// Cell side, band and scale for linking length ll; ext = the largest extent (ll == 0 only).
void set_scale(FofGeom &g, double ll, double ext) {
    if (ll > 0.0) {
        g.cell = ll * (1.0 + 0x1p-20);
        g.inv_scale = 1.0 / ll;
        g.lo = 1.0f - 1e-5f;
        g.hi = 1.0f + 1e-5f;
    } else {
        // ll == 0 links coincident points only: every float candidate is re-tested exactly
        g.cell = ext > 0.0 ? ext * 0x1p-16 : 1.0;
        g.inv_scale = 1.0 / g.cell;
        g.lo = -1.0f;
        g.hi = 1e-6f;
    }
    g.inv_cell = 1.0 / g.cell;
    g.cs = (float)(g.cell * g.inv_scale);
    g.r2 = ll * ll;
}

int g_uf_cap_host = kUfCapDefault;   // guarded by api_mutex()
int g_uf_cap_pushed[64];             // value last copied to each device (0 = never)
bool g_uf_cap_init = false;

// Copies the host's union-find cap to the current device when it differs from the last copy.
int push_uf_cap(cudaStream_t st) {
    if (!g_uf_cap_init) {
        for (int &v : g_uf_cap_pushed) v = kUfCapDefault;   // the __constant__ initialiser
        g_uf_cap_init = true;
    }
    const int dev = current_device();
    if (dev < 0 || dev >= 64) return fail(HALMA_ERR_CAPACITY, "device ordinal %d out of range", dev);
    if (g_uf_cap_pushed[dev] != g_uf_cap_host) {
        HALMA_CUDA(cudaMemcpyToSymbolAsync(c_uf_cap, &g_uf_cap_host, sizeof(int), 0, cudaMemcpyHostToDevice, st));
        HALMA_CUDA(cudaStreamSynchronize(st));
        g_uf_cap_pushed[dev] = g_uf_cap_host;
    }
    return HALMA_OK;
}

// From kPairsByCount particles on, the number of cells comes to the host by a stream of its own (into page-locked memory:
// a copy elsewhere would keep the host from launching what runs meanwhile): in line it took 13 us of a call.
constexpr int kPairsByCount = 1 << 20;

struct CellSide {
    cudaStream_t s = nullptr;
    cudaEvent_t counted = nullptr, copied = nullptr;
    int *cells = nullptr;
};

int cell_side(CellSide **out) {
    static std::map<int, CellSide> m;   // per device, under api_mutex()
    CellSide &c = m[current_device()];
    if (!c.s) HALMA_CUDA(cudaStreamCreateWithFlags(&c.s, cudaStreamNonBlocking));
    for (cudaEvent_t *e : {&c.counted, &c.copied})
        if (!*e) HALMA_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
    if (!c.cells) HALMA_CUDA(cudaMallocHost(reinterpret_cast<void **>(&c.cells), sizeof(int)));
    *out = &c;
    return HALMA_OK;
}

size_t pair_bytes(int ncell) { return sizeof(int2) * 14 * (size_t)std::max(ncell, 1); }

// Keys, sort, cells, links and labels for a geometry whose cell grid is known.
int fof_core(int n, const double *x, const double *y, const double *z, FofGeom g, SegGeom sg, int *labels,
             int64_t *n_groups, cudaStream_t st) {
    g.ky = g.ncy + 1;
    g.kz = g.ncz + 1;
    const long double cells = (long double)g.ncx * g.ky * g.kz;
    if (cells > 4.0e18L)
        return fail(HALMA_ERR_CAPACITY, "cell grid too large (%lld x %lld x %lld cells)", g.ncx, g.ncy, g.ncz);
    const int cell_bits = bits_for((uint64_t)(g.ncx * g.ky * g.kz - 1));
    // half-cells in the key when there is room for them and the linking length is positive
    g.sb = cell_bits <= 61 && g.lo > 0.f ? 3 : 0;
    const int end_bit = cell_bits + g.sb;
    const int sms = device_sm_count();

    const int nruns = (n + kScanRun - 1) / kScanRun;
    const int heavy_cap = std::max(4096, n / 64);
    const size_t sort_b = sort_pairs_u64_i32_bytes(n, end_bit);
    const size_t scan_b = exclusive_sum_i64_bytes(nruns);
    Layout M;
    // the first three are free for the lists of pairs once the cells and nodes are known
    const size_t o_kin = M.add(8ull * n), o_kout = M.add(8ull * n), o_pre = M.add(16ull * n);
    const size_t o_vin = M.add(4ull * n), o_vout = M.add(4ull * n);
    const size_t o_rec = M.add(16ull * n);
    const size_t o_run = M.add(8ull * nruns), o_base = M.add(8ull * nruns);
    const size_t o_nof = M.add(4ull * n), o_nst = M.add(4ull * (n + 1)), o_sub = M.add(1ull * n);
    const size_t o_nrec = M.add(16ull * n), o_ncell = M.add(4ull * n), o_clist = M.add(8ull * n);
    const size_t o_par = M.add(4ull * n), o_root = M.add(4ull * n), o_min = M.add(4ull * n), o_multi = M.add(1ull * n);
    const size_t o_cnode = M.add(4ull * (n + 1)), o_ckey = M.add(8ull * n);
    const size_t o_heavy = M.add(sizeof(HeavyPair) * (size_t)heavy_cap);
    const size_t o_cnt = M.add(64);
    const size_t o_tmp = M.add(std::max(sort_b, scan_b));
    void *base = nullptr;
    HALMA_TRY(push_uf_cap(st));
    HALMA_TRY(workspace(M.total, &base, st));
    auto *kin = at<uint64_t>(base, o_kin), *kout = at<uint64_t>(base, o_kout);
    auto *vin = at<int>(base, o_vin), *vout = at<int>(base, o_vout);
    auto *rec = at<float4>(base, o_rec), *pre = at<float4>(base, o_pre);
    auto *runs = at<int64_t>(base, o_run), *rbase = at<int64_t>(base, o_base);
    int *node_of = at<int>(base, o_nof), *node_start = at<int>(base, o_nst);
    int *parent = at<int>(base, o_par), *root = at<int>(base, o_root), *minidx = at<int>(base, o_min);
    auto *node_sub = at<unsigned char>(base, o_sub), *multi = at<unsigned char>(base, o_multi);
    int *cell_node = at<int>(base, o_cnode);
    auto *cell_key = at<uint64_t>(base, o_ckey);
    // [0] cells [1] nodes [2] groups [3] error [4] pairs for blocks [6..7] cell pairs [8..9] listed pairs of nodes
    // [10] cells, from their count [12..13] pairs for warps
    int *cnt = at<int>(base, o_cnt);
    auto *npairs = at<unsigned long long>(base, o_cnt + 24), *nlist = npairs + 1;
    auto *cell_list = at<long long>(base, o_clist);
    int *node_cell = at<int>(base, o_ncell);
    void *tmp = at<void>(base, o_tmp);
    const int g1 = std::min(sms * 8, grid_for(n, 256));

    Profile &prof = profile();
    const bool stages = !sg.seg_of;   // stage times of the plain FoF only
    auto mark = [&](int k) { return stages ? prof.fof_mark(k, st) : HALMA_OK; };
    HALMA_CUDA(cudaMemsetAsync(cnt, 0, 64, st));
    // the integer map when the coordinates and the grid stay within 2^37 quarter cells (plain
    // FoF; the segmented one has per-segment origins and keeps the FP64 map)
    const double s4 = 4.0 * g.inv_cell, lim = 0x1p37;
    const double bxd = -g.xmin * s4, byd = -g.ymin * s4, bzd = -g.zmin * s4;
    double reach = fmax(fabs(g.xmin), fabs(g.xmin + g.cell * (double)g.ncx));
    reach = fmax(reach, fmax(fabs(g.ymin), fabs(g.ymin + g.cell * (double)g.ncy)));
    reach = fmax(reach, fmax(fabs(g.zmin), fabs(g.zmin + g.cell * (double)g.ncz))) * s4;
    const bool fixed = !sg.seg_of && s4 >= 0x1p-1000 && reach < lim && fabs(bxd) < lim && fabs(byd) < lim &&
                       fabs(bzd) < lim;
    if (fixed)
        HALMA_LAUNCH(keys_kernel<true>, g1, 256, 0, st, x, y, z, n, g, sg, (long long)floor(bxd * 0x1p24),
                     (long long)floor(byd * 0x1p24), (long long)floor(bzd * 0x1p24), kin, vin, pre);
    else
        HALMA_LAUNCH(keys_kernel<false>, g1, 256, 0, st, x, y, z, n, g, sg, 0ll, 0ll, 0ll, kin, vin, pre);
    HALMA_TRY(mark(1));
    HALMA_TRY(sort_pairs_u64_i32(tmp, sort_b, kin, kout, vin, vout, n, end_bit, st));
    HALMA_TRY(mark(2));
    const int gr = grid_for(nruns, 8);
    HALMA_LAUNCH(head_count_kernel, gr, 256, 0, st, n, g.sb, kout, runs, nruns, cnt + 10);
    CellSide *side = nullptr;
    if (n > kPairsByCount) {   // the cells' number, on its way to the host while the two kernels below run
        HALMA_TRY(cell_side(&side));
        HALMA_CUDA(cudaEventRecord(side->counted, st));
        HALMA_CUDA(cudaStreamWaitEvent(side->s, side->counted, 0));
        HALMA_CUDA(cudaMemcpyAsync(side->cells, cnt + 10, sizeof(int), cudaMemcpyDeviceToHost, side->s));
        HALMA_CUDA(cudaEventRecord(side->copied, side->s));
    }
    HALMA_TRY(exclusive_sum_i64(tmp, scan_b, runs, rbase, nruns, st));
    HALMA_LAUNCH(head_apply_kernel, gr, 256, 0, st, n, g.sb, kout, vout, pre, rbase, nruns, rec, node_of, node_start,
                 node_cell, node_sub, at<float4>(base, o_nrec), parent, minidx, multi, cell_node, cell_key, cnt);
    HALMA_TRY(mark(3));
    // The list of cell pairs (at most 14 x 8 bytes per occupied cell) in its own cached buffer: of a size for as many cells as
    // particles up to kPairsByCount of them (117 MB), and for the cells there are above that, or where there is no room.
    int ncell = n;
    void *pbase = nullptr;
    int got = HALMA_ERR_NOMEM;
    if (n <= kPairsByCount) {
        got = workspace(pair_bytes(n), &pbase, st, 10);
    } else {
        HALMA_CUDA(cudaEventSynchronize(side->copied));
        ncell = *side->cells;
    }
    if (got == HALMA_ERR_NOMEM) {
        if (n <= kPairsByCount) {
            HALMA_CUDA(cudaMemcpyAsync(&ncell, cnt + 0, sizeof(int), cudaMemcpyDeviceToHost, st));
            HALMA_CUDA(cudaStreamSynchronize(st));
        }
        got = workspace(pair_bytes(ncell), &pbase, st, 10);
    }
    HALMA_TRY(got);
    int2 *pairs = static_cast<int2 *>(pbase);
    const int gc = std::min(sms * 8, grid_for(ncell, 256));
    if (g.sb)
        HALMA_LAUNCH(cell_pair_kernel<true>, gc, 256, 0, st, cnt, cell_node, cell_key, g.ky, g.kz, pairs, cell_list,
                     npairs);
    else
        HALMA_LAUNCH(cell_pair_kernel<false>, gc, 256, 0, st, cnt, cell_node, cell_key, g.ky, g.kz, pairs, cell_list,
                     npairs);
    HALMA_TRY(mark(4));
    LinkArgs A{cnt, pairs, npairs, cell_list, cell_node, node_start, node_cell, node_sub, cell_key, rec,
               at<float4>(base, o_nrec), x, y, z, parent, cnt + 3, at<unsigned long long>(base, o_kin), npairs + 3, n,
               at<HeavyPair>(base, o_heavy), cnt + 4, heavy_cap};
    if (g.sb) {
        auto *list = at<unsigned long long>(base, o_kout);   // kout and pre: 3 n entries
        const long long cap = 3ll * n;
        HALMA_LAUNCH(hook_kernel, g1, 256, 0, st, A, g);
        HALMA_LAUNCH(flatten_kernel, g1, 256, 0, st, cnt, parent, root, cnt + 3);
        HALMA_LAUNCH(sweep_kernel, g1, 256, 0, st, A, g, root, list, cap, nlist);
        HALMA_TRY(mark(5));
        HALMA_LAUNCH(link_kernel, g1, 256, 0, st, A, g, list, cap, nlist);
    } else {
        HALMA_TRY(mark(5));
        HALMA_LAUNCH(hook_particles_kernel, g1, 256, 0, st, A, g);
        HALMA_LAUNCH(link_particles_kernel, std::min(sms * 8, grid_for(4ll * ncell, 256)), 256, 0, st, A, g);
    }
    HALMA_LAUNCH(crowd_kernel, sms * 8, 256, 0, st, A, g, g.sb ? 1 : 0);
    HALMA_LAUNCH(heavy_kernel, sms * 4, 256, 0, st, A, g, node_of, g.sb ? 1 : 0);
    HALMA_TRY(mark(6));
    HALMA_LAUNCH(root_kernel, g1, 256, 0, st, cnt, node_start, parent, root, minidx, multi, cnt + 3);
    HALMA_LAUNCH(label_kernel, g1, 256, 0, st, n, vout, node_of, root, minidx, multi, labels, cnt + 2);
    HALMA_TRY(mark(7));
    int hc[4];
    HALMA_CUDA(cudaMemcpyAsync(hc, cnt, sizeof(hc), cudaMemcpyDeviceToHost, st));
    HALMA_CUDA(cudaStreamSynchronize(st));
    if (hc[3]) return fail(HALMA_ERR_NOT_CONVERGED, "union-find iteration cap reached");
    if (n_groups) *n_groups = hc[2];
    return HALMA_OK;
}

// The small path (see kSmallFof).
int fof_small(int n, const double *x, const double *y, const double *z, double ll, int *labels, int64_t *n_groups,
              cudaStream_t st) {
    Layout L;
    const size_t o_hi = L.add(sizeof(float4) * n), o_lo = L.add(sizeof(float4) * n), o_par = L.add(4ull * n);
    const size_t o_first = L.add(4ull * n), o_cnt = L.add(64);
    void *base = nullptr;
    HALMA_TRY(push_uf_cap(st));
    HALMA_TRY(workspace(L.total, &base, st));
    int *cnt = at<int>(base, o_cnt);   // [0] non-finite [1] FP64 tests [2] groups [3] error
    int *parent = at<int>(base, o_par);
    Profile &prof = profile();
    FofGeom g{};
    set_scale(g, ll, 0.0);
    HALMA_CUDA(cudaMemsetAsync(cnt, 0, 64, st));
    const int gt = grid_for(n, 256);
    SmallArgs A{n,   x,      y,      z, at<float4>(base, o_hi), at<float4>(base, o_lo),
                cnt, parent, at<int>(base, o_first), cnt + 3, g.lo, g.hi, g.r2};
    HALMA_LAUNCH(small_prep_kernel, gt, 256, 0, st, A, g.inv_scale);
    for (int k = 1; k <= 5; ++k) HALMA_TRY(prof.fof_mark(k, st));
    HALMA_LAUNCH(small_near_kernel, dim3(gt, (n + kNearLen - 1) / kNearLen), 256, 0, st, A);
    HALMA_CUDA(cudaFuncSetAttribute(small_union_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kSmallFof));
    HALMA_LAUNCH(small_union_kernel, 1, 1024, 4 * n, st, A);
    HALMA_LAUNCH(small_sweep_kernel, dim3(grid_for(n, 8 * kSweepT), (n + kSweepLen - 1) / kSweepLen), 256, 0, st, A);
    HALMA_TRY(prof.fof_mark(6, st));
    HALMA_CUDA(cudaFuncSetAttribute(small_label_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * kSmallFof));
    HALMA_LAUNCH(small_label_kernel, 1, 1024, 8 * n, st, n, parent, cnt, labels, cnt + 2, cnt + 3);
    HALMA_TRY(prof.fof_mark(7, st));
    int hc[4];
    HALMA_CUDA(cudaMemcpyAsync(hc, cnt, sizeof(hc), cudaMemcpyDeviceToHost, st));
    HALMA_CUDA(cudaStreamSynchronize(st));
    if (hc[0]) return fail(HALMA_ERR_INVALID, "non-finite particle position");
    if (hc[3]) return fail(HALMA_ERR_NOT_CONVERGED, "union-find iteration cap reached");
    if (n_groups) *n_groups = hc[2];
    return HALMA_OK;
}

}  // namespace

// Bounding box of n > 0 device points, returned on the host: min x, y, z, max x, y, z, and a
// non-zero seventh value if any coordinate is not finite.  Uses workspace slot 0.
int bbox_device(int n, const double *x, const double *y, const double *z, double bb[7], cudaStream_t st) {
    const int gb = std::min(device_sm_count() * 4, grid_for(n, 256));
    Layout L;
    const size_t o_part = L.add(sizeof(double) * 7 * gb);
    const size_t o_out = L.add(sizeof(double) * 8);
    void *base = nullptr;
    HALMA_TRY(workspace(L.total, &base, st));
    HALMA_LAUNCH(bbox_partial_kernel, gb, 256, 0, st, x, y, z, n, at<long long>(base, o_part));
    HALMA_LAUNCH(bbox_final_kernel, 1, 256, 0, st, at<long long>(base, o_part), gb, at<double>(base, o_out));
    HALMA_CUDA(cudaMemcpyAsync(bb, at<double>(base, o_out), 7 * sizeof(double), cudaMemcpyDeviceToHost, st));
    HALMA_CUDA(cudaStreamSynchronize(st));
    return HALMA_OK;
}

// Full FoF on device arrays (no staging, no locking); used by halma_fof and the pipeline.
int fof_device(int n, const double *x, const double *y, const double *z, double ll, int *labels,
               int64_t *n_groups, cudaStream_t st) {
    if (n == 0) {
        if (n_groups) *n_groups = 0;
        return HALMA_OK;
    }
    FofGeom g{};
    HALMA_TRY(profile().fof_mark(0, st));
    if (n <= kSmallFof) return fof_small(n, x, y, z, ll, labels, n_groups, st);
    {
        double bb[7];
        HALMA_TRY(bbox_device(n, x, y, z, bb, st));
        if (bb[6] != 0.0) return fail(HALMA_ERR_INVALID, "non-finite particle position");
        g.xmin = bb[0];
        g.ymin = bb[1];
        g.zmin = bb[2];
        const double ext = std::max(bb[3] - bb[0], std::max(bb[4] - bb[1], bb[5] - bb[2]));
        set_scale(g, ll, ext);
        g.ncx = (long long)floor((bb[3] - bb[0]) * g.inv_cell) + 1;
        g.ncy = (long long)floor((bb[4] - bb[1]) * g.inv_cell) + 1;
        g.ncz = (long long)floor((bb[5] - bb[2]) * g.inv_cell) + 1;
    }
    return fof_core(n, x, y, z, g, SegGeom{}, labels, n_groups, st);
}

// FoF inside segments (particles of segment s are rows off[s] .. off[s+1], off on the
// device): one launch sequence for all segments.  Labels are the smallest row index of each
// component, -1 for rows without a friend in their own segment.  The per-segment geometry
// lives in workspace slot 2, the linking scratch in slot 0.
int fof_segmented_device(int n, int nseg, const int64_t *off, const double *x, const double *y, const double *z,
                         double ll, int *labels, int64_t *n_groups, cudaStream_t st) {
    if (n == 0 || nseg == 0) {
        if (n_groups) *n_groups = 0;
        return HALMA_OK;
    }
    Layout L;
    const size_t o_seg = L.add(4ull * n), o_box = L.add(48ull * nseg), o_min = L.add(24ull * nseg);
    const size_t o_col = L.add(32ull * nseg), o_cnt = L.add(64);
    void *base = nullptr;
    HALMA_TRY(workspace(L.total, &base, st, 2));
    int *seg_of = at<int>(base, o_seg);
    double *sbox = at<double>(base, o_box), *smin = at<double>(base, o_min);
    long long *scol = at<long long>(base, o_col);
    unsigned long long *ext_bits = at<unsigned long long>(base, o_cnt);
    int *bad = at<int>(base, o_cnt + 8);
    long long *cols = at<long long>(base, o_cnt + 16);
    const int gs = std::min(nseg, device_sm_count() * 16);
    HALMA_CUDA(cudaMemsetAsync(at<void>(base, o_cnt), 0, 64, st));
    HALMA_LAUNCH(seg_fill_kernel, gs, 256, 0, st, nseg, off, seg_of);
    HALMA_LAUNCH(seg_bbox_kernel, gs, 256, 0, st, nseg, off, x, y, z, sbox, ext_bits, bad);
    long long hc[2];
    HALMA_CUDA(cudaMemcpyAsync(hc, at<void>(base, o_cnt), 16, cudaMemcpyDeviceToHost, st));
    HALMA_CUDA(cudaStreamSynchronize(st));
    if ((int)hc[1] != 0) return fail(HALMA_ERR_INVALID, "non-finite particle position");
    double ext;
    memcpy(&ext, &hc[0], 8);
    FofGeom g{};
    set_scale(g, ll, ext);
    HALMA_LAUNCH(seg_cols_kernel, 1, 1024, 0, st, nseg, sbox, g.inv_cell, smin, scol, cols);
    long long cc[3];
    HALMA_CUDA(cudaMemcpyAsync(cc, cols, sizeof(cc), cudaMemcpyDeviceToHost, st));
    HALMA_CUDA(cudaStreamSynchronize(st));
    g.ncx = cc[0];
    g.ncy = cc[1];
    g.ncz = cc[2];
    SegGeom sg;
    sg.seg_of = seg_of;
    sg.smin = smin;
    sg.scol = scol;
    return fof_core(n, x, y, z, g, sg, labels, n_groups, st);
}

}  // namespace halma

using namespace halma;

extern "C" int halma_set_union_find_cap(int32_t cap) {
    std::lock_guard<std::mutex> guard(api_mutex());
    g_uf_cap_host = cap < 0 ? kUfCapDefault : cap;
    return HALMA_OK;
}

extern "C" int halma_fof(int64_t n, const double *x, const double *y, const double *z, double linking_length,
                         int32_t *labels, int64_t *n_groups, halma_stream_t stream) {
    if (n < 0) return fail(HALMA_ERR_INVALID, "negative particle count");
    if (n >= INT_MAX) return fail(HALMA_ERR_CAPACITY, "at most 2^31-2 particles per call");
    if (!(linking_length >= 0.0) || !isfinite(linking_length))
        return fail(HALMA_ERR_INVALID, "linking length must be finite and >= 0");
    if (n > 0 && (!x || !y || !z || !labels)) return fail(HALMA_ERR_INVALID, "null pointer");
    if (n == 0) {
        if (n_groups) *n_groups = 0;
        return HALMA_OK;
    }
    std::lock_guard<std::mutex> guard(api_mutex());
    cudaStream_t st = (cudaStream_t)stream;
    Stager sg;
    const double *dx = nullptr, *dy = nullptr, *dz = nullptr;
    int32_t *dl = nullptr;
    sg.add(x, n, true, false, &dx);
    sg.add(y, n, true, false, &dy);
    sg.add(z, n, true, false, &dz);
    sg.add((const int32_t *)labels, n, false, true, &dl);
    if (sg.any_host) {
        // host arrays live in their own allocation so the FoF scratch can reuse the workspace
        std::vector<void *> owned;
        Layout L;
        sg.plan(L);
        void *stage = nullptr;
        HALMA_CUDA(cudaMallocAsync(&stage, L.total, st));
        int s = sg.bind_and_upload(stage, st);
        if (s == HALMA_OK) s = fof_device((int)n, dx, dy, dz, linking_length, dl, n_groups, st);
        if (s == HALMA_OK) s = sg.download(st);
        cudaFreeAsync(stage, st);
        cudaStreamSynchronize(st);
        return s;
    }
    HALMA_TRY(sg.bind_and_upload(nullptr, st));
    return fof_device((int)n, dx, dy, dz, linking_length, dl, n_groups, st);
}

namespace halma {
namespace {

// Members per label (a label is the smallest index of its group), one atomic per distinct
// label among the lanes of a warp: group members are often neighbours in index order.
__global__ void group_count_kernel(int n, const int *__restrict__ labels, int *__restrict__ gsize,
                                   int *__restrict__ bad) {
    const int lane = threadIdx.x & 31;
    for (int i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + threadIdx.x;
        int l = i < n ? labels[i] : -1;
        if (l < -1 || l >= n) {   // not a particle index: reported, counted nowhere
            atomicOr(bad, 1);
            l = -1;
        }
        const unsigned peers = __match_any_sync(0xffffffffu, l);
        if (l >= 0 && lane == __ffs(peers) - 1) atomicAdd(gsize + l, __popc(peers));
    }
}

// Per particle: kept (its group has >= minp members) in the low 32 bits and group head (kept,
// and the smallest index of its group) in the high 32 bits, for one exclusive scan giving every
// kept particle its position among the kept particles and every group its index: the heads
// appear in index order, which is the order of the groups' smallest members.
__global__ void group_flag_kernel(int n, const int *__restrict__ labels, const int *__restrict__ gsize, int minp,
                                  long long *__restrict__ flags) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int l = labels[i];
        const bool keep = l >= 0 && l < n && gsize[l] >= minp;
        flags[i] = keep ? (1ll | (l == i ? 1ll << 32 : 0ll)) : 0ll;
    }
}

// Kept particles in index order, keyed by their group's index; the counts go to cnt[2..3]
// and the member count to offsets[groups].
__global__ void group_scatter_kernel(int n, const int *__restrict__ labels, const long long *__restrict__ flags,
                                     const long long *__restrict__ pre, uint32_t *__restrict__ keys,
                                     int *__restrict__ vals, int *__restrict__ cnt, int64_t *__restrict__ offsets) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const long long f = flags[i];
        if (f) {
            const int pos = (int)(pre[i] & 0xffffffffll);
            keys[pos] = (uint32_t)(pre[labels[i]] >> 32);   // heads before the group's head
            vals[pos] = i;
        }
        if (i == n - 1) {
            const long long t = pre[i] + f;
            cnt[2] = (int)(t >> 32);
            cnt[3] = (int)(t & 0xffffffffll);
            offsets[t >> 32] = t & 0xffffffffll;
        }
    }
}

// Group offsets from the sorted keys: a group starts where its index first appears.
__global__ void group_offsets_kernel(int nm, const uint32_t *__restrict__ keys, int64_t *__restrict__ offsets) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nm; k += gridDim.x * blockDim.x)
        if (k == 0 || keys[k] != keys[k - 1]) offsets[keys[k]] = k;
}

// All of the grouping for up to kSmallGroups particles in one block of 1024 threads, the labels' counts and the groups'
// first places in shared memory: one launch and one round trip instead of ten and two.  A call takes 105 us at 5,000
// particles (124 on the general path) and as much as that at 12,000.  A member's place in its group is the number of earlier
// members: per chunk of 1024 particles the warps take their places one after another, from counters that hold the members
// of earlier chunks and warps.
// cnt: [0] label outside [-1, n), [1] labels that are not their groups' members (the caller then takes the general
// path), [2] groups, [3] members.
constexpr int kSmallGroups = 8192;

__global__ void __launch_bounds__(1024) small_groups_kernel(int n, const int *__restrict__ labels, int minp,
                                                            int64_t *__restrict__ offsets, int *__restrict__ members,
                                                            int *__restrict__ cnt) {
    extern __shared__ int sg_smem[];
    int *size = sg_smem, *place = sg_smem + n;   // by label: members; next free place
    __shared__ int2 wsum[32];
    __shared__ int2 run;   // groups and members before the chunk
    __shared__ int bad;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    for (int i = t; i < n; i += 1024) size[i] = place[i] = 0;
    if (t == 0) {
        run = make_int2(0, 0);
        bad = 0;
    }
    __syncthreads();
    for (int i = t; i < n; i += 1024) {
        const int l = labels[i];
        if (l < -1 || l >= n) bad = 1;
        else if (l >= 0) atomicAdd(size + l, 1);
    }
    __syncthreads();
    if (bad) {
        if (t == 0) cnt[0] = 1;
        return;
    }
    // the kept groups in order of their heads: a group's head carries its own index
    for (int c = 0; c < n; c += 1024) {
        const int i = c + t;
        const bool head = i < n && labels[i] == i && size[i] >= minp;
        const int sz = head ? size[i] : 0;
        int hc = head ? 1 : 0, sc = sz;
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, hc, o), b = __shfl_up_sync(0xffffffffu, sc, o);
            if (lane >= o) {
                hc += a;
                sc += b;
            }
        }
        if (lane == 31) wsum[w] = make_int2(hc, sc);
        __syncthreads();
        int2 before = run, all = make_int2(0, 0);
        for (int k = 0; k < 32; ++k) {
            if (k < w) {
                before.x += wsum[k].x;
                before.y += wsum[k].y;
            }
            all.x += wsum[k].x;
            all.y += wsum[k].y;
        }
        if (head) {
            place[i] = before.y + sc - sz;
            offsets[before.x + hc - 1] = before.y + sc - sz;
        }
        __syncthreads();
        if (t == 0) run = make_int2(run.x + all.x, run.y + all.y);
        __syncthreads();
    }
    if (t == 0) {
        offsets[run.x] = run.y;
        cnt[2] = run.x;
        cnt[3] = run.y;
    }
    for (int c = 0; c < n; c += 1024) {
        const int i = c + t;
        const int l = i < n ? labels[i] : -1;
        const bool keep = l >= 0 && size[l] >= minp;
        if (keep && labels[l] != l) cnt[1] = 1;   // a label that its own particle does not carry
        const unsigned peers = __match_any_sync(0xffffffffu, keep ? l : -1);
        const int rank = __popc(peers & ((1u << lane) - 1u)), many = __popc(peers);
        for (int k = 0; k < 32; ++k) {
            if (k == w) {
                const int p = keep ? place[l] : 0;
                __syncwarp();
                if (keep) {
                    if (rank == 0) place[l] = p + many;
                    if (p + rank < n) members[p + rank] = i;
                }
            }
            __syncthreads();
        }
    }
}

}  // namespace

// Groups of >= minp members in the reference order, on device arrays: members per label,
// flags and one scan over the particles (position among the kept, group index), the kept
// particles keyed by group index in index order, one stable radix sort over the bits of the
// group count, offsets from the sorted keys.  The counts are returned on the host (one
// synchronisation, before the sort).
int fof_groups_device(int n, const int *labels, int minp, int64_t *offsets, int *members,
                      int64_t *n_groups, int64_t *n_members, cudaStream_t st) {
    if (n <= kSmallGroups) {
        void *base = nullptr;
        HALMA_TRY(workspace(64, &base, st));
        int *cnt = static_cast<int *>(base);
        HALMA_CUDA(cudaMemsetAsync(cnt, 0, 64, st));
        const int smem = 2 * 4 * n;
        HALMA_CUDA(cudaFuncSetAttribute(small_groups_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        2 * 4 * kSmallGroups));
        HALMA_LAUNCH(small_groups_kernel, 1, 1024, smem, st, n, labels, std::max(minp, 1), offsets, members, cnt);
        int hc[4];
        HALMA_CUDA(cudaMemcpyAsync(hc, cnt, sizeof(hc), cudaMemcpyDeviceToHost, st));
        HALMA_CUDA(cudaStreamSynchronize(st));
        if (hc[0]) return fail(HALMA_ERR_INVALID, "labels must be particle indices in [0, n) or -1");
        if (!hc[1]) {
            *n_groups = hc[2];
            if (n_members) *n_members = hc[3];
            return HALMA_OK;
        }
    }
    const size_t sort_b = sort_pairs_u32_i32_bytes(n);
    const size_t scan_b = exclusive_sum_i64_bytes(n);
    Layout L;
    const size_t o_gsize = L.add(4ull * n), o_flag = L.add(8ull * n), o_pre = L.add(8ull * n);
    const size_t o_kin = L.add(4ull * n), o_kout = L.add(4ull * n), o_vin = L.add(4ull * n);
    const size_t o_cnt = L.add(64), o_tmp = L.add(std::max(sort_b, scan_b));
    void *base = nullptr;
    HALMA_TRY(workspace(L.total, &base, st));
    auto *gsize = at<int>(base, o_gsize);
    auto *flags = at<long long>(base, o_flag), *pre = at<long long>(base, o_pre);
    auto *kin = at<uint32_t>(base, o_kin), *kout = at<uint32_t>(base, o_kout);
    auto *vin = at<int>(base, o_vin);
    int *cnt = at<int>(base, o_cnt);
    void *tmp = at<void>(base, o_tmp);
    const int g1 = std::min(device_sm_count() * 8, grid_for(n, 256));
    HALMA_CUDA(cudaMemsetAsync(cnt, 0, 64, st));
    HALMA_CUDA(cudaMemsetAsync(gsize, 0, 4ull * n, st));
    HALMA_LAUNCH(group_count_kernel, g1, 256, 0, st, n, labels, gsize, cnt);
    HALMA_LAUNCH(group_flag_kernel, g1, 256, 0, st, n, labels, gsize, std::max(minp, 1), flags);
    HALMA_TRY(exclusive_sum_i64(tmp, scan_b, reinterpret_cast<const int64_t *>(flags),
                                reinterpret_cast<int64_t *>(pre), n, st));
    HALMA_LAUNCH(group_scatter_kernel, g1, 256, 0, st, n, labels, flags, pre, kin, vin, cnt, offsets);
    int hc[4];
    HALMA_CUDA(cudaMemcpyAsync(hc, cnt, sizeof(hc), cudaMemcpyDeviceToHost, st));
    HALMA_CUDA(cudaStreamSynchronize(st));
    if (hc[0]) return fail(HALMA_ERR_INVALID, "labels must be particle indices in [0, n) or -1");
    const int ng = hc[2], nm = hc[3];
    if (nm > 0) {
        if (ng > 1)
            HALMA_TRY(sort_pairs_u32_i32(tmp, sort_b, kin, kout, vin, members, nm, bits_for((uint64_t)(ng - 1)), st));
        else   // one group: already in order
            HALMA_CUDA(cudaMemcpyAsync(members, vin, 4ull * nm, cudaMemcpyDeviceToDevice, st));
        HALMA_LAUNCH(group_offsets_kernel, std::min(device_sm_count() * 8, grid_for(nm, 256)), 256, 0, st, nm,
                     ng > 1 ? kout : kin, offsets);
    }
    *n_groups = ng;
    if (n_members) *n_members = nm;
    return HALMA_OK;
}

}  // namespace halma

extern "C" int halma_fof_groups(int64_t n, const int32_t *labels, int32_t min_members, int64_t *offsets,
                                int32_t *members, int64_t *n_groups, halma_stream_t stream) {
    if (n < 0) return fail(HALMA_ERR_INVALID, "negative particle count");
    if (n >= INT_MAX) return fail(HALMA_ERR_CAPACITY, "at most 2^31-2 particles per call");
    if (!offsets || !n_groups || (n > 0 && (!labels || !members))) return fail(HALMA_ERR_INVALID, "null pointer");
    if (n == 0) {
        *n_groups = 0;
        int64_t zero = 0;
        if (is_device_pointer(offsets)) HALMA_CUDA(cudaMemcpy(offsets, &zero, 8, cudaMemcpyHostToDevice));
        else offsets[0] = 0;
        set_group_members(0);
        return HALMA_OK;
    }
    std::lock_guard<std::mutex> guard(api_mutex());
    cudaStream_t st = (cudaStream_t)stream;
    const bool h_lab = !is_device_pointer(labels), h_off = !is_device_pointer(offsets),
               h_mem = !is_device_pointer(members);
    void *stage = nullptr;
    const int *dl = labels;
    int64_t *doff = offsets;
    int *dmem = members;
    if (h_lab || h_off || h_mem) {
        Layout L;
        const size_t a = L.add(4ull * n), b = L.add(8ull * (n + 1)), c = L.add(4ull * n);
        HALMA_CUDA(cudaMallocAsync(&stage, L.total, st));
        if (h_lab) {
            dl = at<int>(stage, a);
            HALMA_CUDA(cudaMemcpyAsync((void *)dl, labels, 4ull * n, cudaMemcpyHostToDevice, st));
        }
        if (h_off) doff = at<int64_t>(stage, b);
        if (h_mem) dmem = at<int>(stage, c);
    }
    int64_t ng = 0, nm = 0;
    int s = fof_groups_device((int)n, dl, min_members, doff, dmem, &ng, &nm, st);
    if (s == HALMA_OK) {
        if (h_off && cudaMemcpyAsync(offsets, doff, 8ull * (ng + 1), cudaMemcpyDeviceToHost, st) != cudaSuccess)
            s = fail(HALMA_ERR_CUDA, "copy of group offsets failed");
        if (h_mem && nm > 0 && cudaMemcpyAsync(members, dmem, 4ull * nm, cudaMemcpyDeviceToHost, st) != cudaSuccess)
            s = fail(HALMA_ERR_CUDA, "copy of group members failed");
        *n_groups = ng;
    }
    if (stage) cudaFreeAsync(stage, st);
    cudaStreamSynchronize(st);
    if (s == HALMA_OK) set_group_members(nm);
    return s;
}
