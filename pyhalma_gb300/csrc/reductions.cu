// Per-halo FP64 reductions over CSR halo segments (python_scripts/halo_properties.py):
//   total_mass (:16-24), center_of_mass (:26-43), CM_velocity (:45-60),
//   furthest_particle (:98-111), half_mass_radius (:365-392), sigma_effective (:607-625).
// The half-mass radius needs the members in increasing distance from the centre: one stable radix sort over all
// particles by (halo, leading bits of the FP64 distance), the runs of equal leading bits put in order
// by the full distance, after which each halo walks its own segment.
#include <cooperative_groups.h>
#include <limits.h>
#include <math.h>
#include <string.h>

#include "common.cuh"
#include "sort.cuh"
#include "unbind.cuh"

namespace halma {
namespace {

struct Red {
    double M, cx, cy, cz, vx, vy, vz, rmax, r05, sigma, n, mref, plain;
};

__device__ __forceinline__ double wsum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double wmax(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

template <int NV>
__device__ void bsum(double (&v)[NV], double (*sh)[32]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        const double s = wsum(v[q]);
        if (lane == 0) sh[q][w] = s;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            double s = lane < nw ? sh[q][lane] : 0.0;
            s = wsum(s);
            if (lane == 0) sh[q][0] = s;
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; ++q) v[q] = sh[q][0];
    __syncthreads();
}

// The rows of the reductions.  With period > 0 they are sets of hp haloes each over the same members: halo h
// is halo h % hp of set h / hp, which has its own positions (rows start at set * period); velocities,
// masses and mask are the members' own (no mask with sets).
struct RedIn {
    const double *x[kRedSets], *y[kRedSets], *z[kRedSets];
    const double *vx, *vy, *vz, *m;
    const unsigned char *mask;
    int64_t period;
    int hp;
    __device__ __forceinline__ int set(int h) const { return period ? h / hp : 0; }
};

// The member range of every halo is cut into chunks of at most kRedChunk members, so that a
// big halo's FP64 sums are spread over many blocks (GB300 issues FP64 instructions at a small
// fraction of its FP32 rate, so one block per halo would leave the biggest halo's SM as the
// critical path).  Chunk c belongs to halo chunk_h[c] and covers its members
// off[h] + (c - cstart[h]) * kRedChunk onward.  The partial sums of a halo's chunks are added
// in chunk order, so results do not depend on scheduling.
constexpr int kRedChunk = 4096;
constexpr int kRedParts = 9;   // M, Mx, My, Mz, Mvx, Mvy, Mvz, count, masses the integer walk cannot take

__global__ void red_chunks_kernel(int nh, const int64_t *__restrict__ off, int *__restrict__ cnum,
                                  int *__restrict__ longest) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *longest = 0;   // see red_ties_kernel
    for (int h = blockIdx.x * blockDim.x + threadIdx.x; h <= nh; h += gridDim.x * blockDim.x) {
        const int64_t n = h < nh ? off[h + 1] - off[h] : 0;
        cnum[h] = h < nh ? (int)(n > 0 ? (n + kRedChunk - 1) / kRedChunk : 1) : 0;
    }
}

__global__ void red_owner_kernel(int nh, const int *__restrict__ cstart, int *__restrict__ chunk_h) {
    for (int h = blockIdx.x * blockDim.x + threadIdx.x; h < nh; h += gridDim.x * blockDim.x)
        for (int c = cstart[h]; c < cstart[h + 1]; ++c) chunk_h[c] = h;
}

struct Chunk {
    int h;
    int64_t b, e;
};

__device__ __forceinline__ bool chunk_of(int c, int nh, const int64_t *__restrict__ off, const int *__restrict__ cstart,
                                         const int *__restrict__ chunk_h, Chunk &k) {
    if (c >= cstart[nh]) return false;
    k.h = chunk_h[c];
    k.b = off[k.h] + (int64_t)(c - cstart[k.h]) * kRedChunk;
    k.e = min(off[k.h + 1], k.b + (int64_t)kRedChunk);
    return true;
}

// Per chunk: FP64 sums of m, m x, m v, the member count, and the number of masses that are
// negative, -0.0 or not finite (those haloes walk with plain FP64 adds).  SUMS = false leaves the sums zero, for
// callers that give centre, velocity, mass and all (the FP64 pipe is the kernel's bound with them).
template <bool SUMS>
__global__ void __launch_bounds__(256) red_part_kernel(int nh, const int64_t *__restrict__ off,
                                                       const int *__restrict__ cstart, const int *__restrict__ chunk_h,
                                                       RedIn in, double *__restrict__ part) {
    Chunk k;
    if (!chunk_of(blockIdx.x, nh, off, cstart, chunk_h, k)) return;
    const int set = in.set(k.h);
    const int64_t shift = (int64_t)set * in.period;
    const double *__restrict__ x = in.x[set], *__restrict__ y = in.y[set], *__restrict__ z = in.z[set];
    __shared__ double sh[kRedParts - 2][32];
    __shared__ int cnt[2];
    if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
    double v[kRedParts - 2] = {0, 0, 0, 0, 0, 0, 0};
    int members = 0, odd = 0;
    for (int64_t r = k.b + threadIdx.x; r < k.e; r += blockDim.x) {
        const int64_t i = r - shift;
        if (in.mask && !in.mask[i]) continue;
        const double mi = in.m[i];
        if (SUMS) {
            v[0] += mi;
            v[1] += mi * x[i];
            v[2] += mi * y[i];
            v[3] += mi * z[i];
            v[4] += mi * in.vx[i];
            v[5] += mi * in.vy[i];
            v[6] += mi * in.vz[i];
        }
        ++members;
        const unsigned long long bits = (unsigned long long)__double_as_longlong(mi);
        if ((bits >> 63) || ((bits >> 52) & 0x7ff) == 0x7ff) ++odd;
    }
    __syncthreads();
    members = __reduce_add_sync(0xffffffffu, members);
    odd = __reduce_add_sync(0xffffffffu, odd);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&cnt[0], members);
        atomicAdd(&cnt[1], odd);
    }
    if (SUMS) bsum<kRedParts - 2>(v, sh);
    __syncthreads();
    double *p = part + (int64_t)blockIdx.x * kRedParts;
    if (threadIdx.x < kRedParts - 2) p[threadIdx.x] = SUMS ? sh[threadIdx.x][0] : 0.0;
    else if (threadIdx.x < kRedParts) p[threadIdx.x] = (double)cnt[threadIdx.x - (kRedParts - 2)];
}

// One thread per halo: the chunks' sums in order, centre, bulk velocity (or the caller's),
// reference mass and R05; rmax starts at 0 for the distance kernel's atomic maximum.  NaN in the caller's row is a value to
// be computed here; with SUMS = false, where no sums were formed, the row is complete and a NaN is its value.
template <bool SUMS>
__global__ void red_center_kernel(int nh, const int *__restrict__ cstart, const double *__restrict__ part,
                                  const double *__restrict__ about, Red *__restrict__ red) {
    for (int h = blockIdx.x * blockDim.x + threadIdx.x; h < nh; h += gridDim.x * blockDim.x) {
        double v[kRedParts] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int c = cstart[h]; c < cstart[h + 1]; ++c)
#pragma unroll
            for (int q = 0; q < kRedParts; ++q) v[q] += part[(int64_t)c * kRedParts + q];
        const double M = v[0];
        double cx = 0, cy = 0, cz = 0, ux = 0, uy = 0, uz = 0;
        if (M > 0) {
            cx = v[1] / M; cy = v[2] / M; cz = v[3] / M;
            ux = v[4] / M; uy = v[5] / M; uz = v[6] / M;
        }
        double Mref = M, r05_in = NAN;
        if (about) {
            const double *a = about + (int64_t)h * HALMA_ABOUT_NFIELDS;
            auto take = [&](double &v, int f) {
                if (!SUMS || !isnan(a[f])) v = a[f];
            };
            take(cx, HALMA_ABOUT_CX);
            take(cy, HALMA_ABOUT_CY);
            take(cz, HALMA_ABOUT_CZ);
            take(ux, HALMA_ABOUT_VX);
            take(uy, HALMA_ABOUT_VY);
            take(uz, HALMA_ABOUT_VZ);
            take(Mref, HALMA_ABOUT_MASS);
            r05_in = a[HALMA_ABOUT_R05];
        }
        Red o;
        o.M = M; o.cx = cx; o.cy = cy; o.cz = cz; o.vx = ux; o.vy = uy; o.vz = uz;
        o.rmax = 0.0; o.r05 = r05_in; o.sigma = 0; o.n = v[7]; o.mref = Mref; o.plain = v[8];
        red[h] = o;
    }
}

// What the members are sorted by inside a halo, in 63 bits: excluded particles after every finite distance, NaN last.
// A NaN may come with its sign set (infinity - infinity does), which has no place here: above the leading bits of
// the distance stands the halo.  (A minimum, not a mask: the compiler takes it for granted that a square root has none.)
__device__ __forceinline__ uint64_t full_key(double d, bool member) {
    const uint64_t bits = (uint64_t)__double_as_longlong(d);
    return !member ? 0x7ff0000000000000ull : bits < 0x7ff8000000000000ull ? bits : 0x7ff8000000000000ull;
}

// Per chunk: distances, sort keys (halo, leading dbits bits of the distance's bit pattern, which orders
// non-negative doubles) and the halo's R_max.
__global__ void __launch_bounds__(256) red_dist_kernel(int nh, const int64_t *__restrict__ off,
                                                       const int *__restrict__ cstart, const int *__restrict__ chunk_h,
                                                       RedIn in, int dbits, Red *__restrict__ red,
                                                       uint64_t *__restrict__ key, int *__restrict__ val,
                                                       double *__restrict__ dist) {
    Chunk k;
    if (!chunk_of(blockIdx.x, nh, off, cstart, chunk_h, k)) return;
    const int set = in.set(k.h);
    const int64_t shift = (int64_t)set * in.period;
    const double *__restrict__ x = in.x[set], *__restrict__ y = in.y[set], *__restrict__ z = in.z[set];
    const double cx = red[k.h].cx, cy = red[k.h].cy, cz = red[k.h].cz;
    double rmax = 0.0;
    for (int64_t r = k.b + threadIdx.x; r < k.e; r += blockDim.x) {
        const int64_t i = r - shift;
        const bool member = !in.mask || in.mask[i];
        const double dx = cx - x[i], dy = cy - y[i], dz = cz - z[i];
        // (dx**2 + dy**2 + dz**2)**0.5 as the reference evaluates it (halo_properties.py:104-107),
        // each operation rounded on its own so that d < R05 splits members the same way
        const double d = sqrt(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
        dist[r] = d;
        if (member) rmax = fmax(rmax, d);
        key[r] = (uint64_t)k.h << dbits | full_key(d, member) >> (63 - dbits);
        val[r] = (int)r;
    }
    __shared__ double shm[32];
    const double wm = wmax(rmax);
    if ((threadIdx.x & 31) == 0) shm[threadIdx.x >> 5] = wm;
    __syncthreads();
    if (threadIdx.x == 0) {
        double r = 0.0;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) r = fmax(r, shm[q]);
        // non-negative doubles order like their bit patterns
        atomicMax(reinterpret_cast<unsigned long long *>(&red[k.h].rmax), (unsigned long long)__double_as_longlong(r));
    }
}

// The sorted rows with the runs of equal keys in order of the full distance (equal distances stay in row
// order).  In a run of up to kShortRun rows, nearly all of them, a row goes to the run's start plus the number of
// rows before it.  Longer ones (members at one distance, on a shell, about a far centre) keep their
// order here, which the stable sort has made right where their distances are all the same; *longest is
// the length of the longest that has to be put in order (red_runs_kernel), run[p] a long run's start and length (0 elsewhere).
// Rows at no finite distance and excluded ones keep their place: what they are sorted by is one value.
// (Counted by every row, the masses of 2e6 members, a call without positions, took 3.9 s, now 11 ms with their copies.
// 100 haloes of 10,000 about a centre at 10^5 times their size, runs of up to 75 rows: 689 us with runs of up to 32 counted, 555
// with 128, 550 with 256; at 10^7 times, runs of up to 4,500, 1.28 ms with two blocks an SM in red_runs_kernel, 1.17 with four.
// 10 haloes of 30,000 at 10^7 times, up to 2,400: 695 us with 32, 710 with 128, 725 with 256, all with two blocks an SM.)
constexpr int kShortRun = 128;

__global__ void __launch_bounds__(256) red_ties_kernel(int n, const uint64_t *__restrict__ key,
                                                       const int *__restrict__ val, const double *__restrict__ dist,
                                                       const unsigned char *__restrict__ mask, int *__restrict__ order,
                                                       int2 *__restrict__ run, int *__restrict__ longest) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t k = key[p];
        const int i = val[p];
        int64_t to = p;
        int2 r = make_int2(0, 0);
        if ((p > 0 && key[p - 1] == k) || (p + 1 < n && key[p + 1] == k)) {
            const uint64_t fi = full_key(dist[i], !mask || mask[i]);
            if (fi < 0x7ff0000000000000ull) {
                // the run's first row and the one past its last: doubling steps away from p, then bisection
                int64_t lo = p, hi = p, step = 1;   // lo is in the run
                while (lo - step >= 0 && key[lo - step] == k) {
                    lo -= step;
                    step <<= 1;
                }
                for (; step > 0; step >>= 1)
                    if (lo - step >= 0 && key[lo - step] == k) lo -= step;
                step = 1;
                while (hi + step < n && key[hi + step] == k) {
                    hi += step;
                    step <<= 1;
                }
                for (; step > 0; step >>= 1)
                    if (hi + step < n && key[hi + step] == k) hi += step;
                ++hi;
                if (hi - lo <= kShortRun) {
                    to = lo;
                    for (int64_t q = lo; q < hi; ++q) {
                        const int j = val[q];
                        const uint64_t fj = full_key(dist[j], !mask || mask[j]);
                        if (fj < fi || (fj == fi && q < p)) ++to;
                    }
                } else {
                    r = make_int2((int)lo, (int)(hi - lo));
                    if (p > lo) {
                        const int j = val[p - 1];
                        if (full_key(dist[j], !mask || mask[j]) > fi) atomicMax(longest, r.y);
                    }
                }
            }
        }
        order[to] = i;
        run[p] = r;
    }
}

// The long runs in order: tiles of kRunTile rows by counting, then merges of neighbours twice as long each time, a row
// finding its place in the other half by bisection (n log^2 n steps in all, over the whole grid).  Nothing to do for nearly
// every call.  All rows of long runs lie at finite distances, which order as doubles.  (da, a) and (db, b): the rows'
// distances and numbers, from one to the other; order is a.  One cooperative launch, whose barriers separate the merges.
constexpr int kRunTile = 64;

__global__ void __launch_bounds__(256) red_runs_kernel(int n, const int *__restrict__ longest,
                                                       const int2 *__restrict__ run, const int *__restrict__ val,
                                                       const double *__restrict__ dist, double *da, int *a, double *db,
                                                       int *b) {
    const int most = *longest;
    if (most == 0) return;   // the same for the whole grid
    cooperative_groups::grid_group grid = cooperative_groups::this_grid();
    const int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    int merges = 0;
    while (((int64_t)kRunTile << merges) < most) ++merges;
    double *ds = merges & 1 ? db : da, *dd = merges & 1 ? da : db;   // the last merge ends in (da, a)
    int *is = merges & 1 ? b : a, *id = merges & 1 ? a : b;
    for (int64_t p = first; p < n; p += step) {
        const int2 r = run[p];
        if (r.y == 0) continue;
        const int64_t t0 = r.x + (p - r.x) / kRunTile * kRunTile, t1 = min(t0 + kRunTile, (int64_t)r.x + r.y);
        const int i = val[p];
        const double d = dist[i];
        int64_t to = t0;
        for (int64_t q = t0; q < t1; ++q) {
            const double e = dist[val[q]];
            if (e < d || (e == d && q < p)) ++to;
        }
        ds[to] = d;
        is[to] = i;
    }
    for (int64_t w = kRunTile; w < most; w <<= 1) {
        grid.sync();
        for (int64_t p = first; p < n; p += step) {
            const int2 r = run[p];
            if (r.y == 0) continue;
            const int64_t end_run = (int64_t)r.x + r.y, base = r.x + (p - r.x) / (2 * w) * (2 * w);
            const int64_t mid = min(base + w, end_run), end = min(base + 2 * w, end_run);
            const double d = ds[p];
            const bool left = p < mid;
            // rows of the other half before this one: smaller, or of the left half equal
            int64_t lo = left ? mid : base, hi = left ? end : mid;
            const int64_t from = lo;
            while (lo < hi) {
                const int64_t m = (lo + hi) >> 1;
                const double e = ds[m];
                if (left ? e < d : e <= d) lo = m + 1;
                else hi = m;
            }
            const int64_t to = base + (p - (left ? base : mid)) + (lo - from);
            dd[to] = d;
            id[to] = is[p];
        }
        double *const td = ds;
        ds = dd;
        dd = td;
        int *const ti = is;
        is = id;
        id = ti;
    }
}

// The half-mass walk's running sum (halo_properties.py:385-390: cumulative mass in increasing
// distance, compared with M/2 after every addition) is a chain of dependent FP64 adds, which
// GB300 runs at a small fraction of its integer rate.  For non-negative masses the walk keeps
// the sum as an integer number S of ulps of its binade [2^e, 2^(e+1)), ulp = 2^(e-52): while the
// sum stays in the binade, __dadd_rn(sum, m) equals (S + round(m / ulp)) * ulp, with m / ulp
// rounded to the nearest integer and a tie (a remainder of exactly half an ulp) going to the
// even sum.  So the adds are exact integer adds of per-mass increments that do not depend on
// the sum, except for the parity at a tie.  A step that leaves the binade (or starts from a sum
// that is zero or subnormal) is one __dadd_rn, after which the binade is read from the result.
struct SeqSum {
    double c;       // the sum (current only when !nrm; otherwise S * ulp)
    long long S;    // the sum in ulps of its binade, in [2^52, 2^53), when nrm
    long long hl;   // S > hl  <=>  sum > half
    int e;          // binade exponent
    bool nrm;       // the sum is a normal number
};

constexpr long long kTwo53 = 1ll << 53;

__device__ __forceinline__ void seq_set(SeqSum &q, double c, double half) {
    q.c = c;
    const unsigned long long b = (unsigned long long)__double_as_longlong(c);
    const int ef = (int)((b >> 52) & 0x7ff);
    q.nrm = ef != 0 && ef != 0x7ff && !(b >> 63);
    if (q.nrm) {
        q.e = ef - 1023;
        q.S = (long long)((b & 0xfffffffffffffull) | (1ull << 52));
        const double hs = ldexp(half, 52 - q.e);   // half in ulps of the binade (exact scaling)
        q.hl = !(hs < (double)kTwo53) ? kTwo53 : (hs < 0.0 ? -1ll : (long long)floor(hs));
    }
}

// m / ulp for ulp = 2^(e-52): integer part fl and the rounding of the remainder (0 below half
// an ulp, 1 above, 2 exactly half); big when m / ulp >= 2^53 could not be held.  m is finite,
// non-negative and has a clear sign bit.
__device__ __forceinline__ void mass_ulps(double m, int e, long long &fl, int &code, bool &big) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(m);
    const int ef = (int)(b >> 52);
    const unsigned long long M = (b & 0xfffffffffffffull) | (ef ? (1ull << 52) : 0ull);
    const int d = (e - 52) - (ef ? ef - 1075 : -1074);   // m = M * 2^(e - 52 - d)
    big = d < 0;
    if (d <= 0) {
        fl = (long long)M;
        code = 0;
    } else if (d >= 64) {
        fl = 0;
        code = 0;
    } else {
        fl = (long long)(M >> d);
        const unsigned long long rem = M & ((1ull << d) - 1ull), hb = 1ull << (d - 1);
        code = rem > hb ? 1 : (rem == hb ? 2 : 0);
    }
}

__device__ __forceinline__ long long inc_sum(long long S, long long fl, int code) {
    const long long base = S + fl;
    return base + (code == 1 ? 1 : (code == 2 ? (base & 1) : 0));
}

// One mass; true once the sum exceeds half.
__device__ __forceinline__ bool seq_add(SeqSum &q, double m, double half) {
    if (q.nrm) {
        long long fl;
        int code;
        bool big;
        mass_ulps(m, q.e, fl, code, big);
        const long long T = inc_sum(q.S, fl, code);
        if (!big && T < kTwo53) {
            q.S = T;
            return T > q.hl;
        }
        q.c = ldexp((double)q.S, q.e - 52);   // exact
    }
    seq_set(q, __dadd_rn(q.c, m), half);
    return q.c > half;
}

// Half-mass radius: walk the halo's members by increasing distance with the running sum;
// R05 is the distance of the last member before the sum first exceeds M/2 (the smallest
// distance if the first member already exceeds it, the largest if none does).  The block
// stages 1024 masses at a time in shared memory and sums the tile at once: every thread rounds four masses to
// ulps, and their sum gives the tile's end.  Only a tile that leaves the binade, holds a tie or crosses M/2 is
// taken by warp 0, 32 masses at a time in the same way, and of those only a batch with such a step is
// replayed one mass at a time by lane 0.  Bound: latency per tile (32 at a time throughout, 177 us for the
// 9,750 masses that a group of 19,500 members is walked).  Haloes with a
// negative, -0.0 or non-finite mass walk with plain __dadd_rn.
__global__ void __launch_bounds__(256) red_walk_kernel(const int64_t *__restrict__ off, const int *__restrict__ order,
                                                       const double *__restrict__ dist, RedIn in,
                                                       Red *__restrict__ red) {
    const int h = blockIdx.x;
    const int64_t b = off[h];
    const double *__restrict__ m = in.m - (int64_t)in.set(h) * in.period;
    const Red r = red[h];
    if (!isnan(r.r05)) return;   // caller supplied R05
    const int64_t nmem = (int64_t)r.n;
    const double half = 0.5 * r.mref;
    const int lane = threadIdx.x & 31;
    __shared__ double tile[2][1024];   // the next one's masses are written before this one is walked
    __shared__ long long first;
    if (threadIdx.x == 0) first = LLONG_MAX;
    SeqSum q;   // lane 0's state (warp 0)
    q.c = 0.0;
    q.nrm = false;
    q.S = 0;
    q.hl = 0;
    q.e = 0;
    const bool plain = r.plain != 0.0;
    __shared__ long long wsums[8];
    __shared__ int wodd[8], state;   // state: the sum's binade exponent, or kNoBinade; after a tile, whether it was taken
    constexpr int kNoBinade = INT_MIN;
    for (int i = threadIdx.x; i < (nmem < 1024 ? (int)nmem : 1024); i += blockDim.x) tile[0][i] = m[order[b + i]];
    if (threadIdx.x == 0) state = kNoBinade;
    __syncthreads();
    int cur = 0;
    for (int64_t k0 = 0; k0 < nmem; k0 += 1024, cur ^= 1) {
        const int cnt = nmem - k0 < 1024 ? (int)(nmem - k0) : 1024;
        // the next tile's masses, on their way while this one is summed
        double next[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t i = k0 + 1024 + u * 256 + threadIdx.x;
            next[u] = i < nmem ? m[order[b + i]] : 0.0;
        }
        // the whole tile at once, four masses a thread, when the sum stays short of half and of its binade's end
        const int e = state;
        long long inc = 0;
        bool odd = false;
        if (!plain && e != kNoBinade) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = u * 256 + threadIdx.x;
                if (i >= cnt) continue;
                long long fl;
                int code;
                bool big;
                mass_ulps(tile[cur][i], e, fl, code, big);
                odd |= big || code == 2 || fl > (1ll << 51);   // inc < 1024 * 2^51: no overflow
                inc += fl + (code == 1 ? 1 : 0);
            }
        }
        odd = __any_sync(0xffffffffu, odd);
        for (int o = 16; o > 0; o >>= 1) inc += __shfl_xor_sync(0xffffffffu, inc, o);
        if (lane == 0) {
            wsums[threadIdx.x >> 5] = inc;
            wodd[threadIdx.x >> 5] = odd;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) tile[cur ^ 1][u * 256 + threadIdx.x] = next[u];
        __syncthreads();
        if (threadIdx.x == 0) {
            long long T = q.S;
            bool any = plain || e == kNoBinade;
            for (int u = 0; u < 8; ++u) {
                T += wsums[u];
                any |= wodd[u] != 0;
            }
            const bool taken = !any && q.nrm && T < kTwo53 && T <= q.hl;
            if (taken) q.S = T;
            state = taken;
        }
        __syncthreads();
        const bool took = state != 0;
        __syncthreads();   // every thread has read state, which is written again below
        if (took) {
            if (threadIdx.x == 0) state = e;
            __syncthreads();
            continue;
        }
        if (threadIdx.x < 32) {
            long long f = LLONG_MAX;
            for (int q0 = 0; q0 < cnt && f == LLONG_MAX; q0 += 32) {
                const int nb = min(32, cnt - q0);
                bool replay = true;
                if (!plain) {
                    // lane 0's binade, broadcast; a batch from a non-normal sum is replayed
                    const int nrm = __shfl_sync(0xffffffffu, (int)q.nrm, 0);
                    if (nrm) {
                        const int e = __shfl_sync(0xffffffffu, q.e, 0);
                        long long fl = 0;
                        int code = 0;
                        bool big = false;
                        if (lane < nb) mass_ulps(tile[cur][q0 + lane], e, fl, code, big);
                        // increments without ties; a tie or a big mass forces the replay
                        const bool odd = big || code == 2;
                        long long inc = fl + (code == 1 ? 1 : 0);
                        for (int o = 16; o > 0; o >>= 1) inc += __shfl_xor_sync(0xffffffffu, inc, o);
                        if (!__any_sync(0xffffffffu, odd) && lane == 0) {
                            const long long T = q.S + inc;   // no overflow: inc < 32 * 2^53
                            if (T < kTwo53 && T <= q.hl) {
                                q.S = T;
                                replay = false;
                            }
                        }
                        replay = __shfl_sync(0xffffffffu, (int)replay, 0);
                    }
                }
                if (replay && lane == 0) {
                    for (int u = 0; u < nb; ++u) {
                        const bool over = plain ? ((q.c = __dadd_rn(q.c, tile[cur][q0 + u])) > half)
                                                : seq_add(q, tile[cur][q0 + u], half);
                        if (over) {
                            f = k0 + q0 + u;
                            break;
                        }
                    }
                }
                f = __shfl_sync(0xffffffffu, f, 0);
            }
            if (lane == 0) {
                if (f != LLONG_MAX) first = f;
                state = q.nrm ? q.e : kNoBinade;
            }
        }
        __syncthreads();
        if (first != LLONG_MAX) break;
    }
    if (threadIdx.x == 0) {
        double r05 = 0.0;
        if (nmem > 0) {
            const long long f = first == LLONG_MAX ? -1 : first;
            if (f > 0) r05 = dist[order[b + f - 1]];
            else if (f == 0) r05 = dist[order[b]];
            else r05 = dist[order[b + nmem - 1]];
        }
        red[h].r05 = r05;
    }
}

// Per chunk: sum of |v - v_bulk|^2 and count of the members closer than R05.
__global__ void __launch_bounds__(256) red_sigma_kernel(int nh, const int64_t *__restrict__ off,
                                                        const int *__restrict__ cstart, const int *__restrict__ chunk_h,
                                                        const double *__restrict__ dist, RedIn in,
                                                        const Red *__restrict__ red, double *__restrict__ part) {
    Chunk k;
    if (!chunk_of(blockIdx.x, nh, off, cstart, chunk_h, k)) return;
    const Red r = red[k.h];
    const int64_t shift = (int64_t)in.set(k.h) * in.period;
    __shared__ double sh[2][32];
    double v[2] = {0, 0};
    const int64_t e = in.set(k.h) > 0 ? k.b : k.e;   // of sets, the first alone is asked for its dispersion
    for (int64_t q = k.b + threadIdx.x; q < e; q += blockDim.x) {
        const int64_t i = q - shift;
        if (in.mask && !in.mask[i]) continue;
        if (dist[q] < r.r05) {
            const double dx = in.vx[i] - r.vx, dy = in.vy[i] - r.vy, dz = in.vz[i] - r.vz;
            v[0] += dx * dx + dy * dy + dz * dz;
            v[1] += 1.0;
        }
    }
    bsum<2>(v, sh);
    if (threadIdx.x < 2) part[(int64_t)blockIdx.x * 2 + threadIdx.x] = v[threadIdx.x];
}

__global__ void red_out_kernel(int nh, const int *__restrict__ cstart, const double *__restrict__ part,
                               const Red *__restrict__ red, double *__restrict__ out) {
    for (int h = blockIdx.x * blockDim.x + threadIdx.x; h < nh; h += gridDim.x * blockDim.x) {
        const Red r = red[h];
        double s = 0.0, c = 0.0;
        for (int k = cstart[h]; k < cstart[h + 1]; ++k) {
            s += part[(int64_t)k * 2];
            c += part[(int64_t)k * 2 + 1];
        }
        double *o = out + (int64_t)h * HALMA_RED_NFIELDS;
        o[HALMA_RED_MASS] = r.M;
        o[HALMA_RED_CX] = r.cx; o[HALMA_RED_CY] = r.cy; o[HALMA_RED_CZ] = r.cz;
        o[HALMA_RED_VX] = r.vx; o[HALMA_RED_VY] = r.vy; o[HALMA_RED_VZ] = r.vz;
        o[HALMA_RED_RMAX] = r.rmax;
        o[HALMA_RED_R05] = r.r05;
        o[HALMA_RED_SIGMA] = c > 0 ? sqrt(s / 3.0 / c) : 0.0;
        o[HALMA_RED_N] = r.n;
    }
}

int launch_runs(int n, const int *longest, const int2 *run, const int *val, const double *dist, double *da, int *a,
                double *db, int *b, cudaStream_t st) {
    const int grid = std::min(device_sm_count() * 4, grid_for(n, 256));   // all blocks are on the GPU at once (five an SM fit)
    void *args[] = {&n, &longest, &run, &val, &dist, &da, &a, &db, &b};
    HALMA_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void *>(&red_runs_kernel), dim3((unsigned)grid), dim3(256), args,
                                           0, st));
    count_launch();
    return HALMA_OK;
}

}  // namespace

static int reductions_run(int64_t n, int nh, const int64_t *off, const RedIn &in, bool sums,
                          const double *about, double *out, cudaStream_t st) {
    if (nh <= 0) return HALMA_OK;
    const int N = (int)std::max<int64_t>(n, 1);
    const int cmax = nh + (int)(n / kRedChunk) + 1;   // chunks: sum over haloes of max(1, ceil(n_h / kRedChunk))
    int hbits = 1;
    while (hbits < 32 && ((uint64_t)(nh - 1) >> hbits) != 0) ++hbits;
    // Whole radix digits (8 bits), at least 11 bits of exponent and as many of mantissa as number the members, 26 at most:
    // then even the members of one octave of one halo seldom share a key, and red_ties_kernel orders those that do.  (26 for
    // all: one more pass, 22 us of the 1.6e6 rows of four half-mass radii of 4e5 members; one set of 120 haloes 333 us, now 306.)
    const int64_t members = in.period > 0 ? in.period : n;
    int mbits = 8;
    while (mbits < 26 && (members >> mbits) != 0) ++mbits;
    const int kbits = std::min(64, (hbits + 11 + mbits + 7) / 8 * 8), dbits = std::min(63, kbits - hbits);
    const size_t s64 = sort_pairs_u64_i32_bytes(N, hbits + dbits), sc = exclusive_sum_i32_bytes(nh + 1);
    Layout L;
    const size_t o_red = L.add(sizeof(Red) * nh);
    const size_t o_k = L.add(8ull * N), o_k2 = L.add(8ull * N), o_dist = L.add(8ull * N);
    const size_t o_v0 = L.add(4ull * N), o_v1 = L.add(4ull * N);
    const size_t o_cnum = L.add(4ull * (nh + 1)), o_cst = L.add(4ull * (nh + 1)), o_ch = L.add(4ull * cmax);
    const size_t o_part = L.add(8ull * kRedParts * cmax), o_part2 = L.add(16ull * cmax);
    const size_t o_run = L.add(8ull * N), o_long = L.add(4);
    // of the sort, and afterwards of the long runs' merges
    const size_t merge_d = align_up(8ull * N, 256);
    const size_t o_tmp = L.add(std::max(std::max(s64, sc), merge_d + sizeof(int) * (size_t)N));
    void *base = nullptr;
    HALMA_TRY(workspace(L.total, &base, st));
    Red *red = at<Red>(base, o_red);
    auto *key = at<uint64_t>(base, o_k), *key2 = at<uint64_t>(base, o_k2);
    auto *dist = at<double>(base, o_dist);
    auto *v0 = at<int>(base, o_v0), *v1 = at<int>(base, o_v1);
    int *cnum = at<int>(base, o_cnum), *cst = at<int>(base, o_cst), *chunk_h = at<int>(base, o_ch);
    double *part = at<double>(base, o_part), *part2 = at<double>(base, o_part2);
    void *tmp = at<void>(base, o_tmp);
    const int gh = grid_for(nh + 1, 256);
    auto *run = at<int2>(base, o_run);
    int *longest = at<int>(base, o_long);
    HALMA_LAUNCH(red_chunks_kernel, gh, 256, 0, st, nh, off, cnum, longest);
    HALMA_TRY(exclusive_sum_i32(tmp, sc, cnum, cst, nh + 1, st));
    HALMA_LAUNCH(red_owner_kernel, gh, 256, 0, st, nh, cst, chunk_h);
    if (sums) {
        HALMA_LAUNCH(red_part_kernel<true>, cmax, 256, 0, st, nh, off, cst, chunk_h, in, part);
        HALMA_LAUNCH(red_center_kernel<true>, gh, 256, 0, st, nh, cst, part, about, red);
    } else {
        HALMA_LAUNCH(red_part_kernel<false>, cmax, 256, 0, st, nh, off, cst, chunk_h, in, part);
        HALMA_LAUNCH(red_center_kernel<false>, gh, 256, 0, st, nh, cst, part, about, red);
    }
    HALMA_LAUNCH(red_dist_kernel, cmax, 256, 0, st, nh, off, cst, chunk_h, in, dbits, red, key, v0, dist);
    if (n > 0) {
        HALMA_TRY(sort_pairs_u64_i32(tmp, s64, key, key2, v0, v1, (int)n, hbits + dbits, st));
        HALMA_LAUNCH(red_ties_kernel, std::min(device_sm_count() * 8, grid_for(n, 256)), 256, 0, st, (int)n, key2, v1,
                     dist, in.mask, v0, run, longest);
        HALMA_TRY(launch_runs((int)n, longest, run, v1, dist, reinterpret_cast<double *>(key), v0, at<double>(base, o_tmp),
                              at<int>(base, o_tmp + merge_d), st));
    }
    HALMA_LAUNCH(red_walk_kernel, nh, 256, 0, st, off, v0, dist, in, red);
    HALMA_LAUNCH(red_sigma_kernel, cmax, 256, 0, st, nh, off, cst, chunk_h, dist, in, red, part2);
    HALMA_LAUNCH(red_out_kernel, gh, 256, 0, st, nh, cst, part2, red, out);
    return HALMA_OK;
}

int reductions_device(int64_t n, int nh, const int64_t *off, const double *x, const double *y, const double *z,
                      const double *vx, const double *vy, const double *vz, const double *m,
                      const unsigned char *mask, const double *about, double *out, cudaStream_t st) {
    const RedIn in{{x}, {y}, {z}, vx, vy, vz, m, mask, 0, 1};
    return reductions_run(n, nh, off, in, true, about, out, st);
}

// The same for kRedSets sets of positions over the same n members of nh haloes, in one run: off has kRedSets * nh + 1
// entries (set s, halo h: s * n + the member offset), about and out kRedSets * nh rows, about complete but for
// R05.  out holds R05 and R_max, and sigma for the first set; the sums that about replaces are not formed.  One run
// keeps four times as many walks in flight: 120 groups of 4e5 members took 4 x 0.17 ms for them, now 0.14.
int reductions_sets_device(int64_t n, int nh, const int64_t *off, const double *const (*pos)[3], const double *vx,
                           const double *vy, const double *vz, const double *m, const double *about, double *out,
                           cudaStream_t st) {
    RedIn in{};
    for (int s = 0; s < kRedSets; ++s) {
        in.x[s] = pos[s][0];
        in.y[s] = pos[s][1];
        in.z[s] = pos[s][2];
    }
    in.vx = vx;
    in.vy = vy;
    in.vz = vz;
    in.m = m;
    in.period = n;
    in.hp = nh;
    return reductions_run(kRedSets * n, kRedSets * nh, off, in, false, about, out, st);
}

}  // namespace halma

using namespace halma;

extern "C" int halma_halo_reductions(int64_t n, int64_t n_haloes, const int64_t *offsets, const double *x,
                                     const double *y, const double *z, const double *vx, const double *vy,
                                     const double *vz, const double *m, const uint8_t *mask, const double *about_, double *out,
                                     halma_stream_t stream) {
    if (n < 0 || n_haloes < 0) return fail(HALMA_ERR_INVALID, "negative size");
    if (n >= (1ll << 31) - 1 || n_haloes >= (1ll << 31) - 1) return fail(HALMA_ERR_CAPACITY, "too many particles or haloes");
    if (n_haloes == 0) return HALMA_OK;
    if (!offsets || !out || (n > 0 && (!x || !y || !z || !vx || !vy || !vz || !m)))
        return fail(HALMA_ERR_INVALID, "null pointer");
    cudaStream_t st = (cudaStream_t)stream;
    // the segments must cover the n rows in order (checked on the host: the kernels size
    // their chunk table from n, index the rows through the offsets and sort all n rows by
    // the halo each belongs to)
    {
        std::vector<int64_t> h_off(n_haloes + 1);
        if (is_device_pointer(offsets)) {
            HALMA_CUDA(cudaMemcpyAsync(h_off.data(), offsets, 8ull * (n_haloes + 1), cudaMemcpyDeviceToHost, st));
            HALMA_CUDA(cudaStreamSynchronize(st));
        } else {
            memcpy(h_off.data(), offsets, 8ull * (n_haloes + 1));
        }
        if (h_off[0] != 0 || h_off[n_haloes] != n) return fail(HALMA_ERR_INVALID, "halo offsets must run from 0 to n");
        for (int64_t h = 0; h < n_haloes; ++h)
            if (h_off[h + 1] < h_off[h]) return fail(HALMA_ERR_INVALID, "halo offsets must not decrease");
    }
    std::lock_guard<std::mutex> guard(api_mutex());
    Stager sg;
    const int64_t *off = nullptr;
    const double *dx = nullptr, *dy = nullptr, *dz = nullptr, *dvx = nullptr, *dvy = nullptr, *dvz = nullptr,
                 *dm = nullptr;
    const uint8_t *dmask = nullptr;
    double *dout = nullptr;
    sg.add(offsets, n_haloes + 1, true, false, &off);
    sg.add(x, n, true, false, &dx);
    sg.add(y, n, true, false, &dy);
    sg.add(z, n, true, false, &dz);
    sg.add(vx, n, true, false, &dvx);
    sg.add(vy, n, true, false, &dvy);
    sg.add(vz, n, true, false, &dvz);
    sg.add(m, n, true, false, &dm);
    sg.add(mask, mask ? n : 0, true, false, &dmask);
    const double *dabout = nullptr;
    sg.add(about_, about_ ? n_haloes * HALMA_ABOUT_NFIELDS : 0, true, false, &dabout);
    sg.add((const double *)out, n_haloes * HALMA_RED_NFIELDS, false, true, &dout);
    void *stage = nullptr;
    if (sg.any_host) {
        Layout L;
        sg.plan(L);
        HALMA_CUDA(cudaMallocAsync(&stage, L.total, st));
    }
    int s = sg.bind_and_upload(stage, st);
    if (s == HALMA_OK)
        s = reductions_device(n, (int)n_haloes, off, dx, dy, dz, dvx, dvy, dvz, dm, dmask, dabout, dout, st);
    if (s == HALMA_OK) s = sg.download(st);
    if (stage) {
        cudaFreeAsync(stage, st);
        cudaStreamSynchronize(st);
    }
    return s;
}
