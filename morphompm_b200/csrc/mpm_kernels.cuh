// Kernels of one MLS-MPM growth step and of its reverse.
//
// Forward (python/morphompm/transfer.py:33-79):
//   bin_kernel        cell key of every particle (stencil base, exact rounding)
//   cluster sort      (cluster_sort.cuh) small plans: sorted order, segments and
//                     active tiles in one launch, instead of the next three
//   radix sort        (sort.cuh) cell-sorted particle order, deterministic
//   seg_* kernels     segment table of the occupied cells + active tile flags
//   compact_tiles     active node tiles -> compact grid slots
//   prepass_kernel    stress and the P2G record of every particle (particle order);
//                     in a chain of steps the previous G2P forms them instead
//   cell_sums_kernel  P2G phase 1: per occupied cell, its 27 stencil sums, from
//                     records staged in shared memory
//   node_sums_kernel  P2G phase 2: per node, the sums of its 27 source cells
//                     in a fixed order, + grid update with boundary conditions
//   g2p_kernel        gather, advect, F update; clears the cell marks; in a
//                     chain also bins the new state and forms its P2G records
// Reverse (python/morphompm/transfer.py:82-158):
//   cell_sums<ADJ>    gv_b scatter phase 1 (nv_b, Cn_b' formed per particle)
//   node_sums<1>      gv_b gather + grid adjoint (gmom_b, gm_b)
//   bwd_particle_kernel  P2G adjoint, constitutive VJP, volume path, x_b terms
//
// P2G determinism: particles are sorted by cell, every occupied cell's sums
// are formed in sorted particle order (one thread per x-offset of the stencil), and every node adds its
// source cells in the fixed order of the stencil offsets.  No atomics, no
// shared-memory races: the result does not depend on scheduling.
#pragma once

#include <limits.h>

#include "mpm_common.cuh"
#include "constitutive.cuh"

namespace mpm {

constexpr int PAYLOAD = 16;   // fx[3], m, a[3], B[9]

template <typename R> struct Vec4;
template <> struct Vec4<float> { using T = float4; };
template <> struct Vec4<double> { using T = double2; };

template <typename R>
__device__ __forceinline__ void load_record(const R* __restrict__ base, long long q, R r[PAYLOAD]) {
    using V = typename Vec4<R>::T;
    const V* p = reinterpret_cast<const V*>(base + q * PAYLOAD);
    constexpr int per = sizeof(V) / sizeof(R);
#pragma unroll
    for (int i = 0; i < PAYLOAD / per; ++i) {
        V v = __ldg(p + i);
        const R* e = reinterpret_cast<const R*>(&v);
#pragma unroll
        for (int k = 0; k < per; ++k) r[i * per + k] = e[k];
    }
}
template <typename R>
__device__ __forceinline__ void store_record(R* __restrict__ base, long long q, const R r[PAYLOAD]) {
    using V = typename Vec4<R>::T;
    V* p = reinterpret_cast<V*>(base + q * PAYLOAD);
    constexpr int per = sizeof(V) / sizeof(R);
#pragma unroll
    for (int i = 0; i < PAYLOAD / per; ++i) {
        V v;
        R* e = reinterpret_cast<R*>(&v);
#pragma unroll
        for (int k = 0; k < per; ++k) e[k] = r[i * per + k];
        p[i] = v;
    }
}
template <typename R>
__device__ __forceinline__ void load_node(const R* __restrict__ g, long long idx, R o[4]) {
    if constexpr (sizeof(R) == 4) {
        float4 v = __ldg(reinterpret_cast<const float4*>(g) + idx);
        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    } else {
        const double2* p = reinterpret_cast<const double2*>(g) + 2 * idx;
        double2 a = __ldg(p), b = __ldg(p + 1);
        o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
    }
}
template <typename R>
__device__ __forceinline__ void store_node(R* __restrict__ g, long long idx, const R o[4]) {
    if constexpr (sizeof(R) == 4) {
        reinterpret_cast<float4*>(g)[idx] = make_float4(o[0], o[1], o[2], o[3]);
    } else {
        double2* p = reinterpret_cast<double2*>(g) + 2 * idx;
        p[0] = make_double2(o[0], o[1]);
        p[1] = make_double2(o[2], o[3]);
    }
}

template <typename R>
__device__ __forceinline__ bool node_free(const SceneK<R>& sc, int i, int j, int k) {
    if (sc.wall > 0) {
        int w = sc.wall;
        if (i < w || j < w || k < w || i >= sc.shape[0] - w || j >= sc.shape[1] - w || k >= sc.shape[2] - w)
            return false;
    }
    if (sc.clamp_lo[0] < sc.clamp_hi[0] && sc.clamp_lo[1] < sc.clamp_hi[1] && sc.clamp_lo[2] < sc.clamp_hi[2]) {
        if (i >= sc.clamp_lo[0] && i < sc.clamp_hi[0] && j >= sc.clamp_lo[1] && j < sc.clamp_hi[1] &&
            k >= sc.clamp_lo[2] && k < sc.clamp_hi[2])
            return false;
    }
    return true;
}

// The growth law's factor of particle p at step t (growth_mode 1: Fg = g I),
// and its derivative d g / d A
template <typename R>
__device__ __forceinline__ R growth_factor(const Ctx& ctx, const SceneK<R>& sc, long long p, int t, R& gphi) {
    const R phi = ctx.phi ? static_cast<const R*>(ctx.phi)[p] : R(1);
    const double ramp = growth_ramp(sc, t);
    gphi = (R)ramp * phi;
    return R(1) + (R)(sc.growth_A * ramp) * phi;
}

// Fg of particle p (read, or the growth law)
template <typename R>
__device__ __forceinline__ void load_Fg(const Ctx& ctx, const SceneK<R>& sc, const MpmParticles& P, long long p,
                                        int t, R Fg[9], R& gphi) {
    if (sc.growth_mode == 1) {
        const R g = growth_factor(ctx, sc, p, t, gphi);
#pragma unroll
        for (int i = 0; i < 9; ++i) Fg[i] = (i % 4 == 0) ? g : R(0);
    } else {
        ld9<R>(P.Fg, p, P.sp9, P.sc9, Fg);
        gphi = R(0);
    }
}

// Growth of a particle in the form a kernel is compiled for: ISO (every scene
// of the plan follows its growth law) keeps g alone.
template <typename R, bool ISO> struct Growth;
template <typename R> struct Growth<R, true> {
    GrowthIso<R> g;
    __device__ __forceinline__ void load(const Ctx& ctx, const SceneK<R>& sc, const MpmParticles&, long long p, int t,
                                         R& gphi) {
        g.g = growth_factor(ctx, sc, p, t, gphi);
    }
};
template <typename R> struct Growth<R, false> {
    GrowthFull<R> g;
    __device__ __forceinline__ void load(const Ctx& ctx, const SceneK<R>& sc, const MpmParticles& P, long long p,
                                         int t, R& gphi) {
        load_Fg(ctx, sc, P, p, t, g.Fg, gphi);
    }
};

// ---------------------------------------------------------------------------
// binning
// ---------------------------------------------------------------------------
// Active tiles of the next step: the node tiles that the stencil of a particle
// inside the grid touches (nodes base..base+2 clipped to the grid), flagged
// where its cell key is formed.  Every particle of an occupied cell flags the
// same tiles; the flags are plain stores of 1.
template <typename R>
__device__ __forceinline__ void flag_stencil_tiles(const Ctx& ctx, const SceneK<R>& sc, const SceneAux& ax,
                                                   const int base[3]) {
    int tlo[3], thi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int sh = d == 2 ? ctx.tile_z_shift : ctx.tile_xy_shift;
        const int lo = base[d] < 0 ? 0 : base[d];
        const int hi = base[d] + 2 > sc.shape[d] - 1 ? sc.shape[d] - 1 : base[d] + 2;
        tlo[d] = lo >> sh;
        thi[d] = hi >> sh;
    }
    // three nodes lie in at most two tiles per axis (tiles have 4 nodes or more):
    // up to eight stores, without a loop (over lo..hi per axis: binning of 4.7M
    // particles 56 us, now 42; emitting G2P 382, now 356; with a test of the flag
    // before the store 83 and 430)
    const int n1 = ax.ntile[1], n2 = ax.ntile[2];
    const long long t0 = ax.tile_begin + ((tlo[0] * n1 + tlo[1]) * n2 + tlo[2]);
    const bool two[3] = {thi[0] > tlo[0], thi[1] > tlo[1], thi[2] > tlo[2]};
#pragma unroll
    for (int o = 0; o < 8; ++o) {
        const int a = o >> 2, b = (o >> 1) & 1, c = o & 1;
        if ((a && !two[0]) || (b && !two[1]) || (c && !two[2])) continue;
        const long long ti = t0 + ((a * n1 + b) * n2 + c);
        if (MPM_INB(ti, ctx.n_tiles, 1)) ctx.tile_flag[ti] = 1;
    }
}

// Cell key of a particle at x (its padded stencil-base cell, or the scene's
// "outside" key) and its fractional position fx in the stencil; flags the tiles
// of a particle inside.
template <typename R>
__device__ __forceinline__ unsigned particle_key(const Ctx& ctx, const SceneK<R>& sc, const SceneAux& ax,
                                                 const R x[3], R fx[3]) {
    int base[3];
    const bool inside = bin_particle(x, sc.inv_dx, sc.shape, base, fx);
    // a scene's padded cells fit 32 bits; an outside particle's value is not used
    const unsigned cell = ((unsigned)(base[0] + 2) * (unsigned)(sc.shape[1] + 2) + (unsigned)(base[1] + 2)) *
                              (unsigned)(sc.shape[2] + 2) + (unsigned)(base[2] + 2);
    // the lanes of a warp in the same cell flag the same tiles: one of them does
    const unsigned tag = inside ? (unsigned)(ax.cell_begin + cell) : 0xffffffffu;
    const unsigned peers = __match_any_sync(__activemask(), tag);
    const bool leader = (peers & ((1u << (threadIdx.x & 31)) - 1u)) == 0u;
    if (inside) {
        if (leader) flag_stencil_tiles(ctx, sc, ax, base);
        return tag;
    }
    raise_status(ctx.status, MPM_WARN_OUTSIDE);
    return (unsigned)(ax.cell_begin + ax.ncells);
}

template <typename R>
__global__ void __launch_bounds__(256)
bin_kernel(Ctx ctx, MpmParticles P, unsigned* __restrict__ keys) {
    long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= ctx.n) return;
    int s = ctx.scene_of[p];
    R x[3], fx[3];
    ld3<R>(P.x, p, P.sp3, P.sc3, x);
    keys[p] = particle_key<R>(ctx, static_cast<const SceneK<R>*>(ctx.sk)[s], ctx.aux[s], x, fx);
}

// keys of a single scene (C ABI mpm_bin_keys); local keys, no plan
template <typename R>
__global__ void bin_keys_single(MpmScene sc, long long n, const R* __restrict__ x, int* __restrict__ keys) {
    long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    R xp[3] = {x[3 * p], x[3 * p + 1], x[3 * p + 2]};
    int base[3];
    R fx[3];
    bool inside = bin_particle(xp, (R)(1.0 / sc.dx), sc.shape, base, fx);
    long long P0 = sc.shape[0] + 2, P1 = sc.shape[1] + 2, P2 = sc.shape[2] + 2;
    keys[p] = inside ? (int)(((base[0] + 2) * P1 + (base[1] + 2)) * P2 + (base[2] + 2)) : (int)(P0 * P1 * P2);
}

// ---------------------------------------------------------------------------
// segment tables: one segment per occupied cell (a run of equal sorted keys).
// Three kernels: per-block counts of segment starts, a
// single-block scan of the counts, and the writes of seg_first / seg_last /
// cell_seg with each slot's segment id from the scan.  "Outside" keys (stencil
// entirely off the grid) form no segment.
// ---------------------------------------------------------------------------
constexpr int SEG_THREADS = 256;

// Segment kernels: SEGK_ITEMS warp-striped rounds of slots per block (slot =
// block base + round*256 + thread, every key load coalesced), all their loads
// issued before any is used, few registers: a block waits on one chain of
// memory latencies (key, then its scene), not one per round.
#ifndef MPM_SEGK_ITEMS          // slots per thread (build-time; 4 measured fastest of 1, 2, 4, 8)
#define MPM_SEGK_ITEMS 4
#endif
constexpr int SEGK_ITEMS = MPM_SEGK_ITEMS;
constexpr int SEGK_TILE = SEG_THREADS * SEGK_ITEMS;

// Bit r of start / last: slot base + r*256 + thread starts / ends an inside
// segment (a run of equal keys whose cell lies in its scene's grid).
__device__ __forceinline__ void seg_flags(const Ctx& ctx, const unsigned* __restrict__ skeys, long long base,
                                          unsigned key[SEGK_ITEMS], unsigned& start, unsigned& last) {
    const int lane = threadIdx.x & 31;
    const long long n = ctx.n;
    unsigned edge[SEGK_ITEMS];
    int sid[SEGK_ITEMS];
#pragma unroll
    for (int r = 0; r < SEGK_ITEMS; ++r) {
        const long long s = base + (long long)r * SEG_THREADS + threadIdx.x;
        const bool valid = s < n;
        key[r] = valid ? skeys[s] : 0u;
        sid[r] = valid ? ctx.scene_of[s] : 0;
        // lane 0 needs the key before it, lane 31 the key after it
        const long long e = lane == 0 ? s - 1 : s + 1;
        edge[r] = ((lane == 0 || lane == 31) && e >= 0 && e < n) ? skeys[e] : 0u;
    }
    start = 0;
    last = 0;
#pragma unroll
    for (int r = 0; r < SEGK_ITEMS; ++r) {
        const long long s = base + (long long)r * SEG_THREADS + threadIdx.x;
        unsigned prv = __shfl_up_sync(0xffffffffu, key[r], 1);
        unsigned nxt = __shfl_down_sync(0xffffffffu, key[r], 1);
        if (lane == 0) prv = edge[r];
        if (lane == 31) nxt = edge[r];
        const bool valid = s < n;
        const bool a = valid && (s == 0 || prv != key[r]);
        const bool b = valid && (s == n - 1 || nxt != key[r]);
        if (a || b) {
            const SceneAux& ax = ctx.aux[sid[r]];
            if ((long long)key[r] - ax.cell_begin < ax.ncells) {
                start |= (a ? 1u : 0u) << r;
                last |= (b ? 1u : 0u) << r;
            }
        }
    }
}

__global__ void __launch_bounds__(SEG_THREADS)
seg_count_kernel(Ctx ctx, const unsigned* __restrict__ skeys) {
    __shared__ unsigned red[SEG_THREADS / 32];
    unsigned key[SEGK_ITEMS], start, last;
    seg_flags(ctx, skeys, (long long)blockIdx.x * SEGK_TILE, key, start, last);
    unsigned cnt = __popc(start);
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = 0;
        for (int w = 0; w < SEG_THREADS / 32; ++w) t += red[w];
        ctx.blk_count[blockIdx.x] = t;
    }
}

// exclusive scan of per-block counts in place (single block of 1024 threads);
// the total, clamped to cap, goes to *total (a total above cap raises
// MPM_ERR_ARG).  Each thread sums a run of consecutive counts, the runs are
// scanned by warp shuffles and one pass over the 32 warp sums.
__global__ void __launch_bounds__(1024)
scan_counts_kernel(unsigned* __restrict__ cnt, int nblk, int* __restrict__ total, int cap, int* __restrict__ status) {
    __shared__ unsigned wsum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (nblk + 1023) / 1024;
    const long long b0 = (long long)threadIdx.x * per;
    unsigned loc = 0;
    for (int j = 0; j < per; ++j)
        if (b0 + j < nblk) loc += cnt[b0 + j];
    unsigned inc = loc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const unsigned w = wsum[lane];
        unsigned wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        wsum[lane] = wi - w;
    }
    __syncthreads();
    unsigned run = wsum[warp] + inc - loc;
    for (int j = 0; j < per; ++j) {
        if (b0 + j < nblk) {
            const unsigned v = cnt[b0 + j];
            cnt[b0 + j] = run;
            run += v;
        }
    }
    if (threadIdx.x == 1023) {       // its run ends at the grand total
        unsigned c = run;
        if (c > (unsigned)cap) {
            raise_status(status, MPM_ERR_ARG);
            c = (unsigned)cap;
        }
        *total = (int)c;
    }
}

// exclusive scan, in place, of a block's E (round, warp) counts (round-major;
// warp 0, E / 32 per lane, or one per lane for E <= 32); call from all threads
template <int E>
__device__ __forceinline__ void scan_round_warp_counts(unsigned* pre) {
    static_assert(E <= 32 || E % 32 == 0, "E <= 32 or a multiple of 32");
    constexpr int PER = E <= 32 ? 1 : E / 32;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    if ((threadIdx.x >> 5) == 0) {
        unsigned v[PER], tot = 0;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            v[j] = PER * lane + j < E ? pre[PER * lane + j] : 0u;
            tot += v[j];
        }
        unsigned inc = tot;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        unsigned ex = inc - tot;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            if (PER * lane + j < E) pre[PER * lane + j] = ex;
            ex += v[j];
        }
    }
    __syncthreads();
}

// Active-tile list: the flagged tiles, in tile order.  Per-block counts, the
// block scan above, then ranks from warp ballots; the flags are reset for the
// next step.  A block covers TILEK_ITEMS warp-striped rounds of tiles (every
// load coalesced), and all its flag loads are issued before any is used; one
// scan of the (round, warp) counts replaces a barrier pair per round.
#ifndef MPM_TILEK_ITEMS         // tiles per thread (build-time; 4 measured faster than 16)
#define MPM_TILEK_ITEMS 4
#endif
constexpr int TILEK_ITEMS = MPM_TILEK_ITEMS;
constexpr int TILEK_TILE = SEG_THREADS * TILEK_ITEMS;
// Bit r: tile base + r*256 + thread is flagged.
__device__ __forceinline__ unsigned tile_flags(const int* __restrict__ flag, long long n_tiles, long long base) {
    unsigned on = 0;
    int f[TILEK_ITEMS];
#pragma unroll
    for (int r = 0; r < TILEK_ITEMS; ++r) {
        const long long t = base + (long long)r * SEG_THREADS + threadIdx.x;
        f[r] = t < n_tiles ? flag[t] : 0;
    }
#pragma unroll
    for (int r = 0; r < TILEK_ITEMS; ++r) on |= (f[r] != 0 ? 1u : 0u) << r;
    return on;
}

__global__ void __launch_bounds__(SEG_THREADS)
tile_count_kernel(const int* __restrict__ flag, long long n_tiles, unsigned* __restrict__ blk) {
    __shared__ unsigned red[SEG_THREADS / 32];
    unsigned cnt = __popc(tile_flags(flag, n_tiles, (long long)blockIdx.x * TILEK_TILE));
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t = 0;
        for (int w = 0; w < SEG_THREADS / 32; ++w) t += red[w];
        blk[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(SEG_THREADS)
tile_write_kernel(int* __restrict__ flag, long long n_tiles, const unsigned* __restrict__ blk,
                  int* __restrict__ active, int cap) {
    constexpr int NW = SEG_THREADS / 32;
    __shared__ unsigned pre[TILEK_ITEMS * NW];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const long long base = (long long)blockIdx.x * TILEK_TILE;
    const unsigned on = tile_flags(flag, n_tiles, base);
#pragma unroll
    for (int r = 0; r < TILEK_ITEMS; ++r) {
        const unsigned ball = __ballot_sync(0xffffffffu, (on >> r) & 1u);
        if (lane == 0) pre[r * NW + warp] = __popc(ball);
    }
    scan_round_warp_counts<TILEK_ITEMS * NW>(pre);
    const unsigned run = blk[blockIdx.x];
#pragma unroll
    for (int r = 0; r < TILEK_ITEMS; ++r) {
        const long long t = base + (long long)r * SEG_THREADS + threadIdx.x;
        const bool a = (on >> r) & 1u;
        const unsigned ball = __ballot_sync(0xffffffffu, a);
        if (a) {
            const unsigned before = run + pre[r * NW + warp] + __popc(ball & lt);
            if (before < (unsigned)cap) active[before] = (int)t;
            flag[t] = 0;
        }
    }
}

// Writes seg_first / seg_last / cell_seg.  A slot's segment id is the number of
// segment starts up to and including it: the block's count from the scan, the
// starts of the earlier (round, warp) pairs of the block (one exclusive scan
// of the SEGK_ITEMS x 8 warp counts) and the lanes before it.
__global__ void __launch_bounds__(SEG_THREADS)
seg_write_kernel(Ctx ctx, const unsigned* __restrict__ skeys) {
    constexpr int NW = SEG_THREADS / 32;
    constexpr int E = SEGK_ITEMS * NW;
    __shared__ unsigned pre[SEGK_ITEMS * NW];      // round-major
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const long long base = (long long)blockIdx.x * SEGK_TILE;
    unsigned key[SEGK_ITEMS], start, last;
    seg_flags(ctx, skeys, base, key, start, last);
#pragma unroll
    for (int r = 0; r < SEGK_ITEMS; ++r) {
        const unsigned ball = __ballot_sync(0xffffffffu, (start >> r) & 1u);
        if (lane == 0) pre[r * NW + warp] = __popc(ball);
    }
    scan_round_warp_counts<E>(pre);
    const unsigned run = ctx.blk_count[blockIdx.x];     // segments started before this block
#pragma unroll
    for (int r = 0; r < SEGK_ITEMS; ++r) {
        const long long s = base + (long long)r * SEG_THREADS + threadIdx.x;
        const bool st = (start >> r) & 1u;
        const unsigned ball = __ballot_sync(0xffffffffu, st);
        const unsigned id = run + pre[r * NW + warp] + __popc(ball & lt) + (st ? 1u : 0u);
        if (st && MPM_INB(id - 1, ctx.n, 3)) {
            ctx.seg_first[id - 1] = (int)s;
            if (MPM_INB(key[r], ctx.n_keys, 2)) ctx.cell_seg[key[r]] = (int)id;
        }
        if (((last >> r) & 1u) && id > 0 && MPM_INB(id - 1, ctx.n, 3)) ctx.seg_last[id - 1] = (int)(s + 1);
    }
}

// ---------------------------------------------------------------------------
// forward prepass: stress -> P2G record, stored in particle order
// record: fx[0..2], pmass, a = pmass v, B = (pmass C + dt sk) dx
// ---------------------------------------------------------------------------
template <typename R, int KIND = -1, typename G>
__device__ __forceinline__ void p2g_record(const Ctx& ctx, const SceneK<R>& sc, long long p, const R fx[3],
                                           const R v[3], const R C[9], const R F[9], const G& growth,
                                           R rec[PAYLOAD]) {
    ModelParams<R> M;
    M.load(sc);
    if constexpr (KIND >= 0) M.kind = KIND;     // a launch over scenes of one model
    const R dx = sc.dx, dt = sc.dt, inv_dx = sc.inv_dx;
    const R k4 = R(4) * inv_dx * inv_dx;
    R tau[9];
    bool fb = false;
    if (M.kind == MPM_MODEL_EXTERNAL)
        ld9<R>(ctx.ext_tau, p, 9, 1, tau);      // the caller's stress
    else
        fb = model_stress(M, ctx.gap_thresh, F, growth, C, tau);
    if (fb) atomicAdd(ctx.fallbacks, 1ull);
    R pm, vol0;
    particle_mass<R>(ctx, sc, p, pm, vol0);
    R c = -k4 * vol0 * growth.det();
    rec[0] = fx[0]; rec[1] = fx[1]; rec[2] = fx[2]; rec[3] = pm;
#pragma unroll
    for (int i = 0; i < 3; ++i) rec[4 + i] = pm * v[i];
#pragma unroll
    for (int i = 0; i < 9; ++i) rec[7 + i] = (pm * C[i] + dt * (c * tau[i])) * dx;
    if (!finite9(tau)) raise_status(ctx.status, MPM_ERR_NONFINITE);
}

template <typename R>
__global__ void __launch_bounds__(256, 3)
prepass_kernel(Ctx ctx, MpmParticles P, R* __restrict__ payload, int t) {
    long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= ctx.n) return;
    const SceneK<R>& sc = static_cast<const SceneK<R>*>(ctx.sk)[ctx.scene_of[p]];
    R x[3], v[3], C[9], F[9], Fg[9], gphi;
    ld3<R>(P.x, p, P.sp3, P.sc3, x);
    ld3<R>(P.v, p, P.sp3, P.sc3, v);
    ld9<R>(P.C, p, P.sp9, P.sc9, C);
    ld9<R>(P.F, p, P.sp9, P.sc9, F);
    load_Fg<R>(ctx, sc, P, p, t, Fg, gphi);
    int base[3];
    R fx[3];
    bin_particle(x, sc.inv_dx, sc.shape, base, fx);
    R rec[PAYLOAD];
    p2g_record<R>(ctx, sc, p, fx, v, C, F, GrowthFull<R>(Fg), rec);
    store_record(payload, p, rec);
}

// ---------------------------------------------------------------------------
// P2G, phase 1: per-cell sums.  For every segment (occupied cell) the sums of
// its particles' contributions to the 27 stencil nodes, in sorted order,
// stored at sum_at(o, segment) (o = 9 ox + 3 oy + oz).
// Forward: channels (m, mom[3]), from the P2G records.
// ADJ (transfer.py:99-119, the scatter of gv_b): w (nv_b + k4 Cn_b' dp), with
// nv_b = vn_b + dt xn_b (advect) and Cn_b' = Cn_b + dt Fn_b F^T formed here
// from the cotangents of the step's output; the cell marks, cleared by the
// forward G2P, are restored for the node gather.
// ---------------------------------------------------------------------------
// Entry of stencil offset o of segment id in the sums: blocks of SUM_BLOCK
// segments hold their 27 offsets together, so that the entries that a warp
// touches lie in a few kilobytes and not in 27 arrays of n entries.
constexpr int SUM_BLOCK = 32;
__host__ __device__ __forceinline__ long long sum_at(int o, int id) {
    return ((long long)(id / SUM_BLOCK) * 27 + o) * SUM_BLOCK + id % SUM_BLOCK;
}
__host__ __device__ __forceinline__ long long sum_entries(long long n) {
    return (n + SUM_BLOCK - 1) / SUM_BLOCK * SUM_BLOCK * 27;
}

template <typename R>
__device__ __forceinline__ void store_sum(R* __restrict__ S, long long idx, const R v[4]) {
    if constexpr (sizeof(R) == 4) {
        reinterpret_cast<float4*>(S)[idx] = make_float4(v[0], v[1], v[2], v[3]);
    } else {
        double2* p = reinterpret_cast<double2*>(S) + 2 * idx;
        p[0] = make_double2(v[0], v[1]);
        p[1] = make_double2(v[2], v[3]);
    }
}

// What bounds it: with one thread per cell every load touched 32 sectors, and
// a cell's particles were re-read from L2 (FP64: in three passes of the
// registers' choosing).  On 4.7M FP32 particles the reverse took 284 us and the
// forward 166, now 224 and 145; on 0.76M FP64 particles 529 and 93, now 80 and
// 61; on 4096 FP64 particles 33 and 18, now 6.4 and 5.4 (8 per cell).  At 4.7M it moves its
// 0.95 GB (reverse) at 4.2 TB/s; the rest is the wait between a warp's loading
// and adding (45% of the issue slots used).
//
// A warp takes CS_CELLS (or 32, see CS_SPARSE_CELLS) consecutive segments, whose
// particles are consecutive sorted slots.  Its lanes first bring the particles' records into shared
// memory, one particle per lane (every load coalesced), at most CS_SLOTS slots
// at a time; then three lanes per cell, one per stencil x-offset, add them up
// in sorted order.  CS_STRIDE: reals per record in shared memory, 16 padded so
// that the 16-byte accesses of consecutive slots fall on distinct banks.
// MIN_CTAS: registers for a round's loads in flight come before more warps
// (FP64 reverse 105 us with 5 CTAs per SM, 80 with 4; FP32 on (n, 3, 3) fields
// 103 with 6, 85 with 5, and on rows of n 231 with 6, 224 with 5, 239 with 4).
constexpr int CS_CELLS = 10;
constexpr int CS_SLOTS = 96;
// Cells of more slots than a window: with CS_SHARE_CELLS of them or more still to
// be added each gets CS_SHARE places of every window, so that their lanes add
// at the same time; fewer cells take windows of consecutive slots in turn.  FP32
// reverse, 150 particles per cell: 32 us for 3 and 4 cells, in turn 48 and 62, for
// 2 in turn 32; ten cells of 300 in turn took 309 us, with shares 120.
constexpr int CS_SHARE = 8, CS_SHARE_CELLS = 3;
// Two particles per cell or fewer leave most lanes without a record, and a
// warp's ten cells write pieces of 160 bytes: from CS_SPARSE_CELLS cells on a warp
// takes 32 cells, one lane each, for the three x-offsets in turn.  FP32 reverse
// with one particle in each of 30,000 cells 6.8 us both ways, 60,000 10.4 against
// 7.8, 400,000 70 against 44 (two per cell: 50,000 10.3 and 9.7, 15,000 5.2 and
// 6.4; three per cell gain nothing below 100,000 cells).
constexpr int CS_SPARSE_CELLS = 32768;
template <typename R> struct CellSums;
template <> struct CellSums<float>  { static constexpr int WARPS = 4, STRIDE = 20, MIN_CTAS = 5; };
template <> struct CellSums<double> { static constexpr int WARPS = 3, STRIDE = 18, MIN_CTAS = 4; };

// Offset of a slot's record.  Another 16 bytes after every 8 slots: with 8
// particles per cell the ten cells' lanes read slots 8 apart, which would
// otherwise all start on the same bank.
template <typename R>
__host__ __device__ constexpr int rec_at(int slot) {
    return slot * CellSums<R>::STRIDE + (slot >> 3) * (int)(16 / sizeof(R));
}

template <typename R>
__device__ __forceinline__ void put_record(R* at, const R r[PAYLOAD]) {
    using V = typename Vec4<R>::T;
    constexpr int per = sizeof(V) / sizeof(R);
#pragma unroll
    for (int i = 0; i < PAYLOAD / per; ++i) reinterpret_cast<V*>(at)[i] = reinterpret_cast<const V*>(r)[i];
}
template <typename R>
__device__ __forceinline__ void get_record(const R* at, R r[PAYLOAD]) {
    using V = typename Vec4<R>::T;
    constexpr int per = sizeof(V) / sizeof(R);
#pragma unroll
    for (int i = 0; i < PAYLOAD / per; ++i) {
        const V v = reinterpret_cast<const V*>(at)[i];
        const R* e = reinterpret_cast<const R*>(&v);
#pragma unroll
        for (int k = 0; k < per; ++k) r[i * per + k] = e[k];
    }
}

// The reverse record of particle p (fx, -, nv_b, k4 Cn_b' dx)
template <typename R>
__device__ __forceinline__ void adj_record(const Ctx& ctx, const MpmParticles& in, const MpmCotangents& ob, int advect,
                                           int scene, long long p, R r[PAYLOAD]) {
    const SceneK<R>& sk = static_cast<const SceneK<R>*>(ctx.sk)[scene];
    const R dx = sk.dx, dt = sk.dt, inv_dx = sk.inv_dx;
    const R kdx = R(4) * inv_dx * inv_dx * dx;
    R x[3], nv[3], F[9], Fb[9], Cb[9];
    ld3<R>(in.x, p, in.sp3, in.sc3, x);
    ld9<R>(in.F, p, in.sp9, in.sc9, F);
    ld9<R>(ob.F, p, ob.sp9, ob.sc9, Fb);
    ld9<R>(ob.C, p, ob.sp9, ob.sc9, Cb);
    ld3<R>(ob.v, p, ob.sp3, ob.sc3, nv);
    if (advect) {
        R xb[3];
        ld3<R>(ob.x, p, ob.sp3, ob.sc3, xb);
#pragma unroll
        for (int i = 0; i < 3; ++i) nv[i] += dt * xb[i];
    }
    R FbFt[9];
    mmT(Fb, F, FbFt);
    int base[3];
    R fx[3];
    bin_particle(x, inv_dx, sk.shape, base, fx);
    r[0] = fx[0]; r[1] = fx[1]; r[2] = fx[2]; r[3] = R(0);
#pragma unroll
    for (int i = 0; i < 3; ++i) r[4 + i] = nv[i];
#pragma unroll
    for (int i = 0; i < 9; ++i) r[7 + i] = kdx * (Cb[i] + dt * FbFt[i]);
}

// Adds one record's contributions at the stencil x-offset ox: w(o) (a + B dp(o))
// and (forward) w(o) m in channel 0, dp = o - fx in cell units.
template <typename R, bool ADJ>
__device__ __forceinline__ void accumulate_record(const R r[PAYLOAD], int ox, R acc[3][3][ADJ ? 3 : 4]) {
    R wy[3], wz[3], wx;
    {
        const R a = R(1.5) - r[1], b = r[1] - R(1.0), c = r[1] - R(0.5);
        wy[0] = R(0.5) * a * a;
        wy[1] = R(0.75) - b * b;
        wy[2] = R(0.5) * c * c;
    }
    {
        const R a = R(1.5) - r[2], b = r[2] - R(1.0), c = r[2] - R(0.5);
        wz[0] = R(0.5) * a * a;
        wz[1] = R(0.75) - b * b;
        wz[2] = R(0.5) * c * c;
    }
    {
        const R a = (ox == 0 ? R(1.5) : R(0.5)) - r[0], b = r[0] - R(1.0);     // (c)^2 = (-c)^2
        wx = ox == 1 ? R(0.75) - b * b : R(0.5) * a * a;
    }
    const R dz[3] = {R(0) - r[2], R(1) - r[2], R(2) - r[2]};
    const R dy[3] = {R(0) - r[1], R(1) - r[1], R(2) - r[1]};
    const R dpx = R(ox) - r[0];
    // a + B dp with dp = (dpx, dy, dz), x part hoisted
    const R ax0 = r[4] + r[7] * dpx, ax1 = r[5] + r[10] * dpx, ax2 = r[6] + r[13] * dpx;
    constexpr int M = ADJ ? 0 : 1;
#pragma unroll
    for (int oy = 0; oy < 3; ++oy) {
        const R wxy = wx * wy[oy];
        const R ay0 = ax0 + r[8] * dy[oy], ay1 = ax1 + r[11] * dy[oy], ay2 = ax2 + r[14] * dy[oy];
#pragma unroll
        for (int oz = 0; oz < 3; ++oz) {
            const R wt = wxy * wz[oz];
            if constexpr (!ADJ) acc[oy][oz][0] += wt * r[3];
            acc[oy][oz][M + 0] += wt * (ay0 + r[9] * dz[oz]);
            acc[oy][oz][M + 1] += wt * (ay1 + r[12] * dz[oz]);
            acc[oy][oz][M + 2] += wt * (ay2 + r[15] * dz[oz]);
        }
    }
}

// Brings the records of the slots slot(k) < stop(k) to places 32 k + lane.
template <typename R, bool ADJ, typename Slot, typename Stop>
__device__ __forceinline__ void stage_records(const Ctx& ctx, const unsigned* __restrict__ perm,
                                              const R* __restrict__ payload, const MpmParticles& in,
                                              const MpmCotangents& ob, int advect, Slot&& slot, Stop&& stop, R* rec) {
    const int lane = threadIdx.x & 31;
    unsigned p[CS_SLOTS / 32];
#pragma unroll
    for (int k = 0; k < CS_SLOTS / 32; ++k) p[k] = slot(k) < stop(k) ? perm[slot(k)] : 0xffffffffu;
#pragma unroll
    for (int k = 0; k < CS_SLOTS / 32; ++k) {
        if (slot(k) < stop(k)) {
            R r[PAYLOAD];
            if (!MPM_INB(p[k], ctx.n, 9)) {
#pragma unroll
                for (int i = 0; i < PAYLOAD; ++i) r[i] = R(0);
            } else if constexpr (ADJ) {
                adj_record<R>(ctx, in, ob, advect, ctx.scene_of[slot(k)], p[k], r);
            } else {
                load_record(payload, p[k], r);
            }
            put_record(rec + rec_at<R>(32 * k + lane), r);
        }
    }
    __syncwarp();
}

// Sums of a warp's cells g .. stop - 1 (at most 32 / LANES): LANES = 3 lanes per
// cell, one per stencil x-offset, or one lane that takes the offsets in turn.
// With one lane the cells' records must fit one window (otherwise false, and
// nothing is done).
template <typename R, bool ADJ, int LANES>
__device__ __forceinline__ bool sum_cells(const Ctx& ctx, const unsigned* __restrict__ skeys,
                                          const unsigned* __restrict__ perm, const R* __restrict__ payload,
                                          const MpmParticles& in, const MpmCotangents& ob, R* __restrict__ S,
                                          int advect, int g, int stop, R* rec) {
    constexpr int CH = ADJ ? 3 : 4;
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31, c = lane / LANES, id = g + c;
    const bool mine = c < 32 / LANES && id < stop;
    int first = mine ? ctx.seg_first[id] : 0;
    int last = mine ? ctx.seg_last[id] : 0;
    if (!(MPM_INB(first, ctx.n + 1, 11) && MPM_INB(last, ctx.n + 1, 11))) first = last = 0;
    const int end = __reduce_max_sync(ALL, last), begin = __reduce_min_sync(ALL, mine ? first : INT_MAX);
    const bool one_window = __builtin_expect(end - begin <= CS_SLOTS, 1);
    if (LANES == 1 && !one_window) return false;
    if constexpr (ADJ) {
        if (mine && lane % LANES == 0 && first < last) {
            const unsigned key = skeys[first];
            if (MPM_INB(key, ctx.n_keys, 2)) ctx.cell_seg[key] = id + 1;
        }
    }
    if (one_window)
        stage_records<R, ADJ>(ctx, perm, payload, in, ob, advect, [&](int k) { return begin + 32 * k + lane; },
                              [&](int) { return end; }, rec);
#pragma unroll 1
    for (int pass = 0; pass < 3 / LANES; ++pass) {
        const int ox = LANES == 3 ? lane % 3 : pass;
        R acc[3][3][CH];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b)
#pragma unroll
                for (int h = 0; h < CH; ++h) acc[a][b][h] = R(0);
        // adds the records at place `at` and following, up to slot `stop`
        auto add = [&](int& cur, int stop, int at) {
            for (; cur < stop; ++cur, ++at) {
                R r[PAYLOAD];
                get_record(rec + rec_at<R>(at), r);
                accumulate_record<R, ADJ>(r, ox, acc);
            }
        };
        int cur = first;
        if (LANES == 1 || one_window) {
            add(cur, last, cur - begin);
        } else {
            for (;;) {
                // the next window starts at the first slot still to be added (slots
                // between the cells hold particles outside the grid)
                const int w0 = __reduce_min_sync(ALL, cur < last ? cur : INT_MAX);
                if (w0 == INT_MAX) break;
                // several cells that do not fit it take the same share of it each
                const bool share = end - w0 > CS_SLOTS && __popc(__ballot_sync(ALL, cur < last)) >= 3 * CS_SHARE_CELLS;
                int from[CS_SLOTS / 32], upto[CS_SLOTS / 32];
#pragma unroll
                for (int k = 0; k < CS_SLOTS / 32; ++k) {
                    const int l = 32 * k + lane, owner = 3 * (l / CS_SHARE);    // a lane of the cell
                    const int f = __shfl_sync(ALL, cur, owner) + l % CS_SHARE, u = __shfl_sync(ALL, last, owner);
                    from[k] = share ? f : w0 + l;
                    upto[k] = !share ? end : (owner < 3 * CS_CELLS ? u : 0);
                }
                stage_records<R, ADJ>(ctx, perm, payload, in, ob, advect, [&](int k) { return from[k]; },
                                      [&](int k) { return upto[k]; }, rec);
                const int upper = share ? cur + CS_SHARE : w0 + CS_SLOTS;
                add(cur, last < upper ? last : upper, share ? CS_SHARE * c : cur - w0);
                __syncwarp();
            }
        }
        if (mine) {
#pragma unroll
            for (int oy = 0; oy < 3; ++oy)
#pragma unroll
                for (int oz = 0; oz < 3; ++oz) {
                    const long long at = sum_at(9 * ox + 3 * oy + oz, id);
                    R v[4];
#pragma unroll
                    for (int h = 0; h < 4; ++h) v[h] = h < CH ? acc[oy][oz][h] : R(0);
                    if (MPM_INB(at, sum_entries(ctx.n), 4)) store_sum(S, at, v);
                }
        }
    }
    __syncwarp();       // the records are read: the warp's next cells may take their place
    return true;
}

// SPARSE: the plan has particles enough for CS_SPARSE_CELLS cells (asked at run time,
// the question alone costs 0.1 to 0.3 us of 4 to 6 on small plans).
template <typename R, bool ADJ, bool SPARSE>
__global__ void __launch_bounds__(32 * CellSums<R>::WARPS, CellSums<R>::MIN_CTAS)
cell_sums_kernel(Ctx ctx, const unsigned* __restrict__ skeys, const unsigned* __restrict__ perm,
                 const R* __restrict__ payload, MpmParticles in, MpmCotangents ob, R* __restrict__ S, int advect) {
    constexpr int W = CellSums<R>::WARPS;
    __shared__ __align__(16) R rec_s[W][rec_at<R>(CS_SLOTS)];
    const int nseg = *ctx.n_seg, w = blockIdx.x * W + (threadIdx.x >> 5), nw = gridDim.x * W;
    R* rec = rec_s[threadIdx.x >> 5];
    if constexpr (SPARSE) {
        if (nseg >= CS_SPARSE_CELLS && 2ll * nseg >= ctx.n) {
            for (int g = w * 32; g < nseg; g += nw * 32) {
                const int stop = nseg - g < 32 ? nseg : g + 32;
                if (sum_cells<R, ADJ, 1>(ctx, skeys, perm, payload, in, ob, S, advect, g, stop, rec)) continue;
                for (int h = g; h < stop; h += CS_CELLS)
                    sum_cells<R, ADJ, 3>(ctx, skeys, perm, payload, in, ob, S, advect, h, stop, rec);
            }
            return;
        }
    }
    for (int g = w * CS_CELLS; g < nseg; g += nw * CS_CELLS)
        sum_cells<R, ADJ, 3>(ctx, skeys, perm, payload, in, ob, S, advect, g, nseg, rec);
}

// ---------------------------------------------------------------------------
// P2G, phase 2: node gather + grid update.  One thread per node of the
// active node tiles (persistent grid over the active list); every node adds
// the sums of its 27 source cells in the fixed order o = 0..26, then
// MODE 0: grid update -> (m, v[3]) with v = s mom/m + s dt g on free nodes;
// MODE 1: grid adjoint -> (gm_b, gmom_b[3]) from gv_b and the forward record,
// which is also restored into the dense scratch for the reverse particle kernel.
// ---------------------------------------------------------------------------
template <typename R>
__device__ __forceinline__ void load_sum(const R* __restrict__ S, long long idx, R o[4]) {
    if constexpr (sizeof(R) == 4) {
        float4 v = __ldg(reinterpret_cast<const float4*>(S) + idx);
        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    } else {
        const double2* p = reinterpret_cast<const double2*>(S) + 2 * idx;
        double2 a = __ldg(p), b = __ldg(p + 1);
        o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
    }
}

// What bounds it: the latency of scattered loads (a node's 27 sums are 27 short
// runs shared with its z-neighbours), so the loads are issued in groups: IDS
// source cells' segment ids, then their sums SUMS at a time, in 64 (FP64: 80)
// registers.  Left to the compiler's schedule the same loop took 95 to 185 us
// on 4.7M particles, depending on the registers it settled for; in this form
// 105 us forward and 116 us reverse, and on 4096 particles 6.5 us against 7.5
// with 1024-thread blocks, which put a small scene on a handful of SMs.
constexpr int NODE_THREADS = 128;
template <typename R> struct NodeSums;
template <> struct NodeSums<float>  { static constexpr int IDS = 9, SUMS = 9, MIN_CTAS = 8; };
template <> struct NodeSums<double> { static constexpr int IDS = 27, SUMS = 3, MIN_CTAS = 6; };
template <typename R, int T, int TZ, int MODE>
__global__ void __launch_bounds__(NODE_THREADS, NodeSums<R>::MIN_CTAS)
node_sums_kernel(Ctx ctx, const R* __restrict__ S, const int* __restrict__ active,
                 const int* __restrict__ n_active, R* __restrict__ grid_out, const R* __restrict__ grid_fwd,
                 int advect) {
    constexpr unsigned TN = T * T * TZ;
    constexpr int IDS = NodeSums<R>::IDS, G = NodeSums<R>::SUMS;
    // one thread per node of the active tiles (tile-major, z fastest), grid-strided
    const long long total = (long long)(*n_active) * TN;
    for (long long gidx = (long long)blockIdx.x * NODE_THREADS + threadIdx.x; gidx < total;
         gidx += (long long)gridDim.x * NODE_THREADS) {
        const int tile = active[gidx / TN];
        const unsigned node = (unsigned)(gidx % TN);
        const int s = ctx.tile_scene[tile];
        const SceneK<R>& sc = static_cast<const SceneK<R>*>(ctx.sk)[s];
        const SceneAux& ax = ctx.aux[s];
        // the scene's tiles and nodes fit 32 bits (its padded cells do)
        const unsigned lt = (unsigned)(tile - ax.tile_begin), nt1 = ax.ntile[1], nt2 = ax.ntile[2];
        const unsigned row = lt / nt2, tx = row / nt1;
        const int i = (int)(tx * T + node / (TZ * T)), j = (int)((row - tx * nt1) * T + (node / TZ) % T),
                  k = (int)((lt - row * nt2) * TZ + node % TZ);
        if (i >= sc.shape[0] || j >= sc.shape[1] || k >= sc.shape[2]) continue;
        const int P1 = sc.shape[1] + 2, P2 = sc.shape[2] + 2;
        const long long cbase = ax.cell_begin + (((i + 2) * P1 + (j + 2)) * P2 + (k + 2));
        R f[4];
        if (MODE == 1 && MPM_INB(gidx, ctx.grid_nodes, 8)) load_node(grid_fwd, gidx, f);
        R acc[4] = {R(0), R(0), R(0), R(0)};
#pragma unroll
        for (int o0 = 0; o0 < 27; o0 += IDS) {
            int id[IDS];
#pragma unroll
            for (int g = 0; g < IDS; ++g) {
                const int o = o0 + g;
                const long long ci = cbase - ((o / 9) * P1 + (o / 3) % 3) * P2 - o % 3;
                id[g] = MPM_INB(ci, ctx.n_keys, 6) ? ctx.cell_seg[ci] : 0;
            }
#pragma unroll
            for (int g0 = 0; g0 < IDS; g0 += G) {
                R v[G][4];
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const long long si = sum_at(o0 + g0 + g, id[g0 + g] - 1);
#pragma unroll
                    for (int h = 0; h < 4; ++h) v[g][h] = R(0);
                    if (id[g0 + g] != 0 && MPM_INB(si, sum_entries(ctx.n), 5)) load_sum(S, si, v[g]);
                }
#pragma unroll
                for (int g = 0; g < G; ++g)
#pragma unroll
                    for (int h = 0; h < (MODE == 0 ? 4 : 3); ++h) acc[h] += v[g][h];
            }
        }
        const long long didx = ax.node_begin + ((i * sc.shape[1] + j) * sc.shape[2] + k);
        if (!(MPM_INB(didx, ctx.n_nodes, 7) && MPM_INB(gidx, ctx.grid_nodes, 8))) continue;
        const R s_damp = sc.s_damp, dt = sc.dt;
        R rec[4] = {R(0), R(0), R(0), R(0)};
        if constexpr (MODE == 0) {
            const R m = acc[0];
            rec[0] = m;
            if (m > sc.mass_eps && node_free(sc, i, j, k)) {
#pragma unroll
                for (int d = 0; d < 3; ++d) rec[1 + d] = (s_damp * acc[1 + d]) / m + s_damp * dt * sc.gravity[d];
            }
            store_node(grid_out, gidx, rec);
            store_node(static_cast<R*>(ctx.dense_f), didx, rec);
        } else {
            store_node(static_cast<R*>(ctx.dense_f), didx, f);
            const R m = f[0];
            if (m > sc.mass_eps && node_free(sc, i, j, k)) {
#pragma unroll
                for (int d = 0; d < 3; ++d) rec[1 + d] = (s_damp * acc[d]) / m;
                if (advect) {
                    const R sd = s_damp * dt;
                    rec[0] = -(acc[0] * (f[1] - sd * sc.gravity[0]) + acc[1] * (f[2] - sd * sc.gravity[1])
                             + acc[2] * (f[3] - sd * sc.gravity[2])) / m;
                }
            }
            store_node(static_cast<R*>(ctx.dense_b), didx, rec);
        }
    }
}

// ---------------------------------------------------------------------------
// stencil addressing into the dense node scratch: node (i,j,k) of a scene is
// node_begin + (i ny + j) nz + k.  Where the 27 nodes of every particle of a warp
// lie in the grid, the loop is unrolled without a test per node: one address per
// stencil row, the three nodes of a row at constant offsets.  A warp with a
// stencil at a face of the grid takes a rolled loop over the rows for all its
// particles (stencil_rows): the same terms in the same order, so a particle's
// result does not depend on its neighbours in the warp.  With a loop of their own
// for the particles at the faces, warps that mix both ran the two one after the
// other: on a grid of 256 x 256 x 4 nodes the reverse kernel took 87 us for 300,000
// FP32 neo-Hookean particles (Hencky 98) and G2P 42 (51), now 52 (67) and 31 (34).
// ---------------------------------------------------------------------------
template <typename R>
__device__ __forceinline__ bool stencil_interior(const SceneK<R>& sc, const int base[3]) {
    return base[0] >= 0 && base[1] >= 0 && base[2] >= 0 && base[0] + 2 < sc.shape[0] && base[1] + 2 < sc.shape[1] &&
           base[2] + 2 < sc.shape[2];
}
// Orders the loads at `at` after the computation of v: without a test per node
// the compiler would start all 54 node loads of the reverse kernel at once and
// spill what it holds; a third of them at a time is enough in flight (Hencky
// 419 -> 401 us on 2.5M particles, Herschel-Bulkley 336 -> 317 on 2.1M).
__device__ __forceinline__ void loads_after(long long& at, float& v) { asm volatile("" : "+l"(at), "+f"(v)); }
__device__ __forceinline__ void loads_after(long long& at, double& v) { asm volatile("" : "+l"(at), "+d"(v)); }
// weight of stencil offset o at fractional position f, and its derivative
template <typename R>
__device__ __forceinline__ R weight_at(int o, R f) {
    const R a = (o == 0 ? R(1.5) : R(0.5)) - f, b = f - R(1.0);
    return o == 1 ? R(0.75) - b * b : R(0.5) * a * a;
}
template <typename R>
__device__ __forceinline__ R weight_grad_at(int o, R f) {
    return o == 0 ? -(R(1.5) - f) : (o == 1 ? R(-2.0) * (f - R(1.0)) : f - R(0.5));
}
// whether the lanes that are here together all have it
__device__ __forceinline__ bool warp_all(bool have) { return __all_sync(__activemask(), have); }
// A stencil's nodes on one axis: nodes outside the grid have weight 0 and the
// place of the nearest node inside, which the stencil has too.
template <typename R>
struct AxisNode {
    int at;
    R w, dw;
    __device__ __forceinline__ AxisNode(int o, int base, R f, int n) {
        const int i = base + o;
        const bool in = i >= 0 && i < n;
        at = i < 0 ? 0 : (i < n ? i : n - 1);
        w = in ? weight_at(o, f) : R(0);
        dw = in ? weight_grad_at(o, f) : R(0);
    }
};
// row(a, b, the row's x and y weights and derivatives, the z ones, nodes) for the
// rows of a stencil that has nodes in the grid.  The axes' nodes are formed again
// for every row (the fence on base_z): kept, they would take registers from the
// kernel's other paths (FP32 G2P at 5 CTAs per SM: 146 -> 154 us on 2.2M particles).
template <typename R, typename Fn>
__device__ __forceinline__ void stencil_rows(const SceneK<R>& sc, const SceneAux& ax, const int base[3], const R fx[3],
                                             Fn&& row) {
#pragma unroll
    for (int d = 0; d < 3; ++d)
        if (base[d] < -2 || base[d] >= sc.shape[d]) return;
    int base_z = base[2];
#pragma unroll 1
    for (int ab = 0; ab < 9; ++ab) {
        const int a = ab / 3, b = ab - 3 * a;
        asm volatile("" : "+r"(base_z));
        const AxisNode<R> x(a, base[0], fx[0], sc.shape[0]), y(b, base[1], fx[1], sc.shape[1]);
        const AxisNode<R> z[3] = {{0, base_z, fx[2], sc.shape[2]}, {1, base_z, fx[2], sc.shape[2]},
                                  {2, base_z, fx[2], sc.shape[2]}};
        const long long first = ax.node_begin + (x.at * sc.shape[1] + y.at) * sc.shape[2];
        const long long node[3] = {first + z[0].at, first + z[1].at, first + z[2].at};
        const R wz[3] = {z[0].w, z[1].w, z[2].w}, dwz[3] = {z[0].dw, z[1].dw, z[2].dw};
        row(a, b, x.w, x.dw, y.w, y.dw, wz, dwz, node);
    }
}

__device__ __forceinline__ void unmark_cell(const Ctx& ctx, const SceneAux& ax, const unsigned* __restrict__ skeys,
                                            long long sidx) {
    unsigned k = skeys[sidx];
    if ((sidx == 0 || skeys[sidx - 1] != k) && (long long)k - ax.cell_begin < ax.ncells && MPM_INB(k, ctx.n_keys, 2))
        ctx.cell_seg[k] = 0;
}

// ---------------------------------------------------------------------------
// G2P + advection + F update (transfer.py:61-79); writes the output state in
// the input's particle order and clears the cell marks of this step.
// ---------------------------------------------------------------------------
// Sorted slots [s_begin, s_end).  KIND >= 0: every scene of these slots uses
// material model KIND, so the kernel carries that model's code only.
// ISO: see Growth (emitting kernels only).
// FULL: the plan fills the GPU.  Then warps in flight count more than spills:
// the emitting kernel at 5 CTAs per SM (48 registers) takes 154 us on 2.2M
// neo-Hookean and 142 on 2.1M Herschel-Bulkley particles, 164 and 148 at 4, 190
// and 174 at 3; on 4096 particles, where it waits for its own instructions and
// loads, 3 CTAs' registers give 6.3 us and 5 CTAs' 7.7.  FP32 Hencky keeps 3: at 5
// it would take 197 us for 222 on 2.5M, but its eigensolve is contracted
// differently there and the FP32 results move by a rounding.
template <typename R, bool EMIT, int KIND, bool ISO, bool FULL>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? (EMIT ? (FULL ? 5 : 3) : 4) : (EMIT && FULL ? 3 : 2))
g2p_kernel(Ctx ctx, Tape<R> tp, MpmParticles in, MpmParticles out, int advect, unsigned* __restrict__ keys,
           R* __restrict__ payload, int t, long long s_begin, long long s_end) {
    long long sidx = s_begin + (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (sidx >= s_end) return;
    long long p = tp.perm[sidx];
    if (!MPM_INB(p, ctx.n, 9)) return;
    const int s = ctx.scene_of[sidx];
    const SceneK<R>& sc = static_cast<const SceneK<R>*>(ctx.sk)[s];
    const SceneAux& ax = ctx.aux[s];
    const R dx = sc.dx, dt = sc.dt, inv_dx = sc.inv_dx;
    const R k4 = R(4) * inv_dx * inv_dx;
    R x[3];
    ld3<R>(in.x, p, in.sp3, in.sc3, x);
    int base[3];
    R fx[3];
    bin_particle(x, inv_dx, sc.shape, base, fx);
    const R* __restrict__ dense = static_cast<const R*>(ctx.dense_f);
    // nC = k4 sum w g (o - fx)^T dx = k4 dx (G - nv fx^T),  G[i][d] = sum w g_i o_d
    R nv[3] = {0, 0, 0}, G[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    auto row = [&](int a, int b, R wa, R wb, const R wz[3], const long long node[3]) {
        // column sums over z: sum w_c g and sum c w_c g
        R Zg[3] = {0, 0, 0}, Zc[3] = {0, 0, 0};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            R g[4];
            if (!MPM_INB(node[c], ctx.n_nodes, 7)) continue;
            load_node(dense, node[c], g);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                Zg[i] += wz[c] * g[1 + i];
                if (c) Zc[i] += (R(c) * wz[c]) * g[1 + i];
            }
        }
        const R wab = wa * wb;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            nv[i] += wab * Zg[i];
            if (a) G[3 * i + 0] += (R(a) * wab) * Zg[i];
            if (b) G[3 * i + 1] += (R(b) * wab) * Zg[i];
            G[3 * i + 2] += wab * Zc[i];
        }
    };
    if (warp_all(stencil_interior(sc, base))) {
        R w[3][3];
        bspline(fx, w);
        const R wz[3] = {w[0][2], w[1][2], w[2][2]};
        const int ny = sc.shape[1], nz = sc.shape[2];
        const long long n0 = ax.node_begin + ((base[0] * ny + base[1]) * nz + base[2]);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const long long r = n0 + (a * ny + b) * nz;
                const long long node[3] = {r, r + 1, r + 2};
                row(a, b, w[a][0], w[b][1], wz, node);
            }
        }
    } else {
        stencil_rows(sc, ax, base, fx, [&](int a, int b, R wa, R, R wb, R, const R wz[3], const R*,
                                           const long long node[3]) { row(a, b, wa, wb, wz, node); });
    }
    R nC[9];
    const R kd = k4 * dx;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int d = 0; d < 3; ++d) nC[3 * i + d] = kd * (G[3 * i + d] - nv[i] * fx[d]);
    R F[9];
    ld9<R>(in.F, p, in.sp9, in.sc9, F);
    R xn[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) xn[i] = advect ? x[i] + dt * nv[i] : x[i];
    R A[9], Fn[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) A[i] = ((i % 4 == 0) ? R(1) : R(0)) + dt * nC[i];
    mm(A, F, Fn);
    st3<R>(out.x, p, out.sp3, out.sc3, xn);
    st3<R>(out.v, p, out.sp3, out.sc3, nv);
    st9<R>(out.C, p, out.sp9, out.sc9, nC);
    st9<R>(out.F, p, out.sp9, out.sc9, Fn);
    if (!ISO && sc.growth_mode == 0 && out.Fg != nullptr && out.Fg != in.Fg) {
        R Fg[9];
        ld9<R>(in.Fg, p, in.sp9, in.sc9, Fg);
        st9<R>(out.Fg, p, out.sp9, out.sc9, Fg);
    }
    if (!finite9(Fn) || !(xn[0] * R(0) == R(0) && xn[1] * R(0) == R(0) && xn[2] * R(0) == R(0)))
        raise_status(ctx.status, MPM_ERR_NONFINITE);
    unmark_cell(ctx, ax, tp.skeys, sidx);
    if constexpr (EMIT) {
        // the next step's binning and P2G record of the new state (what the
        // bin and prepass kernels of step t+1 would compute from memory)
        R fxn[3], gphi, rec[PAYLOAD];
        const unsigned kn = particle_key<R>(ctx, sc, ax, xn, fxn);
        keys[p] = kn;
        // movers of this step's sorted order (the next step's re-sort)
        if (ctx.moved_count) {
            const unsigned act = __activemask();
            const unsigned ball = __ballot_sync(act, kn != tp.skeys[sidx]);
            if (ball && (threadIdx.x & 31) == __ffs(act) - 1) atomicAdd(ctx.moved_count, (unsigned)__popc(ball));
        }
        if (ctx.mover_flag) {
            const unsigned char moved = kn != tp.skeys[sidx] ? 1 : 0;
            ctx.mover_flag[sidx] = moved;
            ctx.mover_pflag[p] = moved;
        }
        Growth<R, ISO> gr;
        gr.load(ctx, sc, in, p, t + 1, gphi);
        p2g_record<R, KIND>(ctx, sc, p, fxn, nv, nC, Fn, gr.g, rec);
        store_record(payload, p, rec);
    }
}

// ---------------------------------------------------------------------------
// reverse: per-particle cotangents (transfer.py:99-119 x_b terms, 129-156).
// The x_b terms of the reference are regrouped per node as
//   x_b += [nv_b.gv + pm mb.v + pm gm_b + (M1 gv + M2 mb).dp] dW
// with M1 = k4 Cn_b'^T, M2 = pm C^T + dt sk^T, and the weight-only terms are
// summed once per particle: x_b -= M1 sum(w gv) + M2 sum(w mb).
// ---------------------------------------------------------------------------
// MAT: also the material-parameter gradients per slot, dmat[sidx] (mu) and
// dmat[n + sidx] (lambda).  EXT: the plan has MPM_MODEL_EXTERNAL scenes.
// Sorted slots [s_begin, s_end); KIND as in g2p_kernel.
// What bounds it: instruction issue and load latency together, at 16 warps per
// SM (128 registers; more CTAs spill and are slower).  Scene constants in the
// plan's type, one address per stencil row without a test per node, and g
// alone for isotropic growth cut its instructions: on 4.7M particles of two
// models 886 -> 730 us (FP64, 0.76M: 382 -> 269), on 4096 11.0 -> 8.8.
// ISO: see Growth, and no Fg cotangent is asked for (ib.Fg null).
template <typename R, bool MAT, bool EXT, int KIND, bool ISO>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 2 : 1)
bwd_particle_kernel(Ctx ctx, Tape<R> tp, MpmParticles in, const R* __restrict__ outC,
                    MpmCotangents ob, MpmCotangents ib, double* __restrict__ dA, double* __restrict__ dmat,
                    int advect, int t, long long s_begin, long long s_end) {
    long long sidx = s_begin + (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (sidx >= s_end) return;
    long long p = tp.perm[sidx];
    if (!MPM_INB(p, ctx.n, 9)) return;
    const int s = ctx.scene_of[sidx];
    const SceneK<R>& sc = static_cast<const SceneK<R>*>(ctx.sk)[s];
    const SceneAux& ax = ctx.aux[s];
    ModelParams<R> M;
    M.load(sc);
    if constexpr (KIND >= 0) M.kind = KIND;
    const R dx = sc.dx, dt = sc.dt, inv_dx = sc.inv_dx;
    const R k4 = R(4) * inv_dx * inv_dx;
    R pm, vol0;
    particle_mass<R>(ctx, sc, p, pm, vol0);
    R x[3], C[9], F[9];
    R gphi;
    Growth<R, ISO> gr;
    ld3<R>(in.x, p, in.sp3, in.sc3, x);
    ld9<R>(in.C, p, in.sp9, in.sc9, C);
    ld9<R>(in.F, p, in.sp9, in.sc9, F);
    gr.load(ctx, sc, in, p, t, gphi);

    R tau[9], keep[13];
    bool fb = false;
    if (EXT && M.kind == MPM_MODEL_EXTERNAL)
        ld9<R>(ctx.ext_tau, p, 9, 1, tau);      // the caller's stress
    else
        fb = model_stress_keep(M, ctx.gap_thresh, F, gr.g, C, tau, keep);
    // the kept eigendecomposition waits in shared memory (one column per
    // thread) while the node loop holds the registers
    __shared__ R keep_s[13][256];
#pragma unroll
    for (int i = 0; i < 13; ++i) keep_s[i][threadIdx.x] = keep[i];
    const R c = -k4 * vol0 * gr.g.det();

    // per-particle matrices of the regrouped x_b terms
    R M1[9], M2[9], nvb[3], pv[3];
    {
        R xnb[3], vnb[3], Cnb[9], Fnb[9], v[3];
        ld3<R>(ob.x, p, ob.sp3, ob.sc3, xnb);
        ld3<R>(ob.v, p, ob.sp3, ob.sc3, vnb);
        ld9<R>(ob.C, p, ob.sp9, ob.sc9, Cnb);
        ld9<R>(ob.F, p, ob.sp9, ob.sc9, Fnb);
        ld3<R>(in.v, p, in.sp3, in.sc3, v);
        R FbFt[9];
        mmT(Fnb, F, FbFt);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            nvb[i] = advect ? vnb[i] + dt * xnb[i] : vnb[i];
            // rounded products for two components, a fused one for the third: the
            // roundings this kernel has always had, kept whatever the compiler
            // would contract, so that FP32 gradients stay the same bit for bit
            pv[i] = i < 2 ? Num<R>::mul_rn(pm, v[i]) : v[i];
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                M1[3 * i + j] = k4 * (Cnb[3 * j + i] + dt * FbFt[3 * j + i]);       // k4 Cn_b'^T
                M2[3 * i + j] = pm * C[3 * j + i] + dt * (c * tau[3 * j + i]);       // pm C^T + dt sk^T
            }
        }
    }
    // the new C, first read after the node loop, on its way to L2 meanwhile (rows
    // of n: 407 -> 399 and 327 -> 322 us on 2.5M and 2.2M particles; a particle's
    // nine values side by side gain nothing, 326 -> 338 on 1M)
    if (in.sc9 != 1) {
        const R* oc = outC + p * in.sp9;
#pragma unroll
        for (int i = 0; i < 9; ++i) asm volatile("prefetch.global.L2 [%0];" :: "l"(oc + i * in.sc9));
    }
    int base[3];
    R fx[3];
    bin_particle(x, inv_dx, sc.shape, base, fx);
    // The node loop is evaluated as separable sums: per stencil column (a,b)
    // the z-weighted sums of gv, mb and c*mb, and of the advect factor
    //   sfac(o) = gv.U(o) + mb.V(o) + pm gm_b,  U(o) = nv_b + M1^T dp, V(o) = pm v + M2^T dp
    // (dp = (o - fx) dx, so U and V are affine in o: U = U0 + dx (a M1_0 + b M1_1 + c M1_2)
    // with M1_i the rows of M1), then the column sums are weighted by w_a w_b.
    // Sb = sum w mb (o - fx)^T dx = dx (GB - wmb fx^T),  GB[i][d] = sum w mb_i o_d
    R D1[9], D2[9], U0[3], V0[3];
#pragma unroll
    for (int q = 0; q < 9; ++q) { D1[q] = dx * M1[q]; D2[q] = dx * M2[q]; }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        U0[j] = nvb[j] - (D1[j] * fx[0] + D1[3 + j] * fx[1] + D1[6 + j] * fx[2]);
        const R vs = D2[j] * fx[0] + D2[3 + j] * fx[1] + D2[6 + j] * fx[2];
        V0[j] = j < 2 ? pv[j] - vs : fma(pm, pv[j], -vs);
    }
    const R* __restrict__ dfw = static_cast<const R*>(ctx.dense_f);
    const R* __restrict__ dbw = static_cast<const R*>(ctx.dense_b);
    R xs[3] = {0, 0, 0}, wgv[3] = {0, 0, 0}, wmb[3] = {0, 0, 0}, GB[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) GB[q] = R(0);
    auto row = [&](int a, int b, R wa, R dwa, R wb, R dwb, const R w2[3], const R dw2[3], const long long node[3]) {
        R Zg[3] = {0, 0, 0}, Zm[3] = {0, 0, 0}, Zc[3] = {0, 0, 0}, Sab = 0, Tab = 0;
        R Uab[3], Vab[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            Uab[j] = U0[j] + R(a) * D1[j] + R(b) * D1[3 + j];
            Vab[j] = V0[j] + R(a) * D2[j] + R(b) * D2[3 + j];
        }
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) {
            R gf[4], gb[4];
            if (!MPM_INB(node[cc], ctx.n_nodes, 7)) continue;
            load_node(dfw, node[cc], gf);
            load_node(dbw, node[cc], gb);
            const R* gv = gf + 1;
            const R* mb = gb + 1;
            const R wz = w2[cc];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                Zg[i] += wz * gv[i];
                Zm[i] += wz * mb[i];
                if (cc) Zc[i] += (R(cc) * wz) * mb[i];
            }
            if (advect) {
                R sfac = gb[0] * pm;
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    sfac += gv[j] * (Uab[j] + R(cc) * D1[6 + j]) + mb[j] * (Vab[j] + R(cc) * D2[6 + j]);
                Sab += wz * sfac;
                Tab += dw2[cc] * sfac;
            }
        }
        const R wab = wa * wb;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            wgv[i] += wab * Zg[i];
            wmb[i] += wab * Zm[i];
            if (a) GB[3 * i + 0] += (R(a) * wab) * Zm[i];
            if (b) GB[3 * i + 1] += (R(b) * wab) * Zm[i];
            GB[3 * i + 2] += wab * Zc[i];
        }
        if (advect) {
            xs[0] += (dwa * wb) * Sab;
            xs[1] += (wa * dwb) * Sab;
            xs[2] += wab * Tab;
        }
    };
    if (warp_all(stencil_interior(sc, base))) {
        R w[3][3], dw[3][3];
        bspline(fx, w);
        bspline_grad(fx, dw);
        const R wz[3] = {w[0][2], w[1][2], w[2][2]}, dwz[3] = {dw[0][2], dw[1][2], dw[2][2]};
        const int ny = sc.shape[1], nz = sc.shape[2];
        long long n0 = ax.node_begin + ((base[0] * ny + base[1]) * nz + base[2]);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (a) loads_after(n0, xs[2]);
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const long long r = n0 + (a * ny + b) * nz;
                const long long node[3] = {r, r + 1, r + 2};
                row(a, b, w[a][0], dw[a][0], w[b][1], dw[b][1], wz, dwz, node);
            }
        }
    } else {
        stencil_rows(sc, ax, base, fx, row);
    }
    R xb[3] = {xs[0] * inv_dx, xs[1] * inv_dx, xs[2] * inv_dx};
    R Sb[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int d = 0; d < 3; ++d) Sb[3 * i + d] = dx * (GB[3 * i + d] - wmb[i] * fx[d]);
    // the constitutive VJP needs F, C, Fg again: reload rather than keep them live
    ld9<R>(in.C, p, in.sp9, in.sc9, C);
    ld9<R>(in.F, p, in.sp9, in.sc9, F);
    gr.load(ctx, sc, in, p, t, gphi);
    R Fb[9], vb[3], Cb[9], skb[9], taub[9];
    {
        R Cn[9], Fnb[9];
        ld9<R>(outC, p, in.sp9, in.sc9, Cn);
        ld9<R>(ob.F, p, ob.sp9, ob.sc9, Fnb);
        R A[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) A[i] = ((i % 4 == 0) ? R(1) : R(0)) + dt * Cn[i];
        mTm(A, Fnb, Fb);   // (I + dt Cn)^T Fn_b
    }
    if (advect) {
        R xnb[3];
        ld3<R>(ob.x, p, ob.sp3, ob.sc3, xnb);
#pragma unroll
        for (int i = 0; i < 3; ++i)
            xb[i] += xnb[i] - inv_dx * (D1[3 * i] * wgv[0] + D1[3 * i + 1] * wgv[1] + D1[3 * i + 2] * wgv[2]
                                      + D2[3 * i] * wmb[0] + D2[3 * i + 1] * wmb[1] + D2[3 * i + 2] * wmb[2]);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) vb[i] = pm * wmb[i];
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        Cb[i] = pm * Sb[i];
        skb[i] = dt * Sb[i];
        taub[i] = c * skb[i];
    }
    R Fb2[9], Fgb[9], Cb2[9];
    {
        // volatile: reload here rather than keep the values live in registers
        volatile R* ks = &keep_s[0][threadIdx.x];
#pragma unroll
        for (int i = 0; i < 13; ++i) keep[i] = ks[i * 256];
    }
    if (EXT && M.kind == MPM_MODEL_EXTERNAL) {
        // the caller applies its own stress VJP to tau_bar
        st9<R>(ctx.ext_tau_bar, p, 9, 1, taub);
#pragma unroll
        for (int i = 0; i < 9; ++i) Fb2[i] = Fgb[i] = Cb2[i] = R(0);
    } else {
        fb |= model_vjp_keep(M, ctx.gap_thresh, F, gr.g, C, taub, keep, Fb2, Fgb, Cb2);
    }
    if (fb) atomicAdd(ctx.fallbacks, 1ull);
    if constexpr (MAT) {
        double gm[2];
        model_param_grad(M, F, gr.g, keep, taub, gm);
        dmat[sidx] = gm[0];
        dmat[ctx.n + sidx] = gm[1];
    }
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        Fb[i] += Fb2[i];
        Cb[i] += Cb2[i];
    }
    // volume path: c = -k4 vol0 det(Fg)
    R Fgi[9];
    R dFg = gr.g.inverse(Fgi);
    R vol = frob(skb, tau) * (-k4 * vol0) * dFg;
    double Fgl[9];      // with ISO only the diagonal is used
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) Fgl[3 * i + j] = (double)Fgb[3 * i + j] + (double)(vol * Fgi[3 * j + i]);

    st3<R>(ib.x, p, ib.sp3, ib.sc3, xb);
    st3<R>(ib.v, p, ib.sp3, ib.sc3, vb);
    st9<R>(ib.C, p, ib.sp9, ib.sc9, Cb);
    st9<R>(ib.F, p, ib.sp9, ib.sc9, Fb);
    if (!ISO && ib.Fg) {
        double* o = ib.Fg + p * ib.sp9;
        const double* in_g = ob.Fg ? ob.Fg + p * ob.sp9 : nullptr;
#pragma unroll
        for (int i = 0; i < 9; ++i) o[i * ib.sc9] = (in_g ? in_g[i * ob.sc9] : 0.0) + Fgl[i];
    }
    if (dA) dA[sidx] = (sc.growth_mode == 1) ? (Fgl[0] + Fgl[4] + Fgl[8]) * (double)gphi : 0.0;
    if (!finite9(Fb) || !finite9(Cb)) raise_status(ctx.status, MPM_ERR_NONFINITE);
    unmark_cell(ctx, ax, tp.skeys, sidx);
}

// ---------------------------------------------------------------------------
// deterministic per-scene reduction of a per-slot double buffer:
// out[s * stride] = (accumulate ? out[s * stride] : 0) + scale_s * sum_{slots of s} v
// scale_s = 1 (mode 0) or 1/n_s (mode 1)
// Each block sums one chunk of REDUCE_CHUNK slots of a scene (an empty scene has
// one chunk too); the last block of a scene to arrive (a counter per scene, back
// at 0 afterwards) adds the chunks' sums in chunk order, so the order depends
// only on the scene's size.  The chunks come from a table: scenes by chunks of
// the largest one as a grid launched 248,000 blocks for 4062 chunks on 4000
// scenes of 50 particles beside one of 2M (671 us, now 44).
// One block per scene took 242 us on a scene of 2.1M particles, on one SM; its
// 64 chunks take 10 us.  A second block costs about 1 us of waiting, so a
// chunk is as large as still pays: one scene of 32768 particles 4.3 us whole,
// 5.3 in two chunks; 256 scenes of up to 65536 14.8 us, 19.1 in chunks of 8192.
// ---------------------------------------------------------------------------
constexpr int REDUCE_THREADS = 1024;
constexpr int REDUCE_CHUNK = 32768;
struct SumChunk {
    long long begin, end;       // the scene's slots
    int scene;
    int first;                  // its first chunk in the table
};
// sum of one value per thread over the block, on thread 0 (fixed shuffle tree)
__device__ __forceinline__ double reduce_block(double acc, double* wsum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) wsum[warp] = acc;
    __syncthreads();
    double r = 0.0;
    if (warp == 0) {
        r = wsum[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    }
    return r;
}
__global__ void __launch_bounds__(REDUCE_THREADS)
scene_reduce_kernel(const double* __restrict__ v, double* __restrict__ out, double* __restrict__ part,
                    unsigned* __restrict__ arrived, const SumChunk* __restrict__ table, int accumulate, int mean,
                    int stride) {
    __shared__ double wsum[REDUCE_THREADS / 32];
    __shared__ bool is_last;
    const SumChunk chunk = table[blockIdx.x];
    const int s = chunk.scene, first = chunk.first, c = (int)blockIdx.x - first;
    const long long b = chunk.begin, e = chunk.end;
    const int chunks = e > b ? (int)((e - b + REDUCE_CHUNK - 1) / REDUCE_CHUNK) : 1;
    const long long c0 = b + (long long)c * REDUCE_CHUNK, c1 = c0 + REDUCE_CHUNK < e ? c0 + REDUCE_CHUNK : e;
    // two interleaved chains per thread, then a fixed shuffle tree
    double a0 = 0.0, a1 = 0.0;
    long long i = c0 + threadIdx.x;
#pragma unroll 4
    for (; i + REDUCE_THREADS < c1; i += 2 * REDUCE_THREADS) {
        a0 += v[i];
        a1 += v[i + REDUCE_THREADS];
    }
    if (i < c1) a0 += v[i];
    double r = reduce_block(a0 + a1, wsum);
    if (chunks > 1) {
        double* mine = part + first;
        if (threadIdx.x == 0) {
            mine[c] = r;
            __threadfence();
            is_last = atomicAdd(arrived + s, 1u) == (unsigned)chunks - 1u;
        }
        __syncthreads();
        if (!is_last) return;
        __threadfence();
        double a = 0.0;
        for (int k = threadIdx.x; k < chunks; k += REDUCE_THREADS) a += __ldcg(mine + k);
        r = reduce_block(a, wsum);
        if (threadIdx.x == 0) arrived[s] = 0u;
    }
    if (threadIdx.x == 0) {
        if (mean) r /= (double)(e - b > 0 ? e - b : 1);
        out[(long long)s * stride] = accumulate ? out[(long long)s * stride] + r : r;
    }
}

// dst[r][i] = src[r][order[i]]: a thread takes one column, its index read once,
// eight rows' loads in flight.  torch.index_select over (24, n) re-reads the
// 8-byte indices for every element: 232 us on 4.7M FP32 particles of 256 scenes
// and 164 on a sheet of 2.1M, here 181 and 81 (0.9 and 0.4 GB).
constexpr int GATHER_ROWS = 8;
template <typename R>
__global__ void __launch_bounds__(256)
gather_columns_kernel(const R* __restrict__ src, R* __restrict__ dst, const int* __restrict__ order, int rows,
                      long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int q = order[i];
    if (!MPM_INB(q, n, 9)) return;
    for (int r0 = 0; r0 < rows; r0 += GATHER_ROWS) {
        R v[GATHER_ROWS];
#pragma unroll
        for (int r = 0; r < GATHER_ROWS; ++r)
            if (r0 + r < rows) v[r] = src[(r0 + r) * n + q];
#pragma unroll
        for (int r = 0; r < GATHER_ROWS; ++r)
            if (r0 + r < rows) dst[(r0 + r) * n + i] = v[r];
    }
}

// loss seeds (integrate.py:41-52): sum det F with F_bar = det F F^{-T};
// mean |x - x_obs|^2 with x_bar = 2 (x - x_obs) / n_s
template <typename R>
__global__ void __launch_bounds__(256)
loss_detF_kernel(Ctx ctx, const R* __restrict__ F, long long sp9, long long sc9, double* __restrict__ vals,
                 R* __restrict__ Fb) {
    long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= ctx.n) return;
    R A[9], Ai[9];
    ld9<R>(F, p, sp9, sc9, A);
    R d = inv3(A, Ai);
    vals[p] = (double)d;
    if (Fb) {
        R o[9];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) o[3 * i + j] = d * Ai[3 * j + i];
        st9<R>(Fb, p, sp9, sc9, o);
    }
}
template <typename R>
__global__ void __launch_bounds__(256)
loss_mse_kernel(Ctx ctx, const R* __restrict__ x, long long sp3, long long sc3, const R* __restrict__ xo,
                double* __restrict__ vals, R* __restrict__ xb) {
    long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= ctx.n) return;
    const MpmScene& sc = ctx.scenes[ctx.scene_of[p]];
    R a[3], b[3];
    ld3<R>(x, p, sp3, sc3, a);
    ld3<R>(xo, p, sp3, sc3, b);
    double n = (double)(sc.p_end - sc.p_begin);
    double acc = 0.0;
    R o[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        R d = a[i] - b[i];
        acc += (double)d * (double)d;
        o[i] = (R)(2.0 / n) * d;
    }
    vals[p] = acc;
    if (xb) st3<R>(xb, p, sp3, sc3, o);
}

// ---------------------------------------------------------------------------
// constitutive seam, batched over n particles of one model.  The (n, 3, 3)
// arrays are contiguous: a warp moves the 288 values of its 32 particles as
// nine coalesced rows through shared memory (a lane's own nine values lie 9
// apart there, on distinct banks), so every sector is fetched once.  With the
// strided loads and the out-of-line Hencky VJP, whose arrays went through the
// local-memory stack, the pair took 207 us on 1.05M FP32 Hencky particles (37
// stress, 167 VJP), now 101 (39 and 62: the eigensolve's instructions bound
// both); neo-Hookean 192, now 71; Herschel-Bulkley 189, now 86; FP64 368, 260
// and 266, now 241, 108 and 157.
// ---------------------------------------------------------------------------
constexpr int SEAM_THREADS = 128;
template <typename R>
__device__ __forceinline__ void seam_load(const R* __restrict__ A, long long w0, long long n, R* sh, R o[9]) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const long long e = 9 * w0 + 32 * k + lane;
        sh[32 * k + lane] = e < 9 * n ? A[e] : ((32 * k + lane) % 9 % 4 == 0 ? R(1) : R(0));
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 9; ++i) o[i] = sh[9 * lane + i];
}
template <typename R>
__device__ __forceinline__ void seam_store(R* __restrict__ A, long long w0, long long n, R* sh, const R o[9]) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 9; ++i) sh[9 * lane + i] = o[i];
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const long long e = 9 * w0 + 32 * k + lane;
        if (e < 9 * n) A[e] = sh[32 * k + lane];
    }
}
// KIND: the scene's model.  The elastic models do not read C.
template <typename R, int KIND>
__global__ void __launch_bounds__(SEAM_THREADS, sizeof(R) == 4 ? 10 : 8)
stress_kernel(MpmScene sc, long long n, const R* __restrict__ F, const R* __restrict__ Fg, const R* __restrict__ C,
              R* __restrict__ tau, float thresh) {
    __shared__ R sh_all[SEAM_THREADS / 32][288];
    R* sh = sh_all[threadIdx.x >> 5];
    const long long w0 = (long long)blockIdx.x * SEAM_THREADS + (threadIdx.x & ~31);    // the warp's first particle
    if (w0 >= n) return;
    ModelParams<R> M;
    M.load(sc);
    M.kind = KIND;
    R f[9], g[9], c[9], t[9];
    seam_load(F, w0, n, sh, f);
    seam_load(Fg, w0, n, sh, g);
#pragma unroll
    for (int i = 0; i < 9; ++i) c[i] = R(0);
    if (KIND == MPM_MODEL_HERSCHEL_BULKLEY && C) seam_load(C, w0, n, sh, c);
    model_stress(M, thresh, f, GrowthFull<R>(g), c, t);
    seam_store(tau, w0, n, sh, t);
}
template <typename R, int KIND>
__global__ void __launch_bounds__(SEAM_THREADS, sizeof(R) == 4 ? 7 : 5)
stress_vjp_kernel(MpmScene sc, long long n, const R* __restrict__ F, const R* __restrict__ Fg,
                  const R* __restrict__ C, const R* __restrict__ tb, R* __restrict__ Fb, R* __restrict__ Fgb,
                  R* __restrict__ Cb, float thresh) {
    __shared__ R sh_all[SEAM_THREADS / 32][288];
    R* sh = sh_all[threadIdx.x >> 5];
    const long long w0 = (long long)blockIdx.x * SEAM_THREADS + (threadIdx.x & ~31);
    if (w0 >= n) return;
    ModelParams<R> M;
    M.load(sc);
    M.kind = KIND;
    R f[9], g[9], c[9], t[9], a[9], b[9], e[9];
    seam_load(F, w0, n, sh, f);
    seam_load(Fg, w0, n, sh, g);
    seam_load(tb, w0, n, sh, t);
#pragma unroll
    for (int i = 0; i < 9; ++i) c[i] = e[i] = R(0);
    if (KIND == MPM_MODEL_HERSCHEL_BULKLEY && C) seam_load(C, w0, n, sh, c);
    model_vjp(M, thresh, f, GrowthFull<R>(g), c, t, a, b, e);
    seam_store(Fb, w0, n, sh, a);
    seam_store(Fgb, w0, n, sh, b);
    if (Cb) seam_store(Cb, w0, n, sh, e);
}

}  // namespace mpm
