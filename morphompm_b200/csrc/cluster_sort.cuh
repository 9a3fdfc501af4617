// One-launch sort of a small plan: the full radix sort of the cell keys, the
// segment table and the active-tile list of one step, by one thread-block
// cluster whose CTAs hold the keys in shared memory and exchange them through
// distributed shared memory.
//
// What bounds it: latency.  A plan of a few thousand particles is sorted in
// microseconds, but the general path (sort.cuh and the seg_* / tile_* kernels)
// spends 14 to 24 dependent launches of 1.5 to 4 us on it.  In a captured
// forward + adjoint trajectory the passes take 9.7 us for 4096 particles (two
// of 8 bits) and 17.6 us for 32768 (two of 9 bits) against about 46 us for
// those launches: 40 FP32 steps 4.23 -> 2.76 ms and 4.78 -> 3.48 ms, bitwise
// the same results.  About a quarter of that at 32768 is the scatter through
// distributed shared memory (4000 to 6000 cycles a pass).
#pragma once

#include <cooperative_groups.h>

#include "mpm_common.cuh"
#include "sort.cuh"

namespace mpm {

constexpr int CS_THREADS = 1024;
constexpr int CS_WARPS = CS_THREADS / 32;
// 8 CTAs, the portable cluster size (16 measured slower: 32768 particles 20.1 us
// against 19.1, 64^3 grid 26.9 against 24.5)
constexpr int CS_MAX_CTAS = 8;
constexpr int CS_MAX_ITEMS = 8;         // keys per thread
constexpr int CS_MAX_BITS = 10;         // digit bits per pass
constexpr unsigned CS_MOVERS = 1024;    // particles of a merge (ranked by counting): at most CS_THREADS
// A plan up to CS_MAX_N particles takes this path: the size the 8 CTAs hold at
// CS_MAX_ITEMS keys per thread.  It is still the faster side there (40 FP32
// steps of 64000 particles, with the general path and with the passes: 5.25 and
// 4.19 ms on a 40^3 grid, 5.91 and 4.64 ms on 150^3, 55k tiles).  Its CTAs walk
// all tiles of the grid, hence the cap on them: with few particles, so few CTAs,
// it is still the faster side there (forward + reverse step of 1000 FP32 particles
// on 64,000 tiles 81 us, on 68,921 by the general path 155; 61 us on 4096 tiles).
// The cluster takes its CTAs before a thread takes a second key (4096
// particles: 9.7 us with 4 CTAs, 11.3 with 2, 12.9 with 1).
constexpr long long CS_MAX_TILES = 1 << 16;
constexpr long long CS_MAX_N = (long long)CS_MAX_CTAS * CS_THREADS * CS_MAX_ITEMS;

// dynamic shared memory of one CTA: keys and values of its slots, the digit
// totals and offsets, and the per-warp digit counts
inline size_t cluster_sort_smem(int items, int bits) {
    return (size_t)items * CS_THREADS * 8 + (size_t)(1 << CS_MAX_BITS) * 8 + (size_t)CS_WARPS * (size_t)(1 << bits) * 2;
}

// exclusive prefix over the block of one value per thread
__device__ __forceinline__ unsigned cs_block_exclusive(unsigned v, unsigned* wsum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned inc = v;
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
    return wsum[warp] + inc - v;
}

// CTA r of the cluster owns the sorted slots [r S, (r + 1) S), S = 1024 ITEMS;
// warp w of it the consecutive chunk of 32 ITEMS slots.  Each pass is a stable
// counting sort by one digit: every key's rank among its warp's equal digits
// (warp match masks), a prefix of the warps' counts per digit, the CTAs' digit
// totals read over distributed shared memory, and a scatter into the owning
// CTA's shared memory.  The result is the stable radix sort's: (key, particle)
// order.  Then the segment table (as seg_write_kernel) and the active-tile
// list (as tile_write_kernel) come from one exchange of the CTAs' counts.
//
// A chained step starts from the previous step's order (old_keys, old_perm;
// null otherwise; possibly skeys and perm themselves).  When at most CS_MOVERS
// particles changed their key, the passes are replaced by a merge, as in the
// incremental re-sort of sort.cuh: every CTA collects all movers, ranks them by
// (key, particle) and places the slots it owns.  32768 particles with about 160
// movers: 13.1 us against 17.6 for two passes of 9 bits; 4096: 8.4 against 9.7.
template <int ITEMS>
__global__ void __launch_bounds__(CS_THREADS, 1)
cluster_sort_kernel(Ctx ctx, const unsigned* __restrict__ keys, const unsigned* old_keys, const unsigned* old_perm,
                    unsigned* skeys, unsigned* perm, int passes, int bits, int* __restrict__ tile_flag,
                    int* __restrict__ active, int* __restrict__ n_active) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    constexpr int S = ITEMS * CS_THREADS;
    constexpr int SHIFT = 10 + (ITEMS == 8 ? 3 : (ITEMS == 4 ? 2 : (ITEMS == 2 ? 1 : 0)));
    extern __shared__ __align__(16) unsigned cs_smem[];
    uint2* kv_s = reinterpret_cast<uint2*>(cs_smem);      // (key, particle) of this CTA's slots
    unsigned* tot_s = cs_smem + 2 * S;
    unsigned* base_s = tot_s + (1 << CS_MAX_BITS);
    unsigned short* wh = reinterpret_cast<unsigned short*>(base_s + (1 << CS_MAX_BITS));
    __shared__ unsigned wsum[CS_WARPS];
    __shared__ uint2 cta_cnt;                // segment starts, active tiles of this CTA
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int rank = (int)cluster.block_rank(), C = (int)cluster.num_blocks();
    const long long n = ctx.n;
    const int R = 1 << bits;
    const int loc0 = warp * (32 * ITEMS) + lane;      // this thread's first slot in the CTA
    const long long q0 = (long long)rank * S + loc0;
    unsigned short* wrow = wh + (size_t)warp * R;

    // active tiles of this warp's chunk of the tile range
    const long long per_warp = ((ctx.n_tiles + (long long)C * CS_WARPS - 1) / ((long long)C * CS_WARPS) + 31) / 32 * 32;
    const long long t0 = ((long long)rank * CS_WARPS + warp) * per_warp;
    const long long t1 = t0 + per_warp < ctx.n_tiles ? t0 + per_warp : ctx.n_tiles;
    const long long cell0 = ctx.aux[0].cell_begin, ncells = ctx.aux[0].ncells;
    unsigned k[ITEMS], v[ITEMS], rk[ITEMS];
    // the movers that the emitting G2P counted (read by all CTAs before the
    // first cluster barrier, set back after it)
    const unsigned n_moved = *(volatile unsigned*)ctx.moved_count;
    // (the passes' keys do not wait for that count)
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const long long q = q0 + i * 32;
        k[i] = q < n ? keys[q] : 0xffffffffu;
        v[i] = (unsigned)q;
    }
    unsigned tiles = 0;
    for (long long t = t0; t < t1; t += 32) {
        const bool on = t + lane < t1 && tile_flag[t + lane] != 0;
        tiles += __popc(__ballot_sync(0xffffffffu, on));
    }

    const bool merged = old_keys && n_moved <= CS_MOVERS;
    if (merged) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const long long q = q0 + i * 32;
            k[i] = q < n ? old_keys[q] : 0xffffffffu;
            v[i] = q < n ? old_perm[q] : 0u;
        }
        __shared__ unsigned long long mine_s[CS_MOVERS], all_s[CS_MOVERS], sorted_s[CS_MOVERS];
        __shared__ unsigned mpre[CS_WARPS];
        __shared__ unsigned cta_movers;
        // movers of this CTA's slots, in slot order
        unsigned moved = 0, count = 0;
        unsigned nk[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) nk[i] = q0 + i * 32 < n && MPM_INB(v[i], n, 9) ? keys[v[i]] : k[i];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const bool mv = nk[i] != k[i];
            moved |= (mv ? 1u : 0u) << i;
            count += __popc(__ballot_sync(0xffffffffu, mv));
        }
        // the pair before each round's first slot (lane 0)
        unsigned long long before_pair[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const long long q = q0 + i * 32;
            before_pair[i] = lane == 0 && q > 0 && q < n ? pair_key(old_keys[q - 1], old_perm[q - 1]) : 0ull;
        }
        if (lane == 0) mpre[warp] = count;
        __syncthreads();
        if (warp == 0) {
            const unsigned c = mpre[lane];
            unsigned inc = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned t = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += t;
            }
            mpre[lane] = inc - c;
            if (lane == 31) cta_movers = inc;
        }
        __syncthreads();
        unsigned run = mpre[warp];               // movers of this CTA before the round
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const bool mv = (moved >> i) & 1u;
            const unsigned ball = __ballot_sync(0xffffffffu, mv);
            const unsigned at = run + __popc(ball & lt);
            rk[i] = at;                          // movers of this CTA before the slot
            if (mv && at < CS_MOVERS) mine_s[at] = pair_key(nk[i], v[i]);
            run += __popc(ball);
        }
        cluster.sync();
        unsigned m = 0, m_before = 0, first[CS_MAX_CTAS];
#pragma unroll
        for (int r = 0; r < CS_MAX_CTAS; ++r) {
            const unsigned c = r < C ? *cluster.map_shared_rank(&cta_movers, r) : 0u;
            first[r] = m;
            m_before += r < rank ? c : 0u;
            m += c;
        }
        m = m < CS_MOVERS ? m : CS_MOVERS;       // (equal to n_moved)
        for (unsigned t = threadIdx.x; t < m; t += CS_THREADS) {
            int owner = 0;
            unsigned from = 0;
#pragma unroll
            for (int r = 1; r < CS_MAX_CTAS; ++r)
                if (r < C && t >= first[r]) {
                    owner = r;
                    from = first[r];
                }
            all_s[t] = cluster.map_shared_rank(mine_s, owner)[t - from];
        }
        __syncthreads();
        // ranks by counting, `sub` lanes to a mover: a few movers by every CTA for
        // itself, more of them in shares that are sent to all CTAs
        const bool split = m > CS_THREADS / 4;
        const unsigned share = split ? (m + C - 1) / C : m;
        unsigned sub = 32;
        while (sub > 1 && share * sub > CS_THREADS) sub >>= 1;
        // share * sub <= CS_THREADS: one mover per group of sub lanes
        const unsigned part = threadIdx.x % sub, g = threadIdx.x / sub, t = (split ? rank * share : 0u) + g;
        const bool has = g < share && t < m;
        const unsigned long long mine = has ? all_s[t] : 0ull;
        unsigned less = 0;
        if (has) {
#pragma unroll 4
            for (unsigned j = part; j < m; j += sub) less += all_s[j] < mine ? 1u : 0u;
        }
        for (unsigned o = sub >> 1; o > 0; o >>= 1) less += __shfl_xor_sync(0xffffffffu, less, o);
        if (split) {
            if (has)
                for (int r = (int)part; r < C; r += (int)sub) cluster.map_shared_rank(sorted_s, r)[less] = mine;
            cluster.sync();
        } else {
            if (has && part == 0) sorted_s[less] = mine;
            __syncthreads();
        }
        // movers ordered before the pair p
        auto bound = [&](unsigned long long p) {
            unsigned lo = 0, hi = m;
            while (lo < hi) {
                const unsigned mid = (lo + hi) >> 1;
                if (sorted_s[mid] < p) lo = mid + 1;
                else hi = mid;
            }
            return lo;
        };
        auto put = [&](long long pos, unsigned key, unsigned part) {
            if (MPM_INB(pos, n, 10))
                cluster.map_shared_rank(kv_s, (int)(pos >> SHIFT))[pos & (S - 1)] = make_uint2(key, part);
        };
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const long long q = q0 + i * 32;
            const unsigned b = q < n ? bound(pair_key(k[i], v[i])) : m;
            unsigned b_prev = __shfl_up_sync(0xffffffffu, b, 1);
            if (lane == 0) b_prev = q > 0 && q < n ? bound(before_pair[i]) : 0u;
            if (q < n) {
                // slots that keep their key before this one
                const long long stay = q - (long long)(m_before + rk[i]);
                if (!((moved >> i) & 1u)) put(stay + b, k[i], v[i]);
                for (unsigned j = b_prev; j < b; ++j) {
                    const unsigned long long p = sorted_s[j];
                    put(stay + j, (unsigned)(p >> 32), (unsigned)p);
                }
                if (q + 1 == n)
                    for (unsigned j = b; j < m; ++j) {
                        const unsigned long long p = sorted_s[j];
                        put(n - (long long)m + j, (unsigned)(p >> 32), (unsigned)p);
                    }
            }
        }
        cluster.sync();
    }
    for (int pass = 0; pass < (merged ? 0 : passes); ++pass) {
        const int shift = pass * bits;
        if (pass > 0) {
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const uint2 kv = kv_s[loc0 + i * 32];
                k[i] = kv.x;
                v[i] = kv.y;
            }
        }
        for (int d = lane; d < R / 2; d += 32) reinterpret_cast<unsigned*>(wrow)[d] = 0;
        __syncwarp();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const bool valid = q0 + i * 32 < n;
            const unsigned dig = (k[i] >> shift) & (R - 1);
            const unsigned peers = __match_any_sync(0xffffffffu, valid ? dig : 0xffffffffu);
            const unsigned cnt = valid ? wrow[dig] : 0u;
            __syncwarp();
            if (valid && (peers & lt) == 0u) wrow[dig] = (unsigned short)(cnt + __popc(peers));
            __syncwarp();
            rk[i] = cnt + __popc(peers & lt);
        }
        __syncthreads();
        if (threadIdx.x < R) {
            // all of a half's loads before its stores: one shared-memory latency, not 16
            unsigned run = 0;
            unsigned short* col = wh + threadIdx.x;
#pragma unroll
            for (int w0 = 0; w0 < CS_WARPS; w0 += 16) {
                unsigned c[16];
#pragma unroll
                for (int w = 0; w < 16; ++w) c[w] = col[(w0 + w) * R];
#pragma unroll
                for (int w = 0; w < 16; ++w) {
                    col[(w0 + w) * R] = (unsigned short)run;
                    run += c[w];
                }
            }
            tot_s[threadIdx.x] = run;
        }
        cluster.sync();
        unsigned all = 0, before = 0;
        if (threadIdx.x < R) {
#pragma unroll
            for (int r = 0; r < CS_MAX_CTAS; ++r) {      // unrolled: the remote loads are in flight together
                const unsigned t = r < C ? cluster.map_shared_rank(tot_s, r)[threadIdx.x] : 0u;
                all += t;
                before += r < rank ? t : 0u;
            }
        }
        const unsigned ex = cs_block_exclusive(all, wsum);
        if (threadIdx.x < R) base_s[threadIdx.x] = ex + before;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (q0 + i * 32 < n) {
                const unsigned dig = (k[i] >> shift) & (R - 1);
                const unsigned pos = base_s[dig] + wrow[dig] + rk[i];
                if (MPM_INB(pos, n, 10)) {
                    const int dst = (int)(pos >> SHIFT), off = (int)(pos & (S - 1));
                    cluster.map_shared_rank(kv_s, dst)[off] = make_uint2(k[i], v[i]);
                }
            }
        }
        cluster.sync();
    }

    // sorted order out; segment starts and ends
    unsigned start = 0, last = 0, starts = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const long long q = q0 + i * 32;
        const int l = loc0 + i * 32;
        const bool valid = q < n;
        bool a = false, b = false;
        if (valid) {
            const uint2 kv = kv_s[l];
            k[i] = kv.x;
            skeys[q] = kv.x;
            perm[q] = kv.y;
            const unsigned prv = l > 0 ? kv_s[l - 1].x : (rank > 0 ? cluster.map_shared_rank(kv_s, rank - 1)[S - 1].x : 0u);
            a = q == 0 || prv != k[i];
            unsigned nxt = 0;
            if (q + 1 < n) nxt = l < S - 1 ? kv_s[l + 1].x : cluster.map_shared_rank(kv_s, rank + 1)[0].x;
            b = q + 1 == n || nxt != k[i];
            if (a || b) {
                long long c0 = cell0, nc = ncells;
                if (ctx.n_scenes > 1) {
                    const SceneAux& ax = ctx.aux[ctx.scene_of[q]];
                    c0 = ax.cell_begin;
                    nc = ax.ncells;
                }
                if ((long long)k[i] - c0 >= nc) a = b = false;
            }
        }
        start |= (a ? 1u : 0u) << i;
        last |= (b ? 1u : 0u) << i;
        starts += __popc(__ballot_sync(0xffffffffu, a));
    }
    // the warps' prefixes of starts and tiles (lane 0 carries its warp's counts), then the CTAs'
    __shared__ unsigned wpre[2][CS_WARPS];
    if (lane == 0) {
        wpre[0][warp] = starts;
        wpre[1][warp] = tiles;
    }
    __syncthreads();
    if (warp < 2) {
        const unsigned c = wpre[warp][lane];
        unsigned inc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        wpre[warp][lane] = inc - c;
        if (lane == 31) (warp == 0 ? cta_cnt.x : cta_cnt.y) = inc;
    }
    cluster.sync();
    unsigned seg_before = 0, tile_before = 0, seg_all = 0, tile_all = 0;
#pragma unroll
    for (int r = 0; r < CS_MAX_CTAS; ++r) {
        const uint2 c = r < C ? *cluster.map_shared_rank(&cta_cnt, r) : make_uint2(0u, 0u);
        seg_before += r < rank ? c.x : 0u;
        tile_before += r < rank ? c.y : 0u;
        seg_all += c.x;
        tile_all += c.y;
    }
    cluster.sync();           // no CTA's shared memory is read after this
    unsigned run = seg_before + wpre[0][warp];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const long long q = q0 + i * 32;
        const bool st = (start >> i) & 1u;
        const unsigned ball = __ballot_sync(0xffffffffu, st);
        const unsigned id = run + __popc(ball & lt) + (st ? 1u : 0u);
        if (st && MPM_INB(id - 1, n, 3)) {
            ctx.seg_first[id - 1] = (int)q;
            if (MPM_INB(k[i], ctx.n_keys, 2)) ctx.cell_seg[k[i]] = (int)id;
        }
        if (((last >> i) & 1u) && id > 0 && MPM_INB(id - 1, n, 3)) ctx.seg_last[id - 1] = (int)(q + 1);
        run += __popc(ball);
    }
    unsigned tr = tile_before + wpre[1][warp];
    for (long long t = t0; t < t1; t += 32) {
        const bool on = t + lane < t1 && tile_flag[t + lane] != 0;
        const unsigned ball = __ballot_sync(0xffffffffu, on);
        if (on) {
            const unsigned at = tr + __popc(ball & lt);
            if (at < (unsigned)ctx.active_cap) active[at] = (int)(t + lane);
            tile_flag[t + lane] = 0;
        }
        tr += __popc(ball);
    }
    if (rank == 0 && threadIdx.x == 0) {
        *ctx.moved_count = 0u;
        *ctx.n_seg = (int)seg_all;
        if (tile_all > (unsigned)ctx.active_cap) {
            raise_status(ctx.status, MPM_ERR_ARG);
            tile_all = (unsigned)ctx.active_cap;
        }
        *n_active = (int)tile_all;
    }
}

}  // namespace mpm
