// Refinement (sources/refinement.cu:18-582 and kernels/refinement.cu:9-652 restated with exact
// integer arithmetic and a sparse per-hyperedge census instead of the dense E x K table).
//
// One round:
//  1. census: for every hyperedge the partitions among its pins with (pins, destination pins), a
//     set in no particular order; partition sizes and distinct-inbound counts. k-way rounds without
//     an inbound limit keep two masks per hyperedge instead (k_kway_records).
//  2. gains: every node's best feasible target among the partitions adjacent to it; only moves
//     with positive gain are proposed. From per-hyperedge partition masks (O(K/32) per incidence
//     and lane) or from sums by partition or hash (O(lambda) per incidence).
//  3. rank by (gain desc, id asc), k-way in pairs.
//  4. cascade: each move's gain recomputed assuming every better-ranked move is applied. Hyperedges
//     of at most CM_LEN pins compare ranks pin by pin; longer ones gather their movers once and
//     sweep over them in rank order with exact prefix counts, or count events by partition.
//  5. prefix sums of cascaded gains; size-excess and inbound-validity of every prefix from sorted
//     event streams (sources/refinement.cu:239-491); best prefix by best_move_functor
//     (headers/data_types.cuh:113-136); apply when valid with non-negative prefix gain.
//
// Work lists that depend only on the level (hyperedge-length tiers, per-node gain-work bounds)
// are built once per level. Inside a round every count stays in device memory; the host reads a
// single word per round (whether moves were applied), which drives the round schedule.
#include <cstdlib>
#include <type_traits>

#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"
#include "blocksort.cuh"

namespace cg = cooperative_groups;

namespace axc {
namespace {

constexpr u32 CS_WARP_CAP = 256;
constexpr u32 CS_BLOCK_CAP = 4096;
constexpr u32 CS_WARPS = 4;

// Slots of a block's census or candidate hash table for `len` keys: a power of two, at most 2/3
// full. The hyperedge's entries and their order do not depend on it.
__host__ __device__ __forceinline__ u32 cs_cap(u64 len) {
    u32 cap = 32;
    while (cap < len + (len >> 1)) cap <<= 1;
    return cap;
}
// Bytes of dynamic shared memory this launch was given.
__device__ __forceinline__ u32 dyn_smem_bytes() {
    u32 b;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(b));
    return b;
}

// What a node saves by leaving partition p of a hyperedge (weight w) where p holds c of its pins:
// INCC (encourage) floor(w / c^2), k-way w when the node is the last pin in p.
__device__ __forceinline__ i64 leave_gain(int encourage, u32 w, u32 c) {
    if (encourage) return c >= 1 ? (i64)((u64)w / ((u64)c * c)) : 0;
    return c == 1 ? (i64)w : 0;
}

// ------------------------------------------------------------------ census
struct CensusArgs {
    const u64 *off;
    const u32 *pins, *nsrc, *part;
    u32 *cpart, *ccnt, *cdcnt, *lam;
    u32 *status;
    // when set: every pin adds leave_gain(w, count of its partition) to its node's saving
    unsigned long long *save;
    const u32 *wfx;
    int encourage;
    // partition-indexed census only, when set: the hyperedge's masks of partitions present and
    // with destination pins, mw words each
    u32 *mask, *dmask;
    u32 mw;
    // when set (kernel timer on k_census_direct_warp): each hyperedge's algorithmic bytes are added
    unsigned long long *pbytes;
};

// insert phase: keys = partition, mn = first position, cnt/dcnt counters
__device__ __forceinline__ void cs_insert(const CensusArgs &A, u64 a, u64 b, u64 s, u32 *keys, u32 *mn, u32 *cnt,
                                          u32 *dcnt, u32 mask, u32 t, u32 nt) {
    for (u64 k = a + t; k < b; k += nt) {
        u32 p = A.part[A.pins[k]];
        u32 slot = hash_find_or_insert(keys, mask, p);
        if (slot == NONE) { atomicExch(A.status, DEV_HASH_FULL); continue; }
        atomicMin(&mn[slot], (u32)(k - a));
        atomicAdd(&cnt[slot], 1u);
        if (k >= s) atomicAdd(&dcnt[slot], 1u);
    }
}

// The hashed census by hyperedge length. Every kernel reads a pin's partition once; the entries of a
// hyperedge come in no particular order (all consumers read them as a set).
//  - at most CS_SHORT pins: a warp stages the partitions of consecutive hyperedges in shared memory
//    and every pin counts its own among its hyperedge's (no table);
//  - up to CS_WARP_CAP: one warp, a hash table of packed counts; the pin that inserts a partition
//    writes its entry;
//  - up to CS_BLOCK_CAP: one block, the same with the counts indexed by partition up to CS_DIRECT_K
//    partitions, hashed above;
//  - longer: one block, a table in device memory (k_census_block).
constexpr u32 CS_SHORT = 32;
constexpr u32 CS_STAGE = 512;        // pins a warp stages
constexpr u32 CS_THREADS = 256;
constexpr u32 CS_DIRECT_K = 16384;

// Bound by the partitions' gathers. Measured: 1M nets 651 us by a warp and a table per net, 92.
__global__ void __launch_bounds__(CS_THREADS) k_census_short(u32 e, CensusArgs A, u32 per_warp) {
    constexpr u32 NW = CS_THREADS / 32;
    __shared__ u32 sp[NW][CS_STAGE];
    __shared__ u32 sn[NW][32];
    const u32 w = threadIdx.x >> 5, lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    u32 *st = sp[w], *num = sn[w];
    const u32 step = gridDim.x * NW * per_warp;
    for (u32 h0 = (blockIdx.x * NW + w) * per_warp; h0 < e; h0 += step) {
        const u32 h = h0 + lane;
        const bool mine = lane < per_warp && h < e;
        const u64 a = mine ? A.off[h] : 0, len64 = mine ? A.off[h + 1] - a : 0;
        const bool take = mine && len64 <= CS_SHORT;
        const u32 len = take ? (u32)len64 : 0u, ns = take ? A.nsrc[h] : 0u;
        const u32 wh = take && A.save ? A.wfx[h] : 0u;
        u32 x = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if ((int)lane >= o) x += y;
        }
        const u32 excl = x - len;
        num[lane] = 0;
        for (u32 lo = 0; lo < 32;) {  // as many of the hyperedges as the stage holds at a time
            const u32 b0 = __shfl_sync(0xFFFFFFFFu, excl, lo);
            const u32 hi = lo + __popc(__ballot_sync(0xFFFFFFFFu, lane >= lo && x - b0 <= CS_STAGE));
            const u32 T = __shfl_sync(0xFFFFFFFFu, x, hi - 1) - b0;
            for (u32 pass = 0; pass < 2; ++pass) {
                for (u32 f0 = 0; f0 < T; f0 += 32) {
                    const u32 f = f0 + lane;
                    u32 ol = lo, oh = hi - 1;  // owner: the last hyperedge starting at or before f
                    for (int it = 0; it < 5; ++it) {
                        const u32 mid = (ol + oh + 1) >> 1;
                        const u32 em = __shfl_sync(0xFFFFFFFFu, excl, mid & 31);
                        if (ol < oh) { if (em - b0 <= f) ol = mid; else oh = mid - 1; }
                    }
                    const u32 eo = __shfl_sync(0xFFFFFFFFu, excl, ol) - b0;
                    const u64 ao = __shfl_sync(0xFFFFFFFFu, a, ol);
                    const bool in = f < T;
                    if (pass == 0) {
                        if (in) st[f] = A.part[A.pins[ao + (f - eo)]];
                        continue;
                    }
                    const u32 lo_len = __shfl_sync(0xFFFFFFFFu, len, ol), no = __shfl_sync(0xFFFFFFFFu, ns, ol);
                    const u32 wo = __shfl_sync(0xFFFFFFFFu, wh, ol);
                    u32 c = 0, dc = 0, p = 0;
                    bool first = in;
                    if (in) {
                        p = st[f];
                        for (u32 j = 0; j < lo_len; ++j) {
                            const bool same = st[eo + j] == p;
                            c += same;
                            dc += same && j >= no;
                            first = first && !(same && eo + j < f);
                        }
                        if (A.save) {
                            const i64 g = leave_gain(A.encourage, wo, c);
                            if (g) atomicAdd(&A.save[A.pins[ao + (f - eo)]], (unsigned long long)g);
                        }
                    }
                    // the firsts of one hyperedge in this chunk are consecutive lanes, after those of
                    // earlier chunks (num)
                    const u32 bal = __ballot_sync(0xFFFFFFFFu, first);
                    const u32 s0 = in && eo > f0 ? eo - f0 : 0;  // the owner's first lane of this chunk
                    const u32 seg = s0 < 32 ? 0xFFFFFFFFu << s0 : 0u;
                    const u32 had = in ? num[ol] : 0u;
                    __syncwarp();
                    if (first) {
                        const u64 dst = ao + had + __popc(bal & lt & seg);
                        A.cpart[dst] = p;
                        A.ccnt[dst] = c;
                        A.cdcnt[dst] = dc;
                    }
                    // the owner's last lane of this chunk
                    if (in && (lane == 31 || f + 1 == eo + lo_len || f + 1 == T))
                        num[ol] = had + __popc(bal & (lt | (1u << lane)) & seg);
                    __syncwarp();
                }
                __syncwarp();
            }
            lo = hi;
        }
        if (take) A.lam[h] = num[lane];
        __syncwarp();  // num is no longer read
    }
}

// Measured with k_census_mid: 20 x 5000 network at some 10k partitions 1060 us by hash tables sized
// by the hyperedge, 185 + 338 (34M gathers).
__global__ void __launch_bounds__(CS_WARPS * 32) k_census_warp(u32 e, CensusArgs A, u32 per_warp) {
    __shared__ u32 tk[CS_WARPS][2 * CS_WARP_CAP], tv[CS_WARPS][2 * CS_WARP_CAP];
    constexpr u32 R = CS_WARP_CAP / 32;
    const u32 w = threadIdx.x >> 5, lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    const u32 h0 = (blockIdx.x * CS_WARPS + w) * per_warp;
    u32 *keys = tk[w], *val = tv[w];
    const u32 hl = h0 + lane;
    const u64 al = lane < per_warp && hl < e ? A.off[hl] : 0, ll = lane < per_warp && hl < e ? A.off[hl + 1] - al : 0;
    u32 todo = __ballot_sync(0xFFFFFFFFu, ll > CS_SHORT && ll <= CS_WARP_CAP);
    while (todo) {
        const u32 t = __ffs(todo) - 1;
        todo &= todo - 1;
        const u32 h = h0 + t, len = (u32)__shfl_sync(0xFFFFFFFFu, ll, t);
        const u64 a = __shfl_sync(0xFFFFFFFFu, al, t);
        const u32 ns = A.nsrc[h], wh = A.save ? A.wfx[h] : 0u;
        u32 cap = 64;
        while (cap < 2 * len) cap <<= 1;
        u32 v[R], q[R];
#pragma unroll
        for (u32 i = 0; i < R; ++i) v[i] = lane + 32 * i < len ? A.pins[a + lane + 32 * i] : 0;
#pragma unroll
        for (u32 i = 0; i < R; ++i) q[i] = lane + 32 * i < len ? A.part[v[i]] : 0;
        for (u32 i = lane; i < cap; i += 32) { keys[i] = NONE; val[i] = 0; }
        __syncwarp();
        u32 fresh = 0;  // bit i: this lane's pin i inserted its partition
#pragma unroll
        for (u32 i = 0; i < R; ++i) {
            if (lane + 32 * i >= len) continue;
            bool f;
            const u32 slot = hash_insert_fresh(keys, cap - 1, q[i], f);
            if (slot == NONE) { atomicExch(A.status, DEV_HASH_FULL); q[i] = 0; continue; }
            atomicAdd(&val[slot], (1u << 16) | (lane + 32 * i >= ns ? 1u : 0u));
            q[i] = slot;
            fresh |= (u32)f << i;
        }
        __syncwarp();
        u32 o = 0;
#pragma unroll
        for (u32 i = 0; i < R; ++i) {
            if (32 * i >= len) break;
            const bool in = lane + 32 * i < len;
            const u32 c = in ? val[q[i]] : 0u;
            if (A.save && in) {
                const i64 g = leave_gain(A.encourage, wh, c >> 16);
                if (g) atomicAdd(&A.save[v[i]], (unsigned long long)g);
            }
            const bool f = (fresh >> i) & 1u;
            const u32 bal = __ballot_sync(0xFFFFFFFFu, f);
            if (f) {
                const u64 dst = a + o + __popc(bal & lt);
                A.cpart[dst] = keys[q[i]];
                A.ccnt[dst] = c >> 16;
                A.cdcnt[dst] = c & 0xFFFFu;
            }
            o += __popc(bal);
        }
        if (lane == 0) A.lam[h] = o;
        __syncwarp();  // the tables are no longer read
    }
}

// Listed hyperedges of CS_WARP_CAP < |e| <= CS_BLOCK_CAP pins, one block at a time each. DIRECT: the
// counts are indexed by partition (T = K words, all zero between hyperedges), else a hash table
// sized by the hyperedge (T slots at most).
template <bool DIRECT>
__global__ void __launch_bounds__(CS_THREADS) k_census_mid(const u32 *__restrict__ list, u32 nlist, CensusArgs A, u32 T) {
    extern __shared__ u32 cm_dyn[];
    __shared__ unsigned short slot[CS_BLOCK_CAP];
    __shared__ u32 s_n;
    constexpr u32 FRESH = 0x8000u;
    static_assert(CS_DIRECT_K <= FRESH && 2 * CS_BLOCK_CAP <= FRESH, "a slot and its flag fit 16 bits");
    u32 *val = cm_dyn, *keys = cm_dyn + T;
    const u32 lane = threadIdx.x & 31u;
    if (DIRECT)
        for (u32 i = threadIdx.x; i < T; i += CS_THREADS) val[i] = 0;
    for (u32 idx = blockIdx.x; idx < nlist; idx += gridDim.x) {
        const u32 h = list[idx];
        const u64 a = A.off[h];
        const u32 len = (u32)(A.off[h + 1] - a), ns = A.nsrc[h];
        const u32 cap = DIRECT ? 0 : cs_cap(len);
        if (!DIRECT && cap > T) {  // launched with too small a table: refuse
            if (threadIdx.x == 0) atomicExch(A.status, DEV_HASH_FULL);
            continue;
        }
        if (!DIRECT)
            for (u32 i = threadIdx.x; i < cap; i += CS_THREADS) { keys[i] = NONE; val[i] = 0; }
        if (threadIdx.x == 0) s_n = 0;
        __syncthreads();
        constexpr u32 U = 4;
        for (u32 k0 = threadIdx.x; k0 < len; k0 += U * CS_THREADS) {
            u32 q[U];
#pragma unroll
            for (u32 x = 0; x < U; ++x) q[x] = k0 + x * CS_THREADS < len ? A.pins[a + k0 + x * CS_THREADS] : 0;
#pragma unroll
            for (u32 x = 0; x < U; ++x) q[x] = k0 + x * CS_THREADS < len ? A.part[q[x]] : 0;
#pragma unroll
            for (u32 x = 0; x < U; ++x) {
                const u32 k = k0 + x * CS_THREADS;
                if (k >= len) continue;
                u32 s = q[x];
                bool f = false;
                if (!DIRECT) {
                    s = hash_insert_fresh(keys, cap - 1, q[x], f);
                    if (s == NONE) { atomicExch(A.status, DEV_HASH_FULL); slot[k] = 0; continue; }
                }
                const u32 old = atomicAdd(&val[s], (1u << 16) | (k >= ns ? 1u : 0u));
                if (DIRECT) f = old == 0;
                slot[k] = (unsigned short)(s | (f ? FRESH : 0u));
            }
        }
        __syncthreads();
        const u32 wh = A.save ? A.wfx[h] : 0u;
        for (u32 kb = 0; kb < len; kb += CS_THREADS) {
            const u32 k = kb + threadIdx.x;
            const u32 s = k < len ? slot[k] : 0u;
            const u32 c = k < len ? val[s & (FRESH - 1)] : 0u;
            if (A.save && k < len) {
                const i64 g = leave_gain(A.encourage, wh, c >> 16);
                if (g) atomicAdd(&A.save[A.pins[a + k]], (unsigned long long)g);
            }
            const bool f = (s & FRESH) != 0;
            const u32 bal = __ballot_sync(0xFFFFFFFFu, f);
            u32 at = 0;
            if (lane == 0 && bal) at = atomicAdd(&s_n, (u32)__popc(bal));
            at = __shfl_sync(0xFFFFFFFFu, at, 0);
            if (f) {
                const u64 dst = a + at + __popc(bal & ((1u << lane) - 1u));
                A.cpart[dst] = DIRECT ? (s & (FRESH - 1)) : keys[s & (FRESH - 1)];
                A.ccnt[dst] = c >> 16;
                A.cdcnt[dst] = c & 0xFFFFu;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) A.lam[h] = s_n;
        if (DIRECT)
            for (u32 k = threadIdx.x; k < len; k += CS_THREADS)
                if (slot[k] & FRESH) val[slot[k] & (FRESH - 1)] = 0;
        __syncthreads();
    }
}

// Hyperedges of more than CS_BLOCK_CAP pins: one block each, the table (keys, first positions, counts)
// in device memory.
__global__ void k_census_block(const u32 *__restrict__ list, u32 nlist, CensusArgs A, u32 *gtab,
                               const u64 *__restrict__ gtab_off) {
    __shared__ u32 wsum[33];
    if (blockIdx.x >= nlist) return;
    const u32 h = list[blockIdx.x];
    const u64 a = A.off[h], b = A.off[h + 1], s = a + A.nsrc[h];
    const u32 len = (u32)(b - a);
    const u32 cap = cs_cap(len);
    u32 *keys = gtab + 4 * gtab_off[blockIdx.x];
    u32 *mn = keys + cap, *cnt = mn + cap, *dcnt = cnt + cap;
    for (u32 i = threadIdx.x; i < cap; i += blockDim.x) { keys[i] = NONE; mn[i] = NONE; cnt[i] = 0; dcnt[i] = 0; }
    __syncthreads();
    cs_insert(A, a, b, s, keys, mn, cnt, dcnt, cap - 1, threadIdx.x, blockDim.x);
    __syncthreads();
    u32 o = 0;  // running count, identical in every thread
    const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (u64 base = a; base < b; base += blockDim.x) {
        u64 k = base + threadIdx.x;
        u32 slot = NONE, p = 0;
        if (k < b) {
            p = A.part[A.pins[k]];
            slot = hash_find(keys, cap - 1, p);
        }
        if (A.save && slot != NONE)
            atomicAdd(&A.save[A.pins[k]], (unsigned long long)leave_gain(A.encourage, A.wfx[h], cnt[slot]));
        bool first = slot != NONE && mn[slot] == (u32)(k - a);
        u32 bal = __ballot_sync(0xFFFFFFFFu, first);
        if (lane == 0) wsum[w] = __popc(bal);
        __syncthreads();
        u32 before = 0, tot = 0;
        for (u32 i = 0; i < nw; ++i) {
            if (i < w) before += wsum[i];
            tot += wsum[i];
        }
        if (first) {
            u64 dst = a + o + before + __popc(bal & ((1u << lane) - 1u));
            A.cpart[dst] = p;
            A.ccnt[dst] = cnt[slot];
            A.cdcnt[dst] = dcnt[slot];
        }
        o += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) A.lam[h] = o;
}

// Partition-indexed census for K <= CD_K: the counters are K-slot arrays indexed by partition id,
// so a hyperedge of any length fits in shared memory and needs no hashing. Entries are emitted in
// ascending partition order (the hashed census emits them in no order; every
// consumer reads them as a set). With A.save set, every pin then adds its saving from the count
// of its own partition.
constexpr u32 CD_K = 256;
constexpr u32 CD_WARP_LEN = 1024;  // longer hyperedges take a block

// Counts of hyperedge h's pins over [t0, len) step nt into cnt / dcnt (shared, zeroed).
__device__ __forceinline__ void cd_count(const CensusArgs &A, u64 a, u64 b, u64 s, u32 *cnt, u32 *dcnt, u32 t0,
                                         u32 nt) {
    for (u64 k = a + t0; k < b; k += nt) {
        const u32 q = A.part[A.pins[k]];
        atomicAdd(&cnt[q], 1u);
        if (k >= s) atomicAdd(&dcnt[q], 1u);
    }
}
// Returns how many savings this thread added.
__device__ __forceinline__ u32 cd_save(const CensusArgs &A, u32 h, u64 a, u64 b, const u32 *cnt, u32 t0, u32 nt) {
    if (!A.save) return 0;
    const u32 w = A.wfx[h];
    u32 added = 0;
    for (u64 k = a + t0; k < b; k += nt) {
        const u32 v = A.pins[k];
        const i64 g = leave_gain(A.encourage, w, cnt[A.part[v]]);
        if (g) {
            atomicAdd(&A.save[v], (unsigned long long)g);
            ++added;
        }
    }
    return added;
}
// One warp: the nonzero counters in ascending partition order, then lam. The ballots of the
// counters are the hyperedge's masks, written when A.mask is set.
// Returns the entries written (lam).
__device__ __forceinline__ u32 cd_emit(const CensusArgs &A, u32 h, u64 a, const u32 *cnt, const u32 *dcnt, u32 K) {
    const u32 lane = threadIdx.x & 31;
    u32 o = 0;
    const u32 qend = A.mask ? 32 * A.mw : K;
    for (u32 qb = 0; qb < qend; qb += 32) {
        const u32 q = qb + lane;
        const u32 c = q < K ? cnt[q] : 0;
        const u32 bal = __ballot_sync(0xFFFFFFFFu, c > 0);
        if (A.mask) {
            const u32 dbal = __ballot_sync(0xFFFFFFFFu, c > 0 && dcnt[q] > 0);
            if (lane == 0) {
                A.mask[(u64)h * A.mw + qb / 32] = bal;
                A.dmask[(u64)h * A.mw + qb / 32] = dbal;
            }
        }
        if (c > 0) {
            const u64 dst = a + o + __popc(bal & ((1u << lane) - 1u));
            A.cpart[dst] = q;
            A.ccnt[dst] = c;
            A.cdcnt[dst] = dcnt[q];
        }
        o += __popc(bal);
    }
    if (lane == 0) A.lam[h] = o;
    return o;
}

__global__ void k_census_direct_warp(u32 e, CensusArgs A, u32 K) {
    __shared__ u32 tc[CS_WARPS][CD_K], td[CS_WARPS][CD_K];
    const u32 w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u32 h = blockIdx.x * CS_WARPS + w;
    if (h >= e) return;
    const u64 a = A.off[h], b = A.off[h + 1], s = a + A.nsrc[h];
    if (b - a > CD_WARP_LEN) return;
    u32 *cnt = tc[w], *dcnt = td[w];
    for (u32 i = lane; i < K; i += 32) { cnt[i] = 0; dcnt[i] = 0; }
    __syncwarp();
    cd_count(A, a, b, s, cnt, dcnt, lane, 32);
    __syncwarp();
    const u32 saved = __reduce_add_sync(0xFFFFFFFFu, cd_save(A, h, a, b, cnt, lane, 32));
    const u32 lm = cd_emit(A, h, a, cnt, dcnt, K);
    if (A.pbytes && lane == 0)  // algorithmic bytes (kernel timer): offsets and source count, each
        // pin's id and partition, the entries and their count, the masks, the weight and savings
        prof_add(A.pbytes, h, 20 + 8 * (b - a) + 12ull * lm + 4 + (A.mask ? 8ull * A.mw : 0) +
                                  (A.save ? 4 + 8ull * saved : 0));
}

__global__ void k_census_direct_block(const u32 *__restrict__ list, u32 nlist, CensusArgs A, u32 K) {
    __shared__ u32 cnt[CD_K], dcnt[CD_K];
    for (u32 idx = blockIdx.x; idx < nlist; idx += gridDim.x) {
        const u32 h = list[idx];
        const u64 a = A.off[h], b = A.off[h + 1], s = a + A.nsrc[h];
        for (u32 i = threadIdx.x; i < K; i += blockDim.x) { cnt[i] = 0; dcnt[i] = 0; }
        __syncthreads();
        cd_count(A, a, b, s, cnt, dcnt, threadIdx.x, blockDim.x);
        __syncthreads();
        cd_save(A, h, a, b, cnt, threadIdx.x, blockDim.x);
        if (threadIdx.x < 32) cd_emit(A, h, a, cnt, dcnt, K);
        __syncthreads();
    }
}

// ---- incremental partition-indexed census (levels that are not small, K <= CD_K) ---------------
// The level keeps one census across its rounds. Round r recomputes only the hyperedges holding a
// node that moved in round r - 1 (all of them in round 0): their entries, count and masks are
// rewritten, and each pin's saving changes by leave_gain(w, its partition's new count) minus
// leave_gain(w, its partition's count at the previous census). A node's partition at the
// previous census is its current one, unless it moved in round r - 1: then the apply kernel kept
// the old one in prev[] and stamped the move with the round counter. The results are those of a
// census rebuilt from scratch (integer sums, the same entries in the same order).
struct IncArgs {
    const u32 *list, *nlist;   // the hyperedges to recompute
    u32 *work;                 // the warps' work counter (zeroed before the launch)
    const u32 *dirty;          // their flags (the block kernel's filter)
    const u32 *prev, *stamp;   // [n]
    const u32 *ctr;            // rounds run at this level (0 in round 0)
};

// Old counts from the hyperedge's previous entries [a, a + lm) into ocnt (zeroed, K slots).
__device__ __forceinline__ void ci_old_counts(const CensusArgs &A, u64 a, u32 lm, u32 *ocnt, u32 t0, u32 nt) {
    for (u32 j = t0; j < lm; j += nt) ocnt[A.cpart[a + j]] = A.ccnt[a + j];
}
// The savings' change of pins t0, t0 + nt, ... (all of their saving in round 0); returns how many
// this thread added.
__device__ __forceinline__ u32 ci_save(const CensusArgs &A, const IncArgs &I, u32 h, u64 a, u64 b, const u32 *cnt,
                                       const u32 *ocnt, u32 r, u32 t0, u32 nt) {
    const u32 w = A.wfx[h];
    u32 added = 0;
    for (u64 k = a + t0; k < b; k += nt) {
        const u32 v = A.pins[k], p = A.part[v];
        i64 g = leave_gain(A.encourage, w, cnt[p]);
        if (r) {
            const u32 po = I.stamp[v] == r - 1 ? I.prev[v] : p;
            g -= leave_gain(A.encourage, w, ocnt[po]);
        }
        if (g) {
            atomicAdd(&A.save[v], (unsigned long long)g);
            ++added;
        }
    }
    return added;
}

// Listed hyperedges of at most CD_WARP_LEN pins, one warp each; warps take 32 list entries at a
// time from a shared counter.
__global__ void k_census_inc_warp(CensusArgs A, u32 K, IncArgs I) {
    __shared__ u32 tc[CS_WARPS][CD_K], td[CS_WARPS][CD_K], to[CS_WARPS][CD_K];
    const u32 w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u32 nl = *I.nlist, r = *I.ctr;
    u32 *cnt = tc[w], *dcnt = td[w], *ocnt = to[w];
    u64 bytes = 0;  // algorithmic bytes of this warp's hyperedges (kernel timer)
    for (;;) {
        u32 base = 0;
        if (lane == 0) base = atomicAdd(I.work, 32u);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= nl) break;
        const u32 end = base + 32 < nl ? base + 32 : nl;
        for (u32 idx = base; idx < end; ++idx) {
            const u32 h = I.list[idx];
            const u64 a = A.off[h], b = A.off[h + 1], s = a + A.nsrc[h];
            if (b - a > CD_WARP_LEN) continue;  // the block kernel's
            const u32 lm_old = r ? A.lam[h] : 0;
            __syncwarp();  // the previous hyperedge's tables are no longer read
            for (u32 i = lane; i < K; i += 32) { cnt[i] = 0; dcnt[i] = 0; ocnt[i] = 0; }
            __syncwarp();
            if (r) ci_old_counts(A, a, lm_old, ocnt, lane, 32);
            cd_count(A, a, b, s, cnt, dcnt, lane, 32);
            __syncwarp();  // old entries read, counts complete, before the entries are rewritten
            const u32 saved = __reduce_add_sync(0xFFFFFFFFu, ci_save(A, I, h, a, b, cnt, ocnt, r, lane, 32));
            const u32 lm = cd_emit(A, h, a, cnt, dcnt, K);
            // the list entry, offsets and source count, each pin's id, partition (and move stamp),
            // the old entries, the new entries and their count, the masks, the weight and savings
            bytes += 24 + 12 * (b - a) + 8ull * lm_old + 12ull * lm + 4 + (A.mask ? 8ull * A.mw : 0) + 4 +
                     8ull * saved;
        }
    }
    if (A.pbytes && lane == 0 && bytes) prof_add(A.pbytes, blockIdx.x * CS_WARPS + w, bytes);
}

// Hyperedges of more than CD_WARP_LEN pins (the level's block list), one block each, when flagged.
__global__ void k_census_inc_block(const u32 *__restrict__ list, u32 nlist, CensusArgs A, u32 K, IncArgs I) {
    __shared__ u32 cnt[CD_K], dcnt[CD_K], ocnt[CD_K];
    const u32 r = *I.ctr;
    for (u32 idx = blockIdx.x; idx < nlist; idx += gridDim.x) {
        const u32 h = list[idx];
        if (!I.dirty[h]) continue;  // uniform over the block
        const u64 a = A.off[h], b = A.off[h + 1], s = a + A.nsrc[h];
        const u32 lm_old = r ? A.lam[h] : 0;
        for (u32 i = threadIdx.x; i < K; i += blockDim.x) { cnt[i] = 0; dcnt[i] = 0; ocnt[i] = 0; }
        __syncthreads();
        if (r) ci_old_counts(A, a, lm_old, ocnt, threadIdx.x, blockDim.x);
        cd_count(A, a, b, s, cnt, dcnt, threadIdx.x, blockDim.x);
        __syncthreads();
        ci_save(A, I, h, a, b, cnt, ocnt, r, threadIdx.x, blockDim.x);
        __syncthreads();  // every thread has read lam and the old entries
        if (threadIdx.x < 32) cd_emit(A, h, a, cnt, dcnt, K);
        __syncthreads();
    }
}

// After the apply: the hyperedges of the nodes this round moved (stamped with the round counter)
// are flagged for the next round's census. One warp per mover.
__global__ void k_mark_moved(const u32 *__restrict__ mv, const u32 *__restrict__ dM, const u32 *__restrict__ stamp,
                             const u32 *__restrict__ ctr, const u64 *__restrict__ toff, const u32 *__restrict__ touch,
                             u32 *__restrict__ dirty) {
    const u32 lane = threadIdx.x & 31u, nw = (gridDim.x * blockDim.x) >> 5;
    const u32 M = *dM, r = *ctr;
    for (u32 i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < M; i += nw) {
        const u32 v = mv[i];
        if (stamp[v] != r) continue;  // not applied this round
        for (u64 j = toff[v] + lane; j < toff[v + 1]; j += 32) dirty[touch[j]] = 1u;
    }
}
__global__ void k_round_tick(u32 *ctr) {
    if (threadIdx.x == 0 && blockIdx.x == 0) ctr[0] += 1;
}

// The hashed census's block (n[0]) and device-table (n[1]) hyperedges.
__global__ void __launch_bounds__(1024) k_census_lists(u32 e, const u64 *__restrict__ off, u32 *mid, u32 *huge,
                                                       u32 *__restrict__ n) {
    __shared__ u32 sh[33];
    const u32 h = blockIdx.x * blockDim.x + threadIdx.x;
    const u64 len = h < e ? off[h + 1] - off[h] : 0;
    if (!__syncthreads_or(len > CS_WARP_CAP)) return;
    const bool m = len > CS_WARP_CAP && len <= CS_BLOCK_CAP, g = len > CS_BLOCK_CAP;
    const u32 am = block_append(m, n, sh);
    if (m) mid[am] = h;
    if (!__syncthreads_or(g)) return;
    const u32 ag = block_append(g, n + 1, sh);
    if (g) huge[ag] = h;
}
__global__ void k_tab_sizes(const u32 *__restrict__ list, u32 nl, const u64 *__restrict__ off, u64 *__restrict__ sz) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == nl) sz[i] = 0;
    if (i >= nl) return;
    u32 h = list[i];
    u64 len = off[h + 1] - off[h], cap = 32;
    while (cap < 2 * len) cap <<= 1;
    sz[i] = cap;
}

__global__ void k_part_sizes(u32 n, const u32 *__restrict__ part, const u32 *__restrict__ nsize,
                             unsigned long long *__restrict__ ps) {
    u32 v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) atomicAdd(&ps[part[v]], (unsigned long long)(nsize ? nsize[v] : 1u));
}
// Few partitions (K <= PS_SMEM_K): per-block sums in shared memory, one global add per partition
// and block. A size is added in 16-bit halves, each a native 32-bit add (64-bit ones would be
// compare-and-swap loops on a few words), so a block takes at most PS_NODES nodes. Where the room
// allows, a partition has a counter per lane (rep = 32): lanes of one partition do not collide.
constexpr u32 PS_SMEM_K = 1024;
constexpr u32 PS_NODES = 65536;
__global__ void __launch_bounds__(256) k_part_sizes_smem(u32 n, u32 K, u32 rep, u32 per_block,
                                                         const u32 *__restrict__ part, const u32 *__restrict__ nsize,
                                                         unsigned long long *__restrict__ ps) {
    extern __shared__ u32 ps_sh[];  // lo[K * rep], hi[K * rep]
    u32 *lo = ps_sh, *hi = ps_sh + K * rep;
    for (u32 i = threadIdx.x; i < 2 * K * rep; i += blockDim.x) ps_sh[i] = 0;
    __syncthreads();
    const u32 l = threadIdx.x & (rep - 1);
    const u64 v0 = (u64)blockIdx.x * per_block, v1 = v0 + per_block < n ? v0 + per_block : n;
#pragma unroll 4
    for (u64 v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
        const u32 q = part[v], s = nsize ? nsize[v] : 1u;
        if (q >= K) continue;  // ids are below K by contract
        atomicAdd(&lo[q * rep + l], s & 0xFFFFu);
        if (s >> 16) atomicAdd(&hi[q * rep + l], s >> 16);
    }
    __syncthreads();
    for (u32 i = threadIdx.x; i < K; i += blockDim.x) {
        u64 t = 0;
        for (u32 x = 0; x < rep; ++x) {
            const u32 y = i * rep + ((x + i) & (rep - 1));
            t += (u64)lo[y] + ((u64)hi[y] << 16);
        }
        if (t) atomicAdd(&ps[i], (unsigned long long)t);
    }
}
__global__ void k_part_inbound(u32 e, const u64 *__restrict__ off, const u32 *__restrict__ lam,
                               const u32 *__restrict__ cpart, const u32 *__restrict__ cdcnt,
                               unsigned long long *__restrict__ pinb) {
    const u32 h = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (h >= e) return;
    const u64 a = off[h];
    for (u32 j = lane; j < lam[h]; j += 32)
        if (cdcnt[a + j] > 0) atomicAdd(&pinb[cpart[a + j]], 1ull);
}

constexpr u32 PI_SMEM_K = 49152;
constexpr u32 PI_THREADS = 1024;
// k_part_inbound for K <= PI_SMEM_K: groups of G lanes stride over the hyperedges and count into a
// shared histogram, which the block adds to pinb once: one large block per SM, since every block
// adds up to K words to the same places. G follows the mean length (a census has no more entries).
// Measured: 1M nets 495 us with a warp per net, 44; 20 x 5000 network 292 us by global atomics, 159
// in shared memory.
template <u32 G>
__global__ void __launch_bounds__(PI_THREADS) k_part_inbound_smem(u32 e, const u64 *__restrict__ off,
                                                                  const u32 *__restrict__ lam,
                                                                  const u32 *__restrict__ cpart,
                                                                  const u32 *__restrict__ cdcnt, u32 K,
                                                                  unsigned long long *__restrict__ pinb) {
    extern __shared__ u32 hist[];
    for (u32 i = threadIdx.x; i < K; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const u32 gl = threadIdx.x & (G - 1);
    constexpr u32 per = PI_THREADS / G;
    for (u32 h = blockIdx.x * per + threadIdx.x / G; h < e; h += gridDim.x * per) {
        const u64 a = off[h];
        const u32 lm = lam[h];
        for (u32 j = gl; j < lm; j += G)
            if (cdcnt[a + j] > 0) atomicAdd(&hist[cpart[a + j]], 1u);
    }
    __syncthreads();
    for (u32 i = threadIdx.x; i < K; i += blockDim.x)
        if (hist[i]) atomicAdd(&pinb[i], (unsigned long long)hist[i]);
}

// ------------------------------------------------------------------ gains
struct GainArgs {
    u32 n, omega, delta, discount, round;
    u32 seed;
    int encourage;
    const u64 *off;
    const u32 *lam, *cpart, *ccnt, *cdcnt, *wfx;
    const u32 *pins, *nsrc;  // the level's hyperedges (pin-centric passes)
    const u64 *toff;
    const u32 *touch, *nin, *nsize, *part;
    const u64 *psize, *pinb;
    u32 *target;
    i64 *gain;
    u32 *status;
    const u32 *dyn;  // when set: discount and round read from device memory (graph replays)
    const i64 *save; // partition-indexed gains: each node's saving from leaving its partition
    u32 K;           // partitions
};

constexpr u32 GN_DIRECT_K = 256;

// Slots of a node's hash table from its work bound.
__device__ __forceinline__ u32 gain_cap(u64 work, u32 cap_max) {
    u32 cap = 32;
    while (cap < 2 * work && cap < cap_max) cap <<= 1;
    return cap;
}

// The launch's arguments with the per-round scalars resolved.
__device__ __forceinline__ GainArgs gain_args_now(const GainArgs &A0) {
    GainArgs A = A0;
    if (A0.dyn) {
        A.discount = A0.dyn[0];
        A.round = A0.dyn[1];
    }
    return A;
}

// Per-level bounds of a node's gain work: the partitions adjacent to it in any round number at
// most min(sum over incident hyperedges of min(|e|, K), K), which sizes its accumulator table; the
// sum of incident weights bounds its gain. G lanes a node; the block takes those of more than
// GB_HEAVY incidences a lane (GB_HEAVY_WARP for a warp) together.
// Measured: 1M nodes 169 us a level, 664 at the first (an atomic per node at one address), 45. A node of
// 300,000 incidences among 120,000 of few: 10.3 ms with four lanes, 3.8 with a warp, 0.37 with the block.
constexpr u32 GB_HEAVY = 64, GB_HEAVY_WARP = 8192;
template <u32 G>
__global__ void __launch_bounds__(256) k_gain_bounds(u32 n, u32 K, const u64 *__restrict__ toff,
                                                     const u32 *__restrict__ touch, const u64 *__restrict__ off,
                                                     const u32 *__restrict__ wfx, u64 *__restrict__ work,
                                                     u64 *__restrict__ wsum, unsigned long long *__restrict__ wmax) {
    __shared__ u64 top[8], rs[8];
    __shared__ u32 heavy[256 / G], nheavy;
    if (threadIdx.x == 0) nheavy = 0;
    __syncthreads();
    const u32 u = (blockIdx.x * 256 + threadIdx.x) / G, own = threadIdx.x & (G - 1);
    u64 s = 0, ws = 0;
    const auto add = [&](u64 j0, u64 j1, u32 step) {
        for (u64 j = j0; j < j1; j += step) {
            const u32 h = touch[j];
            const u64 len = off[h + 1] - off[h];
            s += len < K ? len : K;
            ws += wfx[h];
        }
    };
    bool light = false;
    if (u < n) {
        const u64 t0 = toff[u], t1 = toff[u + 1];
        light = t1 - t0 <= (G == 32 ? GB_HEAVY_WARP : GB_HEAVY * G);
        if (light) add(t0 + own, t1, G);
        else if (own == 0) heavy[atomicAdd(&nheavy, 1u)] = u;
    }
#pragma unroll
    for (u32 o = G / 2; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
        ws += __shfl_xor_sync(0xFFFFFFFFu, ws, o);
    }
    if (light && own == 0) {
        work[u] = s < K ? s : K;
        if (wsum) wsum[u] = ws;
    }
    // the largest of the block in one atomic: one per node met at a single address
    u64 most = warp_max_u64(ws);
    __syncthreads();
    for (u32 i = 0; i < nheavy; ++i) {
        const u32 v = heavy[i];
        s = ws = 0;
        add(toff[v] + threadIdx.x, toff[v + 1], 256);
        s = warp_sum(s);
        ws = warp_sum(ws);
        if ((threadIdx.x & 31) == 0) {
            rs[threadIdx.x >> 5] = s;
            top[threadIdx.x >> 5] = ws;
        }
        __syncthreads();
        s = ws = 0;
        for (u32 x = 0; x < 8; ++x) {
            s += rs[x];
            ws += top[x];
        }
        if (threadIdx.x == 0) {
            work[v] = s < K ? s : K;
            if (wsum) wsum[v] = ws;
        }
        most = ws > most ? ws : most;
        __syncthreads();  // rs and top are no longer read
    }
    if ((threadIdx.x & 31) == 0) top[threadIdx.x >> 5] = most;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (u32 i = 1; i < 8; ++i) most = top[i] > most ? top[i] : most;
        if (most) atomicMax(wmax, (unsigned long long)most);
    }
}

// Accumulate node u's adjacency to other partitions into (keys, conn, dconn). Warp-cooperative:
// the calling warp takes the node's incidences in batches of 32 starting at `first`, every
// `stride` entries. A batch's hyperedge metadata loads in parallel; its census entries are then
// flattened across the lanes (each lane finds its entry's hyperedge by a 5-step search over the
// prefix of the batch's lambdas). saving and wtot are per-lane partial sums.
template <bool WIDE>
__device__ __forceinline__ void gain_flat(const GainArgs &A, u32 u, u32 p, u32 *keys, u32 *conn, u32 *high, u32 *dconn,
                                          u32 mask, u32 first, u32 stride, i64 &saving, i64 &wtot) {
    const u32 lane = threadIdx.x & 31u;
    const u64 t0 = A.toff[u];
    const u32 deg = (u32)(A.toff[u + 1] - t0), nin_u = A.nin[u];
    for (u32 jb = first; jb < deg; jb += stride) {
        const u32 j = jb + lane;
        const bool has = j < deg;
        const u32 h = has ? A.touch[t0 + j] : 0;
        const u32 lm = has ? A.lam[h] : 0;
        const u32 wh = has ? A.wfx[h] : 0;
        const u64 ah = has ? A.off[h] : 0;
        const u32 ib = (has && j < nin_u) ? 1u : 0u;
        wtot += wh;
        u32 x = lm;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            u32 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if ((int)lane >= o) x += y;
        }
        const u32 total = __shfl_sync(0xFFFFFFFFu, x, 31), excl = x - lm;
        const u32 chunk = (deg - jb) < 32 ? (deg - jb) : 32;
        for (u32 fb = 0; fb < total; fb += 32) {
            const u32 f = fb + lane;
            u32 lo = 0, hi = chunk - 1;
            for (int it = 0; it < 5; ++it) {
                const u32 mid = (lo + hi + 1) >> 1;
                const u32 em = __shfl_sync(0xFFFFFFFFu, excl, mid & 31);
                if (lo < hi) { if (em <= f) lo = mid; else hi = mid - 1; }
            }
            const u32 eo = __shfl_sync(0xFFFFFFFFu, excl, lo);
            const u64 ao = __shfl_sync(0xFFFFFFFFu, ah, lo);
            const u32 wo = __shfl_sync(0xFFFFFFFFu, wh, lo);
            const u32 io = __shfl_sync(0xFFFFFFFFu, ib, lo);
            if (f >= total) continue;
            const u64 k = ao + (f - eo);
            const u32 q = A.cpart[k];
            if (q == p) {
                saving += leave_gain(A.encourage, wo, A.ccnt[k]);
                continue;
            }
            const u32 slot = hash_find_or_insert(keys, mask, q);
            if (slot == NONE) { atomicExch(A.status, DEV_HASH_FULL); continue; }
            const u32 old = atomicAdd(&conn[slot], wo);
            if (WIDE && old + wo < old) atomicAdd(&high[slot], 1u);
            if (io && A.cdcnt[k] > 0) atomicAdd(&dconn[slot], 1u);
        }
    }
}

// candidate key: the larger wins. (gain, tie-hash, -id) packed into two u64 words.
struct Cand {
    i64 g;
    u64 tie;  // hash << 32 | ~q
};
__device__ __forceinline__ bool cand_better(const Cand &x, const Cand &y) {
    return x.g > y.g || (x.g == y.g && x.tie > y.tie);
}

__device__ __forceinline__ Cand gain_candidate(const GainArgs &A, u32 u, u32 q, u64 cw, u32 dc, i64 saving,
                                               i64 wtot) {
    Cand c{INT64_MIN, 0};
    const u64 s = A.nsize[u];
    if (A.psize[q] + s - s / A.discount > A.omega) return c;
    if (A.pinb[q] + (u64)(A.nin[u] - dc) > A.delta) return c;
    c.g = saving - (wtot - (i64)cw);
    c.tie = ((u64)mix32(q + A.round + A.seed) << 32) | (u64)(~q);
    return c;
}

__device__ __forceinline__ Cand warp_best(Cand c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Cand d;
        d.g = __shfl_xor_sync(0xFFFFFFFFu, c.g, o);
        d.tie = __shfl_xor_sync(0xFFFFFFFFu, c.tie, o);
        if (cand_better(d, c)) c = d;
    }
    return c;
}

constexpr u32 GN_WARP_W = 128;
constexpr u32 GN_WARPS = 4;
constexpr u32 GN_BLOCK = 256;
constexpr u32 GN_BLOCK_W = 4096;
constexpr u32 GN_WARP_DEG = 256;      // incidences one warp takes; more go to a block
constexpr u32 GN_SMALL_LEVEL = 1024;  // levels with at most this many nodes use blocks only
constexpr u32 KW_WARP_DEG = 1024;     // incidences one group of lanes takes in the k-way gains
constexpr u32 GM_WARP_DEG = 4096;     // incidences one warp takes in the mask gains; more go to a block

// ------------------------------------------------------------------ partition-indexed gains
// For K <= GN_DIRECT_K a hyperedge's census is also kept as two K-bit masks of MW words: the
// partitions present, and those holding destination pins. A node's table is then MW registers
// per lane (lane l owns partitions l, l + 32, ...), so an incidence costs O(MW) per lane whatever
// its lambda, against lambda hash updates in the general path. The node's saving from leaving
// its own partition comes from the census pass (Census::save); candidates, connectivity and the
// inbound count per candidate are the same quantities the general path accumulates.

template <u32 MW>
__device__ __forceinline__ void load_words(const u32 *p, u32 (&w)[MW]) {
    if constexpr (MW == 1) {
        w[0] = *p;
    } else if constexpr (MW == 2) {
        const uint2 v = *(const uint2 *)p;
        w[0] = v.x; w[1] = v.y;
    } else {
#pragma unroll
        for (u32 k = 0; k < MW; k += 4) {
            const uint4 v = *(const uint4 *)(p + k);
            w[k] = v.x; w[k + 1] = v.y; w[k + 2] = v.z; w[k + 3] = v.w;
        }
    }
}
template <u32 MW>
__device__ __forceinline__ void store_words(u32 *p, const u32 (&w)[MW]) {
    if constexpr (MW == 1) {
        *p = w[0];
    } else if constexpr (MW == 2) {
        *(uint2 *)p = make_uint2(w[0], w[1]);
    } else {
#pragma unroll
        for (u32 k = 0; k < MW; k += 4) *(uint4 *)(p + k) = make_uint4(w[k], w[k + 1], w[k + 2], w[k + 3]);
    }
}

template <u32 MW>
struct MaskAcc {
    unsigned long long conn[MW];  // this lane's partitions: summed weights of incidences holding them
    u32 dconn[MW];                // inbound incidences with destination pins in them
    u32 pres[MW];                 // OR of the mask words seen (bit `lane` of word k: partition lane + 32k)
};

// Accumulate node u's incidences first, first + stride, ... in batches of 32 (one warp). Each
// batch stages its masks in the warp's shared slots (sm, sd, sw: 32 entries), which every lane
// then reads as broadcasts.
template <u32 MW>
__device__ __forceinline__ void gain_mask_acc(const GainArgs &A, const u32 *mask,
                                              const u32 *dmask, u32 u, u32 first, u32 stride,
                                              u32 (*sm)[MW], u32 (*sd)[MW], u32 *sw, MaskAcc<MW> &acc, i64 &wtot) {
    const u32 lane = threadIdx.x & 31u;
    const u64 t0 = A.toff[u];
    const u32 deg = (u32)(A.toff[u + 1] - t0), nin_u = A.nin[u];
    for (u32 jb = first; jb < deg; jb += stride) {
        const u32 j = jb + lane;
        const bool has = j < deg;
        const u32 h = has ? A.touch[t0 + j] : 0;
        const u32 wh = has ? A.wfx[h] : 0;
        wtot += wh;
        u32 mw[MW], dw[MW];
#pragma unroll
        for (u32 k = 0; k < MW; ++k) mw[k] = dw[k] = 0;
        if (has) load_words<MW>(mask + (u64)h * MW, mw);
        if (has && j < nin_u) load_words<MW>(dmask + (u64)h * MW, dw);
        store_words<MW>(sm[lane], mw);
        store_words<MW>(sd[lane], dw);
        sw[lane] = wh;
        __syncwarp();
        const u32 chunk = (deg - jb) < 32 ? (deg - jb) : 32;
        for (u32 t = 0; t < chunk; ++t) {
            const u32 wt = sw[t];
            u32 mk[MW], dk[MW];
            load_words<MW>(sm[t], mk);
            load_words<MW>(sd[t], dk);
#pragma unroll
            for (u32 k = 0; k < MW; ++k) {
                if ((mk[k] >> lane) & 1u) acc.conn[k] += wt;
                acc.dconn[k] += (dk[k] >> lane) & 1u;
                acc.pres[k] |= mk[k];
            }
        }
        __syncwarp();
    }
}

template <u32 MW>
__device__ __forceinline__ Cand mask_best(const GainArgs &A, u32 u, u32 p, const MaskAcc<MW> &acc, i64 saving,
                                          i64 wtot) {
    const u32 lane = threadIdx.x & 31u;
    Cand best{INT64_MIN, 0};
#pragma unroll
    for (u32 k = 0; k < MW; ++k) {
        const u32 q = lane + 32 * k;
        if (q < A.K && q != p && ((acc.pres[k] >> lane) & 1u)) {
            const Cand c = gain_candidate(A, u, q, acc.conn[k], acc.dconn[k], saving, wtot);
            if (cand_better(c, best)) best = c;
        }
    }
    return warp_best(best);
}

__device__ __forceinline__ void write_move(const GainArgs &A, u32 u, const Cand &b) {
    if (b.g != INT64_MIN && b.g > 0) {
        A.target[u] = ~(u32)b.tie;
        A.gain[u] = b.g;
    } else {
        A.target[u] = NONE;
        A.gain[u] = 0;
    }
}

// One warp per node.
template <u32 MW>
__global__ void __launch_bounds__(GN_WARPS * 32) k_gain_mask_warp(GainArgs A0, const u32 *__restrict__ list, u32 nl,
                                                                 const u32 *__restrict__ mask,
                                                                 const u32 *__restrict__ dmask) {
    const GainArgs A = gain_args_now(A0);
    __shared__ __align__(16) u32 sm[GN_WARPS][32][MW], sd[GN_WARPS][32][MW];
    __shared__ u32 sw[GN_WARPS][32];
    const u32 w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u32 idx = blockIdx.x * GN_WARPS + w;
    if (idx >= nl) return;
    const u32 u = list[idx], p = A.part[u];
    MaskAcc<MW> acc;
#pragma unroll
    for (u32 k = 0; k < MW; ++k) { acc.conn[k] = 0; acc.dconn[k] = 0; acc.pres[k] = 0; }
    i64 wtot = 0;
    gain_mask_acc<MW>(A, mask, dmask, u, 0, 32, sm[w], sd[w], sw[w], acc, wtot);
    wtot = warp_sum(wtot);
    const Cand best = mask_best<MW>(A, u, p, acc, A.save[u], wtot);
    if (lane == 0) write_move(A, u, best);
}

// One block per node (its warps split the incidences), for heavy nodes and small levels; the
// warps' tables are summed in shared memory.
template <u32 MW>
__global__ void __launch_bounds__(GN_BLOCK) k_gain_mask_block(GainArgs A0, const u32 *__restrict__ list, u32 nl,
                                                             const u32 *__restrict__ mask,
                                                             const u32 *__restrict__ dmask) {
    constexpr u32 NW = GN_BLOCK / 32;
    const GainArgs A = gain_args_now(A0);
    __shared__ __align__(16) u32 sm[NW][32][MW], sd[NW][32][MW];
    __shared__ u32 sw[NW][32];
    __shared__ unsigned long long rc[MW][32];
    __shared__ u32 rd[MW][32], rp[MW];
    __shared__ i64 rw[NW];
    const u32 w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (u32 i = threadIdx.x; i < MW * 32; i += blockDim.x) { rc[i / 32][i % 32] = 0; rd[i / 32][i % 32] = 0; }
    if (threadIdx.x < MW) rp[threadIdx.x] = 0;
    __syncthreads();
    for (u32 idx = blockIdx.x; idx < nl; idx += gridDim.x) {
        const u32 u = list[idx], p = A.part[u];
        MaskAcc<MW> acc;
#pragma unroll
        for (u32 k = 0; k < MW; ++k) { acc.conn[k] = 0; acc.dconn[k] = 0; acc.pres[k] = 0; }
        i64 wtot = 0;
        gain_mask_acc<MW>(A, mask, dmask, u, 32 * w, GN_BLOCK, sm[w], sd[w], sw[w], acc, wtot);
        wtot = warp_sum(wtot);
#pragma unroll
        for (u32 k = 0; k < MW; ++k) {
            if (acc.conn[k]) atomicAdd(&rc[k][lane], acc.conn[k]);
            if (acc.dconn[k]) atomicAdd(&rd[k][lane], acc.dconn[k]);
            if (lane == 0 && acc.pres[k]) atomicOr(&rp[k], acc.pres[k]);
        }
        if (lane == 0) rw[w] = wtot;
        __syncthreads();
        if (w == 0) {
#pragma unroll
            for (u32 k = 0; k < MW; ++k) {
                acc.conn[k] = rc[k][lane];
                acc.dconn[k] = rd[k][lane];
                acc.pres[k] = rp[k];
            }
            wtot = 0;
            for (u32 i = 0; i < NW; ++i) wtot += rw[i];
            const Cand best = mask_best<MW>(A, u, p, acc, A.save[u], wtot);
            if (lane == 0) write_move(A, u, best);
        }
        __syncthreads();  // warp 0 has read the sums: clear them for the next node
        for (u32 i = threadIdx.x; i < MW * 32; i += blockDim.x) { rc[i / 32][i % 32] = 0; rd[i / 32][i % 32] = 0; }
        if (threadIdx.x < MW) rp[threadIdx.x] = 0;
        __syncthreads();
    }
}

// WIDE: some node's incident weights pass 2^32, and a connectivity is a low and a high word (64-bit
// shared adds would be compare-and-swap loops).
// Bound by latency (touch list, census offsets, entries). Measured: 120k-node netlist 57 us, 46.
template <bool WIDE>
__global__ void __launch_bounds__(GN_WARPS * 32) k_gain_warp(GainArgs A0, const u32 *__restrict__ list, u32 nl,
                                                             const u64 *__restrict__ work) {
    const GainArgs A = gain_args_now(A0);
    __shared__ u32 tk[GN_WARPS][2 * GN_WARP_W], td[GN_WARPS][2 * GN_WARP_W], tl[GN_WARPS][2 * GN_WARP_W],
        th[WIDE ? GN_WARPS : 1][WIDE ? 2 * GN_WARP_W : 1];
    const u32 w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u32 idx = blockIdx.x * GN_WARPS + w;
    if (idx >= nl) return;
    const u32 u = list[idx], p = A.part[u];
    u32 *keys = tk[w], *dconn = td[w], *lo = tl[w], *hi = th[WIDE ? w : 0];
    const u32 cap = gain_cap(work[u], 2 * GN_WARP_W);
    for (u32 i = lane; i < cap; i += 32) {
        keys[i] = NONE;
        dconn[i] = 0;
        lo[i] = 0;
        if (WIDE) hi[i] = 0;
    }
    __syncwarp();
    i64 saving = 0, wtot = 0;
    gain_flat<WIDE>(A, u, p, keys, lo, hi, dconn, cap - 1, 0, 32, saving, wtot);
    saving = warp_sum(saving);
    wtot = warp_sum(wtot);
    __syncwarp();
    Cand best{INT64_MIN, 0};
    for (u32 i = lane; i < cap; i += 32) {
        if (keys[i] == NONE) continue;
        const u64 conn = WIDE ? ((u64)hi[i] << 32) | lo[i] : (u64)lo[i];
        if (saving - (wtot - (i64)conn) <= 0) continue;  // no move
        const Cand c = gain_candidate(A, u, keys[i], conn, dconn[i], saving, wtot);
        if (cand_better(c, best)) best = c;
    }
    best = warp_best(best);
    if (lane == 0) write_move(A, u, best);
}

// ------------------------------------------------------------------ sampled gains (K > AXC_SPARSE_GAIN_K)
// With more partitions than AXC_SPARSE_GAIN_K a heavy node's adjacent partitions number in the
// tens of thousands and no per-node table fits on chip. Its gains follow the sampled rule of
// include/axc.h in two kernels:
//  - k_gain_sample (one block per node, the sample table in shared memory) finds the sample
//    prefix, accumulates the sampled connectivity and, when the prefix is the whole node, settles
//    the node exactly; otherwise it writes the node's candidates;
//  - k_cands_warp / k_cands_block (one warp or block per hyperedge holding such a node) put the
//    hyperedge's census in a hash table and add, for each such pin, the hyperedge's weight to its
//    candidates' sums, and k_cands_best picks each node's best feasible candidate. A node's exact
//    pass so costs its incidences times GS_C + 1 lookups, not its whole census.
constexpr u32 GS_K = AXC_SPARSE_GAIN_K;
constexpr u32 GS_SAMPLE = AXC_SPARSE_GAIN_SAMPLE;
constexpr u32 GS_C = AXC_SPARSE_GAIN_CANDIDATES;
constexpr u32 GS_TAB = 2 * GS_SAMPLE;  // hashed sample table: at most half full
constexpr u32 GS_BLOCK = 256;
constexpr u32 GS_LIST = 256;           // keys the final selection of the candidates looks at
constexpr u32 GS_HIST = 32;            // equal weights: slots are counted by incidences from GS_BAND up ...
constexpr u32 GS_BAND = 3;             // (nearly every slot reaches one or two)
constexpr u32 GS_BAND_MIN = 16;        // ... and looked at in bands of at least so many
// A slot of the sample table holds a partition's sampled connectivity and inbound count in 32-bit
// words (64-bit shared adds would be compare-and-swap loops). Equal weights: one word, incidences
// holding the partition above, inbound ones with a destination pin in it below. Else the low word
// of the connectivity, and a word with its carries above, the inbound count below and GS_ZERO set
// by a zero weight, so that a present slot is never all zero.
constexpr u32 GS_HI = 16, GS_LOW = 0xFFFFu, GS_ZERO = 0x80000000u;
static_assert(GS_SAMPLE < GS_LOW / 2, "counts and carries fit their half words");
// The table is indexed by partition where that takes no more room than the hashed one (UNI: one
// word per slot against a key and one), which also makes its scans read psize and pinb in order.
constexpr u32 GS_DIRECT_UNI = 2 * GS_TAB, GS_DIRECT_GEN = GS_TAB + GS_TAB / 2;
// Nodes outside the sampled kernels (gain tiers 0 and 1) have at most GN_BLOCK_W census entries,
// so their sample would be the whole node and the exact kernels give the rule's result.
static_assert(GN_BLOCK_W <= GS_SAMPLE, "tier-1 nodes must fit the sample");

// The census entries [ao, ao + lo) of one hyperedge read by the whole calling warp, CF_UNROLL
// independent loads in flight per lane: f(k, cpart[k], w, inbound) for each entry k.
constexpr u32 CF_UNROLL = 8;
template <class F>
__device__ __forceinline__ void census_edge_warp(const GainArgs &A, u64 ao, u32 lo, u32 w, u32 io, F &&f) {
    const u32 lane = threadIdx.x & 31u;
    for (u32 i0 = 0; i0 < lo; i0 += 32 * CF_UNROLL) {
        u32 x[CF_UNROLL];
#pragma unroll
        for (u32 r = 0; r < CF_UNROLL; ++r) {
            const u32 i = i0 + 32 * r + lane;
            x[r] = i < lo ? A.cpart[ao + i] : NONE;
        }
#pragma unroll
        for (u32 r = 0; r < CF_UNROLL; ++r) {
            const u32 i = i0 + 32 * r + lane;
            if (i < lo) f(ao + i, x[r], w, io);
        }
    }
}

// Census entries of u's incidences j = first, first + stride, ... below jend, flattened across the
// calling warp's lanes in batches of 32 incidences (the scheme of gain_flat): f(k, cpart[k], w,
// inbound) is called for each entry k, and every incidence adds its weight to wtot once (per
// lane). A batch whose entries average CF_LONG or more per incidence is read one hyperedge at a
// time by the whole warp instead (coalesced, no search). The calls are the same set either way.
constexpr u32 CF_LONG = 16;
template <class F>
__device__ __forceinline__ void census_flat(const GainArgs &A, u32 u, u32 first, u32 stride, u32 jend, i64 &wtot,
                                            F &&f) {
    const u32 lane = threadIdx.x & 31u;
    const u64 t0 = A.toff[u];
    const u32 nin_u = A.nin[u];
    for (u32 jb = first; jb < jend; jb += stride) {
        const u32 j = jb + lane;
        const bool has = j < jend;
        const u32 h = has ? A.touch[t0 + j] : 0;
        const u32 lm = has ? A.lam[h] : 0;
        const u32 wh = has ? A.wfx[h] : 0;
        const u64 ah = has ? A.off[h] : 0;
        const u32 ib = (has && j < nin_u) ? 1u : 0u;
        wtot += wh;
        u32 x = lm;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if ((int)lane >= o) x += y;
        }
        const u32 total = __shfl_sync(0xFFFFFFFFu, x, 31), excl = x - lm;
        const u32 chunk = (jend - jb) < 32 ? (jend - jb) : 32;
        if (total >= 32 * CF_LONG) {  // long lists: the warp reads one hyperedge's entries at a time
            for (u32 t = 0; t < chunk; ++t) {
                const u64 ao = __shfl_sync(0xFFFFFFFFu, ah, t);
                const u32 lo = __shfl_sync(0xFFFFFFFFu, lm, t), wo = __shfl_sync(0xFFFFFFFFu, wh, t);
                const u32 io = __shfl_sync(0xFFFFFFFFu, ib, t);
                census_edge_warp(A, ao, lo, wo, io, f);
            }
            continue;
        }
        for (u32 fb = 0; fb < total; fb += 32) {
            const u32 fi = fb + lane;
            u32 lo = 0, hi = chunk - 1;
            for (int it = 0; it < 5; ++it) {
                const u32 mid = (lo + hi + 1) >> 1;
                const u32 em = __shfl_sync(0xFFFFFFFFu, excl, mid & 31);
                if (lo < hi) { if (em <= fi) lo = mid; else hi = mid - 1; }
            }
            const u32 eo = __shfl_sync(0xFFFFFFFFu, excl, lo);
            const u64 ao = __shfl_sync(0xFFFFFFFFu, ah, lo);
            const u32 wo = __shfl_sync(0xFFFFFFFFu, wh, lo);
            const u32 io = __shfl_sync(0xFFFFFFFFu, ib, lo);
            if (fi < total) f(ao + (fi - eo), A.cpart[ao + (fi - eo)], wo, io);
        }
    }
}

// ------------------------------------------------------------------ gains for GN_DIRECT_K < K <= GS_K
// Nodes beyond a warp's hash table take a block and sums indexed by partition. What bounds them is
// the census entries of a node's hyperedges (tens of thousands at a spiking network's
// partitions), so there are two forms, chosen per level by run_gains:
//  - k_gain_table: one shared add per census entry into K-entry tables. The connectivity is one
//    u32 where no node's incident weights pass 2^32, else a low and a high word: 64-bit shared
//    adds would be compare-and-swap loops. NT threads: 64 at moderate degrees, where more nodes in
//    flight hide the loads' latency better than more threads per node, and no node of more than
//    GT_SMALL_DEG incidences, whose walk by two warps would outlast the level's other nodes.
//  - k_gain_planes: for equal weights and hyperedges of at least as many pins as mask words. A
//    candidate's connectivity is then a count of incidences whose K-bit mask holds it. A lane owns
//    one mask word and adds whole words into bit-plane counters (carry-save adders, eight
//    incidences at a time): 32 partitions per instruction, whatever the number of entries.
// Measured: 120k-node netlist 134 us hashed, 64 (64 threads) and 68 (256); with a node of 300,000
// incidences 20.8 ms (64) and 2.8 (256).
constexpr u32 GT_SMALL_DEG = 4096;
template <bool WIDE, u32 NT>
__global__ void __launch_bounds__(NT) k_gain_table(GainArgs A0, const u32 *__restrict__ list, u32 nl) {
    const GainArgs A = gain_args_now(A0);
    extern __shared__ u32 gt_dyn[];
    u32 *lo = gt_dyn, *dconn = lo + A.K, *hi = dconn + A.K;  // hi only when WIDE
    __shared__ i64 red[2][NT / 32];
    __shared__ Cand cred[NT / 32];
    const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (u32 idx = blockIdx.x; idx < nl; idx += gridDim.x) {
        const u32 u = list[idx], p = A.part[u];
        const u32 deg = (u32)(A.toff[u + 1] - A.toff[u]);
        for (u32 i = threadIdx.x; i < (WIDE ? 3 : 2) * A.K; i += NT) gt_dyn[i] = 0;
        __syncthreads();
        i64 saving = 0, wtot = 0;
        census_flat(A, u, 32 * warp, NT, deg, wtot, [&](u64 k, u32 q, u32 w, u32 io) {
            if (q == p) { saving += leave_gain(A.encourage, w, A.ccnt[k]); return; }
            if (io && A.cdcnt[k] > 0) atomicAdd(&dconn[q], 1u);
            if (WIDE) {
                const u32 old = atomicAdd(&lo[q], w);
                if (old + w < old) atomicAdd(&hi[q], 1u);
            } else {
                atomicAdd(&lo[q], w);
            }
        });
        saving = warp_sum(saving);
        wtot = warp_sum(wtot);
        if (lane == 0) { red[0][warp] = saving; red[1][warp] = wtot; }
        __syncthreads();
        saving = wtot = 0;
        for (u32 i = 0; i < NT / 32; ++i) { saving += red[0][i]; wtot += red[1][i]; }
        Cand best{INT64_MIN, 0};
        for (u32 q = threadIdx.x; q < A.K; q += NT) {
            const u64 conn = WIDE ? ((u64)hi[q] << 32) | lo[q] : (u64)lo[q];
            if (saving - (wtot - (i64)conn) <= 0) continue;  // absent, or no move
            const Cand c = gain_candidate(A, u, q, conn, dconn[q], saving, wtot);
            if (cand_better(c, best)) best = c;
        }
        best = warp_best(best);
        if (lane == 0) cred[warp] = best;
        __syncthreads();
        if (threadIdx.x == 0) {
            Cand b = cred[0];
            for (u32 i = 1; i < NT / 32; ++i)
                if (cand_better(cred[i], b)) b = cred[i];
            write_move(A, u, b);
        }
        __syncthreads();
    }
}

constexpr u32 GP_PLANES = 14;   // bits of a lane's counters
constexpr u32 GP_MAX_MW = 128;  // mask words (K <= GS_K)
static_assert(GS_K <= 32 * GP_MAX_MW, "every K of the plane gains has a mask");

// Per-hyperedge masks of MW <= GP_MAX_MW words from the census entries; one warp per hyperedge.
__global__ void __launch_bounds__(128) k_census_masks_wide(u32 e, const u64 *__restrict__ off,
                                                           const u32 *__restrict__ lam, const u32 *__restrict__ cpart,
                                                           const u32 *__restrict__ cdcnt, u32 MW,
                                                           u32 *__restrict__ mask, u32 *__restrict__ dmask) {
    __shared__ u32 sm[4][GP_MAX_MW], sd[4][GP_MAX_MW];
    const u32 w = threadIdx.x >> 5, lane = threadIdx.x & 31, h = blockIdx.x * 4 + w;
    if (h >= e) return;
    for (u32 i = lane; i < MW; i += 32) sm[w][i] = sd[w][i] = 0;
    __syncwarp();
    const u64 a = off[h];
    const u32 lm = lam[h];
    for (u32 j = lane; j < lm; j += 32) {
        const u32 q = cpart[a + j], bit = 1u << (q & 31u);
        atomicOr(&sm[w][q >> 5], bit);
        if (cdcnt[a + j] > 0) atomicOr(&sd[w][q >> 5], bit);
    }
    __syncwarp();
    for (u32 i = lane; i < MW; i += 32) {
        mask[(u64)h * MW + i] = sm[w][i];
        dmask[(u64)h * MW + i] = sd[w][i];
    }
}

// a + b + c of one bit position: sum into l, carry into h.
__device__ __forceinline__ void csa(u32 &h, u32 &l, u32 a, u32 b, u32 c) {
    const u32 x = a ^ b;
    h = (a & b) | (x & c);
    l = x ^ c;
}
// Bit-plane counters of mask word `wl` (of MW, pitch words apart) over the incidences slot, slot + S,
// ... below jend of the node's list t: plane b of bit i counts 2^b incidences whose word has bit i.
template <u32 NP>
__device__ __forceinline__ void plane_count(const u32 *__restrict__ t, u32 jend, const u32 *__restrict__ mask, u32 pitch,
                                            u32 MW, u32 wl, u32 slot, u32 S, u32 (&pl)[NP]) {
#pragma unroll
    for (u32 b = 0; b < NP; ++b) pl[b] = 0;
    for (u32 j = slot; j < jend; j += 8 * S) {
        u32 x[8];
#pragma unroll
        for (u32 r = 0; r < 8; ++r) x[r] = j + r * S < jend ? t[j + r * S] : NONE;
#pragma unroll
        for (u32 r = 0; r < 8; ++r) x[r] = x[r] != NONE && wl < MW ? mask[(u64)x[r] * pitch + wl] : 0u;
        u32 t0, t1, f0, f1, e0;
        csa(t0, pl[0], pl[0], x[0], x[1]);
        csa(t1, pl[0], pl[0], x[2], x[3]);
        csa(f0, pl[1], pl[1], t0, t1);
        csa(t0, pl[0], pl[0], x[4], x[5]);
        csa(t1, pl[0], pl[0], x[6], x[7]);
        csa(f1, pl[1], pl[1], t0, t1);
        csa(e0, pl[2], pl[2], f0, f1);
#pragma unroll
        for (u32 b = 3; b < NP; ++b) {
            const u32 c = pl[b] & e0;
            pl[b] ^= e0;
            e0 = c;
        }
    }
}
// The counters of lanes l and l ^ o added (both get the sum).
template <u32 NP>
__device__ __forceinline__ void plane_merge(u32 (&pl)[NP], u32 o) {
    u32 c = 0;
#pragma unroll
    for (u32 b = 0; b < NP; ++b) {
        const u32 y = __shfl_xor_sync(0xFFFFFFFFu, pl[b], o);
        u32 h;
        csa(h, pl[b], pl[b], y, c);
        c = h;
    }
}

// One block per node; MWP, the power of two from MW up, lanes per incidence. w: the level's weight.
// Bound by issue: about five instructions per mask word. Measured: 20 x 500 network, 10k nodes of
// some 340 incidences at 500 partitions, 3056 us hashed, 107.
template <u32 MWP>
__global__ void __launch_bounds__(GN_BLOCK) k_gain_planes(GainArgs A0, const u32 *__restrict__ list, u32 nl,
                                                         const u32 *__restrict__ mask, const u32 *__restrict__ dmask,
                                                         u32 MW, u32 w) {
    constexpr u32 S = GN_BLOCK / MWP;                // incidences side by side
    constexpr u32 ROWS = MWP < 32 ? GN_BLOCK / 32 : S;  // counters per word once a warp's are merged
    const GainArgs A = gain_args_now(A0);
    __shared__ u32 pc[GP_PLANES][ROWS * MWP], pd[GP_PLANES][ROWS * MWP];
    __shared__ Cand cred[GN_BLOCK / 32];
    const u32 wl = threadIdx.x & (MWP - 1), slot = threadIdx.x / MWP;
    const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (u32 idx = blockIdx.x; idx < nl; idx += gridDim.x) {
        const u32 u = list[idx], p = A.part[u];
        const u64 t0 = A.toff[u];
        const u32 deg = (u32)(A.toff[u + 1] - t0), nin = A.nin[u];
        // planes that can be set: the bits of the most incidences one counter sees
        u32 nb = 32 - __clz((deg + S - 1) / S * (MWP < 32 ? 32 / MWP : 1));
        nb = nb < GP_PLANES ? nb : GP_PLANES;
        const auto count = [&](u32 jend, const u32 *m, u32 (&out)[GP_PLANES][ROWS * MWP]) {
            u32 pl[GP_PLANES];
            plane_count<GP_PLANES>(A.touch + t0, jend, m, MW, MW, wl, slot, S, pl);
            if (MWP < 32)
#pragma unroll
                for (u32 o = 16; o >= MWP; o >>= 1) plane_merge<GP_PLANES>(pl, o);
            const u32 row = MWP < 32 ? warp * MWP + wl : threadIdx.x;
            if (MWP >= 32 || lane < MWP)
#pragma unroll
                for (u32 b = 0; b < GP_PLANES; ++b)
                    if (b < nb) out[b][row] = pl[b];
        };
        const auto total = [&](const u32 (&in)[GP_PLANES][ROWS * MWP], u32 q) {
            const u32 wd = q >> 5, sh = q & 31u;
            u32 cnt = 0;
            for (u32 b = 0; b < nb; ++b) {
                u32 c = 0;
#pragma unroll
                for (u32 r = 0; r < ROWS; ++r) c += (in[b][r * MWP + wd] >> sh) & 1u;
                cnt += c << b;
            }
            return cnt;
        };
        count(deg, mask, pc);
        __syncthreads();
        // A partition whose connectivity does not outweigh what the node pays, or that has no room, is
        // no target whatever its inbound count: the destination planes are counted only where some
        // partition is left (bit k of pos: this thread's k-th), which late rounds rarely have.
        const i64 saving = A.save[u], wtot = (i64)((u64)deg * w);
        const u64 s = A.nsize[u], need = s - s / A.discount;
        u32 pos = 0;
        {
            u32 k = 0;
            for (u32 q = threadIdx.x; q < A.K; q += GN_BLOCK, ++k) {
                const i64 conn = (i64)((u64)total(pc, q) * w);
                if (q != p && saving - (wtot - conn) > 0 && A.psize[q] + need <= A.omega) pos |= 1u << k;
            }
        }
        static_assert(GS_K / GN_BLOCK <= 32, "a thread's partitions fit its mask");
        Cand best{INT64_MIN, 0};
        if (__syncthreads_or(pos)) {
            count(nin, dmask, pd);
            __syncthreads();
            for (u32 k = 0; pos >> k; ++k) {
                if (!((pos >> k) & 1u)) continue;
                const u32 q = threadIdx.x + k * GN_BLOCK;
                const Cand c = gain_candidate(A, u, q, (u64)total(pc, q) * w, total(pd, q), saving, wtot);
                if (cand_better(c, best)) best = c;
            }
        }
        best = warp_best(best);
        if (lane == 0) cred[warp] = best;
        __syncthreads();
        if (threadIdx.x == 0) {
            Cand b = cred[0];
            for (u32 i = 1; i < GN_BLOCK / 32; ++i)
                if (cand_better(cred[i], b)) b = cred[i];
            write_move(A, u, b);
        }
        // the next node's counters are written after every thread has passed this barrier and
        // read the previous ones before it
        __syncthreads();
    }
}

// Block-wide sum of a u64 over GS_BLOCK threads (every thread gets it). `sh` holds one word per warp.
__device__ __forceinline__ u64 block_sum_u64(u64 v, unsigned long long *sh) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    u64 t = 0;
    for (u32 i = 0; i < blockDim.x / 32; ++i) t += sh[i];
    return t;
}

// Sampled-connectivity order of the candidate selection: (sconn desc, hash desc, id asc) as one
// (hi, lo) pair compared as unsigned, the larger first.
struct SKey {
    u64 hi, lo;
};
__device__ __forceinline__ bool skey_better(const SKey &a, const SKey &b) {
    return a.hi > b.hi || (a.hi == b.hi && a.lo > b.lo);
}

// Candidates and sums of the sampled rule's exact pass (k_cands_*), by node. With equal weights a
// sum is one word, the incidences holding the candidate above and the inbound ones with a
// destination pin in it below; else conn is the weight and dcon the inbound count.
struct CandAcc {
    u32 *cand;                 // [n * GS_C], NONE-padded; all NONE for nodes without candidates
    unsigned long long *conn;  // [n * GS_C]
    u32 *dcon;                 // [n * GS_C], null with equal weights
    const u64 *wsum;           // [n] summed weights of a node's hyperedges
    u32 weight;                // with equal weights
};
constexpr unsigned long long CV_ONE = 1ull << 32;

// What a partition can still take, in one word: nodes (omega - size) below, inbound hyperedges
// (delta - inbound) above, each at most RM_MORE; RM_NONE where the limit is already passed. The scans
// of k_gain_sample read it for every partition near a node, at a quarter of the two counts' bytes.
constexpr u32 RM_MORE = 0xFFFEu, RM_NONE = 0xFFFFu;
static_assert(GS_BLOCK == 256, "32 groups of 8 threads");
static_assert(GS_SAMPLE < RM_MORE, "a sample's incidences compare exactly");
__global__ void k_part_room(u32 K, u32 omega, u32 delta, const u64 *__restrict__ psize, const u64 *__restrict__ pinb,
                            u32 *__restrict__ room) {
    const u32 q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= K) return;
    const u64 s = psize[q], b = pinb[q];
    const u32 rs = s > omega ? RM_NONE : (u32)(omega - s < RM_MORE ? omega - s : RM_MORE);
    const u32 rb = b > delta ? RM_NONE : (u32)(delta - b < RM_MORE ? delta - b : RM_MORE);
    room[q] = rs | rb << 16;
}

// UNI: every hyperedge has the weight w. DIRECT: slots are partitions (T = K), else a hash table of
// T = GS_TAB slots. One block per node at a time; the table is empty between nodes: the last scan
// of a node clears it.
// Bound by the shared adds and the block's barriers. Measured: 20 x 5000 network 1422 us (and 315
// for the middling nodes' own kernel), 529 a launch, two launches a round.
template <bool UNI, bool DIRECT>
__global__ void __launch_bounds__(GS_BLOCK, 4) k_gain_sample(GainArgs A0, const u32 *__restrict__ list, u32 nl, CandAcc C,
                                                         u32 T, u32 weight, const u32 *__restrict__ room) {
    const GainArgs A = gain_args_now(A0);
    extern __shared__ __align__(16) u32 gs_tab[];
    u32 *v0 = gs_tab, *v1 = UNI ? nullptr : gs_tab + T, *keys = DIRECT ? nullptr : gs_tab + (UNI ? 1 : 2) * T;
    constexpr u32 NW = GS_BLOCK / 32;
    __shared__ unsigned long long wsh[NW];
    __shared__ unsigned long long s_acc;
    __shared__ Cand cred[NW];
    __shared__ SKey kred[32], kout[GS_C], klist[GS_LIST];
    __shared__ u32 nkeys;
    // the first GS_BLOCK incidences: exclusive census prefix (entry m = the sample's total when m is
    // at most GS_BLOCK), census offset and weight
    __shared__ u32 s_ex[GS_BLOCK + 1], s_w[GS_BLOCK];
    __shared__ u64 s_off[GS_BLOCK];
    __shared__ u32 hist[UNI ? GS_HIST : 1];  // [c]: slots of at least c incidences, c >= GS_BAND
    if (UNI && threadIdx.x < GS_HIST) hist[threadIdx.x] = 0;
    const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (u32 i = threadIdx.x; i < T; i += GS_BLOCK) {
        v0[i] = 0;
        if (!UNI) v1[i] = 0;
        if (!DIRECT) keys[i] = NONE;
    }
    // slot contents (x, y): the words of v0 and v1
    const auto conn_of = [&](u32 x, u32 y) {
        return UNI ? (u64)(x >> GS_HI) * weight : ((u64)((y & ~GS_ZERO) >> GS_HI) << 32) | x;
    };
    const auto dcon_of = [&](u32 x, u32 y) { return (UNI ? x : y) & GS_LOW; };
    const auto part_of = [&](u32 i) { return DIRECT ? i : keys[i]; };
    const auto key_of = [&](u32 q, u64 conn) {
        return SKey{conn, ((u64)mix32(q + A.round + A.seed) << 32) | (u64)(~q)};
    };
    // f(i, x, y) for every present slot, four slots per load (T is a multiple of 4)
    const auto scan = [&](auto &&f) {
        for (u32 i4 = threadIdx.x; i4 < T / 4; i4 += GS_BLOCK) {
            const uint4 x = ((const uint4 *)v0)[i4];
            const uint4 y = UNI ? make_uint4(0, 0, 0, 0) : ((const uint4 *)v1)[i4];
            if (x.x | y.x) f(4 * i4, x.x, y.x);
            if (x.y | y.y) f(4 * i4 + 1, x.y, y.y);
            if (x.z | y.z) f(4 * i4 + 2, x.z, y.z);
            if (x.w | y.w) f(4 * i4 + 3, x.w, y.w);
        }
    };
    const auto clear_all = [&]() {
        if (UNI && threadIdx.x < GS_HIST) hist[threadIdx.x] = 0;
        for (u32 i4 = threadIdx.x; i4 < T / 4; i4 += GS_BLOCK) {
            ((uint4 *)v0)[i4] = make_uint4(0, 0, 0, 0);
            if (!UNI) ((uint4 *)v1)[i4] = make_uint4(0, 0, 0, 0);
            if (!DIRECT) ((uint4 *)keys)[i4] = make_uint4(NONE, NONE, NONE, NONE);
        }
    };
    for (u32 idx = blockIdx.x; idx < nl; idx += gridDim.x) {
        const u32 u = list[idx], p = A.part[u];
        const u64 t0 = A.toff[u];
        const u32 deg = (u32)(A.toff[u + 1] - t0), nin_u = A.nin[u];
        // 1. the sample: the longest incidence prefix with at most GS_SAMPLE census entries. Nodes at
        // this many partitions mostly pass it within 32 incidences, which every warp looks at.
        u32 m = 0;
        u64 acc = 0;
        {
            const u32 h = lane < deg ? A.touch[t0 + lane] : 0;
            const u32 lm = lane < deg ? A.lam[h] : 0;
            const u64 ah = warp == 0 && lane < deg ? A.off[h] : 0;  // in flight with lam
            u64 x = lm;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const u64 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if ((int)lane >= o) x += y;
            }
            m = __popc(__ballot_sync(0xFFFFFFFFu, lane < deg && x <= GS_SAMPLE));
            if (m) acc = __shfl_sync(0xFFFFFFFFu, x, m - 1);
            if (warp == 0 && lane < m) {
                s_off[lane] = ah;
                s_w[lane] = UNI ? weight : A.wfx[h];
                s_ex[lane] = (u32)(x - lm);
                if (lane == m - 1) s_ex[m] = (u32)x;
            }
        }
        if (m == 32 && deg > 32) {  // uniform over the block: the general prefix
            __syncthreads();
            m = 0;
            acc = 0;
            for (u32 base = 0; base < deg; base += GS_BLOCK) {
                const u32 j = base + threadIdx.x;
                const u32 h = j < deg ? A.touch[t0 + j] : 0;
                const u32 lm = j < deg ? A.lam[h] : 0;
                if (base == 0 && j < deg) {
                    s_off[j] = A.off[h];
                    s_w[j] = A.wfx[h];
                }
                u64 x = lm;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const u64 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                    if ((int)lane >= o) x += y;
                }
                if (lane == 31) wsh[warp] = x;
                __syncthreads();
                for (u32 i = 0; i < warp; ++i) x += wsh[i];
                if (base == 0) s_ex[threadIdx.x] = (u32)(x - lm < GS_SAMPLE ? x - lm : GS_SAMPLE);  // exact for j < m
                const bool take = j < deg && acc + x <= GS_SAMPLE;
                const u32 cnt = (u32)__syncthreads_count(take);
                if (cnt > 0 && threadIdx.x == cnt - 1) s_acc = acc + x;
                __syncthreads();
                m += cnt;
                if (cnt > 0) acc = s_acc;
                if (cnt < GS_BLOCK) break;
            }
            if (threadIdx.x == 0 && m <= GS_BLOCK) s_ex[m] = (u32)acc;
        }
        __syncthreads();
        // 2. sampled connectivity; saving and wtot are exact when the sample is the whole node
        i64 saving = 0, wtot = 0;
        const auto put = [&](u64 k, u32 q, u32 w, bool dst) {
            if (q == p) { saving += leave_gain(A.encourage, w, A.ccnt[k]); return; }
            u32 slot = q;
            if (!DIRECT) {
                slot = hash_find_or_insert(keys, T - 1, q);
                if (slot == NONE) { atomicExch(A.status, DEV_HASH_FULL); return; }
            }
            if (UNI) {
                const u32 cnt = (atomicAdd(&v0[slot], (1u << GS_HI) | (dst ? 1u : 0u)) >> GS_HI) + 1;
                if (cnt >= GS_BAND && cnt < GS_HIST) atomicAdd(&hist[cnt], 1u);
            } else {
                const u32 old = atomicAdd(&v0[slot], w);
                const u32 up = (old + w < old ? 1u << GS_HI : 0u) | (dst ? 1u : 0u);
                if (up) atomicAdd(&v1[slot], up);
                if (w == 0) atomicOr(&v1[slot], GS_ZERO);
            }
        };
        if (m <= GS_BLOCK) {
            // the sample's acc entries split evenly over the block: thread t takes entries t,
            // t + GS_BLOCK, ..., finding each one's incidence with a cursor over s_ex
            constexpr u32 U = 8;
            u32 j = 0;
            for (u32 f0 = threadIdx.x; f0 < acc; f0 += U * GS_BLOCK) {
                u32 xx[U], jj[U], dd[U];
#pragma unroll
                for (u32 r = 0; r < U; ++r) {
                    const u32 f = f0 + r * GS_BLOCK;
                    jj[r] = NONE;
                    if (f < acc) {
                        while (s_ex[j + 1] <= f) ++j;  // s_ex[m] = acc > f ends it below m
                        jj[r] = j;
                        const u64 k = s_off[j] + (f - s_ex[j]);
                        xx[r] = A.cpart[k];
                        dd[r] = j < nin_u ? A.cdcnt[k] : 0;
                    }
                }
#pragma unroll
                for (u32 r = 0; r < U; ++r)
                    if (jj[r] != NONE)
                        put(s_off[jj[r]] + (f0 + r * GS_BLOCK - s_ex[jj[r]]), xx[r], UNI ? weight : s_w[jj[r]], dd[r] > 0);
            }
            if (threadIdx.x < m) wtot = s_w[threadIdx.x];
        } else {
            census_flat(A, u, 32 * warp, GS_BLOCK, m, wtot,
                        [&](u64 k, u32 q, u32 w, u32 io) { put(k, q, w, io && q != p && A.cdcnt[k] > 0); });
        }
        if (threadIdx.x == 0) nkeys = 0;
        __syncthreads();
        const u64 s = A.nsize[u];
        if (m == deg) {  // 3a. the whole node: exact, as the table kernels
            saving = (i64)block_sum_u64((u64)saving, wsh);
            wtot = (i64)block_sum_u64((u64)wtot, wsh);
            Cand best{INT64_MIN, 0};
            scan([&](u32 i, u32 x, u32 y) {
                const Cand c = gain_candidate(A, u, part_of(i), conn_of(x, y), dcon_of(x, y), saving, wtot);
                if (cand_better(c, best)) best = c;
            });
            best = warp_best(best);
            if (lane == 0) cred[warp] = best;
            __syncthreads();
            if (threadIdx.x == 0) {
                Cand b = cred[0];
                for (u32 i = 1; i < NW; ++i)
                    if (cand_better(cred[i], b)) b = cred[i];
                write_move(A, u, b);  // its candidates stay NONE
            }
            clear_all();
            __syncthreads();
            continue;
        }
        // 3b. with equal weights the histogram says where the few dozen best connected slots lie: slots are
        // looked at in bands of falling counts until GS_C keys stand that the size limit and the inbound
        // bound do not rule out, so only a band's slots look up their partition's room. A band with more
        // keys than the list holds, and other weights, take the general selection.
        const u64 in_sample = m < nin_u ? m : nin_u, need = s - s / A.discount;
        const auto ruled_out = [&](u32 q, u32 dcon) {
            const u32 rm = room[q], rs = rm & 0xFFFFu, rb = rm >> 16;
            if (rs == RM_NONE || rb == RM_NONE || in_sample - dcon > rb) return true;
            // a clamped room is at least RM_MORE nodes: larger nodes look at the size itself
            return rs == RM_MORE ? (need > RM_MORE && A.psize[q] + need > A.omega) : need > rs;
        };
        u32 nk = GS_LIST + 1;
        if (threadIdx.x < GS_C) kout[threadIdx.x] = SKey{0, 0};
        if (UNI && weight) {
            u32 top = NONE, seen = 0;  // the seen slots of count top and more were looked at
            do {
                u32 c = (top < GS_HIST ? top : GS_HIST) - 1;
                while (c >= GS_BAND && hist[c] < seen + GS_BAND_MIN) --c;
                seen = c >= GS_BAND ? hist[c] : 0;
                const u32 x0 = c << GS_HI, x1 = top < GS_HIST ? (top << GS_HI) - 1 : NONE;
                scan([&](u32 i, u32 x, u32) {
                    if (x < x0 || x > x1) return;
                    const u32 q = part_of(i);
                    if (ruled_out(q, dcon_of(x, 0))) return;
                    const u32 at = atomicAdd(&nkeys, 1u);
                    if (at < GS_LIST) klist[at] = key_of(q, conn_of(x, 0));
                });
                __syncthreads();
                nk = nkeys;
                __syncthreads();  // read before the next band, or the reset below
                top = c;
            } while (nk < GS_C && top > 1);
        }
        // The general selection: the GS_C best by (sampled connectivity, tie hash, -id) among the keys
        // that are not ruled out. Pass 1 empties the ruled-out slots and takes the best key
        // of each group of 8 threads; the GS_C-th of those 32 keys is no better than the GS_C-th of
        // all, so pass 2 lists the keys at or above it (a dozen or so), whose ranks are counted
        // pairwise. (The least of the warps' best keys listed hundreds where a warp's slots, a range
        // of partitions, lie away from the node's.)
        if (nk > GS_LIST) {
            if (threadIdx.x == 0) nkeys = 0;
            SKey best1{0, 0};
            scan([&](u32 i, u32 x, u32 y) {
                const u32 q = part_of(i);
                if (ruled_out(q, dcon_of(x, y))) {  // the slot is emptied (its key may stay: nothing is inserted any more)
                    v0[i] = 0;
                    if (!UNI) v1[i] = 0;
                    return;
                }
                const u64 conn = conn_of(x, y);
                if (conn < best1.hi) return;
                const SKey k = key_of(q, conn);
                if (skey_better(k, best1)) best1 = k;
            });
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {  // 32 groups of 8 threads
                const SKey c{__shfl_xor_sync(0xFFFFFFFFu, best1.hi, o), __shfl_xor_sync(0xFFFFFFFFu, best1.lo, o)};
                if (skey_better(c, best1)) best1 = c;
            }
            if ((lane & 7u) == 0) kred[threadIdx.x / 8] = best1;
            __syncthreads();
            SKey thr{0, 0};
            {
                const SKey mine = kred[lane];
                u32 rank = 0;
                for (u32 j = 0; j < 32; ++j) rank += skey_better(kred[j], mine);
                const u32 bal = __ballot_sync(0xFFFFFFFFu, rank == GS_C - 1 && (mine.hi | mine.lo));
                if (bal) thr = kred[__ffs(bal) - 1];  // keys are unique: one lane
            }
            scan([&](u32 i, u32 x, u32 y) {
                const u64 conn = conn_of(x, y);
                if (conn < thr.hi) return;
                const SKey k = key_of(part_of(i), conn);
                if (skey_better(thr, k)) return;
                const u32 at = atomicAdd(&nkeys, 1u);
                if (at < GS_LIST) klist[at] = k;
            });
            __syncthreads();
            nk = nkeys;
        }
        if (nk <= GS_LIST) {
            if (threadIdx.x < nk) {
                const SKey k = klist[threadIdx.x];
                u32 rank = 0;
                for (u32 j = 0; j < nk && rank < GS_C; ++j) rank += skey_better(klist[j], k);
                if (rank < GS_C) kout[rank] = k;
            }
        } else {  // fewer than GS_C groups hold a key and some hold very many: GS_C block-wide maxima
            SKey prev{~0ull, ~0ull};
            for (u32 r = 0; r < GS_C; ++r) {
                SKey b{0, 0};
                scan([&](u32 i, u32 x, u32 y) {
                    const SKey k = key_of(part_of(i), conn_of(x, y));
                    if (skey_better(prev, k) && skey_better(k, b)) b = k;
                });
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const SKey c{__shfl_xor_sync(0xFFFFFFFFu, b.hi, o), __shfl_xor_sync(0xFFFFFFFFu, b.lo, o)};
                    if (skey_better(c, b)) b = c;
                }
                __syncthreads();
                if (lane == 0) kred[warp] = b;
                __syncthreads();
                b = kred[0];
                for (u32 w2 = 1; w2 < NW; ++w2)
                    if (skey_better(kred[w2], b)) b = kred[w2];
                if (threadIdx.x == 0) kout[r] = b;
                prev = b;
                if (!(b.hi | b.lo)) break;  // no key is left
            }
        }
        __syncthreads();
        clear_all();
        if (threadIdx.x < GS_C) {  // the candidates and their zeroed sums
            const SKey b = kout[threadIdx.x];
            C.cand[(u64)u * GS_C + threadIdx.x] = (b.hi | b.lo) ? ~(u32)b.lo : NONE;
            C.conn[(u64)u * GS_C + threadIdx.x] = 0;
            if (!UNI) C.dcon[(u64)u * GS_C + threadIdx.x] = 0;
            // no candidate: the exact pass will not see the node
            if (threadIdx.x == 0 && !(b.hi | b.lo)) write_move(A, u, Cand{INT64_MIN, 0});
        }
        __syncthreads();
    }
}

// The exact pass of the sampled rule, pin-centric. One pass over the hyperedges fills the sums of
// the listed nodes' candidates: a hyperedge's census goes into shared memory and each pin with
// candidates looks them up. k_cands_best then takes the best feasible candidate from these integer
// sums, which are those a scan of each node's incidences would give; what the node saves by
// leaving comes from the census pass and its total weight from the level. Two forms of the census:
//  - up to CV_BITS_K partitions two bitmaps by partition (present, with a destination pin), so a
//    lookup is one word, and only the words that were set are cleared again;
//  - above, a hash table (partition -> has-destination bit).
static_assert(GS_C == 8, "k_cands_* read a node's candidates as two 16-byte words");
constexpr u32 CV_WARPS = 4;
constexpr u32 CV_WARP_LEN = 256;      // longer hyperedges take a block (CS_WARP_CAP)
constexpr u32 CV_BLOCK_LEN = 4096;    // hashed, longer still: a table in device memory (CS_BLOCK_CAP)
constexpr u32 CV_BLOCK = 256;
constexpr size_t CV_BLOCK_SMEM = (size_t)8 * 8192;  // keys and values of cs_cap(CV_BLOCK_LEN) slots
constexpr u32 CV_BITS_K = 16384;      // two bitmaps of 2 KB

struct CvBits {
    u32 *any, *dst;
    __device__ __forceinline__ bool has(u32 q, bool &d) const {
        const u32 bit = 1u << (q & 31u);
        d = (dst[q >> 5] & bit) != 0;
        return (any[q >> 5] & bit) != 0;
    }
    __device__ __forceinline__ void put(const GainArgs &A, u32 q, bool d) {
        const u32 bit = 1u << (q & 31u);
        atomicOr(&any[q >> 5], bit);
        if (d) atomicOr(&dst[q >> 5], bit);
    }
};
struct CvHash {
    u32 *keys, *vals, mask;
    __device__ __forceinline__ bool has(u32 q, bool &d) const {
        const u32 s = hash_find(keys, mask, q);
        d = s != NONE && vals[s];
        return s != NONE;
    }
    __device__ __forceinline__ void put(const GainArgs &A, u32 q, bool d) {  // each partition once
        const u32 s = hash_find_or_insert(keys, mask, q);
        if (s == NONE) { atomicExch(A.status, DEV_HASH_FULL); return; }
        vals[s] = d;
    }
};
// The sums of pin v's candidates over one hyperedge of weight w; io: v is one of its destinations.
template <class M>
__device__ __forceinline__ void cv_pin(const CandAcc &C, u32 v, bool io, u32 w, const M &map) {
    const uint4 *cp = reinterpret_cast<const uint4 *>(C.cand + (u64)v * GS_C);
    const uint4 c0 = cp[0], c1 = cp[1];
    const u32 q[GS_C] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
    for (u32 i = 0; i < GS_C; ++i) {
        if (q[i] == NONE) break;
        bool d;
        if (!map.has(q[i], d)) continue;
        const u64 at = (u64)v * GS_C + i;
        if (!C.dcon) {
            atomicAdd(&C.conn[at], CV_ONE | (io && d ? 1ull : 0ull));
        } else {
            if (w) atomicAdd(&C.conn[at], (unsigned long long)w);
            if (io && d) atomicAdd(&C.dcon[at], 1u);
        }
    }
}

// One warp per hyperedge of at most CV_WARP_LEN pins; skipped when no pin has candidates. BITS: mw
// words per bitmap.
// Bound by the candidates' 32-byte gathers and the 64-bit atomics. Measured with k_cands_block: 20
// x 5000 network 5060 us with nine hash probes and up to eighteen atomics per pin, 159 + 297.
template <bool BITS>
__global__ void __launch_bounds__(CV_WARPS * 32) k_cands_warp(GainArgs A, CandAcc C, u32 e, u32 mw) {
    extern __shared__ u32 cv_dyn[];
    const u32 wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    u32 *t0 = cv_dyn + wp * (BITS ? 2 * mw : 4 * CV_WARP_LEN);
    if (BITS)
        for (u32 i = lane; i < 2 * mw; i += 32) t0[i] = 0;
    constexpr u32 R = CV_WARP_LEN / 32;
    for (u32 h = blockIdx.x * CV_WARPS + wp; h < e; h += gridDim.x * CV_WARPS) {
        const u64 a = A.off[h], b = A.off[h + 1];
        if (b - a > CV_WARP_LEN) continue;
        u32 pv[R];
        bool any = false;
#pragma unroll
        for (u32 i = 0; i < R; ++i) {
            const u64 k = a + lane + 32 * i;
            pv[i] = k < b ? A.pins[k] : NONE;
        }
#pragma unroll
        for (u32 i = 0; i < R; ++i) {
            if (pv[i] != NONE && C.cand[(u64)pv[i] * GS_C] == NONE) pv[i] = NONE;
            any |= pv[i] != NONE;
        }
        if (!__any_sync(0xFFFFFFFFu, any)) continue;
        const u32 lm = A.lam[h], w = A.wfx[h];
        const u64 s = a + A.nsrc[h];
        const u32 cap = cs_cap(lm);
        if (!BITS)
            for (u32 i = lane; i < cap; i += 32) t0[i] = NONE;
        __syncwarp();
        CvBits bits{t0, t0 + mw};
        CvHash hash{t0, t0 + 2 * CV_WARP_LEN, cap - 1};
        for (u32 j = lane; j < lm; j += 32) {
            if (BITS) bits.put(A, A.cpart[a + j], A.cdcnt[a + j] > 0);
            else hash.put(A, A.cpart[a + j], A.cdcnt[a + j] > 0);
        }
        __syncwarp();
#pragma unroll
        for (u32 i = 0; i < R; ++i)
            if (pv[i] != NONE) {
                if (BITS) cv_pin(C, pv[i], a + lane + 32 * i >= s, w, bits);
                else cv_pin(C, pv[i], a + lane + 32 * i >= s, w, hash);
            }
        __syncwarp();
        if (BITS) {
            for (u32 j = lane; j < lm; j += 32) {
                const u32 x = A.cpart[a + j] >> 5;
                t0[x] = 0;
                t0[mw + x] = 0;
            }
            __syncwarp();
        }
    }
}

// One block per listed hyperedge: BITS, or hashed those of CV_WARP_LEN < |e| <= CV_BLOCK_LEN pins
// (tables in shared memory) or, with gtab set, the longer ones (tables at gtab + 2 * gtab_off[i],
// 2 * |e| slots rounded up to a power of two, as k_tab_sizes sizes them).
template <bool BITS>
__global__ void __launch_bounds__(CV_BLOCK) k_cands_block(GainArgs A, CandAcc C, const u32 *__restrict__ list,
                                                          u32 nlist, u32 mw, u32 *gtab,
                                                          const u64 *__restrict__ gtab_off) {
    extern __shared__ u32 cv_dyn[];
    if (blockIdx.x >= nlist) return;
    const u32 h = list[blockIdx.x];
    const u64 a = A.off[h], b = A.off[h + 1];
    bool any = false;
    for (u64 k = a + threadIdx.x; k < b && !any; k += CV_BLOCK) any = C.cand[(u64)A.pins[k] * GS_C] != NONE;
    if (!__syncthreads_or(any)) return;
    const u32 lm = A.lam[h];
    const u32 cap = BITS ? 0 : cs_cap(lm);
    if (!BITS && !gtab && 8ull * cap > dyn_smem_bytes()) {  // launched with too small a table: refuse
        if (threadIdx.x == 0) atomicExch(A.status, DEV_HASH_FULL);
        return;
    }
    u32 *t0 = !BITS && gtab ? gtab + 2 * gtab_off[blockIdx.x] : cv_dyn;
    const u32 n0 = BITS ? 2 * mw : cap;
    for (u32 i = threadIdx.x; i < n0; i += CV_BLOCK) t0[i] = BITS ? 0u : NONE;
    __syncthreads();
    CvBits bits{t0, t0 + mw};
    CvHash hash{t0, t0 + cap, cap - 1};
    for (u32 j = threadIdx.x; j < lm; j += CV_BLOCK) {
        if (BITS) bits.put(A, A.cpart[a + j], A.cdcnt[a + j] > 0);
        else hash.put(A, A.cpart[a + j], A.cdcnt[a + j] > 0);
    }
    __syncthreads();
    const u32 w = A.wfx[h];
    const u64 s = a + A.nsrc[h];
    for (u64 k = a + threadIdx.x; k < b; k += CV_BLOCK) {
        if (BITS) cv_pin(C, A.pins[k], k >= s, w, bits);
        else cv_pin(C, A.pins[k], k >= s, w, hash);
    }
}

// Each node with candidates: its best feasible one (the order of gain_candidate).
__global__ void k_cands_best(GainArgs A0, CandAcc C, const u32 *__restrict__ list, u32 nl) {
    const GainArgs A = gain_args_now(A0);
    const u32 idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nl) return;
    const u32 u = list[idx];
    if (C.cand[(u64)u * GS_C] == NONE) return;  // settled by k_gain_sample
    const i64 saving = A.save[u], wtot = (i64)C.wsum[u];
    Cand best{INT64_MIN, 0};
#pragma unroll
    for (u32 i = 0; i < GS_C; ++i) {
        const u64 at = (u64)u * GS_C + i;
        const u32 q = C.cand[at];
        if (q == NONE) break;
        const u64 x = C.conn[at];
        const u64 conn = C.dcon ? x : (x >> 32) * C.weight;
        const Cand c = gain_candidate(A, u, q, conn, C.dcon ? C.dcon[at] : (u32)x, saving, wtot);
        if (cand_better(c, best)) best = c;
    }
    write_move(A, u, best);
}

__global__ void k_list_degree(const u32 *__restrict__ list, u32 nl, const u64 *__restrict__ toff,
                              unsigned long long *__restrict__ out) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    u64 d = i < nl ? toff[list[i] + 1] - toff[list[i]] : 0;
    d = warp_sum(d);
    if ((threadIdx.x & 31) == 0 && d) atomicAdd(out, (unsigned long long)d);
}
// Gain tiers: 0 = one warp (small table, at most GN_WARP_DEG incidences), 1 = one block with the
// table in shared memory, 2 = one block with the table in global scratch. Levels of at most
// GN_SMALL_LEVEL nodes use no warp tier: their few nodes carry long census chains, which a block
// splits over its warps while the rest of the GPU would idle anyway.
__device__ __forceinline__ u32 gain_tier(u32 n, u32 K, u64 wk, u64 deg, u32 kway) {
    if (kway) return (n > GN_SMALL_LEVEL && deg <= KW_WARP_DEG) ? 0u : 1u;
    if (K <= GN_DIRECT_K)  // partition-indexed gains: a warp or a block, by incidences
        return (n > GN_SMALL_LEVEL && deg <= GM_WARP_DEG) ? 0u : 1u;
    if (wk > GN_BLOCK_W) return 2u;
    return (n > GN_SMALL_LEVEL && wk <= GN_WARP_W && deg <= GN_WARP_DEG) ? 0u : 1u;
}
// The tiers' node lists, the largest work bound over all nodes (out[0]) and over the block tier
// (out[1]), and the largest degree (out[2]); cnt: three list counts in u64 words.
// Measured: 1M nodes 12 us, in place of a launch and a scan per list.
__global__ void __launch_bounds__(1024) k_tier_lists(u32 n, u32 K, const u64 *__restrict__ work,
                                                     const u64 *__restrict__ toff, u32 kway, u32 *l0, u32 *l1, u32 *l2,
                                                     u64 *__restrict__ cnt, unsigned long long *__restrict__ out) {
    __shared__ u32 sh[33];
    const u32 u = blockIdx.x * blockDim.x + threadIdx.x;
    u64 all = 0, blk = 0, deg = 0;
    u32 t = 3;
    if (u < n) {
        all = work[u];
        deg = toff[u + 1] - toff[u];
        t = gain_tier(n, K, all, deg, kway);
        if (t == 1u) blk = all;
    }
    u32 *lists[3] = {l0, l1, l2};
#pragma unroll
    for (u32 i = 0; i < 3; ++i) {
        if (!__syncthreads_or(t == i)) continue;
        const u32 at = block_append(t == i, (u32 *)(cnt + i), sh);
        if (t == i) lists[i][at] = u;
    }
    all = warp_max_u64(all);
    blk = warp_max_u64(blk);
    deg = warp_max_u64(deg);
    if ((threadIdx.x & 31) == 0) {
        if (all) atomicMax(&out[0], (unsigned long long)all);
        if (blk) atomicMax(&out[1], (unsigned long long)blk);
        if (deg) atomicMax(&out[2], (unsigned long long)deg);
    }
}

// ------------------------------------------------------------------ ranking
// A node's state in the cascade: {rank, place}, rank NONE unless it moves. One 8-byte gather tells a
// hyperedge's pin apart from an earlier mover: the place is the node's partition, and up to
// STATE_PACK_K partitions a mover's target above it, which larger levels gather besides (scattered
// loads and adds were three quarters of the long hyperedges' kernel).
constexpr u32 STATE_PACK_K = 65536;
__device__ __forceinline__ u32 state_place(u32 part, u32 target, int packed) { return packed ? part | target << 16 : part; }
// Mover flags, and every node's state without a rank (k_set_rank then ranks the movers) and
// cascaded gain zeroed.
__global__ void k_move_flags(u32 n, const u32 *__restrict__ target, const u32 *__restrict__ part,
                             u32 *__restrict__ flag, uint2 *__restrict__ state, unsigned long long *__restrict__ g2,
                             int packed) {
    u32 v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) {
        flag[v] = target[v] != NONE ? 1u : 0u;
        state[v] = make_uint2(NONE, state_place(part[v], target[v], packed));
        g2[v] = 0;
    }
}
__global__ void k_move_keys(const u32 *__restrict__ mv, const u32 *__restrict__ dM, const i64 *__restrict__ gain,
                            u64 gbound, u32 *__restrict__ hi, u32 *__restrict__ lo) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *dM) return;
    u64 k = gbound - (u64)gain[mv[i]];  // ascending key = descending gain
    hi[i] = (u32)(k >> 32);
    lo[i] = (u32)k;
}
// The rank of mover mv[i] is i; also the size-event count 2M into *twice.
__global__ void k_set_rank(const u32 *__restrict__ mv, const u32 *__restrict__ dM, uint2 *__restrict__ state,
                           u32 *__restrict__ twice) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *twice = 2 * *dM;
    if (i < *dM) state[mv[i]].x = i;
}

// k-way pair ranking (include/axc.h AXC_PAIR_RANK_MAX_K): the moves, in (gain desc, id asc)
// order, get the key of their direction group: (min(p,q) * K + max(p,q)) * 2 + (p > q).
constexpr u32 PAIR_RANK_MAX_K = AXC_PAIR_RANK_MAX_K;
__global__ void k_pair_group(const u32 *__restrict__ mv, const u32 *__restrict__ dM, const u32 *__restrict__ part,
                             const u32 *__restrict__ target, u32 K, u32 *__restrict__ gk, u32 *__restrict__ pos) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *dM) return;
    const u32 u = mv[i], p = part[u], q = target[u];
    gk[i] = (((p < q ? p : q) * K + (p < q ? q : p)) << 1) | (p < q ? 0u : 1u);
    pos[i] = i;
}
__device__ __forceinline__ u32 lower_bound_u32(const u32 *a, u32 n, u32 x) {
    u32 lo = 0, hi = n;
    while (lo < hi) {
        const u32 mid = (lo + hi) >> 1;
        if (a[mid] < x) lo = mid + 1; else hi = mid;
    }
    return lo;
}
// After the stable sort by group key: the move at position j is the i-th of its group; the i-th of
// the opposite direction is its partner. Pair gain into psn[node] (indexed by node, so later
// passes can rebuild the key after any permutation). The order by (pair position, direction), a
// pair's first direction at its own position and the second one after it, needs no sort: follow[j]
// counts the moves placed at position j (both of a pair at its first direction's, none at its
// second's), and its prefix sums are the places; pk[j] is a paired second direction's pair
// position, else NONE.
__global__ void k_pair_keys(const u32 *__restrict__ gk, const u32 *__restrict__ pos, const u32 *__restrict__ dM, u32 n,
                            const u32 *__restrict__ mv, const i64 *__restrict__ gain, i64 *__restrict__ psn,
                            u32 *__restrict__ pk, u32 *__restrict__ node, u32 *__restrict__ follow) {
    const u32 M = *dM, j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= M) {
        if (j < n) follow[j] = 0;
        return;
    }
    const u32 g = gk[j], d = g & 1u;
    const u32 i = j - lower_bound_u32(gk, M, g);
    const u32 s2 = lower_bound_u32(gk, M, g ^ 1u), e2 = lower_bound_u32(gk, M, (g ^ 1u) + 1u);
    const u32 u = mv[pos[j]];
    i64 ps = gain[u];
    const bool paired = i < e2 - s2;
    if (paired) ps += gain[mv[pos[s2 + i]]];
    psn[u] = ps;
    pk[j] = paired && d ? s2 + i : NONE;
    follow[j] = paired ? (d ? 0u : 2u) : 1u;
    node[j] = u;
}
// Each move at its place, with the low word of its descending pair-gain key (pbound - ps).
__global__ void k_pair_place(const u32 *__restrict__ node, const u32 *__restrict__ dM, const u32 *__restrict__ pk,
                             const u32 *__restrict__ place, const i64 *__restrict__ psn, u64 pbound,
                             u32 *__restrict__ mv, u32 *__restrict__ lo) {
    const u32 j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= *dM) return;
    const u32 u = node[j], at = pk[j] != NONE ? place[pk[j]] + 1 : place[j];
    mv[at] = u;
    lo[at] = (u32)(pbound - (u64)psn[u]);
}
// High words of the permuted movers' descending pair-gain keys.
__global__ void k_pair_gain_high(const u32 *__restrict__ mv, const u32 *__restrict__ dM, const i64 *__restrict__ psn,
                                 u64 pbound, u32 *__restrict__ hi) {
    const u32 j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < *dM) hi[j] = (u32)((pbound - (u64)psn[mv[j]]) >> 32);
}

// ------------------------------------------------------------------ cascade

struct CascadeArgs {
    u32 e;
    int encourage;
    const u64 *off;
    const u32 *pins, *nsrc, *wfx, *lam, *cpart, *ccnt, *cdcnt, *part, *target;
    const uint2 *state;  // [n] {rank, place}
    int packed;          // places hold targets
    unsigned long long *g2;
    // inbound-set transitions (INCC): a (partition, hyperedge) destination count going 0 -> 1 or
    // 1 -> 0 at a move's rank; appended as (partition, rank, +-1)
    int track;
    u32 *tp, *tr;
    int32_t *tdv;
    u32 *dT;
    u64 tcap;
    // when set (small levels), transitions are summed per (partition, rank) instead: entry
    // p * dense_stride + r gets ((d << 32) + 1) per transition, its count below and its net above
    unsigned long long *tdense;
    u32 dense_stride;
    u32 *status;
    u32 K;  // partitions: with K <= CC_DIRECT_BLOCK_K the per-hyperedge tables are indexed by partition id
    // without a census (k-way levels of few partitions per copy): K partitions and ce hyperedges
    // of one copy; the tables hold copy-local partitions, counted from the pins (lam, cpart null)
    u32 ce;
    // movers in slots (k-way copies ranked by one block each): copy t's from slot t * cn, dM[t] of
    // them; 0: ranks [0, *dM)
    u32 cn;
};

constexpr u32 MV_DST = 0x80000000u;  // mover flag in the node field: the pin is a destination
constexpr u32 CC_DIRECT_BLOCK_K = 1024;  // tables indexed by partition up to this many

// The partition of a node and the target of mover v, from its state.
__device__ __forceinline__ u32 state_part(const CascadeArgs &A, const uint2 &s) { return A.packed ? s.y & 0xFFFFu : s.y; }
__device__ __forceinline__ u32 state_target(const CascadeArgs &A, const uint2 &s, u32 v) {
    return A.packed ? s.y >> 16 : A.target[v];
}
__device__ __forceinline__ u32 cascade_base(const CascadeArgs &A, u32 h) { return A.ce ? (h / A.ce) * A.K : 0u; }

// The hyperedge's census into the table: partition -> (pins, destination pins). Block- or
// warp-wide over threads [t0, t0 + nt); direct tables hold K slots, hashed ones `cap`.
__device__ __forceinline__ void cascade_fill(const CascadeArgs &A, u32 h, u64 a, u64 b, u32 lm, u32 *tk, u32 *tc,
                                             u32 *td, u32 cap, bool direct, u32 t0, u32 nt) {
    if (!A.lam) {
        const u32 base = cascade_base(A, h);
        for (u64 k = a + t0; k < b; k += nt) atomicAdd(&tc[state_part(A, A.state[A.pins[k]]) - base], 1u);
        return;
    }
    for (u32 i = t0; i < lm; i += nt) {
        const u32 q = A.cpart[a + i];
        const u32 s = direct ? q : hash_find_or_insert(tk, cap - 1, q);
        if (s != NONE) { tc[s] = A.ccnt[a + i]; td[s] = A.cdcnt[a + i]; }
    }
}

__device__ __forceinline__ void emit_at(const CascadeArgs &A, u32 s, u32 p, u32 r, int32_t d) {
    if (A.tdense) {
        atomicAdd(&A.tdense[(u64)p * A.dense_stride + r], ((unsigned long long)(i64)d << 32) + 1ull);
        return;
    }
    if (s >= A.tcap) { atomicExch(A.status, DEV_BAD_INDEX); return; }
    A.tp[s] = p;
    A.tr[s] = r;
    A.tdv[s] = d;
}
__device__ __forceinline__ void emit_transition(const CascadeArgs &A, u32 p, u32 r, int32_t d) {
    emit_at(A, atomicAdd(A.dT, 1u), p, r, d);
}
// The transitions of one mover (leave: p loses its last destination pin, join: q gains its first),
// with one reservation for the lanes that call it together.
__device__ __forceinline__ void emit_pair(const CascadeArgs &A, bool leave, u32 p, bool join, u32 q, u32 r) {
    const u32 am = __activemask(), lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    const u32 bp = __ballot_sync(am, leave), bq = __ballot_sync(am, join);
    const u32 tot = __popc(bp) + __popc(bq), lead = __ffs(am) - 1;
    if (!tot) return;
    u32 s0 = 0;
    if (!A.tdense && lane == lead) s0 = atomicAdd(A.dT, tot);
    s0 = __shfl_sync(am, s0, lead);
    if (leave) emit_at(A, s0 + __popc(bp & lt), p, r, -1);
    if (join) emit_at(A, s0 + __popc(bp) + __popc(bq & lt), q, r, +1);
}

// Table slots of every mover's source and target partition, sl[i] = slot(p) | slot(q) << 16,
// gathered in parallel so the sequential sweep reads no global memory. Hashed tables insert the
// partitions missing from the census (their counts stay zero); they need cap <= 65536.
__device__ __forceinline__ void cascade_slots(const CascadeArgs &A, u32 h, const u64 *mv, u32 *sl, u32 m, u32 *tk,
                                              u32 cap, bool direct, u32 t0, u32 nt) {
    const u32 base = cascade_base(A, h);
    for (u32 i = t0; i < m; i += nt) {
        const u32 v = (u32)mv[i] & ~MV_DST;
        const u32 p = A.part[v] - base, q = A.target[v] - base;
        u32 sp = p, sq = q;  // direct tables: the slot is the partition id
        if (!direct) {
            sp = hash_find_or_insert(tk, cap - 1, p);
            sq = hash_find_or_insert(tk, cap - 1, q);
            if (sp == NONE || sq == NONE) { atomicExch(A.status, DEV_HASH_FULL); sp = sq = 0; }
        }
        sl[i] = sp | sq << 16;
    }
}

// Sweep the movers of one hyperedge sequentially in rank order. mv[i] = rank << 32 | dst flag |
// node; tc / td hold the hyperedge's pins / destination pins per partition (hash slots in tk,
// or the partition id itself for direct tables). With sl the slots come precomputed from
// cascade_slots; without it (hashed tables too large for 16-bit slots) they are looked up here.
// One thread; cascade_sweep_warp is the warp-wide form used wherever the slots fit 16 bits.
__device__ void cascade_sweep(const CascadeArgs &A, u32 h, const u64 *mv, const u32 *sl, u32 m, u32 *tk, u32 *tc,
                              u32 *td, u32 mask, bool direct) {
    const u32 w = A.wfx[h];
    for (u32 i = 0; i < m; ++i) {
        const u32 lowv = (u32)mv[i], r = (u32)(mv[i] >> 32);
        const u32 v = lowv & ~MV_DST;
        u32 sp, sq;
        if (sl) {
            sp = sl[i] & 0xFFFFu;
            sq = sl[i] >> 16;
        } else {
            sp = A.part[v];
            sq = A.target[v];
            if (!direct) {
                sp = hash_find_or_insert(tk, mask, sp);
                sq = hash_find_or_insert(tk, mask, sq);
                if (sp == NONE || sq == NONE) { atomicExch(A.status, DEV_HASH_FULL); return; }
            }
        }
        const u32 cp = tc[sp], cq = tc[sq];
        const i64 d = leave_gain(A.encourage, w, cp) - (cq == 0 ? (i64)w : 0);
        atomicAdd(&A.g2[v], (unsigned long long)d);
        tc[sp] = cp - 1;
        tc[sq] = tc[sq] + 1;
        if (A.track && (lowv & MV_DST)) {
            if (td[sp] == 1) emit_transition(A, direct ? sp : tk[sp], r, -1);
            if (td[sq] == 0) emit_transition(A, direct ? sq : tk[sq], r, +1);
            td[sp] -= 1;
            td[sq] += 1;
        }
    }
}

// Table size for a hyperedge with lm census partitions and m movers: its keys are the census
// partitions plus at most m targets, at load factor <= 1/2.
__host__ __device__ __forceinline__ u64 cascade_cap(u64 lm, u64 m) {
    u64 cap = 32;
    while (cap < 2 * (lm + m)) cap <<= 1;
    return cap;
}
__device__ __forceinline__ u32 cascade_cap32(u32 lm, u32 m) {
    const u64 cap = cascade_cap(lm, m);
    return cap > (1ull << 31) ? (1u << 31) : (u32)cap;
}

// The same sweep with a whole warp, 32 movers at a time (slots from cascade_slots required). The
// counts a mover sees are the table's counts before its chunk plus what the chunk's earlier lanes
// did to its two partitions: leaves of the same source (match_any), joins of the same target
// (match_any), and the cross terms, lanes whose target is its source or whose source is its
// target (one shuffle pass over the chunk). The tables are then updated by the whole chunk at once.
// Equal to the sequential sweep: the counts are exact prefix sums, and transitions are a set.
__device__ void cascade_sweep_warp(const CascadeArgs &A, u32 h, const u64 *mv, const u32 *sl, u32 m, const u32 *tk,
                                   u32 *tc, u32 *td, u32 *lmask) {
    const u32 lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    const u32 w = A.wfx[h];
    const bool direct = lmask != nullptr;
    for (u32 base = 0; base < m; base += 32) {
        const u32 i = base + lane;
        const bool act = i < m;
        const u64 e = act ? mv[i] : 0;
        // inactive lanes get slots no table has (slots are below 65536), distinct per lane
        const u32 sp = act ? (sl[i] & 0xFFFFu) : 0x10000u + lane, sq = act ? (sl[i] >> 16) : 0x20000u + lane;
        const bool dst = act && ((u32)e & MV_DST);
        const u32 dmask = __ballot_sync(0xFFFFFFFFu, dst);
        u32 m_pp, m_qq, m_qp = 0, m_pq = 0;  // lanes with my source / my target as source / target
        if (lmask) {  // direct tables: lmask[x] / lmask[K + x] = lanes with source / target x
            u32 *pm = lmask, *qm = lmask + A.K;
            if (act) {
                atomicOr(&pm[sp], 1u << lane);
                atomicOr(&qm[sq], 1u << lane);
            }
            __syncwarp();
            m_pp = act ? pm[sp] : 0u;
            m_qq = act ? qm[sq] : 0u;
            m_qp = act ? qm[sp] : 0u;
            m_pq = act ? pm[sq] : 0u;
            __syncwarp();
            if (act) {
                pm[sp] = 0;
                qm[sq] = 0;
            }
        } else {
            m_pp = __match_any_sync(0xFFFFFFFFu, sp);
            m_qq = __match_any_sync(0xFFFFFFFFu, sq);
#pragma unroll 8
            for (u32 j = 0; j < 32; ++j) {
                const u32 spj = __shfl_sync(0xFFFFFFFFu, sp, j), sqj = __shfl_sync(0xFFFFFFFFu, sq, j);
                m_qp |= (u32)(sqj == sp) << j;
                m_pq |= (u32)(spj == sq) << j;
            }
        }
        const int before_p = __popc(m_qp & lt) - __popc(m_pp & lt);
        const int before_q = __popc(m_qq & lt) - __popc(m_pq & lt);
        if (act) {
            const u32 cp = (u32)((int)tc[sp] + before_p), cq = (u32)((int)tc[sq] + before_q);
            const i64 d = leave_gain(A.encourage, w, cp) - (cq == 0 ? (i64)w : 0);
            atomicAdd(&A.g2[(u32)e & ~MV_DST], (unsigned long long)d);
        }
        if (A.track) {  // warp-uniform
            bool ep = false, eq = false;
            if (dst) {
                const int dp = __popc(m_qp & lt & dmask) - __popc(m_pp & lt & dmask);
                const int dq = __popc(m_qq & lt & dmask) - __popc(m_pq & lt & dmask);
                ep = (int)td[sp] + dp == 1;
                eq = (int)td[sq] + dq == 0;
            }
            // one reservation per chunk: p-transitions first, then q-transitions
            const u32 bp = __ballot_sync(0xFFFFFFFFu, ep), bq = __ballot_sync(0xFFFFFFFFu, eq);
            const u32 tot = __popc(bp) + __popc(bq);
            u32 s0 = 0;
            if (lane == 0 && tot) s0 = atomicAdd(A.dT, tot);
            s0 = __shfl_sync(0xFFFFFFFFu, s0, 0);
            const u32 r = (u32)(e >> 32);
            if (ep) emit_at(A, s0 + __popc(bp & lt), direct ? sp : tk[sp], r, -1);
            if (eq) emit_at(A, s0 + __popc(bp) + __popc(bq & lt), direct ? sq : tk[sq], r, +1);
        }
        __syncwarp();
        if (act) {
            atomicSub(&tc[sp], 1u);
            atomicAdd(&tc[sq], 1u);
            if (dst) {
                atomicSub(&td[sp], 1u);
                atomicAdd(&td[sq], 1u);
            }
        }
        __syncwarp();
    }
}

// The cascade over hyperedges of at most CM_LEN pins needs no table and no sort of a hyperedge's
// movers: a pin whose rank is below a mover's counts in its target partition, every other pin in its
// own, which gives the counts the mover finds when all better-ranked moves are applied. Two
// kernels, of which one acts, by the round's mover count (cascade_dense):
//  - few movers, k_cascade_movers: G lanes take one mover, a lane one incidence at a time, and
//    re-read the hyperedge's pins. Its cost follows the movers alone, and a mover's gain is one
//    sum over its lanes.
//  - many movers, k_cascade_dense: a warp stages the pins of consecutive hyperedges in shared
//    memory, each read once, and every mover among them runs over its hyperedge there.
constexpr u32 CM_LEN = 128;
constexpr u32 CM_THREADS = 256;
constexpr u32 CD_STAGE = 512;        // pins a warp of the dense kernel stages at a time
constexpr u32 CD_MAX_K = 32768;      // partitions its staged words hold
static_assert(CD_MAX_K <= STATE_PACK_K, "its nodes' places hold targets");
static_assert(CM_LEN <= CD_STAGE, "every short hyperedge fits the stage");

struct MoverArgs {
    const u32 *mv, *dM;
    const u64 *toff;
    const u32 *touch, *nin;
    int longs;  // the level holds longer hyperedges, whose kernels add to g2 as well
    int dense;  // k_cascade_dense is launched too
    u32 n, copies;     // nodes; counters in dM (one per copy with slots)
    u64 len16;         // 16 times the mean length of the short hyperedge at a short incidence
    u32 per_warp;      // hyperedges a warp of the dense kernel looks at
};

// Whether the dense kernel acts: the movers' incidences hold at least as many pins as the level.
__device__ __forceinline__ bool cascade_dense(const MoverArgs &V) {
    if (!V.dense) return false;
    u64 M = 0;
    for (u32 t = 0; t < V.copies; ++t) M += V.dM[t];
    return M * V.len16 >= 16ull * V.n;
}

// One incidence of the mover of rank r (node u, moving p -> q) in hyperedge h: its part of the
// cascaded gain, and its inbound transitions when u is one of h's destinations.
template <bool TRACK>
__device__ __forceinline__ i64 cascade_incidence(const CascadeArgs &A, u32 h, u32 u, u32 r, u32 p, u32 q, bool dst) {
    const u64 a = A.off[h], len64 = A.off[h + 1] - a;
    if (len64 > CM_LEN) return 0;
    const u32 len = (u32)len64, w = A.wfx[h], ns = TRACK ? A.nsrc[h] : 0u;
    u32 cp = 0, cq = 0, dp = 0, dq = 0;
    constexpr u32 U = 4;  // pins whose loads are in flight together
    for (u32 i0 = 0; i0 < len; i0 += U) {
        u32 v[U];
        uint2 st[U];
#pragma unroll
        for (u32 x = 0; x < U; ++x) v[x] = i0 + x < len ? A.pins[a + i0 + x] : u;
#pragma unroll
        for (u32 x = 0; x < U; ++x) st[x] = A.state[v[x]];
#pragma unroll
        for (u32 x = 0; x < U; ++x)
            if (i0 + x < len) {
                const u32 s = st[x].x < r ? state_target(A, st[x], v[x]) : state_part(A, st[x]);
                cp += s == p;
                cq += s == q;
                if (TRACK && i0 + x >= ns) {
                    dp += s == p;
                    dq += s == q;
                }
            }
    }
    if (TRACK) emit_pair(A, dst && dp == 1, p, dst && dq == 0, q, r);
    return leave_gain(A.encourage, w, cp) - (cq == 0 ? (i64)w : 0);
}

// Movers of at most CM_HEAVY * G incidences (a lane's share stays bounded); the others take a block
// each (k_cascade_movers_heavy).
constexpr u32 CM_HEAVY = 128;
// Bound by latency; its cost follows the movers. Measured with the dense kernel, per round: 200k
// nodes 64 parts 658 us by a sorted sweep per net, 67; 1M nodes 16 parts 656, 93.
template <u32 G, bool TRACK>
__global__ void __launch_bounds__(CM_THREADS) k_cascade_movers(CascadeArgs A, MoverArgs V) {
    const u32 lane = threadIdx.x & 31u, gl = lane & (G - 1);
    const u32 gmask = G == 32 ? 0xFFFFFFFFu : ((1u << G) - 1u) << (lane & ~(G - 1));
    if (cascade_dense(V)) return;
    const u32 ng = gridDim.x * (CM_THREADS / G), end = A.cn ? V.n : *V.dM;
    for (u32 x = blockIdx.x * (CM_THREADS / G) + threadIdx.x / G; x < end; x += ng) {
        const u32 r = A.cn ? x % A.cn : x;
        if (A.cn && r >= V.dM[x / A.cn]) continue;
        const u32 u = V.mv[x];
        const u64 t0 = V.toff[u], deg = V.toff[u + 1] - t0;
        if (deg > CM_HEAVY * G) continue;
        const u32 p = A.part[u], q = A.target[u], nin_u = TRACK ? V.nin[u] : 0u;
        i64 sum = 0;
        for (u32 j = gl; j < (u32)deg; j += G)
            sum += cascade_incidence<TRACK>(A, V.touch[t0 + j], u, r, p, q, TRACK && j < nin_u);
        __syncwarp(gmask);
#pragma unroll
        for (u32 o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(gmask, sum, o);
        if (gl == 0) {
            if (V.longs) atomicAdd(&A.g2[u], (unsigned long long)sum);
            else A.g2[u] = (unsigned long long)sum;
        }
    }
}
template <bool TRACK>
__global__ void __launch_bounds__(CM_THREADS) k_cascade_movers_heavy(CascadeArgs A, MoverArgs V, u32 min_deg) {
    if (cascade_dense(V)) return;
    const u32 end = A.cn ? V.n : *V.dM;
    for (u32 x = blockIdx.x; x < end; x += gridDim.x) {
        const u32 r = A.cn ? x % A.cn : x;
        if (A.cn && r >= V.dM[x / A.cn]) continue;
        const u32 u = V.mv[x];
        const u64 t0 = V.toff[u], deg = V.toff[u + 1] - t0;
        if (deg <= min_deg) continue;
        const u32 p = A.part[u], q = A.target[u], nin_u = TRACK ? V.nin[u] : 0u;
        i64 sum = 0;
        for (u64 j = threadIdx.x; j < deg; j += CM_THREADS)
            sum += cascade_incidence<TRACK>(A, V.touch[t0 + j], u, r, p, q, TRACK && j < nin_u);
        sum = warp_sum(sum);
        if ((threadIdx.x & 31u) == 0 && sum) atomicAdd(&A.g2[u], (unsigned long long)sum);  // g2 starts at zero
    }
}

// A staged pin: its rank, and partition | target << 15 | destination << 31 (target 0 without a
// rank); its node beside it.
// Warp `warp` of `warps`; st and nd hold STAGE staged pins of this warp.
template <bool TRACK, u32 STAGE>
__device__ __forceinline__ void cascade_dense_body(const CascadeArgs &A, const MoverArgs &V, u32 warp, u32 warps, uint2 *st,
                                                   u32 *nd) {
    const u32 lane = threadIdx.x & 31u;
    const u32 step = warps * V.per_warp;
    for (u32 h0 = warp * V.per_warp; h0 < A.e; h0 += step) {
        const u32 h = h0 + lane;
        const bool mine = lane < V.per_warp && h < A.e;
        const u64 a = mine ? A.off[h] : 0, len64 = mine ? A.off[h + 1] - a : 0;
        const u32 len = len64 <= CM_LEN ? (u32)len64 : 0u;  // longer ones are not taken here
        const u32 wh = mine ? A.wfx[h] : 0u, ns = TRACK && mine ? A.nsrc[h] : 0u;
        u32 x = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if ((int)lane >= o) x += y;
        }
        const u32 excl = x - len;
        // as many of the hyperedges as the stage holds at a time
        for (u32 lo = 0; lo < 32;) {
            const u32 b0 = __shfl_sync(0xFFFFFFFFu, excl, lo);
            const u32 hi = lo + __popc(__ballot_sync(0xFFFFFFFFu, lane >= lo && x - b0 <= STAGE));
            const u32 T = __shfl_sync(0xFFFFFFFFu, x, hi - 1) - b0;
            bool movers = false;
            // a pin and its state are a chain of loads: U pins of a lane go through it together
            constexpr u32 U = 4;
            for (u32 f0 = 0; f0 < T; f0 += 32 * U) {
                u32 v[U], dst = 0;
                uint2 s[U];
#pragma unroll
                for (u32 x = 0; x < U; ++x) {
                    v[x] = NONE;
                    if (f0 + 32 * x >= T) continue;  // uniform over the warp
                    const u32 f = f0 + 32 * x + lane;
                    u32 ol = lo, oh = hi - 1;  // owner: the last hyperedge starting at or before f
                    for (int it = 0; it < 5; ++it) {
                        const u32 mid = (ol + oh + 1) >> 1;
                        const u32 em = __shfl_sync(0xFFFFFFFFu, excl, mid & 31);
                        if (ol < oh) { if (em - b0 <= f) ol = mid; else oh = mid - 1; }
                    }
                    const u32 eo = __shfl_sync(0xFFFFFFFFu, excl, ol) - b0;
                    const u64 ao = __shfl_sync(0xFFFFFFFFu, a, ol);
                    const u32 no = TRACK ? __shfl_sync(0xFFFFFFFFu, ns, ol) : 0u;
                    if (f < T) v[x] = A.pins[ao + (f - eo)];
                    if (TRACK && f - eo >= no) dst |= 1u << x;
                }
#pragma unroll
                for (u32 x = 0; x < U; ++x) s[x] = v[x] != NONE ? A.state[v[x]] : make_uint2(NONE, 0);
#pragma unroll
                for (u32 x = 0; x < U; ++x) {
                    if (v[x] == NONE) continue;
                    const u32 f = f0 + 32 * x + lane;
                    movers |= s[x].x != NONE;
                    const u32 q = s[x].x != NONE ? s[x].y >> 16 : 0u;
                    st[f] = make_uint2(s[x].x, (s[x].y & 0xFFFFu) | q << 15 | (TRACK ? (dst >> x) << 31 : 0u));
                    nd[f] = v[x];
                }
            }
            __syncwarp();
            if (__any_sync(0xFFFFFFFFu, movers)) {
                for (u32 f0 = 0; f0 < T; f0 += 32) {
                    const u32 f = f0 + lane;
                    const uint2 me = f < T ? st[f] : make_uint2(NONE, 0);
                    const bool act = me.x != NONE;
                    if (!__any_sync(0xFFFFFFFFu, act)) continue;
                    u32 ol = lo, oh = hi - 1;
                    for (int it = 0; it < 5; ++it) {
                        const u32 mid = (ol + oh + 1) >> 1;
                        const u32 em = __shfl_sync(0xFFFFFFFFu, excl, mid & 31);
                        if (ol < oh) { if (em - b0 <= f) ol = mid; else oh = mid - 1; }
                    }
                    const u32 eo = __shfl_sync(0xFFFFFFFFu, excl, ol) - b0, lno = __shfl_sync(0xFFFFFFFFu, len, ol);
                    const u32 wo = __shfl_sync(0xFFFFFFFFu, wh, ol);
                    const u32 p = me.y & 0x7FFFu, q = (me.y >> 15) & 0x7FFFu;
                    u32 cp = 0, cq = 0, dp = 0, dq = 0;
                    if (act) {
#pragma unroll 4
                        for (u32 j = eo; j < eo + lno; ++j) {
                            const uint2 o = st[j];
                            const u32 s = (o.x < me.x ? o.y >> 15 : o.y) & 0x7FFFu;
                            cp += s == p;
                            cq += s == q;
                            if (TRACK) {
                                dp += s == p && (o.y >> 31);
                                dq += s == q && (o.y >> 31);
                            }
                        }
                        const i64 d = leave_gain(A.encourage, wo, cp) - (cq == 0 ? (i64)wo : 0);
                        if (d) atomicAdd(&A.g2[nd[f]], (unsigned long long)d);
                    }
                    if (TRACK) {
                        __syncwarp();
                        const bool dst = act && (me.y >> 31);
                        emit_pair(A, dst && dp == 1, p, dst && dq == 0, q, me.x);
                    }
                }
            }
            __syncwarp();  // the stage is no longer read
            lo = hi;
        }
    }
}

// Bound by issue on nets of a few pins (about 170 instructions per 32 pins, then ten per pin and
// mover). Measured: 20 x 5000 network 75 us (137 with up to 32 hyperedges a warp).
template <bool TRACK>
__global__ void __launch_bounds__(CM_THREADS) k_cascade_dense(CascadeArgs A, MoverArgs V) {
    constexpr u32 NW = CM_THREADS / 32;
    __shared__ uint2 ss[NW][CD_STAGE];
    __shared__ u32 sn[NW][CD_STAGE];
    if (!cascade_dense(V)) return;
    const u32 w = threadIdx.x >> 5;
    cascade_dense_body<TRACK, CD_STAGE>(A, V, blockIdx.x * NW + w, gridDim.x * NW, ss[w], sn[w]);
}

// The hyperedges of more than CM_LEN pins that hold a mover. Few movers: every such incidence of
// every mover flags its hyperedge (mark[]: 0, or 2 where the hyperedge is short and not to be
// flagged, restored before), and the level's long hyperedges that are flagged form the cascade's
// list. Many movers (cascade_dense): all of them do. One warp per mover.
__global__ void k_mover_hedges(CascadeArgs A, MoverArgs V, uint8_t *__restrict__ mark) {
    if (cascade_dense(V)) return;
    const u32 lane = threadIdx.x & 31u, nw = (gridDim.x * blockDim.x) >> 5;
    const u32 end = A.cn ? V.n : *V.dM;
    for (u32 x = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; x < end; x += nw) {
        if (A.cn && x % A.cn >= V.dM[x / A.cn]) continue;
        const u32 u = V.mv[x];
        const u64 t1 = V.toff[u + 1];
        for (u64 j = V.toff[u] + lane; j < t1; j += 32) {
            const u32 h = V.touch[j];
            if (!mark[h]) mark[h] = 1;
        }
    }
}
// Measured: 100k hyperedges 4 us; with k_mover_hedges 190 before, when every incidence's flag was
// stored.
__global__ void k_long_list(MoverArgs V, const u32 *__restrict__ longs, u32 nlong, const uint8_t *__restrict__ mark,
                            u32 *__restrict__ list, u32 *__restrict__ nlist) {
    const bool all = cascade_dense(V);
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    const u32 h = i < nlong ? longs[i] : 0;
    const bool f = i < nlong && (all || mark[h] == 1);
    const u32 bal = __ballot_sync(0xFFFFFFFFu, f);
    u32 at = 0;
    if (lane == 0 && bal) at = atomicAdd(nlist, (u32)__popc(bal));
    at = __shfl_sync(0xFFFFFFFFu, at, 0);
    if (f) list[at + __popc(bal & ((1u << lane) - 1u))] = h;
}
// Long hyperedges with at most MV movers, one warp each: the gather, the order by rank and the sweep
// are chains of dependent loads, so what counts is the hyperedges in flight, and a warp needs no
// block barrier between its phases. Everything a mover needs is loaded in the gather.
//  - DIRECT (partitions of one copy up to CC_DIRECT_BLOCK_K): a counter word per partition (pins
//    below, destination pins above), counted from the pins themselves;
//  - hashed: only the movers' sources and targets are keys (at most 2 MV of them, 4 MV slots), and the
//    hyperedge's census entries fill in the counts of those.
// Hyperedges with more movers, or too many pins for 16-bit counts, go on to the block kernel.
constexpr u32 CL_WARPS = 4;
constexpr u32 CL_BINS = 256;
constexpr u32 CL_MAX_LEN = 65535;
// Movers a warp takes. Hashed, a mover's slots are most of the warp's shared memory, and the warps in
// flight count for more than the hyperedges that go on to the wide kernel (20 x 5000 network: 456 ms
// with 256, 424 with 128, 413 with 64); by index 512 (128 parts: 156 ms, with 256 165).
constexpr u32 CL_MOV_DIRECT = 512, CL_MOV_HASH = 64;
// Bytes of one warp's shared memory.
__host__ __device__ __forceinline__ u32 cl_bytes(bool direct, u32 K, u32 MV) {
    const u32 common = MV * 8 + MV * 4 + 2 * MV * 2 + CL_BINS * 4 + 16;
    return (common + (direct ? 3 * K * 4 : MV * 4 + 4 * MV * 8) + 15) & ~15u;
}

// Places of the m movers by rank (the high word of mv): ord[i] is the index of the i-th. Ranks spread
// over CL_BINS bins by their leading bits; a mover's place in its bin is the number of smaller ranks.
__device__ __forceinline__ void warp_rank_order(const u64 *mv, u32 m, u32 rmax, u32 *bins, unsigned short *idx,
                                                unsigned short *ord) {
    const u32 lane = threadIdx.x & 31u;
    const u32 nb = 32 - __clz(rmax), sh = nb > 8 ? nb - 8 : 0;
    static_assert(CL_BINS == 256, "eight leading bits");
    for (u32 i = lane; i < CL_BINS; i += 32) bins[i] = 0;
    __syncwarp();
    // arrival places are kept in ord until the movers are listed by bin in idx
    for (u32 i = lane; i < m; i += 32) ord[i] = (unsigned short)atomicAdd(&bins[(u32)(mv[i] >> 32) >> sh], 1u);
    __syncwarp();
    u32 c[8], s = 0;
#pragma unroll
    for (u32 k = 0; k < 8; ++k) { c[k] = bins[lane * 8 + k]; s += c[k]; }
    u32 x = s;
#pragma unroll
    for (u32 o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    u32 pre = x - s;
#pragma unroll
    for (u32 k = 0; k < 8; ++k) { bins[lane * 8 + k] = pre; pre += c[k]; }
    if (lane == 31) bins[CL_BINS] = m;
    __syncwarp();
    for (u32 i = lane; i < m; i += 32) idx[bins[(u32)(mv[i] >> 32) >> sh] + ord[i]] = (unsigned short)i;
    __syncwarp();
    for (u32 i0 = 0; i0 < m; i0 += 32) {
        const u32 i = i0 + lane;
        u32 p = 0;
        if (i < m) {
            const u64 key = mv[i];
            const u32 b = (u32)(key >> 32) >> sh, lo = bins[b], hi = bins[b + 1];
            p = lo;
            for (u32 j = lo; j < hi; ++j) p += mv[idx[j]] < key;
        }
        __syncwarp();
        if (i < m) ord[p] = (unsigned short)i;  // arrival places are no longer read
    }
    __syncwarp();
}

// The sweep of one warp over its hyperedge's movers [i0, i1) in rank order, 32 at a time
// (cascade_sweep_warp). cnt: pins below, destination pins above, as the first of them finds them.
template <bool DIRECT>
__device__ __forceinline__ void cl_sweep(const CascadeArgs &A, const u64 *mv, const u32 *sl, const unsigned short *ord,
                                         u32 i0, u32 i1, u32 *cnt, u32 *pm, u32 *qm, const u32 *keys, u32 wh, u32 base) {
    const u32 lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    for (u32 b0 = i0; b0 < i1; b0 += 32) {
        const bool act = b0 + lane < i1;
        const u32 i = act ? ord[b0 + lane] : 0;
        const u64 e = act ? mv[i] : 0;
        const u32 pq = sl[i];
        const u32 sp = act ? pq & 0xFFFFu : 0x10000u + lane, sqx = act ? pq >> 16 : 0x20000u + lane;
        const bool dst = act && ((u32)e & MV_DST);
        const u32 dmask = __ballot_sync(0xFFFFFFFFu, dst);
        u32 m_pp, m_qq, m_qp = 0, m_pq = 0;  // lanes with my source / my target as source / target
        if (DIRECT) {
            if (act) {
                atomicOr(&pm[sp], 1u << lane);
                atomicOr(&qm[sqx], 1u << lane);
            }
            __syncwarp();
            m_pp = act ? pm[sp] : 0u;
            m_qq = act ? qm[sqx] : 0u;
            m_qp = act ? qm[sp] : 0u;
            m_pq = act ? pm[sqx] : 0u;
            __syncwarp();
            if (act) {
                pm[sp] = 0;
                qm[sqx] = 0;
            }
        } else {
            m_pp = __match_any_sync(0xFFFFFFFFu, sp);
            m_qq = __match_any_sync(0xFFFFFFFFu, sqx);
#pragma unroll 8
            for (u32 j = 0; j < 32; ++j) {
                const u32 spj = __shfl_sync(0xFFFFFFFFu, sp, j), sqj = __shfl_sync(0xFFFFFFFFu, sqx, j);
                m_qp |= (u32)(sqj == sp) << j;
                m_pq |= (u32)(spj == sqx) << j;
            }
        }
        const u32 cP = act ? cnt[sp] : 0, cQ = act ? cnt[sqx] : 0;
        if (act) {
            const u32 cp = (u32)((int)(cP & 0xFFFFu) + __popc(m_qp & lt) - __popc(m_pp & lt));
            const u32 cq = (u32)((int)(cQ & 0xFFFFu) + __popc(m_qq & lt) - __popc(m_pq & lt));
            const i64 d = leave_gain(A.encourage, wh, cp) - (cq == 0 ? (i64)wh : 0);
            if (d) atomicAdd(&A.g2[(u32)e & ~MV_DST], (unsigned long long)d);
        }
        if (A.track) {  // warp-uniform
            bool ep = false, eq = false;
            if (dst) {
                ep = (int)(cP >> 16) + __popc(m_qp & lt & dmask) - __popc(m_pp & lt & dmask) == 1;
                eq = (int)(cQ >> 16) + __popc(m_qq & lt & dmask) - __popc(m_pq & lt & dmask) == 0;
            }
            const u32 r = (u32)(e >> 32);
            const u32 pid = DIRECT ? sp + base : ep ? keys[sp] : 0, qid = DIRECT ? sqx + base : eq ? keys[sqx] : 0;
            __syncwarp();
            emit_pair(A, ep, pid, eq, qid, r);
        }
        __syncwarp();
        if (act) {  // counts stay within their halves once the whole chunk is in
            const u32 one = dst ? 0x10001u : 1u;
            atomicSub(&cnt[sp], one);
            atomicAdd(&cnt[sqx], one);
        }
        __syncwarp();
    }
}

// Bound by scattered loads and adds (L1 at 82% of its peak). Measured per round, short hyperedges
// included: 20 x 5000 network, 128 parts 353 us in a warp and 1710 in a block kernel, now 500, 248
// in the wide and 120 in the dense one; 20 x 500 595, now 105, 56 and 64.
template <bool DIRECT>
__global__ void __launch_bounds__(CL_WARPS * 32) k_cascade_long(CascadeArgs A, const u32 *__restrict__ list,
                                                               const u32 *__restrict__ nlist, u32 MV, u32 per,
                                                               u32 *__restrict__ big, u32 *__restrict__ nbig) {
    extern __shared__ __align__(16) unsigned char cl_smem[];
    const u32 w = threadIdx.x >> 5, lane = threadIdx.x & 31u, lt = (1u << lane) - 1u, nl = *nlist;
    u64 *mv = (u64 *)(cl_smem + w * per);
    u32 *sl = (u32 *)(mv + MV);
    unsigned short *idx = (unsigned short *)(sl + MV), *ord = idx + MV;
    u32 *bins = (u32 *)(ord + MV), *rest = bins + CL_BINS + 4;
    u32 *tc = rest, *pm = tc + A.K, *qm = pm + A.K;                     // DIRECT
    u32 *sq = rest, *keys = sq + MV, *hc = keys + 4 * MV;               // hashed
    if (DIRECT)
        for (u32 i = lane; i < 2 * A.K; i += 32) pm[i] = 0;
    for (u32 li = blockIdx.x * CL_WARPS + w; li < nl; li += gridDim.x * CL_WARPS) {
        __syncwarp();  // the previous hyperedge's shared state is no longer read
        const u32 h = list[li];
        const u64 a = A.off[h], len64 = A.off[h + 1] - a;
        const u32 len = len64 <= CL_MAX_LEN ? (u32)len64 : 0u, ns = A.nsrc[h], base = cascade_base(A, h);
        if (DIRECT)
            for (u32 i = lane; i < A.K; i += 32) tc[i] = 0;
        __syncwarp();
        u32 m = 0, rmax = 0;
        constexpr u32 U = 4;
        for (u32 k0 = 0; k0 < len; k0 += 32 * U) {
            u32 v[U], q[U];
            uint2 st[U];
#pragma unroll
            for (u32 x = 0; x < U; ++x) v[x] = k0 + 32 * x + lane < len ? A.pins[a + k0 + 32 * x + lane] : NONE;
#pragma unroll
            for (u32 x = 0; x < U; ++x) st[x] = v[x] != NONE ? A.state[v[x]] : make_uint2(NONE, 0);
#pragma unroll
            for (u32 x = 0; x < U; ++x) {
                q[x] = st[x].x != NONE ? state_target(A, st[x], v[x]) : 0;
                st[x].y = state_part(A, st[x]);
            }
#pragma unroll
            for (u32 x = 0; x < U; ++x) {
                const bool in = v[x] != NONE, dst = in && k0 + 32 * x + lane >= ns, mover = st[x].x != NONE;
                if (DIRECT && in) atomicAdd(&tc[st[x].y - base], dst ? 0x10001u : 1u);
                const u32 bal = __ballot_sync(0xFFFFFFFFu, mover);
                const u32 at = m + __popc(bal & lt);
                if (mover && at < MV) {
                    mv[at] = ((u64)st[x].x << 32) | (dst ? MV_DST : 0u) | v[x];
                    if (DIRECT) {
                        sl[at] = (st[x].y - base) | (q[x] - base) << 16;
                    } else {
                        sl[at] = st[x].y;
                        sq[at] = q[x];
                    }
                    rmax = st[x].x > rmax ? st[x].x : rmax;
                }
                m += __popc(bal);
            }
        }
        if (m > MV || len64 > CL_MAX_LEN) {
            if (lane == 0) big[atomicAdd(nbig, 1u)] = h;
            continue;
        }
        if (m == 0) continue;
        rmax = __reduce_max_sync(0xFFFFFFFFu, rmax);
        u32 cap = 32;
        if (!DIRECT) {
            while (cap < 4 * m) cap <<= 1;  // at most 4 * MV
            for (u32 i = lane; i < cap; i += 32) { keys[i] = NONE; hc[i] = 0; }
        }
        __syncwarp();
        if (!DIRECT) {
            for (u32 i = lane; i < m; i += 32) {
                const u32 sp = hash_find_or_insert(keys, cap - 1, sl[i]), st = hash_find_or_insert(keys, cap - 1, sq[i]);
                if (sp == NONE || st == NONE) atomicExch(A.status, DEV_HASH_FULL);
                sl[i] = (sp & 0xFFFFu) | st << 16;
            }
            __syncwarp();
            const u32 lm = A.lam[h];
            for (u32 j = lane; j < lm; j += 32) {  // each partition once
                const u32 s = hash_find(keys, cap - 1, A.cpart[a + j]);
                if (s != NONE) hc[s] = A.ccnt[a + j] | A.cdcnt[a + j] << 16;
            }
        }
        warp_rank_order(mv, m, rmax, bins, idx, ord);
        u32 *cnt = DIRECT ? tc : hc;
        cl_sweep<DIRECT>(A, mv, sl, ord, 0, m, cnt, pm, qm, keys, A.wfx[h], base);
    }
}

// Hyperedges with more movers than a warp takes, a block each; everything a mover needs is loaded in one
// gather. The counts a mover finds come in one of two ways:
//  - CW_SWEEP, up to CW_SWEEP_K partitions by index: the movers are ordered by rank, and each warp sweeps
//    over its share of them with a table of its own, which holds the counts its first mover finds
//    (the hyperedge's, plus what the earlier shares did). The block kernel has one warp sweep over all.
//  - CW_EVENTS by index and CW_HASH, more partitions: the movers' leave and join events are dealt out by
//    partition, and a mover counts those of smaller rank in its source and its target: no order and no
//    chain at all. With m movers over K partitions a list holds about 2m / K events; a hyperedge whose
//    lists hold more than CW_PAIRS events per mover goes on to the block kernel.
// So do those with more movers than MV or too many pins for 16-bit counts.
enum WideForm { CW_SWEEP, CW_EVENTS, CW_HASH };
constexpr u32 CW_SWEEP_K = 256;
constexpr u32 CW_PAIRS = 256;
constexpr u32 CW_BINS = 1024;
__host__ __device__ constexpr u32 cw_threads(WideForm f) { return f == CW_SWEEP ? 256u : 512u; }
constexpr u32 cw_movers(WideForm f) { return f == CW_SWEEP ? 2048u : f == CW_EVENTS ? 4096u : 1024u; }
// Words of the events, or of the sweep's order (two shorts per mover, then the bins).
__host__ __device__ constexpr u32 cw_event_words(WideForm f, u32 MV) {
    return f == CW_SWEEP ? MV + CW_BINS + 1 : 2 * MV;
}
__host__ __device__ constexpr u32 cw_bytes(WideForm f, u32 K, u32 MV) {
    return (MV * 12 + cw_event_words(f, MV) * 4 +
            (f == CW_SWEEP ? (1 + 3 * (cw_threads(f) / 32)) * K : f == CW_EVENTS ? 2 * K : 12 * MV) * 4 + 15) & ~15u;
}
// Counts c[0, S) into exclusive prefix sums; returns the sum of the counts' squares.
template <u32 NT>
__device__ __forceinline__ u32 cw_starts(u32 *c, u32 S, u32 *wsum) {
    constexpr u32 NW = NT / 32;
    const u32 lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    u32 carry = 0, sq = 0;
    for (u32 base = 0; base < S; base += NT) {
        const u32 i = base + threadIdx.x, v = i < S ? c[i] : 0;
        sq += v * v;
        u32 x = v;
#pragma unroll
        for (u32 o = 1; o < 32; o <<= 1) {
            const u32 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        u32 tot = 0;
        for (u32 k = 0; k < NW; ++k) {
            if (k == w) x += tot;
            tot += wsum[k];
        }
        __syncthreads();
        if (i < S) c[i] = carry + x - v;
        carry += tot;
    }
    sq = __reduce_add_sync(0xFFFFFFFFu, sq);
    if (lane == 0) wsum[w] = sq;
    __syncthreads();
    sq = 0;
    for (u32 k = 0; k < NW; ++k) sq += wsum[k];
    return sq;
}

// Places of the m movers by rank, block-wide (warp_rank_order).
template <u32 NT>
__device__ __forceinline__ void cw_rank_order(const u64 *mv, u32 m, u32 rmax, u32 *bins, unsigned short *idx,
                                              unsigned short *ord, u32 *wsum) {
    const u32 t = threadIdx.x, nb = 32 - __clz(rmax), sh = nb > 10 ? nb - 10 : 0;
    static_assert(CW_BINS == 1024, "ten leading bits");
    for (u32 i = t; i <= CW_BINS; i += NT) bins[i] = 0;
    __syncthreads();
    // arrival places are kept in ord until the movers are listed by bin in idx
    for (u32 i = t; i < m; i += NT) ord[i] = (unsigned short)atomicAdd(&bins[(u32)(mv[i] >> 32) >> sh], 1u);
    __syncthreads();
    cw_starts<NT>(bins, CW_BINS + 1, wsum);
    __syncthreads();
    for (u32 i = t; i < m; i += NT) idx[bins[(u32)(mv[i] >> 32) >> sh] + ord[i]] = (unsigned short)i;
    __syncthreads();
    for (u32 i = t; i < m; i += NT) {
        const u64 key = mv[i];
        const u32 b = (u32)(key >> 32) >> sh, lo = bins[b], hi = bins[b + 1];
        u32 p = lo;
        for (u32 j = lo; j < hi; ++j) p += mv[idx[j]] < key;
        ord[p] = (unsigned short)i;  // arrival places are no longer read
    }
    __syncthreads();
}

// Measured: 20 x 5000 network, 128 parts, 248 us where the block kernel took 693; 20 x 500 (500
// partitions) 56 a round by events, 155 by the block and scratch kernels.
template <WideForm FORM>
__global__ void __launch_bounds__(cw_threads(FORM)) k_cascade_wide(CascadeArgs A, const u32 *__restrict__ list,
                                                            const u32 *__restrict__ nlist, u32 MV,
                                                            u32 *__restrict__ big, u32 *__restrict__ nbig) {
    extern __shared__ __align__(16) unsigned char cw_smem[];
    constexpr bool DIRECT = FORM != CW_HASH;
    constexpr u32 NT = cw_threads(FORM), NW = NT / 32;
    __shared__ u32 wsum[NW], cm, smax;
    const u32 t = threadIdx.x, lane = t & 31u, lt = (1u << lane) - 1u, nl = *nlist;
    u64 *mv = (u64 *)cw_smem;
    u32 *sl = (u32 *)(mv + MV), *ev = sl + MV, *tc = ev + cw_event_words(FORM, MV);
    u32 *ec = tc + (DIRECT ? A.K : 4 * MV);  // events per partition; the sweep: tables per warp
    u32 *keys = ec + 4 * MV, *sq = ev;  // hashed
    for (u32 li = blockIdx.x; li < nl; li += gridDim.x) {
        __syncthreads();  // the previous hyperedge's shared state is no longer read
        const u32 h = list[li];
        const u64 a = A.off[h], len64 = A.off[h + 1] - a;
        const u32 len = len64 <= CL_MAX_LEN ? (u32)len64 : 0u, ns = A.nsrc[h], base = cascade_base(A, h);
        if (DIRECT)
            for (u32 i = t; i < (FORM == CW_SWEEP ? 1 + 3 * NW : 2) * A.K; i += NT) tc[i] = 0;  // and ec
        if (t == 0) cm = smax = 0;
        __syncthreads();
        u32 rmax = 0;
        constexpr u32 U = 4;
        for (u32 k0 = 0; k0 < len; k0 += NT * U) {
            u32 v[U], q[U];
            uint2 st[U];
#pragma unroll
            for (u32 x = 0; x < U; ++x) v[x] = k0 + NT * x + t < len ? A.pins[a + k0 + NT * x + t] : NONE;
#pragma unroll
            for (u32 x = 0; x < U; ++x) st[x] = v[x] != NONE ? A.state[v[x]] : make_uint2(NONE, 0);
#pragma unroll
            for (u32 x = 0; x < U; ++x) {
                q[x] = st[x].x != NONE ? state_target(A, st[x], v[x]) : 0;
                st[x].y = state_part(A, st[x]);
            }
#pragma unroll
            for (u32 x = 0; x < U; ++x) {
                const bool in = v[x] != NONE, dst = in && k0 + NT * x + t >= ns, mover = st[x].x != NONE;
                if (DIRECT && in) atomicAdd(&tc[st[x].y - base], dst ? 0x10001u : 1u);
                const u32 bal = __ballot_sync(0xFFFFFFFFu, mover);
                u32 at = 0;
                if (lane == 0 && bal) at = atomicAdd(&cm, (u32)__popc(bal));
                at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(bal & lt);
                if (mover && at < MV) {
                    mv[at] = ((u64)st[x].x << 32) | (dst ? MV_DST : 0u) | v[x];
                    if (DIRECT) {
                        const u32 p = st[x].y - base, to = q[x] - base;
                        sl[at] = p | to << 16;
                        if (FORM == CW_EVENTS) {
                            atomicAdd(&ec[p], 1u);
                            atomicAdd(&ec[to], 1u);
                        }
                        rmax = st[x].x > rmax ? st[x].x : rmax;
                    } else {
                        sl[at] = st[x].y;
                        sq[at] = q[x];
                    }
                }
            }
        }
        if (FORM == CW_SWEEP) {
            rmax = __reduce_max_sync(0xFFFFFFFFu, rmax);
            if (lane == 0) atomicMax(&smax, rmax);
        }
        __syncthreads();
        const u32 m = cm;
        if (m > MV || len64 > CL_MAX_LEN) {
            if (t == 0) big[atomicAdd(nbig, 1u)] = h;
            continue;
        }
        if (FORM == CW_SWEEP) {
            unsigned short *idx = (unsigned short *)ev, *ord = idx + MV;
            cw_rank_order<NT>(mv, m, smax, ev + MV, idx, ord, wsum);
            // what each share of the movers changes, then the counts its first one finds
            const u32 w = t >> 5, per = (m + 32 * NW - 1) / (32 * NW) * 32;
            const u32 i0 = w * per < m ? w * per : m, i1 = i0 + per < m ? i0 + per : m;
            u32 *cnt = ec + w * A.K, *pm = ec + (NW + 2 * w) * A.K;
            for (u32 i = i0 + lane; i < i1; i += 32) {
                const u32 pq = sl[ord[i]], one = (u32)mv[ord[i]] & MV_DST ? 0x10001u : 1u;
                atomicSub(&cnt[pq & 0xFFFFu], one);
                atomicAdd(&cnt[pq >> 16], one);
            }
            __syncthreads();
            for (u32 q = t; q < A.K; q += NT) {
                u32 run = tc[q];
#pragma unroll
                for (u32 k = 0; k < NW; ++k) {
                    const u32 d = ec[k * A.K + q];
                    ec[k * A.K + q] = run;
                    run += d;
                }
            }
            __syncthreads();
            cl_sweep<true>(A, mv, sl, ord, i0, i1, cnt, pm, pm + A.K, nullptr, A.wfx[h], base);
            continue;
        }
        u32 cap = 32;
        if (!DIRECT) {
            while (cap < 4 * m) cap <<= 1;  // at most 4 * MV
            for (u32 i = t; i < cap; i += NT) {
                keys[i] = NONE;
                tc[i] = 0;
                ec[i] = 0;
            }
            __syncthreads();
            for (u32 i = t; i < m; i += NT) {
                const u32 sp = hash_find_or_insert(keys, cap - 1, sl[i]), st = hash_find_or_insert(keys, cap - 1, sq[i]);
                if (sp == NONE || st == NONE) {
                    atomicExch(A.status, DEV_HASH_FULL);
                    sl[i] = 0;
                    continue;
                }
                sl[i] = sp | st << 16;
                atomicAdd(&ec[sp], 1u);
                atomicAdd(&ec[st], 1u);
            }
            __syncthreads();
            const u32 lm = A.lam[h];
            for (u32 j = t; j < lm; j += NT) {  // each partition once
                const u32 s = hash_find(keys, cap - 1, A.cpart[a + j]);
                if (s != NONE) tc[s] = A.ccnt[a + j] | A.cdcnt[a + j] << 16;
            }
        }
        if (cw_starts<NT>(ec, DIRECT ? A.K : cap, wsum) > CW_PAIRS * m) {
            if (t == 0) big[atomicAdd(nbig, 1u)] = h;
            continue;
        }
        // events: rank, join, destination pin; ec[b] becomes the end of partition b's
        for (u32 i = t; i < m; i += NT) {
            const u64 e = mv[i];
            const u32 pq = sl[i], x = (u32)(e >> 32) << 2 | ((u32)e & MV_DST ? 1u : 0u);
            ev[atomicAdd(&ec[pq & 0xFFFFu], 1u)] = x;
            ev[atomicAdd(&ec[pq >> 16], 1u)] = x | 2u;
        }
        __syncthreads();
        const u32 wh = A.wfx[h];
        for (u32 b0 = 0; b0 < m; b0 += NT) {
            const bool act = b0 + t < m;
            const u64 e = act ? mv[b0 + t] : 0;
            const u32 pq = act ? sl[b0 + t] : 0, sp = pq & 0xFFFFu, st = pq >> 16, r4 = (u32)(e >> 32) << 2;
            const auto found = [&](u32 b) {  // pins below, destination pins above
                u32 x = tc[b];
                for (u32 j = b ? ec[b - 1] : 0, end = ec[b]; j < end; ++j) {
                    const u32 y = ev[j];
                    if (y < r4) x += ((y & 2u) - 1u) * ((y & 1u) << 16 | 1u);
                }
                return x;
            };
            const u32 cP = act ? found(sp) : 0, cQ = act ? found(st) : 0;
            if (act) {
                const i64 d = leave_gain(A.encourage, wh, cP & 0xFFFFu) - ((cQ & 0xFFFFu) == 0 ? (i64)wh : 0);
                if (d) atomicAdd(&A.g2[(u32)e & ~MV_DST], (unsigned long long)d);
            }
            if (A.track) {  // uniform over the grid
                const bool dst = act && ((u32)e & MV_DST), ep = dst && cP >> 16 == 1, eq = dst && cQ >> 16 == 0;
                const u32 pid = DIRECT ? sp + base : ep ? keys[sp] : 0, qid = DIRECT ? st + base : eq ? keys[st] : 0;
                __syncwarp();
                emit_pair(A, ep, pid, eq, qid, (u32)(e >> 32));
            }
        }
    }
}

// Block-wide bitonic sort of buf[0, P) ascending (P a power of two).
__device__ void block_bitonic_u64(u64 *buf, u32 P) {
    for (u32 k = 2; k <= P; k <<= 1) {
        for (u32 j = k >> 1; j > 0; j >>= 1) {
            for (u32 i = threadIdx.x; i < P; i += blockDim.x) {
                const u32 ixj = i ^ j;
                if (ixj > i) {
                    const u64 x = buf[i], y = buf[ixj];
                    if ((x > y) == ((i & k) == 0)) {
                        buf[i] = y;
                        buf[ixj] = x;
                    }
                }
            }
            __syncthreads();
        }
    }
}

constexpr u32 CB_THREADS = 128;
constexpr u32 CB_MOV_MAX = 2048;  // movers of the block kernel, in shared memory
constexpr u32 CB_TAB_HASH = 8192; // hashed table slots of the block kernel, at most
constexpr size_t CB_DYN_MAX = (size_t)CB_MOV_MAX * 12 + (size_t)CB_TAB_HASH * 12;
// The block kernel's middle tier: hyperedges with at most CB_MID_MOV movers and, hashed, CB_MID_TAB
// table slots take blocks small enough for several per SM; the rest go on to the
// launch sized by the level's largest hyperedge.
constexpr u32 CB_MID_MOV = 512;
constexpr u32 CB_MID_TAB = 2048;

// Gather the movers of hyperedge h (rank << 32 | dst flag | node) into mvs[0, min(m, lim)) with
// the whole block; returns m (all of them, counted past lim) and their largest rank in *rmax.
// Warps reserve their movers' slots with one atomic each. Ends with the block synchronised.
__device__ __forceinline__ u32 cascade_gather(const CascadeArgs &A, u32 h, u64 *mvs, u32 lim, u32 *cntm, u32 *smax,
                                              u32 &rmax) {
    const u64 a = A.off[h], b = A.off[h + 1], d0 = a + A.nsrc[h];
    const u32 lane = threadIdx.x & 31;
    if (threadIdx.x == 0) { *cntm = 0; *smax = 0; }
    __syncthreads();
    u32 mymax = 0;
    for (u64 base = a; base < b; base += blockDim.x) {  // same trip count in every thread
        const u64 k = base + threadIdx.x;
        const u32 v = k < b ? A.pins[k] : 0, r = k < b ? A.state[v].x : NONE;
        const bool mvr = r != NONE;
        const u32 bal = __ballot_sync(0xFFFFFFFFu, mvr);
        u32 wbase = 0;
        if (lane == 0 && bal) wbase = atomicAdd(cntm, (u32)__popc(bal));
        wbase = __shfl_sync(0xFFFFFFFFu, wbase, 0);
        if (mvr) {
            const u32 pos = wbase + __popc(bal & ((1u << lane) - 1u));
            if (pos < lim) mvs[pos] = ((u64)r << 32) | (k >= d0 ? MV_DST : 0u) | v;
            mymax = r > mymax ? r : mymax;
        }
    }
    mymax = __reduce_max_sync(0xFFFFFFFFu, mymax);
    if (lane == 0 && mymax) atomicMax(smax, mymax);
    __syncthreads();
    const u32 m = *cntm;
    rmax = *smax;
    __syncthreads();  // read before the next hyperedge resets them
    return m;
}

constexpr u32 CB_SORT_R = 8;                          // keys per thread in the block bin sort
constexpr u32 CB_BIN_MAX = CB_SORT_R * CB_THREADS;    // more movers sort bitonically
constexpr u32 CB_BINS = 512;

// Sort of buf[0, m) (m <= CB_BIN_MAX, CB_THREADS threads) by the rank in the high word: ranks spread
// over CB_BINS bins by their leading bits, and a key's place in its bin is the number of smaller
// ranks there, one or two keys as a rule. About a tenth of a radix sort's instructions, which made
// up most of the block kernel's. idx holds 2 * CB_BIN_MAX shorts of scratch (the slots' array).
__device__ __forceinline__ void block_bin_sort_hi(u64 *buf, unsigned short *idx, u32 m, u32 rmax, u32 *bins, u32 *wsum) {
    constexpr u32 NW = CB_THREADS / 32, PER = CB_BINS / CB_THREADS;
    const u32 t = threadIdx.x, lane = t & 31, w = t >> 5;
    const u32 nb = 32 - __clz(rmax), sh = nb > 9 ? nb - 9 : 0;  // rank >> sh < CB_BINS
    static_assert(CB_BINS == 512, "nine leading bits");
    for (u32 i = t; i < CB_BINS; i += CB_THREADS) bins[i] = 0;
    __syncthreads();
    u64 key[CB_SORT_R];
    u32 at[CB_SORT_R];
#pragma unroll
    for (u32 r = 0; r < CB_SORT_R; ++r) {
        const u32 i = t + r * CB_THREADS;
        if (i >= m) continue;
        key[r] = buf[i];
        at[r] = atomicAdd(&bins[(u32)(key[r] >> 32) >> sh], 1u);
    }
    __syncthreads();
    u32 c[PER], s = 0;
#pragma unroll
    for (u32 k = 0; k < PER; ++k) { c[k] = bins[t * PER + k]; s += c[k]; }
    u32 x = s;
#pragma unroll
    for (u32 o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    u32 pre = x - s;
#pragma unroll
    for (u32 i = 0; i < NW; ++i)
        if (i < w) pre += wsum[i];
#pragma unroll
    for (u32 k = 0; k < PER; ++k) { bins[t * PER + k] = pre; pre += c[k]; }
    if (t == CB_THREADS - 1) bins[CB_BINS] = m;
    __syncthreads();
#pragma unroll
    for (u32 r = 0; r < CB_SORT_R; ++r) {
        const u32 i = t + r * CB_THREADS;
        if (i < m) idx[bins[(u32)(key[r] >> 32) >> sh] + at[r]] = (unsigned short)i;
    }
    __syncthreads();
#pragma unroll
    for (u32 r = 0; r < CB_SORT_R; ++r) {
        if (t + r * CB_THREADS >= m) continue;
        const u32 b = (u32)(key[r] >> 32) >> sh, lo = bins[b], hi = bins[b + 1];
        u32 p = lo;
        for (u32 j = lo; j < hi; ++j) p += buf[idx[j]] < key[r];
        at[r] = p;
    }
    __syncthreads();
#pragma unroll
    for (u32 r = 0; r < CB_SORT_R; ++r)
        if (t + r * CB_THREADS < m) buf[at[r]] = key[r];
    __syncthreads();
}

// Sort, tables, slots and sweep of one hyperedge whose m movers (largest rank rmax) are in mvs,
// block-wide. The shared-memory kernel sorts up to CB_BIN_MAX of them with the block bin sort (bins
// set); more, and the scratch kernel's, sort bitonically. Direct tables leave tk to the sweep's lane
// masks (2K words, zeroed).
__device__ __forceinline__ void cascade_block_one(const CascadeArgs &A, u32 h, u64 *mvs, u32 *sl, u32 m, u32 rmax,
                                                  u32 *tk, u32 *tc, u32 *td, u32 cap, bool direct, u32 *bins,
                                                  u32 *wsum) {
    u32 P = 1;
    while (P < m) P <<= 1;
    const bool binned = bins && m <= CB_BIN_MAX;
    if (!binned)
        for (u32 i = m + threadIdx.x; i < P; i += blockDim.x) mvs[i] = ~0ull;
    for (u32 i = threadIdx.x; i < cap; i += blockDim.x) { tc[i] = 0; td[i] = 0; }
    const u32 ntk = direct ? 2 * A.K : cap;
    for (u32 i = threadIdx.x; i < ntk; i += blockDim.x) tk[i] = direct ? 0u : NONE;
    __syncthreads();
    if (binned) block_bin_sort_hi(mvs, (unsigned short *)sl, m, rmax, bins, wsum);
    else block_bitonic_u64(mvs, P);
    cascade_fill(A, h, A.off[h], A.off[h + 1], A.lam ? A.lam[h] : 0, tk, tc, td, cap, direct, threadIdx.x, blockDim.x);
    __syncthreads();
    if (sl) {
        cascade_slots(A, h, mvs, sl, m, tk, cap, direct, threadIdx.x, blockDim.x);
        __syncthreads();
    }
    if (sl) {
        if (threadIdx.x < 32) cascade_sweep_warp(A, h, mvs, sl, m, tk, tc, td, direct ? tk : nullptr);
    } else if (threadIdx.x == 0) {
        cascade_sweep(A, h, mvs, sl, m, tk, tc, td, cap - 1, direct);
    }
    __syncthreads();
}

// Hyperedges with more movers than a warp takes: one block per hyperedge, everything in shared
// memory (dynamic: smov movers and their slots, then three tables of stab slots). A hyperedge
// with more than smov movers, or a hashed table above stab slots, is appended to `huge`.
__global__ void __launch_bounds__(CB_THREADS) k_cascade_block(CascadeArgs A, const u32 *__restrict__ list,
                                                              const u32 *__restrict__ nl, u32 smov, u32 stab,
                                                              u32 *__restrict__ huge, u32 *__restrict__ nhuge) {
    extern __shared__ __align__(16) unsigned char cb_smem[];
    __shared__ u32 cntm, smax;
    __shared__ u32 wsum[CB_THREADS / 32], bins[CB_BINS + 1];
    u64 *mvs = (u64 *)cb_smem;
    u32 *sl = (u32 *)(mvs + smov), *tk = sl + smov, *tc = tk + stab, *td = tc + stab;
    const bool direct = A.K <= CC_DIRECT_BLOCK_K;
    for (u32 idx = blockIdx.x; idx < *nl; idx += gridDim.x) {
        const u32 h = list[idx];
        u32 rmax;
        const u32 m = cascade_gather(A, h, mvs, smov, &cntm, &smax, rmax);
        const u32 cap = direct ? A.K : cascade_cap32(A.lam[h], m);
        if (m > smov || cap > stab) {
            if (threadIdx.x == 0) huge[atomicAdd(nhuge, 1u)] = h;
            continue;
        }
        cascade_block_one(A, h, mvs, sl, m, rmax, tk, tc, td, cap, direct, bins, wsum);
    }
}

// The rest: one block per SM, each with its slice of scratch regions sized by the level's
// largest hyperedge (mv_cap movers and slots, three tables of tab_cap slots).
__global__ void __launch_bounds__(CB_THREADS) k_cascade_huge(CascadeArgs A, const u32 *__restrict__ list,
                                                             const u32 *__restrict__ nl, u64 *scratch_mv,
                                                             u32 *scratch_sl, u32 *scratch_tab, u64 mv_cap,
                                                             u64 tab_cap) {
    __shared__ u32 cntm, smax;
    u64 *mvs = scratch_mv + (u64)blockIdx.x * mv_cap;
    u32 *tk = scratch_tab + (u64)blockIdx.x * 3 * tab_cap, *tc = tk + tab_cap, *td = tc + tab_cap;
    const bool direct = A.K <= CC_DIRECT_BLOCK_K;
    for (u32 idx = blockIdx.x; idx < *nl; idx += gridDim.x) {
        const u32 h = list[idx];
        u32 rmax;
        const u32 m = cascade_gather(A, h, mvs, (u32)mv_cap, &cntm, &smax, rmax);
        const u32 cap = direct ? A.K : cascade_cap32(A.lam[h], m);
        // 16-bit slots cover every direct table and hashed tables of up to 65536 slots
        u32 *sl = (direct || cap <= 65536) ? scratch_sl + (u64)blockIdx.x * mv_cap : nullptr;
        cascade_block_one(A, h, mvs, sl, m, rmax, tk, tc, td, cap, direct, nullptr, nullptr);
    }
}

// ------------------------------------------------------------------ prefix and validity
// G[i] = the cascaded gain of the i-th mover; the two following nmax-entry blocks (the size and
// inbound violations) start at zero.
__global__ void k_gather_g2(const u32 *__restrict__ mv, const u32 *__restrict__ dM, u32 nmax,
                            const unsigned long long *__restrict__ g2, i64 *__restrict__ G) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nmax) {
        G[i] = i < *dM ? (i64)g2[mv[i]] : 0;
        G[(u64)nmax + i] = 0;
        G[2 * (u64)nmax + i] = 0;
    }
}

// The event kernels loop over the device's counts: their capacities (two events per node, two
// transitions per destination pin) are mostly empty.
__device__ __forceinline__ u64 grid_first() { return (u64)blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ u64 grid_step() { return (u64)gridDim.x * blockDim.x; }
// size events: 2r = leave p, 2r+1 = join q
__global__ void k_size_events(const u32 *__restrict__ mv, const u32 *__restrict__ dM, const u32 *__restrict__ part,
                              const u32 *__restrict__ target, u32 *__restrict__ key, u32 *__restrict__ val) {
    const u64 ne = 2 * (u64)*dM;
    for (u64 i = grid_first(); i < ne; i += grid_step()) {
        const u32 v = mv[i >> 1];
        key[i] = (i & 1) ? target[v] : part[v];
        val[i] = (u32)i;
    }
}
__global__ void k_size_delta(const u32 *__restrict__ mv, const u32 *__restrict__ val, const u32 *__restrict__ dne,
                             const u32 *__restrict__ nsize, i64 *__restrict__ d) {
    const u32 ne = *dne;
    for (u64 i = grid_first(); i < ne; i += grid_step()) {
        const u32 ev = val[i];
        const i64 s = nsize[mv[ev >> 1]];
        d[i] = (ev & 1) ? s : -s;
    }
}
__global__ void k_size_flags(const u32 *__restrict__ key, const u32 *__restrict__ val, const i64 *__restrict__ d,
                             const i64 *__restrict__ E, const u32 *__restrict__ dne, const u64 *__restrict__ psize,
                             u64 omega, unsigned long long *__restrict__ Vs) {
    const u32 ne = *dne;
    for (u64 i = grid_first(); i < ne; i += grid_step()) {
        const u32 p = key[i];
        const u32 st = lower_bound_u32(key, ne, p);
        const i64 before = (i64)psize[p] + (E[i] - E[st]);
        const i64 after = before + d[i];
        const i64 exb = before > (i64)omega ? before - (i64)omega : 0;
        const i64 exa = after > (i64)omega ? after - (i64)omega : 0;
        if (exa != exb) atomicAdd(&Vs[val[i] >> 1], (unsigned long long)(exa - exb));
    }
}

__global__ void k_gather_by_dn(const u32 *__restrict__ src, const u32 *__restrict__ idx, u32 *__restrict__ dst,
                               const u32 *__restrict__ dn) {
    const u32 n = *dn;
    for (u64 i = grid_first(); i < n; i += grid_step()) dst[i] = src[idx[i]];
}
// transition keys: (partition, rank) in one word when both fit, else the rank alone (the
// partition is then a second stable pass). The count is clamped to the capacity nmax first (an
// overflow has already set the status word); later kernels read the clamped count.
__global__ void k_trans_keys(u32 *__restrict__ dT, u64 nmax, const u32 *__restrict__ tp,
                             const u32 *__restrict__ tr, u32 rbits, int combined, u32 *__restrict__ key,
                             u32 *__restrict__ perm) {
    const u64 j0 = grid_first(), cnt = *dT < nmax ? *dT : nmax;
    if (j0 == 0 && cnt < *dT) atomicMin(dT, (u32)cnt);
    for (u64 j = j0; j < cnt; j += grid_step()) {
        key[j] = combined ? ((tp[j] << rbits) | tr[j]) : tr[j];
        perm[j] = (u32)j;
    }
}
// after ordering by (p, r): partition, rank and delta of position i; the deltas of [*dT, nz) are zero
__global__ void k_trans_perm(const u32 *__restrict__ perm, const u32 *__restrict__ dT, u64 nz,
                             const u32 *__restrict__ tp, const u32 *__restrict__ tr, const int32_t *__restrict__ td,
                             u32 *__restrict__ sp, u32 *__restrict__ sr, i64 *__restrict__ sd) {
    const u64 nt = *dT, end = nt > nz ? nt : nz;
    for (u64 i = grid_first(); i < end; i += grid_step()) {
        if (i >= nt) { sd[i] = 0; continue; }
        const u32 j = perm[i];
        sp[i] = tp[j];
        sr[i] = tr[j];
        sd[i] = td[j];
    }
}
// per partition, the running inbound-set size along the move sequence; an event that makes the
// partition exceed delta adds +1 at its rank, one that brings it back adds -1. The first event of a
// partition assumes it started valid (kernels/refinement.cu:632-651).
__global__ void k_trans_flags(const u32 *__restrict__ sp, const u32 *__restrict__ sr, const i64 *__restrict__ sd,
                              const i64 *__restrict__ E, const u32 *__restrict__ dT, const u64 *__restrict__ pinb,
                              u64 delta, unsigned long long *__restrict__ Vi) {
    const u32 nt = *dT;
    for (u64 j = grid_first(); j < nt; j += grid_step()) {
        const u32 p = sp[j];
        const u32 st = lower_bound_u32(sp, nt, p);  // the partition's first transition (sp is sorted)
        const i64 before = (i64)pinb[p] + (E[j] - E[st]);
        const i64 after = before + sd[j];
        const bool was_bad = (j != st) && before > (i64)delta;
        const bool is_bad = after > (i64)delta;
        if (was_bad != is_bad) atomicAdd(&Vi[sr[j]], (unsigned long long)(i64)(is_bad ? 1 : -1));
    }
}

// ---- size and inbound validity of every prefix on small levels: one block per partition ----------
// The same quantities as the event pipelines above (k_size_events ... k_size_flags and
// k_trans_keys ... k_trans_flags), without sorting: a partition's size events are its movers in
// rank order, and its inbound transitions arrive summed per rank (CascadeArgs::tdense).
//  - sizes: Vs[r] += excess(after rank r) - excess(before), excess = max(size - omega, 0);
//  - inbound: Vi[r] += bad(after r) - bad(before r) at each rank with transitions, bad = the
//    running inbound count above delta, and "before" taken as good at the partition's first
//    such rank (kernels/refinement.cu:632-651). Both telescope over the events of one rank, so
//    the order of events within a rank does not matter.
constexpr u32 VS_THREADS = 1024;
constexpr u32 VS_MAX_K = 256;    // partitions (blocks)

__device__ __forceinline__ i64 block_incl_scan_i64(i64 v, i64 *sh, i64 &total) {
    const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const i64 y = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if ((int)lane >= o) v += y;
    }
    __syncthreads();
    if (lane == 31) sh[w] = v;
    __syncthreads();
    if (w == 0) {
        i64 x = lane < (blockDim.x >> 5) ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const i64 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if ((int)lane >= o) x += y;
        }
        sh[lane] = x;  // inclusive warp prefixes
    }
    __syncthreads();
    total = sh[(blockDim.x >> 5) - 1];
    return v + (w ? sh[w - 1] : 0);
}
// Partition p by the calling block of VS_THREADS threads. CLEAR: the transitions read are zeroed.
template <bool CLEAR>
__device__ __forceinline__ void validity_small_body(u32 p, u32 M, const u32 *mv, const u32 *part, const u32 *target,
                                                    const u32 *nsize, const u64 *psize, u64 omega, unsigned long long *Vs,
                                                    int track, unsigned long long *tdense, u32 stride, const u64 *pinb,
                                                    u64 delta, unsigned long long *Vi) {
    __shared__ i64 sh[32];
    i64 run = (i64)psize[p];
    const i64 om = (i64)omega;
    for (u32 base = 0; base < M; base += VS_THREADS) {
        const u32 r = base + threadIdx.x;
        i64 d = 0;
        if (r < M) {
            const u32 v = mv[r];
            if (part[v] == p) d = -(i64)nsize[v];
            else if (target[v] == p) d = (i64)nsize[v];
        }
        i64 tot;
        const i64 incl = block_incl_scan_i64(d, sh, tot);
        if (d != 0) {
            const i64 after = run + incl, before = after - d;
            const i64 dx = (after > om ? after - om : 0) - (before > om ? before - om : 0);
            if (dx) atomicAdd(&Vs[r], (unsigned long long)dx);
        }
        run += tot;
    }
    if (!track) return;
    const i64 dl = (i64)delta;
    i64 run2 = (i64)pinb[p];
    bool seen = false;  // a rank with transitions of p came before this chunk
    for (u32 base = 0; base < M; base += VS_THREADS) {
        const u32 r = base + threadIdx.x;
        const unsigned long long x = r < M ? tdense[(u64)p * stride + r] : 0ull;
        if (CLEAR && x) tdense[(u64)p * stride + r] = 0;
        const bool has = (u32)x != 0u;
        const i64 D = has ? (i64)(int32_t)(u32)(x >> 32) : 0;
        i64 tot, htot;
        const i64 incl = block_incl_scan_i64(D, sh, tot);
        const i64 hincl = block_incl_scan_i64(has ? 1 : 0, sh, htot);
        if (has) {
            const i64 after = run2 + incl, before = after - D;
            const bool first = !seen && hincl == 1;
            const bool bad_before = !first && before > dl, bad_after = after > dl;
            if (bad_before != bad_after) atomicAdd(&Vi[r], (unsigned long long)(i64)(bad_after ? 1 : -1));
        }
        run2 += tot;
        seen = seen || htot > 0;
    }
}
__global__ void __launch_bounds__(VS_THREADS) k_validity_small(
    const u32 *__restrict__ mv, const u32 *__restrict__ dM, const u32 *__restrict__ part,
    const u32 *__restrict__ target, const u32 *__restrict__ nsize, const u64 *__restrict__ psize, u64 omega,
    unsigned long long *__restrict__ Vs, int track, unsigned long long *__restrict__ tdense, u32 stride,
    const u64 *__restrict__ pinb, u64 delta, unsigned long long *__restrict__ Vi) {
    validity_small_body<false>(blockIdx.x, *dM, mv, part, target, nsize, psize, omega, Vs, track, tdense, stride, pinb, delta,
                               Vi);
}

// best prefix (best_move_functor): inbound-valid first, then fewer size violations, then larger
// gain, then the earlier rank.
struct Best {
    u32 ok;
    i64 vs, g;
    u32 r;
};
__device__ __forceinline__ bool best_better(const Best &b, const Best &a) {  // is b better than a
    if (a.ok != b.ok) return b.ok > a.ok;
    if (!a.ok) return b.r < a.r;
    if (a.vs != b.vs) return b.vs < a.vs;
    if (a.g != b.g) return b.g > a.g;
    return b.r < a.r;
}
__device__ __forceinline__ Best best_pick(const Best &a, const Best &b) {  // the better one; r = ~0 is empty
    if (b.r == 0xFFFFFFFFu) return a;
    if (a.r == 0xFFFFFFFFu) return b;
    return best_better(b, a) ? b : a;
}
__device__ __forceinline__ Best warp_best_prefix(Best b) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Best c;
        c.ok = __shfl_xor_sync(0xFFFFFFFFu, b.ok, o);
        c.vs = __shfl_xor_sync(0xFFFFFFFFu, b.vs, o);
        c.g = __shfl_xor_sync(0xFFFFFFFFu, b.g, o);
        c.r = __shfl_xor_sync(0xFFFFFFFFu, b.r, o);
        b = best_pick(b, c);
    }
    return b;
}
// ---- small levels (n <= RSS_CAP): ranking, and prefix sums + best prefix + apply, one block each ----
// The movers in id order, ranked by (gain desc, id asc): compaction by block scans, the stable
// radix sort of the descending gain keys (a second pass over the high words when the gain bound
// needs more than 32 bits), then the ranks. Also resets every node's rank and cascaded gain and
// writes the mover count and the size-event count, as k_move_flags ... k_set_rank do.
// sm: RSS_SMEM bytes. Returns the mover count.
__device__ __forceinline__ u32 rank_small_body(u32 *sm, u32 n, const u32 *target, const i64 *gain, u64 gbound, u32 kb,
                                               const u32 *part, u32 *mv, uint2 *state, unsigned long long *g2) {
    static_assert(VS_MAX_K <= STATE_PACK_K, "places hold targets");
    __shared__ i64 sh[32];
    u32 M = 0;
    for (u32 b = 0; b < n; b += blockDim.x) {
        const u32 v = b + threadIdx.x;
        const bool f = v < n && target[v] != NONE;
        if (v < n) { state[v] = make_uint2(NONE, state_place(part[v], target[v], 1)); g2[v] = 0; }
        i64 tot;
        const i64 incl = block_incl_scan_i64(f ? 1 : 0, sh, tot);
        if (f) {
            const u32 pos = M + (u32)incl - 1;
            sm[pos] = (u32)(gbound - (u64)gain[v]);
            sm[RSS_CAP + pos] = v;
        }
        M += (u32)tot;
    }
    const u32 *ko, *vo;
    block_radix_sort(sm, M, kb < 32 ? kb : 32, ko, vo);
    if (kb > 32) {  // high words of the movers in their low-word order
        u32 hv[RSS_ITEMS], nv[RSS_ITEMS];
#pragma unroll
        for (int k = 0; k < RSS_ITEMS; ++k) {
            const u32 i = threadIdx.x + (u32)k * blockDim.x;
            nv[k] = i < M ? vo[i] : 0u;
            hv[k] = i < M ? (u32)((gbound - (u64)gain[nv[k]]) >> 32) : 0u;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < RSS_ITEMS; ++k) {
            const u32 i = threadIdx.x + (u32)k * blockDim.x;
            if (i < M) { sm[i] = hv[k]; sm[RSS_CAP + i] = nv[k]; }
        }
        block_radix_sort(sm, M, kb - 32, ko, vo);
    }
    for (u32 i = threadIdx.x; i < M; i += blockDim.x) {
        const u32 v = vo[i];
        mv[i] = v;
        state[v].x = i;
    }
    return M;
}
__global__ void __launch_bounds__(RSS_WARPS * 32) k_rank_small(u32 n, const u32 *__restrict__ target,
                                                              const i64 *__restrict__ gain, u64 gbound, u32 kb,
                                                              const u32 *__restrict__ part, u32 *__restrict__ mv,
                                                              uint2 *__restrict__ state,
                                                              unsigned long long *__restrict__ g2, u32 *__restrict__ dM,
                                                              u32 *__restrict__ twice) {
    extern __shared__ u32 sm[];
    const u32 M = rank_small_body(sm, n, target, gain, gbound, kb, part, mv, state, g2);
    if (threadIdx.x == 0) {
        *dM = M;
        *twice = 2 * M;
    }
}

// The inclusive prefix sums by rank of the cascaded gains, size violations (Vs) and inbound
// violations (Vi), the best prefix by best_better, and its application when it is valid with a
// non-negative gain: k_gather_g2, the 3n scan, k_best, k_best_final and k_apply in one block.
// The block's best prefix: the number of movers to apply (0: none).
__device__ __forceinline__ u32 tail_small_body(u32 M, const u32 *mv, const unsigned long long *g2, const i64 *Vs,
                                               const i64 *Vi, int has_vi) {
    __shared__ i64 sh[32];
    __shared__ Best bsh[32];
    __shared__ i64 vsh[32];
    __shared__ Best s_best;
    __shared__ i64 s_vi;
    const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) { s_best = Best{0, 0, 0, 0xFFFFFFFFu}; s_vi = 0; }
    i64 rg = 0, rs = 0, ri = 0;
    for (u32 base = 0; base < M; base += blockDim.x) {
        const u32 r = base + threadIdx.x;
        const bool in = r < M;
        i64 tg, ts, ti;
        const i64 pg = rg + block_incl_scan_i64(in ? (i64)g2[mv[r]] : 0, sh, tg);
        const i64 ps = rs + block_incl_scan_i64(in ? Vs[r] : 0, sh, ts);
        const i64 pi = ri + block_incl_scan_i64(in ? Vi[r] : 0, sh, ti);
        Best b{has_vi ? (pi == 0 ? 1u : 0u) : 1u, ps, pg, in ? r : 0xFFFFFFFFu};
        i64 bvi = pi;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            Best c;
            c.ok = __shfl_xor_sync(0xFFFFFFFFu, b.ok, o);
            c.vs = __shfl_xor_sync(0xFFFFFFFFu, b.vs, o);
            c.g = __shfl_xor_sync(0xFFFFFFFFu, b.g, o);
            c.r = __shfl_xor_sync(0xFFFFFFFFu, b.r, o);
            const i64 cvi = __shfl_xor_sync(0xFFFFFFFFu, bvi, o);
            const Best x = best_pick(b, c);
            if (x.r != b.r) bvi = cvi;
            b = x;
        }
        if (lane == 0) { bsh[w] = b; vsh[w] = bvi; }
        __syncthreads();
        if (threadIdx.x == 0) {
            Best x = s_best;
            i64 xv = s_vi;
            for (u32 k = 0; k < blockDim.x / 32; ++k) {
                const Best y = best_pick(x, bsh[k]);
                if (y.r != x.r) xv = vsh[k];
                x = y;
            }
            s_best = x;
            s_vi = xv;
        }
        rg += tg;
        rs += ts;
        ri += ti;
    }
    __syncthreads();
    const Best x = s_best;
    const i64 vi = has_vi ? s_vi : 0;
    const bool ok = x.r != 0xFFFFFFFFu && x.vs <= 0 && vi <= 0 && x.g >= 0;
    return ok ? x.r + 1 : 0u;
}
__global__ void __launch_bounds__(1024) k_tail_small(const u32 *__restrict__ mv, const u32 *__restrict__ dM,
                                                     const unsigned long long *__restrict__ g2,
                                                     const i64 *__restrict__ Vs, const i64 *__restrict__ Vi, int has_vi,
                                                     const u32 *__restrict__ target, u32 *__restrict__ part,
                                                     u32 *__restrict__ apply) {
    const u32 end = tail_small_body(*dM, mv, g2, Vs, Vi, has_vi);
    if (threadIdx.x == 0) *apply = end ? 1u : 0u;
    for (u32 i = threadIdx.x; i < end; i += blockDim.x) {
        const u32 v = mv[i];
        part[v] = target[v];
    }
}

// best_better is a strict total order (ties end on the rank), so the tree reduction picks the
// same prefix as a sequential scan would.
// pre = inclusive scan of [gain deltas | size-violation deltas | inbound-violation deltas] by rank,
// each n long: the prefix of segment s at rank r is pre[s*n + r] - pre[s*n - 1].
__device__ __forceinline__ i64 seg_prefix(const i64 *pre, u32 n, u32 s, u32 r) {
    const u64 base = (u64)s * n;
    return pre[base + r] - (s ? pre[base - 1] : 0);
}
__global__ void k_best(const i64 *__restrict__ pre, u32 n, int has_vi, const u32 *__restrict__ dM,
                       Best *__restrict__ out) {
    __shared__ Best sh[32];
    Best b{0, 0, 0, 0xFFFFFFFFu};
    const u32 M = *dM;
    for (u32 r = blockIdx.x * blockDim.x + threadIdx.x; r < M; r += gridDim.x * blockDim.x) {
        const u32 ok = has_vi ? (seg_prefix(pre, n, 2, r) == 0 ? 1u : 0u) : 1u;
        Best c{ok, seg_prefix(pre, n, 1, r), seg_prefix(pre, n, 0, r), r};
        b = best_pick(b, c);
    }
    b = warp_best_prefix(b);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x < 32) {
        Best x = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : Best{0, 0, 0, 0xFFFFFFFFu};
        x = warp_best_prefix(x);
        if (threadIdx.x == 0) out[blockIdx.x] = x;
    }
}
__global__ void __launch_bounds__(32) k_best_final(const Best *__restrict__ in, u32 nb, const i64 *__restrict__ pre,
                                                   u32 n, int has_vi, Best *__restrict__ out, u32 *__restrict__ apply) {
    Best x{0, 0, 0, 0xFFFFFFFFu};
    for (u32 i = threadIdx.x; i < nb; i += 32) x = best_pick(x, in[i]);
    x = warp_best_prefix(x);
    if (threadIdx.x) return;
    *out = x;
    const i64 vi = (has_vi && x.r != 0xFFFFFFFFu) ? seg_prefix(pre, n, 2, x.r) : 0;
    *apply = (x.r != 0xFFFFFFFFu && x.vs <= 0 && vi <= 0 && x.g >= 0) ? 1u : 0u;
}
// With prev set (incremental census), a moved node's old partition and the round counter are kept.
__global__ void k_apply(const u32 *__restrict__ mv, const u32 *__restrict__ target, const Best *__restrict__ best,
                        const u32 *__restrict__ apply, u32 *__restrict__ part, u32 *__restrict__ prev,
                        u32 *__restrict__ stamp, const u32 *__restrict__ ctr) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (!*apply || i > best->r) return;
    u32 v = mv[i];
    if (prev) {
        prev[v] = part[v];
        stamp[v] = *ctr;
    }
    part[v] = target[v];
}

// Copies (the k-way multi-start): moves are sorted by copy last, so every copy owns one rank
// segment; ck[r] is the copy of rank r. One block per copy finds its segment's best prefix with
// the prefix values taken relative to the segment start, and decides its own application.
__global__ void k_copy_keys(const u32 *__restrict__ mv, const u32 *__restrict__ dM, u32 copy_n, u32 *__restrict__ ck) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < *dM) ck[i] = mv[i] / copy_n;
}
__global__ void k_best_seg(const i64 *__restrict__ pre, u32 n, int has_vi, const u32 *__restrict__ dM,
                           const u32 *__restrict__ ck, Best *__restrict__ best, u32 *__restrict__ capply,
                           u32 *__restrict__ apply) {
    __shared__ Best sh[32];
    const u32 M = *dM, t = blockIdx.x;
    const u32 s = lower_bound_u32(ck, M, t), e = lower_bound_u32(ck, M, t + 1);
    const i64 g0 = s ? seg_prefix(pre, n, 0, s - 1) : 0, v0 = s ? seg_prefix(pre, n, 1, s - 1) : 0;
    const i64 i0 = (s && has_vi) ? seg_prefix(pre, n, 2, s - 1) : 0;
    Best b{0, 0, 0, 0xFFFFFFFFu};
    for (u32 r = s + threadIdx.x; r < e; r += blockDim.x) {
        const u32 ok = has_vi ? (seg_prefix(pre, n, 2, r) - i0 == 0 ? 1u : 0u) : 1u;
        Best c{ok, seg_prefix(pre, n, 1, r) - v0, seg_prefix(pre, n, 0, r) - g0, r};
        b = best_pick(b, c);
    }
    b = warp_best_prefix(b);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x < 32) {
        Best x = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : Best{0, 0, 0, 0xFFFFFFFFu};
        x = warp_best_prefix(x);
        if (threadIdx.x == 0) {
            best[t] = x;
            const i64 vi = (has_vi && x.r != 0xFFFFFFFFu) ? seg_prefix(pre, n, 2, x.r) - i0 : 0;
            const u32 ap = (x.r != 0xFFFFFFFFu && x.vs <= 0 && vi <= 0 && x.g >= 0) ? 1u : 0u;
            capply[t] = ap;
            if (ap) atomicOr(apply, 1u);
        }
    }
}
__global__ void k_apply_seg(const u32 *__restrict__ mv, const u32 *__restrict__ dM, const u32 *__restrict__ ck,
                            const u32 *__restrict__ target, const Best *__restrict__ best,
                            const u32 *__restrict__ capply, u32 *__restrict__ part, u32 *__restrict__ prev,
                            u32 *__restrict__ stamp, const u32 *__restrict__ ctr) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *dM) return;
    const u32 t = ck[i];
    if (!capply[t] || i > best[t].r) return;
    const u32 v = mv[i];
    if (prev) {
        prev[v] = part[v];
        stamp[v] = *ctr;
    }
    part[v] = target[v];
}

// ------------------------------------------------------------------ k-way levels of few partitions
// K-way rounds without an inbound limit need no census entries when a copy holds at most KW_K
// partitions. A hyperedge's record is two K-bit masks of MW words: the partitions present, and
// those holding exactly one of its pins. With w its weight, a node in partition p gains w for
// every incidence where p is single (what leaving saves) and pays w for every incidence where
// the target is absent: both are bits, so a node's gains are sums over its incidences' records
// and no per-pin sums are kept. A level keeps its records across its rounds; after each apply
// the hyperedges of the moved nodes are flagged, and the next round rewrites only those. The
// copies of a multi-start use partition ids local to their copy, so a record is as wide as one
// copy's partitions whatever the number of copies.
constexpr u32 KW_K = 256;
constexpr u32 KW_SHORT = 8;      // pins one lane reads; longer hyperedges take the warp
constexpr u32 KW_THREADS = 256;

struct KwArgs {
    const u64 *off;
    const u32 *pins, *part;
    u32 e, ce, k;    // hyperedges; hyperedges and partitions of one copy
    u32 *rec;        // [e * 2 * MW]: present words, then single words
    uint8_t *dirty;  // [e]
    u32 per_warp;    // hyperedges one warp looks at (at most 32)
};

template <u32 MW>
__device__ __forceinline__ void kw_add(u32 (&any)[MW], u32 (&mul)[MW], u32 q) {
    const u32 bit = 1u << (q & 31u);
#pragma unroll
    for (u32 x = 0; x < MW; ++x) {  // no branch: the words stay in registers
        const u32 m = MW == 1 || x == (q >> 5) ? bit : 0u;
        mul[x] |= any[x] & m;
        any[x] |= m;
    }
}
template <u32 MW>
__device__ __forceinline__ void kw_store(u32 *rec, const u32 (&any)[MW], const u32 (&mul)[MW]) {
    u32 out[2 * MW];
#pragma unroll
    for (u32 x = 0; x < MW; ++x) {
        out[x] = any[x];
        out[MW + x] = any[x] & ~mul[x];
    }
    store_words<2 * MW>(rec, out);
}

// The records of the flagged hyperedges, which are unflagged. A warp looks at per_warp hyperedges:
// a lane does its own when it has at most KW_SHORT pins, the warp the others one by one.
// Measured: the multi-start of 200k nodes, 64 parts, 896 partitions in all: 1074 us a hashed
// census, 8 with only the moved nodes' hyperedges rewritten.
template <u32 MW>
__global__ void __launch_bounds__(KW_THREADS) k_kway_records(KwArgs A) {
    const u32 lane = threadIdx.x & 31u;
    const u32 h0 = (blockIdx.x * (KW_THREADS / 32) + (threadIdx.x >> 5)) * A.per_warp;
    const u32 h = h0 + lane;
    bool mine = lane < A.per_warp && h < A.e && A.dirty[h];
    const u64 a = mine ? A.off[h] : 0, len64 = mine ? A.off[h + 1] - a : 0;
    mine = mine && len64 <= CD_WARP_LEN;  // longer ones are k_kway_records_block's
    const u32 len = mine ? (u32)len64 : 0;
    const u32 base = mine ? (h / A.ce) * A.k : 0;
    if (mine) A.dirty[h] = 0;
    u32 any[MW], mul[MW];
#pragma unroll
    for (u32 x = 0; x < MW; ++x) any[x] = mul[x] = 0;
    if (mine && len <= KW_SHORT) {
        u32 q[KW_SHORT];
#pragma unroll
        for (u32 i = 0; i < KW_SHORT; ++i) q[i] = i < len ? A.part[A.pins[a + i]] - base : NONE;
#pragma unroll
        for (u32 i = 0; i < KW_SHORT; ++i)
            if (i < len) kw_add<MW>(any, mul, q[i]);
        kw_store<MW>(A.rec + (u64)h * (2 * MW), any, mul);
    }
    u32 rest = __ballot_sync(0xFFFFFFFFu, mine && len > KW_SHORT);
    while (rest) {
        const u32 t = __ffs(rest) - 1;
        rest &= rest - 1;
        const u64 at = __shfl_sync(0xFFFFFFFFu, a, t);
        const u32 lt = __shfl_sync(0xFFFFFFFFu, len, t), bt = __shfl_sync(0xFFFFFFFFu, base, t);
#pragma unroll
        for (u32 x = 0; x < MW; ++x) any[x] = mul[x] = 0;
#pragma unroll 4
        for (u32 i = lane; i < lt; i += 32) kw_add<MW>(any, mul, A.part[A.pins[at + i]] - bt);
#pragma unroll
        for (u32 o = 16; o > 0; o >>= 1)
#pragma unroll
            for (u32 x = 0; x < MW; ++x) {
                const u32 a2 = __shfl_xor_sync(0xFFFFFFFFu, any[x], o), m2 = __shfl_xor_sync(0xFFFFFFFFu, mul[x], o);
                mul[x] |= m2 | (any[x] & a2);
                any[x] |= a2;
            }
        if (lane == 0) kw_store<MW>(A.rec + (u64)(h0 + t) * (2 * MW), any, mul);
    }
}

// Hyperedges above CD_WARP_LEN pins (the level's block list), one block each, when flagged.
template <u32 MW>
__global__ void __launch_bounds__(KW_THREADS) k_kway_records_block(KwArgs A, const u32 *__restrict__ list, u32 nlist) {
    __shared__ u32 cnt[MW * 32];
    for (u32 idx = blockIdx.x; idx < nlist; idx += gridDim.x) {
        const u32 h = list[idx];
        if (!A.dirty[h]) continue;  // uniform over the block
        const u64 a = A.off[h], b = A.off[h + 1];
        const u32 base = (h / A.ce) * A.k;
        for (u32 i = threadIdx.x; i < MW * 32; i += KW_THREADS) cnt[i] = 0;
        __syncthreads();
        for (u64 i = a + threadIdx.x; i < b; i += KW_THREADS) atomicAdd(&cnt[A.part[A.pins[i]] - base], 1u);
        __syncthreads();
        for (u32 x = threadIdx.x >> 5; x < MW; x += KW_THREADS / 32) {
            const u32 c = cnt[x * 32 + (threadIdx.x & 31u)];
            const u32 any = __ballot_sync(0xFFFFFFFFu, c > 0), one = __ballot_sync(0xFFFFFFFFu, c == 1);
            if ((threadIdx.x & 31u) == 0) {
                A.rec[(u64)h * (2 * MW) + x] = any;
                A.rec[(u64)h * (2 * MW) + MW + x] = one;
            }
        }
        if (threadIdx.x == 0) A.dirty[h] = 0;
        __syncthreads();
    }
}

// Connectivity of every copy from the records: conn[t] += w * (partitions present - 1).
template <u32 MW>
__global__ void __launch_bounds__(KW_THREADS) k_kway_conn(KwArgs A, const u32 *__restrict__ wfx,
                                                          unsigned long long *__restrict__ conn) {
    const u32 t = blockIdx.y;
    u64 s = 0;
    for (u32 j = blockIdx.x * KW_THREADS + threadIdx.x; j < A.ce; j += gridDim.x * KW_THREADS) {
        const u64 h = (u64)t * A.ce + j;
        u32 any[MW], l = 0;
        load_words<MW>(A.rec + h * (2 * MW), any);
#pragma unroll
        for (u32 x = 0; x < MW; ++x) l += __popc(any[x]);
        if (l > 1) s += (u64)wfx[h] * (l - 1);
    }
    s = warp_sum(s);
    if ((threadIdx.x & 31u) == 0 && s) atomicAdd(&conn[t], (unsigned long long)s);
}

struct KwGain {
    const u32 *rec;
    u32 k, cn;  // partitions and nodes of one copy
    const u32 *list;
    u32 nl;
    int uni;     // every hyperedge has the weight `weight`
    u32 weight;
};

// Best target of node u from the lanes' connectivities: lane `own` of a group of G holds those of
// its partitions own, own + G, ... (conn[x]); the group's lane 0 writes the move. A partition
// without connectivity gains at most saving - wtot <= 0, so presence needs no test.
// EARLY: a partition's gain is looked at before its size, and a group without a gain skips the
// reduction, as most do in the later rounds (the plane kernels, which come here once per hundreds of
// incidences, got slower by it: 110 -> 130 us a launch).
template <u32 G, u32 C, class T, bool EARLY = false>
__device__ __forceinline__ void kw_move(const GainArgs &A, u32 u, u32 base, u32 pl, u32 k, u32 own, u32 gmask,
                                        const T (&conn)[C], T saving, T wtot) {
    Cand best{INT64_MIN, 0};
    const u64 s = A.nsize[u], need = s - s / A.discount;
#pragma unroll
    for (u32 x = 0; x < C; ++x) {
        const u32 q = own + G * x;
        const i64 g = (i64)saving - ((i64)wtot - (i64)conn[x]);
        if (q >= k || q == pl || (EARLY ? g <= 0 : conn[x] == 0)) continue;
        if (A.psize[base + q] + need > A.omega) continue;
        const Cand c{g, ((u64)mix32(base + q + A.round + A.seed) << 32) | (u64)(~(base + q))};
        if (cand_better(c, best)) best = c;
    }
    if (EARLY && !__any_sync(gmask, best.g > 0)) {
        if (own == 0) write_move(A, u, best);
        return;
    }
#pragma unroll
    for (u32 o = G / 2; o > 0; o >>= 1) {
        Cand d;
        d.g = __shfl_xor_sync(gmask, best.g, o);
        d.tie = __shfl_xor_sync(gmask, best.tie, o);
        if (cand_better(d, best)) best = d;
    }
    if (own == 0) write_move(A, u, best);
}

// One group of G lanes per node (G a power of two, at least k for one word): lane l owns
// partitions l, l + G, ... (C of them) and reads every incidence's record, the same addresses across the group. T: u32 when
// no node's incident weights pass 2^32, else u64.
// Bound by issue and the records' L2 reads. Measured: the same multi-start 1970 us hashed, 46 to
// 70; 1M nodes 16 parts 218 from the census' masks, 101.
template <u32 MW, u32 G, class T>
__global__ void __launch_bounds__(KW_THREADS) k_kway_gain(GainArgs A0, KwGain V) {
    static_assert(MW == 1 || G == 32, "one word: a lane per partition; more: a lane per bit of each");
    constexpr u32 C = MW;
    const GainArgs A = gain_args_now(A0);
    const u32 lane = threadIdx.x & 31u, own = lane & (G - 1);
    const u32 gmask = G == 32 ? 0xFFFFFFFFu : ((1u << G) - 1u) << (lane & ~(G - 1));
    const u32 idx = blockIdx.x * (KW_THREADS / G) + threadIdx.x / G;
    if (idx >= V.nl) return;
    const u32 u = V.list[idx], base = (u / V.cn) * V.k, pl = A.part[u] - base;
    const u64 t0 = A.toff[u];
    const u32 deg = (u32)(A.toff[u + 1] - t0);
    T conn[C], saving = 0, wtot = 0;
#pragma unroll
    for (u32 x = 0; x < C; ++x) conn[x] = 0;
#pragma unroll 4
    for (u32 j = 0; j < deg; ++j) {
        const u32 h = A.touch[t0 + j], w = V.uni ? V.weight : A.wfx[h];
        const u32 *r = V.rec + (u64)h * (2 * MW);
        u32 any[MW];
        u32 sg;
        if constexpr (MW == 1) {
            const uint2 v = *(const uint2 *)r;
            any[0] = v.x;
            sg = v.y;
        } else {
            load_words<MW>(r, any);
            sg = r[MW + (pl >> 5)];
        }
        wtot += w;
        if ((sg >> (pl & 31u)) & 1u) saving += w;
#pragma unroll
        for (u32 x = 0; x < C; ++x)
            if ((any[x] >> own) & 1u) conn[x] += w;
    }
    kw_move<G, C, T, true>(A, u, base, pl, V.k, own, gmask, conn, saving, wtot);
}

// At most 4 partitions: a group of G lanes per node takes the incidences side by side, each lane
// with a sum per partition, summed over the group at the end.
template <u32 G, class T>
__global__ void __launch_bounds__(KW_THREADS) k_kway_gain_few(GainArgs A0, KwGain V) {
    const GainArgs A = gain_args_now(A0);
    const u32 lane = threadIdx.x & 31u, own = lane & (G - 1);
    const u32 gmask = G == 32 ? 0xFFFFFFFFu : ((1u << G) - 1u) << (lane & ~(G - 1));
    const u32 idx = blockIdx.x * (KW_THREADS / G) + threadIdx.x / G;
    if (idx >= V.nl) return;
    const u32 u = V.list[idx], base = (u / V.cn) * V.k, pl = A.part[u] - base;
    const u64 t0 = A.toff[u];
    const u32 deg = (u32)(A.toff[u + 1] - t0);
    T conn[4] = {0, 0, 0, 0}, saving = 0, wtot = 0;
#pragma unroll 2
    for (u32 j = own; j < deg; j += G) {
        const u32 h = A.touch[t0 + j], w = V.uni ? V.weight : A.wfx[h];
        const uint2 r = *(const uint2 *)(V.rec + (u64)h * 2);
        wtot += w;
        if ((r.y >> pl) & 1u) saving += w;
#pragma unroll
        for (u32 x = 0; x < 4; ++x)
            if ((r.x >> x) & 1u) conn[x] += w;
    }
    __syncwarp(gmask);
#pragma unroll
    for (u32 o = G / 2; o > 0; o >>= 1) {
        wtot += __shfl_xor_sync(gmask, wtot, o);
        saving += __shfl_xor_sync(gmask, saving, o);
#pragma unroll
        for (u32 x = 0; x < 4; ++x) conn[x] += __shfl_xor_sync(gmask, conn[x], o);
    }
    T mine[1] = {own == 0 ? conn[0] : own == 1 ? conn[1] : own == 2 ? conn[2] : own == 3 ? conn[3] : (T)0};
    kw_move<G, 1, T, true>(A, u, base, pl, V.k, own, gmask, mine, saving, wtot);
}

// One block per node (heavy nodes and small levels): each warp takes every eighth incidence with a
// lane per 32 partitions as above, and the warps' sums meet in shared memory.
template <u32 MW, class T>
__global__ void __launch_bounds__(KW_THREADS) k_kway_gain_block(GainArgs A0, KwGain V) {
    constexpr u32 NW = KW_THREADS / 32;
    const GainArgs A = gain_args_now(A0);
    __shared__ T sc[NW][MW * 32], ss[NW], sw[NW];
    const u32 lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    for (u32 idx = blockIdx.x; idx < V.nl; idx += gridDim.x) {
        const u32 u = V.list[idx], base = (u / V.cn) * V.k, pl = A.part[u] - base;
        const u64 t0 = A.toff[u], deg = A.toff[u + 1] - t0;
        T conn[MW], saving = 0, wtot = 0;
#pragma unroll
        for (u32 x = 0; x < MW; ++x) conn[x] = 0;
#pragma unroll 4
        for (u64 j = w; j < deg; j += NW) {
            const u32 h = A.touch[t0 + j], wh = V.uni ? V.weight : A.wfx[h];
            const u32 *r = V.rec + (u64)h * (2 * MW);
            u32 any[MW];
            load_words<MW>(r, any);
            const u32 sg = r[MW + (pl >> 5)];
            wtot += wh;
            if ((sg >> (pl & 31u)) & 1u) saving += wh;
#pragma unroll
            for (u32 x = 0; x < MW; ++x)
                if ((any[x] >> lane) & 1u) conn[x] += wh;
        }
#pragma unroll
        for (u32 x = 0; x < MW; ++x) sc[w][x * 32 + lane] = conn[x];
        if (lane == 0) { ss[w] = saving; sw[w] = wtot; }
        __syncthreads();
        if (w == 0) {
            saving = wtot = 0;
            for (u32 i = 0; i < NW; ++i) { saving += ss[i]; wtot += sw[i]; }
#pragma unroll
            for (u32 x = 0; x < MW; ++x) {
                conn[x] = 0;
                for (u32 i = 0; i < NW; ++i) conn[x] += sc[i][x * 32 + lane];
            }
            kw_move<32, MW, T>(A, u, base, pl, V.k, lane, 0xFFFFFFFFu, conn, saving, wtot);
        }
        __syncthreads();  // warp 0 has read the sums
    }
}

// Equal weights and many incidences per node: connectivity as a count, by bit planes (k_gain_planes)
// over the records' present words. A lane owns one word of an incidence, so 32 / MW incidences go
// side by side and an incidence costs a lane a few bit operations for 32 partitions, against one
// test and add per partition. A warp per node, or with BLOCK a block of KW_THREADS whose warps split
// the incidences. NP: planes, enough for a warp's incidences.
constexpr u32 KP_PLANES = 11, KP_PLANES_BLOCK = 14;
static_assert(KW_WARP_DEG < (1u << KP_PLANES), "a warp's counters hold its node's incidences");
// Measured: 20 x 5000 network, 128 parts 1069 us from the census' masks, 109 and 155 (light and
// heavy nodes).
template <u32 MW, bool BLOCK>
__global__ void __launch_bounds__(KW_THREADS) k_kway_planes(GainArgs A0, KwGain V) {
    constexpr u32 NP = BLOCK ? KP_PLANES_BLOCK : KP_PLANES, NW = KW_THREADS / 32, S = 32 / MW;
    const GainArgs A = gain_args_now(A0);
    __shared__ u32 sc[BLOCK ? NW : 1][MW * 32], ss[NW];
    const u32 lane = threadIdx.x & 31u, w = threadIdx.x >> 5, wl = lane & (MW - 1), slot = lane / MW;
    const u32 first = BLOCK ? blockIdx.x : blockIdx.x * NW + w, step = BLOCK ? gridDim.x : gridDim.x * NW;
    for (u32 idx = first; idx < V.nl; idx += step) {
        const u32 u = V.list[idx], base = (u / V.cn) * V.k, pl = A.part[u] - base;
        const u64 t0 = A.toff[u];
        const u32 deg = (u32)(A.toff[u + 1] - t0);
        // BLOCK: warp w takes incidences [j0, j1)
        const u32 share = BLOCK ? (deg + NW - 1) / NW : deg, j0 = BLOCK ? min(deg, w * share) : 0;
        const u32 cnt = BLOCK ? min(share, deg - j0) : deg;
        const u32 *t = A.touch + t0 + j0;
        u32 pc[NP];
        plane_count<NP>(t, cnt, V.rec, 2 * MW, MW, wl, slot, S, pc);
#pragma unroll
        for (u32 o = 16; o >= MW; o >>= 1) plane_merge<NP>(pc, o);
        u32 one = 0;  // incidences whose only pin in u's partition is u
        for (u32 j = lane; j < cnt; j += 32)
            one += (V.rec[(u64)t[j] * (2 * MW) + MW + (pl >> 5)] >> (pl & 31u)) & 1u;
        one = __reduce_add_sync(0xFFFFFFFFu, one);
        unsigned long long conn[MW];
#pragma unroll
        for (u32 x = 0; x < MW; ++x) {
            u32 c = 0;
#pragma unroll
            for (u32 b = 0; b < NP; ++b) c += ((__shfl_sync(0xFFFFFFFFu, pc[b], x) >> lane) & 1u) << b;
            if (BLOCK) sc[w][x * 32 + lane] = c;
            else conn[x] = (unsigned long long)c * V.weight;
        }
        if (BLOCK) {
            if (lane == 0) ss[w] = one;
            __syncthreads();
            if (w == 0) {
                one = 0;
                for (u32 i = 0; i < NW; ++i) one += ss[i];
#pragma unroll
                for (u32 x = 0; x < MW; ++x) {
                    u32 c = 0;
                    for (u32 i = 0; i < NW; ++i) c += sc[i][x * 32 + lane];
                    conn[x] = (unsigned long long)c * V.weight;
                }
            }
        }
        if (!BLOCK || w == 0)
            kw_move<32, MW, unsigned long long>(A, u, base, pl, V.k, lane, 0xFFFFFFFFu, conn,
                                                (unsigned long long)one * V.weight, (unsigned long long)deg * V.weight);
        if (BLOCK) __syncthreads();  // warp 0 has read the sums
    }
}

// After the apply: the hyperedges of the moved nodes are flagged for the next round's records. The
// movers of copy t are mv[t * cn, ...) in rank order and its first applied[t] moved (one copy:
// the movers up to the best prefix's rank).
__global__ void k_kway_mark(const u32 *__restrict__ mv, u32 cn, u32 copies, const u32 *__restrict__ applied,
                            const u64 *__restrict__ toff, const u32 *__restrict__ touch, uint8_t *__restrict__ dirty) {
    const u32 lane = threadIdx.x & 31u, nw = (gridDim.x * blockDim.x) >> 5;
    const u32 w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    for (u32 t = 0; t < copies; ++t) {
        const u32 M = applied[t];
        for (u32 i = w0; i < M; i += nw) {
            const u32 v = mv[(u64)t * cn + i];
            for (u64 j = toff[v] + lane; j < toff[v + 1]; j += 32) dirty[touch[j]] = 1;
        }
    }
}

// The same after the ranking of larger levels: the movers mv[0, *dM) in rank order, their copies in
// ck (null: one copy), those up to their copy's best rank moved where its apply flag is set.
__global__ void k_kway_mark_ranked(const u32 *__restrict__ mv, const u32 *__restrict__ dM, const u32 *__restrict__ ck,
                                   const Best *__restrict__ best, const u32 *__restrict__ apply,
                                   const u64 *__restrict__ toff, const u32 *__restrict__ touch,
                                   uint8_t *__restrict__ dirty) {
    const u32 lane = threadIdx.x & 31u, nw = (gridDim.x * blockDim.x) >> 5, M = *dM;
    for (u32 i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < M; i += nw) {
        const u32 t = ck ? ck[i] : 0;
        if (!apply[t] || i > best[t].r) continue;
        const u32 v = mv[i];
        for (u64 j = toff[v] + lane; j < toff[v + 1]; j += 32) dirty[touch[j]] = 1;
    }
}

// ---- ranking, validity and the best prefix of k-way copies of at most RSS_CAP nodes -----------
// A copy's moves depend on no other copy, so one block ranks each copy's moves in shared memory
// (a level of one copy is the case copies = 1), and ranks, prefixes and the best prefix are per
// copy. The order is that of the launches for larger levels: moves by (gain desc, id asc), the
// i-th of a -> b beside the i-th of b -> a, pairs by (pair gain desc, position, direction).
struct CopyArgs {
    u32 cn, k;                  // nodes and partitions of one copy
    u32 n;                      // nodes of all copies
    const u32 *target, *nsize;
    const i64 *gain;
    u32 *part;
    u64 gbound, pbound;         // bounds of the gains and of the pair gains
    u32 kb, pb, gb;             // their bits; bits of a direction group
    u32 *mv;                    // [n] movers of copy t in rank order from t * cn
    u32 *dM;                    // [copies] movers
    uint2 *state;               // [n]
    unsigned long long *g2;     // [n] cascaded gains (zeroed here)
    i64 *psn;                   // [n] pair gain of a mover
    i64 *vs;                    // [n] size violations by rank (zeroed here)
    u64 *psize;                 // [copies * k]
    u32 *applied;               // [copies]
    u32 *apply;                 // any copy moved
    u64 omega;
    int packed;                 // states hold targets
};

// Stable sort of the block's (key, node) pairs by a 64-bit key of `bits` bits: the low words are in
// sm (as block_radix_sort takes them), the high words come from hi(node).
template <class F>
__device__ __forceinline__ void copy_sort64(u32 *sm, u32 M, u32 bits, const u32 *&ko, const u32 *&vo, F &&hi) {
    block_radix_sort(sm, M, bits < 32 ? bits : 32, ko, vo);
    if (bits <= 32) return;
    u32 hv[RSS_ITEMS], nv[RSS_ITEMS];
#pragma unroll
    for (int x = 0; x < RSS_ITEMS; ++x) {
        const u32 i = threadIdx.x + (u32)x * blockDim.x;
        nv[x] = i < M ? vo[i] : 0u;
        hv[x] = i < M ? hi(nv[x]) : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int x = 0; x < RSS_ITEMS; ++x) {
        const u32 i = threadIdx.x + (u32)x * blockDim.x;
        if (i < M) { sm[i] = hv[x]; sm[RSS_CAP + i] = nv[x]; }
    }
    block_radix_sort(sm, M, bits - 32, ko, vo);
}

// Bound by one block's latency per copy. Measured: 14 copies 66 us, with k_copy_sizes 38 and
// k_copy_tail 22, in place of about 60 launches a round.
__global__ void __launch_bounds__(RSS_WARPS * 32) k_copy_rank(CopyArgs A) {
    extern __shared__ u32 sm[];
    __shared__ i64 sh[32];
    const u32 t = blockIdx.x, v0 = t * A.cn, base = t * A.k, T = blockDim.x;
    u32 M = 0;
    for (u32 b = 0; b < A.cn; b += T) {
        const u32 i = b + threadIdx.x, v = v0 + i;
        const bool f = i < A.cn && A.target[v] != NONE;
        if (i < A.cn) {
            A.state[v] = make_uint2(NONE, state_place(A.part[v], A.target[v], A.packed));
            A.g2[v] = 0;
            A.vs[v] = 0;
        }
        i64 tot;
        const i64 incl = block_incl_scan_i64(f ? 1 : 0, sh, tot);
        if (f) {
            const u32 pos = M + (u32)incl - 1;
            sm[pos] = (u32)(A.gbound - (u64)A.gain[v]);
            sm[RSS_CAP + pos] = v;
        }
        M += (u32)tot;
    }
    const u32 *ko, *vo;
    copy_sort64(sm, M, A.kb, ko, vo, [&](u32 v) { return (u32)((A.gbound - (u64)A.gain[v]) >> 32); });
    // by direction group, each in gain order
    u32 key[RSS_ITEMS], nd[RSS_ITEMS];
#pragma unroll
    for (int x = 0; x < RSS_ITEMS; ++x) {
        const u32 i = threadIdx.x + (u32)x * T;
        if (i >= M) continue;
        const u32 u = vo[i], p = A.part[u] - base, q = A.target[u] - base;
        nd[x] = u;
        key[x] = (((p < q ? p : q) * A.k + (p < q ? q : p)) << 1) | (p < q ? 0u : 1u);
    }
    __syncthreads();
#pragma unroll
    for (int x = 0; x < RSS_ITEMS; ++x) {
        const u32 i = threadIdx.x + (u32)x * T;
        if (i < M) { sm[i] = key[x]; sm[RSS_CAP + i] = nd[x]; }
    }
    block_radix_sort(sm, M, A.gb, ko, vo);
    // partners: the i-th move of a group and the i-th of the opposite one. fl[j] counts the moves
    // that follow the group order at position j: both of a pair at its first direction's position.
    u32 pk[RSS_ITEMS];  // a paired second direction's partner position, else NONE
    i64 ps[RSS_ITEMS];
    u32 *fl = const_cast<u32 *>(ko == sm ? sm + 2 * RSS_CAP : sm);  // the buffers not holding (ko, vo)
#pragma unroll
    for (int x = 0; x < RSS_ITEMS; ++x) {
        const u32 j = threadIdx.x + (u32)x * T;
        if (j >= M) continue;
        const u32 g = ko[j], d = g & 1u, u = vo[j];
        const u32 i = j - lower_bound_u32(ko, M, g);
        const u32 s2 = lower_bound_u32(ko, M, g ^ 1u), e2 = lower_bound_u32(ko, M, (g ^ 1u) + 1u);
        nd[x] = u;
        ps[x] = A.gain[u];
        pk[x] = NONE;
        u32 f = 1;
        if (i < e2 - s2) {
            ps[x] += A.gain[vo[s2 + i]];
            if (d) pk[x] = s2 + i;
            f = d ? 0u : 2u;
        }
        fl[j] = f;
    }
    __syncthreads();
    // exclusive prefix of fl in place: a move's place by (pair position, direction)
    {
        u32 run = 0;
        for (u32 b = 0; b < M; b += T) {
            const u32 j = b + threadIdx.x;
            const u32 f = j < M ? fl[j] : 0u;
            i64 tot;
            const i64 incl = block_incl_scan_i64((i64)f, sh, tot);
            if (j < M) fl[j] = run + (u32)incl - f;
            run += (u32)tot;
        }
    }
    __syncthreads();
    u32 at[RSS_ITEMS];
#pragma unroll
    for (int x = 0; x < RSS_ITEMS; ++x) {
        const u32 j = threadIdx.x + (u32)x * T;
        if (j < M) at[x] = pk[x] != NONE ? fl[pk[x]] + 1 : fl[j];
    }
    __syncthreads();
#pragma unroll
    for (int x = 0; x < RSS_ITEMS; ++x) {
        const u32 j = threadIdx.x + (u32)x * T;
        if (j >= M) continue;
        sm[at[x]] = (u32)(A.pbound - (u64)ps[x]);
        sm[RSS_CAP + at[x]] = nd[x];
        if (A.pb > 32) A.psn[nd[x]] = ps[x];
    }
    __syncthreads();
    copy_sort64(sm, M, A.pb, ko, vo, [&](u32 v) { return (u32)((A.pbound - (u64)A.psn[v]) >> 32); });
    for (u32 i = threadIdx.x; i < M; i += T) {
        const u32 v = vo[i];
        A.mv[v0 + i] = v;
        A.state[v].x = i;
    }
    if (threadIdx.x == 0) {
        A.dM[t] = M;
        if (t == 0) *A.apply = 0;
    }
}

// Size violations of every prefix: one block per partition of every copy runs its size along the
// copy's movers; vs[r] += excess(after rank r) - excess(before).
constexpr u32 CV_SIZE_THREADS = 512;
__global__ void __launch_bounds__(CV_SIZE_THREADS) k_copy_sizes(CopyArgs A) {
    __shared__ i64 sh[32];
    const u32 p = blockIdx.x, t = p / A.k, v0 = t * A.cn, M = A.dM[t];
    i64 run = (i64)A.psize[p];
    const i64 om = (i64)A.omega;
    for (u32 b = 0; b < M; b += CV_SIZE_THREADS) {
        const u32 r = b + threadIdx.x;
        i64 d = 0;
        if (r < M) {
            const u32 v = A.mv[v0 + r];
            if (A.part[v] == p) d = -(i64)A.nsize[v];
            else if (A.target[v] == p) d = (i64)A.nsize[v];
        }
        if (!__syncthreads_or(d != 0)) continue;
        i64 tot;
        const i64 incl = block_incl_scan_i64(d, sh, tot);
        if (d != 0) {
            const i64 after = run + incl, before = after - d;
            const i64 dx = (after > om ? after - om : 0) - (before > om ? before - om : 0);
            if (dx) atomicAdd((unsigned long long *)&A.vs[v0 + r], (unsigned long long)dx);
        }
        run += tot;
    }
}

// The best prefix of every copy and its application, one block each; the partition sizes follow.
__global__ void __launch_bounds__(1024) k_copy_tail(CopyArgs A) {
    __shared__ i64 sh[32];
    __shared__ Best bsh[32];
    __shared__ Best s_best;
    __shared__ int dlo[KW_K], dhi[KW_K];  // size changes in units of 1 and 2^16: at most RSS_CAP terms each
    const u32 t = blockIdx.x, v0 = t * A.cn, base = t * A.k, M = A.dM[t];
    const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_best = Best{0, 0, 0, 0xFFFFFFFFu};
    for (u32 i = threadIdx.x; i < A.k; i += blockDim.x) dlo[i] = dhi[i] = 0;
    i64 rg = 0, rs = 0;
    for (u32 b0 = 0; b0 < M; b0 += blockDim.x) {
        const u32 r = b0 + threadIdx.x;
        const bool in = r < M;
        i64 tg, ts;
        const i64 pg = rg + block_incl_scan_i64(in ? (i64)A.g2[A.mv[v0 + r]] : 0, sh, tg);
        const i64 ps = rs + block_incl_scan_i64(in ? A.vs[v0 + r] : 0, sh, ts);
        const Best b = warp_best_prefix(Best{1u, ps, pg, in ? r : 0xFFFFFFFFu});
        if (lane == 0) bsh[w] = b;
        __syncthreads();
        if (w == 0) {
            const Best x = warp_best_prefix(bsh[lane]);
            if (lane == 0) s_best = best_pick(s_best, x);
        }
        rg += tg;
        rs += ts;
    }
    __syncthreads();
    const Best x = s_best;
    const bool ok = x.r != 0xFFFFFFFFu && x.vs <= 0 && x.g >= 0;
    if (threadIdx.x == 0) {
        A.applied[t] = ok ? x.r + 1 : 0u;
        if (ok) *A.apply = 1u;
    }
    if (!ok) return;
    for (u32 i = threadIdx.x; i <= x.r; i += blockDim.x) {
        const u32 v = A.mv[v0 + i], p = A.part[v] - base, q = A.target[v] - base, s = A.nsize[v];
        A.part[v] = base + q;
        atomicAdd(&dlo[p], -(int)(s & 0xFFFFu));
        atomicAdd(&dlo[q], (int)(s & 0xFFFFu));
        if (s >> 16) {
            atomicAdd(&dhi[p], -(int)(s >> 16));
            atomicAdd(&dhi[q], (int)(s >> 16));
        }
    }
    __syncthreads();
    for (u32 i = threadIdx.x; i < A.k; i += blockDim.x)
        A.psize[base + i] = (u64)((i64)A.psize[base + i] + (i64)dlo[i] + ((i64)dhi[i] << 16));
}

// ------------------------------------------------------------------ all rounds of a small level
// Inbound-constrained levels of at most RSS_CAP nodes, VS_MAX_K partitions and CM_LEN pins per
// hyperedge: every round of the level in one cooperative launch. Such a round is a handful of
// microseconds per phase, and as launches it was bound by their number and by capturing and
// instantiating a graph per level. The phases are those of round_body on a small level, a grid
// barrier apart; ranking and the best prefix run on block 0. What a phase accumulates into is
// cleared by the phase that reads it last.
constexpr u32 SR_THREADS = 1024;
constexpr u32 SR_STAGE = 256;  // pins a warp of the cascade stages
constexpr size_t SR_SMEM = RSS_SMEM;
static_assert(SR_SMEM >= (size_t)SR_THREADS / 32 * SR_STAGE * 12 && SR_SMEM >= (size_t)SR_THREADS / 32 * 2 * CD_K * 4 &&
                  SR_SMEM >= (size_t)SR_THREADS / 32 * 32 * (2 * 8 + 1) * 4 + 8 * 32 * 12 + 1024 && CM_LEN <= SR_STAGE &&
                  VS_THREADS == SR_THREADS,
              "every phase's shared state fits the launch");
struct SmallArgs {
    CensusArgs C;
    GainArgs G;
    CascadeArgs D;
    MoverArgs V;
    u32 R, kb;
    u64 gbound;
    u32 *mv, *dM;
    uint2 *state;
    unsigned long long *Vs, *Vi;
    u32 *part;
    u64 *psize, *pinb;
    i64 *save;
    u32 *rs;     // [0] round, [1] rounds done, [2] go on
    int track;
};

// Bound by its grid barriers. Measured: 8 x 512 network 12.0 ms with a graph of some 40 launches a
// round, 10.0; 4 x 64 6.5 and 3.5.
template <u32 MW>
__global__ void __launch_bounds__(SR_THREADS) k_small_rounds(SmallArgs S) {
    cg::grid_group grid = cg::this_grid();
    extern __shared__ __align__(16) u32 sr_sm[];
    __shared__ u32 s_pinb[CD_K];
    constexpr u32 NW = SR_THREADS / 32;
    const u32 w = threadIdx.x >> 5, lane = threadIdx.x & 31u, K = S.G.K, n = S.G.n;
    const u32 warp = blockIdx.x * NW + w, warps = gridDim.x * NW;
    const u32 R = S.R;
    for (u32 round = 0;;) {
        // 1. census, savings and masks; the partitions' inbound counts
        for (u32 i = threadIdx.x; i < K; i += SR_THREADS) s_pinb[i] = 0;
        __syncthreads();
        {
            u32 *cnt = sr_sm + w * 2 * CD_K, *dcnt = cnt + CD_K;
            for (u32 h = warp; h < S.D.e; h += warps) {
                const u64 a = S.C.off[h], b = S.C.off[h + 1], s = a + S.C.nsrc[h];
                for (u32 i = lane; i < K; i += 32) { cnt[i] = 0; dcnt[i] = 0; }
                __syncwarp();
                cd_count(S.C, a, b, s, cnt, dcnt, lane, 32);
                __syncwarp();
                cd_save(S.C, h, a, b, cnt, lane, 32);
                cd_emit(S.C, h, a, cnt, dcnt, K);
                for (u32 q = lane; q < K; q += 32)
                    if (dcnt[q]) atomicAdd(&s_pinb[q], 1u);
                __syncwarp();
            }
        }
        __syncthreads();
        for (u32 i = threadIdx.x; i < K; i += SR_THREADS)
            if (s_pinb[i]) atomicAdd((unsigned long long *)&S.pinb[i], (unsigned long long)s_pinb[i]);
        grid.sync();
        // 2. gains: a warp per node, or a block per node where the nodes are few
        GainArgs A = S.G;
        A.discount = round < R / 3 ? 1u : (round < 2 * R / 3 ? 2u : 0xFFFFFFFFu);
        A.round = round;
        {
            u32(*sm)[MW] = (u32(*)[MW])(sr_sm + w * 32 * (2 * MW + 1)), (*sd)[MW] = sm + 32;
            u32 *sw = (u32 *)(sd + 32);
            u32 *rest = sr_sm + NW * 32 * (2 * MW + 1);
            if (n > warps / 2) {
                for (u32 u = warp; u < n; u += warps) {
                    MaskAcc<MW> acc;
#pragma unroll
                    for (u32 k = 0; k < MW; ++k) { acc.conn[k] = 0; acc.dconn[k] = 0; acc.pres[k] = 0; }
                    i64 wtot = 0;
                    gain_mask_acc<MW>(A, S.C.mask, S.C.dmask, u, 0, 32, sm, sd, sw, acc, wtot);
                    wtot = warp_sum(wtot);
                    const Cand best = mask_best<MW>(A, u, S.part[u], acc, S.save[u], wtot);
                    if (lane == 0) {
                        write_move(A, u, best);
                        S.save[u] = 0;
                    }
                }
            } else {
                unsigned long long *rc = (unsigned long long *)rest;  // [MW * 32]
                u32 *rd = (u32 *)(rc + MW * 32), *rp = rd + MW * 32;  // [MW * 32], [MW]
                i64 *rw = (i64 *)(rp + 8);                            // [NW]
                for (u32 u = blockIdx.x; u < n; u += gridDim.x) {
                    for (u32 i = threadIdx.x; i < MW * 32; i += SR_THREADS) { rc[i] = 0; rd[i] = 0; }
                    if (threadIdx.x < MW) rp[threadIdx.x] = 0;
                    __syncthreads();
                    MaskAcc<MW> acc;
#pragma unroll
                    for (u32 k = 0; k < MW; ++k) { acc.conn[k] = 0; acc.dconn[k] = 0; acc.pres[k] = 0; }
                    i64 wtot = 0;
                    gain_mask_acc<MW>(A, S.C.mask, S.C.dmask, u, 32 * w, SR_THREADS, sm, sd, sw, acc, wtot);
                    wtot = warp_sum(wtot);
#pragma unroll
                    for (u32 k = 0; k < MW; ++k) {
                        if (acc.conn[k]) atomicAdd(&rc[k * 32 + lane], acc.conn[k]);
                        if (acc.dconn[k]) atomicAdd(&rd[k * 32 + lane], acc.dconn[k]);
                        if (lane == 0 && acc.pres[k]) atomicOr(&rp[k], acc.pres[k]);
                    }
                    if (lane == 0) rw[w] = wtot;
                    __syncthreads();
                    if (w == 0) {
#pragma unroll
                        for (u32 k = 0; k < MW; ++k) {
                            acc.conn[k] = rc[k * 32 + lane];
                            acc.dconn[k] = rd[k * 32 + lane];
                            acc.pres[k] = rp[k];
                        }
                        wtot = 0;
                        for (u32 i = 0; i < NW; ++i) wtot += rw[i];
                        const Cand best = mask_best<MW>(A, u, S.part[u], acc, S.save[u], wtot);
                        if (lane == 0) {
                            write_move(A, u, best);
                            S.save[u] = 0;
                        }
                    }
                    __syncthreads();
                }
            }
        }
        grid.sync();
        // 3. ranks
        if (blockIdx.x == 0) {
            const u32 M = rank_small_body(sr_sm, n, A.target, A.gain, S.gbound, S.kb, S.part, S.mv, S.state, S.D.g2);
            for (u32 i = threadIdx.x; i < M; i += SR_THREADS) S.Vs[i] = S.Vi[i] = 0;
            if (threadIdx.x == 0) *S.dM = M;
        }
        grid.sync();
        const u32 M = *(volatile u32 *)S.dM;
        if (M) {
            // 4. the cascade
            {
                uint2 *st = (uint2 *)sr_sm + w * SR_STAGE;
                u32 *nd = sr_sm + NW * SR_STAGE * 2 + w * SR_STAGE;
                if (S.track) cascade_dense_body<true, SR_STAGE>(S.D, S.V, warp, warps, st, nd);
                else cascade_dense_body<false, SR_STAGE>(S.D, S.V, warp, warps, st, nd);
            }
            grid.sync();
            // 5. size and inbound validity of every prefix
            for (u32 p = blockIdx.x; p < K; p += gridDim.x)
                validity_small_body<true>(p, M, S.mv, S.part, A.target, A.nsize, S.psize, A.omega, S.Vs, S.track, S.D.tdense, n,
                                          S.pinb, A.delta, S.Vi);
            grid.sync();
        }
        // 6. the best prefix, its application, and the schedule (k_round_next)
        if (blockIdx.x == 0) {
            const u32 end = M ? tail_small_body(M, S.mv, S.D.g2, (const i64 *)S.Vs, (const i64 *)S.Vi, S.track) : 0u;
            for (u32 i = threadIdx.x; i < end; i += SR_THREADS) {
                const u32 v = S.mv[i], p = S.part[v], q = A.target[v];
                atomicAdd((unsigned long long *)&S.psize[p], 0ull - (unsigned long long)A.nsize[v]);
                atomicAdd((unsigned long long *)&S.psize[q], (unsigned long long)A.nsize[v]);
                S.part[v] = q;
            }
            for (u32 i = threadIdx.x; i < K; i += SR_THREADS) S.pinb[i] = 0;
            if (threadIdx.x == 0) {
                u32 x = round;
                if (!end) {
                    if (x < R / 3) x = R / 2;
                    else if (x < 2 * R / 3) x = 2 * R / 3;
                    else x = R;
                }
                x += 1;
                S.rs[0] = x;
                S.rs[1] += 1;
                S.rs[2] = x < R && *(volatile const u32 *)S.C.status == 0;
            }
        }
        grid.sync();
        if (!*(volatile u32 *)&S.rs[2]) return;
        round = *(volatile u32 *)&S.rs[0];
    }
}

GainArgs make_gain_args(const DLevel &L, const u32 *wfx, const RefineParams &rp, const Census &cs, const u32 *part,
                        const u64 *psize, const u64 *pinb, u32 discount, u32 round, u32 *target, i64 *gain,
                        u32 *status) {
    GainArgs A;
    A.n = L.n; A.omega = rp.omega; A.delta = rp.delta; A.discount = discount; A.round = round; A.K = rp.K;
    A.seed = (u32)rp.seed; A.encourage = rp.encourage ? 1 : 0;
    A.off = L.off; A.pins = L.pins; A.nsrc = L.nsrc; A.lam = cs.lam; A.cpart = cs.part; A.ccnt = cs.cnt; A.cdcnt = cs.dcnt; A.wfx = wfx;
    A.toff = L.toff; A.touch = L.touch; A.nin = L.nin; A.nsize = L.nsize; A.part = part;
    A.psize = psize; A.pinb = pinb; A.target = target; A.gain = gain; A.status = status;
    A.dyn = nullptr;
    A.save = cs.save;
    return A;
}

}  // namespace

// Work lists of one level for the census (hyperedge length tiers) and the gains (node gain-work
// bound tiers), plus the bounds that size per-round buffers. Built once per level.
struct LevelPrep {
    u32 *hblock = nullptr, n_hblock = 0;       // 256 < |e| <= 4096
    u32 *hhuge = nullptr, n_hhuge = 0;         // |e| > 4096
    u64 *huge_tab = nullptr, huge_tot = 0;     // table offsets of the huge hyperedges
    u32 *ntier[3] = {nullptr, nullptr, nullptr};
    u32 ncount[3] = {0, 0, 0};
    u64 *work = nullptr;     // per-node table bound of the gains
    u64 *wsum = nullptr;     // K > GS_K: per-node summed weights of its hyperedges
    u64 gain_bound = 0;     // no gain exceeds this (sum of incident weights)
    u64 max_len = 0;         // largest hyperedge
    u32 *hlong = nullptr, n_hlong = 0;         // |e| > CM_LEN
    uint8_t *hclass = nullptr;                 // [e] 0 for those, else 2 (k_mover_hedges)
    u64 max_deg = 0;         // largest degree
    u64 short_pins = 0, short_sq = 0;  // pins of hyperedges of at most CM_LEN pins; sum of their squared lengths
    bool uniform = false;    // every hyperedge has the weight `weight`
    u32 weight = 0;
    u64 dst_pins = 0;        // destination pins (bounds the inbound events: 2 per pin)
    u64 tier_deg[3] = {0, 0, 0};  // incidence entries of each gain tier (kernel timer only)
    u32 census_K = 0;        // nonzero: partition-indexed census over this many partitions, and
                             // hblock holds the hyperedges above CD_WARP_LEN pins
};

// Movers the cascade's block kernel keeps in shared memory: CB_MOV_MAX, or less when the context's
// tuning (c.tune.cascade_movers) or the environment variable AXC_CASCADE_BLOCK_MOVERS asks for it
// (a power of two >= 128), which sends hyperedges with more movers to the scratch kernel; the tests
// use it to reach that kernel on small inputs. Read at each level's launch.
static u32 cascade_block_movers(const Ctx &c) {
    unsigned long v = c.tune.cascade_movers;
    if (!v) {
        const char *s = std::getenv("AXC_CASCADE_BLOCK_MOVERS");
        if (!s || !*s) return CB_MOV_MAX;
        v = std::strtoul(s, nullptr, 10);
    }
    u32 lim = 128;
    while ((unsigned long)lim * 2 <= v && lim < CB_MOV_MAX) lim <<= 1;
    return lim;
}

// The incremental census is on unless the environment variable AXC_INC_CENSUS is "0" (then every
// round rebuilds the census; the same results).
static bool inc_census_enabled() {
    const char *s = std::getenv("AXC_INC_CENSUS");
    return !(s && s[0] == '0');
}

static bool round_loop_enabled() {
    const char *s = std::getenv("AXC_ROUND_LOOP");
    return !(s && s[0] == '0');
}

void setup_refine_kernels(Ctx &c) {
    AXC_CUDA(cudaFuncSetAttribute(k_census_mid<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CS_DIRECT_K * 4));
    AXC_CUDA(cudaFuncSetAttribute(k_census_mid<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * CS_BLOCK_CAP * 8));
    AXC_CUDA(cudaFuncSetAttribute(k_part_inbound_smem<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PI_SMEM_K * 4));
    AXC_CUDA(cudaFuncSetAttribute(k_part_inbound_smem<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PI_SMEM_K * 4));
    AXC_CUDA(cudaFuncSetAttribute(k_part_inbound_smem<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PI_SMEM_K * 4));
    AXC_CUDA(cudaFuncSetAttribute(k_gain_table<true, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GS_K * 12));
    AXC_CUDA(cudaFuncSetAttribute(k_gain_table<true, GN_BLOCK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GS_K * 12));
    AXC_CUDA(cudaFuncSetAttribute(k_cascade_long<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(CL_WARPS * cl_bytes(true, CC_DIRECT_BLOCK_K, CL_MOV_DIRECT))));
    AXC_CUDA(cudaFuncSetAttribute(k_cascade_long<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(CL_WARPS * cl_bytes(false, 0, CL_MOV_HASH))));
    AXC_CUDA(cudaFuncSetAttribute(k_cascade_wide<CW_SWEEP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)cw_bytes(CW_SWEEP, CW_SWEEP_K, cw_movers(CW_SWEEP))));
    AXC_CUDA(cudaFuncSetAttribute(k_cascade_wide<CW_EVENTS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)cw_bytes(CW_EVENTS, CC_DIRECT_BLOCK_K, cw_movers(CW_EVENTS))));
    AXC_CUDA(cudaFuncSetAttribute(k_cascade_wide<CW_HASH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)cw_bytes(CW_HASH, 0, cw_movers(CW_HASH))));
    AXC_CUDA(cudaFuncSetAttribute(k_cascade_block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CB_DYN_MAX));
    AXC_CUDA(cudaFuncSetAttribute(k_gain_sample<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GS_DIRECT_UNI * 4));
    AXC_CUDA(cudaFuncSetAttribute(k_gain_sample<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GS_TAB * 8));
    AXC_CUDA(cudaFuncSetAttribute(k_gain_sample<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GS_DIRECT_GEN * 8));
    AXC_CUDA(cudaFuncSetAttribute(k_gain_sample<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GS_TAB * 12));
    AXC_CUDA(cudaFuncSetAttribute(k_cands_block<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CV_BLOCK_SMEM));
    AXC_CUDA(cudaFuncSetAttribute(k_rank_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RSS_SMEM));
    AXC_CUDA(cudaFuncSetAttribute(k_copy_rank, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RSS_SMEM));
    AXC_CUDA(cudaFuncSetAttribute(k_small_rounds<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SR_SMEM));
    AXC_CUDA(cudaFuncSetAttribute(k_small_rounds<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SR_SMEM));
    AXC_CUDA(cudaFuncSetAttribute(k_small_rounds<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SR_SMEM));
    AXC_CUDA(cudaFuncSetAttribute(k_small_rounds<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SR_SMEM));
}

// The level's hyperedge lists and bounds in one pass; dc as in prepare_level: the lists of lo < |e| <=
// hi pins ([0]), longer ones ([1]) and those above CM_LEN ([15]), with cls their class
// (k_mover_hedges); the longest, the destination pins, the extreme weights, and the pins and squared
// lengths of the short ones ([9] to [14]).
// Measured: 1M nets 138 us, 16.
__global__ void __launch_bounds__(1024) k_level_hedges(u32 e, const u64 *__restrict__ off, const u32 *__restrict__ nsrc,
                                                       const u32 *__restrict__ wfx, u64 lo, u64 hi, u32 *mid, u32 *huge,
                                                       u32 *lng, uint8_t *__restrict__ cls, u64 *__restrict__ dc) {
    __shared__ u32 sh[33];
    const u32 h = blockIdx.x * blockDim.x + threadIdx.x;
    u64 len = 0, dst = 0, sp = 0, sq = 0;
    u32 w = 0, nw = 0;
    if (h < e) {
        len = off[h + 1] - off[h];
        dst = len - nsrc[h];
        w = wfx[h];
        nw = ~w;
        cls[h] = len > CM_LEN ? 0 : 2;
        if (len <= CM_LEN) { sp = len; sq = len * len; }
    }
    if (__syncthreads_or(len > CM_LEN)) {
        const u32 at = block_append(len > CM_LEN, (u32 *)(dc + 15), sh);
        if (len > CM_LEN) lng[at] = h;
    }
    if (__syncthreads_or(len > lo)) {
        const u32 at = block_append(len > lo && len <= hi, (u32 *)(dc + 0), sh);
        if (len > lo && len <= hi) mid[at] = h;
        if (__syncthreads_or(len > hi)) {
            const u32 ah = block_append(len > hi, (u32 *)(dc + 1), sh);
            if (len > hi) huge[ah] = h;
        }
    }
    // one atomic per block and word: one per warp met at six addresses
    __shared__ u64 red[6][32];
    const u32 lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const auto reduce = [&]() {
        len = warp_max_u64(len);
        dst = warp_sum(dst);
        sp = warp_sum(sp);
        sq = warp_sum(sq);
        w = __reduce_max_sync(0xFFFFFFFFu, w);
        nw = __reduce_max_sync(0xFFFFFFFFu, nw);
    };
    reduce();
    if (lane == 0) {
        red[0][wp] = len;
        red[1][wp] = dst;
        red[2][wp] = sp;
        red[3][wp] = sq;
        red[4][wp] = w;
        red[5][wp] = nw;
    }
    __syncthreads();
    if (wp) return;
    len = red[0][lane];  // 32 warps
    dst = red[1][lane];
    sp = red[2][lane];
    sq = red[3][lane];
    w = (u32)red[4][lane];
    nw = (u32)red[5][lane];
    reduce();
    if (lane == 0) {
        unsigned long long *out = (unsigned long long *)dc;
        if (len) atomicMax(&out[9], (unsigned long long)len);
        if (dst) atomicAdd(&out[10], (unsigned long long)dst);
        if (w) atomicMax(&out[11], (unsigned long long)w);
        if (nw) atomicMax(&out[12], (unsigned long long)nw);
        if (sp) atomicAdd(&out[13], (unsigned long long)sp);
        if (sq) atomicAdd(&out[14], (unsigned long long)sq);
    }
}

// Everything the level's rounds need sized on the host comes back in one round trip (a second
// one only when some hyperedge is longer than CS_BLOCK_CAP).
// kway: the level's rounds take the k-way records (no census lists; two gain tiers, by degree).
static LevelPrep prepare_level(Ctx &c, const DLevel &L, const u32 *wfx, u32 K, bool kway = false) {
    LevelPrep lp;
    const u32 e = L.e, n = L.n;
    // [0] census block list, [1] census huge list, [2..4] node tiers, [5] gain bound,
    // [6] largest work, [7] largest block-tier work, [8] largest degree, [9] largest hyperedge,
    // [10] destination pins, [11] largest weight, [12] complement of the smallest, [13] pins of short
    // hyperedges, [14] the sum of their squared lengths, [15] hyperedges above CM_LEN pins
    u64 *dc = c.arena.alloc<u64>(16);
    AXC_CUDA(cudaMemsetAsync(dc, 0, 128, c.stream));
    lp.census_K = K <= CD_K || kway ? K : 0;
    if (n) {
        lp.work = c.arena.alloc<u64>(n);
        for (u32 t = 0; t < (kway ? 2u : 3u); ++t) lp.ntier[t] = c.arena.alloc<u32>(n);
    }
    // what the counts may show to be needless comes last, and is given back then
    const size_t before_wsum = c.arena.mark();
    if (n && K > GS_K) lp.wsum = c.arena.alloc<u64>(n);
    const size_t before_lists = c.arena.mark();
    size_t before_long = before_lists;
    if (e) {
        // census: a warp, a block above CD_WARP_LEN pins (partition-indexed) or CS_WARP_CAP (hashed),
        // and hashed above CS_BLOCK_CAP a table in device memory
        lp.hclass = c.arena.alloc<uint8_t>(e);
        lp.hblock = c.arena.alloc<u32>(e);
        if (!lp.census_K) lp.hhuge = c.arena.alloc<u32>(e);
        before_long = c.arena.mark();
        lp.hlong = c.arena.alloc<u32>(e);
        static_assert(CM_LEN <= CS_WARP_CAP && CM_LEN <= CD_WARP_LEN, "no long hyperedges: the other lists are empty too");
        LAUNCH(c, k_level_hedges, cdiv(e, 1024), 1024, 0, e, L.off, L.nsrc, wfx, lp.census_K ? (u64)CD_WARP_LEN : (u64)CS_WARP_CAP,
               lp.census_K ? ~0ull : (u64)CS_BLOCK_CAP, lp.hblock, lp.hhuge, lp.hlong, lp.hclass, dc);
    }
    if (n) {
        const auto bounds = [&](auto g) {  // lanes per node: as many as a mean node has incidences
            constexpr u32 G = decltype(g)::value;
            LAUNCH_AS(c, "k_gain_bounds", k_gain_bounds<G>, cdiv((u64)n * G, 256), 256, 0, n, K, L.toff, L.touch, L.off, wfx,
                      lp.work, lp.wsum, (unsigned long long *)(dc + 5));
        };
        if (L.P < 8ull * n) bounds(std::integral_constant<u32, 4>());
        else if (L.P < 32ull * n) bounds(std::integral_constant<u32, 8>());
        else bounds(std::integral_constant<u32, 32>());
        LAUNCH(c, k_tier_lists, cdiv(n, 1024), 1024, 0, n, K, lp.work, L.toff, kway ? 1u : 0u, lp.ntier[0], lp.ntier[1],
               lp.ntier[2], dc + 2, (unsigned long long *)(dc + 6));
    }
    u64 h[16];
    fetch(c, h, dc, 128);
    lp.n_hblock = (u32)h[0];
    lp.n_hhuge = (u32)h[1];
    for (int t = 0; t < 3; ++t) lp.ncount[t] = (u32)h[2 + t];
    lp.gain_bound = h[5];
    lp.max_deg = h[8];
    lp.max_len = h[9];
    lp.dst_pins = h[10];
    lp.short_pins = h[13];
    lp.short_sq = h[14];
    lp.n_hlong = (u32)h[15];
    if (lp.n_hlong) {
        c.arena.release(before_long);
        lp.hlong = c.arena.alloc<u32>(lp.n_hlong);  // same address, tighter size
    } else {
        lp.hclass = nullptr;
        lp.hblock = lp.hhuge = lp.hlong = nullptr;
        if (!lp.ncount[2]) lp.wsum = nullptr;
        c.arena.release(lp.wsum ? before_lists : before_wsum);
    }
    if (e && (u32)h[11] == ~(u32)h[12]) {
        lp.uniform = true;
        lp.weight = (u32)h[11];
    }
    if (lp.n_hhuge) {
        lp.huge_tab = c.arena.alloc<u64>(lp.n_hhuge + 1);
        LAUNCH(c, k_tab_sizes, cdiv(lp.n_hhuge + 1, 256), 256, 0, lp.hhuge, lp.n_hhuge, L.off, lp.huge_tab);
        scan_excl_u64(c, lp.huge_tab, lp.huge_tab, lp.n_hhuge + 1);
        lp.huge_tot = fetch1(c, lp.huge_tab + lp.n_hhuge);
    }
    if (n) {
        if (c.prof_on && (c.prof_name.find("gain") != std::string::npos || c.prof_name.find("k_kway") == 0)) {
            unsigned long long *dg = c.arena.alloc<unsigned long long>(3);
            AXC_CUDA(cudaMemsetAsync(dg, 0, 24, c.stream));
            for (int t = 0; t < 3; ++t)
                LAUNCH(c, k_list_degree, cdiv(lp.ncount[t], 256), 256, 0, lp.ntier[t], lp.ncount[t], L.toff, dg + t);
            fetch(c, lp.tier_deg, dg, 24);
        }
    }
    return lp;
}

// Longest hyperedge a block-tier table must hold: the level's longest, capped by the tier's bound
// (the bound itself when the level's is not known).
static u64 block_tier_len(const LevelPrep &lp, u64 bound) { return lp.max_len && lp.max_len < bound ? lp.max_len : bound; }

// K: partition ids are below it (~0 when no bound is known).
static void run_census(Ctx &c, const DLevel &L, const LevelPrep &lp, const u32 *part, u32 K, Census &cs) {
    cs.beg = L.off;
    if (L.e == 0) return;
    CensusArgs A{L.off, L.pins, L.nsrc, part, cs.part, cs.cnt, cs.dcnt, cs.lam, c.d_status,
                 (unsigned long long *)cs.save, cs.wfx, cs.encourage, nullptr, nullptr, 0, nullptr};
    if (c.profiling("k_census_direct_warp")) A.pbytes = c.d_prof_bytes();
    if (lp.census_K) {
        A.mask = cs.mask;  // masks come with the partition-indexed census
        A.dmask = cs.dmask;
        A.mw = cs.mw;
        LAUNCH(c, k_census_direct_warp, cdiv(L.e, CS_WARPS), CS_WARPS * 32, 0, L.e, A, lp.census_K);
        if (lp.n_hblock)
            LAUNCH(c, k_census_direct_block, lp.n_hblock, 256, 0, lp.hblock, lp.n_hblock, A, lp.census_K);
        return;
    }
    // hyperedges a warp looks at: fewer where the mean length leaves it many pins each
    u32 per = 32;
    while (per > 2 && (L.P / L.e * per > 1024 || L.e / per < (u32)c.sms * 16)) per >>= 1;
    LAUNCH(c, k_census_short, std::min<u32>(cdiv(L.e, (CS_THREADS / 32) * per), (u32)c.sms * 8), CS_THREADS, 0, L.e, A, per);
    if (!lp.max_len || lp.max_len > CS_SHORT)
        LAUNCH(c, k_census_warp, cdiv(L.e, CS_WARPS * per), CS_WARPS * 32, 0, L.e, A, per);
    if (lp.n_hblock) {
        const bool direct = K <= CS_DIRECT_K;
        const u32 T = direct ? K : cs_cap(block_tier_len(lp, CS_BLOCK_CAP));
        const size_t smem = (size_t)T * (direct ? 4 : 8);
        const auto launch = [&](auto kernel) {
            int per_sm = 1;
            AXC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, CS_THREADS, smem));
            LAUNCH_AS(c, "k_census_mid", kernel, std::min<u32>(lp.n_hblock, (u32)c.sms * (u32)std::max(per_sm, 1)),
                      CS_THREADS, smem, lp.hblock, lp.n_hblock, A, T);
        };
        if (direct) launch(k_census_mid<true>);
        else launch(k_census_mid<false>);
    }
    if (lp.n_hhuge) {
        size_t m = c.arena.mark();
        u32 *gtab = c.arena.alloc<u32>(4 * lp.huge_tot);
        LAUNCH(c, k_census_block, lp.n_hhuge, 512, 0, lp.hhuge, lp.n_hhuge, A, gtab, (const u64 *)lp.huge_tab);
        c.arena.release(m);
    }
}

static Census alloc_census(Ctx &c, const DLevel &L) {
    Census cs;
    cs.beg = L.off;
    cs.part = c.arena.alloc<u32>(L.P ? L.P : 1);
    cs.cnt = c.arena.alloc<u32>(L.P ? L.P : 1);
    cs.dcnt = c.arena.alloc<u32>(L.P ? L.P : 1);
    cs.lam = c.arena.alloc<u32>(L.e ? L.e : 1);
    return cs;
}

// Algorithmic bytes of one gains launch over a node list: 8 per incidence entry (the touching id
// and the census reads of the node's own and the candidate partitions) and 16 per node (its
// move, gain and rank).
static u64 gain_bytes(const LevelPrep &lp, int t) { return 8 * lp.tier_deg[t] + 16 * (u64)lp.ncount[t]; }

template <u32 MW>
static void run_gains_masked(Ctx &c, const LevelPrep &lp, const GainArgs &A, const Census &cs) {
    if (lp.ncount[0])
        LAUNCH(c, k_gain_mask_warp<MW>, cdiv(lp.ncount[0], GN_WARPS), GN_WARPS * 32, 0, A, lp.ntier[0], lp.ncount[0],
               cs.mask, cs.dmask);
    if (lp.ncount[1])
        LAUNCH(c, k_gain_mask_block<MW>, lp.ncount[1], GN_BLOCK, 0, A, lp.ntier[1], lp.ncount[1], cs.mask, cs.dmask);
}

// Lanes per incidence of k_gain_planes at K partitions: the power of two from its mask words up.
static u32 plane_lanes(u32 K) {
    u32 l = 16;
    while (32 * l < K) l <<= 1;
    return l;
}
// Plane gains: equal weights, a block tier at GN_DIRECT_K < K <= GS_K, counters that hold the
// largest degree, and hyperedges of at least as many pins as mask words on average. A node's work is
// then its incidences times K / 32 words against (at most) times their census entries.
static bool plane_gains(const DLevel &L, const LevelPrep &lp, u32 K) {
    if (!lp.uniform || !lp.ncount[1] || K <= GN_DIRECT_K || K > GS_K || !L.e) return false;
    const u32 lanes = plane_lanes(K), S = GN_BLOCK / lanes, rows = lanes < 32 ? 32 / lanes : 1;
    return (lp.max_deg / S + 1) * rows < (1u << GP_PLANES) && L.P / L.e >= (K + 31) / 32;
}

static void run_gains(Ctx &c, const DLevel &L, const LevelPrep &lp, const GainArgs &A, const Census &cs) {
    if (cs.mask) {  // partition-indexed gains (K <= GN_DIRECT_K); their two tiers write every node
        if (c.profiling("k_gain_mask_warp")) c.prof_bytes += gain_bytes(lp, 0);
        if (c.profiling("k_gain_mask_block")) c.prof_bytes += gain_bytes(lp, 1);
        switch (cs.mw) {
            case 1: run_gains_masked<1>(c, lp, A, cs); break;
            case 2: run_gains_masked<2>(c, lp, A, cs); break;
            case 4: run_gains_masked<4>(c, lp, A, cs); break;
            default: run_gains_masked<8>(c, lp, A, cs); break;
        }
        return;
    }
    fill_u32(c, A.target, NONE, L.n);
    if (c.profiling("k_gain_warp") && lp.ncount[0]) c.prof_bytes += gain_bytes(lp, 0);
    if (lp.gain_bound < (1ull << 32))
        LAUNCH_AS(c, "k_gain_warp", k_gain_warp<false>, cdiv(lp.ncount[0], GN_WARPS), GN_WARPS * 32, 0, A, lp.ntier[0],
                  lp.ncount[0], lp.work);
    else
        LAUNCH_AS(c, "k_gain_warp", k_gain_warp<true>, cdiv(lp.ncount[0], GN_WARPS), GN_WARPS * 32, 0, A, lp.ntier[0],
                  lp.ncount[0], lp.work);
    if (lp.ncount[1] && plane_gains(L, lp, A.K)) {
        const size_t m = c.arena.mark();
        const u32 MW = (A.K + 31) / 32;
        u32 *mask = c.arena.alloc<u32>((u64)L.e * MW), *dmask = c.arena.alloc<u32>((u64)L.e * MW);
        LAUNCH(c, k_census_masks_wide, cdiv(L.e, 4), 128, 0, L.e, L.off, cs.lam, cs.part, cs.dcnt, MW, mask, dmask);
        const auto launch = [&](auto lanes) {
            LAUNCH_AS(c, "k_gain_planes", k_gain_planes<decltype(lanes)::value>, lp.ncount[1], GN_BLOCK, 0, A,
                      lp.ntier[1], lp.ncount[1], mask, dmask, MW, lp.weight);
        };
        switch (plane_lanes(A.K)) {
            case 16: launch(std::integral_constant<u32, 16>()); break;
            case 32: launch(std::integral_constant<u32, 32>()); break;
            case 64: launch(std::integral_constant<u32, 64>()); break;
            default: launch(std::integral_constant<u32, 128>()); break;
        }
        c.arena.release(m);
    } else if (lp.ncount[1] && A.K <= GS_K) {
        const auto launch = [&](auto wide, auto threads) {
            constexpr bool W = decltype(wide)::value;
            constexpr u32 NT = decltype(threads)::value;
            LAUNCH_AS(c, "k_gain_table", (k_gain_table<W, NT>), lp.ncount[1], NT, (size_t)A.K * (W ? 12 : 8), A,
                      lp.ntier[1], lp.ncount[1]);
        };
        const bool wide = lp.gain_bound >= (1ull << 32), small = L.P / L.n <= 256 && lp.max_deg <= GT_SMALL_DEG;
        const std::integral_constant<u32, 64> t64;
        const std::integral_constant<u32, GN_BLOCK> t256;
        if (wide && small) launch(std::true_type(), t64);
        else if (wide) launch(std::true_type(), t256);
        else if (small) launch(std::false_type(), t64);
        else launch(std::false_type(), t256);
    }
    if (A.K > GS_K && lp.ncount[1] + lp.ncount[2]) {  // the sampled rule (include/axc.h AXC_SPARSE_GAIN_*)
        size_t m = c.arena.mark();
        const u32 rows = lp.ncount[2];
        CandAcc C{nullptr, nullptr, nullptr, lp.wsum, lp.weight};
        if (rows) {  // tier 1 has no candidates: its nodes' samples are the whole nodes
            C.cand = c.arena.alloc<u32>((u64)L.n * GS_C);
            C.conn = c.arena.alloc<unsigned long long>((u64)L.n * GS_C);
            if (!lp.uniform) C.dcon = c.arena.alloc<u32>((u64)L.n * GS_C);
            AXC_CUDA(cudaMemsetAsync(C.cand, 0xFF, (size_t)L.n * GS_C * 4, c.stream));  // NONE
        }
        u32 *room = c.arena.alloc<u32>(A.K);
        LAUNCH(c, k_part_room, cdiv(A.K, 256), 256, 0, A.K, A.omega, A.delta, A.psize, A.pinb, room);
        const auto sample = [&](auto uni, auto direct) {
            constexpr bool U = decltype(uni)::value, D = decltype(direct)::value;
            const u32 T = D ? (A.K + 3) & ~3u : GS_TAB;
            const size_t smem = (size_t)T * 4 * ((U ? 1 : 2) + (D ? 0 : 1));
            int per_sm = 1;
            AXC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gain_sample<U, D>, GS_BLOCK, smem));
            // tier 1: nodes whose bound fits the sample are settled exactly
            for (u32 t = 1; t <= 2; ++t)
                LAUNCH_AS(c, "k_gain_sample", (k_gain_sample<U, D>),
                          std::min<u32>(lp.ncount[t], (u32)c.sms * (u32)std::max(per_sm, 1)), GS_BLOCK, smem, A, lp.ntier[t],
                          lp.ncount[t], C, T, lp.weight, room);
        };
        const std::true_type yes;
        const std::false_type no;
        if (lp.uniform && A.K <= GS_DIRECT_UNI) sample(yes, yes);
        else if (lp.uniform) sample(yes, no);
        else if (A.K <= GS_DIRECT_GEN) sample(no, yes);
        else sample(no, no);
        const auto exact = [&](auto bitmaps) {
            constexpr bool B = decltype(bitmaps)::value;
            const u32 mw = (A.K + 31) / 32;
            const size_t ws = B ? (size_t)CV_WARPS * 2 * mw * 4 : (size_t)CV_WARPS * 4 * CV_WARP_LEN * 4;
            int per_sm = 1;
            AXC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cands_warp<B>, CV_WARPS * 32, ws));
            LAUNCH_AS(c, "k_cands_warp", k_cands_warp<B>,
                      std::min<u32>(cdiv(L.e, CV_WARPS), (u32)c.sms * (u32)std::max(per_sm, 1)), CV_WARPS * 32, ws, A, C,
                      L.e, mw);
            const size_t bs = B ? (size_t)2 * mw * 4 : 8 * (size_t)cs_cap(block_tier_len(lp, CV_BLOCK_LEN));
            if (lp.n_hblock)
                LAUNCH_AS(c, "k_cands_block", k_cands_block<B>, lp.n_hblock, CV_BLOCK, bs, A, C, lp.hblock, lp.n_hblock,
                          mw, (u32 *)nullptr, (const u64 *)nullptr);
            if (lp.n_hhuge) {
                u32 *gtab = B ? nullptr : c.arena.alloc<u32>(2 * lp.huge_tot);
                LAUNCH_AS(c, "k_cands_block", k_cands_block<B>, lp.n_hhuge, CV_BLOCK, B ? bs : 0, A, C, lp.hhuge,
                          lp.n_hhuge, mw, gtab, (const u64 *)lp.huge_tab);
            }
        };
        if (rows && A.K <= CV_BITS_K) exact(yes);
        else if (rows) exact(no);
        LAUNCH(c, k_cands_best, cdiv(rows, 256), 256, 0, A, C, lp.ntier[2], rows);
        c.arena.release(m);
    }
}

__global__ void k_copy_conn(u64 eS, u32 e2, const u32 *__restrict__ lam, const u32 *__restrict__ wfxS,
                            unsigned long long *__restrict__ conn) {
    const u64 h = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= eS) return;
    const u32 l = lam[h];
    if (l > 1) atomicAdd(&conn[h / e2], (unsigned long long)wfxS[h] * (l - 1));
}

Census build_census(Ctx &c, const DLevel &L, const u32 *part, u32 K) {
    Census cs = alloc_census(c, L);
    size_t m = c.arena.mark();
    LevelPrep lp;
    if (L.e) {
        lp.hblock = c.arena.alloc<u32>(L.e);
        lp.hhuge = c.arena.alloc<u32>(L.e);
        u32 *cnt = c.arena.alloc<u32>(2);
        AXC_CUDA(cudaMemsetAsync(cnt, 0, 8, c.stream));
        LAUNCH(c, k_census_lists, cdiv(L.e, 1024), 1024, 0, L.e, L.off, lp.hblock, lp.hhuge, cnt);
        u64 h;
        fetch(c, &h, cnt, 8);
        lp.n_hblock = (u32)h;
        lp.n_hhuge = (u32)(h >> 32);
        if (lp.n_hhuge) {
            lp.huge_tab = c.arena.alloc<u64>(lp.n_hhuge + 1);
            LAUNCH(c, k_tab_sizes, cdiv(lp.n_hhuge + 1, 256), 256, 0, lp.hhuge, lp.n_hhuge, L.off, lp.huge_tab);
            scan_excl_u64(c, lp.huge_tab, lp.huge_tab, lp.n_hhuge + 1);
            lp.huge_tot = fetch1(c, lp.huge_tab + lp.n_hhuge);
        }
    }
    run_census(c, L, lp, part, K, cs);
    c.arena.release(m);
    return cs;
}

void part_sizes(Ctx &c, u32 n, const u32 *part, const u32 *nsize, u64 *psize, u32 K) {
    AXC_CUDA(cudaMemsetAsync(psize, 0, (size_t)K * 8, c.stream));
    if (n && K <= PS_SMEM_K) {
        const u32 rep = K <= 64 ? 32u : 1u;
        const u32 per = std::min<u32>(PS_NODES, std::max<u32>(1024, cdiv(n, (u64)c.sms * 4)));
        LAUNCH(c, k_part_sizes_smem, cdiv(n, per), 256, (size_t)2 * K * rep * 4, n, K, rep, per, part, nsize,
               (unsigned long long *)psize);
    } else if (n)
        LAUNCH(c, k_part_sizes, cdiv(n, 256), 256, 0, n, part, nsize, (unsigned long long *)psize);
}
void part_inbound(Ctx &c, const DLevel &L, const Census &cs, u64 *pinb, u32 K) {
    AXC_CUDA(cudaMemsetAsync(pinb, 0, (size_t)K * 8, c.stream));
    if (L.e && K <= PI_SMEM_K) {  // per-block counts in shared memory, one global add per partition
        const auto launch = [&](auto g) {
            constexpr u32 G = decltype(g)::value;
            LAUNCH_AS(c, "k_part_inbound_smem", k_part_inbound_smem<G>,
                      std::min<u32>(cdiv(L.e, PI_THREADS / G), (u32)c.sms), PI_THREADS, (size_t)K * 4, L.e, L.off, cs.lam,
                      cs.part, cs.dcnt, K, (unsigned long long *)pinb);
        };
        const u64 len = L.P / L.e;
        if (len <= 6) launch(std::integral_constant<u32, 4>());
        else if (len <= 24) launch(std::integral_constant<u32, 8>());
        else launch(std::integral_constant<u32, 32>());
    } else if (L.e)
        LAUNCH(c, k_part_inbound, cdiv((u64)L.e * 32, 256), 256, 0, L.e, L.off, cs.lam, cs.part, cs.dcnt,
               (unsigned long long *)pinb);
}

// Whether a round needs the partitions' inbound counts. With no inbound limit (delta 2^31 - 1,
// k-way) the inbound check pinb[q] + nin[u] - dc > delta never holds while the level has fewer
// than 2^30 hyperedges (both terms are at most e), so zero counts decide it the same way.
static bool inbound_binds(const DLevel &L, const RefineParams &rp) {
    return rp.delta < 0x7FFFFFFFu || (u64)L.e >= (1ull << 30);
}

// Mask words per hyperedge for K partitions: 1, 2, 4 or 8.
static u32 mask_words(u32 K) {
    u32 mw = 1;
    while (32 * mw < K) mw <<= 1;
    return mw;
}

// The round's census, with the extras of the partition-indexed gains when K <= GN_DIRECT_K:
// each node's saving (pushed by the census pass) and the per-hyperedge masks.
static Census census_for_gains(Ctx &c, const DLevel &L, const LevelPrep &lp, const u32 *wfx, const RefineParams &rp,
                               const u32 *part) {
    Census cs = alloc_census(c, L);
    const bool direct = rp.K <= GN_DIRECT_K;
    if (direct || plane_gains(L, lp, rp.K) || (rp.K > GS_K && lp.ncount[1] + lp.ncount[2])) {
        cs.save = c.arena.alloc<i64>(L.n ? L.n : 1);
        AXC_CUDA(cudaMemsetAsync(cs.save, 0, (size_t)L.n * 8, c.stream));
        cs.wfx = wfx;
        cs.encourage = rp.encourage ? 1 : 0;
    }
    if (direct) {
        cs.mw = mask_words(rp.K);
        cs.mask = c.arena.alloc<u32>((u64)(L.e ? L.e : 1) * cs.mw);
        cs.dmask = c.arena.alloc<u32>((u64)(L.e ? L.e : 1) * cs.mw);
    }
    run_census(c, L, lp, part, rp.K, cs);
    return cs;
}

void refine_gains_only(Ctx &c, const DLevel &L, const u32 *wfx, const RefineParams &rp, const u32 *part,
                       u32 discount, u32 round, u32 *target, i64 *gain) {
    size_t m = c.arena.mark();
    LevelPrep lp = prepare_level(c, L, wfx, rp.K);
    Census cs = census_for_gains(c, L, lp, wfx, rp, part);
    u64 *psize = c.arena.alloc<u64>(rp.K), *pinb = c.arena.alloc<u64>(rp.K);
    part_sizes(c, L.n, part, L.nsize, psize, rp.K);
    part_inbound(c, L, cs, pinb, rp.K);
    GainArgs A = make_gain_args(L, wfx, rp, cs, part, psize, pinb, discount, round, target, gain, c.d_status);
    run_gains(c, L, lp, A, cs);
    check_status(c);
    c.arena.release(m);
}

// The level-persistent census of the incremental rounds (k_census_inc_*), for levels with a
// partition-indexed census (K <= CD_K) that are not small.
struct IncCensus {
    Census cs;              // entries, counts, masks and node savings, kept across the rounds
    u32 *dirty = nullptr;   // [e] hyperedges to recompute at the next census (all before round 0)
    u32 *dlist = nullptr;   // [e] their compacted list
    u32 *prev = nullptr;    // [n] a moved node's partition before its last move
    u32 *stamp = nullptr;   // [n] the round counter at the node's last move (NONE: none)
    u32 *ctr = nullptr;     // [0] rounds run at this level, [1] the list count, [2] the warps' work
};

static bool inc_census_eligible(const DLevel &L, const LevelPrep &lp, const RefineParams &rp) {
    const bool small = rp.K <= VS_MAX_K && L.n <= (u32)RSS_CAP && rp.copies == 1;
    return lp.census_K && rp.K <= GN_DIRECT_K && !small && L.e;
}

static void inc_census_init(Ctx &c, const DLevel &L, const u32 *wfx, const RefineParams &rp, IncCensus &ic) {
    ic.cs = alloc_census(c, L);
    ic.cs.save = c.arena.alloc<i64>(L.n ? L.n : 1);
    AXC_CUDA(cudaMemsetAsync(ic.cs.save, 0, (size_t)L.n * 8, c.stream));
    ic.cs.wfx = wfx;
    ic.cs.encourage = rp.encourage ? 1 : 0;
    ic.cs.mw = mask_words(rp.K);
    ic.cs.mask = c.arena.alloc<u32>((u64)L.e * ic.cs.mw);
    ic.cs.dmask = c.arena.alloc<u32>((u64)L.e * ic.cs.mw);
    ic.dirty = c.arena.alloc<u32>(L.e);
    ic.dlist = c.arena.alloc<u32>(L.e);
    ic.prev = c.arena.alloc<u32>(L.n ? L.n : 1);
    ic.stamp = c.arena.alloc<u32>(L.n ? L.n : 1);
    ic.ctr = c.arena.alloc<u32>(4);
    fill_u32(c, ic.dirty, 1u, L.e);
    fill_u32(c, ic.stamp, NONE, L.n);
    AXC_CUDA(cudaMemsetAsync(ic.ctr, 0, 16, c.stream));
}

// The round's census in incremental form: the flagged hyperedges are listed, recomputed and
// unflagged.
static void inc_census_round(Ctx &c, const DLevel &L, const LevelPrep &lp, const u32 *part, IncCensus &ic) {
    const Census &cs = ic.cs;
    CensusArgs A{L.off, L.pins, L.nsrc, part, cs.part, cs.cnt, cs.dcnt, cs.lam, c.d_status,
                 (unsigned long long *)cs.save, cs.wfx, cs.encourage, cs.mask, cs.dmask, cs.mw, nullptr};
    if (c.profiling("k_census_inc_warp")) A.pbytes = c.d_prof_bytes();
    compact_indices_dn(c, ic.dirty, ic.dlist, L.e, ic.ctr + 1);
    AXC_CUDA(cudaMemsetAsync(ic.ctr + 2, 0, 4, c.stream));
    const IncArgs I{ic.dlist, ic.ctr + 1, ic.ctr + 2, ic.dirty, ic.prev, ic.stamp, ic.ctr};
    int per_sm = 1;
    AXC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_census_inc_warp, CS_WARPS * 32, 0));
    LAUNCH(c, k_census_inc_warp, std::min<u32>(cdiv(L.e, CS_WARPS), (u32)c.sms * (u32)std::max(per_sm, 1)),
           CS_WARPS * 32, 0, A, lp.census_K, I);
    if (lp.n_hblock) LAUNCH(c, k_census_inc_block, lp.n_hblock, 256, 0, lp.hblock, lp.n_hblock, A, lp.census_K, I);
    AXC_CUDA(cudaMemsetAsync(ic.dirty, 0, (size_t)L.e * 4, c.stream));
}

// The lanes per mover follow the level's mean degree.
template <u32 G, bool TRACK>
static void run_cascade_movers_g(Ctx &c, const CascadeArgs &C, const MoverArgs &V, u32 n, u64 max_deg) {
    LAUNCH_AS(c, "k_cascade_movers", (k_cascade_movers<G, TRACK>),
              std::min<u32>(cdiv((u64)n * G, CM_THREADS), (u32)c.sms * 8), CM_THREADS, 0, C, V);
    if (max_deg > CM_HEAVY * G)
        LAUNCH_AS(c, "k_cascade_movers_heavy", (k_cascade_movers_heavy<TRACK>), (u32)c.sms * 4, CM_THREADS, 0, C, V,
                  CM_HEAVY * G);
}
template <bool TRACK>
static void run_cascade_movers(Ctx &c, const CascadeArgs &C, const MoverArgs &V, u32 n, u64 P, u64 max_deg) {
    if (V.dense)
        LAUNCH_AS(c, "k_cascade_dense", k_cascade_dense<TRACK>,
                  std::min<u32>(cdiv(C.e, (CM_THREADS / 32) * V.per_warp), (u32)c.sms * 4), CM_THREADS, 0, C, V);
    const u64 deg = P / n;
    if (deg < 6) run_cascade_movers_g<4, TRACK>(c, C, V, n, max_deg);
    else if (deg < 12) run_cascade_movers_g<8, TRACK>(c, C, V, n, max_deg);
    else if (deg < 24) run_cascade_movers_g<16, TRACK>(c, C, V, n, max_deg);
    else run_cascade_movers_g<32, TRACK>(c, C, V, n, max_deg);
}

// The records of a level's k-way rounds (k_kway_*), kept across them.
struct KwayLevel {
    u32 k = 0, mw = 0, cn = 0, ce = 0;  // partitions, mask words, nodes and hyperedges of one copy
    u32 *rec = nullptr;                 // [e * 2 * mw]
    uint8_t *dirty = nullptr;           // [e]
    bool slots = false;                 // copies ranked by one block each (k_copy_*)
    u64 *psize = nullptr;               // [K] with slots: kept by k_copy_tail
};

// K-way rounds without an inbound limit whose copies hold at most KW_K partitions.
static bool kway_eligible(const DLevel &L, const RefineParams &rp) {
    return !rp.encourage && !inbound_binds(L, rp) && L.e && rp.K / rp.copies <= KW_K;
}

static void kway_init(Ctx &c, const DLevel &L, const RefineParams &rp, const u32 *part, KwayLevel &kw) {
    kw.k = rp.K / rp.copies;
    kw.mw = mask_words(kw.k);
    kw.cn = L.n / rp.copies;
    kw.ce = L.e / rp.copies;
    kw.slots = kw.cn <= (u32)RSS_CAP;
    kw.rec = c.arena.alloc<u32>((u64)L.e * 2 * kw.mw);
    kw.dirty = c.arena.alloc<uint8_t>(L.e);
    AXC_CUDA(cudaMemsetAsync(kw.dirty, 1, L.e, c.stream));
    if (kw.slots) {
        kw.psize = c.arena.alloc<u64>(rp.K);
        part_sizes(c, L.n, part, L.nsize, kw.psize, rp.K);
    }
}

static KwArgs kway_args(const DLevel &L, const u32 *part, const KwayLevel &kw) {
    // a lane per hyperedge where most have few pins; fewer per warp where the warp reads each
    const u64 len = L.P / L.e;
    return KwArgs{L.off, L.pins, part, L.e, kw.ce, kw.k, kw.rec, kw.dirty, len <= 2 * KW_SHORT ? 32u : len <= 64 ? 8u : 2u};
}

// Runs f(MW) for the level's mask words.
template <class F>
static void kway_words(u32 mw, F &&f) {
    switch (mw) {
        case 1: f(std::integral_constant<u32, 1>()); break;
        case 2: f(std::integral_constant<u32, 2>()); break;
        case 4: f(std::integral_constant<u32, 4>()); break;
        default: f(std::integral_constant<u32, 8>()); break;
    }
}

static void kway_records(Ctx &c, const DLevel &L, const LevelPrep &lp, const u32 *part, const KwayLevel &kw) {
    const KwArgs A = kway_args(L, part, kw);
    kway_words(kw.mw, [&](auto mw) {
        constexpr u32 MW = decltype(mw)::value;
        LAUNCH_AS(c, "k_kway_records", k_kway_records<MW>, cdiv(L.e, (KW_THREADS / 32) * A.per_warp), KW_THREADS, 0, A);
        if (lp.n_hblock)
            LAUNCH_AS(c, "k_kway_records_block", k_kway_records_block<MW>, lp.n_hblock, KW_THREADS, 0, A, lp.hblock,
                      lp.n_hblock);
    });
}

// Gains from the records. Light nodes: a group of lanes per node, at least one lane per partition
// up to 32 (at most 4 partitions: lanes side by side over the incidences, as many as the mean
// degree fills); heavy nodes and small levels: a block per node.
template <class T>
static void kway_gains_t(Ctx &c, const DLevel &L, const LevelPrep &lp, const GainArgs &A, const KwayLevel &kw) {
    KwGain V{kw.rec, kw.k, kw.cn, lp.ntier[0], lp.ncount[0], lp.uniform ? 1 : 0, lp.weight};
    // planes: merging a warp's counters costs as much as a few dozen incidences the other way
    const bool planes = lp.uniform && kw.k > 8 && L.P / L.n >= 48;
    const auto grid = [&](u32 G) { return cdiv((u64)lp.ncount[0] * G, KW_THREADS); };
    // kernel timer, per incidence: hyperedge id, a word of single pins, the present words, the weight
    // where unequal
    const auto add_bytes = [&](const char *kernel, int t) {
        if (c.profiling(kernel))
            c.prof_bytes += (8 + 4 * kw.mw + (lp.uniform ? 0 : 4)) * lp.tier_deg[t] + 16 * (u64)lp.ncount[t];
    };
    if (lp.ncount[0]) add_bytes(planes ? "k_kway_planes" : "k_kway_gain", 0);
    if (lp.ncount[0] && kw.k <= 4) {
        const u64 deg = L.P / L.n;
        if (deg < 8) LAUNCH_AS(c, "k_kway_gain", (k_kway_gain_few<4, T>), grid(4), KW_THREADS, 0, A, V);
        else if (deg < 24) LAUNCH_AS(c, "k_kway_gain", (k_kway_gain_few<8, T>), grid(8), KW_THREADS, 0, A, V);
        else if (deg < 64) LAUNCH_AS(c, "k_kway_gain", (k_kway_gain_few<16, T>), grid(16), KW_THREADS, 0, A, V);
        else LAUNCH_AS(c, "k_kway_gain", (k_kway_gain_few<32, T>), grid(32), KW_THREADS, 0, A, V);
    } else if (lp.ncount[0] && planes) {
        kway_words(kw.mw, [&](auto mw) {
            LAUNCH_AS(c, "k_kway_planes", (k_kway_planes<decltype(mw)::value, false>), cdiv(lp.ncount[0], KW_THREADS / 32),
                      KW_THREADS, 0, A, V);
        });
    } else if (lp.ncount[0]) {
        if (kw.k <= 8) LAUNCH_AS(c, "k_kway_gain", (k_kway_gain<1, 8, T>), grid(8), KW_THREADS, 0, A, V);
        else if (kw.k <= 16) LAUNCH_AS(c, "k_kway_gain", (k_kway_gain<1, 16, T>), grid(16), KW_THREADS, 0, A, V);
        else if (kw.k <= 32) LAUNCH_AS(c, "k_kway_gain", (k_kway_gain<1, 32, T>), grid(32), KW_THREADS, 0, A, V);
        else if (kw.k <= 64) LAUNCH_AS(c, "k_kway_gain", (k_kway_gain<2, 32, T>), grid(32), KW_THREADS, 0, A, V);
        else if (kw.k <= 128) LAUNCH_AS(c, "k_kway_gain", (k_kway_gain<4, 32, T>), grid(32), KW_THREADS, 0, A, V);
        else LAUNCH_AS(c, "k_kway_gain", (k_kway_gain<8, 32, T>), grid(32), KW_THREADS, 0, A, V);
    }
    if (lp.ncount[1]) {
        V.list = lp.ntier[1];
        V.nl = lp.ncount[1];
        const bool wide = planes && lp.max_deg / (KW_THREADS / 32) + 1 < (1u << KP_PLANES_BLOCK);
        add_bytes(wide ? "k_kway_planes_block" : "k_kway_gain_block", 1);
        kway_words(kw.mw, [&](auto mw) {
            if (wide)
                LAUNCH_AS(c, "k_kway_planes_block", (k_kway_planes<decltype(mw)::value, true>), lp.ncount[1], KW_THREADS, 0, A,
                          V);
            else
            LAUNCH_AS(c, "k_kway_gain_block", (k_kway_gain_block<decltype(mw)::value, T>), lp.ncount[1], KW_THREADS, 0, A,
                      V);
        });
    }
}
static void kway_gains(Ctx &c, const DLevel &L, const LevelPrep &lp, const GainArgs &A, const KwayLevel &kw) {
    if (lp.gain_bound < (1ull << 32)) kway_gains_t<u32>(c, L, lp, A, kw);
    else kway_gains_t<unsigned long long>(c, L, lp, A, kw);
}

// The launches of one round, with no host synchronization: safe to capture in a CUDA graph.
// dyn (device, optional) holds the round's discount and round number for graph replays. Returns
// the device word that says whether the moves were applied; its arena slot lies below `keep`,
// the mark the caller releases to after reading it.
static u32 *round_body(Ctx &c, const DLevel &L, const LevelPrep &lp, const u32 *wfx, const RefineParams &rp,
                       u32 *part, u32 discount, u32 round, const u32 *dyn, size_t &keep, IncCensus *ic,
                       const KwayLevel *kw) {
    const u32 n = L.n;
    const bool slots = kw && kw->slots;
    u32 *apply = c.arena.alloc<u32>(1);
    keep = c.arena.mark();
    Census cs;
    if (kw) {
        kway_records(c, L, lp, part, *kw);
    } else if (ic) {
        inc_census_round(c, L, lp, part, *ic);
        cs = ic->cs;
    } else {
        cs = census_for_gains(c, L, lp, wfx, rp, part);
    }
    u64 *psize = slots ? kw->psize : c.arena.alloc<u64>(rp.K), *pinb = kw ? nullptr : c.arena.alloc<u64>(rp.K);
    if (!slots) part_sizes(c, n, part, L.nsize, psize, rp.K);
    if (kw) {  // no inbound limit, and gains that read no inbound counts
    } else if (inbound_binds(L, rp)) {
        part_inbound(c, L, cs, pinb, rp.K);
    } else {
        AXC_CUDA(cudaMemsetAsync(pinb, 0, (size_t)rp.K * 8, c.stream));
    }
    u32 *target = c.arena.alloc<u32>(n);
    i64 *gain = c.arena.alloc<i64>(n);
    GainArgs A = make_gain_args(L, wfx, rp, cs, part, psize, pinb, discount, round, target, gain, c.d_status);
    A.dyn = dyn;
    if (kw) kway_gains(c, L, lp, A, *kw);
    else run_gains(c, L, lp, A, cs);
    // counters on the device: [0] M movers, [1] 2M size events, [2] inbound transitions,
    // [3] cascade hyperedges left by the warp kernel, [4] for the scratch kernel, [5] for the block
    // kernel's full-size launch after its middle tier, [6] holding a mover, [7] left by the wide kernel
    u32 *cnt = c.arena.alloc<u32>(8);
    AXC_CUDA(cudaMemsetAsync(cnt, 0, 32, c.stream));
    u32 *dM = cnt, *dSE = cnt + 1, *dT = cnt + 2, *dBig = cnt + 3, *dHuge = cnt + 4, *dBig2 = cnt + 5;
    u32 *dHl = cnt + 6, *dBigW = cnt + 7;  // hyperedges holding a mover; the wide kernel's leftovers
    // small levels: ranking, validity and the best prefix in one block each (SMALL_*)
    const bool small = !slots && rp.K <= VS_MAX_K && n <= (u32)RSS_CAP && rp.copies == 1;
    CopyArgs ca{};
    // movers in id order, then ranked by (gain desc, id asc)
    u32 *mv = c.arena.alloc<u32>(n);
    uint2 *state = (uint2 *)c.arena.alloc<u64>(n);
    unsigned long long *g2 = c.arena.alloc<unsigned long long>(n);  // cascaded gains, zeroed here
    u32 *ck = rp.copies > 1 && !slots ? c.arena.alloc<u32>(n) : nullptr;  // copies: the copy of every rank, ascending
    const size_t ranking = c.arena.mark();  // its scratch is given back once the movers are ranked
    u32 *flag = slots ? nullptr : c.arena.alloc<u32>(n), *klo = slots ? nullptr : c.arena.alloc<u32>(n);
    u32 *khi = flag;  // the flags are spent when the keys are made
    const u32 kb = bits_for(lp.gain_bound);
    const int packed = rp.K <= STATE_PACK_K ? 1 : 0;
    if (slots) {
        const u64 pbound = 2 * lp.gain_bound;
        u32 *dMc = c.arena.alloc<u32>(2 * (u64)rp.copies);
        ca = CopyArgs{kw->cn, kw->k, n, target, L.nsize, gain, part, lp.gain_bound, pbound, kb, bits_for(pbound),
                      bits_for(2 * (u64)kw->k * kw->k), mv, dMc, state, g2, c.arena.alloc<i64>(n),
                      c.arena.alloc<i64>(n), psize, dMc + rp.copies, apply, rp.omega, packed};
        dM = dMc;
        LAUNCH(c, k_copy_rank, rp.copies, RSS_WARPS * 32, RSS_SMEM, ca);
    } else if (small) {
        LAUNCH(c, k_rank_small, 1, RSS_WARPS * 32, RSS_SMEM, n, target, gain, lp.gain_bound, kb, part, mv, state,
               g2, dM, dSE);
    } else {
    LAUNCH(c, k_move_flags, cdiv(n, 256), 256, 0, n, target, part, flag, state, g2, packed);
    compact_indices_dn(c, flag, mv, n, dM);
    LAUNCH(c, k_move_keys, cdiv(n, 256), 256, 0, mv, dM, gain, lp.gain_bound, khi, klo);
    if (kb > 32) {
        // stable by the low word, then by the high word (a 64-bit LSD sort); the high words are
        // recomputed for the permuted movers between the two passes
        u32 *tmp = c.arena.alloc<u32>(n);
        radix_sort_pairs_dn(c, klo, mv, dM, n, 32);
        LAUNCH(c, k_move_keys, cdiv(n, 256), 256, 0, mv, dM, gain, lp.gain_bound, khi, tmp);
        radix_sort_pairs_dn(c, khi, mv, dM, n, kb - 32);
    } else {
        radix_sort_pairs_dn(c, klo, mv, dM, n, kb);
    }
    }
    const bool pairs = !slots && !rp.encourage && rp.K <= PAIR_RANK_MAX_K;
    if (pairs) {  // k-way: moves in p <-> q pairs
        u32 *gk = khi, *pos = klo;  // the gain keys are spent
        LAUNCH(c, k_pair_group, cdiv(n, 256), 256, 0, mv, dM, part, target, rp.K, gk, pos);
        radix_sort_pairs_dn(c, gk, pos, dM, n, bits_for(2 * (u64)rp.K * rp.K));
        i64 *psn = c.arena.alloc<i64>(n);
        u32 *pk = c.arena.alloc<u32>(n), *node = c.arena.alloc<u32>(n), *follow = c.arena.alloc<u32>(n);
        LAUNCH(c, k_pair_keys, cdiv(n, 256), 256, 0, gk, pos, dM, n, mv, gain, psn, pk, node, follow);
        scan_excl_u32(c, follow, follow, n);
        const u64 pbound = 2 * lp.gain_bound;
        const u32 pb = bits_for(pbound);
        LAUNCH(c, k_pair_place, cdiv(n, 256), 256, 0, node, dM, pk, follow, psn, pbound, mv, klo);
        radix_sort_pairs_dn(c, klo, mv, dM, n, pb < 32 ? pb : 32);
        if (pb > 32) {
            LAUNCH(c, k_pair_gain_high, cdiv(n, 256), 256, 0, mv, dM, psn, pbound, khi);
            radix_sort_pairs_dn(c, khi, mv, dM, n, pb - 32);
        }
    }
    if (ck) {
        LAUNCH(c, k_copy_keys, cdiv(n, 256), 256, 0, mv, dM, rp.copy_n, ck);
        radix_sort_pairs_dn(c, ck, mv, dM, n, bits_for(rp.copies - 1));
    }
    if (!slots && (!small || pairs || rp.copies > 1)) LAUNCH(c, k_set_rank, cdiv(n, 256), 256, 0, mv, dM, state, dSE);
    if (!slots) c.arena.release(ranking);
    // cascade

    // inbound-set transitions (INCC): each destination pin of a mover gives at most two
    const bool track = rp.delta < 0x7FFFFFFFu && lp.dst_pins;
    // small levels check every prefix with one block per partition (k_validity_small), the
    // transitions summed per (partition, rank) in a dense K x n table
    const u64 tcap = track && !small ? 2 * lp.dst_pins : 0;
    u32 *tp = nullptr, *tr = nullptr;
    int32_t *tdv = nullptr;
    unsigned long long *tdense = nullptr;
    if (track && small) {
        tdense = c.arena.alloc<unsigned long long>((u64)rp.K * n);
        AXC_CUDA(cudaMemsetAsync(tdense, 0, (size_t)rp.K * n * 8, c.stream));
    } else if (track) {
        tp = c.arena.alloc<u32>(tcap);
        tr = c.arena.alloc<u32>(tcap);
        tdv = (int32_t *)c.arena.alloc<u32>(tcap);
    }
    {
        CascadeArgs C;
        C.e = L.e; C.encourage = rp.encourage ? 1 : 0; C.off = L.off; C.pins = L.pins; C.nsrc = L.nsrc;
        C.wfx = wfx; C.lam = cs.lam; C.cpart = cs.part; C.ccnt = cs.cnt; C.cdcnt = cs.dcnt; C.state = state; C.packed = packed;
        C.part = part; C.target = target; C.g2 = g2;
        C.track = track ? 1 : 0; C.tp = tp; C.tr = tr; C.tdv = tdv; C.dT = dT; C.tcap = tcap;
        C.tdense = tdense; C.dense_stride = n;
        C.status = c.d_status;
        C.K = kw ? kw->k : rp.K;
        C.ce = kw ? kw->ce : 0;
        C.cn = slots ? kw->cn : 0;
        const bool direct = C.K <= CC_DIRECT_BLOCK_K;
        size_t m1 = c.arena.mark();
        const bool longs = lp.max_len > CM_LEN;
        // a warp of the dense kernel looks at 32 hyperedges, or fewer where that leaves the GPU idle or
        // gives some warps several times the work of others (at 60 pins a hyperedge and 32 to a warp a
        // fifth of the warps were busy on average)
        u32 per_warp = 32;
        while (per_warp > 4 && L.e / per_warp < (u32)c.sms * 16) per_warp >>= 1;
        while (per_warp > 2 && per_warp * lp.short_pins > 192ull * L.e) per_warp >>= 1;
        // few nodes of many short incidences: a lane of the mover kernel would walk through several
        // of them one after the other while the dense kernel reads the whole level in a few microseconds
        const bool always = L.P / n > 128 && lp.short_pins <= (2u << 20);
        const MoverArgs V{mv, dM, L.toff, L.touch, L.nin, longs ? 1 : 0, rp.K <= CD_MAX_K ? 1 : 0, n, C.cn ? rp.copies : 1u,
                          always ? 1ull << 40 : lp.short_pins ? 16 * lp.short_sq / lp.short_pins : 0, per_warp};
        if (lp.short_pins && track) run_cascade_movers<true>(c, C, V, n, L.P, lp.max_deg);
        else if (lp.short_pins) run_cascade_movers<false>(c, C, V, n, L.P, lp.max_deg);
        if (longs) {
            u32 *big = c.arena.alloc<u32>(L.e), *huge = c.arena.alloc<u32>(L.e), *big2 = c.arena.alloc<u32>(L.e);
            // only the long hyperedges that hold a mover
            u32 *hlist = c.arena.alloc<u32>(L.e);
            uint8_t *mark = c.arena.alloc<uint8_t>(L.e);
            AXC_CUDA(cudaMemcpyAsync(mark, lp.hclass, L.e, cudaMemcpyDeviceToDevice, c.stream));
            LAUNCH(c, k_mover_hedges, (u32)c.sms * 8, 256, 0, C, V, mark);
            LAUNCH(c, k_long_list, cdiv(lp.n_hlong, 256), 256, 0, V, lp.hlong, lp.n_hlong, mark, hlist, dHl);
            const u32 lim = cascade_block_movers(c);
            // a warp per hyperedge: as many movers as 512 (hashed 64) leave room for
            u32 mvs = 64;
            while (mvs < (direct ? CL_MOV_DIRECT : CL_MOV_HASH) && mvs < lp.max_len) mvs <<= 1;
            mvs = std::min(mvs, lim);
            const u32 per = cl_bytes(direct, C.K, mvs);
            const auto lng = [&](auto kernel) {
                int per_w = 1;
                AXC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_w, kernel, CL_WARPS * 32, CL_WARPS * per));
                LAUNCH_AS(c, "k_cascade_long", kernel,
                          std::min<u32>(cdiv(lp.n_hlong, CL_WARPS), (u32)c.sms * (u32)std::max(per_w, 1)), CL_WARPS * 32,
                          CL_WARPS * per, C, hlist, dHl, mvs, per, big, dBig);
            };
            if (direct) lng(k_cascade_long<true>);
            else lng(k_cascade_long<false>);
            const u32 *blist = big, *bcount = dBig;
            const auto wide = [&](auto form) {
                constexpr WideForm F = decltype(form)::value;
                u32 mvw = mvs;
                while (mvw < cw_movers(F) && mvw < lp.max_len) mvw <<= 1;
                if (lim < CB_MOV_MAX) mvw = std::min(mvw, lim);
                if (mvw <= mvs) return;  // no hyperedge has more movers than a warp takes
                u32 *bigw = c.arena.alloc<u32>(L.e);
                const u32 bytes = cw_bytes(F, C.K, mvw);
                int per_w = 1;
                AXC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_w, k_cascade_wide<F>, cw_threads(F), bytes));
                LAUNCH_AS(c, "k_cascade_wide", k_cascade_wide<F>,
                          std::min<u32>(lp.n_hlong, (u32)c.sms * (u32)std::max(per_w, 1)), cw_threads(F), bytes, C, blist,
                          bcount, mvw, bigw, dBigW);
                blist = bigw;
                bcount = dBigW;
            };
            if (C.K <= CW_SWEEP_K) wide(std::integral_constant<WideForm, CW_SWEEP>());
            else if (n < (1u << 30)) {  // an event holds 30 bits of rank
                if (direct) wide(std::integral_constant<WideForm, CW_EVENTS>());
                else wide(std::integral_constant<WideForm, CW_HASH>());
            }
            // block kernel: shared memory sized by the level's largest hyperedge, all resident blocks
            u32 smov = 128;
            while (smov < lp.max_len && smov < lim) smov <<= 1;
            // hashed tables: sized for the level's largest hyperedge within the block's limit
            const u32 stab = direct ? std::max(2 * C.K, 32u)  // tk: the sweep's 2K lane masks
                                    : (u32)std::min<u64>(cascade_cap(std::min<u64>(lp.max_len, rp.K),
                                                                     std::min<u64>(lp.max_len, smov)),
                                                         CB_TAB_HASH);
            if (smov > CB_MID_MOV || (!direct && stab > CB_MID_TAB)) {  // middle tier first
                const u32 smid = std::min(smov, CB_MID_MOV), tmid = direct ? stab : std::min(stab, CB_MID_TAB);
                const size_t dmid = (size_t)smid * 12 + (size_t)tmid * 12;
                int per_mid = 1;
                AXC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_mid, k_cascade_block, CB_THREADS, dmid));
                LAUNCH(c, k_cascade_block, (u32)c.sms * (u32)std::max(per_mid, 1), CB_THREADS, dmid, C, blist, bcount, smid,
                       tmid, big2, dBig2);
                blist = big2;
                bcount = dBig2;
            }
            const size_t dyn = (size_t)smov * 12 + (size_t)stab * 12;
            int per_sm = 1;
            AXC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cascade_block, CB_THREADS, dyn));
            const u32 grid = (u32)c.sms * (u32)std::max(per_sm, 1);
            LAUNCH(c, k_cascade_block, grid, CB_THREADS, dyn, C, blist, bcount, smov, stab, huge, dHuge);
            // scratch kernel, only when some hyperedge can outgrow the block kernel: one slice of
            // movers, slots and tables per block, at most 1 GiB in all
            u64 mv_cap = 1;
            while (mv_cap < lp.max_len) mv_cap <<= 1;
            const u64 tab_cap = direct ? stab : cascade_cap(std::min<u64>(lp.max_len, rp.K), lp.max_len);
            if (mv_cap > smov || tab_cap > stab) {
                const u64 per_block = mv_cap * 12 + tab_cap * 12;
                const u32 gh = (u32)std::max<u64>(1, std::min<u64>((u64)c.sms, (1ull << 30) / per_block));
                u64 *smv = c.arena.alloc<u64>((u64)gh * mv_cap);
                u32 *ssl = c.arena.alloc<u32>((u64)gh * mv_cap);
                u32 *stb = c.arena.alloc<u32>((u64)gh * 3 * tab_cap);
                LAUNCH(c, k_cascade_huge, gh, CB_THREADS, 0, C, huge, dHuge, smv, ssl, stb, mv_cap, tab_cap);
            }
        }
        c.arena.release(m1);
    }
    if (slots) {  // every copy's prefixes, application and partition sizes
        LAUNCH(c, k_copy_sizes, rp.K, CV_SIZE_THREADS, 0, ca);
        LAUNCH(c, k_copy_tail, rp.copies, 1024, 0, ca);
        LAUNCH(c, k_kway_mark, (u32)c.sms * 8, 256, 0, mv, kw->cn, rp.copies, ca.applied, L.toff, L.touch, kw->dirty);
        c.arena.release(keep);
        return apply;
    }
    // prefix gains in rank order
    // per-rank deltas of the cascaded gain, the size violations and the inbound violations, in
    // one buffer [G | Vs | Vi] so one inclusive scan makes all three prefix sums
    i64 *raw = c.arena.alloc<i64>(3 * (u64)n), *pre = c.arena.alloc<i64>(3 * (u64)n);
    i64 *Gx = raw, *Vs = raw + n, *Vi = raw + 2 * (u64)n;
    if (small) {
        AXC_CUDA(cudaMemsetAsync(Vs, 0, 2 * (size_t)n * 8, c.stream));  // Vs and Vi
        LAUNCH(c, k_validity_small, rp.K, VS_THREADS, 0, mv, dM, part, target, L.nsize, psize, (u64)rp.omega,
               (unsigned long long *)Vs, track ? 1 : 0, tdense, n, pinb, (u64)rp.delta, (unsigned long long *)Vi);
        LAUNCH(c, k_tail_small, 1, 1024, 0, mv, dM, (const unsigned long long *)g2, Vs, Vi, track ? 1 : 0, target,
               part, apply);
        c.arena.release(keep);
        return apply;
    }
    LAUNCH(c, k_gather_g2, cdiv(n, 256), 256, 0, mv, dM, n, g2, Gx);  // also zeroes Vs and Vi
    // size validity
    {
        size_t m1 = c.arena.mark();
        const u32 nemax = 2 * n;
        u32 *key = c.arena.alloc<u32>(nemax), *val = c.arena.alloc<u32>(nemax);
        const u32 ge = std::min<u32>(cdiv(nemax, 256), (u32)c.sms * 8);
        LAUNCH(c, k_size_events, ge, 256, 0, mv, dM, part, target, key, val);
        radix_sort_pairs_dn(c, key, val, dSE, nemax, bits_for(rp.K ? rp.K - 1 : 0));
        i64 *d = c.arena.alloc<i64>(nemax), *E = c.arena.alloc<i64>(nemax);
        LAUNCH(c, k_size_delta, ge, 256, 0, mv, val, dSE, L.nsize, d);
        scan_excl_i64_dn(c, d, E, dSE, nemax);
        LAUNCH(c, k_size_flags, ge, 256, 0, key, val, d, E, dSE, psize, (u64)rp.omega,
               (unsigned long long *)Vs);
        c.arena.release(m1);
    }
    // inbound validity (INCC only): the transitions ordered by (partition, rank), the running
    // inbound-set size of each partition along them
    if (track) {
        size_t m1 = c.arena.mark();
        const u64 nt = tcap;
        const u32 rb = bits_for(n ? n - 1 : 0), pb = bits_for(rp.K ? rp.K - 1 : 0);
        const bool combined = rb + pb <= 32;
        u32 *key = c.arena.alloc<u32>(nt), *perm = c.arena.alloc<u32>(nt);
        const u32 gt = std::min<u32>(cdiv(nt, 256), (u32)c.sms * 8);
        LAUNCH(c, k_trans_keys, gt, 256, 0, dT, nt, tp, tr, rb, combined ? 1 : 0, key, perm);
        if (combined) {
            radix_sort_pairs_dn(c, key, perm, dT, nt, rb + pb);
        } else {
            radix_sort_pairs_dn(c, key, perm, dT, nt, rb);
            LAUNCH(c, k_gather_by_dn, gt, 256, 0, tp, perm, key, dT);
            radix_sort_pairs_dn(c, key, perm, dT, nt, pb);
        }
        u32 *sp = c.arena.alloc<u32>(nt), *sr = key;
        i64 *sd = c.arena.alloc<i64>(nt), *E2 = c.arena.alloc<i64>(nt);
        const bool fits = scan_fits(c, nt);  // else the whole capacity is scanned, past the count as zeros
        LAUNCH(c, k_trans_perm, fits ? gt : cdiv(nt, 256), 256, 0, perm, dT, fits ? 0 : nt, tp, tr, tdv, sp, sr, sd);
        if (fits) scan_excl_i64_dn(c, sd, E2, dT, nt);
        else scan_excl_i64(c, sd, E2, nt);
        LAUNCH(c, k_trans_flags, gt, 256, 0, sp, sr, sd, E2, dT, pinb, (u64)rp.delta,
               (unsigned long long *)Vi);
        c.arena.release(m1);
    }
    scan_incl_i64(c, raw, pre, 3 * (u64)n);
    // best prefix and apply
    if (rp.copies > 1) {  // every copy its own
        Best *bs = (Best *)c.arena.alloc<u64>(4 * (u64)rp.copies);
        u32 *capply = c.arena.alloc<u32>(rp.copies);
        AXC_CUDA(cudaMemsetAsync(apply, 0, 4, c.stream));
        LAUNCH(c, k_best_seg, rp.copies, 256, 0, pre, n, track ? 1 : 0, dM, ck, bs, capply, apply);
        LAUNCH(c, k_apply_seg, cdiv(n, 256), 256, 0, mv, dM, ck, target, bs, capply, part, ic ? ic->prev : nullptr,
               ic ? ic->stamp : nullptr, ic ? (const u32 *)ic->ctr : nullptr);
        if (kw)
            LAUNCH(c, k_kway_mark_ranked, (u32)c.sms * 8, 256, 0, mv, dM, ck, bs, capply, L.toff, L.touch, kw->dirty);
    } else {
        const u32 nbk = cdiv(n, 256) < 64u ? cdiv(n, 256) : 64u;
        Best *bb = (Best *)c.arena.alloc<u64>(4 * (nbk + 1));
        LAUNCH(c, k_best, nbk, 256, 0, pre, n, track ? 1 : 0, dM, bb + 1);
        LAUNCH(c, k_best_final, 1, 32, 0, bb + 1, nbk, pre, n, track ? 1 : 0, bb, apply);
        LAUNCH(c, k_apply, cdiv(n, 256), 256, 0, mv, target, bb, apply, part, ic ? ic->prev : nullptr,
               ic ? ic->stamp : nullptr, ic ? (const u32 *)ic->ctr : nullptr);
        if (kw)
            LAUNCH(c, k_kway_mark_ranked, (u32)c.sms * 8, 256, 0, mv, dM, (const u32 *)nullptr, bb, apply, L.toff,
                   L.touch, kw->dirty);
    }
    if (ic) {  // flag the moved nodes' hyperedges for the next census, then count the round
        LAUNCH(c, k_mark_moved, (u32)c.sms * 8, 256, 0, mv, dM, ic->stamp, ic->ctr, L.toff, L.touch, ic->dirty);
        LAUNCH(c, k_round_tick, 1, 32, 0, ic->ctr);
    }
    c.arena.release(keep);
    return apply;
}

// The round's one host round trip: the apply flag and the status word.
static bool round_result(Ctx &c, const u32 *apply) {
    AXC_CUDA(cudaMemcpyAsync(c.h_pinned, apply, 4, cudaMemcpyDeviceToHost, c.stream));
    AXC_CUDA(cudaMemcpyAsync((char *)c.h_pinned + 4, c.d_status, 4, cudaMemcpyDeviceToHost, c.stream));
    AXC_CUDA(cudaStreamSynchronize(c.stream));
    u32 hv[2];
    memcpy(hv, c.h_pinned, 8);
    if (hv[1] != DEV_OK) {
        AXC_CUDA(cudaMemsetAsync(c.d_status, 0, 4, c.stream));
        throw Error(AXC_EINTERNAL, "device status word = " + std::to_string(hv[1]));
    }
    return hv[0] != 0;
}

// One round, launched eagerly; returns true when moves were applied.
static bool refine_round(Ctx &c, const DLevel &L, const LevelPrep &lp, const u32 *wfx, const RefineParams &rp,
                         u32 *part, u32 discount, u32 round, IncCensus *ic, const KwayLevel *kw) {
    const size_t m0 = c.arena.mark();
    size_t keep;
    const u32 *apply = round_body(c, L, lp, wfx, rp, part, discount, round, nullptr, keep, ic, kw);
    const bool r = round_result(c, apply);
    c.arena.release(m0);
    return r;
}

// The rounds of one level replayed from one CUDA graph of the round body.
struct RoundGraph {
    cudaGraph_t g = nullptr;
    cudaGraphExec_t x = nullptr;
    ~RoundGraph() {
        if (x) cudaGraphExecDestroy(x);
        if (g) cudaGraphDestroy(g);
    }
};

// Kernel nodes of a captured graph (memset and copy nodes are not kernel launches).
static u32 rg_kernels(cudaGraph_t g) {
    size_t k = 0;
    if (cudaGraphGetNodes(g, nullptr, &k) != cudaSuccess || k == 0) return 0;
    std::vector<cudaGraphNode_t> nodes(k);
    if (cudaGraphGetNodes(g, nodes.data(), &k) != cudaSuccess) return 0;
    u32 kernels = 0;
    for (size_t i = 0; i < k; ++i) {
        cudaGraphNodeType t;
        if (cudaGraphNodeGetType(nodes[i], &t) == cudaSuccess && t == cudaGraphNodeTypeKernel) ++kernels;
    }
    return kernels;
}

// The round schedule on the device, for the level's rounds run as the body of one conditional
// WHILE graph node. rs = {r, R, rounds done}; after each round: the next r by the skip rule after
// a round without moves (sources/refinement.cu:539-542; the host loop of refine_level is the same
// rule), its discount (1, 2, none by thirds) and round number into dyn, and the loop goes on while
// r < R and the status word is clear.
__global__ void k_round_next(cudaGraphConditionalHandle h, u32 *__restrict__ rs, u32 *__restrict__ dyn,
                             const u32 *__restrict__ apply, const u32 *__restrict__ status) {
    u32 r = rs[0];
    const u32 R = rs[1];
    rs[2] += 1;
    if (!*apply) {
        if (r < R / 3) r = R / 2;
        else if (r < 2 * R / 3) r = 2 * R / 3;
        else r = R;
    }
    r += 1;
    rs[0] = r;
    const bool go = r < R && *(volatile const u32 *)status == 0;
    if (go) {
        dyn[0] = r < R / 3 ? 1u : (r < 2 * R / 3 ? 2u : 0xFFFFFFFFu);
        dyn[1] = r;
    }
    cudaGraphSetConditional(h, go ? 1u : 0u);
}

// All rounds of a level in one graph launch: a conditional WHILE node whose body is one round
// (round_body) followed by k_round_next, which applies the round schedule on the device. Returns
// the rounds run.
static u32 refine_level_loop(Ctx &c, const DLevel &L, const LevelPrep &lp, const u32 *wfx, const RefineParams &rp,
                             u32 *part, IncCensus *ic, const KwayLevel *kw) {
    const u32 R = rp.rounds;
    u32 *dyn = c.arena.alloc<u32>(2), *rs = c.arena.alloc<u32>(4);
    {
        u32 *hp = (u32 *)((char *)c.h_pinned + 64);
        hp[0] = 0 < R / 3 ? 1u : (0 < 2 * R / 3 ? 2u : 0xFFFFFFFFu);  // discount of round 0 (2 when R = 2)
        hp[1] = 0u;
        hp[2] = 0u;  // rs: r, R, rounds done
        hp[3] = R;
        hp[4] = 0u;
        hp[5] = 0u;
        AXC_CUDA(cudaMemcpyAsync(dyn, hp, 8, cudaMemcpyHostToDevice, c.stream));
        AXC_CUDA(cudaMemcpyAsync(rs, hp + 2, 16, cudaMemcpyHostToDevice, c.stream));
    }
    RoundGraph rg;
    AXC_CUDA(cudaGraphCreate(&rg.g, 0));
    cudaGraphConditionalHandle h;
    AXC_CUDA(cudaGraphConditionalHandleCreate(&h, rg.g, 1u, cudaGraphCondAssignDefault));
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t wn;
    AXC_CUDA(cudaGraphAddNode(&wn, rg.g, nullptr, 0, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    const size_t m1 = c.arena.mark();
    const u32 launches0 = c.launches;
    size_t keep;
    u32 *apply = nullptr;
    AXC_CUDA(cudaStreamBeginCaptureToGraph(c.stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    c.capturing = true;
    try {
        apply = round_body(c, L, lp, wfx, rp, part, 1, 0, dyn, keep, ic, kw);
        LAUNCH(c, k_round_next, 1, 1, 0, h, rs, dyn, apply, c.d_status);
    } catch (...) {
        c.capturing = false;
        cudaGraph_t junk = nullptr;
        cudaStreamEndCapture(c.stream, &junk);
        throw;
    }
    c.capturing = false;
    AXC_CUDA(cudaStreamEndCapture(c.stream, &body));
    c.launches = launches0;
    const u32 body_kernels = rg_kernels(body);
    AXC_CUDA(cudaGraphInstantiate(&rg.x, rg.g, 0));
    // the round's scratch above m1 stays unallocated, and nothing else allocates, while the graph runs
    c.arena.release(m1);
    AXC_CUDA(cudaGraphLaunch(rg.x, c.stream));
    u32 *hp = (u32 *)((char *)c.h_pinned + 64);
    AXC_CUDA(cudaMemcpyAsync(hp, rs, 16, cudaMemcpyDeviceToHost, c.stream));
    AXC_CUDA(cudaMemcpyAsync(hp + 4, c.d_status, 4, cudaMemcpyDeviceToHost, c.stream));
    AXC_CUDA(cudaStreamSynchronize(c.stream));
    const u32 done = hp[2];
    c.launches += done * body_kernels;
    if (hp[4] != DEV_OK) {
        AXC_CUDA(cudaMemsetAsync(c.d_status, 0, 4, c.stream));
        throw Error(AXC_EINTERNAL, "device status word = " + std::to_string(hp[4]));
    }
    return done;
}

// Blocks of k_small_rounds: a warp per two or so hyperedges and per node, at most one block per SM.
static u32 small_rounds_grid(const Ctx &c, const DLevel &L) {
    return std::max(1u, std::min<u32>((u32)c.sms, cdiv(std::max<u64>(L.e, L.n), 2 * (SR_THREADS / 32))));
}

// Levels whose rounds run in one launch (k_small_rounds). A node takes a warp there where the nodes are
// many; a level with one of more than GM_WARP_DEG incidences then keeps the rounds' own launches, which
// give such nodes a block (20,000 nodes, one of 300,000 incidences, 156 parts: 1559 ms in one launch, 316).
static bool small_rounds_eligible(const Ctx &c, const DLevel &L, const LevelPrep &lp, const RefineParams &rp) {
    return rp.encourage && rp.copies == 1 && rp.K <= VS_MAX_K && L.n <= (u32)RSS_CAP && L.e && lp.max_len <= CM_LEN &&
           (lp.max_deg <= GM_WARP_DEG || L.n <= small_rounds_grid(c, L) * (SR_THREADS / 32) / 2) && c.coop_supported &&
           !c.prof_on && round_loop_enabled();
}

static u32 small_rounds(Ctx &c, const DLevel &L, const LevelPrep &lp, const u32 *wfx, const RefineParams &rp, u32 *part) {
    const u32 n = L.n, K = rp.K;
    Census cs = alloc_census(c, L);
    cs.save = c.arena.alloc<i64>(n);
    AXC_CUDA(cudaMemsetAsync(cs.save, 0, (size_t)n * 8, c.stream));
    cs.wfx = wfx;
    cs.encourage = 1;
    cs.mw = mask_words(K);
    cs.mask = c.arena.alloc<u32>((u64)L.e * cs.mw);
    cs.dmask = c.arena.alloc<u32>((u64)L.e * cs.mw);
    u64 *psize = c.arena.alloc<u64>(K), *pinb = c.arena.alloc<u64>(K);
    part_sizes(c, n, part, L.nsize, psize, K);
    AXC_CUDA(cudaMemsetAsync(pinb, 0, (size_t)K * 8, c.stream));
    const bool track = rp.delta < 0x7FFFFFFFu && lp.dst_pins;
    unsigned long long *tdense = nullptr;
    if (track) {
        tdense = c.arena.alloc<unsigned long long>((u64)K * n);
        AXC_CUDA(cudaMemsetAsync(tdense, 0, (size_t)K * n * 8, c.stream));
    }
    u32 *target = c.arena.alloc<u32>(n);
    i64 *gain = c.arena.alloc<i64>(n);
    u32 *ctl = c.arena.alloc<u32>(8);  // [0, 3) schedule, [3] movers, [4] transitions (unused: summed)
    AXC_CUDA(cudaMemsetAsync(ctl, 0, 32, c.stream));
    SmallArgs S{};
    S.C = CensusArgs{L.off, L.pins, L.nsrc, part, cs.part, cs.cnt, cs.dcnt, cs.lam, c.d_status,
                     (unsigned long long *)cs.save, wfx, 1, cs.mask, cs.dmask, cs.mw, nullptr};
    S.G = make_gain_args(L, wfx, rp, cs, part, psize, pinb, 1, 0, target, gain, c.d_status);
    S.mv = c.arena.alloc<u32>(n);
    S.dM = ctl + 3;
    S.state = (uint2 *)c.arena.alloc<u64>(n);
    S.D.e = L.e; S.D.encourage = 1; S.D.off = L.off; S.D.pins = L.pins; S.D.nsrc = L.nsrc; S.D.wfx = wfx;
    S.D.part = part; S.D.target = target; S.D.state = S.state; S.D.packed = 1;
    S.D.g2 = c.arena.alloc<unsigned long long>(n);
    S.D.track = track ? 1 : 0; S.D.dT = ctl + 4; S.D.tdense = tdense; S.D.dense_stride = n; S.D.status = c.d_status;
    S.D.K = K;
    S.Vs = c.arena.alloc<unsigned long long>(n);
    S.Vi = c.arena.alloc<unsigned long long>(n);
    S.R = rp.rounds; S.kb = bits_for(lp.gain_bound); S.gbound = lp.gain_bound;
    S.part = part; S.psize = psize; S.pinb = pinb; S.save = cs.save; S.rs = ctl; S.track = track ? 1 : 0;
    const u32 grid = small_rounds_grid(c, L);
    S.V.per_warp = 32;
    while (S.V.per_warp > 2 && L.e / S.V.per_warp < grid * (SR_THREADS / 32)) S.V.per_warp >>= 1;
    const void *k = cs.mw == 1 ? (const void *)k_small_rounds<1> : cs.mw == 2 ? (const void *)k_small_rounds<2>
                  : cs.mw == 4 ? (const void *)k_small_rounds<4> : (const void *)k_small_rounds<8>;
    void *args[] = {(void *)&S};
    AXC_CUDA(cudaLaunchCooperativeKernel(k, grid, SR_THREADS, args, SR_SMEM, c.stream));
    c.launches++;
    u64 res[3];
    AXC_CUDA(cudaMemcpyAsync(ctl + 5, c.d_status, 4, cudaMemcpyDeviceToDevice, c.stream));
    fetch(c, res, ctl, 24);
    if ((u32)(res[2] >> 32) != DEV_OK) check_status(c);
    return (u32)(res[0] >> 32);
}

static u32 refine_rounds(Ctx &c, const DLevel &L, const LevelPrep &lp, const u32 *wfx, const RefineParams &rp, u32 *part,
                         IncCensus *ic, const KwayLevel *kw) {
    const u32 R = rp.rounds;
    // Graph replays need the round's scalars in device memory. Kernel-timer pairs captured in the
    // graph are read back after every replay; the bytes of the captured launches count per replay.
    const bool graph = R > 1;
    // Without the kernel timer the rounds run as one conditional WHILE graph: the schedule lives
    // on the device and the host waits once per level. With the timer on, each round is one replay
    // of the round graph, so that its event pairs are read after every round. The environment
    // variable AXC_ROUND_LOOP=0 also selects the replays (the same kernels and results; profilers
    // that do not follow kernels into conditional graph nodes see them then).
    if (graph && !c.prof_on && round_loop_enabled()) {
        return refine_level_loop(c, L, lp, wfx, rp, part, ic, kw);
    }
    size_t ev0 = 0, ev1 = 0;
    u64 bytes_per_round = 0;
    RoundGraph rg;
    u32 *dyn = nullptr, *apply = nullptr, graph_kernels = 0;
    if (graph) {
        dyn = c.arena.alloc<u32>(2);
        const size_t m1 = c.arena.mark();
        size_t keep;
        const u32 launches0 = c.launches;  // captured launches run only when replayed
        const u64 bytes0 = c.prof_bytes;
        ev0 = c.prof_used;
        AXC_CUDA(cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal));
        c.capturing = true;
        try {
            apply = round_body(c, L, lp, wfx, rp, part, 1, 0, dyn, keep, ic, kw);
        } catch (...) {
            c.capturing = false;
            cudaGraph_t junk = nullptr;
            cudaStreamEndCapture(c.stream, &junk);
            if (junk) cudaGraphDestroy(junk);
            throw;
        }
        c.capturing = false;
        ev1 = c.prof_used;
        bytes_per_round = c.prof_bytes - bytes0;
        c.prof_bytes = bytes0;
        AXC_CUDA(cudaStreamEndCapture(c.stream, &rg.g));
        AXC_CUDA(cudaGraphInstantiate(&rg.x, rg.g, 0));
        c.launches = launches0;
        graph_kernels = rg_kernels(rg.g);
        c.arena.release(m1);
        c.arena.alloc<u32>(1);  // keep the apply word below the round's scratch, as captured
    }
    u32 done = 0;
    for (u32 r = 0; r < R; ++r) {
        const u32 discount = r < R / 3 ? 1u : (r < 2 * R / 3 ? 2u : 0xFFFFFFFFu);
        ++done;
        bool applied;
        if (graph) {
            u32 *hp = (u32 *)((char *)c.h_pinned + 64);
            hp[0] = discount;
            hp[1] = r;
            AXC_CUDA(cudaMemcpyAsync(dyn, hp, 8, cudaMemcpyHostToDevice, c.stream));
            AXC_CUDA(cudaGraphLaunch(rg.x, c.stream));
            c.launches += graph_kernels;
            applied = round_result(c, apply);
            c.prof_collect(ev0, ev1);
            c.prof_bytes += bytes_per_round;
        } else {
            applied = refine_round(c, L, lp, wfx, rp, part, discount, r, ic, kw);
        }
        if (!applied) {
            if (r < R / 3) r = R / 2;
            else if (r < 2 * R / 3) r = 2 * R / 3;
            else r = R;
        }
    }
    if (graph) c.prof_used = ev0;  // the captured pairs go back to the pool with the graph
    return done;
}

u32 refine_level(Ctx &c, const DLevel &L, const u32 *wfx, const RefineParams &rp, u32 *part,
                 unsigned long long *copy_conn) {
    if (rp.rounds == 0 || L.n == 0) return 0;
    const size_t m = c.arena.mark();
    const bool kway = kway_eligible(L, rp);
    const LevelPrep lp = prepare_level(c, L, wfx, rp.K, kway);
    // state kept across the rounds: the k-way records, or one census where the level allows it
    KwayLevel kw;
    IncCensus ic;
    const bool inc = !kway && inc_census_eligible(L, lp, rp) && inc_census_enabled();
    if (!kway && small_rounds_eligible(c, L, lp, rp)) {
        const u32 done = small_rounds(c, L, lp, wfx, rp, part);
        c.arena.release(m);
        return done;
    }
    if (kway) kway_init(c, L, rp, part, kw);
    if (inc) inc_census_init(c, L, wfx, rp, ic);
    const u32 done = refine_rounds(c, L, lp, wfx, rp, part, inc ? &ic : nullptr, kway ? &kw : nullptr);
    if (copy_conn && kway) {  // from the records, brought up to date with the last round's moves
        kway_records(c, L, lp, part, kw);
        const KwArgs A = kway_args(L, part, kw);
        const dim3 grid(std::min<u32>(cdiv(kw.ce, KW_THREADS), std::max(1u, (u32)c.sms * 8 / rp.copies)), rp.copies);
        kway_words(kw.mw, [&](auto mw) {
            k_kway_conn<decltype(mw)::value><<<grid, KW_THREADS, 0, c.stream>>>(A, wfx, copy_conn);
            c.launches++;
            AXC_CUDA(cudaGetLastError());
        });
    } else if (copy_conn) {
        const Census cs = build_census(c, L, part, rp.K);
        LAUNCH(c, k_copy_conn, cdiv((u64)L.e, 256), 256, 0, (u64)L.e, L.e / rp.copies, cs.lam, wfx, copy_conn);
    }
    c.arena.release(m);
    return done;
}

}  // namespace axc
