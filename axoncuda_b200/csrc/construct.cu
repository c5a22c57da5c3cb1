// Construction kernels: fixed-point weights, per-hyperedge uniqueness (level-0 rule-2 dedupe and
// level-to-level contraction share one kernel family), compaction into a new pin CSR, and the
// incidence ("touching") CSR built as a stable transpose.
//
// Uniqueness rule. Every pin occurrence k of hyperedge h gets a key (the pin, or its group at
// contraction) and a priority (cls << 31 | position). For each key the occurrence of minimum
// priority survives. Level 0 (includes/hgraph.hpp:518-581, rule 2): cls = 0 everywhere, so the
// first occurrence in flat order survives and sources (stored first) win over destinations.
// Contraction (kernels/construction.cu:304-489): cls = 1 for sources, 0 for destinations, so a
// group that is both keeps its destination occurrence. Survivors are compacted in position order,
// so the output keeps sources first and is deterministic.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace axc {
namespace {

__global__ void k_wfx(const float *__restrict__ w, u32 *__restrict__ wfx, u32 e) {
    u32 h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h >= e) return;
    float x = w ? w[h] : 1.0f;
    double y = x > 0.0f ? floor((double)x * 262144.0) : 0.0;
    wfx[h] = y >= 4294967295.0 ? 0xFFFFFFFFu : (u32)y;
}

constexpr u32 UQ_WARP_CAP = 256;      // hyperedges up to this size: one warp, table in smem
constexpr u32 UQ_MID_CAP = 2048;      // up to this size: one block, 32 KB of table (several per SM)
constexpr u32 UQ_BLOCK_CAP = 8192;    // up to this size: one block, 128 KB of table
constexpr u32 UQ_WARPS = 8;

__device__ __forceinline__ u32 uq_key(const u32 *pins, const u32 *groups, u64 k) {
    u32 v = pins[k];
    return groups ? groups[v] : v;
}

// Insert all occurrences of hyperedge [a,b) into the table (keys/vals, size mask+1), then mark
// survivors. Threads [t0, t0+nt) of the caller cooperate; caller syncs between phases.
__device__ __forceinline__ void uq_insert(const u32 *pins, const u32 *groups, u64 a, u64 b, u64 s,
                                          bool dst_wins, u32 *keys, u32 *vals, u32 mask, u32 t,
                                          u32 nt, u32 *status) {
    for (u64 k = a + t; k < b; k += nt) {
        u32 key = uq_key(pins, groups, k);
        u32 pri = ((dst_wins && k < s) ? 0x80000000u : 0u) | (u32)(k - a);
        u32 slot = hash_find_or_insert(keys, mask, key);
        if (slot == NONE) { atomicExch(status, DEV_HASH_FULL); continue; }
        atomicMin(&vals[slot], pri);
    }
}
__device__ __forceinline__ void uq_mark(const u32 *pins, const u32 *groups, u64 a, u64 b, u64 s,
                                        bool dst_wins, const u32 *keys, const u32 *vals, u32 mask,
                                        u32 t, u32 nt, uint8_t *keep, u32 &kept, u32 &kept_src) {
    for (u64 k = a + t; k < b; k += nt) {
        u32 key = uq_key(pins, groups, k);
        u32 pri = ((dst_wins && k < s) ? 0x80000000u : 0u) | (u32)(k - a);
        u32 slot = hash_find(keys, mask, key);
        bool kp = slot != NONE && vals[slot] == pri;
        keep[k] = kp;
        if (kp) { ++kept; if (k < s) ++kept_src; }
    }
}

// A warp's consecutive hyperedges: 32 where most have a handful of pins, fewer where they are long or
// few. A warp per hyperedge left seven lanes in eight idle on a netlist.
static u32 hedges_per_warp(const Ctx &c, u32 e, u64 P) {
    u32 per = P <= 16ull * e ? 32u : P <= 64ull * e ? 8u : 1u;
    while (per > 1 && e / per < (u32)c.sms * 16) per >>= 1;
    return per;
}
// The lane l whose item holds position f, given the items' exclusive prefix sums less b0 (lanes
// [lo, hi)): the last that starts at or before f. All lanes take part.
__device__ __forceinline__ u32 owner_lane(u32 excl, u32 b0, u32 lo, u32 hi, u32 f) {
    u32 l = lo, h = hi - 1;
    for (int it = 0; it < 5; ++it) {
        const u32 mid = (l + h + 1) >> 1;
        const u32 em = __shfl_sync(0xFFFFFFFFu, excl, mid & 31);
        if (l < h) { if (em - b0 <= f) l = mid; else h = mid - 1; }
    }
    return l;
}
__device__ __forceinline__ u32 warp_incl(u32 x, u32 lane) {
#pragma unroll
    for (u32 o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// One warp per `per` consecutive hyperedges. Those of at most 32 pins are packed into the warp's
// lanes, a pin each: the lanes holding the same pin of the same hyperedge find each other by a match,
// no table. Then those up to UQ_WARP_CAP, one after the other, by a table in shared memory.
// Measured per level: 1M nets of about 5 pins 355 us with a warp and a table per net, 103 packed;
// 220k nets 72 and 39.
__global__ void __launch_bounds__(UQ_WARPS * 32, 7) k_uniq_warp(u32 e, const u64 *__restrict__ off,
                                                             const u32 *__restrict__ pins, const u32 *__restrict__ nsrc,
                                                             const u32 *__restrict__ groups, int dst_wins, u32 per,
                                                             uint8_t *__restrict__ keep, u32 *__restrict__ cnt,
                                                             u32 *__restrict__ cnt_src, u32 *status) {
    __shared__ u32 tk[UQ_WARPS][2 * UQ_WARP_CAP], tv[UQ_WARPS][2 * UQ_WARP_CAP];
    const u32 w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u64 h0 = ((u64)blockIdx.x * UQ_WARPS + w) * per;
    if (h0 >= e) return;
    const u32 nh = (u32)(e - h0 < per ? e - h0 : per), h = (u32)h0 + lane;
    const bool mine = lane < nh;
    const u64 a = mine ? off[h] : 0, len64 = mine ? off[h + 1] - a : 0;
    const u32 ns = mine ? nsrc[h] : 0, few = len64 <= 32 ? (u32)len64 : 0u;
    const u32 x = warp_incl(few, lane), excl = x - few;
    for (u32 lo = 0; lo < nh;) {
        const u32 b0 = __shfl_sync(0xFFFFFFFFu, excl, lo);
        const u32 hi = lo + __popc(__ballot_sync(0xFFFFFFFFu, lane >= lo && lane < nh && x - b0 <= 32));
        const u32 T = __shfl_sync(0xFFFFFFFFu, x, hi - 1) - b0;
        if (T == 0) {  // only longer or empty ones (uniform over the warp)
            if (lane >= lo && lane < hi && len64 == 0) cnt[h] = cnt_src[h] = 0;
            lo = hi;
            continue;
        }
        const u32 ol = owner_lane(excl, b0, lo, hi, lane);
        const u32 at = lane - (__shfl_sync(0xFFFFFFFFu, excl, ol) - b0);  // in the hyperedge
        const u64 k = __shfl_sync(0xFFFFFFFFu, a, ol) + at;
        const bool in = lane < T, src = at < __shfl_sync(0xFFFFFFFFu, ns, ol);
        const u64 key = in ? (u64)ol << 32 | uq_key(pins, groups, k) : (u64)(32 + lane) << 32;
        const u32 same = __match_any_sync(0xFFFFFFFFu, key), dsts = __ballot_sync(0xFFFFFFFFu, in && !src);
        const u32 from = dst_wins && (same & dsts) ? same & dsts : same;
        const bool kp = in && (u32)__ffs(from) == lane + 1;
        if (in) keep[k] = kp;
        const u32 kb = __ballot_sync(0xFFFFFFFFu, kp), sb = __ballot_sync(0xFFFFFFFFu, kp && src);
        if (lane >= lo && lane < hi && len64 <= 32) {
            const u32 run = few ? (0xFFFFFFFFu >> (32 - few)) << (excl - b0) : 0u;
            cnt[h] = __popc(kb & run);
            cnt_src[h] = __popc(sb & run);
        }
        lo = hi;
    }
    u32 *keys = tk[w], *vals = tv[w];
    for (u32 left = __ballot_sync(0xFFFFFFFFu, len64 > 32 && len64 <= UQ_WARP_CAP); left; left &= left - 1) {
        const u32 i = __ffs(left) - 1, len = (u32)__shfl_sync(0xFFFFFFFFu, len64, i);
        const u64 ai = __shfl_sync(0xFFFFFFFFu, a, i), bi = ai + len, si = ai + __shfl_sync(0xFFFFFFFFu, ns, i);
        u32 cap = 64;
        while (cap < 2 * len) cap <<= 1;
        for (u32 j = lane; j < cap; j += 32) { keys[j] = NONE; vals[j] = NONE; }
        __syncwarp();
        uq_insert(pins, groups, ai, bi, si, dst_wins, keys, vals, cap - 1, lane, 32, status);
        __syncwarp();
        u32 kept = 0, ks = 0;
        uq_mark(pins, groups, ai, bi, si, dst_wins, keys, vals, cap - 1, lane, 32, keep, kept, ks);
        kept = warp_sum(kept);
        ks = warp_sum(ks);
        if (lane == i) { cnt[h] = kept; cnt_src[h] = ks; }
        __syncwarp();  // the table is no longer read
    }
}

// One block per listed hyperedge (the count in device memory when d_n is set).
// Measured: 20 x 5000 network (34M pins) 1350 us a level with one launch sized on the host, 440
// with one per table size looping over the device's lists.
__global__ void k_uniq_block(const u32 *__restrict__ list, u32 nlist, const u32 *__restrict__ d_n,
                             const u64 *__restrict__ off,
                             const u32 *__restrict__ pins, const u32 *__restrict__ nsrc,
                             const u32 *__restrict__ groups, int dst_wins, uint8_t *__restrict__ keep,
                             u32 *__restrict__ cnt, u32 *__restrict__ cnt_src, u32 *gtab,
                             const u64 *__restrict__ gtab_off, u32 *status) {
    extern __shared__ u32 dyn[];
    __shared__ u32 red[2][32];
    if (d_n) nlist = *d_n;
    for (u32 idx = blockIdx.x; idx < nlist; idx += gridDim.x) {
        const u32 h = list[idx];
        const u64 a = off[h], b = off[h + 1], s = a + nsrc[h];
        const u32 len = (u32)(b - a);
        u32 cap = 64;
        while (cap < 2 * len) cap <<= 1;
        u32 *keys = gtab ? gtab + 2 * gtab_off[idx] : dyn, *vals = keys + cap;
        for (u32 i = threadIdx.x; i < cap; i += blockDim.x) { keys[i] = NONE; vals[i] = NONE; }
        __syncthreads();
        uq_insert(pins, groups, a, b, s, dst_wins, keys, vals, cap - 1, threadIdx.x, blockDim.x, status);
        __syncthreads();
        u32 kept = 0, ks = 0;
        uq_mark(pins, groups, a, b, s, dst_wins, keys, vals, cap - 1, threadIdx.x, blockDim.x, keep, kept, ks);
        kept = warp_sum(kept);
        ks = warp_sum(ks);
        if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = kept; red[1][threadIdx.x >> 5] = ks; }
        __syncthreads();
        if (threadIdx.x == 0) {
            u32 t0 = 0, t1 = 0;
            for (u32 i = 0; i < blockDim.x / 32; ++i) { t0 += red[0][i]; t1 += red[1][i]; }
            cnt[h] = t0;
            cnt_src[h] = t1;
        }
        __syncthreads();  // the table and red are no longer read
    }
}

// Stable compaction of survivors: a warp per `per` consecutive hyperedges, whose pins follow one
// another before and after.
// Measured: 1M nets 152 us with a warp per net, 15.
__global__ void k_uniq_compact(u32 e, const u64 *__restrict__ off, const u32 *__restrict__ pins,
                               const u32 *__restrict__ groups, const uint8_t *__restrict__ keep, u32 per,
                               const u64 *__restrict__ new_off, u32 *__restrict__ new_pins) {
    const u32 lane = threadIdx.x & 31;
    const u64 h0 = (((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per;
    if (h0 >= e) return;
    const u64 a = off[h0], b = off[h0 + per < e ? h0 + per : e];
    u64 o = new_off[h0];
    constexpr u32 U = 4;
    for (u64 base = a; base < b; base += 32 * U) {
        bool kp[U];
        u32 v[U];
#pragma unroll
        for (u32 r = 0; r < U; ++r) {
            const u64 k = base + 32 * r + lane;
            kp[r] = k < b && keep[k];
            v[r] = k < b ? pins[k] : 0;
        }
#pragma unroll
        for (u32 r = 0; r < U; ++r)
            if (kp[r] && groups) v[r] = groups[v[r]];
#pragma unroll
        for (u32 r = 0; r < U; ++r) {
            const u32 bal = __ballot_sync(0xFFFFFFFFu, kp[r]);
            if (kp[r]) new_pins[o + __popc(bal & ((1u << lane) - 1u))] = v[r];
            o += __popc(bal);
        }
    }
}

// The hyperedges beyond a warp's table by length: up to UQ_MID_CAP, up to UQ_BLOCK_CAP, longer.
// Measured: 1M nets 4.5 us; a flag, scan and scatter launch per list before.
__global__ void __launch_bounds__(1024) k_uniq_lists(u32 e, const u64 *__restrict__ off, u32 *mid, u32 *big, u32 *huge,
                                                     u32 *__restrict__ n) {
    __shared__ u32 sh[33];
    const u32 h = blockIdx.x * blockDim.x + threadIdx.x;
    const u64 len = h < e ? off[h + 1] - off[h] : 0;
    const u32 t = len <= UQ_WARP_CAP ? 3u : len <= UQ_MID_CAP ? 0u : len <= UQ_BLOCK_CAP ? 1u : 2u;
    if (!__syncthreads_or(t < 3)) return;
    u32 *lists[3] = {mid, big, huge};
#pragma unroll
    for (u32 i = 0; i < 3; ++i) {
        if (!__syncthreads_or(t == i)) continue;
        const u32 at = block_append(t == i, n + i, sh);
        if (t == i) lists[i][at] = h;
    }
}
__global__ void k_table_sizes(const u32 *__restrict__ list, u32 nlist, const u64 *__restrict__ off,
                              u64 *__restrict__ sz) {
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == nlist) sz[i] = 0;
    if (i >= nlist) return;
    u32 h = list[i];
    u64 len = off[h + 1] - off[h], cap = 64;
    while (cap < 2 * len) cap <<= 1;
    sz[i] = cap;
}

// ---------------------------------------------------------------- transpose
// key = 2*pin + is_source, value = hyperedge: a stable sort by key lists, per node, its inbound
// hyperedges ascending and then its outbound ones ascending (sources/construction.cu:17-62).
// A warp per `per` consecutive hyperedges, their pins side by side.
// Measured: 1M nets 124 us with a warp per net, 18; 34M pins 78 us (about 1090 with two counting
// atomics per pin).
__global__ void k_touch_keys(u32 e, const u64 *__restrict__ off, const u32 *__restrict__ pins,
                             const u32 *__restrict__ nsrc, u32 per, u32 *__restrict__ keys, u32 *__restrict__ vals) {
    const u32 lane = threadIdx.x & 31;
    const u64 h0 = (((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per;
    if (h0 >= e) return;
    const u32 nh = (u32)(e - h0 < per ? e - h0 : per);
    const u64 a = off[h0], P = off[h0 + nh] - a;
    const u32 h = (u32)h0 + (lane < nh ? lane : nh - 1);
    const u64 at = off[h] - a;
    const u32 ns = nsrc[h];
    if (nh == 1 || P >> 31) {  // one by one (positions below are 32-bit)
        for (u32 i = 0; i < nh; ++i) {
            const u64 s0 = a + __shfl_sync(0xFFFFFFFFu, at, i), s = s0 + __shfl_sync(0xFFFFFFFFu, ns, i);
            const u64 s1 = i + 1 < nh ? a + __shfl_sync(0xFFFFFFFFu, at, (i + 1) & 31) : a + P;
            for (u64 k = s0 + lane; k < s1; k += 32) {
                keys[k] = 2 * pins[k] + (k < s ? 1u : 0u);
                vals[k] = (u32)h0 + i;
            }
        }
        return;
    }
    constexpr u32 U = 4;
    for (u32 f0 = 0; f0 < (u32)P; f0 += 32 * U) {
        u32 v[U], ol[U];
#pragma unroll
        for (u32 r = 0; r < U; ++r) {
            const u32 f = f0 + 32 * r + lane;
            v[r] = f < (u32)P ? pins[a + f] : 0;
        }
#pragma unroll
        for (u32 r = 0; r < U; ++r) {
            const u32 f = f0 + 32 * r + lane;
            ol[r] = owner_lane((u32)at, 0, 0, nh, f);
            const u32 src = f < __shfl_sync(0xFFFFFFFFu, (u32)at + ns, ol[r]) ? 1u : 0u;
            if (f < (u32)P) {
                keys[a + f] = 2 * v[r] + src;
                vals[a + f] = (u32)h0 + ol[r];
            }
        }
    }
}
// Where a node's keys start in the sorted keys, by two binary searches: its offset, and its
// inbound count from the start of its second key. Against counting by atomics (two per pin,
// contended at high-degree nodes) and a scan; the searches' upper steps stay in cache.
__device__ __forceinline__ u64 first_at_least(const u32 *__restrict__ a, u64 lo, u64 hi, u32 x) {
    while (lo < hi) {
        const u64 mid = (lo + hi) >> 1;
        if (a[mid] < x) lo = mid + 1; else hi = mid;
    }
    return lo;
}
// Measured: 1M nodes 20 us.
__global__ void k_touch_starts(u32 n, u64 P, const u32 *__restrict__ keys, u64 *__restrict__ toff,
                               u32 *__restrict__ nin) {
    const u32 v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v > n) return;
    if (v == n) { toff[n] = P; return; }
    const u64 o = first_at_least(keys, 0, P, 2 * v);
    toff[v] = o;
    nin[v] = (u32)(first_at_least(keys, o, P, 2 * v + 1) - o);
}

// Input validation before any id is used as an index: offsets non-decreasing and within the P pins,
// source counts within their hyperedge, pin ids below n. Failures set the status word (no trap).
// The pins are read in order, whatever the hyperedges' lengths.
// Bound by the pins' read. Measured: 1M nets 188 us with a warp per net, 16.
__global__ void k_check_input(u32 n, u32 e, u64 P, const u64 *__restrict__ off, const u32 *__restrict__ pins,
                              const u32 *__restrict__ nsrc, u32 *status) {
    const u64 i0 = (u64)blockIdx.x * blockDim.x + threadIdx.x, step = (u64)gridDim.x * blockDim.x;
    bool bad = false;
    for (u64 h = i0; h < e; h += step) {
        const u64 a = off[h], b = off[h + 1];
        bad |= b < a || b > P || nsrc[h] > b - a;
    }
#pragma unroll 4
    for (u64 k = off[0] + i0; k < P; k += step) bad |= pins[k] >= n;
    if (bad) atomicExch(status, DEV_BAD_INDEX);
}

__global__ void k_group_sizes(u32 n, const u32 *__restrict__ groups, const u32 *__restrict__ nsize,
                              u32 *__restrict__ gsize) {
    u32 v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < n) atomicAdd(&gsize[groups[v]], nsize[v]);
}

}  // namespace

void compute_wfx(Ctx &c, const float *d_w, u32 *d_wfx, u32 e) {
    if (e) LAUNCH(c, k_wfx, cdiv(e, 256), 256, 0, d_w, d_wfx, e);
}

u64 hedge_unique(Ctx &c, u32 e, const u64 *off, const u32 *pins, const u32 *nsrc, const u32 *groups,
                 bool dst_wins, u64 *new_off, u32 *new_pins, u32 *new_nsrc, u64 pins_in) {
    if (e == 0) {
        AXC_CUDA(cudaMemsetAsync(new_off, 0, 8, c.stream));
        return 0;
    }
    size_t m = c.arena.mark();
    uint8_t *keep = c.arena.alloc<uint8_t>(pins_in ? pins_in : 1);
    u32 *cnt = c.arena.alloc<u32>(e);
    const u32 per = hedges_per_warp(c, e, pins_in);
    LAUNCH(c, k_uniq_warp, cdiv(e, UQ_WARPS * per), UQ_WARPS * 32, 0, e, off, pins, nsrc, groups,
           (int)dst_wins, per, keep, cnt, new_nsrc, c.d_status);
    // hyperedges larger than a warp's table: their lists and counts stay on the device, except for
    // those that need tables in device memory, which are rare and sized by the host
    u32 *mid = c.arena.alloc<u32>(e), *big = c.arena.alloc<u32>(e), *huge = c.arena.alloc<u32>(e);
    u64 *res = c.arena.alloc<u64>(4);  // list counts (three words), then the total and the status
    u32 *ln = (u32 *)res;
    AXC_CUDA(cudaMemsetAsync(res, 0, 32, c.stream));
    LAUNCH(c, k_uniq_lists, cdiv(e, 1024), 1024, 0, e, off, mid, big, huge, ln);
    if (pins_in > UQ_WARP_CAP)
        LAUNCH(c, k_uniq_block, std::min<u32>(cdiv(pins_in, UQ_WARP_CAP), (u32)c.sms * 6), 256, 2 * 2 * UQ_MID_CAP * 4, mid, 0u,
               ln, off, pins, nsrc, groups, (int)dst_wins, keep, cnt, new_nsrc, (u32 *)nullptr, (const u64 *)nullptr,
               c.d_status);
    if (pins_in > UQ_MID_CAP)
        LAUNCH(c, k_uniq_block, std::min<u32>(cdiv(pins_in, UQ_MID_CAP), (u32)c.sms), 512, 2 * 2 * UQ_BLOCK_CAP * 4, big, 0u,
               ln + 1, off, pins, nsrc, groups, (int)dst_wins, keep, cnt, new_nsrc, (u32 *)nullptr, (const u64 *)nullptr,
               c.d_status);
    const u32 nh = pins_in > UQ_BLOCK_CAP ? fetch1(c, ln + 2) : 0;
    if (nh) {
        u64 *tsz = c.arena.alloc<u64>(nh + 1);
        LAUNCH(c, k_table_sizes, cdiv(nh + 1, 256), 256, 0, huge, nh, off, tsz);
        scan_excl_u64(c, tsz, tsz, nh + 1);
        u64 tot = fetch1(c, tsz + nh);  // sum of table capacities
        u32 *gtab = c.arena.alloc<u32>(2 * tot);
        LAUNCH(c, k_uniq_block, nh, 512, 0, huge, nh, (const u32 *)nullptr, off, pins, nsrc, groups, (int)dst_wins, keep, cnt,
               new_nsrc, gtab, (const u64 *)tsz, c.d_status);
    }
    offsets_from_counts(c, cnt, new_off, e);
    LAUNCH(c, k_uniq_compact, cdiv(e, 8 * per), 256, 0, e, off, pins, groups, keep, per, new_off, new_pins);
    AXC_CUDA(cudaMemcpyAsync(res + 2, new_off + e, 8, cudaMemcpyDeviceToDevice, c.stream));
    AXC_CUDA(cudaMemcpyAsync(res + 3, c.d_status, 4, cudaMemcpyDeviceToDevice, c.stream));
    u64 fin[2];
    fetch(c, fin, res + 2, 16);
    const u64 total = fin[0];
    if ((u32)fin[1] != DEV_OK) check_status(c);
    c.arena.release(m);
    return total;
}

void build_touching(Ctx &c, u32 n, u32 e, const u64 *off, const u32 *pins, const u32 *nsrc, u64 P,
                    u64 *toff, u32 *touch, u32 *nin) {
    size_t m = c.arena.mark();
    u32 *keys = c.arena.alloc<u32>(P ? P : 1);
    const u32 per = e ? hedges_per_warp(c, e, P) : 1;
    if (e) LAUNCH(c, k_touch_keys, cdiv(e, 8 * per), 256, 0, e, off, pins, nsrc, per, keys, touch);
    radix_sort_pairs(c, keys, touch, P, bits_for(n ? 2ull * n - 1 : 0));
    LAUNCH(c, k_touch_starts, cdiv((u64)n + 1, 256), 256, 0, n, P, keys, toff, nin);
    c.arena.release(m);
}

void check_input(Ctx &c, u32 n, u32 e, u64 P, const u64 *off, const u32 *pins, const u32 *nsrc) {
    if (e)
        LAUNCH(c, k_check_input, std::min<u32>(cdiv(std::max<u64>(P, e), 256), (u32)c.sms * 16), 256, 0, n, e, P, off, pins, nsrc,
               c.d_status);
    u32 s = fetch1(c, c.d_status);
    if (s != DEV_OK) {
        AXC_CUDA(cudaMemsetAsync(c.d_status, 0, 4, c.stream));
        throw Error(AXC_EINVAL, "hypergraph rejected: an offset, source count or pin id is out of range");
    }
}

void group_sizes(Ctx &c, u32 n, const u32 *groups, const u32 *nsize, u32 *gsize, u32 ng) {
    AXC_CUDA(cudaMemsetAsync(gsize, 0, (size_t)ng * 4, c.stream));
    if (n) LAUNCH(c, k_group_sizes, cdiv(n, 256), 256, 0, n, groups, nsize, gsize);
}

void setup_construct_kernels() {
    cudaFuncSetAttribute(k_uniq_block, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * 2 * UQ_BLOCK_CAP * 4);
}

}  // namespace axc
