// Occurrence-table build by literal buckets (createOT, src/cpu/simplify.cpp:35-56;
// GPU reference: histogram.cu:34-52, memory.cu:271-312, create_ot_k kernels.cu:81-96).
//
// The literal slots are cut into buckets of 2^shift consecutive slots. No pass
// issues one device-memory atomic per occurrence, and no pass writes outside the
// range of the bucket it works on:
//   pass 0 (ot_bucket_count_k): every occurrence (a literal of a live clause) adds
//     one to its bucket in a per-block shared histogram; one atomic per bucket per
//     block at the end. An exclusive scan of the bucket counts gives every bucket
//     its range of the table (all its literals' lists, side by side).
//   pass 1 (ot_bucket_fill_k): per tile of clauses, the occurrences are counted per
//     bucket, one reservation per non-empty bucket gives each run its place, a block scan
//     orders the tile by bucket, the occurrences are staged in shared memory in that order
//     (slot in its bucket and clause in its tile: one word) and written out in that order,
//     consecutive threads on consecutive places of a run, clause ids and slots side by side
//     (6 bytes an occurrence).
//   pass 2 (ot_bucket_lists_k): one block per bucket: per-slot counts in shared
//     memory (from the 2-byte slots alone), a block scan gives the list sizes and starts of
//     the bucket's slots, then every occurrence lands in its list inside the bucket's range.
// What bounds it: pass 1 the issue slots of its two walks (74% busy on 28M occurrences,
// 252 us; 295 us when whose literal a lane has was searched for in five shuffles a step),
// pass 2 the scattered 4-byte stores. All tables of a round, before (6,144 occurrences a
// tile staged as 8-byte pairs) and now: 80M community clauses 14.6 and 13.8 ms, 8M 1.41 and
// 1.31. Tiles of 6,144, 8,192, 14,336 and 30,720 occurrences with 4, 3, 2 and 1 blocks an
// SM: 14.9, 14.4, 13.8 and 14.1 ms. (Above 120M literal slots the buckets are as large as
// they get, their counters leave room for one block: 62M variables, 350M occurrences 20.6 ms.)
// Clause headers and literals are read by whole warps, consecutive lanes on
// consecutive literals. The order inside one list is unspecified, as for the
// atomic build: the elected lists are sorted into the reference's order later.
#pragma once

#include "cnf.cuh"

namespace sigma {

#if SIGMA_CUDA

constexpr u32 OTB_FILL_CAP = 14336;  // occurrences of a pass-1 tile ordered in shared memory
                                     // (84 KB)
constexpr u32 OTB_MAX_TILE = 1u << 16;  // clauses of a pass-1 tile
constexpr u32 OTB_MAX_BUCKETS = 4096;
constexpr u32 OTB_FILL_BUCKETS = 3680;  // most buckets with which two blocks of pass 1 fit an SM
static_assert(2 * (OTB_FILL_CAP * 6 + 8 * (OTB_FILL_BUCKETS + 1) + 128 + 1024) <= 228 * 1024,
              "stage, counters, static shared memory and the 1 KB a block reserves, twice");
constexpr u32 OTB_MAX_SHIFT = 15;   // 32,768 slots: 128 KiB of shared counters in pass 2
constexpr u32 OTB_LIST_THREADS = 1024;  // one block a bucket, 32 warps to keep its loads in flight
constexpr unsigned OTB_FULL = 0xffffffffu;
// (clause in the tile, slot) in one word
static_assert(OTB_MAX_SHIFT <= 15 && OTB_MAX_TILE <= 1u << 17, "a staged occurrence is one word");

struct OtbArgs {
    Ctx c;
    u32 shift;        // bucket of literal l: l >> shift
    u32 nb;           // buckets
    u32* count;       // nb: occurrences per bucket (pass 0)
    u32* cursor;      // nb: next free position of every bucket (pass 1; starts at base)
    const u32* base;  // nb + 1: first position of every bucket, base[nb] = occurrences
    u32* tcid;        // occurrences grouped by bucket: clause ids
    unsigned short* tslot;  // and literals, less the bucket's first
    u32 fill_tile;    // clauses per pass-1 tile (a multiple of 32)
};

// The literals of the live clauses c0 .. c1-1, walked by the warps of a block (warp w of nw
// takes every nw-th group of 32 clauses), consecutive lanes on consecutive literals
// (clauses are mostly adjacent in the literal array, so the loads coalesce).
// f(literal, clause id) is called by the lanes that have one. Four steps' loads and the
// next group's headers are in flight together: a walk waits for memory once a group, not
// once a step. Returns the number of literals this warp walked.
template <class F>
DEV u32 warp_clause_literals(const Ctx& c, u32 c0, u32 c1, u32 w, u32 nw, F&& f) {
    const u32 lane = threadIdx.x & 31u;
    auto header = [&](u32 g, u32& start, u32& size) {
        start = size = 0;
        if (g < c1 && lane < c1 - g) {
            const Hdr h = hdr_ro(&c.hdr[g + lane]);
            if (!h_deleted(h.flags)) {
                start = h.start;
                size = h.size;
            }
        }
    };
    u32 sum = 0, start, size;
    header(c0 + w * 32u, start, size);
    for (u32 g = c0 + w * 32u; g < c1; g += nw * 32u) {
        WarpWalk ww;
        ww.init(start, size);
        header(g + nw * 32u, start, size);
        sum += ww.total;
        for (u32 base = 0; base < ww.total; base += 128) {
            u32 k[4], l[4];
#pragma unroll
            for (u32 q = 0; q < 4; q++) {
                u32 src;
                if (base + 32u * q < ww.total) ww.step(base + 32u * q, k[q], src);
                if (base + 32u * q + lane < ww.total) l[q] = __ldg(&c.lits[src]);
            }
#pragma unroll
            for (u32 q = 0; q < 4; q++)
                if (base + 32u * q + lane < ww.total) f(l[q], g + k[q]);
        }
    }
    return sum;
}

// Pass 0: occurrences per bucket.
__global__ void __launch_bounds__(256) ot_bucket_count_k(OtbArgs a) {
    extern __shared__ u32 otb_hist[];
    for (u32 b = threadIdx.x; b < a.nb; b += blockDim.x) otb_hist[b] = 0;
    __syncthreads();
    const u32 nw = blockDim.x >> 5;
    warp_clause_literals(a.c, 0, a.c.ncls, blockIdx.x * nw + (threadIdx.x >> 5), gridDim.x * nw,
                         [&](u32 lit, u32) { atomicAdd(&otb_hist[lit >> a.shift], 1u); });
    __syncthreads();
    for (u32 b = threadIdx.x; b < a.nb; b += blockDim.x)
        if (otb_hist[b]) atomicAdd(&a.count[b], otb_hist[b]);
}

// Block-wide exclusive scan of cnt[0, n) in place; returns the total. Every thread
// of the block calls it.
DEV u32 otb_block_scan(u32* cnt, u32 n, u32* warp_tot, u32* carry) {
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    if (tid == 0) *carry = 0;
    __syncthreads();
    for (u32 i0 = 0; i0 < n; i0 += blockDim.x) {
        const u32 i = i0 + tid;
        const u32 v = i < n ? cnt[i] : 0u;
        u32 incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 t = __shfl_up_sync(OTB_FULL, incl, o);
            if ((int)lane >= o) incl += t;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        u32 before = *carry;
        for (u32 w = 0; w < warp; w++) before += warp_tot[w];
        if (i < n) cnt[i] = before + incl - v;
        __syncthreads();
        if (tid == blockDim.x - 1) *carry = before + incl;
        __syncthreads();
    }
    return *carry;
}

// Pass 1: occurrences grouped by bucket. The tile's literals are walked twice (the second
// time mostly cache hits): once to count them per bucket, once to place them. A tile with
// more occurrences than shared memory holds (very long clauses) writes them to their runs
// directly instead. Tiles hold fill_tile clauses, sized from the mean clause length so
// that a tile's occurrences nearly fill the stage.
constexpr u32 OTB_FILL_THREADS = 768;
__global__ void __launch_bounds__(OTB_FILL_THREADS, 2) ot_bucket_fill_k(OtbArgs a) {
    extern __shared__ u32 otb_fsm[];
    u32* stage = otb_fsm;              // OTB_FILL_CAP: clause in the tile << OTB_MAX_SHIFT | slot
    unsigned short* bucket = reinterpret_cast<unsigned short*>(stage + OTB_FILL_CAP);  // OTB_FILL_CAP
    u32* cur = stage + OTB_FILL_CAP + OTB_FILL_CAP / 2;  // nb: counts, then places
    u32* run = cur + a.nb;                               // nb: global start of the tile's run, less its place
    __shared__ u32 warp_tot[OTB_FILL_THREADS / 32];
    __shared__ u32 carry, ntile;
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const u32 T = a.fill_tile, smask = (1u << a.shift) - 1u;
    const u32 ntiles = (a.c.ncls + T - 1u) / T;
    for (u32 t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const u32 c0 = t * T, c1 = a.c.ncls - c0 < T ? a.c.ncls : c0 + T;
        for (u32 b = threadIdx.x; b < a.nb; b += blockDim.x) cur[b] = 0;
        if (threadIdx.x == 0) ntile = 0;
        __syncthreads();
        const u32 nwarp = warp_clause_literals(a.c, c0, c1, warp, nw,
                                               [&](u32 lit, u32) { atomicAdd(&cur[lit >> a.shift], 1u); });
        if (lane == 0 && nwarp) atomicAdd(&ntile, nwarp);
        __syncthreads();
        const u32 n = ntile;
        for (u32 b = threadIdx.x; b < a.nb; b += blockDim.x) {
            const u32 k = cur[b];
            run[b] = k ? atomicAdd(&a.cursor[b], k) : 0u;
        }
        if (n <= OTB_FILL_CAP) {
            otb_block_scan(cur, a.nb, warp_tot, &carry);
            for (u32 b = threadIdx.x; b < a.nb; b += blockDim.x) run[b] -= cur[b];
            __syncthreads();
            warp_clause_literals(a.c, c0, c1, warp, nw, [&](u32 lit, u32 cid) {
                const u32 b = lit >> a.shift, q = atomicAdd(&cur[b], 1u);
                stage[q] = (cid - c0) << OTB_MAX_SHIFT | (lit & smask);
                bucket[q] = (unsigned short)b;
            });
            __syncthreads();
            for (u32 i = threadIdx.x; i < n; i += blockDim.x) {
                const u32 x = stage[i], q = run[bucket[i]] + i;
                a.tcid[q] = c0 + (x >> OTB_MAX_SHIFT);
                a.tslot[q] = (unsigned short)(x & ((1u << OTB_MAX_SHIFT) - 1u));
            }
        } else {
            __syncthreads();
            for (u32 b = threadIdx.x; b < a.nb; b += blockDim.x) cur[b] = 0;
            __syncthreads();
            warp_clause_literals(a.c, c0, c1, warp, nw, [&](u32 lit, u32 cid) {
                const u32 b = lit >> a.shift;
                const u32 q = run[b] + atomicAdd(&cur[b], 1u);
                a.tcid[q] = cid;
                a.tslot[q] = (unsigned short)(lit & smask);
            });
        }
        __syncthreads();
    }
}

// Pass 2: one block per bucket. Shared memory: 2^shift slot counters.
__global__ void __launch_bounds__(OTB_LIST_THREADS) ot_bucket_lists_k(OtbArgs a) {
    extern __shared__ u32 otb_cnt[];
    __shared__ u32 warp_tot[OTB_LIST_THREADS / 32];
    __shared__ u32 carry;
    const u32 b = blockIdx.x;
    const u32 l0 = b << a.shift;
    const u32 D = a.c.D;
    const u32 nl = D - l0 < (1u << a.shift) ? D - l0 : (1u << a.shift);
    const u32 p0 = a.base[b], p1 = a.base[b + 1];
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    for (u32 i = tid; i < nl; i += blockDim.x) otb_cnt[i] = 0;
    if (tid == 0) carry = 0;
    __syncthreads();
    // four consecutive occurrences per thread per step, in one load each; the staged
    // words are read for the last time in the second walk (evicted first), the lists'
    // lines are filled by scattered stores and kept while they fill
    const u64 pf = l2_policy_first(), pl = l2_policy_last();
    const u32 step = 4u * blockDim.x;
    const u32 a0 = p0 & ~3u;  // the arrays are 16-byte aligned
    for (u32 k0 = a0 + 4u * tid; k0 < p1; k0 += step) {
        const ushort4 x = __ldcg(reinterpret_cast<const ushort4*>(a.tslot + k0));
        if (k0 >= p0) atomicAdd(&otb_cnt[x.x], 1u);
        if (k0 + 1 >= p0 && k0 + 1 < p1) atomicAdd(&otb_cnt[x.y], 1u);
        if (k0 + 2 >= p0 && k0 + 2 < p1) atomicAdd(&otb_cnt[x.z], 1u);
        if (k0 + 3 >= p0 && k0 + 3 < p1) atomicAdd(&otb_cnt[x.w], 1u);
    }
    __syncthreads();
    // block scan of the slot counts, blockDim.x slots per step: list sizes and starts
    for (u32 i0 = 0; i0 < nl; i0 += blockDim.x) {
        const u32 i = i0 + tid;
        const u32 v = i < nl ? otb_cnt[i] : 0u;
        u32 incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 t = __shfl_up_sync(OTB_FULL, incl, o);
            if ((int)lane >= o) incl += t;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        u32 before = carry;
        for (u32 w = 0; w < warp; w++) before += warp_tot[w];
        const u32 excl = before + incl - v;
        if (i < nl) {
            a.c.ot_size[l0 + i] = v;
            a.c.ot_off[l0 + i] = p0 + excl;
            otb_cnt[i] = excl;
        }
        __syncthreads();
        if (tid == blockDim.x - 1) carry = excl + v;
        __syncthreads();
    }
    for (u32 k0 = a0 + 4u * tid; k0 < p1; k0 += step) {
        const ushort4 x = __ldcg(reinterpret_cast<const ushort4*>(a.tslot + k0));
        const Q4 id = ldro4_hint(reinterpret_cast<const Q4*>(a.tcid + k0), pf);
        u32* refs = a.c.ot_refs + p0;
        if (k0 >= p0) st_hint(&refs[atomicAdd(&otb_cnt[x.x], 1u)], id.x, pl);
        if (k0 + 1 >= p0 && k0 + 1 < p1) st_hint(&refs[atomicAdd(&otb_cnt[x.y], 1u)], id.y, pl);
        if (k0 + 2 >= p0 && k0 + 2 < p1) st_hint(&refs[atomicAdd(&otb_cnt[x.z], 1u)], id.z, pl);
        if (k0 + 3 >= p0 && k0 + 3 < p1) st_hint(&refs[atomicAdd(&otb_cnt[x.w], 1u)], id.w, pl);
    }
}

#endif  // SIGMA_CUDA

}  // namespace sigma
