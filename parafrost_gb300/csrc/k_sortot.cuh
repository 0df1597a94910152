// sortOT (src/cpu/simplify.cpp:81-93): the two lists of every elected variable in
// CNF_CMP_KEY order (size, first literal, last literal, signature;
// src/cpu/simplify.h:29-42) using the reference's own sort (insertion sort up to
// 20 entries, libstdc++ std::sort above). The lists are first put back into
// clause-store order, the order the reference's lists have when it sorts them,
// so equal keys end up in the reference's relative order.
#pragma once

#include "cnf.cuh"
#include "introsort.cuh"

namespace sigma {

struct KeyLess {
    const Hdr* hdr;
    const u32* lits;
    HD bool operator()(u32 a, u32 b) const {
        const Hdr x = hdr[a], y = hdr[b];
        if (x.size != y.size) return x.size < y.size;
        const u32 x0 = lits[x.start], y0 = lits[y.start];
        if (x0 != y0) return x0 < y0;
        const u32 xb = lits[x.start + x.size - 1], yb = lits[y.start + y.size - 1];
        if (xb != yb) return xb < yb;
        return x.sig < y.sig;
    }
};

struct IdLess {
    HD bool operator()(u32 a, u32 b) const { return a < b; }
};

struct SortArgs {
    Ctx c;
    const u32* pvs;
    u64* ws_bytes;  // kSpreadSlots words summing the elected lists' working set (4*occ + sum(8 + 4*len))
    // per elected variable: work-order key and rank (pv_order_key), words of BVE scratch
    u32 npvs, n_first;
    u32* key;
    u32* perm;
    u64* need;
};

// Work-order key of elected variable k with occ occurrences: descending clause count.
// Elected variables from n_first on (a batch's stopping formulas) come after the
// others; clause counts from 127 up share the first place (one 8-bit radix pass).
HD u32 pv_order_key(u32 k, u32 n_first, u32 occ) {
    return (k >= n_first ? 0x80u : 0u) | (0x7Fu - (occ < 0x7Fu ? occ : 0x7Fu));
}

// List d of n clauses by one thread: store order, then the reference's sort.
HD void sort_one_list(const Ctx& c, u32* d, u32 n) {
    if (n <= 1) return;
    if (n <= 20) ref_insertion_sort(d, (int)n, IdLess());
    else std_sort_replica(d, d + n, IdLess());
    reference_list_sort(d, (int)n, KeyLess{c.hdr, c.lits});
}

#if !SIGMA_CUDA
// One item per elected variable: its two lists.
HD void k_sort_pv(const SortArgs& a, u32 k) {
    u64 ws = 0;
    const u32 p = V2L(a.pvs[k]);
    for (u32 l = p; l <= p + 1; l++) {
        const u32 n = a.c.ot_size[l];
        u32* d = a.c.ot_refs + a.c.ot_off[l];
        ws += 4ull * n;
        for (u32 i = 0; i < n; i++) ws += 8ull + 4ull * a.c.hdr[d[i]].size;
        sort_one_list(a.c, d, n);
    }
    const u32 occ = a.c.ot_size[p] + a.c.ot_size[p + 1];
    a.key[k] = pv_order_key(k, a.n_first, occ);
    a.perm[k] = k;
    a.need[k] = (u64)occ + 2;
    spread_sum_add64(a.ws_bytes, ws);
}
#else
// A warp takes the lists of 16 elected variables, a lane each, and sorts those of up to
// SORT_LIST clauses together: their clauses' keys are staged in shared memory by
// consecutive lanes (four clauses a lane in flight), a clause's place is the number of
// smaller keys in its list, and the list is written back in one pass. Up to 20 clauses
// the reference's sort is stable over store order, so (key, clause id) is the order; above
// that it is std::sort, whose result is the same for any sort as long as no two keys are
// equal: a list with equal keys, and a longer one, is sorted by its lane as the reference
// does it. One thread a list compared keys in memory, a chain of four dependent loads
// a comparison. The stage (with the work-order sort) before and now: 10k-variable 3-SAT
// 213 and 107 us, 1M mixed clauses 373 and 228, a 6.8M-clause AIG 1.00 and 0.71 ms, 384
// mixed formulas 1.80 and 1.11, 80M community clauses 3.9 and 2.9.
constexpr u32 SORT_LIST = 32;    // longest list sorted by the warp
constexpr u32 SORT_STAGE = 192;  // clauses staged at a time
constexpr u32 SORT_WARPS = 8;

struct SortStage {
    u64 a[SORT_STAGE], b[SORT_STAGE];  // (size, first literal), (last literal, signature)
    u32 id[SORT_STAGE];
};

__global__ void __launch_bounds__(SORT_WARPS * 32) sort_lists_k(SortArgs a) {
    extern __shared__ u64 sort_smem[];
    SortStage& s = reinterpret_cast<SortStage*>(sort_smem)[threadIdx.x >> 5];
    const Ctx& c = a.c;
    const u32 lane = threadIdx.x & 31u;
    const u32 nwarps = (gridDim.x * blockDim.x) >> 5;
    u64 ws = 0;
    for (u32 k0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 16u; k0 < a.npvs; k0 += nwarps * 16u) {
        // lane: list side lane & 1 of variable k0 + lane / 2
        const u32 k = k0 + (lane >> 1);
        u32 n = 0, off = 0;
        if (k < a.npvs) {
            const u32 l = V2L(a.pvs[k]) + (lane & 1u);
            n = c.ot_size[l];
            off = c.ot_off[l];
        }
        const u32 occ = n + __shfl_xor_sync(kFull, n, 1);
        if (k < a.npvs && !(lane & 1u)) {
            a.key[k] = pv_order_key(k, a.n_first, occ);
            a.perm[k] = k;
            a.need[k] = (u64)occ + 2;
        }
        ws += 4ull * n;
        u32 alone = __ballot_sync(kFull, n > SORT_LIST);  // lists left to their lanes
        const u32 len = n > SORT_LIST ? 0u : n;
        if (n > SORT_LIST)
            for (u32 i = 0; i < n; i++) ws += 8ull + 4ull * c.hdr[c.ot_refs[off + i]].size;
        u32 next = 0;  // lists before this one are done
        while (next < 32) {
            // as many of the lists from `next` on as the stage holds
            const u32 mine = lane >= next ? len : 0u;
            u32 incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const u32 t = __shfl_up_sync(kFull, incl, o);
                if ((int)lane >= o) incl += t;
            }
            const u32 over = __ballot_sync(kFull, lane >= next && incl > SORT_STAGE);
            const u32 end = over ? (u32)(__ffs(over) - 1) : 32u;
            WarpWalk w;
            w.init(off, lane < end ? mine : 0u);
            for (u32 base = 0; base < w.total; base += 128) {
                u32 id[4];
                Hdr h[4];
#pragma unroll
                for (u32 q = 0; q < 4; q++) {
                    u32 o, src;
                    const u32 j = base + 32u * q + lane;
                    if (base + 32u * q < w.total) w.step(base + 32u * q, o, src);
                    id[q] = j < w.total ? c.ot_refs[src] : 0u;
                }
#pragma unroll
                for (u32 q = 0; q < 4; q++)
                    if (base + 32u * q + lane < w.total) h[q] = hdr_ro(&c.hdr[id[q]]);
#pragma unroll
                for (u32 q = 0; q < 4; q++) {
                    const u32 j = base + 32u * q + lane;
                    if (j >= w.total) continue;
                    const u32 *lits = c.lits + h[q].start;
                    s.a[j] = (u64)h[q].size << 32 | lits[0];
                    s.b[j] = (u64)lits[h[q].size ? h[q].size - 1u : 0u] << 32 | h[q].sig;
                    s.id[j] = id[q];
                    ws += 8ull + 4ull * h[q].size;
                }
            }
            __syncwarp();
            // places; a list above 20 with two equal keys goes to its lane unchanged
            WarpWalk v;
            v.init(off, lane < end ? mine : 0u);
            for (u32 base = 0; base < v.total; base += 32) {
                u32 o, src;
                v.step(base, o, src);
                const u32 j = base + lane;
                const u32 ex = __shfl_sync(kFull, v.excl, (int)o), m = __shfl_sync(kFull, mine, (int)o);
                bool tie = false;
                u32 rank = 0;
                if (j < v.total) {
                    const u64 ka = s.a[j], kb = s.b[j];
                    const u32 ki = s.id[j];
                    for (u32 e = ex; e < ex + m; e++) {
                        const u64 ea = s.a[e], eb = s.b[e];
                        const bool same = ea == ka && eb == kb;
                        rank += ea < ka || (ea == ka && (eb < kb || (same && s.id[e] < ki)));
                        tie |= same && e != j;
                    }
                    tie = tie && m > 20u;
                }
                alone |= __reduce_or_sync(kFull, tie ? 1u << o : 0u);
                if (j < v.total) c.ot_refs[src - (j - ex) + rank] = s.id[j];
            }
            __syncwarp();
            next = end;
        }
        // what is left to single lanes (a list with equal keys is back in some order of its
        // clauses, which the sort by id below undoes)
        if ((alone >> lane) & 1u) sort_one_list(c, c.ot_refs + off, n);
        __syncwarp();
    }
    for (int o = 16; o; o >>= 1) ws += __shfl_xor_sync(kFull, ws, o);
    if (lane == 0 && ws) atomicAdd((unsigned long long*)(a.ws_bytes + (blockIdx.x & (kSpreadSlots - 1u))), (unsigned long long)ws);
}
#endif

}  // namespace sigma
