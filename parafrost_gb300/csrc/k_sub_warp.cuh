// SUB with one warp per elected variable (self_sub_x, src/cpu/subsume.h:144-179).
//
// The candidate loop stays in list order: whether a candidate is strengthened or
// deleted depends on what happened to the earlier ones. The two searches inside
// one candidate step are split over the lanes: the self-subsumption search over
// the opposite list (subsume.h:123-142: first clause that strengthens the
// candidate, stopping at the first clause longer than it) and the subsumption
// search over the earlier candidates (subsume.h:105-121: first clause that
// subsumes it). Each takes the first hit in list order, so the outcome is the
// sequential one. Writes to the clauses happen on lane 0 between warp barriers.
//
// For most variables nothing is subsumed or strengthened, and the loop is a chain of
// two searches per candidate, each waiting for headers in memory. So the warp first
// looks at all pairs of the two lists at once, with the headers staged in shared memory
// (sub_nothing): when no pair as it stands would subsume or strengthen, no step of the
// loop could change anything and only the deleted clauses leave the lists.
// SUB of a round, before and now: 6.8M-clause AIG 2.49 and 1.38 ms, 80M community clauses
// 8.8 and 6.8 (5M variables of 14 clauses), 384 mixed formulas 3.8 and 2.7, 10k 3-SAT 108
// and 75 us.
#pragma once

#include "k_sub.cuh"

namespace sigma {

// Candidates of list lx against the opposite list lo (x: the candidates' literal of
// the elected variable, fx its negation).
HD void sub_warp_side(const SubArgs& a, u32 k, u32 p, u32 lx, u32 lo, SubLocal& L) {
    const Ctx& c = a.c;
    const u32* cands = c.ot_refs + c.ot_off[lx];
    const u32* opp = c.ot_refs + c.ot_off[lo];
    const u32 cs = c.ot_size[lx];
    for (u32 i = 0; i < cs; i++) {
        const u32 r = cands[i];
        const Hdr h = c.hdr[r];
        if (h.size > HSE_MAX_CL_SIZE) break;
        if (h_deleted(h.flags)) continue;
        // self-subsumption: first opposite clause that strengthens r, or the first
        // one longer than r (where the reference's scan stops)
        const u32 ls = c.ot_size[lo];
        const u32* cl = c.lits + h.start;
        const u32 js = wfirst(ls, [&](u32 j) {
            const Hdr s = c.hdr[opp[j]];
            if (s.size > h.size) return true;
            return !h_deleted(s.flags) && s.size > 1 && sig_selfsub(s.sig, h.sig) &&
                   clause_selfsub(lx, lo, c.lits + s.start, s.size, cl, h.size);
        });
        if (js != NONE_IDX && c.hdr[opp[js]].size <= h.size) {
            wone([&] {
                sub_strengthen(a, k, p, r, lx, L);
                set_molten(c, r, true);
            });
        }
        // subsumption by an earlier candidate
        const Hdr cand = c.hdr[r];
        const u32* cl2 = c.lits + cand.start;
        const u32 jb = wfirst(i, [&](u32 j) {
            const Hdr s = c.hdr[cands[j]];
            if (h_deleted(s.flags)) return false;
            if (h_molten(cand.flags) && s.size > cand.size) return false;
            return s.size > 1 && sig_sub(s.sig, cand.sig) && clause_sub(c.lits + s.start, s.size, cl2, cand.size);
        });
        if (jb != NONE_IDX) {
            wone([&] {
                const u32 sr = cands[jb];
                const Hdr s = c.hdr[sr];
                if (h_learnt(s.flags) && h_original(cand.flags)) {
                    c.hdr[sr].flags = (s.flags & ~3u) | ST_ORIGINAL;
                    touch(c, sr);
                }
                proof_delete(c, r);
                mark_deleted(c, r);
            });
        }
    }
    wone([&] { sub_update_list(c, lx); });
}

// Staged headers of a variable's two lists, entry after entry.
constexpr u32 SUB_STAGE = 64;
constexpr u32 SUB_SLOT = 4 * SUB_STAGE;  // words per warp

// True when SUB changes no clause of the np + nn <= SUB_STAGE entries (its updateOL is
// then done here); false leaves everything to the candidate loop. The pairs tested hold
// every pair that the loop can act on as long as it has not acted: an earlier entry of
// the same list that subsumes, an entry of the other list, no longer, that strengthens.
HD bool sub_nothing(const Ctx& c, u32 p, u32 np, u32 nn, u32* slot) {
    u32 *id = slot, *size = id + SUB_STAGE, *sig = size + SUB_STAGE, *start = sig + SUB_STAGE;
    const u32 tot = np + nn;
    u32* lp = c.ot_refs + c.ot_off[p];
    u32* ln = c.ot_refs + c.ot_off[p + 1];
    const u32 odd = wsum(tot, [&](u32 i) {  // deleted entries in the low half, molten ones in the high
        const u32 r = i < np ? lp[i] : ln[i - np];
        const Hdr h = c.hdr[r];
        const bool dead = h_deleted(h.flags);
        id[i] = r;
        size[i] = dead ? 0u : h.size;  // no live clause is empty
        sig[i] = h.sig;
        start[i] = h.start;
        return (dead ? 1u : 0u) + (h_molten(h.flags) ? 0x10000u : 0u);
    });
    wsync();
    if (odd >> 16) return false;
    const u32 inv = ((1u << 20) + tot - 1) / (tot ? tot : 1u);  // t / tot for t < 64 * 64
    const u32 hit = wfirst(tot * tot, [&](u32 t) {
        const u32 i = (t * inv) >> 20, j = t - i * tot;
        const u32 si = size[i], sj = size[j];
        if (sj < 2 || sj > si) return false;
        const bool same = (i < np) == (j < np);
        if (same) {
            if (j >= i || !sig_sub(sig[j], sig[i])) return false;
            return clause_sub(c.lits + start[j], sj, c.lits + start[i], si);
        }
        if (!sig_selfsub(sig[j], sig[i])) return false;
        const u32 x = i < np ? p : NEG(p);
        return clause_selfsub(x, FLIP(x), c.lits + start[j], sj, c.lits + start[i], si);
    });
    if (hit != NONE_IDX) return false;
    if (!odd) return true;
    // updateOL of both lists: the live entries move up in order
    for (u32 side = 0; side < 2; side++) {
        const u32 b = side ? np : 0u, n = side ? nn : np;
        u32* l = side ? ln : lp;
        u32 out = 0;
        for (u32 base = 0; base < n; base += 32) {
            const u32 m = wballot([&](u32 q) { return base + q < n && size[b + base + q] != 0; });
            wfor(32, [&](u32 q) {
                if ((m >> q) & 1u) l[out + (u32)popc32(m & ((1u << q) - 1u))] = id[b + base + q];
            });
            out += (u32)popc32(m);
        }
        wone([&] { c.ot_size[p + side] = out; });
    }
    return true;
}

// What a pass needs to know of elected variable k before its lists; false: not its turn,
// or a list past the bound. SUB changes list sizes only of the variable it works on.
struct SubHead {
    u32 k, v, np, nn;
};
HD bool sub_head(const SubArgs& a, u32 k, SubHead& h) {
    if (a.run && !a.run[k]) return false;
    h.k = k;
    h.v = a.pvs[k];
    h.np = a.c.ot_size[V2L(h.v)];
    h.nn = a.c.ot_size[NEG(V2L(h.v))];
    return h.np <= a.sub_max && h.nn <= a.sub_max;
}

HD void sub_warp_pv(const SubArgs& a, const SubHead& h, u32* slot) {
    const Ctx& c = a.c;
    const u32 k = h.k, np = h.np, nn = h.nn;
    const u32 p = V2L(h.v), n = NEG(p);
    const bool pre = a.pre_off && a.pre_off[k] < a.pre_off[k + 1];
    wsync();
    if (!pre && np + nn <= SUB_STAGE && sub_nothing(c, p, np, nn, slot)) return;
    SubLocal L;  // lane 0's (only lane 0 strengthens)
    L.n = 0;
    if (a.pre_off) {
        wone([&] {
            for (u32 i = a.pre_off[k]; i < a.pre_off[k + 1]; i++) sub_local_oblivion(c, p, a.pre_lits[i]);
        });
    }
    sub_warp_side(a, k, p, p, n, L);
    sub_warp_side(a, k, p, n, p, L);
}

#if SIGMA_CUDA
// Warps take elected variables in work order (perm), a few at a time. The heads of a grab
// are loaded by its lanes at once: one after the other they were a chain of three loads a
// variable, and a pass over variables that are mostly not its turn (`run`) did little else;
// such a pass takes 32 a grab. The pass waits for its lists' headers and literals (half of
// the issue slots idle), so with more variables than resident warps eight blocks an SM pay
// although 32 registers spill a little; below that the spills are all that shows. SUB stage
// with one head after the other, heads at once, and eight blocks: 80M community clauses
// 6.87, 6.09 and 5.56 ms; 6.8M AIG clauses 1.40, 1.33 and 1.16; 10k 3-SAT variables 72, 75
// and 81 us.
template <int MinBlocks>
__global__ void __launch_bounds__(256, MinBlocks) sub_warp_k(SubArgs a, const u32* perm, u32 n, u32* next) {
    __shared__ u32 slots[8][SUB_SLOT];
    u32* slot = slots[threadIdx.x >> 5];
    const u32 lane = threadIdx.x & 31u;
    auto grab = [&](u32 left) {
        const u32 x = warp_chunk(left);
        return a.run && x == kWarpChunkFar ? 32u : x;
    };
    u32 chunk = grab(n);
    while (true) {
        u32 j0 = 0;
        if (lane == 0) j0 = atomicAdd(next, chunk);
        j0 = __shfl_sync(kFull, j0, 0);
        if (j0 >= n) break;
        const u32 j1 = j0 + chunk < n ? j0 + chunk : n;
        SubHead h{0, 0, 0, 0};
        const bool go = j0 + lane < j1 && sub_head(a, perm[j0 + lane], h);
        for (u32 m = __ballot_sync(kFull, go); m; m &= m - 1u) {
            const int q = __ffs(m) - 1;
            const SubHead x{__shfl_sync(kFull, h.k, q), __shfl_sync(kFull, h.v, q), __shfl_sync(kFull, h.np, q),
                            __shfl_sync(kFull, h.nn, q)};
            sub_warp_pv(a, x, slot);
        }
        chunk = grab(n - j1);
    }
}
#endif

}  // namespace sigma
