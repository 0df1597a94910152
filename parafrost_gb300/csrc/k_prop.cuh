// In-round unit propagation: ParaFROST::prop (src/cpu/elimination.cpp:41-99;
// GPU reference elimbcp.cu:103-192, which runs it on the host).
//
// The reference walks the trail in order; for each assigned literal t it strips
// -t from the clauses of ot[-t] (deleting those satisfied by a literal already
// true), enqueues the units this creates, then empties ot[-t] and deletes every
// clause of ot[t]. Here the pending literals of one wave are processed together:
//   wave A (per pending literal t): delete ot[t], collect ot[-t] into a worklist;
//   wave B (per collected clause): delete it if any literal is true, else remove
//          every false literal; an empty clause is a conflict, a unit is claimed
//          with a compare-and-swap on its variable and appended to the trail.
// Waves repeat until no new unit appears. (That is the serial form of the emulation
// build; the GPU's waves only judge clauses and strip them once at the end, see
// prop_waves_k.) The final state is the propagation
// fixpoint the reference reaches: the same clauses deleted, the same live-clause
// contents and signatures, the same set of assigned literals, the same emptied
// lists, and a conflict exactly when the reference finds one. Only the order of
// the trail and the literal contents of clauses that end up deleted can differ.
#pragma once

#include "cnf.cuh"

namespace sigma {

struct PropArgs {
    Ctx c;
    u32 head;        // first pending trail index of this wave
    u32 stamp;       // wave stamp (not used before; the launch of all waves takes one per wave)
    u32* cl_stamp;   // per clause: last wave that collected it
#if !SIGMA_CUDA
    u32* work;       // collected clause ids
    u32* nwork;      // their count
    u32 cap_work;
#endif
};

constexpr u32 PROP_SHORT = 4;  // literals of a clause loaded together

#if !SIGMA_CUDA
// The waves of the emulation build, one item after another. They share the fixpoint with
// the GPU's waves, not their walks, chases, list parts and strip: those run on a GPU only.
//
// Wave A: one item per pending literal.
HD void k_prop_lists(const PropArgs& a, u32 k) {
    const Ctx& c = a.c;
    const u32 t = c.trail[a.head + k];
    const u32 f = FLIP(t);
    // collect ot[-t]
    const u32 fo = c.ot_off[f], fs = c.ot_size[f];
    for (u32 i = 0; i < fs; i++) {
        const u32 r = c.ot_refs[fo + i];
        const bool take = !h_deleted(c.hdr[r].flags) && atom_exch(&a.cl_stamp[r], a.stamp) != a.stamp;
        const u32 pos = warp_append(a.nwork, take);  // one reservation per group of lanes
        if (!take) continue;
        if (pos < a.cap_work) a.work[pos] = r;
        else set_err(c, ERR_CAP_SCRATCH);
    }
    // toblivion(ot[t])
    const u32 to = c.ot_off[t], ts = c.ot_size[t];
    for (u32 i = 0; i < ts; i++) {
        const u32 r = c.ot_refs[to + i];
        c.hdr[r].flags = (c.hdr[r].flags & ~3u) | ST_DELETED;
        touch(c, r);
    }
    c.ot_size[t] = 0;
    c.ot_size[f] = 0;
}

// Wave B: one item per collected clause.
HD void k_prop_clause(const PropArgs& a, u32 k) {
    const Ctx& c = a.c;
    const u32 r = a.work[k];
    Hdr h = c.hdr[r];
    if (h_deleted(h.flags)) return;
    u32* l = c.lits + h.start;
    const u32 v0 = ABS(l[0]);  // names the formula if the clause empties
    u32 n = 0, sig = 0;
    if (h.size <= PROP_SHORT) {
        // short clause: all literals and their values loaded together
        u32 L[PROP_SHORT];
        int val[PROP_SHORT];
#pragma unroll
        for (u32 j = 0; j < PROP_SHORT; j++) L[j] = j < h.size ? l[j] : 0u;
#pragma unroll
        for (u32 j = 0; j < PROP_SHORT; j++) val[j] = j < h.size ? lit_value(c, L[j]) : 0;
        bool sat = false;
#pragma unroll
        for (u32 j = 0; j < PROP_SHORT; j++) sat |= val[j] == 1;
        if (sat) {
            c.hdr[r].flags = (h.flags & ~3u) | ST_DELETED;
            touch(c, r);
            return;
        }
#pragma unroll
        for (u32 j = 0; j < PROP_SHORT; j++) {
            if (j < h.size && val[j] != 0) {
                l[n++] = L[j];
                sig |= MAPHASH(L[j]);
            }
        }
    } else {
        // satisfied?
        for (u32 i = 0; i < h.size; i++) {
            if (lit_value(c, l[i]) == 1) {
                c.hdr[r].flags = (h.flags & ~3u) | ST_DELETED;
                touch(c, r);
                return;
            }
        }
        for (u32 i = 0; i < h.size; i++) {
            const u32 lit = l[i];
            if (lit_value(c, lit) == 0) continue;
            l[n++] = lit;
            sig |= MAPHASH(lit);
        }
    }
    h.size = n;
    h.sig = sig;
    c.hdr[r] = h;
    touch(c, r);
    if (n == 0) {
        set_unsat(c, v0);
        // in a batch the other formulas go on: keep no empty live clause around
        if (c.var_fid) {
            c.hdr[r].flags = (h.flags & ~3u) | ST_DELETED;
            touch(c, r);
        }
        return;
    }
    if (n == 1) claim_unit(c, l[0]);
}

// Sweep wave: when the pending literals' lists cover a large part of the store (a
// propagation cascade), every clause of the store is checked against the current
// assignment instead, in store order (streaming reads, no list walk, no collection):
// a clause with a true literal is deleted, one with false literals loses them (a
// unit is claimed, an empty clause is a conflict); a clause without an assigned
// literal is left alone. Literals assigned during the sweep are pending for the next
// wave, so the fixpoint is the one the list waves reach.
HD void k_prop_sweep(const PropArgs& a, u32 r) {
    const Ctx& c = a.c;
    Hdr h = c.hdr[r];
    if (h_deleted(h.flags)) return;
    u32* l = c.lits + h.start;
    u32 nfalse = 0;
    for (u32 i = 0; i < h.size; i++) {
        const int v = lit_value(c, l[i]);
        if (v == 1) {
            c.hdr[r].flags = (h.flags & ~3u) | ST_DELETED;
            touch(c, r);
            return;
        }
        nfalse += v == 0;
    }
    if (!nfalse) return;
    const u32 v0 = ABS(l[0]);
    u32 n = 0, sig = 0;
    for (u32 i = 0; i < h.size; i++) {
        const u32 lit = l[i];
        if (lit_value(c, lit) == 0) continue;
        l[n++] = lit;
        sig |= MAPHASH(lit);
    }
    h.size = n;
    h.sig = sig;
    c.hdr[r] = h;
    touch(c, r);
    if (n == 0) {
        set_unsat(c, v0);
        if (c.var_fid) {
            c.hdr[r].flags = (h.flags & ~3u) | ST_DELETED;
            touch(c, r);
        }
        return;
    }
    if (n == 1) claim_unit(c, l[0]);
}
// The lists of a swept wave's literals end empty, as the list waves leave them.
HD void k_prop_sweep_lists(const PropArgs& a, u32 k) {
    const u32 t = a.c.trail[a.head + k];
    a.c.ot_size[t] = 0;
    a.c.ot_size[FLIP(t)] = 0;
}
// Sweep rather than walk: the pending literals' lists (estimated from the mean list
// length) exceed a fraction of the store; scale = mean list length x the divisor of
// that fraction (0: never sweep).
HD bool prop_use_sweep(u32 pending, u32 scale, u32 ncls) { return scale && (u64)pending * scale > (u64)ncls; }
#else
// Clause r, which holds a literal that has become false, judged against the current
// assignment (read at L2: other warps assign meanwhile) without being changed, except
// that a clause with a true literal is deleted. Two unassigned literals end the look (a
// true literal further on has its own walk, which deletes the clause). Returns the
// clause's one unassigned literal, or 0. A clause without any is a conflict.
DEV u32 prop_judge(const Ctx& c, u32 r) {
    const Hdr h = c.hdr[r];
    if (h_deleted(h.flags)) return 0;
    const u32* l = c.lits + h.start;
    u32 und = 0, unit = 0;
    for (u32 k0 = 0; k0 < h.size && und < 2; k0 += PROP_SHORT) {
        u32 L[PROP_SHORT], v[PROP_SHORT];
#pragma unroll
        for (u32 j = 0; j < PROP_SHORT; j++) L[j] = k0 + j < h.size ? l[k0 + j] : 0u;
#pragma unroll
        for (u32 j = 0; j < PROP_SHORT; j++) v[j] = k0 + j < h.size ? __ldcg(&c.asg[ABS(L[j])]) : FLIP(L[j]);
        bool sat = false;
#pragma unroll
        for (u32 j = 0; j < PROP_SHORT; j++) {
            sat |= v[j] == L[j];
            if (!v[j]) {
                und++;
                unit = L[j];
            }
        }
        if (sat) {
            c.hdr[r].flags = (h.flags & ~3u) | ST_DELETED;
            touch(c, r);
            return 0;
        }
    }
    if (und == 0) set_unsat(c, ABS(l[0]));
    return und == 1 ? unit : 0u;
}

// Claims u (0: none); true when it is newly assigned, opposite: a conflict.
DEV bool prop_assign(const Ctx& c, u32 u) {
    if (!u) return false;
    const u32 old = atomicCAS(&c.asg[ABS(u)], 0u, u);
    if (old == FLIP(u)) set_unsat(c, ABS(u));
    return old == 0;
}

// Lists longer than PROP_PART entries are cut: the first part is walked at once, the
// others go to the part list (literal << 32 | first entry) and are walked by all warps
// in the next wave, so a hub's list is not one warp's critical path.
constexpr u32 PROP_PART = 128;
// Walks of a warp in one wave, and the list entries of a walk after the first: what is
// past them goes to the next wave, where all warps share it. Measured on the unrolled AIG
// above: 1 walk a wave 8.3 ms (every link a barrier), 2 4.8, 4 3.7, 8 4.2, 16 5.4 (few warps
// with most of the work); 32, 64 and 96 entries at 4 walks 3.74, 3.89 and 4.04 ms.
constexpr u32 PROP_STEPS = 4;
constexpr u32 PROP_CAP = 32;
constexpr u32 PROP_OUT = 64;  // newly assigned literals that a warp stages before it writes them to the trail

struct PropOut {
    u32* pend;    // the next wave's literals
    u32* npend;
    u64* parts;   // the next wave's list parts
    u32* nparts;
    u32 cap_parts;
};
// A warp's shared words: the literals it assigned (to go to the trail), and the ones it
// walks next.
struct PropWarp {
    u32 out[PROP_OUT];
    u32 q[32];
};

// The staged literals to the trail, and with o to the next wave's.
DEV void prop_flush(const Ctx& c, PropWarp& s, u32& nout, const PropOut* o = nullptr) {
    const u32 lane = threadIdx.x & 31u;
    __syncwarp();
    if (!nout) return;
    u32 base = 0, pb = 0;
    if (lane == 0) {
        base = atomicAdd(c.ntrail, nout);
        if (o) pb = atomicAdd(o->npend, nout);
    }
    base = __shfl_sync(kFull, base, 0);
    pb = __shfl_sync(kFull, pb, 0);
    for (u32 i = lane; i < nout; i += 32) {
        const u32 u = s.out[i];
        c.trail[base + i] = u;
        if (o) o->pend[pb + i] = u;
        proof_line(c, &u, 1);  // learnUnit's proof.addUnit (src/cpu/solve.h:475-479)
    }
    nout = 0;
    __syncwarp();
}
// Stages the lanes' newly assigned literals; a full stage goes out first.
DEV u32 prop_stage(const Ctx& c, PropWarp& s, u32& nout, bool fresh, u32 u, const PropOut* o = nullptr) {
    const u32 m = __ballot_sync(kFull, fresh);
    if (!m) return 0;
    const u32 cnt = (u32)__popc(m);
    if (nout + cnt > PROP_OUT) prop_flush(c, s, nout, o);
    if (fresh) s.out[nout + (u32)__popc(m & ((1u << (threadIdx.x & 31u)) - 1u))] = u;
    nout += cnt;
    return m;
}

// The parts of a list of n > PROP_PART entries from entry s0 on, but the first.
DEV void prop_cut(const Ctx& c, const PropOut& o, u32 t, u32 s0, u32 n) {
    const u32 k = (n - 1u) / PROP_PART;
    const u32 at = atomicAdd(o.nparts, k);
    for (u32 i = 0; i < k; i++) {
        if (at + i < o.cap_parts) o.parts[at + i] = (u64)t << 32 | (s0 + (i + 1u) * PROP_PART);
        else set_err(c, ERR_CAP_SCRATCH);
    }
}

// Owner of entry j among the lanes' ranges (incl: inclusive prefix of their lengths).
DEV u32 prop_owner(u32 incl, u32 j) {
    u32 k = 0;  // the first lane with incl > j
#pragma unroll
    for (u32 step = 16; step; step >>= 1) {
        const u32 x = __shfl_sync(kFull, incl, k + step - 1);
        if (x <= j) k += step;
    }
    return k & 31u;
}
DEV u32 prop_prefix(u32 n) {
    const u32 lane = threadIdx.x & 31u;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const u32 x = __shfl_up_sync(kFull, n, d);
        if ((int)lane >= d) n += x;
    }
    return n;
}

// Up to 32 literals of one warp (lane i: true literal t, 0 none; its lists seen as one
// range from entry s0 on: first ot[-t], whose clauses are judged, then ot[t], whose
// clauses are deleted): the entries of all of them are walked by consecutive lanes.
// cap: entries at most; the literals past them go to the next wave. The newly assigned
// literals are left in s.q (their number returned), what does not fit goes to the next
// wave.
DEV u32 prop_walk(const Ctx& c, const PropOut& o, PropWarp& s, u32& nout, u32 t, u32 s0, bool cut, u32 cap) {
    const u32 lane = threadIdx.x & 31u;
    u32 fo = 0, to = 0, fs = 0, n = 0;
    if (t) {
        const u32 f = FLIP(t);
        fo = c.ot_off[f];
        to = c.ot_off[t];
        fs = c.ot_size[f];
        n = fs + c.ot_size[t] - s0;
    }
    u32 incl = prop_prefix(n);
    if (incl > cap) {  // (the first ones' prefixes are the smaller)
        o.pend[atomicAdd(o.npend, 1u)] = t;
        t = 0;
        n = 0;
    } else if (n > PROP_PART) {
        if (cut) prop_cut(c, o, t, s0, n);
        n = PROP_PART;
    }
    __syncwarp();
    incl = prop_prefix(n);
    const u32 excl = incl - n;
    const u32 total = __shfl_sync(kFull, incl, 31);
    u32 nq = 0;
    for (u32 base = 0; base < total; base += 32) {
        const u32 j = base + lane;
        const u32 k = prop_owner(incl, j);
        const u32 e = j - __shfl_sync(kFull, excl, k) + __shfl_sync(kFull, s0, k);
        const u32 kfs = __shfl_sync(kFull, fs, k), kfo = __shfl_sync(kFull, fo, k), kto = __shfl_sync(kFull, to, k);
        u32 u = 0;
        if (j < total) {
            if (e < kfs) {
                u = prop_judge(c, c.ot_refs[kfo + e]);
            } else {
                const u32 r = c.ot_refs[kto + (e - kfs)];
                const u32 fl = c.hdr[r].flags;
                if (!h_deleted(fl)) {
                    c.hdr[r].flags = (fl & ~3u) | ST_DELETED;
                    touch(c, r);
                }
            }
        }
        const bool fresh = prop_assign(c, u);
        const u32 m = prop_stage(c, s, nout, fresh, u);
        if (!m) continue;
        const u32 cnt = (u32)__popc(m), rank = (u32)__popc(m & ((1u << lane) - 1u));
        const u32 fit = nq < 32u ? (cnt < 32u - nq ? cnt : 32u - nq) : 0u;
        u32 g = 0;
        if (lane == 0 && cnt > fit) g = atomicAdd(o.npend, cnt - fit);
        g = __shfl_sync(kFull, g, 0);
        if (fresh) {
            if (rank < fit) s.q[nq + rank] = u;
            else o.pend[g + rank - fit] = u;
        }
        nq += fit;
    }
    return nq;
}

// A warp walks its literals, then the ones that its walk assigned, and so on: a chain of
// implications costs a walk a link, not a grid barrier a link.
DEV void prop_chase(const Ctx& c, const PropOut& o, PropWarp& s, u32 t, u32 s0, bool cut) {
    const u32 lane = threadIdx.x & 31u;
    u32 nout = 0;
    u32 nq = prop_walk(c, o, s, nout, t, s0, cut, 0xFFFFFFFFu);
    for (u32 step = 1; step < PROP_STEPS && nq; step++) {
        __syncwarp();
        const u32 x = lane < nq ? s.q[lane] : 0u;
        __syncwarp();
        nq = prop_walk(c, o, s, nout, x, 0, true, PROP_CAP);
    }
    prop_flush(c, s, nout);
    if (nq) {
        u32 g = 0;
        if (lane == 0) g = atomicAdd(o.npend, nq);
        g = __shfl_sync(kFull, g, 0);
        if (lane < nq) o.pend[g + lane] = s.q[lane];
        __syncwarp();
    }
}

// Header of clause r as another block may have left it; of no clause: deleted.
DEV Hdr prop_hdr(const Ctx& c, u32 r, bool has) {
    Hdr h;
    h.start = h.size = h.sig = 0;
    h.flags = ST_DELETED;
    if (has) {
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(&c.hdr[r]));
        h.start = v.x;
        h.size = v.y;
        h.sig = v.z;
        h.flags = v.w;
    }
    return h;
}
// k_prop_clause (Always) or k_prop_sweep (not Always) for up to 32 clauses by one
// warp: lane i holds the header of clause r; the live clauses' literals are then read and valued by consecutive lanes, 32 literals of the
// warp's clauses per step, and each literal's value is read once. Every literal that
// is not false moves down to its place among its clause's kept literals (it is
// written only when its place changes, so a clause without false literals is not
// written), its signature bit goes to the clause's word in shared memory, and lane i
// learns from the step's ballots whether its clause has a true literal and how many
// false ones. A clause with a true literal is deleted (its literal contents do not
// matter then); otherwise, when it had false literals (or always, for Always), its
// header takes the kept size and signature, as the per-thread versions leave it.
// Returns the literal of a clause left with one, or 0.
// sm: 3 words per thread of the block (signature, unit, first variable of a clause).
template <bool Always>
DEV u32 prop_warp_clauses(const PropArgs& a, u32* sm, u32 r, Hdr h) {
    const Ctx& c = a.c;
    const u32 lane = threadIdx.x & 31u, wb = threadIdx.x & ~31u;
    u32* s_sig = sm;
    u32* s_unit = sm + blockDim.x;
    u32* s_v0 = sm + 2 * blockDim.x;
    const bool live = !h_deleted(h.flags);
    const u32 sz = live ? h.size : 0u;
    u32 incl = sz;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const u32 t = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)lane >= o) incl += t;
    }
    const u32 excl = incl - sz;
    const u32 total = __shfl_sync(0xffffffffu, incl, 31);
    s_sig[wb + lane] = 0;
    __syncwarp();
    bool sat = false;
    u32 nfalse = 0, kept = 0;
    for (u32 base = 0; base < total; base += 32) {
        const u32 j = base + lane;
        u32 k = 0;  // the lane whose clause holds literal j: the first with incl > j
#pragma unroll
        for (u32 step = 16; step; step >>= 1) {
            const u32 v = __shfl_sync(0xffffffffu, incl, k + step - 1);
            if (v <= j) k += step;
        }
        k &= 31u;
        const u32 st = __shfl_sync(0xffffffffu, h.start, k), ex = __shfl_sync(0xffffffffu, excl, k);
        const u32 kc = __shfl_sync(0xffffffffu, kept, k);  // the clause's literals kept in earlier steps
        const bool in = j < total;
        const u32 lit = in ? __ldcg(&c.lits[st + (j - ex)]) : 0u;
        const int val = in ? lit_value(c, lit) : VAL_UNDEF;
        const bool keep = in && val != 0;
        const u32 bt = __ballot_sync(0xffffffffu, in && val == 1), bf = __ballot_sync(0xffffffffu, in && val == 0);
        const u32 bk = __ballot_sync(0xffffffffu, keep);
        if (in) {
            const u32 pos = j - ex;  // place in the clause
            if (pos == 0) s_v0[wb + k] = ABS(lit);
            if (keep) {
                // the clause's lanes of this step start at lane max(ex - base, 0)
                const u32 lo = ex > base ? ex - base : 0u;
                const u32 below = bk & ((1u << lane) - 1u) & ~((1u << lo) - 1u);
                const u32 p = kc + (u32)__popc(below);
                if (p != pos) c.lits[st + p] = lit;
                if (p == 0) s_unit[wb + k] = lit;
                atomicOr(&s_sig[wb + k], MAPHASH(lit));
            }
        }
        // this lane's literals in the step: [excl - base, incl - base) clipped to the warp
        const int lo = max((int)excl - (int)base, 0), hi = min((int)incl - (int)base, 32);
        if (lo < hi) {
            const u32 m = (hi - lo == 32 ? 0xffffffffu : ((1u << (hi - lo)) - 1u)) << lo;
            sat |= (bt & m) != 0;
            nfalse += (u32)__popc(bf & m);
            kept += (u32)__popc(bk & m);
        }
    }
    __syncwarp();
    if (!live) return 0;
    if (sat) {
        c.hdr[r].flags = (h.flags & ~3u) | ST_DELETED;
        touch(c, r);
        return 0;
    }
    if (!Always && !nfalse) return 0;
    const u32 n = kept;
    h.size = n;
    h.sig = s_sig[wb + lane];
    c.hdr[r] = h;
    touch(c, r);
    if (n == 0) {
        set_unsat(c, s_v0[wb + lane]);  // names the formula the clause emptied in
        if (c.var_fid) {
            c.hdr[r].flags = (h.flags & ~3u) | ST_DELETED;
            touch(c, r);
        }
        return 0;
    }
    return n == 1 ? s_unit[wb + lane] : 0u;
}

// The strip of the clauses that hold -t for the lanes' true literals t (list entries from
// s0 on, as prop_walk's): each live one is taken once (cl_stamp), loses its false
// literals, and a unit it leaves (one that no walk saw) goes to the next wave.
DEV void prop_strip(const PropArgs& a, const PropOut& o, u32* sm, PropWarp& s, u32 stamp, u32 t, u32 s0, bool cut) {
    const Ctx& c = a.c;
    const u32 lane = threadIdx.x & 31u;
    u32 fo = 0, n = 0, nout = 0;
    if (t) {
        fo = c.ot_off[FLIP(t)] + s0;
        n = c.ot_size[FLIP(t)] - s0;
    }
    if (n > PROP_PART) {
        if (cut) prop_cut(c, o, t, s0, n);
        n = PROP_PART;
    }
    __syncwarp();
    const u32 incl = prop_prefix(n), excl = incl - n, total = __shfl_sync(kFull, incl, 31);
    for (u32 base = 0; base < total; base += 32) {
        const u32 j = base + lane;
        const u32 k = prop_owner(incl, j);
        const u32 kex = __shfl_sync(kFull, excl, k), kfo = __shfl_sync(kFull, fo, k);
        u32 r = 0;
        bool take = false;
        if (j < total) {
            r = c.ot_refs[kfo + (j - kex)];
            take = !h_deleted(__ldcg(&c.hdr[r].flags)) && atomicExch(&a.cl_stamp[r], stamp) != stamp;
        }
        const u32 u = prop_warp_clauses<true>(a, sm, r, prop_hdr(c, r, take));
        prop_stage(c, s, nout, prop_assign(c, u), u, &o);
    }
    prop_flush(c, s, nout, &o);
}

// A whole propagation in one cooperative launch. A wave takes the pending literals: list
// walks by warps, each of which goes on with the literals that it assigns itself
// (prop_chase), or one sweep over the store when the pending lists cover a large part of
// it. The walks only judge and delete clauses; once nothing is pending, a strip takes the
// false literals out of the clauses that a sweep has not stripped already, and every
// clause it strips is looked at once more under the whole assignment, so nothing depends
// on what a walk saw of another walk's assignments. The lists of the assigned literals
// end empty. A wave of walks is one barrier.
//
// What bounds it: a narrow cascade is a chain of some seven dependent loads and an atomic
// a link; a wide one the random sectors of headers, literals and values, and a sweep's
// latency (hence four groups' headers in flight). Before, a wave collected clauses, crossed
// a barrier and stripped them at once. Device time before and now: 1.1M-clause unrolled
// AIG (a cascade 580 links deep, some 600 literals wide) 10.6 and 3.7 ms; community formula
// with 80M clauses, 10.2M literals assigned, 11.8 and 8.4 ms; with 8M clauses 1.87 and 0.94.
struct PropWaves {
    u32* pend[2];       // pending literals of odd and even waves
    u64* parts[2];      // list parts
    u32* ctr;           // three sets of two counters: pending literals, parts
    u32* bar;           // grid barrier words
    u32* waves;         // out: waves run
    u32 max_waves;
    u32 sweep_scale;    // mean occurrences per literal x sweep divisor (0: never sweep)
    u32 sweep_div;
    u32* trace;         // optional: per wave [pending, parts | sweep << 31, start (ns / 1024)]
    u32 trace_cap;      // waves the trace holds
    u32 cap_parts;
    u32* tail;          // the trail's length at the start of the wave (set before the launch
                        // and by the barrier that ends each wave)
};

// Blocks per SM by the store's size: on a small one most waves are small and the barrier
// between them costs an arrival per block; on a large one sweeps and wide walks want every
// warp the registers allow. Propagation at 1, 2, 4 and 6 blocks an SM: 1.1M-clause unrolled
// AIG 3.5, 3.2, 3.7 and 4.9 ms; 120k clauses with learnt ones 186, 201, 268 and 340 us; 8M
// community clauses 2.48, 1.41, 0.93 and 0.92 ms; 80M 26.1, 14.0, 8.4 and 7.1.
constexpr u32 PROP_LARGE = 1u << 22;  // clauses
constexpr int PROP_BLOCKS_SMALL = 2, PROP_BLOCKS_LARGE = 6;
template <int MinBlocks>
__global__ void __launch_bounds__(256, MinBlocks) prop_waves_k(PropArgs a, PropWaves w) {
    __shared__ u32 sm[3 * 256];
    __shared__ PropWarp pw[8];
    const u32 tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    const u32 lane = threadIdx.x & 31u, nwarps = nth >> 5;
    // consecutive warp numbers on different SMs: a few literals spread over the chip
    const u32 warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    PropWarp& s = pw[threadIdx.x >> 5];
    u32 strip_from = a.head;  // trail literals from here on are still to be stripped
    u32 strip_end = a.head;   // while a strip's list parts are left: the literals it took end here
    u32 stamp = a.stamp;      // of the strip
    u32 wave = 0, walks = 0;
    for (;; wave++) {
        const u32 cur = wave % 3, nxt = (wave + 1) % 3, old = (wave + 2) % 3;
        const u32 tail = vload(w.tail);
        const u32 np = wave ? vload(&w.ctr[2 * cur]) : tail - a.head;
        const u32 nq = vload(&w.ctr[2 * cur + 1]);
        if (!nq) strip_from = strip_end;
        const bool stripping = strip_end != strip_from;  // the last wave was a strip: nq are its parts
        if (!np && !nq && tail == strip_from && !stripping) break;
        // walks and sweeps count against the bound, one more than level by level: the parts of
        // a list come a wave after its front
        if ((np || nq) && !stripping && walks++ > w.max_waves) {
            if (tid == 0) atomicOr(a.c.err, ERR_ITER);
            return;
        }
        if (tid == 0) w.ctr[2 * old] = w.ctr[2 * old + 1] = 0;
        const bool odd = wave & 1;
        const u32* pend = odd ? w.pend[1] : w.pend[0];
        const u64* parts = odd ? w.parts[1] : w.parts[0];
        PropOut o;
        o.pend = odd ? w.pend[0] : w.pend[1];
        o.parts = odd ? w.parts[0] : w.parts[1];
        o.npend = &w.ctr[2 * nxt];
        o.nparts = &w.ctr[2 * nxt + 1];
        o.cap_parts = w.cap_parts;
        const bool sweep = !stripping && (np || nq) && w.sweep_scale &&
                           (u64)np * w.sweep_scale + (u64)nq * PROP_PART * w.sweep_div > (u64)a.c.ncls;
        if (tid == 0 && w.trace && wave < w.trace_cap) {
            w.trace[3 * wave] = np;
            w.trace[3 * wave + 1] = nq | (sweep ? 1u << 31 : 0u);
            w.trace[3 * wave + 2] = (u32)(global_ns() >> 10);
        }
        // as many literals a warp as spread them over all warps
        auto spread = [&](u32 n) { return n <= nwarps ? 1u : n >= 32u * nwarps ? 32u : (n + nwarps - 1u) / nwarps; };
        const u32 per = spread(np);
        if (sweep) {
            u32 nout = 0;
            // four groups' headers in flight
            const u32 ng = (a.c.ncls + 31u) / 32u;
            for (u32 g0 = tid >> 5; g0 < ng; g0 += 4u * nwarps) {
                Hdr h[4];
#pragma unroll
                for (u32 k = 0; k < 4; k++) {
                    const u64 r = ((u64)g0 + (u64)k * nwarps) * 32u + lane;
                    h[k] = prop_hdr(a.c, (u32)r, r < a.c.ncls);
                }
#pragma unroll
                for (u32 k = 0; k < 4; k++) {
                    if (!__any_sync(kFull, !h_deleted(h[k].flags))) continue;
                    const u32 u = prop_warp_clauses<false>(a, sm, (g0 + k * nwarps) * 32u + lane, h[k]);
                    prop_stage(a.c, s, nout, prop_assign(a.c, u), u, &o);
                }
            }
            prop_flush(a.c, s, nout, &o);
            strip_from = strip_end = tail;
        } else if (stripping) {
            for (u32 i = warp; i < nq; i += nwarps) {
                const u64 x = __ldcg(&parts[i]);
                prop_strip(a, o, sm, s, stamp, lane ? 0u : (u32)(x >> 32), lane ? 0u : (u32)x, false);
            }
            // units that the strip itself found wait for their walk (none in theory)
            for (u32 i = tid; i < np; i += nth) o.pend[atomicAdd(o.npend, 1u)] = __ldcg(&pend[i]);
            strip_from = strip_end;
        } else if (!np && !nq) {
            const u32 ns = tail - strip_from, each = spread(ns);
            stamp = a.stamp + wave;
            for (u32 i = warp * each; i < ns; i += nwarps * each) {
                const bool has = lane < each && i + lane < ns;
                prop_strip(a, o, sm, s, stamp, has ? __ldcg(&a.c.trail[strip_from + i + lane]) : 0u, 0, true);
            }
            strip_end = tail;
        } else {
            for (u32 i = warp; i < nq; i += nwarps) {
                const u64 x = __ldcg(&parts[i]);
                prop_chase(a.c, o, s, lane ? 0u : (u32)(x >> 32), lane ? 0u : (u32)x, false);
            }
            for (u32 i = warp * per; i < np; i += nwarps * per) {
                const bool has = lane < per && i + lane < np;
                const u32 t = !has ? 0u : wave ? __ldcg(&pend[i + lane]) : a.c.trail[a.head + i + lane];
                prop_chase(a.c, o, s, t, 0, true);
            }
        }
        if (!grid_barrier(w.bar, a.c.err, a.c.ntrail, w.tail)) return;
    }
    if (tid == 0) *w.waves = wave;
    for (u32 i = a.head + tid; i < strip_from; i += nth) {
        const u32 t = __ldcg(&a.c.trail[i]);
        a.c.ot_size[t] = 0;
        a.c.ot_size[FLIP(t)] = 0;
    }
}
#endif

// reduceOT (src/cpu/simplify.cpp:58-79), run after propagation when SUB is off:
// drop deleted clauses from every list.
HD void k_reduce_list(const Ctx& c, u32 l) {
    const u32 o = c.ot_off[l], s = c.ot_size[l];
    u32 j = 0;
    for (u32 i = 0; i < s; i++) {
        const u32 r = c.ot_refs[o + i];
        if (!h_deleted(c.hdr[r].flags)) c.ot_refs[o + j++] = r;
    }
    c.ot_size[l] = j;
}

}  // namespace sigma
