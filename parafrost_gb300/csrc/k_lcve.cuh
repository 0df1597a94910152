// LCVE election: ParaFROST::LCVE + depFreeze (src/cpu/lcve.cpp:46-100), with the
// variable order of varReorder (lcve.cpp:25-44, histogram.h:32-41, key.h:57-66).
//
// The reference walks candidates in (score, variable) order, skips eliminated,
// zero-occurrence and frozen ones, stops at the first candidate whose two lists
// reach the freezing temperatures (pt, nt), elects the rest and freezes every
// neighbour v with ps[v] < pt or ns[v] < nt. Writing F for those freezable
// variables, the elected set is the lexicographically-first independent set of
// the co-occurrence graph restricted to F, in rank order, cut at the break
// candidate B = the first valid candidate that is either outside F (it is never
// frozen and its lists are necessarily long) or an independent-set member whose
// lists reach the temperatures. The independent set is the greedy one in rank
// order (a vertex joins when every lower-ranked neighbour is out, leaves when one
// lower-ranked neighbour is in), decided by push/pull rounds over the graph
// (mis_rounds_k below).
#pragma once

#include "cnf.cuh"
#include "prims.cuh"

namespace sigma {

// Independent-set word of a variable, read by every neighbour test: bits 0-29 the
// variable's rank if it is a vertex of the graph (MIS_NO_RANK otherwise; never
// changes while the set is decided), bits 30-31 the decision. Four bytes a
// variable keep the words of a 20M-variable graph (80 MB) in L2 while the walks
// stream clause records past them. Where a vertex's last pull walk stopped (an
// index into its two lists) is a separate word that only the vertex's walk reads.
enum : u32 { MIS_UNDECIDED = 0, MIS_IN = 1, MIS_OUT = 2 };
constexpr u32 MIS_NO_RANK = 0x3FFFFFFFu;
HD u32 mis_rank(u32 w) { return w & MIS_NO_RANK; }
HD u32 mis_dec(u32 w) { return w >> 30; }
HD u32 mis_dec_bits(u32 d) { return d << 30; }

struct LcveArgs {
    Ctx c;
    u32 pt, nt;           // mu_pos << mu_inc, mu_neg << mu_inc
    u32* score;           // nvars+1 (stage dumps)
    u32* cand;            // candidates in variable order (lcve_class in the top bits)
    u32* order;           // the same in (score, variable) order
    u32 ncand;
    bool dirty;           // ps/ns hold the occurrences (else the lists' sizes are they)
    bool all;             // every variable is listed (stage dumps record the whole order)
    u32* max_score;
    u32* key;             // the candidates' scores
    u32* word;            // nvars+1: independent-set words
    u32* resume;          // nvars+1: where each vertex's last pull walk stopped
    const Q4* crec;       // per clause: its first three literals and size | deleted << 31
    u64* ws_bytes;        // kSpreadSlots words summing the graph's working set (4*occ + sum(8 + 4*len))
    u32* bound;           // per formula f: [2f] = B0 (first valid non-F rank), [2f+1] = B
    const u32* f_active;  // batches: formulas taking part in this election (null: all)
    u32* f_npvs;          // batches: elected variables per formula, counted up to lcve_min (at least 1)
    u32 lcve_min;
    u32 nform;            // formulas (1 without a batch)
    u32* pvs;             // elected variables in rank order
    u64 pf = 0, pl = 0;   // L2 policies in the rounds kernel: streams go first, words last
    u32* cmin;            // per clause: the least rank of its graph vertices (MIS_NO_RANK when
                          // it has none or is deleted), built with the clause records
};

// A listed variable carries its class in the two bits above its number (numbers stay
// below 2^30), so the passes over the candidates read nothing else of it.
enum : u32 { LC_FIXED = 0, LC_SMALL = 1, LC_BIG = 2, LC_INVALID = 3 };
constexpr u32 LC_VAR = 0x3FFFFFFFu;
HD u32 lc_var(u32 x) { return x & LC_VAR; }
HD u32 lc_class(u32 x) { return x >> 30; }

HD u32 lcve_ps(const LcveArgs& a, u32 v) { return a.dirty ? a.c.ps[v] : a.c.ot_size[V2L(v)]; }
HD u32 lcve_ns(const LcveArgs& a, u32 v) { return a.dirty ? a.c.ns[v] : a.c.ot_size[NEG(V2L(v))]; }

// The candidates, in variable order: variables that occur, are not eliminated and belong
// to a formula taking part, with their scores (write_scores, histogram.h:32-41: ps*ns,
// 32-bit wrap) as sort keys. The others cannot be elected, bound the election or be a
// neighbour in a live clause, so every later pass of the election runs over the
// candidates alone: a formula that has shrunk costs what is left of it, not its
// variable count (elections without their rounds, six phases over 20M variables of a
// community formula that shrinks to 180 clauses: 13.4 ms over all variables, 7.9 over
// the candidates; a 6.8M-clause AIG 2.1 and 1.4 ms). The largest score goes to max_score (it sets how many radix passes
// the order needs). One scan over the variables (value, then put).
// Class: not freezable (a bound of the election), or freezable with short or long lists.
constexpr u32 MIS_WARP_MIN_OCC = 32;
struct LcveCand {
    LcveArgs a;
    struct State { u32 max_score = 0; };
    static constexpr int kItems = 8;
    HD u32 value(size_t i, State& st) const {
        const u32 v = (u32)i + 1u;
        const u32 p = lcve_ps(a, v), n = lcve_ns(a, v);
        const bool valid = (p || n) && !a.c.vstate[v] && (!a.f_active || a.f_active[fid_of(a.c, v)]);
        a.word[v] = MIS_NO_RANK;
        if (a.all) a.score[v] = p * n;
        if ((valid || a.all) && p * n > st.max_score) st.max_score = p * n;
        return valid || a.all;
    }
    HD void done(const State& st) const { warp_max_atomic(a.max_score, st.max_score); }
    HD void put(size_t i, u32 take, u32 at) const {
        if (!take) return;
        const u32 v = (u32)i + 1u;
        const u32 p = lcve_ps(a, v), n = lcve_ns(a, v);
        u32 cl = LC_FIXED;
        if (a.all && (!(p || n) || a.c.vstate[v])) cl = LC_INVALID;
        else if (p < a.pt || n < a.nt)
            cl = a.c.ot_size[V2L(v)] + a.c.ot_size[NEG(V2L(v))] > MIS_WARP_MIN_OCC ? LC_BIG : LC_SMALL;
        a.key[at] = p * n;
        a.cand[at] = a.order[at] = v | cl << 30;
    }
};

// Place p of the order: a freezable variable's word takes its rank; B0 = first valid
// candidate outside F.
HD void k_rank(const LcveArgs& a, u32 p) {
    const u32 x = a.order[p], cl = lc_class(x), v = lc_var(x);
    if (cl == LC_FIXED) atom_min(&a.bound[2 * fid_of(a.c, v)], p);
    else if (cl != LC_INVALID) a.word[v] = p;
}

// The independent set is decided in rounds. In a round every undecided vertex walks its
// live clauses, from where its last walk stopped, looking at its lower-ranked graph
// neighbours; the first one that is not out stops the walk (the vertex stays undecided
// and resumes there), and a walk that reaches the end finds every lower neighbour out,
// so the vertex goes in and marks its undecided higher-ranked neighbours out.
// A vertex goes in exactly when all its lower neighbours are out, and out when a
// lower neighbour is in, as in the greedy walk in rank order. Both are final and true
// whenever they are found, so the marks need no phase of their own and a walk may see
// decisions of its own round: the set does not depend on the schedule. Out is final, so
// the clauses a walk has passed never need another look. Vertices with more than
// MIS_WARP_MIN_OCC clauses are walked by a whole warp; the others by one thread,
// or by a group of lanes when few of them are left (mis_lanes).
struct MisFront {
    u32* small;   // list of small-adjacency vertices
    u32* nsmall;
    u32* big;     // list of large-adjacency vertices
    u32* nbig;
};

// Graph membership of candidate i (in variable order, so that the walks of neighbouring
// vertices read neighbouring lists): freezable and before the first bound. Every graph
// vertex starts on the undecided lists. The election's bound starts at B0.
HD bool mis_vertex(const LcveArgs& a, u32 i, u32& v, bool& big) {
    if (i < a.nform) a.bound[2 * i + 1] = a.bound[2 * i];
    if (i >= a.ncand) return false;
    const u32 x = a.cand[i], cl = lc_class(x);
    v = lc_var(x);
    big = cl == LC_BIG;
    if (cl != LC_SMALL && cl != LC_BIG) return false;
    if (a.word[v] >= a.bound[2 * fid_of(a.c, v)]) {
        a.word[v] = MIS_NO_RANK;
        return false;
    }
    a.resume[v] = 0;
    return true;
}

#if !SIGMA_CUDA
HD void k_mis_init(const LcveArgs& a, const MisFront& und, u32 i) {
    u32 v = 0;
    bool big = false;
    if (!mis_vertex(a, i, v, big)) return;
    if (big) und.big[atom_add(und.nbig, 1u)] = v;
    else und.small[atom_add(und.nsmall, 1u)] = v;
}
#else
// k_mis_init over n >= max(ncand, nform) items with block-wide appends: a block takes 256
// consecutive candidates a step, ranks its small and big vertices by warp ballots and
// reserves both lists' places with one atomic each (the lists' two counters would
// otherwise take one atomic per warp step over 20M candidates).
__global__ void __launch_bounds__(256) mis_init_k(LcveArgs a, MisFront und, u32 n) {
    __shared__ u32 ws[8], wb[8], base_s, base_b;
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (u32 i0 = blockIdx.x * 256u; i0 < n; i0 += gridDim.x * 256u) {
        u32 v = 0;
        bool big = false;
        const bool in = mis_vertex(a, i0 + threadIdx.x, v, big);
        const bool small = in && !big;
        big = in && big;
        const u32 ms = __ballot_sync(kFull, small), mb = __ballot_sync(kFull, big);
        if (lane == 0) {
            ws[warp] = (u32)__popc(ms);
            wb[warp] = (u32)__popc(mb);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            u32 ts = 0, tb = 0;
            for (u32 k = 0; k < 8; k++) {
                const u32 xs = ws[k], xb = wb[k];
                ws[k] = ts;
                wb[k] = tb;
                ts += xs;
                tb += xb;
            }
            base_s = ts ? atomicAdd(und.nsmall, ts) : 0u;
            base_b = tb ? atomicAdd(und.nbig, tb) : 0u;
        }
        __syncthreads();
        const u32 below = (1u << lane) - 1u;
        if (small) und.small[base_s + ws[warp] + (u32)__popc(ms & below)] = v;
        if (big) und.big[base_b + wb[warp] + (u32)__popc(mb & below)] = v;
        __syncthreads();
    }
}
#endif

// The clause walks read literals four at a time, so the loads (and the pushes'
// atomics) of a chunk are in flight together. Clauses and lists are not written
// while the independent set is decided.
constexpr u32 MIS_CHUNK = 4;

// A clause as the election reads it: one 16-byte record holding its first three
// literals and its size and deleted bit (built once per election), so
// clauses of up to three literals cost one load; longer ones read the rest of
// their literals from the store.
// In the first round no vertex is out yet, so a clause stops a walk of v exactly when
// one of its graph vertices ranks below v: when its least rank (cmin) is below v's.
// The first round's walks then load one word per clause (kept in q.x) instead of the
// record and the neighbours' words.
struct MisCl {
    Q4 q;
    u32 r;
    bool r0;
    HD bool deleted() const { return !r0 && (q.w >> 31) != 0; }
    HD u32 size() const { return q.w & 0x7FFFFFFFu; }
};
HD MisCl mis_cl(const LcveArgs& a, u32 r, bool r0) {
    MisCl cl;
    cl.r = r;
    cl.r0 = r0;
    if (r0) {
        cl.q.x = ldro_hint(&a.cmin[r], a.pf);
        cl.q.y = cl.q.z = cl.q.w = 0;
    } else {
        cl.q = ldro4_hint(&a.crec[r], a.pf);
    }
    return cl;
}
// Literal k of the clause; L is the clause's literal array (read only for k >= 3).
HD u32 mis_lit(const MisCl& cl, const u32* L, u32 k) {
    return k == 0 ? cl.q.x : k == 1 ? cl.q.y : k == 2 ? cl.q.z : ldro(L + k);
}
HD const u32* mis_long_lits(const LcveArgs& a, const MisCl& cl) {
    return cl.size() > 3 ? a.c.lits + hdr_ro(&a.c.hdr[cl.r]).start : nullptr;
}

// The record of clause i, its least graph rank, and the graph's working set: every graph
// vertex's list entry (4 bytes) and, for a live clause, its header and literals
// (8 + 4*len) once per graph vertex in it. Runs after the graph is known.
#if !SIGMA_CUDA
HD void k_mis_rec(const LcveArgs& a, Q4* rec, u32 i) {
    const Ctx& c = a.c;
    const Hdr h = c.hdr[i];
    const u32* l = c.lits + h.start;
    Q4 q;
    q.x = h.size > 0 ? l[0] : 0u;
    q.y = h.size > 1 ? l[1] : 0u;
    q.z = h.size > 2 ? l[2] : 0u;
    q.w = h.size | (h_deleted(h.flags) ? 0x80000000u : 0u);
    rec[i] = q;
    u32 ng = 0, m = MIS_NO_RANK;
    for (u32 k = 0; k < h.size; k++) {
        const u32 rk = mis_rank(a.word[ABS(l[k])]);
        ng += rk != MIS_NO_RANK;
        if (rk < m) m = rk;
    }
    a.cmin[i] = h_deleted(h.flags) ? MIS_NO_RANK : m;
    spread_sum_add64(a.ws_bytes, (u64)ng * (4ull + (h_deleted(h.flags) ? 0ull : 8ull + 4ull * h.size)));
}
#else
// The same for 32 clauses per warp: lane i writes the record of clause id0 + i
// (coalesced 16-byte stores), and the graph working set is summed over the warp's
// literals with consecutive lanes on consecutive literals (coalesced reads), each
// literal of a graph vertex adding 4 bytes and, in a live clause, the clause's
// 8 + 4 * len bytes.
__global__ void __launch_bounds__(256) mis_rec_warp_k(LcveArgs a, Q4* rec) {
    __shared__ u32 s_min[256];  // per lane of the block: the least rank of its clause
    const u32 lane = threadIdx.x & 31u;
    const u32 nw = (gridDim.x * blockDim.x) >> 5;
    const u32 ngroups = (a.c.ncls + 31u) / 32u;
    u64 sum = 0;
    for (u32 g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ngroups; g += nw) {
        const u32 id0 = g * 32u;
        const u32 n = a.c.ncls - id0 < 32u ? a.c.ncls - id0 : 32u;
        u32 start = 0, sz = 0, weight = 0;
        bool dead = true;
        s_min[threadIdx.x] = MIS_NO_RANK;
        __syncwarp();
        if (lane < n) {
            const Hdr h = hdr_ro(&a.c.hdr[id0 + lane]);
            const u32* l = a.c.lits + h.start;
            Q4 q;
            q.x = h.size > 0 ? __ldg(&l[0]) : 0u;
            q.y = h.size > 1 ? __ldg(&l[1]) : 0u;
            q.z = h.size > 2 ? __ldg(&l[2]) : 0u;
            q.w = h.size | (h_deleted(h.flags) ? 0x80000000u : 0u);
            rec[id0 + lane] = q;
            start = h.start;
            sz = h.size;
            weight = 4u + (h_deleted(h.flags) ? 0u : 8u + 4u * h.size);
            dead = h_deleted(h.flags);
        }
        u32 incl = sz;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u32 t = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += t;
        }
        const u32 excl = incl - sz;
        const u32 total = __shfl_sync(0xffffffffu, incl, 31);
        for (u32 base = 0; base < total; base += 32) {
            const u32 j = base + lane;
            u32 k = 0;
#pragma unroll
            for (u32 step = 16; step; step >>= 1) {
                const u32 v = __shfl_sync(0xffffffffu, incl, k + step - 1);
                if (v <= j) k += step;
            }
            const u32 st = __shfl_sync(0xffffffffu, start, k & 31u), ex = __shfl_sync(0xffffffffu, excl, k & 31u);
            const u32 wt = __shfl_sync(0xffffffffu, weight, k & 31u);
            if (j < total) {
                const u32 rk = mis_rank(ldro(&a.word[ABS(__ldg(&a.c.lits[st + (j - ex)]))]));
                if (rk != MIS_NO_RANK) {
                    sum += wt;
                    atomicMin(&s_min[(threadIdx.x & ~31u) + (k & 31u)], rk);
                }
            }
        }
        __syncwarp();
        if (lane < n) a.cmin[id0 + lane] = dead ? MIS_NO_RANK : s_min[threadIdx.x];
    }
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0 && sum) atomicAdd((unsigned long long*)(a.ws_bytes + (blockIdx.x & (kSpreadSlots - 1u))),
                                    (unsigned long long)sum);
}

// The same with a thread a clause, four literals at a time: their loads, then their words'
// loads, are in flight together, and the next clause's header. A warp of the kernel above
// waits for both at every 32 literals, which more warps hide on a large store but nothing
// hides on one that does not fill the chip. Clause records of a round, warps and threads:
// 200 variables 42 and 16 us, 43k clauses 89 and 19, 1M mixed 134 and 98, a 6.8M-clause AIG 362
// and 384, 14M clauses of 384 formulas 1.11 and 1.25 ms, 80M community clauses 3.5 and 4.2:
// threads below MIS_REC_WARPS clauses.
constexpr u32 MIS_REC_WARPS = 1u << 20;
__global__ void __launch_bounds__(256) mis_rec_k(LcveArgs a, Q4* rec) {
    const u32 lane = threadIdx.x & 31u;
    const u32 step = gridDim.x * blockDim.x;
    u64 sum = 0;
    u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    Hdr h{};
    if (i < a.c.ncls) h = hdr_ro(&a.c.hdr[i]);
    for (; i < a.c.ncls;) {
        const Hdr cur = h;
        const u32 at = i;
        i = a.c.ncls - i > step ? i + step : a.c.ncls;
        if (i < a.c.ncls) h = hdr_ro(&a.c.hdr[i]);
        const u32* l = a.c.lits + cur.start;
        const bool dead = h_deleted(cur.flags);
        u32 ng = 0, m = MIS_NO_RANK;
        Q4 q;
        q.x = q.y = q.z = 0u;
        for (u32 k0 = 0; k0 < cur.size; k0 += 4) {
            u32 x[4], w[4];
#pragma unroll
            for (u32 j = 0; j < 4; j++) x[j] = k0 + j < cur.size ? __ldg(&l[k0 + j]) : 0u;
#pragma unroll
            for (u32 j = 0; j < 4; j++) w[j] = k0 + j < cur.size ? ldro(&a.word[ABS(x[j])]) : MIS_NO_RANK;
            if (!k0) {
                q.x = x[0];
                q.y = x[1];
                q.z = x[2];
            }
#pragma unroll
            for (u32 j = 0; j < 4; j++) {
                const u32 rk = mis_rank(w[j]);
                ng += rk != MIS_NO_RANK;
                m = rk < m ? rk : m;
            }
        }
        q.w = cur.size | (dead ? 0x80000000u : 0u);
        rec[at] = q;
        a.cmin[at] = dead ? MIS_NO_RANK : m;
        sum += (u64)ng * (4ull + (dead ? 0ull : 8ull + 4ull * cur.size));
    }
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0 && sum) atomicAdd((unsigned long long*)(a.ws_bytes + (blockIdx.x & (kSpreadSlots - 1u))),
                                    (unsigned long long)sum);
}
#endif

// A graph neighbour of v in clause cl that is ranked below rv and not out (0: none; a
// first-round clause only says that there is one: NONE). Decisions are read through to the
// cache level other SMs write.
HD u32 mis_blocker(const LcveArgs& a, u32 v, u32 rv, const MisCl& cl) {
    if (cl.r0) return cl.q.x < rv ? NONE : 0u;
    if (cl.deleted()) return 0;
    const u32 size = cl.size();
    const u32* L = mis_long_lits(a, cl);
    for (u32 k0 = 0; k0 < size; k0 += MIS_CHUNK) {
        u32 w[MIS_CHUNK];
#pragma unroll
        for (u32 j = 0; j < MIS_CHUNK; j++) w[j] = k0 + j < size ? ABS(mis_lit(cl, L, k0 + j)) : v;
        u32 b = 0;
#pragma unroll
        for (u32 j = 0; j < MIS_CHUNK; j++) {
            if (w[j] == v) continue;
            const u32 g = ldcg_hint(&a.word[w[j]], a.pl);
            if (mis_rank(g) < rv && mis_dec(g) != MIS_OUT) b = w[j];
        }
        if (b) return b;
    }
    return 0;
}

// Vertex v (rank rv) goes in; one whose lists reach the temperatures bounds the election
// (B = min(B0, first member whose lists reach them)).
HD void mis_goes_in(const LcveArgs& a, u32 v, u32 rv, u32 np, u32 nn) {
    atom_or(&a.word[v], mis_dec_bits(MIS_IN));
    if (np >= a.pt && nn >= a.nt) atom_min(&a.bound[2 * fid_of(a.c, v) + 1], rv);
}

// Pull walk of undecided vertex v by one thread: true when v went in; otherwise the
// resume point is stored (v stays undecided). The next clause's record is loaded
// before the current one is examined.
HD bool mis_pull_one(const LcveArgs& a, u32 v, u32 wv, bool r0) {
    const u32 rv = mis_rank(wv);
    const u32 p = V2L(v), np = a.c.ot_size[p], n = np + a.c.ot_size[p + 1];
    const u32 op = a.c.ot_off[p], on = a.c.ot_off[p + 1] - np;
    u32 t = vload(&a.resume[v]);
    if (t < n) {
        MisCl cl = mis_cl(a, ldro_hint(&a.c.ot_refs[t < np ? op + t : on + t], a.pf), r0);
        for (; t < n; t++) {
            MisCl nx = cl;
            if (t + 1 < n) nx = mis_cl(a, ldro_hint(&a.c.ot_refs[t + 1 < np ? op + t + 1 : on + t + 1], a.pf), r0);
            if (mis_blocker(a, v, rv, cl)) {
                a.resume[v] = t;
                return false;
            }
            cl = nx;
        }
    }
    mis_goes_in(a, v, rv, np, n - np);
    return true;
}

// Push of in vertex u (rank ru) through clause cl: undecided higher neighbours go
// out. The rank in a neighbour's word never changes and a decision is final, so a
// plain (possibly older) load decides whether the atomic is needed.
HD void mis_push_clause(const LcveArgs& a, u32 u, u32 ru, const MisCl& cl) {
    if (cl.deleted()) return;
    const u32 size = cl.size();
    const u32* L = mis_long_lits(a, cl);
    for (u32 k0 = 0; k0 < size; k0 += MIS_CHUNK) {
        u32 w[MIS_CHUNK];
#pragma unroll
        for (u32 j = 0; j < MIS_CHUNK; j++) w[j] = k0 + j < size ? ABS(mis_lit(cl, L, k0 + j)) : u;
#pragma unroll
        for (u32 j = 0; j < MIS_CHUNK; j++) {
            if (w[j] == u) continue;
            const u32 g = ldcg_hint(&a.word[w[j]], a.pl);
            if (mis_rank(g) != MIS_NO_RANK && mis_rank(g) > ru && mis_dec(g) == MIS_UNDECIDED)
                atom_or(&a.word[w[j]], mis_dec_bits(MIS_OUT));
        }
    }
}

#if !SIGMA_CUDA
// Serial rounds of the emulation build: what went in marks its neighbours, then the
// undecided vertices walk. (A list that has shrunk ends before the next one's start, so
// an empty positive list's first clause is the negative one's.)
HD void k_mis_push(const LcveArgs& a, const u32* in, u32 idx) {
    const u32 u = in[idx], ru = mis_rank(a.word[u]);
    const u32 p = V2L(u), np = a.c.ot_size[p], n = np + a.c.ot_size[p + 1];
    const u32 op = a.c.ot_off[p], on = a.c.ot_off[p + 1] - np;
    for (u32 t = 0; t < n; t++) mis_push_clause(a, u, ru, mis_cl(a, a.c.ot_refs[t < np ? op + t : on + t], false));
}
HD void k_mis_pull(const LcveArgs& a, const u32* in, const MisFront& und, const MisFront& ins, bool r0, u32 idx) {
    const u32 v = in[idx];
    const u32 wv = a.word[v];
    if (mis_dec(wv) != MIS_UNDECIDED) return;
    const bool big = a.c.ot_size[V2L(v)] + a.c.ot_size[NEG(V2L(v))] > MIS_WARP_MIN_OCC;
    if (mis_pull_one(a, v, wv, r0)) {
        if (big) ins.big[atom_add(ins.nbig, 1u)] = v;
        else ins.small[atom_add(ins.nsmall, 1u)] = v;
    } else {
        if (big) und.big[atom_add(und.nbig, 1u)] = v;
        else und.small[atom_add(und.nsmall, 1u)] = v;
    }
}
#else
// All rounds in one cooperative launch. Round r reads the undecided lists u[r&1]
// (lengths in counter set r%3: small, large) and writes u[(r+1)&1] through counter set
// (r+1)%3; set (r+2)%3, last read in round r-1, is cleared for round r+1. One grid
// barrier ends a round.
//
// What bounds a small election is the chain of dependent decisions: a round costs the
// barrier and some five dependent loads whatever its size. So once every undecided
// vertex has its own lanes (us * lanes <= threads), a group keeps its vertex and tries
// again up to MIS_TRIES times before the round ends, and sees its neighbours' decisions
// as they are made. Device time of a round's elections, before (a push phase and a pull
// phase a round, two barriers) and now: 200 variables 507 and 88 us (18 and 8 rounds),
// 10k-variable 3-SAT 739 and 141, 1M mixed clauses 1245 and 740, a 6.8M-clause AIG 3449
// and 2830 (50 and 23 rounds), 80M community clauses 10.9 and 8.1 ms.
struct MisRounds {
    u32* u_small[2];
    u32* u_big[2];
    u32* ctr;        // three sets of four counters (two used)
    u32* bar;        // grid barrier: [0] arrivals, [1] generation
    u32* rounds;     // out: rounds run
    u32 max_rounds;
    u32* trace;      // optional: per round [undecided small, big, start ns / 1024]
    u32 trace_cap;   // rounds the trace holds
};
constexpr u32 MIS_TRIES = 384;

// Vertices that stay undecided are staged per block in shared memory and copied to the
// next lists with one reservation per block (a vertex that finds its block's queue full
// goes to the list directly).
constexpr u32 MIS_QCAP = 1024;

struct MisBlockQueue {
    u32 small[MIS_QCAP], big[MIS_QCAP];
    u32 ns, nb, base_s, base_b;
};

DEV void mis_queue_push(MisBlockQueue& q, const MisFront& f, bool big, u32 w) {
    if (big) {
        const u32 k = atomicAdd(&q.nb, 1u);
        if (k < MIS_QCAP) q.big[k] = w;
        else f.big[atomicAdd(f.nbig, 1u)] = w;
    } else {
        const u32 k = atomicAdd(&q.ns, 1u);
        if (k < MIS_QCAP) q.small[k] = w;
        else f.small[atomicAdd(f.nsmall, 1u)] = w;
    }
}

// Append of the lanes with pred by one reservation per warp: to the block's queue
// while it has room, the rest to the list. All lanes of the warp take part.
DEV void mis_queue_warp(u32* qa, u32& qn, u32* list, u32* nlist, bool pred, u32 v) {
    const u32 lane = threadIdx.x & 31u;
    const u32 m = __ballot_sync(kFull, pred);
    if (!m) return;
    const u32 cnt = (u32)__popc(m), rank = (u32)__popc(m & ((1u << lane) - 1u));
    u32 k = 0;
    if (lane == 0) k = atomicAdd(&qn, cnt);
    k = __shfl_sync(kFull, k, 0);
    const u32 fit = k < MIS_QCAP ? (cnt < MIS_QCAP - k ? cnt : MIS_QCAP - k) : 0u;
    u32 g = 0;
    if (lane == 0 && cnt > fit) g = atomicAdd(nlist, cnt - fit);
    g = __shfl_sync(kFull, g, 0);
    if (pred) {
        if (rank < fit) qa[k + rank] = v;
        else list[g + rank - fit] = v;
    }
}

// Lanes per vertex for a phase over n small vertices and nth threads: when the list
// is short, each vertex's clauses are spread over a group of up to 32 lanes, so the
// phase waits for one clause walk per vertex instead of a whole list walked by one
// thread.
DEV u32 mis_lanes(u32 n, u32 nth) {
    u32 L = 1;
    while (L < 32u && (u64)n * (2u * L) <= nth) L *= 2u;
    return L;
}

DEV void mis_queue_flush(MisBlockQueue& q, const MisFront& f) {
    __syncthreads();
    const u32 ns = q.ns < MIS_QCAP ? q.ns : MIS_QCAP, nb = q.nb < MIS_QCAP ? q.nb : MIS_QCAP;
    if (threadIdx.x == 0) {
        q.base_s = ns ? atomicAdd(f.nsmall, ns) : 0u;
        q.base_b = nb ? atomicAdd(f.nbig, nb) : 0u;
    }
    __syncthreads();
    for (u32 i = threadIdx.x; i < ns; i += blockDim.x) f.small[q.base_s + i] = q.small[i];
    for (u32 i = threadIdx.x; i < nb; i += blockDim.x) f.big[q.base_b + i] = q.big[i];
    __syncthreads();
    if (threadIdx.x == 0) q.ns = q.nb = 0;
}

// One try at vertex v by the lanes of mask gm (sub: this lane's place among the L of
// them): clauses from `at` on, L at a time in list order, the first blocking one of a
// step (lowest lane) stops the walk. Returns true when v is decided; a walk that
// reaches the end puts v in and marks its neighbours out, the lanes sharing the clauses.
// wait: the neighbour that stopped the last try (0 or NONE: none known). Until it is
// decided only its word and v's own are looked at: one load a try instead of a walk's
// four dependent ones.
// Other blocks decide both words at any time, and the lanes' loads need not be one access:
// the group goes by what its first lane saw, so all of it takes the same branches (the
// collectives below name every lane of the group).
DEV bool mis_try(const LcveArgs& a, u32 v, u32 gm, u32 gbase, u32 sub, u32 L, u32& at, u32& wait, bool r0) {
    const u32 wv = vload(&a.word[v]);
    const bool known = wait && wait != NONE;
    const u32 ww = known ? vload(&a.word[wait]) : 0u;
    const u32 seen = __shfl_sync(gm, mis_dec(wv) | mis_dec(ww) << 2, (int)gbase);
    const u32 dv = seen & 3u, dw = seen >> 2;
    if (dv != MIS_UNDECIDED) return true;
    if (known) {
        if (dw == MIS_UNDECIDED) return false;
        if (dw == MIS_IN) {  // a lower neighbour is in
            if (sub == 0) atomicOr(&a.word[v], mis_dec_bits(MIS_OUT));
            return true;
        }
    }
    const u32 rv = mis_rank(wv);  // (a word's rank does not change)
    const u32 p = V2L(v), np = a.c.ot_size[p], n = np + a.c.ot_size[p + 1];
    const u32 op = a.c.ot_off[p], on = a.c.ot_off[p + 1] - np;
    for (u32 b0 = at; b0 < n; b0 += L) {
        const u32 t = b0 + sub;
        u32 blk = 0;
        if (t < n) blk = mis_blocker(a, v, rv, mis_cl(a, ldro_hint(&a.c.ot_refs[t < np ? op + t : on + t], a.pf), r0));
        const u32 m = (__ballot_sync(gm, blk != 0) & gm) >> gbase;
        if (m) {
            const u32 first = (u32)(__ffs(m) - 1);
            at = b0 + first;
            wait = __shfl_sync(gm, blk, (int)(gbase + first));
            return false;
        }
    }
    if (sub == 0) mis_goes_in(a, v, rv, np, n - np);
    for (u32 t = sub; t < n; t += L)
        mis_push_clause(a, v, rv, mis_cl(a, ldro_hint(&a.c.ot_refs[t < np ? op + t : on + t], a.pf), false));
    return true;
}

// The block marks out the neighbours of the vertices it put in (queue q, n of them),
// eight lanes a vertex.
DEV void mis_push_queue(const LcveArgs& a, const u32* q, u32 n) {
    const u32 sub = threadIdx.x & 7u;
    for (u32 k = threadIdx.x >> 3; k < n; k += blockDim.x >> 3) {
        const u32 u = q[k];
        const u32 ru = mis_rank(vload(&a.word[u]));
        const u32 p = V2L(u), np = a.c.ot_size[p], m = np + a.c.ot_size[p + 1];
        const u32 op = a.c.ot_off[p], on = a.c.ot_off[p + 1] - np;
        for (u32 t = sub; t < m; t += 8)
            mis_push_clause(a, u, ru, mis_cl(a, ldro_hint(&a.c.ot_refs[t < np ? op + t : on + t], a.pf), false));
    }
}

__global__ void __launch_bounds__(256, 6) mis_rounds_k(LcveArgs a0, MisRounds w) {
    LcveArgs a = a0;
    a.pf = l2_policy_first();
    a.pl = l2_policy_last();
    __shared__ MisBlockQueue qu;
    __shared__ u32 qin[MIS_QCAP];
    __shared__ u32 nin;
    const u32 tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
    const u32 lane = threadIdx.x & 31u, nwarps = nth >> 5;
    if (threadIdx.x == 0) qu.ns = qu.nb = nin = 0;
    __syncthreads();
    for (u32 r = 0;; r++) {
        // In the first round no vertex is out yet, so the walks test one word per clause.
        const bool r0 = r == 0;
        const u32 cur = r % 3, nxt = (r + 1) % 3, old = (r + 2) % 3;
        const u32 us = vload(&w.ctr[4 * cur]), ub = vload(&w.ctr[4 * cur + 1]);
        if (!us && !ub) {
            if (tid == 0) *w.rounds = r;
            return;
        }
        if (r >= w.max_rounds) {
            if (tid == 0) atomicOr(a.c.err, ERR_ITER);
            return;
        }
        if (tid == 0)
            for (u32 k = 0; k < 2; k++) w.ctr[4 * old + k] = 0;
        if (tid == 0 && w.trace && r < w.trace_cap) {
            u32* t = w.trace + 3 * r;
            t[0] = us;
            t[1] = ub;
            t[2] = (u32)(global_ns() >> 10);
        }
        MisFront fu;
        const bool odd = r & 1;
        fu.small = odd ? w.u_small[0] : w.u_small[1];
        fu.nsmall = &w.ctr[4 * nxt];
        fu.big = odd ? w.u_big[0] : w.u_big[1];
        fu.nbig = &w.ctr[4 * nxt + 1];
        // (lists written by other blocks: uncached reads)
        const u32* pu_b = odd ? w.u_big[1] : w.u_big[0];
        const u32* pu_s = odd ? w.u_small[1] : w.u_small[0];
        const u32 lu = mis_lanes(us, nth);
        const u32 sub = lane & (lu - 1u), gbase = lane - sub;
        const u32 gm = lu == 32u ? kFull : ((1u << lu) - 1u) << gbase;
        const u32 warp = tid >> 5;
        if (!r0 && (u64)us * lu <= nth && ub <= nwarps) {
            // every undecided vertex has its own lanes: try until it is decided
            const bool hb = warp < ub, hs = tid / lu < us;
            const u32 vb = hb ? vload(&pu_b[warp]) : 0u, vs = hs ? vload(&pu_s[tid / lu]) : 0u;
            u32 ab = hb ? vload(&a.resume[vb]) : 0u, as = hs ? vload(&a.resume[vs]) : 0u;
            u32 nb = 0, ns = 0;  // the neighbours that are waited for
            bool wb = hb, ws = hs;
            for (u32 k = 0; k < MIS_TRIES && __any_sync(kFull, wb || ws); k++) {
                if (wb) wb = !mis_try(a, vb, kFull, 0, lane, 32, ab, nb, false);  // warp-uniform
                if (ws) ws = !mis_try(a, vs, gm, gbase, sub, lu, as, ns, false);  // group-uniform
                __syncwarp();
            }
            if (wb && lane == 0) {
                a.resume[vb] = ab;
                mis_queue_push(qu, fu, true, vb);
            }
            if (ws && sub == 0) a.resume[vs] = as;
            mis_queue_warp(qu.small, qu.ns, fu.small, fu.nsmall, ws && sub == 0, vs);
        } else {
            for (u32 idx = warp; idx < ub; idx += nwarps) {
                const u32 v = vload(&pu_b[idx]);
                u32 at = vload(&a.resume[v]), wait = 0;
                const bool und = !mis_try(a, v, kFull, 0, lane, 32, at, wait, r0);
                if (und && lane == 0) {
                    a.resume[v] = at;
                    mis_queue_push(qu, fu, true, v);
                }
                __syncwarp();
            }
            if (lu == 1) {
                // one thread a vertex; the block's own new in vertices are staged and their
                // neighbours marked by all its threads (block-uniform trip count)
                for (u32 base = blockIdx.x * blockDim.x; base < us; base += nth) {
                    const u32 idx = base + threadIdx.x;
                    u32 v = 0;
                    bool in = false, und = false;
                    if (idx < us) {
                        v = vload(&pu_s[idx]);
                        const u32 wv = vload(&a.word[v]);
                        if (mis_dec(wv) == MIS_UNDECIDED) {
                            in = mis_pull_one(a, v, wv, r0);
                            und = !in;
                        }
                    }
                    mis_queue_warp(qu.small, qu.ns, fu.small, fu.nsmall, und, v);
                    const u32 k = warp_append(&nin, in);
                    if (in) qin[k] = v;
                    __syncthreads();
                    const u32 n = nin;
                    __syncthreads();
                    if (n > MIS_QCAP - 256u || base + nth >= us) {
                        mis_push_queue(a, qin, n);
                        if (threadIdx.x == 0) nin = 0;
                        __syncthreads();
                    }
                }
            } else {
                // a group of lu lanes a vertex
                const u32 gpw = 32u / lu;
                for (u32 base = warp * gpw; base < us; base += nwarps * gpw) {
                    const u32 idx = base + lane / lu;
                    u32 v = 0;
                    bool und = false;
                    if (idx < us) {
                        v = vload(&pu_s[idx]);
                        u32 at = vload(&a.resume[v]), wait = 0;
                        und = !mis_try(a, v, gm, gbase, sub, lu, at, wait, r0);
                        if (und && sub == 0) a.resume[v] = at;
                        und = und && sub == 0;
                    }
                    mis_queue_warp(qu.small, qu.ns, fu.small, fu.nsmall, und, v);
                }
            }
        }
        mis_queue_flush(qu, fu);
        if (!grid_barrier(w.bar, a.c.err)) return;
    }
}
#endif

// The elected variables: the members of the set below their formula's bound, in rank
// order. One scan over the order.
struct LcveElect {
    LcveArgs a;
    typedef ScanNone State;
    static constexpr int kItems = 8;
    HD void done(const State&) const {}
    HD u32 value(size_t p, State&) const {
        const u32 v = lc_var(a.order[p]);
        const u32 w = a.word[v];
        return (u32)p < a.bound[2 * fid_of(a.c, v) + 1] && mis_rank(w) != MIS_NO_RANK && mis_dec(w) == MIS_IN;
    }
    HD void put(size_t p, u32 take, u32 at) const {
        if (!take) return;
        const u32 v = lc_var(a.order[p]);
        a.pvs[at] = v;
        a.c.pvrank[v] = at;
        if (a.f_npvs) {  // one shared word per formula: counted no further than it is asked for
            u32* n = &a.f_npvs[fid_of(a.c, v)];
            if (vload(n) < a.lcve_min) atom_add(n, 1u);
        }
    }
};

}  // namespace sigma
