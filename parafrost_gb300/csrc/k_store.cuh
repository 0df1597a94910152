// Clause-store kernels: upload normalisation, occurrence-table build, survivor
// counts and compaction. Item functions run once per clause / literal slot.
#pragma once

#include "cnf.cuh"
#include "introsort.cuh"
#include "prims.cuh"

namespace sigma {

// ---------------------------------------------------------------- upload
// extract() (src/cpu/simplify.cpp:95-113; GPU: transfer.cu:24-42 + prep_cnf_k,
// kernels.cu:61-70): literals sorted ascending, signature over the clause,
// status from the learnt flag. Rejects literals out of range and clauses that
// repeat a variable. A one-literal clause is not a clause of the store: as the
// reference's parser does (src/cpu/dimacs.cpp:153-159), its literal goes to the
// trail (first claim of the variable wins; the opposite literal already there is
// a contradiction) and the clause is kept as a deleted slot; the round then
// propagates these units before its first phase.
struct UploadArgs {
    Ctx c;
    const u64* off;      // num_clauses + 1
    const uint8_t* learnt;  // may be null
    u64 base;            // literal offset of off[0]
    u64 nlits;           // literals uploaded: every clause must lie in [base, base + nlits)
    // formula batches: nf formulas, formula f holds clauses [f_cls[f], f_cls[f+1])
    // and f_nv[f] variables from f_var[f]+1 on; its literals arrive in its own
    // numbering and are moved to the batch's (nf = 0: a single formula)
    u32 nf;
    const u64* f_cls;
    const u32* f_var;
    const u32* f_nv;
};

// A short clause sorted in registers (an in-place sort waits for memory at every swap):
// all literals loaded together, a transposition network, a store where the order changed.
// Returns whether a literal is out of range or a variable repeated; sig is its signature.
// (Device-side upload of 80M community clauses 3.4 ms in place, 2.2 with the short ones in
// registers.)
constexpr u32 UPLOAD_SHORT = 8;
HD u32 upload_short(u32* l, u32 n, u32 D, u32& sig) {
    u32 x[UPLOAD_SHORT], y[UPLOAD_SHORT];
#pragma unroll
    for (u32 k = 0; k < UPLOAD_SHORT; k++) x[k] = y[k] = k < n ? l[k] : 0xFFFFFFFFu;
    // odd-even transposition: UPLOAD_SHORT rounds sort any order
#pragma unroll
    for (u32 r = 0; r < UPLOAD_SHORT; r++) {
#pragma unroll
        for (u32 k = r & 1u; k + 1 < UPLOAD_SHORT; k += 2) {
            const u32 lo = y[k] < y[k + 1] ? y[k] : y[k + 1], hi = y[k] < y[k + 1] ? y[k + 1] : y[k];
            y[k] = lo;
            y[k + 1] = hi;
        }
    }
    u32 bad = 0;
#pragma unroll
    for (u32 k = 0; k < UPLOAD_SHORT; k++) {
        if (k >= n) continue;
        bad |= y[k] < 2 || y[k] >= D || (k && ABS(y[k]) == ABS(y[k ? k - 1 : 0]));
        sig |= MAPHASH(y[k]);
        if (y[k] != x[k]) l[k] = y[k];
    }
    return bad;
}

HD void k_upload_clause(const UploadArgs& a, u32 i) {
    const u64 o0 = a.off[i], o1 = a.off[i + 1];
    // offsets that go down, or leave the uploaded literals, are rejected before
    // any literal is touched
    if (o0 < a.base || o1 < o0 || o1 - a.base > a.nlits) { set_err(a.c, ERR_INPUT); return; }
    const u64 s = o0 - a.base, e = o1 - a.base;
    u32* l = a.c.lits + s;
    const u32 n = (u32)(e - s);
    if (n == 0) { set_err(a.c, ERR_INPUT); return; }
    if (a.nf) {
        const u32 f = upper_segment(a.f_cls, a.nf, (u64)i);
        const u32 shift = 2u * a.f_var[f], lim = 2u * a.f_nv[f] + 2u;
        for (u32 k = 0; k < n; k++) {
            if (l[k] < 2 || l[k] >= lim) { set_err(a.c, ERR_INPUT); return; }
            l[k] += shift;
        }
    }
    u32 sig = 0, bad = 0;
    if (n <= UPLOAD_SHORT) bad = upload_short(l, n, a.c.D, sig);
    else {
        if (n <= 32) ref_insertion_sort(l, (int)n, LitLess());
        else std_sort_replica(l, l + n, LitLess());
        for (u32 k = 0; k < n; k++) {
            const u32 lit = l[k];
            bad |= lit < 2 || lit >= a.c.D || (k && ABS(lit) == ABS(l[k - 1]));
            sig |= MAPHASH(lit);
        }
    }
    if (bad) { set_err(a.c, ERR_INPUT); return; }
    Hdr h;
    h.start = (u32)s;
    h.size = n;
    h.sig = sig;
    h.flags = (a.learnt && a.learnt[i]) ? ST_LEARNT : ST_ORIGINAL;
    if (n == 1) {
        h.flags = ST_DELETED;
        const u32 u = l[0];
        const u32 old = atom_cas(&a.c.asg[ABS(u)], 0u, u);
        if (old == 0) a.c.trail[atom_add(a.c.ntrail, 1u)] = u;
        else if (old != u) set_unsat(a.c, ABS(u));
    }
    a.c.hdr[i] = h;
}

#if SIGMA_CUDA
// Batch upload from separate host arrays by one launch that reads them in place (devices
// that share the host's page tables): a block copies one piece of a formula's literals or
// offsets to its place in the store, offsets moved from the formula's base to the store's.
// A copy per array, each staged from pageable memory by the driver, took 9.6 ms for 384
// formulas (768 arrays, 317 MB), upload kernel included; reading them in place 3.2 ms.
constexpr u32 PART_WORDS = 1u << 15;  // literals or offsets of a piece
struct UploadPiece {
    const void* src;
    u64 dst;    // first literal or offset of the store
    u64 add;    // offsets: added to each (modulo 2^64)
    u32 n;
    u32 offsets;  // 1: 64-bit offsets, 0: 32-bit literals
};
__global__ void __launch_bounds__(256) upload_pieces_k(const UploadPiece* pieces, u32 np, u32* lits, u64* off) {
    constexpr u32 kFlight = 8;  // loads of a thread on their way over the host link
    for (u32 b = blockIdx.x; b < np; b += gridDim.x) {
        const UploadPiece p = pieces[b];
        for (u32 i0 = threadIdx.x; i0 < p.n; i0 += 256u * kFlight) {
            if (p.offsets) {
                u64 x[kFlight];
#pragma unroll
                for (u32 q = 0; q < kFlight; q++) if (i0 + 256u * q < p.n) x[q] = ((const u64*)p.src)[i0 + 256u * q];
#pragma unroll
                for (u32 q = 0; q < kFlight; q++) if (i0 + 256u * q < p.n) off[p.dst + i0 + 256u * q] = x[q] + p.add;
            } else {
                u32 x[kFlight];
#pragma unroll
                for (u32 q = 0; q < kFlight; q++) if (i0 + 256u * q < p.n) x[q] = ((const u32*)p.src)[i0 + 256u * q];
#pragma unroll
                for (u32 q = 0; q < kFlight; q++) if (i0 + 256u * q < p.n) lits[p.dst + i0 + 256u * q] = x[q];
            }
        }
    }
}
#endif

// ---------------------------------------------------------------- OT build
// createOT (src/cpu/simplify.cpp:35-56) as histogram -> exclusive scan -> scatter
// (GPU reference: histogram.cu:34-52, memory.cu:271-312, create_ot_k kernels.cu:81-96).
HD void k_hist_clause(const Ctx& c, u32 i) {
    const Hdr h = c.hdr[i];
    if (h_deleted(h.flags)) return;
    const u32* l = c.lits + h.start;
    for (u32 k = 0; k < h.size; k++) atom_add(&c.ot_size[l[k]], 1u);
}

HD void k_scatter_clause(const Ctx& c, u32 i) {
    const Hdr h = c.hdr[i];
    if (h_deleted(h.flags)) return;
    const u32* l = c.lits + h.start;
    for (u32 k = 0; k < h.size; k++) {
        const u32 pos = atom_add(&c.ot_cursor[l[k]], 1u);
        if (pos < c.ot_cap) c.ot_refs[pos] = i;
        else set_err(c, ERR_INTERNAL);
    }
}

// Standalone occurrence-table build over a clause list in CSR form (all clauses
// live): histogram into ot_size, exclusive scan into ot_off, then a scatter that
// reuses ot_size (zeroed after the scan) as the per-literal cursor, which leaves
// the list sizes in ot_size again.
struct CsrOtArgs {
    const u32* lits;
    const u64* off;
    u32* ot_off;
    u32* ot_size;
    u32* ot_refs;
    u64 nlits;
    u32 D;
    u32* err;
};
// A clause whose offsets go down or leave [0, nlits) is an input error; neither
// pass reads its literals.
HD bool csr_clause_ok(const CsrOtArgs& a, u32 i) {
    const u64 s = a.off[i], e = a.off[i + 1];
    return s <= e && e <= a.nlits;
}
HD void k_hist_csr(const CsrOtArgs& a, u32 i) {
    if (!csr_clause_ok(a, i)) { atom_or(a.err, ERR_INPUT); return; }
    for (u64 k = a.off[i]; k < a.off[i + 1]; k++) {
        const u32 lit = a.lits[k];
        if (lit < 2 || lit >= a.D) { atom_or(a.err, ERR_INPUT); continue; }
        atom_add(&a.ot_size[lit], 1u);
    }
}
HD void k_scatter_csr(const CsrOtArgs& a, u32 i) {
    if (!csr_clause_ok(a, i)) return;
    for (u64 k = a.off[i]; k < a.off[i + 1]; k++) {
        const u32 lit = a.lits[k];
        if (lit < 2 || lit >= a.D) continue;
        const u32 pos = a.ot_off[lit] + atom_add(&a.ot_size[lit], 1u);
        if (pos < a.nlits) a.ot_refs[pos] = i;
        else atom_or(a.err, ERR_INTERNAL);
    }
}

// occurs[v] = (ps, ns) over live clauses (histSimp, src/cpu/histogram.cpp:82-96).
HD void k_occurs_clause(const Ctx& c, u32 i) {
    const Hdr h = c.hdr[i];
    if (h_deleted(h.flags)) return;
    const u32* l = c.lits + h.start;
    for (u32 k = 0; k < h.size; k++) {
        const u32 lit = l[k];
        atom_add(SIGN(lit) ? &c.ns[ABS(lit)] : &c.ps[ABS(lit)], 1u);
    }
}

// ---------------------------------------------------------------- counts
// countAll (src/cpu/solve.h:724-734): live clauses and their literals.
struct CountArgs {
    Ctx c;
    u64* out;  // [0] clauses, [1] literals
};
HD void k_count_clause(const CountArgs& a, u32 i) {
    const Hdr h = a.c.hdr[i];
    if (h_deleted(h.flags)) return;
    atom_add64(&a.out[0], 1ull);
    atom_add64(&a.out[1], (u64)h.size);
}

// Formula of every variable of a batch (variable 0 belongs to none).
HD void k_var_fid(u32* var_fid, const u32* f_var, u32 nf, u32 v) {
    var_fid[v] = v ? upper_segment(f_var, nf, v - 1) : NONE;
}

// Live clauses and literals per formula of a batch (countAll per formula); a
// clause's formula is that of its first literal's variable.
struct FormulaCountArgs {
    Ctx c;
    u64* f_cls;   // nf
    u64* f_lits;  // nf
};
HD void k_count_formula(const FormulaCountArgs& a, u32 i) {
    const Hdr h = a.c.hdr[i];
    if (h_deleted(h.flags)) return;
    const u32 f = a.c.var_fid[ABS(a.c.lits[h.start])];
    atom_add64(&a.f_cls[f], 1ull);
    atom_add64(&a.f_lits[f], (u64)h.size);
}

#if SIGMA_CUDA
// Same count. A formula's clauses are mostly adjacent, so a warp takes a stretch of
// consecutive clauses and adds only where the formula changes: an atomic per step of 32
// clauses queued 900k of them on 384 words (250 us for 14M clauses of 384 formulas, 167 so).
__global__ void __launch_bounds__(256) count_formula_k(FormulaCountArgs a, u32 n) {
    const u32 lane = threadIdx.x & 31u;
    const u32 warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    const u32 steps = ((n + 31u) / 32u + nwarps - 1u) / nwarps;  // per warp
    const u64 first = (u64)warp * steps * 32u;
    u32 cur = NONE;          // the formula being summed (the same in every lane)
    u32 cls = 0, lits = 0;   // this lane's share
    auto flush = [&]() {
        const u32 tc = __reduce_add_sync(kFull, cls), tl = __reduce_add_sync(kFull, lits);
        if (lane == 0 && tc) {
            atomicAdd((unsigned long long*)&a.f_cls[cur], (unsigned long long)tc);
            atomicAdd((unsigned long long*)&a.f_lits[cur], (unsigned long long)tl);
        }
        cls = lits = 0;
    };
    for (u32 s = 0; s < steps; s++) {
        const u64 i = first + (u64)s * 32u + lane;
        u32 f = NONE, sz = 0;
        if (i < n) {
            const Hdr h = a.c.hdr[i];
            if (!h_deleted(h.flags)) {
                f = a.c.var_fid[ABS(a.c.lits[h.start])];
                sz = h.size;
            }
        }
        u32 left = __ballot_sync(kFull, f != NONE);
        while (left) {
            const u32 g = __shfl_sync(kFull, f, __ffs(left) - 1);
            if (g != cur) {
                flush();
                cur = g;
            }
            const bool mine = f == g;
            cls += mine;
            lits += mine ? sz : 0u;
            left &= ~__ballot_sync(kFull, mine);
        }
    }
    flush();
}

// Same counts with a warp/block reduction and one pair of atomics per block.
__global__ void count_live_k(const Hdr* __restrict__ hdr, u32 n, u64* out) {
    u64 cls = 0, lits = 0;
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += blockDim.x * gridDim.x) {
        const Hdr h = hdr[i];
        if (!h_deleted(h.flags)) { cls++; lits += h.size; }
    }
    for (int o = 16; o; o >>= 1) {
        cls += __shfl_down_sync(0xffffffffu, cls, o);
        lits += __shfl_down_sync(0xffffffffu, lits, o);
    }
    __shared__ u64 s_cls[32], s_lits[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { s_cls[warp] = cls; s_lits[warp] = lits; }
    __syncthreads();
    if (threadIdx.x == 0) {
        u64 c = 0, l = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) { c += s_cls[w]; l += s_lits[w]; }
        atomicAdd((unsigned long long*)&out[0], (unsigned long long)c);
        atomicAdd((unsigned long long*)&out[1], (unsigned long long)l);
    }
}
#endif

// ---------------------------------------------------------------- compaction
// shrinkSimp (src/cpu/simplify.cpp:234-245; GPU: recycle.cu:30-97): drop deleted
// clauses, keep order. One scan over the clauses gives every survivor its new id (the
// sum's high word) and its new literal start (the low word: the literals of a store stay
// below 2^32), and moves it there in the same pass. (Flags, two scans and the move were
// four passes: 3.7 ms for the compactions of a round over 80M community clauses,
// 2.6 in one; 300k clauses 127 and 78 us.)
struct GcMove {
    Ctx c;
    Hdr* new_hdr;
    u32* new_lits;
    u32* new_stamp;  // the clause stamps move with the headers
    typedef ScanNone State;
    static constexpr int kItems = 4;
    static HD u32 clauses(u64 sum) { return (u32)(sum >> 32); }
    static HD u64 lits(u64 sum) { return sum & 0xFFFFFFFFull; }
    HD u64 value(size_t i, State&) const {
        const Hdr h = c.hdr[i];
        return h_deleted(h.flags) ? 0ull : (1ull << 32) + h.size;
    }
    HD void done(const State&) const {}
    HD void put(size_t i, u64 own, u64 at) const {
        if (!own) return;
        const u32 id = clauses(at);
        Hdr h = c.hdr[i];
        const u32* src = c.lits + h.start;
        h.start = (u32)lits(at);
        u32* dst = new_lits + h.start;
        new_hdr[id] = h;
        if (c.cstamp) new_stamp[id] = c.cstamp[i];
        for (u32 k0 = 0; k0 < h.size; k0 += 4) {  // four loads in flight
            u32 l[4];
#pragma unroll
            for (u32 j = 0; j < 4; j++) if (k0 + j < h.size) l[j] = src[k0 + j];
#pragma unroll
            for (u32 j = 0; j < 4; j++) if (k0 + j < h.size) dst[k0 + j] = l[j];
        }
    }
};

}  // namespace sigma
