// Model extension on the device: MODEL::extend (src/cpu/model.cpp:104-138).
//
// The witness stack holds records [witness, other literals..., length]. Walking the
// stack from its end, a record whose other literals are all false under the current
// values sets its witness true. Each record may read values that the records after
// it set, so one formula's walk is one dependent chain; the formulas of a batch are
// walked side by side, one warp per formula.
//
// What bounds it is the latency of that chain: a thread that walks record by record
// waits for four dependent loads a record (7.46 ms for 384 mixed k-SAT formulas with
// 797k witness words). A warp takes 32 records at a time instead: the lanes load their
// records and judge them under the values at the start of the step, all at once; then
// only the records that set a witness go one after the other, lowest lane (latest
// record) first, and the other lanes update what they know of their literals from
// registers. The same 384 formulas: 0.96 ms, and 1.99 ms when a step's loads are not
// spread over the steps before it and a lane asks for the values again instead.
#pragma once

#include "cnf.cuh"

namespace sigma {

struct ExtendArgs {
    const u32* resolved;  // witness stack (the store's numbering)
    uint8_t* value;       // per variable of the store: 1 true, 0 false
    u64 nres;             // single formula: stack length
    // formula batches: records in formula order (stack order inside a formula)
    const u32* rec_start;  // stack position of every record's witness
    const u64* rec_words;  // words of every record (its literals and the length word)
    const u32* order;      // records sorted by formula
    const u32* f_first;    // nf + 1: formula f owns order[f_first[f] .. f_first[f+1])
    u32* err;
};

HD bool ext_true(const uint8_t* value, u32 lit) { return value[ABS(lit)] == (SIGN(lit) ? 0 : 1); }

// One record: literals resolved[st .. st+len), the witness first.
HD void ext_record(const ExtendArgs& a, u64 st, u32 len) {
    for (u32 j = len - 1; j >= 1; j--)
        if (ext_true(a.value, a.resolved[st + j])) return;
    const u32 w = a.resolved[st];
    a.value[ABS(w)] = SIGN(w) ? 0 : 1;
}

// The single formula: records from the end of the stack, found by their length words.
HD void k_extend_single(const ExtendArgs& a) {
    u64 x = a.nres;
    while (x) {
        const u32 len = a.resolved[x - 1];
        if (len == 0 || len > x - 1) {  // malformed stack
            atom_or(a.err, ERR_INTERNAL);
            return;
        }
        const u64 st = x - 1 - len;
        ext_record(a, st, len);
        x = st;
    }
}

// Formula f of a batch: its records from the last to the first.
HD void k_extend_formula(const ExtendArgs& a, u32 f) {
    for (u32 i = a.f_first[f + 1]; i-- > a.f_first[f];) {
        const u32 r = a.order[i];
        ext_record(a, a.rec_start[r], (u32)a.rec_words[r] - 1u);
    }
}

#if SIGMA_CUDA
// Literals of a record that a lane keeps in registers (a longer record's rest is read
// again where it is needed), and the words of the stack a single formula's warp reads
// ahead to find its records.
constexpr u32 EXT_KEEP = 8;
constexpr u32 EXT_AHEAD = 1024;

// A lane's record: n other literals (the first EXT_KEEP in l, all at p), witness w.
struct ExtRec {
    const u32* p;
    u32 n, w;
    u32 l[EXT_KEEP];
    bool has;
};
DEV ExtRec ext_load(const u32* resolved, bool has, u64 st, u32 len) {
    ExtRec r;
    r.has = has;
    r.p = resolved + st + 1;
    r.n = has ? len - 1u : 0u;
    r.w = has ? resolved[st] : 0u;
#pragma unroll
    for (u32 j = 0; j < EXT_KEEP; j++) r.l[j] = j < r.n ? r.p[j] : 0u;
    return r;
}

// 32 records of one formula by one warp, in lane order. A lane keeps a truth bit per
// literal in l and whether its witness is true; a witness that is set goes round by a
// shuffle and updates them, so only records longer than EXT_KEEP + 1 read values again.
DEV void ext_warp_step(uint8_t* value, const ExtRec& r) {
    const u32 lane = threadIdx.x & 31u;
    bool wtrue = r.has && ext_true(value, r.w), rest = false;
    u32 bits = 0;
#pragma unroll
    for (u32 j = 0; j < EXT_KEEP; j++)
        if (j < r.n && ext_true(value, r.l[j])) bits |= 1u << j;
    for (u32 j = EXT_KEEP; j < r.n; j++) rest |= ext_true(value, r.p[j]);
    __syncwarp();
    u32 todo = __ballot_sync(kFull, r.has && !bits && !rest);
    while (todo) {
        const u32 f = (u32)(__ffs(todo) - 1);
        const u32 x = __shfl_sync(kFull, r.w | (wtrue ? 0u : 0x80000000u), (int)f);
        if (x >> 31) {  // the value changes
            const u32 w = x & 0x7FFFFFFFu;
            if (lane == f) value[ABS(w)] = SIGN(w) ? 0 : 1;
            if (ABS(r.w) == ABS(w)) wtrue = r.w == w;
#pragma unroll
            for (u32 j = 0; j < EXT_KEEP; j++) {
                if (r.l[j] == w) bits |= 1u << j;
                else if (r.l[j] == FLIP(w)) bits &= ~(1u << j);
            }
            __syncwarp();
            if (r.n > EXT_KEEP) {
                rest = false;
                for (u32 j = EXT_KEEP; j < r.n; j++) rest |= ext_true(value, r.p[j]);
            }
        }
        todo = __ballot_sync(kFull, r.has && !bits && !rest && lane > f);
    }
    __syncwarp();
}

// Formula f of a batch by warp f: its records from the last to the first. The loads of
// a step are spread over the steps before it (the record's index three steps ahead, its
// place two, its literals one), so a step waits for its values alone.
constexpr u32 EXT_WARPS = 2;
__global__ void __launch_bounds__(EXT_WARPS * 32) extend_formula_k(ExtendArgs a, u32 nf) {
    const u32 lane = threadIdx.x & 31u;
    const u32 f = blockIdx.x * EXT_WARPS + (threadIdx.x >> 5);
    if (f >= nf) return;
    const u32 first = a.f_first[f], n = a.f_first[f + 1] - first;
    // record q counts from the formula's last
    auto index = [&](u32 q) { return q < n ? a.order[first + n - 1u - q] : 0u; };
    auto place = [&](u32 q, u32 i) { return q < n ? a.rec_start[i] : 0u; };
    auto words = [&](u32 q, u32 i) { return q < n ? (u32)a.rec_words[i] - 1u : 0u; };
    const u32 i1 = index(lane + 32u);
    u32 i2 = index(lane + 64u);
    u32 st1, len1;
    ExtRec r;
    {
        const u32 i0 = index(lane);
        r = ext_load(a.resolved, lane < n, place(lane, i0), words(lane, i0));
        st1 = place(lane + 32u, i1);
        len1 = words(lane + 32u, i1);
    }
    for (u32 q = lane; q - lane < n; q += 32) {
        const ExtRec nx = ext_load(a.resolved, q + 32u < n, st1, len1);
        st1 = place(q + 64u, i2);
        len1 = words(q + 64u, i2);
        i2 = index(q + 96u);
        ext_warp_step(a.value, r);
        r = nx;
    }
}

// The single formula by one warp: the end of the stack is copied to shared memory,
// lane 0 finds up to 32 records there by their length words, and the warp takes them.
__global__ void __launch_bounds__(32) extend_single_k(ExtendArgs a) {
    __shared__ u32 ahead[EXT_AHEAD];
    __shared__ u64 rst[32];
    __shared__ u32 rlen[32];
    const u32 lane = threadIdx.x & 31u;
    u64 x = a.nres, lo = a.nres;  // ahead holds the words [lo, lo + EXT_AHEAD) below x
    while (x) {
        if (x - lo < EXT_AHEAD / 4 && lo) {
            lo = x > EXT_AHEAD ? x - EXT_AHEAD : 0;
            __syncwarp();
            for (u32 i = lane; i < (u32)(x - lo); i += 32) ahead[i] = a.resolved[lo + i];
            __syncwarp();
        }
        u32 cnt = 0, bad = 0;
        u64 y = x;
        if (lane == 0) {
            while (cnt < 32 && y > lo) {
                const u32 len = ahead[y - 1 - lo];
                if (len == 0 || len > y - 1) {  // malformed stack
                    bad = 1;
                    break;
                }
                y -= 1 + (u64)len;
                rst[cnt] = y;
                rlen[cnt++] = len;
            }
        }
        __syncwarp();
        cnt = __shfl_sync(kFull, cnt, 0);
        bad = __shfl_sync(kFull, bad, 0);
        x = __shfl_sync(kFull, y, 0);
        if (x < lo) lo = x;  // a record that began before the copy: read on from its start
        const bool has = lane < cnt;
        ext_warp_step(a.value, ext_load(a.resolved, has, has ? rst[lane] : 0ull, has ? rlen[lane] : 0u));
        if (bad) {
            if (lane == 0) atomicOr(a.err, ERR_INTERNAL);
            return;
        }
    }
}
#endif

// First record of every formula in the order sorted by formula (fid: its keys).
HD void k_extend_first(const u32* fid, u32 nrec, u32* f_first, u32 f) {
    u32 lo = 0, hi = nrec;  // the first record whose formula is f or later
    while (lo < hi) {
        const u32 mid = (lo + hi) >> 1;
        if (fid[mid] < f) lo = mid + 1;
        else hi = mid;
    }
    f_first[f] = lo;
}

// Values before the walk: eliminated variables start false (the solver never
// assigns them; MODEL::extend starts them at 0), the round's units hold.
HD void k_extend_clear(const Ctx& c, uint8_t* value, u32 v) {
    if (c.vstate[v]) value[v] = 0;
}
HD void k_extend_unit(const Ctx& c, uint8_t* value, u32 i) {
    const u32 u = c.trail[i];
    value[ABS(u)] = SIGN(u) ? 0 : 1;
}

// Batch values between the caller's layout (formula after formula, num_vars[f] + 1
// entries each, the first unused) and the store's numbering.
struct ExtendMap {
    const u64* p_first;  // nf + 1: first packed position of every formula
    const u32* f_var;    // nf + 1: variable offset of every formula in the store
    u32 nf;
};
HD void k_extend_in(const ExtendMap& m, const uint8_t* packed, uint8_t* value, u32 p) {
    const u32 f = upper_segment(m.p_first, m.nf, (u64)p);
    const u32 local = (u32)(p - m.p_first[f]);
    if (local) value[m.f_var[f] + local] = packed[p] ? 1 : 0;
}
HD void k_extend_out(const ExtendMap& m, const uint8_t* value, uint8_t* packed, u32 p) {
    const u32 f = upper_segment(m.p_first, m.nf, (u64)p);
    const u32 local = (u32)(p - m.p_first[f]);
    if (local) packed[p] = value[m.f_var[f] + local];  // the unused first entry keeps the caller's value
}

}  // namespace sigma
