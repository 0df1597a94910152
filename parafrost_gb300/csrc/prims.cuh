// Device-wide primitives written for this library: exclusive scan and a stable
// LSD radix sort of (key, value) pairs. No CUB/Thrust: each is a few plain
// kernels (block reduce -> scan of block sums -> block scan, or one pass with a
// look-back; one digit histogram for all passes, then one ranked pass per digit).
#pragma once

#include "device.cuh"

#include <algorithm>
#include <vector>

namespace sigma {

// The plain scan of an array (scan1_k's value and put; no state per thread).
struct ScanNone {};
template <class Tin, class T>
struct ScanArray {
    const Tin* in;
    T* out;
    typedef ScanNone State;
    static constexpr int kItems = 16;
    HD T value(size_t i, State&) const { return (T)in[i]; }
    HD void done(const State&) const {}
    HD void put(size_t i, T, T prefix) const { out[i] = prefix; }
};

#if SIGMA_CUDA

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;  // per thread
constexpr int kScanTile = kScanThreads * kScanItems;

template <class T>
__device__ __forceinline__ T warp_incl_scan(T v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

template <class Tin, class T>
__global__ void scan_reduce_k(const Tin* in, size_t n, T* sums) {
    const size_t base = (size_t)blockIdx.x * kScanTile;
    T s = 0;
    for (int k = 0; k < kScanItems; k++) {
        const size_t i = base + (size_t)k * kScanThreads + threadIdx.x;
        if (i < n) s += (T)in[i];
    }
    // block reduce
    for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    __shared__ T ws[kScanThreads / 32];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        T t = 0;
        for (int w = 0; w < kScanThreads / 32; w++) t += ws[w];
        sums[blockIdx.x] = t;
    }
}

// Single block: exclusive scan of the block sums in place; writes the grand total.
template <class T>
__global__ void scan_sums_k(T* sums, size_t nb, T* total) {
    __shared__ T carry_s;
    __shared__ T ws[kScanThreads / 32];
    if (threadIdx.x == 0) carry_s = 0;
    __syncthreads();
    for (size_t base = 0; base < nb; base += kScanThreads) {
        const size_t i = base + threadIdx.x;
        const T v = i < nb ? sums[i] : T(0);
        const T incl = warp_incl_scan(v);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        if (lane == 31) ws[warp] = incl;
        __syncthreads();
        T wpre = 0, btot = 0;
        for (int w = 0; w < kScanThreads / 32; w++) {
            if (w < warp) wpre += ws[w];
            btot += ws[w];
        }
        const T carry = carry_s;
        if (i < nb) sums[i] = carry + wpre + incl - v;
        __syncthreads();
        if (threadIdx.x == 0) carry_s = carry + btot;
        __syncthreads();
    }
    if (threadIdx.x == 0 && total) *total = carry_s;
}

template <class Tin, class T>
__global__ void scan_down_k(const Tin* in, T* out, size_t n, const T* sums) {
    const size_t base = (size_t)blockIdx.x * kScanTile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ T ws[kScanThreads / 32];
    __shared__ T carry_s;
    if (threadIdx.x == 0) carry_s = sums[blockIdx.x];
    __syncthreads();
    for (int k = 0; k < kScanItems; k++) {
        const size_t i = base + (size_t)k * kScanThreads + threadIdx.x;
        const T v = i < n ? (T)in[i] : T(0);
        const T incl = warp_incl_scan(v);
        if (lane == 31) ws[warp] = incl;
        __syncthreads();
        T wpre = 0, btot = 0;
        for (int w = 0; w < kScanThreads / 32; w++) {
            if (w < warp) wpre += ws[w];
            btot += ws[w];
        }
        const T carry = carry_s;
        if (i < n) out[i] = carry + wpre + incl - v;
        __syncthreads();
        if (threadIdx.x == 0) carry_s = carry + btot;
        __syncthreads();
    }
}

// out[i] = sum(in[0..i)), total (device pointer, may be null) = sum(in[0..n)).
// tmp needs scan_tmp_elems(n) elements of T.
inline size_t scan_tmp_elems(size_t n) { return (n + kScanTile - 1) / kScanTile + 1; }

template <class Tin, class T>
void excl_scan(const Tin* in, T* out, size_t n, T* total, T* tmp, cudaStream_t s) {
    const size_t nb = (n + kScanTile - 1) / kScanTile;
    if (n == 0) {
        if (total) cudaMemsetAsync(total, 0, sizeof(T), s);
        return;
    }
    scan_reduce_k<Tin, T><<<(unsigned)nb, kScanThreads, 0, s>>>(in, n, tmp);
    scan_sums_k<T><<<1, kScanThreads, 0, s>>>(tmp, nb, total);
    scan_down_k<Tin, T><<<(unsigned)nb, kScanThreads, 0, s>>>(in, out, n, tmp);
}

// Single-pass exclusive scan (decoupled look-back): each tile takes its index from
// a counter in launch order, publishes its aggregate, adds the aggregates (or the
// first inclusive prefix) of the tiles before it, publishes its inclusive prefix
// and scans itself. Flags carry the scan's epoch, so nothing is cleared between
// scans; a tile index counter keeps running and base is where this scan's tiles
// start. A look-back wait that runs out records ERR_ITER in err.
struct Scan1State {
    u64* agg;       // per tile
    u64* incl;      // per tile
    u32* flag;      // per tile: epoch << 2 | 1 (aggregate) or | 2 (inclusive)
    u32* counter;   // tile index counter
    u32* err;
};

// A tile is F::kItems consecutive items per thread (16 for plain arrays, fewer where put
// has more to do, so that middle-sized scans still have a block for every SM): read once from memory in
// coalesced order into shared memory, scanned per thread in registers, combined
// across the block by one warp scan of the thread sums, and written back in
// coalesced order. Shared-memory positions are padded (one slot per 32) so the
// per-thread runs of consecutive items do not fall on one bank.
__device__ __forceinline__ int scan1_pad(int i) { return i + (i >> 5); }

//
// The scanned values come from f.value(i, state) and go to f.put(i, value, prefix), so a
// pass that selects, ranks and writes items is one launch; a thread's state over its
// values ends in f.done(state), called by whole warps.
template <class T, class F>
__global__ void __launch_bounds__(kScanThreads) scan1_k(F f, size_t n, T* total, Scan1State st, u32 base, u32 epoch) {
    constexpr int kItems = F::kItems, kTile = kScanThreads * kItems;
    __shared__ T items[kTile + kTile / 32];
    __shared__ T ws[kScanThreads / 32];
    __shared__ u32 tile_s;
    __shared__ T carry_s;
    if (threadIdx.x == 0) tile_s = atomicAdd(st.counter, 1u) - base;
    __syncthreads();
    const u32 tile = tile_s;
    const size_t nb = (n + kTile - 1) / kTile;
    const size_t t0 = (size_t)tile * kTile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T own[kItems];
    typename F::State state{};
#pragma unroll
    for (int k = 0; k < kItems; k++) {
        const int j = k * kScanThreads + threadIdx.x;
        const size_t i = t0 + (size_t)j;
        own[k] = i < n ? f.value(i, state) : T(0);
        items[scan1_pad(j)] = own[k];
    }
    f.done(state);
    __syncthreads();
    // this thread's run: items [threadIdx.x * kItems, +kItems)
    T run = 0;
    const int r0 = threadIdx.x * kItems;
#pragma unroll
    for (int k = 0; k < kItems; k++) run += items[scan1_pad(r0 + k)];
    const T incl = warp_incl_scan(run);
    if (lane == 31) ws[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        // block aggregate and per-warp offsets, then the look-back (as before, 32
        // tiles at a time: wait for their flags, add the aggregates after the
        // nearest inclusive prefix and stop there)
        T wv = lane < kScanThreads / 32 ? ws[lane] : T(0);
        const T winc = warp_incl_scan(wv);
        const T a = __shfl_sync(0xffffffffu, winc, kScanThreads / 32 - 1);
        if (lane < kScanThreads / 32) ws[lane] = winc - wv;
        T prefix = 0;
        if (lane == 0) {
            if (tile == 0) st.incl[0] = (u64)a;
            else st.agg[tile] = (u64)a;
            __threadfence();
            atomicExch(&st.flag[tile], (epoch << 2) | (tile == 0 ? 2u : 1u));
        }
        __syncwarp();
        bool late = false;
        for (long long top = (long long)tile - 1; top >= 0 && !late; top -= 32) {
            const long long p = top - lane;
            u32 f = (epoch << 2) | 1u;  // lanes past tile 0 add nothing
            u32 it = 0;
            if (p >= 0) {
                while (((f = *(volatile u32*)&st.flag[p]) >> 2) != epoch) {
                    if (++it > (1u << 24)) {
                        late = true;
                        break;
                    }
                    __nanosleep(32);
                }
            }
            late = __any_sync(0xffffffffu, late);
            if (late) break;
            __threadfence();
            const u32 incl_mask = __ballot_sync(0xffffffffu, p >= 0 && (f & 3u) == 2u);
            const int stop = incl_mask ? __ffs(incl_mask) - 1 : 32;
            T v = 0;
            if (p >= 0 && lane <= stop) {
                v = lane == stop ? (T)(*(volatile u64*)&st.incl[p]) : (T)(*(volatile u64*)&st.agg[p]);
            }
            for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            prefix += __shfl_sync(0xffffffffu, v, 0);
            if (incl_mask) break;
        }
        if (lane == 0) {
            if (late) atomicOr(st.err, ERR_ITER);
            if (tile != 0) {
                st.incl[tile] = (u64)(prefix + a);
                __threadfence();
                atomicExch(&st.flag[tile], (epoch << 2) | 2u);
            }
            if (tile + 1 == nb && total) *total = prefix + a;
            carry_s = prefix;
        }
    }
    __syncthreads();
    // exclusive prefixes of this thread's run, in place
    T acc = carry_s + ws[warp] + incl - run;
#pragma unroll
    for (int k = 0; k < kItems; k++) {
        const int q = scan1_pad(r0 + k);
        const T v = items[q];
        items[q] = acc;
        acc += v;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kItems; k++) {
        const int j = k * kScanThreads + threadIdx.x;
        const size_t i = t0 + (size_t)j;
        if (i < n) f.put(i, own[k], items[scan1_pad(j)]);
    }
}

template <class F>
size_t scan1_tiles(size_t n) { return (n + kScanThreads * F::kItems - 1) / (kScanThreads * F::kItems); }

// ---------------------------------------------------------------- radix sort
// Stable LSD radix sort of pairs, 8 bits a pass. One launch counts the digits of every
// pass; a pass is then one launch: a block ranks a tile of 4096 pairs by digit (warp
// matches, so equal digits keep their order), learns by a decoupled look-back how many
// of each digit the tiles before it hold, orders the tile in shared memory and writes it
// in runs of consecutive places. What bounds a large sort is the pairs' traffic (16 bytes
// a pair and pass, 4 for the count) and the ranking's issue slots, a small one the
// launches: up to one tile is sorted by one block in one launch. Before, a pass took
// five launches (count, three of a scan over 256 counts a tile, a scatter of single
// pairs). The election and list-sort stages
// of a round, which do two sorts a phase, before and now: 200 variables 794 and 562 us,
// 10k variables 1241 and 899, 1M mixed clauses 2105 and 1856; sorts of millions of pairs
// take as long as before.
constexpr int kRadixThreads = 256;
constexpr int kRadixWarps = kRadixThreads / 32;
constexpr int kRadixItems = 16;  // pairs per thread per tile
constexpr int kRadixTile = kRadixThreads * kRadixItems;

struct RadixShared {
    u32 keys[kRadixTile], vals[kRadixTile];
    u32 cnt[kRadixWarps][256];  // per warp: pairs of each digit, then the warp's first place
    u32 start[256];             // the digit's first place in the tile
    u32 wtot[kRadixWarps];
};
static_assert(sizeof(RadixShared) <= 48 * 1024, "more shared memory needs an attribute per device");

// Ranks of a tile's pairs: pair k of a lane (place warp * 512 + k * 32 + lane, those from
// n on left out) goes to place rank[k] of the tile ordered by digit. Thread d gets the
// tile's count of digit d. Ends with the block synchronised.
DEV u32 radix_rank(RadixShared& s, const u32 (&key)[kRadixItems], u32 n, int shift, u32 (&rank)[kRadixItems]) {
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const u32 lt = (1u << lane) - 1u;
    for (u32 d = lane; d < 256; d += 32) s.cnt[warp][d] = 0;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kRadixItems; k++) {
        const bool valid = warp * 512u + k * 32u + lane < n;
        const u32 d = valid ? (key[k] >> shift) & 255u : 256u;
        const u32 peers = __match_any_sync(kFull, d);
        const u32 before = valid ? s.cnt[warp][d] : 0u;
        __syncwarp();
        rank[k] = before + (u32)__popc(peers & lt);
        if (valid && !(peers & lt)) s.cnt[warp][d] = before + (u32)__popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // thread d: the warps' first places among digit d, the tile's count, and by a block
    // scan over the digits the digit's first place
    const u32 d = threadIdx.x;
    u32 total = 0;
#pragma unroll
    for (int w = 0; w < kRadixWarps; w++) {
        const u32 c = s.cnt[w][d];
        s.cnt[w][d] = total;
        total += c;
    }
    const u32 incl = warp_incl_scan(total);
    if (lane == 31) s.wtot[warp] = incl;
    __syncthreads();
    u32 before = 0;
    for (u32 w = 0; w < warp; w++) before += s.wtot[w];
    s.start[d] = before + incl - total;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kRadixItems; k++) {
        const u32 dk = (key[k] >> shift) & 255u;
        rank[k] += s.cnt[warp][dk] + s.start[dk];
    }
    return total;
}

// Digit counts of all passes: hist[pass * 256 + digit].
__global__ void __launch_bounds__(kRadixThreads) radix_count_k(const u32* keys, size_t n, int passes, u64* hist) {
    __shared__ u32 h[4][256];
    for (int i = threadIdx.x; i < 1024; i += blockDim.x) (&h[0][0])[i] = 0;
    __syncthreads();
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t base = (size_t)blockIdx.x * blockDim.x; base < n; base += step) {
        const size_t i = base + threadIdx.x;
        const u32 m = __ballot_sync(kFull, i < n);
        if (i >= n) continue;
        const u32 key = keys[i];
        for (int p = 0; p < passes; p++) {
            const u32 d = (key >> (8 * p)) & 255u;
            int same;
            __match_all_sync(m, d, &same);  // high digits are mostly alike: one add per warp
            if (!same) atomicAdd(&h[p][d], 1u);
            else if ((threadIdx.x & 31u) == (u32)(__ffs(m) - 1)) atomicAdd(&h[p][d], (u32)__popc(m));
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 256 * passes; i += blockDim.x)
        if ((&h[0][0])[i]) atomicAdd((unsigned long long*)&hist[i], (unsigned long long)(&h[0][0])[i]);
}

// One pass. state: one word per (tile, digit), zero before the pass: 1 << 62 | count of
// the tile, or 2 << 62 | count of all tiles up to it. A wait that runs out records
// ERR_ITER (nothing is then written past the arrays).
__global__ void __launch_bounds__(kRadixThreads) radix_pass_k(const u32* keys, const u32* vals, u32* okeys, u32* ovals,
                                                             size_t n, int shift, const u64* hist, u64* state,
                                                             u32* counter, u32* err) {
    extern __shared__ u32 radix_smem[];
    RadixShared& s = *reinterpret_cast<RadixShared*>(radix_smem);
    __shared__ u64 gbase[256];
    __shared__ u64 gtot[kRadixWarps];
    __shared__ u32 tile_s;
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, d = threadIdx.x;
    if (threadIdx.x == 0) tile_s = atomicAdd(counter, 1u);
    __syncthreads();
    const u32 tile = tile_s;
    const size_t t0 = (size_t)tile * kRadixTile;
    const u32 cnt = n - t0 < (size_t)kRadixTile ? (u32)(n - t0) : (u32)kRadixTile;
    u32 key[kRadixItems], val[kRadixItems], rank[kRadixItems];
#pragma unroll
    for (int k = 0; k < kRadixItems; k++) {
        const u32 j = warp * 512u + k * 32u + lane;
        key[k] = j < cnt ? keys[t0 + j] : 0u;
        val[k] = j < cnt ? vals[t0 + j] : 0u;
    }
    const u32 total = radix_rank(s, key, cnt, shift, rank);
    // publish digit d's count, then look back
    volatile u64* st = state;
    constexpr u64 kAgg = 1ull << 62, kIncl = 2ull << 62, kMask = kAgg - 1;
    st[(size_t)tile * 256 + d] = (tile ? kAgg : kIncl) | total;
    u64 before = 0;
    for (u32 t = tile; t-- > 0;) {
        u64 x;
        u32 it = 0;
        while (!(x = st[(size_t)t * 256 + d])) {
            if (++it > (1u << 24)) {
                atomicOr(err, ERR_ITER);
                break;
            }
        }
        before += x & kMask;
        if (!x || (x & kIncl)) break;
    }
    if (tile) st[(size_t)tile * 256 + d] = kIncl | (before + total);
    // exclusive prefix of the pass's digit counts
    const u64 hd = hist[d];
    const u64 incl = warp_incl_scan(hd);
    if (lane == 31) gtot[warp] = incl;
    __syncthreads();
    u64 base = incl - hd;
    for (u32 w = 0; w < warp; w++) base += gtot[w];
    gbase[d] = base + before - s.start[d];  // place i of the ordered tile goes to gbase + i
#pragma unroll
    for (int k = 0; k < kRadixItems; k++) {
        const u32 j = warp * 512u + k * 32u + lane;
        if (j < cnt) {
            s.keys[rank[k]] = key[k];
            s.vals[rank[k]] = val[k];
        }
    }
    __syncthreads();
    for (u32 i = threadIdx.x; i < cnt; i += kRadixThreads) {
        const u32 x = s.keys[i];
        const u64 pos = gbase[(x >> shift) & 255u] + i;
        if (pos < n) {
            okeys[pos] = x;
            ovals[pos] = s.vals[i];
        }
    }
}

// All passes of a sort of at most one tile, in one block.
__global__ void __launch_bounds__(kRadixThreads) radix_small_k(u32* keys, u32* vals, u32 n, int passes) {
    extern __shared__ u32 radix_smem[];
    RadixShared& s = *reinterpret_cast<RadixShared*>(radix_smem);
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    u32 key[kRadixItems], val[kRadixItems], rank[kRadixItems];
#pragma unroll
    for (int k = 0; k < kRadixItems; k++) {
        const u32 j = warp * 512u + k * 32u + lane;
        key[k] = j < n ? keys[j] : 0u;
        val[k] = j < n ? vals[j] : 0u;
    }
    for (int p = 0; p < passes; p++) {
        radix_rank(s, key, n, 8 * p, rank);
#pragma unroll
        for (int k = 0; k < kRadixItems; k++) {
            if (warp * 512u + k * 32u + lane < n) {
                s.keys[rank[k]] = key[k];
                s.vals[rank[k]] = val[k];
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kRadixItems; k++) {
            const u32 j = warp * 512u + k * 32u + lane;
            if (j < n) {
                key[k] = s.keys[j];
                val[k] = s.vals[j];
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < kRadixItems; k++) {
        const u32 j = warp * 512u + k * 32u + lane;
        if (j < n) {
            keys[j] = key[k];
            vals[j] = val[k];
        }
    }
}

// Work words of a sort of n pairs: the digit counts of four passes, the tile counters and
// a state word per tile and digit, all 64-bit.
inline size_t radix_tiles(size_t n) { return (n + kRadixTile - 1) / kRadixTile; }
inline size_t radix_work_elems(size_t n) { return 1024 + 4 + 256 * radix_tiles(n); }

// Stable sort of (keys, vals) by the low `bits` bits of keys, with (k2, v2) as the other
// buffers and radix_work_elems(n) words of work. True when the result is in (k2, v2).
inline bool radix_sort_any(u32* keys, u32* vals, u32* k2, u32* v2, size_t n, int bits, u64* work, u32* err,
                           cudaStream_t s, unsigned& launches) {
    if (n <= 1) return false;
    const int passes = (bits + 7) / 8;
    if (n <= (size_t)kRadixTile) {
        launches++;
        radix_small_k<<<1, kRadixThreads, sizeof(RadixShared), s>>>(keys, vals, (u32)n, passes);
        return false;
    }
    const size_t nb = radix_tiles(n);
    u64* hist = work;
    u32* counter = (u32*)(work + 1024);
    u64* state = work + 1028;
    cudaMemsetAsync(hist, 0, 1028 * 8, s);
    radix_count_k<<<(unsigned)std::min<size_t>((n + 2047) / 2048, 1216), kRadixThreads, 0, s>>>(keys, n, passes, hist);
    u32 *ka = keys, *va = vals, *kb = k2, *vb = v2;
    for (int p = 0; p < passes; p++) {
        cudaMemsetAsync(state, 0, nb * 256 * 8, s);
        radix_pass_k<<<(unsigned)nb, kRadixThreads, sizeof(RadixShared), s>>>(ka, va, kb, vb, n, 8 * p, hist + 256 * p,
                                                                             state, counter + p, err);
        std::swap(ka, kb);
        std::swap(va, vb);
    }
    launches += 1 + passes;
    return passes & 1;
}

#else  // serial emulation

inline size_t scan_tmp_elems(size_t n) { return 1; }
inline size_t radix_work_elems(size_t) { return 1; }

template <class Tin, class T>
void excl_scan(const Tin* in, T* out, size_t n, T* total, T* /*tmp*/, void* /*stream*/) {
    T s = 0;
    for (size_t i = 0; i < n; i++) {
        const T v = (T)in[i];
        out[i] = s;
        s += v;
    }
    if (total) *total = s;
}

inline bool radix_sort_any(u32* keys, u32* vals, u32*, u32*, size_t n, int bits, u64*, u32*, void*, unsigned&) {
    std::vector<size_t> idx(n);
    for (size_t i = 0; i < n; i++) idx[i] = i;
    const u32 mask = bits >= 32 ? 0xFFFFFFFFu : ((1u << bits) - 1u);
    std::stable_sort(idx.begin(), idx.end(), [&](size_t a, size_t b) { return (keys[a] & mask) < (keys[b] & mask); });
    std::vector<u32> k(n), v(n);
    for (size_t i = 0; i < n; i++) { k[i] = keys[idx[i]]; v[i] = vals[idx[i]]; }
    std::copy(k.begin(), k.end(), keys);
    std::copy(v.begin(), v.end(), vals);
    return false;
}

#endif

}  // namespace sigma
