// Single-pass device-wide exclusive scan with decoupled look-back.
//
// Generic over the value type T (a trivially copyable struct of 32-bit
// words), the associative operator, the input functor in(i) -> T and the
// output functor out(i, exclusive_prefix, own_value).  Tiles are numbered by
// an atomic ticket taken when a block starts, so a block only ever waits on
// blocks that are already resident; every wait is bounded (wait_give_up_warp)
// and a timeout sets ERR_TIMEOUT instead of hanging.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace ochre {

// A tile's aggregate and inclusive prefix, every 32-bit word of each in a
// 64-bit word whose high half is its flag: the scan's tag (see ScanSpace) and
// SCAN_AGG or SCAN_INC.  Anything else there (zero, or the tag of an earlier
// scan that used the same memory) means not yet.  One naturally aligned 64-bit access reads or writes a word with
// its flag, so a reader takes a value once all its words carry the flag, with
// relaxed accesses only, and one round of loads reads a predecessor's flags
// and values together.
constexpr uint32_t SCAN_AGG = 1u, SCAN_INC = 2u;
template <class T>
struct ScanStatus {
    static constexpr int W = (int)(sizeof(T) / 4);
    uint64_t agg[W];
    uint64_t inc[W];
};
template <class T>
__device__ __forceinline__ void st_flagged(uint64_t* dst, const T& v, uint32_t flag) {
    const uint32_t* s = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(T) / 4); i++) st_relaxed64(dst + i, ((uint64_t)flag << 32) | s[i]);
}
// True when every word of the value carries `flag`; v receives the words.
template <class T>
__device__ __forceinline__ bool ld_flagged(const uint64_t* src, uint32_t flag, T& v) {
    uint32_t* d = reinterpret_cast<uint32_t*>(&v);
    bool ok = true;
#pragma unroll
    for (int i = 0; i < (int)(sizeof(T) / 4); i++) {
        const uint64_t w = ld_relaxed64(src + i);
        d[i] = (uint32_t)w;
        ok = ok && (uint32_t)(w >> 32) == flag;
    }
    return ok;
}

// The prefix of a tile with aggregate tile_agg: decoupled look-back by one
// whole warp, 32 predecessors per round: lane k inspects tile top - k; the
// window up to the nearest inclusive value is combined in tile order (earlier
// tiles on the left).  Publishes the tile's aggregate and inclusive prefix.
template <class T, class Op>
__device__ __forceinline__ T scan_lookback(uint32_t tile, const T& tile_agg, Op op, const T& identity,
                                           ScanStatus<T>* status, uint32_t tag, uint32_t* err) {
    const int lane = threadIdx.x & 31;
    const uint32_t f_agg = tag << 2 | SCAN_AGG, f_inc = tag << 2 | SCAN_INC;
    T prefix = identity;
    ScanStatus<T>* me = status + tile;
    if (tile == 0) {
        if (lane == 0) st_flagged(me->inc, tile_agg, f_inc);
        return prefix;
    }
    if (lane == 0) st_flagged(me->agg, tile_agg, f_agg);
    int64_t top = (int64_t)tile - 1;
    long long spins = 0;
    const long long poll_limit = spin_limit(err);
    while (top >= 0) {
        const int64_t j = top - lane;
        // the predecessor's inclusive prefix and aggregate, read together
        bool has_inc = true, has_agg = true;   // before tile 0: an inclusive identity
        T vi = identity, va = identity;
        if (j >= 0) {
            has_inc = ld_flagged(status[j].inc, f_inc, vi);
            has_agg = ld_flagged(status[j].agg, f_agg, va);
        }
        const uint32_t m2 = __ballot_sync(0xffffffffu, has_inc);
        const int limit = m2 ? __ffs(m2) - 1 : 31;   // lanes [0, limit] are needed
        const uint32_t need = limit == 31 ? 0xffffffffu : ((1u << (limit + 1)) - 1u);
        if (__ballot_sync(0xffffffffu, !has_inc && !has_agg) & need) {
            if (wait_give_up_warp(spins, poll_limit, err)) break;
            if (spins > 64) __nanosleep(64);
            continue;
        }
        T v = identity;
        if (lane <= limit && j >= 0) v = has_inc ? vi : va;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const T o = shfl_down_T(v, d);
            if (lane + d < 32) v = op(o, v);
        }
        prefix = op(shfl_idx_T(v, 0), prefix);
        if (m2) break;
        top -= 32;
    }
    if (lane == 0) st_flagged(me->inc, op(prefix, tile_agg), f_inc);
    return prefix;
}

// Functors over whole arrays of words may take a thread's items at once, in
// 8- and 16-byte accesses (load_all(i, v), store_all(i, run, v, op) for the
// ITEMS items from i on): item by item a warp's access touches a sector for
// every 8 items and each of them ITEMS times.
template <class F, class = void>
struct takes_all : std::false_type {};
template <class F>
struct takes_all<F, std::void_t<typename F::takes_all>> : std::true_type {};
// N consecutive words (N 2 or 8; the address a multiple of 8 or 16 bytes).
template <int N>
__device__ __forceinline__ void load_words(const uint32_t* p, uint32_t (&w)[N]) {
    static_assert(N == 2 || N % 4 == 0, "pairs or fours");
    if constexpr (N == 2) {
        const uint2 q = *reinterpret_cast<const uint2*>(p);
        w[0] = q.x;
        w[1] = q.y;
    } else {
#pragma unroll
        for (int k = 0; k < N; k += 4) {
            const uint4 q = *reinterpret_cast<const uint4*>(p + k);
            w[k] = q.x;
            w[k + 1] = q.y;
            w[k + 2] = q.z;
            w[k + 3] = q.w;
        }
    }
}
template <int N>
__device__ __forceinline__ void store_words(uint32_t* p, const uint32_t (&w)[N]) {
    static_assert(N == 2 || N % 4 == 0, "pairs or fours");
    if constexpr (N == 2) {
        *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
    } else {
#pragma unroll
        for (int k = 0; k < N; k += 4) *reinterpret_cast<uint4*>(p + k) = make_uint4(w[k], w[k + 1], w[k + 2], w[k + 3]);
    }
}

// N consecutive bytes, as words (a caller's array may lie anywhere).
template <int N>
__device__ __forceinline__ void load_bytes(const uint8_t* p, uint32_t (&b)[N]) {
    if (N == 8 && (reinterpret_cast<uintptr_t>(p) & 7u) == 0u) {
        const uint2 q = *reinterpret_cast<const uint2*>(p);
#pragma unroll
        for (int k = 0; k < N; k++) b[k] = ((k < 4 ? q.x : q.y) >> (8 * (k & 3))) & 0xffu;
    } else {
#pragma unroll
        for (int k = 0; k < N; k++) b[k] = p[k];
    }
}

template <int BLOCK, int ITEMS, class T, class Op, class In, class Out>
__global__ void __launch_bounds__(BLOCK) k_scan(uint64_t n, const uint32_t* n_dev, In in, Out out, Op op,
                                                 T identity, ScanStatus<T>* status, uint32_t* ticket,
                                                 uint32_t ticket_base, uint32_t tag, T* total, uint32_t* err) {
    dependent_start();
    constexpr int WARPS = BLOCK / 32;
    __shared__ uint32_t s_tile;
    __shared__ T s_warp[WARPS];
    __shared__ T s_prefix;
    // A count held on the device (graph replays): the grid covers the
    // capacity n, the scan covers min(*n_dev, n).  Tiles past the count end
    // before publishing anything; no tile that scans waits on them.
    n = dev_count(n, n_dev);
    // an earlier wait of the run gave up: its outputs (this scan's inputs) are
    // not valid; every block ends here, before publishing
    if (run_aborted(err)) return;
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u) - ticket_base;
    __syncthreads();
    const uint32_t tile = s_tile;
    if ((uint64_t)tile * (BLOCK * ITEMS) >= n) return;
    const uint64_t base = (uint64_t)tile * (BLOCK * ITEMS) + (uint64_t)threadIdx.x * ITEMS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    T v[ITEMS];
    T acc = identity;
    const bool whole = base + ITEMS <= n;
    bool loaded = false;
    if constexpr (takes_all<In>::value) {
        if (whole) in.load_all(base, v);
        loaded = whole;
    }
    if (!loaded) {
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            const uint64_t i = base + k;
            v[k] = i < n ? in(i) : identity;
        }
    }
#pragma unroll
    for (int k = 0; k < ITEMS; k++) acc = op(acc, v[k]);
    // warp inclusive scan of per-thread aggregates
    T inc = acc;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T o = shfl_up_T(inc, d);
        if (lane >= d) inc = op(o, inc);
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        T w = lane < WARPS ? s_warp[lane] : identity;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const T o = shfl_up_T(w, d);
            if (lane >= d) w = op(o, w);
        }
        // w = inclusive over warps; turn into exclusive per warp
        const T ex = shfl_up_T(w, 1);
        const T tile_agg = shfl_idx_T(w, WARPS - 1);
        if (lane < WARPS) s_warp[lane] = lane == 0 ? identity : ex;
        const T prefix = scan_lookback(tile, tile_agg, op, identity, status, tag, err);
        if (lane == 0) {
            s_prefix = prefix;
            const uint64_t tile_end = (uint64_t)(tile + 1) * (BLOCK * ITEMS);
            if (tile_end >= n && total != nullptr) *total = op(prefix, tile_agg);
        }
    }
    __syncthreads();
    // exclusive prefix of this thread's first item
    T ex_lane = shfl_up_T(inc, 1);
    if (lane == 0) ex_lane = identity;
    T run = op(op(s_prefix, s_warp[warp]), ex_lane);
    if constexpr (takes_all<Out>::value) {
        if (whole) {
            out.store_all(base, run, v);
            return;
        }
    }
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        const uint64_t i = base + k;
        if (i < n) out(i, run, v[k]);
        run = op(run, v[k]);
    }
}

struct OpSumU32 {
    __device__ __forceinline__ uint32_t operator()(uint32_t a, uint32_t b) const { return a + b; }
};

// Floats of every command.
struct VerbFloats {
    const uint8_t* verbs;
    __device__ __forceinline__ uint32_t operator()(uint64_t i) const { return floats_per_verb(verbs[i]); }
    using takes_all = void;
    template <int N>
    __device__ __forceinline__ void load_all(uint64_t i, uint32_t (&v)[N]) const {
        uint32_t b[N];
        load_bytes(verbs + i, b);
#pragma unroll
        for (int k = 0; k < N; k++) v[k] = floats_per_verb((uint8_t)b[k]);
    }
};
// Every item's exclusive prefix.
struct ScanOff {
    uint32_t* off;
    __device__ __forceinline__ void operator()(uint64_t i, uint32_t ex, uint32_t) const { off[i] = ex; }
    using takes_all = void;
    template <int N>
    __device__ __forceinline__ void store_all(uint64_t i, uint32_t run, const uint32_t (&v)[N]) const {
        uint32_t o[N];
#pragma unroll
        for (int k = 0; k < N; k++) {
            o[k] = run;
            run += v[k];
        }
        store_words(off + i, o);
    }
};

constexpr int SCAN_BLOCK = 256;
constexpr int SCAN_ITEMS = 8;
// Up to SCAN_FEW items a thread takes 2 instead of 8: it reads and writes its
// items one after the other, which is most of a short scan's time (the span
// scan of one path's 2,367 tiles 13.1 -> 9.5 us; 1 and 4 items are 0.5 to 2 us
// slower on one or the other scan).  An arena keeps to 8, so that the
// look-back words take no more of it.
constexpr int SCAN_ITEMS_FEW = 2;
constexpr uint64_t SCAN_FEW = 1u << 16;

// Look-back memory of one scan (scan_space, api.cu).  An eager scan clears
// nothing: its flags carry a tag no earlier scan of the context used, and its
// tickets go on from the last scan's (ticket_base).  Two clears before each of
// a call's eight scans had cost more than a small batch's scans themselves.
struct ScanSpace {
    void* status;
    uint32_t* ticket;
    uint32_t ticket_base, tag;
};
cudaError_t scan_space(ochre_gpu_ctx* ctx, size_t status_bytes, uint32_t tiles, uint32_t first_ticket, cudaStream_t s,
                       ScanSpace* out);

// Launch helper.
// `n_dev` (optional): the count lives on the device and `n` is its capacity.
// `first_ticket` (a test hook, else 0): tiles below it are never taken.
template <class T, class Op, class In, class Out>
cudaError_t launch_scan(ochre_gpu_ctx* ctx, uint64_t n, In in, Out out, Op op, T identity, T* total, cudaStream_t stream,
                        const uint32_t* n_dev = nullptr, uint32_t first_ticket = 0u) {
    if (n == 0) return cudaSuccess;
    const bool few = n <= SCAN_FEW && ctx->scan_status.arena == nullptr && first_ticket == 0u;
    const uint64_t tile = (uint64_t)SCAN_BLOCK * (few ? SCAN_ITEMS_FEW : SCAN_ITEMS), tiles = (n + tile - 1) / tile;
    ScanSpace sp;
    const cudaError_t e = scan_space(ctx, tiles * sizeof(ScanStatus<T>), (uint32_t)tiles, first_ticket, stream, &sp);
    if (e != cudaSuccess) return e;
    auto* status = reinterpret_cast<ScanStatus<T>*>(sp.status);
    uint32_t* err = &dev_scalars(ctx)->err;
    if (few)
        launch_after(k_scan<SCAN_BLOCK, SCAN_ITEMS_FEW, T, Op, In, Out>, (unsigned)tiles, SCAN_BLOCK, 0, stream,
            n, n_dev, in, out, op, identity, status, sp.ticket, sp.ticket_base, sp.tag, total, err);
    else
        launch_after(k_scan<SCAN_BLOCK, SCAN_ITEMS, T, Op, In, Out>, (unsigned)tiles, SCAN_BLOCK, 0, stream,
            n, n_dev, in, out, op, identity, status, sp.ticket, sp.ticket_base, sp.tag, total, err);
    return cudaGetLastError();
}

}  // namespace ochre
