// Stage 3: stable LSD radix sort of (key, value) pairs, onesweep style.
//
// Reference counterpart: the two sort_unstable_by_key calls of finish
// (rasterizer.rs:209, 211).  The reference's sorts are unstable, so the f32
// accumulation order inside a tile is unspecified there; this sort is stable,
// which makes the GPU result deterministic.
//
// Digits are 8 bits wide, or up to 11 (the tunable sort_digit_bits: fewer
// passes, larger per-tile histograms and look-back rows); a sort of k key bits
// takes ceil(k / width) passes of balanced widths.
// One upfront kernel histograms every digit of every pass (and scans the
// counts); each pass then ranks a tile of keys in shared memory (per-warp counters with
// __match_any_sync for stable ranks), publishes its per-digit counts and
// resolves its global offsets by decoupled look-back over earlier tiles
// (bounded spins; a look-back word holds its flag and count together, so
// relaxed accesses suffice), and scatters through shared memory so that
// runs of equal digits leave as contiguous writes.
#include "common.cuh"
#include "internal.h"

#include <algorithm>
#include <utility>

namespace ochre {

constexpr int SORT_BLOCK = 256;
constexpr int SORT_WARPS = SORT_BLOCK / 32;
constexpr int SORT_ITEMS = 15;
constexpr int SORT_TILE = SORT_BLOCK * SORT_ITEMS;
constexpr uint32_t LB_AGG = 1u << 30, LB_INC = 2u << 30, LB_MASK = (1u << 30) - 1u;
constexpr int LB_WINDOW = 8;      // predecessor tiles one digit's look-back reads per round
constexpr int SORT_MAX_PASSES = 8;
constexpr size_t SORT_APART = (size_t)64 << 20;   // bytes that look-back words of passes of their own may take

// The digits of a sort: pass p takes `width[p]` bits from bit `shift[p]`
// (widths balanced over the key bits, at most the digit width RB).
struct SortPlan {
    int passes;
    uint8_t shift[SORT_MAX_PASSES];
    uint8_t width[SORT_MAX_PASSES];
};

// Histograms of every pass's digits; the block that adds its counts last turns
// them into each digit's first output place (`done` counts the blocks).
template <class K, int RB>
__global__ void __launch_bounds__(256) k_sort_hist(const K* keys, uint64_t n, const uint32_t* n_dev,
                                                   SortPlan plan, uint32_t* hist, uint32_t* __restrict__ off,
                                                   uint32_t* done) {
    dependent_start();
    constexpr int RADIX = 1 << RB;
    constexpr int MAXP = (64 + RB - 1) / RB;
    constexpr int PER = RADIX / 256;   // consecutive digits per thread
    __shared__ uint32_t sh[MAXP][RADIX];
    uint32_t* s_scan = &sh[0][0];   // the last block's scan, once the counts have left
    n = dev_count(n, n_dev);
    for (int i = threadIdx.x; i < MAXP * RADIX; i += blockDim.x) (&sh[0][0])[i] = 0u;
    __syncthreads();
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const K k = keys[i];
#pragma unroll
        for (int p = 0; p < MAXP; p++)
            if (p < plan.passes) atomicAdd(&sh[p][(uint32_t)(k >> plan.shift[p]) & ((1u << plan.width[p]) - 1u)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < plan.passes * RADIX; i += blockDim.x) {
        const uint32_t v = (&sh[0][0])[i];
        if (v) atomicAdd(hist + i, v);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_scan[0] = atomicAdd(done, 1u);
    __syncthreads();
    if (s_scan[0] + 1u != gridDim.x) return;
    __threadfence();
    __syncthreads();
    const int t = threadIdx.x;
    for (int p = 0; p < plan.passes; p++) {
        uint32_t v[PER], sum = 0;
#pragma unroll
        for (int q = 0; q < PER; q++) {
            v[q] = __ldcg(hist + p * RADIX + t * PER + q);
            sum += v[q];
        }
        s_scan[t] = sum;
        __syncthreads();
        for (int k = 1; k < 256; k <<= 1) {
            const uint32_t a = t >= k ? s_scan[t - k] : 0u;
            __syncthreads();
            s_scan[t] += a;
            __syncthreads();
        }
        uint32_t run = s_scan[t] - sum;
#pragma unroll
        for (int q = 0; q < PER; q++) {
            off[p * RADIX + t * PER + q] = run;
            run += v[q];
        }
        __syncthreads();
    }
}

// Shared memory of a onesweep block: the tile's keys and values, per-warp
// digit counters, the tile's digit starts and global digit bases, a word.
template <class K, int RB>
constexpr size_t onesweep_smem() {
    return (size_t)SORT_TILE * (sizeof(K) + 4) + ((size_t)SORT_WARPS * (1 << RB) + 2 * (1 << RB) + 4) * 4;
}

// Blocks per SM: three with 8-bit digits (register-bound otherwise: the
// 32-bit-key form would take more than 85 registers and drop to two); wider
// digits are held to two by their shared memory.
template <class K, int RB>
__global__ void __launch_bounds__(SORT_BLOCK, RB <= 8 ? 3 : 2) k_onesweep(
    const K* keys_in, const uint32_t* vals_in, K* __restrict__ keys_out,
    uint32_t* __restrict__ vals_out, uint64_t n, const uint32_t* n_dev, int shift, uint32_t mask,
    const uint32_t* digit_off, uint32_t* lookback, uint32_t* ticket, uint32_t* err) {
    dependent_start();
    constexpr int RADIX = 1 << RB;
    constexpr int PER = RADIX / SORT_BLOCK;   // digits per thread in the offset phase
    extern __shared__ __align__(16) unsigned char smem[];
    K* s_keys = reinterpret_cast<K*>(smem);
    uint32_t* s_vals = reinterpret_cast<uint32_t*>(s_keys + SORT_TILE);
    uint32_t* s_whist = s_vals + SORT_TILE;               // [SORT_WARPS][RADIX]
    uint32_t* s_tile_excl = s_whist + SORT_WARPS * RADIX;  // [RADIX]
    uint32_t* s_gbase = s_tile_excl + RADIX;               // [RADIX]
    uint32_t* s_misc = s_gbase + RADIX;                    // [0]: tile id

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (run_aborted(err)) return;   // an earlier wait of the run gave up
    if (threadIdx.x == 0) s_misc[0] = atomicAdd(ticket, 1u);
    for (int i = lane; i < RADIX; i += 32) s_whist[warp * RADIX + i] = 0u;
    __syncthreads();
    const uint32_t tile = s_misc[0];
    const uint64_t tile_base = (uint64_t)tile * SORT_TILE;
    // device-held count (graph replays): tiles past it end before publishing;
    // every tile that sorts precedes them
    n = dev_count(n, n_dev);
    if (tile_base >= n) return;
    const uint64_t warp_base = tile_base + (uint64_t)warp * 32 * SORT_ITEMS;
    const uint32_t lt_mask = (1u << lane) - 1u;

    K key[SORT_ITEMS];
    uint32_t val[SORT_ITEMS];
    uint32_t rank[SORT_ITEMS];
    uint32_t dig[SORT_ITEMS];
    // every load of the tile first (all in flight together), then the ranking
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; k++) {
        const uint64_t i = warp_base + (uint64_t)k * 32 + lane;
        const bool valid = i < n;
        key[k] = valid ? keys_in[i] : (K)0;
        val[k] = valid ? vals_in[i] : 0u;
    }
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; k++) {
        const uint64_t i = warp_base + (uint64_t)k * 32 + lane;
        const bool valid = i < n;
        const uint32_t d = valid ? ((uint32_t)(key[k] >> shift) & mask) : (uint32_t)RADIX;
        dig[k] = d;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const int leader = __ffs(peers) - 1;
        uint32_t b = 0;
        if (lane == leader && d < (uint32_t)RADIX) {
            b = s_whist[warp * RADIX + d];
            s_whist[warp * RADIX + d] = b + __popc(peers);
        }
        b = __shfl_sync(0xffffffffu, b, leader);
        rank[k] = b + __popc(peers & lt_mask);
        __syncwarp();
    }
    __syncthreads();

    // PER digits per thread: exclusive over warps, tile count, look-back
#pragma unroll 1
    for (int q = 0; q < PER; q++) {
        const int d = threadIdx.x + q * SORT_BLOCK;
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < SORT_WARPS; w++) {
            const uint32_t c = s_whist[w * RADIX + d];
            s_whist[w * RADIX + d] = run;
            run += c;
        }
        uint32_t* my = lookback + (size_t)tile * RADIX + d;
        uint32_t excl = 0;
        if (tile == 0) {
            st_relaxed(my, LB_INC | run);
        } else {
            st_relaxed(my, LB_AGG | run);
            // windowed look-back: LB_WINDOW predecessors per round, read
            // together (one latency per round instead of one per tile), up
            // to the nearest inclusive value
            int64_t top = (int64_t)tile - 1;
            long long spins = 0;
            const long long poll_limit = spin_limit(err);
            // the nearest predecessor alone first: often it is inclusive already
            {
                const uint32_t v = ld_relaxed(lookback + (size_t)top * RADIX + d);
                if ((v & ~LB_MASK) == LB_INC) {
                    excl = v & LB_MASK;
                    top = -1;
                }
            }
            while (top >= 0) {
                uint32_t v[LB_WINDOW];
#pragma unroll
                for (int k = 0; k < LB_WINDOW; k++) {
                    const int64_t j = top - k;
                    v[k] = j >= 0 ? ld_relaxed(lookback + (size_t)j * RADIX + d) : LB_INC;   // before tile 0: an inclusive 0
                }
                int k_inc = LB_WINDOW;
#pragma unroll
                for (int k = LB_WINDOW - 1; k >= 0; k--)
                    if ((v[k] & ~LB_MASK) == LB_INC) k_inc = k;
                bool missing = false;
                uint32_t sum = 0;
#pragma unroll
                for (int k = 0; k < LB_WINDOW; k++) {
                    if (k <= k_inc) {
                        if ((v[k] & ~LB_MASK) == 0u) missing = true;
                        sum += v[k] & LB_MASK;
                    }
                }
                if (missing) {
                    if (wait_give_up(spins, poll_limit, err)) break;
                    if (spins > 64) __nanosleep(64);
                    continue;
                }
                excl += sum;
                if (k_inc < LB_WINDOW) break;
                top -= LB_WINDOW;
            }
            st_relaxed(my, LB_INC | (excl + run));
        }
        s_gbase[d] = digit_off[d] + excl;
        s_tile_excl[d] = run;
    }
    __syncthreads();
    if (warp == 0) {
        // block exclusive scan of the tile's digit counts: RADIX / 32 per lane
        constexpr int PL = RADIX / 32;
        uint32_t v[PL], sum = 0;
#pragma unroll
        for (int q = 0; q < PL; q++) { v[q] = s_tile_excl[lane * PL + q]; sum += v[q]; }
        uint32_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        uint32_t run = inc - sum;
#pragma unroll
        for (int q = 0; q < PL; q++) { s_tile_excl[lane * PL + q] = run; run += v[q]; }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < SORT_ITEMS; k++) {
        const uint32_t d = dig[k];
        if (d < (uint32_t)RADIX) {
            const uint32_t pos = s_tile_excl[d] + s_whist[warp * RADIX + d] + rank[k];
            s_keys[pos] = key[k];
            s_vals[pos] = val[k];
        }
    }
    __syncthreads();
    const uint64_t remain = n - tile_base;
    const int cnt = remain < (uint64_t)SORT_TILE ? (int)remain : SORT_TILE;
    for (int i = threadIdx.x; i < cnt; i += SORT_BLOCK) {
        const K k = s_keys[i];
        const uint32_t d = (uint32_t)(k >> shift) & mask;
        const uint32_t g = s_gbase[d] + ((uint32_t)i - s_tile_excl[d]);
        keys_out[g] = k;
        vals_out[g] = s_vals[i];
    }
}

template <class K, int RB>
static int sort_impl(ochre_gpu_ctx* ctx, uint64_t n, uint32_t key_bits, cudaStream_t s, uint32_t* passes_done,
                     uint32_t first_bit) {
    constexpr int RADIX = 1 << RB;
    DevScalars* ds = dev_scalars(ctx);
    // graph replays: n is the capacity, the count is on the device
    const uint32_t* n_dev = ctx->plan ? &ds->n_entries : nullptr;
    SortPlan plan{};
    const uint32_t kb = std::max<uint32_t>(key_bits, 1u);
    plan.passes = (int)((kb + RB - 1) / RB);
    if (plan.passes > SORT_MAX_PASSES) return OCHRE_E_INVALID;
    for (int p = 0, at = (int)first_bit; p < plan.passes; p++) {
        // balanced widths: the first kb % passes passes take one bit more
        const int w = (int)(kb / plan.passes) + (p < (int)(kb % plan.passes) ? 1 : 0);
        plan.shift[p] = (uint8_t)at;
        plan.width[p] = (uint8_t)w;
        at += w;
    }
    const int passes = plan.passes;
    const uint64_t tiles = (n + SORT_TILE - 1) / SORT_TILE;
    // The counts, the tickets and every pass's look-back words lie together
    // and are cleared once.  In an arena (no allocation), and where a long sort's
    // passes would take more than SORT_APART bytes beyond one pass's words, the
    // passes share those, cleared before each (a clear and a late launch, some 5
    // us of passes that take 500 there).
    // No count is read back: a pass whose digit is the same in all keys runs
    // like any other (the read-back that found it out took longer than most
    // calls' passes: 15 to 20 us of every call).
    const size_t rows = (size_t)tiles * RADIX;
    const bool shared = ctx->sort_lookback.arena != nullptr || (size_t)(passes - 1) * rows * 4 > SORT_APART;
    constexpr size_t TICKETS = 16;   // one per pass, the last one counts k_sort_hist's blocks
    OCHRE_CUDA_TRY(ctx->sort_hist.ensure((size_t)passes * RADIX * 4 * 2));
    const size_t head = shared ? 0 : (size_t)passes * RADIX + TICKETS;
    const size_t words = head + rows * (shared ? 1 : passes);
    OCHRE_CUDA_TRY(ctx->sort_lookback.ensure(words * 4));
    uint32_t* off = ctx->sort_hist.as<uint32_t>();
    uint32_t* hist = shared ? off + passes * RADIX : ctx->sort_lookback.as<uint32_t>();
    uint32_t* tickets = shared ? &ds->sort_ticket : hist + passes * RADIX;
    if (shared) {
        OCHRE_CUDA_TRY(cudaMemsetAsync(hist, 0, (size_t)passes * RADIX * 4, s));
        OCHRE_CUDA_TRY(cudaMemsetAsync(tickets, 0, 4, s));
    } else {
        OCHRE_CUDA_TRY(cudaMemsetAsync(hist, 0, words * 4, s));
    }
    K* kin = ctx->keys.as<K>();
    uint32_t* vin = ctx->vals.as<uint32_t>();
    K* kout = ctx->keys_alt.as<K>();
    uint32_t* vout = ctx->vals_alt.as<uint32_t>();
    {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
        int blocks = (int)std::min<uint64_t>((n + 255) / 256, (uint64_t)std::max(sms, 1) * 8);
        OCHRE_LAUNCH(ctx, "sort_hist", s, launch_after(k_sort_hist<K, RB>, blocks, 256, 0, s,
            kin, n, n_dev, plan, hist, off, shared ? tickets : tickets + TICKETS - 1));
        OCHRE_CUDA_TRY(cudaGetLastError());
    }
    const size_t smem = onesweep_smem<K, RB>();
    OCHRE_CUDA_TRY(cudaFuncSetAttribute(k_onesweep<K, RB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    for (int p = 0; p < passes; p++) {
        uint32_t* lookback = ctx->sort_lookback.as<uint32_t>() + head + (shared ? 0 : p * rows);
        uint32_t* ticket = shared ? tickets : tickets + p;
        if (shared) {
            OCHRE_CUDA_TRY(cudaMemsetAsync(lookback, 0, rows * 4, s));
            OCHRE_CUDA_TRY(cudaMemsetAsync(ticket, 0, 4, s));
        }
        if (ctx->test_skip_sort_ticket) {
            ctx->test_skip_sort_ticket = 0;
            OCHRE_CUDA_TRY(cudaMemsetAsync(ticket, 1, 1, s));   // (its low byte)
        }
        OCHRE_LAUNCH(ctx, "sort_onesweep", s, launch_after(k_onesweep<K, RB>, (unsigned)tiles, SORT_BLOCK, smem, s,
            kin, vin, kout, vout, n, n_dev, plan.shift[p], (1u << plan.width[p]) - 1u, off + p * RADIX, lookback,
            ticket, &ds->err));
        OCHRE_CUDA_TRY(cudaGetLastError());
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    if (kin != ctx->keys.as<K>()) {
        // leave the sorted result in ctx->keys / ctx->vals
        std::swap(ctx->keys, ctx->keys_alt);
        std::swap(ctx->vals, ctx->vals_alt);
    }
    *passes_done = (uint32_t)passes;
    return OCHRE_OK;
}

int stage_sort(ochre_gpu_ctx* ctx, uint64_t n, uint32_t key_bits, cudaStream_t s, uint32_t* passes,
               uint32_t first_bit) {
    *passes = 0;
    if (n <= 1) return OCHRE_OK;
    if (ctx->tune_sort_digit_bits == 11)
        return ctx->keys64 ? sort_impl<uint64_t, 11>(ctx, n, key_bits, s, passes, first_bit)
                           : sort_impl<uint32_t, 11>(ctx, n, key_bits, s, passes, first_bit);
    return ctx->keys64 ? sort_impl<uint64_t, 8>(ctx, n, key_bits, s, passes, first_bit)
                       : sort_impl<uint32_t, 8>(ctx, n, key_bits, s, passes, first_bit);
}

// ---- one block per raster ----
// The entries were emitted raster by raster and a raster's keys are its key
// base plus a number below its own key space, so the order asked for is each
// raster's entries sorted by that number.  Where every raster's entries fit
// one block's shared memory, a block reads their keys once, ranks them there
// (8 bits a pass, as in k_onesweep: lanes with equal digits by ballots, warps
// in entry order, so it is stable) and writes the
// entries once.  An entry is one word, its number and its place among the
// raster's entries; its value is fetched when it is written.  That is one
// launch and 16 bytes an entry, where the device-wide passes move 16 bytes an
// entry each, as many passes as all rasters' key spaces together have digits.
// Bound by the latency of a block's few serial phases, so blocks come in three
// sizes (128, 256 and 512 threads), each raster to the smallest that holds it.
// 1,000 shapes of 2,785 entries (23 key bits, 13 of them within a raster): 124
// us for three passes and their histogram, 40 here; 20,000 strokes of 957: 620
// and 287.
// The lanes of the warp whose digit equals this lane's, among those with
// `valid` set: one ballot per digit bit.  (Here 6 us shorter than
// __match_any_sync for 1,000 shapes; in k_onesweep it is the longer way.)
template <int BITS>
__device__ __forceinline__ uint32_t same_digit(uint32_t d, bool valid) {
    uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < BITS; b++) {
        const bool set = (d >> b) & 1u;
        const uint32_t m = __ballot_sync(0xffffffffu, set);
        peers &= set ? m : ~m;
    }
    return peers;
}

struct LocalSortArgs {
    const RasterRun* run;       // the rasters: small from the front, middle from n_rasters - 1 down, large from n_rasters on
    uint32_t n_rasters, middle, large;
    uint32_t first;             // of the launch, in the order large, middle, small
    const int4* bbox;
    const uint64_t* key_base;
    const uint32_t* line_ent_total;
};
template <int THREADS, int ITEMS>
constexpr size_t local_sort_smem() {
    return (size_t)THREADS * ITEMS * 4 + (size_t)(THREADS / 32) * 256 * 4 + 256 * 4;
}
template <class K, int THREADS, int ITEMS, int BLOCKS>
__global__ void __launch_bounds__(THREADS, BLOCKS) k_sort_local(const K* keys_in,
                                                                const uint32_t* vals_in,
                                                                K* __restrict__ keys_out,
                                                                uint32_t* __restrict__ vals_out, LocalSortArgs A) {
    dependent_start();
    constexpr int WARPS = THREADS / 32;
    constexpr uint32_t FULL = 0xffffffffu;
    constexpr int IDX = LOCAL_SORT_IDX_BITS;
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t* s_word = reinterpret_cast<uint32_t*>(smem);    // [THREADS * ITEMS]
    uint32_t* s_cnt = s_word + THREADS * ITEMS;              // [WARPS][256]
    uint32_t* s_dig = s_cnt + WARPS * 256;                   // [256]
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t q = A.first + blockIdx.x;
    const RasterRun run = A.run[q < A.large              ? A.n_rasters + q
                                : q < A.large + A.middle ? A.n_rasters - 1u - (q - A.large)
                                                         : q - A.large - A.middle];
    const uint32_t r = run.raster, e0 = run.begin, out = run.out;
    const K base = (K)A.key_base[r];
    if (run.n == 0u) {   // no increments: its one entry comes after the lines' entries
        if (tid == 0) {
            const uint32_t at = *A.line_ent_total + (out - e0);
            keys_out[out] = keys_in[at];
            vals_out[out] = vals_in[at];
        }
        return;
    }
    const uint32_t n = min(run.n, (uint32_t)(THREADS * ITEMS));   // (listed by size: it fits)
    const int4 bb = A.bbox[r];
    const uint32_t space = (uint32_t)(bb.z - bb.x + 1) * (uint32_t)(bb.w - bb.y + 1) * 2u;
    const int bits = 32 - __clz(space - 1u);
    const int passes = (bits + 7) / 8;
    const int width = (bits + passes - 1) / passes;
    const uint32_t mask = (1u << width) - 1u;
    // a warp owns `steps` times 32 consecutive entries
    const int steps = (int)((n + THREADS - 1) / THREADS);
    const uint32_t first = warp * 32u * (uint32_t)steps + lane;
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t word[ITEMS], rank[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        const uint32_t i = first + 32u * k;
        word[k] = k < steps && i < n ? (uint32_t)(keys_in[e0 + i] - base) << IDX | i : 0u;
    }
    for (int p = 0; p < passes; p++) {
        const int shift = IDX + p * width;
        for (uint32_t d = lane; d <= mask; d += 32) s_cnt[warp * 256u + d] = 0u;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            if (k >= steps) break;
            const bool valid = first + 32u * k < n;
            const uint32_t d = (word[k] >> shift) & mask;
            const uint32_t peers = same_digit<8>(d, valid);
            const int leader = valid ? __ffs(peers) - 1 : (int)lane;
            uint32_t b = 0;
            if ((int)lane == leader && valid) {
                b = s_cnt[warp * 256u + d];
                s_cnt[warp * 256u + d] = b + (uint32_t)__popc(peers);
            }
            rank[k] = __shfl_sync(FULL, b, leader) + (uint32_t)__popc(peers & lt);
            __syncwarp();
        }
        __syncthreads();
        // per digit: the warps' starts, then the digits' starts
        for (uint32_t d = tid; d < 256u; d += THREADS) {
            uint32_t run = 0;
            if (d <= mask) {
#pragma unroll
                for (int w = 0; w < WARPS; w++) {
                    const uint32_t c = s_cnt[w * 256u + d];
                    s_cnt[w * 256u + d] = run;
                    run += c;
                }
            }
            s_dig[d] = run;
        }
        __syncthreads();
        if (warp == 0) {
            uint32_t v[8], sum = 0;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                v[q] = s_dig[lane * 8u + q];
                sum += v[q];
            }
            uint32_t inc = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, inc, o);
                if (lane >= (uint32_t)o) inc += t;
            }
            uint32_t run = inc - sum;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                s_dig[lane * 8u + q] = run;
                run += v[q];
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; k++) {
            if (k < steps && first + 32u * k < n) {
                const uint32_t d = (word[k] >> shift) & mask;
                s_word[s_dig[d] + s_cnt[warp * 256u + d] + rank[k]] = word[k];
            }
        }
        __syncthreads();
        if (p + 1 < passes) {
#pragma unroll
            for (int k = 0; k < ITEMS; k++) {
                const uint32_t i = first + 32u * k;
                if (k < steps && i < n) word[k] = s_word[i];
            }
        }
    }
    // every value is on its way before the first is written
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        const uint32_t i = tid + k * THREADS;
        if (i < n) {
            word[k] = s_word[i];
            rank[k] = vals_in[e0 + (word[k] & ((1u << IDX) - 1u))];
        }
    }
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        const uint32_t i = tid + k * THREADS;
        if (i < n) {
            keys_out[out + i] = base + (K)(word[k] >> IDX);
            vals_out[out + i] = rank[k];
        }
    }
}

template <class K, int THREADS, int ITEMS, int BLOCKS>
static int launch_sort_local(ochre_gpu_ctx* ctx, LocalSortArgs a, uint32_t first, uint32_t rasters, cudaStream_t s) {
    if (rasters == 0) return OCHRE_OK;
    constexpr size_t smem = local_sort_smem<THREADS, ITEMS>();
    if (smem > 48 * 1024)
        OCHRE_CUDA_TRY(cudaFuncSetAttribute(k_sort_local<K, THREADS, ITEMS, BLOCKS>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    a.first = first;
    OCHRE_LAUNCH(ctx, "sort_local", s, launch_after(
        k_sort_local<K, THREADS, ITEMS, BLOCKS>, rasters, THREADS, smem, s, ctx->keys.as<K>(),
        ctx->vals.as<uint32_t>(), ctx->keys_alt.as<K>(), ctx->vals_alt.as<uint32_t>(), a));
    OCHRE_CUDA_TRY(cudaGetLastError());
    return OCHRE_OK;
}
// Few rasters go in one launch, all to the size the largest of them needs
// (three short launches one after the other took 53 us for a document of 415
// paths, one 16; the device-wide sort 47).
constexpr uint32_t LOCAL_SORT_FEW = 1024;
template <class K>
static int sort_local(ochre_gpu_ctx* ctx, const LocalSortArgs& a, cudaStream_t s) {
    const uint32_t R = a.n_rasters, few = R <= LOCAL_SORT_FEW;
    uint32_t large = a.large, middle = a.middle;
    if (few && large) {
        large = R;
        middle = 0;
    } else if (few && middle) {
        middle = R;
    }
    int st = launch_sort_local<K, 512, 16, 2>(ctx, a, 0u, large, s);
    if (st == OCHRE_OK) st = launch_sort_local<K, 256, 16, 4>(ctx, a, large, middle, s);
    if (st == OCHRE_OK) st = launch_sort_local<K, 128, 8, 8>(ctx, a, large + middle, R - middle - large, s);
    return st;
}
static_assert(LOCAL_SORT_SMALL == 128 * 8 && LOCAL_SORT_MIDDLE == 256 * 16 && LOCAL_SORT_LARGE == 512 * 16 &&
                  LOCAL_SORT_LARGE <= 1u << LOCAL_SORT_IDX_BITS,
              "block sizes");

int stage_sort_local(ochre_gpu_ctx* ctx, const ochre_batch* in, cudaStream_t s) {
    const DevScalars* hs = host_scalars(ctx);
    const LocalSortArgs a{ctx->raster_run.as<RasterRun>(), in->n_rasters, hs->n_sort[0], hs->n_sort[1], 0u,
                          ctx->raster_bbox.as<int4>(), ctx->raster_keybase.as<uint64_t>(),
                          &dev_scalars(ctx)->line_ent_total};
    const int st = ctx->keys64 ? sort_local<uint64_t>(ctx, a, s) : sort_local<uint32_t>(ctx, a, s);
    if (st != OCHRE_OK) return st;
    std::swap(ctx->keys, ctx->keys_alt);
    std::swap(ctx->vals, ctx->vals_alt);
    return OCHRE_OK;
}

}  // namespace ochre
