// Stage 4: sorted entries -> 8x8 alpha tiles and solid spans.
//
// Reference: the tile loop of finish (rasterizer.rs:213-267):
//   * scatter-add area/height of every increment of a tile (:223-228);
//   * alpha = min(|accum + area| * 256, 255) as u8 with accum the running
//     sum of heights along the pixel row, seeded by the carry `prev` from
//     the tiles to the left on the same tile row (:232-239, 243-250);
//   * a span between this tile and the next one on the row when there is a
//     gap and the running tile-row-crossing winding (never reset, so a
//     prefix over the whole raster) is nonzero (:252-265).
//
// Tiles are numbered in sorted order, which is the reference's callback
// order.  One scan over the sorted entries numbers the tiles and their rows and
// sums the crossing signs, and writes each tile's metadata at its head; the
// spans follow from it by a scan over the tiles.
// Coverage (row form) runs one warp per whole tile row (raster, tile_y) at a
// time, taken by ticket: chunk by chunk of TILES_PER_WARP tiles it adds the
// increments the emit walk stored for the chunk's bins into shared-memory
// accumulators, then walks the tiles left to right keeping the row carry in
// registers, so no carry ever crosses warps.  The block form gives each warp
// an aligned block of tiles and takes the carry from the block before by
// look-back.
#include <algorithm>

#include "common.cuh"
#include "internal.h"
#include "scan.cuh"
#include "tiles.cuh"

namespace ochre {

// Tile heads: the first bin entry of every run of equal keys.  One single-pass
// scan numbers the tiles and sums the crossing signs; a tile's winding
// (rasterizer.rs:219, 253-258: the signs of all crossings of its raster sorted
// before it, never reset) is the sum before its head minus that of all earlier
// rasters.
struct HeadScan {
    uint32_t heads;
    int32_t w;
};
struct OpHead {
    __device__ __forceinline__ HeadScan operator()(HeadScan a, HeadScan b) const {
        return HeadScan{a.heads + b.heads, a.w + b.w};
    }
};
// Beside its look-back words every block publishes its last head: 1 + the
// entry (0: the block has none), under the scan's flag.  The last one before a
// block (0: none), by a whole warp, 32 blocks a round.
__device__ __forceinline__ uint32_t head_before(const uint64_t* last_head, uint32_t block, uint32_t flag, uint32_t* err) {
    const uint32_t lane = threadIdx.x & 31u;
    long long spins = 0;
    const long long poll_limit = spin_limit(err);
    for (int64_t top = (int64_t)block - 1; top >= 0;) {
        const int64_t j = top - lane;
        const uint64_t v = j >= 0 ? ld_relaxed64(last_head + j) : (uint64_t)flag << 32;
        if (__any_sync(0xffffffffu, (uint32_t)(v >> 32) != flag)) {   // (published before its look-back: on its way)
            if (wait_give_up_warp(spins, poll_limit, err)) break;
            continue;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, (uint32_t)v != 0u);
        if (m) return __shfl_sync(0xffffffffu, (uint32_t)v, __ffs(m) - 1);
        top -= 32;
    }
    return 0u;
}

// A warp takes HEAD_ITEMS steps of 32 consecutive entries, so every load is
// one segment of 128 bytes, a head's number is a count of ballot bits, and so
// is the sum of the signs before it (they are +-1 but for walks that snap far,
// which take a shuffle scan).  Each head then gathers its bin record once; a
// row starts where raster or tile row differ from the head before, a shuffle
// away.  For a warp's first head that is the last bin before the warp: one of
// the 32 entries there, loaded with the warp's own, and where they are all
// crossings (a tile's crossings may be any number, also of a tile without bins: a
// line that ends in a tile's corner leaves its crossing where it has no cell)
// the last head of the warps and blocks before.  Bound by those gathers.  For the 178 M entries and 70 M tiles of
// 20,000 uneven paths a generic scan (threads own 8 consecutive entries), the
// metadata gathered by a kernel of its own and a scan for the rows took 3.40
// ms; 1.33 ms here (the coverage kernel finds the rows itself).  Few entries
// take 4 steps a warp instead of 16, so that more warps share the gathers'
// latency: one path's 6,339 entries 16 us at 16 steps, 10 us at 4.  The records
// of eight steps are gathered together (one step after the other, the values
// kept in indexed registers, which are memory: 1.34 ms; four steps 1.14; eight 1.04;
// 19 M entries of strokes 162 -> 123 us, one path 10 -> 8 us).
constexpr int HEAD_BLOCK = 256;
struct HeadArgs {
    const uint32_t* vals;
    const BinRec* bins;
    const int32_t* raster_wbase;
    uint64_t n;
    const uint32_t* n_dev;   // device-held entry count (graph replays), else null
    uint32_t n_rasters;
    uint32_t* head;
    uint32_t* xy;
    uint32_t* rf;
    uint32_t* raster_tile_off;
    HeadScan* total;
    uint32_t* n_rows;        // zero before the launch
};
template <class K, int HEAD_ITEMS>
__global__ void __launch_bounds__(HEAD_BLOCK) k_tile_heads(const K* keys, HeadArgs A,
                                                           ScanStatus<HeadScan>* status, uint64_t* last_head,
                                                           uint32_t* ticket, uint32_t ticket_base, uint32_t tag,
                                                           uint32_t* err) {
    dependent_start();
    constexpr int HEAD_GATHER = HEAD_ITEMS < 8 ? HEAD_ITEMS : 8;   // steps whose records are gathered together
    constexpr int WARPS = HEAD_BLOCK / 32, HEAD_TILE = HEAD_BLOCK * HEAD_ITEMS;
    constexpr uint32_t FULL = 0xffffffffu;
    __shared__ uint32_t s_tile, s_rows;
    __shared__ HeadScan s_warp[WARPS];
    __shared__ uint32_t s_last[WARPS];   // 1 + the warp's last head (0: none)
    __shared__ HeadScan s_prefix;
    const uint64_t n = dev_count(A.n, A.n_dev);
    if (run_aborted(err)) return;   // a wait of the sort gave up: the values are not valid indices
    if (threadIdx.x == 0) {
        s_tile = atomicAdd(ticket, 1u) - ticket_base;
        s_rows = 0u;
    }
    __syncthreads();
    const uint32_t tile = s_tile;
    if ((uint64_t)tile * HEAD_TILE >= n) return;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const uint64_t base = (uint64_t)tile * HEAD_TILE + (uint64_t)warp * (32 * HEAD_ITEMS);

    // heads and signs of the warp's entries
    uint32_t val[HEAD_ITEMS];
    uint32_t heads = 0;   // bit k: this lane's entry of step k is a head
    int32_t w = 0;
    uint32_t n_heads = 0;
    const uint32_t near = base > lane && base < n ? A.vals[base - 1 - lane] : CROSS_TAG;   // the entries before the warp
    {
        K key[HEAD_ITEMS];
        K before = 0;     // the key before the warp's first entry
#pragma unroll
        for (int k = 0; k < HEAD_ITEMS; k++) {
            const uint64_t i = base + k * 32 + lane;
            val[k] = i < n ? A.vals[i] : CROSS_TAG;   // (past the end: a crossing without a sign)
            key[k] = i < n ? keys[i] : (K)0;
        }
        if (base > 0 && base < n) before = keys[base - 1];
#pragma unroll
        for (int k = 0; k < HEAD_ITEMS; k++) {
            K left = shfl_up_T(key[k], 1);
            if (lane == 0) left = before;
            before = shfl_idx_T(key[k], 31);
            const uint64_t i = base + k * 32 + lane;
            const bool bin = !(val[k] & CROSS_TAG);
            const bool is = bin && (i == 0 || key[k] != left);
            if (is) heads |= 1u << k;
            n_heads += (uint32_t)__popc(__ballot_sync(FULL, is));
            if (!bin) w += (int32_t)(int8_t)(val[k] & 0xffu);
        }
    }
    const int32_t warp_w = __reduce_add_sync(FULL, w);
    const uint32_t last = __reduce_max_sync(FULL, heads ? (uint32_t)base + (31u - (uint32_t)__clz(heads)) * 32u + lane + 1u : 0u);
    if (lane == 0) {
        s_warp[warp] = HeadScan{n_heads, warp_w};
        s_last[warp] = last;
    }
    // raster and tile row of the last bin before the warp's entries
    uint32_t prev_r = 0xffffffffu;
    int prev_ty = 0;
    auto previous = [&](uint32_t value) {
        const BinRec* rec = A.bins + value;
        prev_r = rec->raster;
        prev_ty = div8((int)rec->y);
    };
    const uint32_t near_bins = __ballot_sync(FULL, !(near & CROSS_TAG));
    if (n_heads && near_bins) previous(__shfl_sync(FULL, near, __ffs(near_bins) - 1));
    __syncthreads();
    if (warp == 0) {
        HeadScan v = lane < (uint32_t)WARPS ? s_warp[lane] : HeadScan{0u, 0};
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const HeadScan o = shfl_up_T(v, d);
            if (lane >= (uint32_t)d) v = OpHead{}(o, v);
        }
        HeadScan ex = shfl_up_T(v, 1);
        if (lane == 0) ex = HeadScan{0u, 0};
        const HeadScan agg = shfl_idx_T(v, WARPS - 1);
        if (lane < (uint32_t)WARPS) s_warp[lane] = ex;
        const uint32_t block_last = __reduce_max_sync(FULL, lane < (uint32_t)WARPS ? s_last[lane] : 0u);
        if (lane == 0) st_relaxed64(last_head + tile, (uint64_t)(tag << 2 | SCAN_INC) << 32 | block_last);
        const HeadScan prefix = scan_lookback(tile, agg, OpHead{}, HeadScan{0u, 0}, status, tag, err);
        if (lane == 0) {
            s_prefix = prefix;
            if ((uint64_t)(tile + 1) * HEAD_TILE >= n) {
                const HeadScan t = OpHead{}(prefix, agg);
                *A.total = t;
                A.raster_tile_off[A.n_rasters] = t.heads;
            }
        }
    }
    __syncthreads();
    uint32_t t0 = s_prefix.heads + s_warp[warp].heads;   // tiles before the step
    int32_t w0 = s_prefix.w + s_warp[warp].w;            // signs before the step
    if (n_heads && !near_bins) {
        uint32_t before = __reduce_max_sync(FULL, lane < warp ? s_last[lane] : 0u);
        if (!before) before = head_before(last_head, tile, tag << 2 | SCAN_INC, err);
        if (before) previous(A.vals[before - 1u]);
    }
    uint32_t rows = 0;
    // HEAD_GATHER steps at a time: their values again (out of the cache) and
    // their records, all in flight before the first is used
#pragma unroll 1
    for (int k0 = 0; k0 < HEAD_ITEMS; k0 += HEAD_GATHER) {
        uint32_t v[HEAD_GATHER], rec_r[HEAD_GATHER], rec_xy[HEAD_GATHER];
#pragma unroll
        for (int q = 0; q < HEAD_GATHER; q++) {
            const uint64_t i = base + (k0 + q) * 32 + lane;
            v[q] = i < n ? A.vals[i] : CROSS_TAG;
        }
#pragma unroll
        for (int q = 0; q < HEAD_GATHER; q++) {
            rec_r[q] = rec_xy[q] = 0u;
            if (heads >> (k0 + q) & 1u) {
                const uint4 rec = *reinterpret_cast<const uint4*>(A.bins + v[q]);
                rec_r[q] = rec.y;
                rec_xy[q] = rec.z;
            }
        }
#pragma unroll
        for (int q = 0; q < HEAD_GATHER; q++) {
            const bool is = heads >> (k0 + q) & 1u;
            const bool cross = (v[q] & CROSS_TAG) != 0u;
            const int sign = cross ? (int)(int8_t)(v[q] & 0xffu) : 0;
            const uint32_t hm = __ballot_sync(FULL, is);
            const uint32_t pos = __ballot_sync(FULL, sign == 1), neg = __ballot_sync(FULL, sign == -1);
            int wb = __popc(pos & lt) - __popc(neg & lt), wt = __popc(pos) - __popc(neg);
            if (__any_sync(FULL, sign > 1 || sign < -1)) {
                int inc = sign;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int o = __shfl_up_sync(FULL, inc, d);
                    if (lane >= (uint32_t)d) inc += o;
                }
                wb = inc - sign;
                wt = __shfl_sync(FULL, inc, 31);
            }
            if (hm) {
                const uint32_t r = rec_r[q], at = rec_xy[q];
                const int tx = div8(tile_tx(at)), ty = div8(tile_ty(at));
                // the head before: in this step, else the last one so far (or the
                // last bin before the warp: the same tile as the head before)
                const uint32_t below = hm & lt;
                const int src = below ? 31 - __clz(below) : 0;
                const uint32_t sr = __shfl_sync(FULL, r, src);
                const int sy = __shfl_sync(FULL, ty, src);
                const uint32_t pr = below ? sr : prev_r;
                const int py = below ? sy : prev_ty;
                const bool row = is && (pr != r || py != ty);
                if (is) {
                    const uint32_t t = t0 + (uint32_t)__popc(below);
                    A.head[t] = (uint32_t)(base + (k0 + q) * 32 + lane);
                    A.xy[t] = pack_tile(tx, ty);
                    A.rf[t] = r | (w0 + wb != A.raster_wbase[r] ? RF_WIND : 0u) | (row ? RF_ROW : 0u);
                    if (pr != r) A.raster_tile_off[r] = t;
                }
                rows += (uint32_t)__popc(__ballot_sync(FULL, row));
                const int last = 31 - __clz(hm);
                prev_r = __shfl_sync(FULL, r, last);
                prev_ty = __shfl_sync(FULL, ty, last);
            }
            t0 += (uint32_t)__popc(hm);
            w0 += wt;
        }
    }
    if (lane == 0 && rows) atomicAdd(&s_rows, rows);
    __syncthreads();
    if (threadIdx.x == 0 && s_rows) atomicAdd(A.n_rows, s_rows);
}

// Graph replays: the tile count against its capacity; above it there is no
// tile, no row and no span to work on.
__global__ void k_plan_tiles(DevScalars* ds, uint32_t cap) {
    dependent_start();
    if (ds->n_tiles > cap) {
        ds->n_tiles = 0u;
        ds->n_rows = 0u;
        atomicOr(&ds->err, ERR_CAPACITY);
    }
}

// Shared-memory accumulators of one tile: per pixel row 8 areas, 8 heights
// and 4 floats of padding, so a cell's place is linear in x and y and the
// 128-bit row loads of eight lanes (rows 0-7 of one tile) hit distinct banks.
constexpr int ACC_ROW = 20;                // floats per pixel row
constexpr int ACC_H = 8;                   // offset of a row's heights
constexpr int ACC_STRIDE = 8 * ACC_ROW;    // floats per tile

// Stage of one batch of bins (per warp).
struct BinStage {
    // first increment less the batch's cells before it (a cell's increment is
    // at that plus its number in the batch); steps (bits 0-15) and place of
    // the first cell (16-31)
    uint2 bin[32];
    // batch's cells before the bin (bits 16-31; [32] all of them), and what a
    // step in y adds to the place (bits 8-15, signed) and, beyond that, a
    // step in x instead (0-7, signed)
    uint32_t pre[33];
};

constexpr int CELL_UNROLL = 4;

// A warp's entry (none: no cells): its bin's record, and the accumulator slot
// of its tile.  Adds the stored increments of the warp's bins into the
// accumulators (rasterizer.rs:223-228).  The bins of the 32 entries are
// staged, then the warp's lanes take equal contiguous ranges of their cells,
// so every lane has cells whatever the bins' lengths; a cell's place follows
// from its bin's first cell and steps.
__device__ __forceinline__ void add_increments(bool bin, uint4 rec, int slot, const float2* incs, float* acc,
                                               BinStage& st) {
    const int lane = threadIdx.x & 31;
    const uint32_t n = bin ? (rec.w >> 16) & 0xffu : 0u;
    uint32_t pre = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, pre, d);
        if (lane >= d) pre += o;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, pre, 31);
    const int sy = rec.w & (2u << 24) ? -ACC_ROW : ACC_ROW, sxy = (rec.w & (1u << 24) ? -1 : 1) - sy;
    const uint32_t place0 = (uint32_t)(slot * ACC_STRIDE) + (rec.z >> 16 & 7u) * ACC_ROW + (rec.z & 7u);
    st.bin[lane] = make_uint2(rec.x - (pre - n), (rec.w & 0xffffu) | place0 << 16);
    st.pre[lane] = (pre - n) << 16 | ((uint32_t)sy & 0xffu) << 8 | ((uint32_t)sxy & 0xffu);
    if (lane == 31) st.pre[32] = total << 16;
    __syncwarp();
    // Each lane takes a contiguous range of the batch's cells: one search
    // for the bin of its first cell, then bin after bin; CELL_UNROLL
    // cells at a time, their increment loads all in flight before the
    // first is added.
    const uint32_t per = (total + 31u) >> 5;
    uint32_t c = lane * per;
    const uint32_t c_end = min(c + per, total);
    if (c < c_end) {
        int b = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
            if (st.pre[b + step] >> 16 <= c) b += step;
        uint32_t own = st.pre[b], after = st.pre[b + 1], base = own >> 16, next = after >> 16;
        uint2 bin_b = st.bin[b];
        while (c < c_end) {
            float2 ah[CELL_UNROLL];
            int where[CELL_UNROLL];   // place, or -1
#pragma unroll
            for (int u = 0; u < CELL_UNROLL; u++) {
                where[u] = -1;
                ah[u] = make_float2(0.0f, 0.0f);
                if (c < c_end) {
                    while (c >= next) {   // on to the next bin with cells
                        b++;
                        own = after;
                        after = st.pre[b + 1];
                        base = next;
                        next = after >> 16;
                        bin_b = st.bin[b];
                    }
                    const uint32_t k = c - base;
                    const int nx = __popc(bin_b.y & ((1u << k) - 1u));
                    where[u] = (int)(bin_b.y >> 16) + (int)k * (int)(int8_t)(own >> 8) + nx * (int)(int8_t)own;
                    ah[u] = incs[bin_b.x + c];
                    c++;
                }
            }
#pragma unroll
            for (int u = 0; u < CELL_UNROLL; u++) {
                if (where[u] < 0) continue;
                atomicAdd(acc + where[u], ah[u].x);
                atomicAdd(acc + where[u] + ACC_H, ah[u].y);
            }
        }
    }
    __syncwarp();
}
// An entry's tile among a chunk's: the heads before the batch and those up to
// it (my_head: lane i holds the first entry of the chunk's i-th later tile).
__device__ __forceinline__ int entry_slot(uint32_t my_head, uint32_t eb) {
    const int before = __popc(__ballot_sync(0xffffffffu, my_head < eb));
    const uint32_t in = __reduce_or_sync(0xffffffffu, my_head - eb < 32u ? 1u << (my_head - eb) : 0u);
    return before + __popc(in & (0xffffffffu >> (31 - (threadIdx.x & 31))));
}

// The entries of a run of tiles, 32 a batch: a batch's entries are loaded
// while the batch before adds, its bins' records when that one is done.
struct EntryRun {
    const uint32_t* vals;
    const BinRec* bins;
    uint32_t end;   // entries there are
    uint32_t eb, v;
    uint4 rec;
    __device__ __forceinline__ void load_vals() {
        const uint32_t e = eb + (threadIdx.x & 31);
        v = e < end ? vals[e] : CROSS_TAG;
    }
    __device__ __forceinline__ void load_recs() {
        rec = v & CROSS_TAG ? make_uint4(0u, 0u, 0u, 0u) : *reinterpret_cast<const uint4*>(bins + v);
    }
    __device__ __forceinline__ void begin(uint32_t e) {
        eb = e;
        load_vals();
        load_recs();
    }
    // Adds the entries up to e1, the end of a chunk of tiles (my_head: see
    // entry_slot; crossing entries in between are skipped).
    __device__ __forceinline__ void add_to(uint32_t e1, uint32_t my_head, const float2* incs, float* acc,
                                           BinStage& st) {
        for (;;) {
            const bool bin = eb + (threadIdx.x & 31) < e1 && !(v & CROSS_TAG);
            const uint4 now = rec;
            const int slot = entry_slot(my_head, eb);
            eb = min(eb + 32u, e1);
            load_vals();
            add_increments(bin, now, slot, incs, acc, st);
            load_recs();
            if (eb >= e1) break;
        }
    }
};

// A tile's pixel row: areas and heights.
__device__ __forceinline__ void load_row(const float* row, float* a, float* h) {
    const float4* q = reinterpret_cast<const float4*>(row);
    const float4 a0 = q[0], a1 = q[1], h0 = q[2], h1 = q[3];
    a[0] = a0.x; a[1] = a0.y; a[2] = a0.z; a[3] = a0.w; a[4] = a1.x; a[5] = a1.y; a[6] = a1.z; a[7] = a1.w;
    h[0] = h0.x; h[1] = h0.y; h[2] = h0.z; h[3] = h0.w; h[4] = h1.x; h[5] = h1.y; h[6] = h1.z; h[7] = h1.w;
}
// The row shaded from the carry into it (rasterizer.rs:232-250): along the row
// the cells are added in the reference's order.
__device__ __forceinline__ void shade_row(const float* a, const float* h, float carry, bool cov_signed, uint32_t t, int y,
                                          uint8_t* __restrict__ out_alpha, float* __restrict__ out_cov) {
    float accum = carry;
    uint32_t al[8];
    float cv[8];
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const float sum = accum + a[c];
        cv[c] = cov_signed ? sum : fabsf(sum);
        al[c] = alpha_bits(sum);
        accum = accum + h[c];
    }
    reinterpret_cast<uint2*>(out_alpha + (size_t)t * 64)[y] =
        make_uint2(pack_bytes(al[0], al[1], al[2], al[3]), pack_bytes(al[4], al[5], al[6], al[7]));
    if (out_cov) {
        float4* o = reinterpret_cast<float4*>(out_cov + (size_t)t * 64 + 8 * y);
        o[0] = make_float4(cv[0], cv[1], cv[2], cv[3]);
        o[1] = make_float4(cv[4], cv[5], cv[6], cv[7]);
    }
}

// Coverage, block form: one warp per aligned block of TILES_PER_WARP
// consecutive tiles (blocks may cross rows).  A block that continues a row
// from the previous block resolves its carry by decoupled look-back: blocks
// publish the row sums of their last row segment (taken by atomic ticket,
// bounded spins).  Used when there are too few tile rows to occupy the GPU
// with one warp per row; with many long rows the look-back chains grow long,
// and the row form below is used instead.  Entries as there: 128 dense scenes
// (382,000 tiles, 16 million bins) 546 -> 532 us, 256 shapes 36 -> 32 us.
template <int CH>
__global__ void __launch_bounds__(128) k_tile_cov_blocks(
    const uint32_t* vals, const BinRec* bins, const float2* incs,
    TileView tiles, uint32_t n_tiles, const uint32_t* n_dev, TileBlockState* state, uint32_t* ticket,
    uint32_t* __restrict__ out_xy, uint8_t* __restrict__ out_alpha, float* __restrict__ out_cov, uint32_t* err,
    bool cov_signed) {
    dependent_start();
    constexpr int WARPS = 4;
    // device-held count (graph replays): blocks past it end before publishing
    n_tiles = (uint32_t)dev_count(n_tiles, n_dev);
    // an earlier wait of the run gave up: the tile data is not valid (the
    // blocks' own waits then give up at once too)
    if (run_aborted(err)) return;
    __shared__ __align__(16) float s_acc[WARPS][CH][ACC_STRIDE];
    __shared__ uint32_t s_head[WARPS][CH + 1];   // (and the end of the block's entries)
    __shared__ uint32_t s_xy[WARPS][CH], s_rf[WARPS][CH];
    __shared__ BinStage s_stage[WARPS];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t blk = 0;
    if (lane == 0) blk = atomicAdd(ticket, 1u);
    blk = __shfl_sync(0xffffffffu, blk, 0);
    const uint32_t t0 = blk * CH;
    if (t0 >= n_tiles) return;
    const int nt = (int)min((uint32_t)CH, n_tiles - t0);
    float (*acc)[ACC_STRIDE] = s_acc[wid];

    // tile metadata
    for (int i = lane; i <= nt; i += 32) {
        s_head[wid][i] = t0 + i < n_tiles ? tiles.head[t0 + i] : tiles.end();
        if (i < nt) {
            s_xy[wid][i] = tiles.xy[t0 + i];
            s_rf[wid][i] = tiles.rf[t0 + i];
        }
    }
    for (int k = lane; k < nt * (ACC_STRIDE / 4); k += 32)
        reinterpret_cast<float4*>(acc[0])[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncwarp();

    // The stored increments of every bin of the block (rasterizer.rs:97-106,
    // 223-228).  The block's entries are contiguous; crossing entries in
    // between are skipped.
    const uint32_t e0 = s_head[wid][0], e1 = s_head[wid][nt];
    const uint32_t my_head = lane > 0 && lane < nt ? s_head[wid][lane] : 0xffffffffu;
    EntryRun run{vals, bins, e1};
    run.begin(e0);
    run.add_to(e1, my_head, incs, acc[0], s_stage[wid]);

    // Each lane owns one pixel row of one tile: lane = 8 * g + y, four tiles
    // (g) per pass.
    const int y = lane & 7, g = lane >> 3;

    // Row sums of the block's last row segment -> publish (decoupled).
    int last_seg = 0;
    for (int i = nt - 1; i > 0; i--)
        if (s_rf[wid][i] & RF_ROW) { last_seg = i; break; }
    const bool starts_mid_row = !(s_rf[wid][0] & RF_ROW);
    const bool one_segment = last_seg == 0 && starts_mid_row;
    float part = 0.0f;
    for (int i = last_seg + g; i < nt; i += 4) {
        const float4 h0 = *reinterpret_cast<const float4*>(&acc[i][ACC_ROW * y + ACC_H]);
        const float4 h1 = *reinterpret_cast<const float4*>(&acc[i][ACC_ROW * y + ACC_H + 4]);
        part += ((h0.x + h0.y) + (h0.z + h0.w)) + ((h1.x + h1.y) + (h1.z + h1.w));
    }
    part += __shfl_xor_sync(0xffffffffu, part, 8);
    part += __shfl_xor_sync(0xffffffffu, part, 16);   // every lane of row y holds its sum
    float seg[8];
#pragma unroll
    for (int r = 0; r < 8; r++) seg[r] = __shfl_sync(0xffffffffu, part, r);
    float carry_in = 0.0f;   // per lane: carry of this lane's pixel row
    if (lane == 0) {
        TileBlockState* me = state + blk;
        if (!one_segment) {
            for (int r = 0; r < 8; r++) st_relaxed(reinterpret_cast<uint32_t*>(&me->inc[r]), __float_as_uint(seg[r]));
            st_release(&me->flag, 2u);
        } else {
            for (int r = 0; r < 8; r++) st_relaxed(reinterpret_cast<uint32_t*>(&me->agg[r]), __float_as_uint(seg[r]));
            st_release(&me->flag, 1u);
        }
    }
    if (starts_mid_row) {
        // Warp-cooperative decoupled look-back over the preceding blocks, 32
        // per round (a long tile row spans many blocks): lane k inspects
        // block top - k; the nearest inclusive value ends the walk.
        float c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        int64_t top = (int64_t)blk - 1;
        long long spins = 0;
        const long long poll_limit = spin_limit(err);
        while (top >= 0) {
            const int64_t j = top - lane;
            uint32_t f = 2u;   // before block 0: an inclusive zero
            if (j >= 0) f = ld_acquire(&state[j].flag);
            const uint32_t m2 = __ballot_sync(0xffffffffu, f == 2u);
            const int limit = m2 ? __ffs(m2) - 1 : 31;   // lanes [0, limit] are needed
            const uint32_t need = limit == 31 ? 0xffffffffu : ((1u << (limit + 1)) - 1u);
            if (__ballot_sync(0xffffffffu, f == 0u) & need) {
                if (wait_give_up_warp(spins, poll_limit, err)) break;
                if (spins > 16) __nanosleep(64);
                continue;
            }
            float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            if (lane <= limit && j >= 0) {
                const float* src = f == 2u ? state[j].inc : state[j].agg;
#pragma unroll
                for (int r = 0; r < 8; r++) v[r] = __uint_as_float(ld_relaxed(reinterpret_cast<const uint32_t*>(src + r)));
            }
#pragma unroll
            for (int r = 0; r < 8; r++) {
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) v[r] += __shfl_xor_sync(0xffffffffu, v[r], d);
                c[r] += v[r];
            }
            if (m2) break;
            top -= 32;
        }
        if (one_segment && lane == 0) {
            TileBlockState* me = state + blk;
            for (int r = 0; r < 8; r++)
                st_relaxed(reinterpret_cast<uint32_t*>(&me->inc[r]), __float_as_uint(c[r] + seg[r]));
            st_release(&me->flag, 2u);
        }
#pragma unroll
        for (int r = 0; r < 8; r++)
            if (y == r) carry_in = c[r];
    }

    // Tiles left to right (rasterizer.rs:232-250): along its row a lane adds
    // the cells in the reference's order; the carry into a tile is the carry
    // into the previous tile of the row plus that tile's row sum (reset at
    // each row start), a segmented scan over the four tiles of a pass.
    float carry_row = carry_in;   // carry into the pass's first tile, row y
    for (int i0 = 0; i0 < nt; i0 += 4) {
        const int i = i0 + g;
        const bool valid = i < nt;
        float a[8], h[8];
        if (valid) {
            load_row(&acc[i][ACC_ROW * y], a, h);
        } else {
#pragma unroll
            for (int c = 0; c < 8; c++) a[c] = h[c] = 0.0f;
        }
        const float rs = ((h[0] + h[1]) + (h[2] + h[3])) + ((h[4] + h[5]) + (h[6] + h[7]));
        const bool head = valid && i > 0 && (s_rf[wid][i] & RF_ROW);
        // segmented inclusive scan of rs over g (lanes 8 apart), then shifted
        // by one tile: ex = the sum of rs since the last row start before g
        float v = rs;
        bool f = head;
#pragma unroll
        for (int d = 8; d < 32; d <<= 1) {
            const float vo = __shfl_up_sync(0xffffffffu, v, d);
            const bool fo = __shfl_up_sync(0xffffffffu, f ? 1 : 0, d) != 0;
            if (lane >= d) {
                if (!f) v = vo + v;
                f = f || fo;
            }
        }
        float ex = __shfl_up_sync(0xffffffffu, v, 8);
        bool exf = __shfl_up_sync(0xffffffffu, f ? 1 : 0, 8) != 0;
        if (g == 0) {
            ex = 0.0f;
            exf = false;
        }
        const float carry = head ? 0.0f : (exf ? ex : carry_row + ex);
        carry_row = __shfl_sync(0xffffffffu, carry + rs, 24 + y);
        if (valid) {
            const uint32_t t = t0 + i;
            shade_row(a, h, carry, cov_signed, t, y, out_alpha, out_cov);
            if (y == 0) {
                const uint32_t xy = s_xy[wid][i];
                out_xy[t] = pack_tile(tile_tx(xy) * 8, tile_ty(xy) * 8);
            }
        }
    }
}

// Coverage, row form: one warp per tile row (see the file comment).  The row
// carry (rasterizer.rs:243-250) never leaves the warp.  A ticket is a range of
// tiles; its warp takes the rows that start there, tile after tile.
//
// Bound by instruction issue and, with the accumulators' shared memory
// limiting the warps in flight, by the chain tile -> entry -> bin -> increment of
// dependent loads.  So the warp holds the metadata of the next 32 to 64 tiles,
// and a batch's entries are loaded while the batch before adds, its bins while
// that one shades; a cell's place is two multiply-adds from its bin's first
// one (rows of 20 floats, areas and heights side by side); and the shading
// leaves the accumulators zero.  70 million tiles, 689 million increments:
// 8.04 ms -> 7.25 ms; 5.8 million tiles of strokes 885 -> 785 us.
constexpr uint32_t ROW_RANGE = 32;   // tiles per ticket, and per window of metadata
template <int CH>
__global__ void __launch_bounds__(128, CH == 8 ? 9 : 1) k_tile_cov(
    const uint32_t* vals, const BinRec* bins, const float2* incs,
    TileView tiles, uint32_t n_tiles, const uint32_t* n_dev, uint32_t* ticket, uint32_t* __restrict__ out_xy,
    uint8_t* __restrict__ out_alpha, float* __restrict__ out_cov, const uint32_t* err, bool cov_signed) {
    dependent_start();
    constexpr int WARPS = 4;
    // an earlier wait of the run gave up: the tile data is not valid
    if (run_aborted(err)) return;
    __shared__ __align__(16) float s_acc[WARPS][CH * ACC_STRIDE];
    __shared__ BinStage s_stage[WARPS];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // lane = 8 * g + y: pixel row y of the g-th tile of a pass of four
    const int y = lane & 7, g = lane >> 3;
    n_tiles = (uint32_t)dev_count(n_tiles, n_dev);
    const uint32_t n_ent = tiles.end();
    float* acc = s_acc[wid];
    for (int q = lane; q < CH * (ACC_STRIDE / 4); q += 32)
        reinterpret_cast<float4*>(acc)[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    // 32 tiles' metadata; past the last tile the end of the entries, a row start
    struct Window {
        uint32_t head, xy, rf;
    };
    auto window = [&](uint32_t t) {
        Window w{n_ent, 0u, RF_ROW};
        t += lane;
        if (t < n_tiles) w = Window{tiles.head[t], tiles.xy[t], tiles.rf[t]};
        return w;
    };
    EntryRun run{vals, bins, n_ent};
    uint32_t range = 0;
    if (lane == 0) range = atomicAdd(ticket, 1u);
    for (;;) {
        uint32_t w0 = __shfl_sync(0xffffffffu, range, 0) * ROW_RANGE;   // the window's first tile
        if (w0 >= n_tiles) return;
        const uint32_t range_end = w0 + ROW_RANGE;
        if (lane == 0) range = atomicAdd(ticket, 1u);
        Window win = window(w0), after = window(range_end);
        const uint32_t starts = __ballot_sync(0xffffffffu, w0 + lane < n_tiles && (win.rf & RF_ROW));
        if (!starts) continue;
        uint32_t t0 = w0 + (uint32_t)__ffs(starts) - 1u;
        run.begin(__shfl_sync(0xffffffffu, win.head, (int)(t0 - w0)));
        float carry_row = 0.0f;   // carry into the next tile, pixel row y
        for (;;) {
            // the chunk: the row's next tiles, at most CH
            const int at = (int)(t0 - w0) + lane;   // (lane <= CH: less than 64)
            auto pick = [&](uint32_t a, uint32_t b) {
                const uint32_t x = __shfl_sync(0xffffffffu, a, at & 31), z = __shfl_sync(0xffffffffu, b, at & 31);
                return at < 32 ? x : z;
            };
            const uint32_t head = pick(win.head, after.head), xy = pick(win.xy, after.xy), rf = pick(win.rf, after.rf);
            const uint32_t em = __ballot_sync(0xffffffffu, lane > 0 && lane <= CH && (rf & RF_ROW));
            const int nt = em ? __ffs(em) - 1 : CH;
            if (lane < nt) out_xy[t0 + lane] = pack_tile(tile_tx(xy) * 8, tile_ty(xy) * 8);
            const uint32_t e1 = __shfl_sync(0xffffffffu, head, nt);
            const uint32_t my_head = lane > 0 && lane < nt ? head : 0xffffffffu;

            // The stored increments of every bin of the chunk
            // (rasterizer.rs:97-106, 223-228).
            run.add_to(e1, my_head, incs, acc, s_stage[wid]);

            // Tiles left to right (rasterizer.rs:232-250); the carry into a
            // tile is the carry into the previous tile plus that tile's row
            // sum.  The accumulators are left zero.
            for (int i0 = 0; i0 < nt; i0 += 4) {
                const int i = i0 + g;
                const bool valid = i < nt;
                float a[8], h[8];
                if (valid) {
                    float* row = acc + i * ACC_STRIDE + ACC_ROW * y;
                    load_row(row, a, h);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        reinterpret_cast<float4*>(row)[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                } else {
#pragma unroll
                    for (int c = 0; c < 8; c++) a[c] = h[c] = 0.0f;
                }
                const float rs = ((h[0] + h[1]) + (h[2] + h[3])) + ((h[4] + h[5]) + (h[6] + h[7]));
                // exclusive sum of rs over the tiles of the pass before this one
                float sum = rs;
#pragma unroll
                for (int d = 8; d < 32; d <<= 1) {
                    const float o = __shfl_up_sync(0xffffffffu, sum, d);
                    if (lane >= d) sum = o + sum;
                }
                float ex = __shfl_up_sync(0xffffffffu, sum, 8);
                if (g == 0) ex = 0.0f;
                const float carry = carry_row + ex;
                carry_row = __shfl_sync(0xffffffffu, carry + rs, 24 + y);
                if (valid) shade_row(a, h, carry, cov_signed, t0 + i, y, out_alpha, out_cov);
            }
            __syncwarp();
            t0 += (uint32_t)nt;
            if (em) {   // the row has ended
                if (t0 >= range_end || t0 >= n_tiles) break;
                carry_row = 0.0f;
            }
            if (t0 - w0 >= ROW_RANGE) {
                w0 += ROW_RANGE;
                win = after;
                after = window(w0 + ROW_RANGE);
            }
        }
    }
}

// Spans (rasterizer.rs:252-265): a tile is followed by one when the next tile
// of its row leaves a gap and its winding is nonzero.  A thread reads its 8
// tiles' metadata in 16-byte accesses (70 M tiles 488 -> 372 us) and writes
// only where there is something to write.
struct SpanIn {
    const uint32_t* xy;
    const uint32_t* rf;
    uint32_t n_tiles;
    const uint32_t* n_dev;   // device-held tile count (graph replays), else null
    __device__ __forceinline__ uint32_t operator()(uint64_t t) const {
        if (t + 1 >= dev_count(n_tiles, n_dev) || (rf[t + 1] & RF_ROW) || !(rf[t] & RF_WIND)) return 0u;
        return tile_tx(xy[t + 1]) > tile_tx(xy[t]) + 1 ? 1u : 0u;
    }
    using takes_all = void;
    template <int N>
    __device__ __forceinline__ void load_all(uint64_t t, uint32_t (&v)[N]) const {
        const bool last = t + N >= dev_count(n_tiles, n_dev);
        uint32_t f[N + 1], p[N + 1], w[N];
        load_words(rf + t, w);
#pragma unroll
        for (int k = 0; k < N; k++) f[k] = w[k];
        load_words(xy + t, w);
#pragma unroll
        for (int k = 0; k < N; k++) p[k] = w[k];
        f[N] = last ? RF_ROW : rf[t + N];
        p[N] = last ? 0u : xy[t + N];
#pragma unroll
        for (int k = 0; k < N; k++)
            v[k] = !(f[k + 1] & RF_ROW) && (f[k] & RF_WIND) && tile_tx(p[k + 1]) > tile_tx(p[k]) + 1 ? 1u : 0u;
    }
};
struct SpanOut {
    const uint32_t* xy;
    const uint32_t* rf;
    uint32_t n_tiles, n_rasters;
    const uint32_t* n_dev;
    uint32_t* out_xy;
    uint16_t* w;
    uint32_t* tile;
    uint32_t* raster_span_off;
    __device__ __forceinline__ void operator()(uint64_t t, uint32_t ex, uint32_t v) const {
        if (v) {
            const int tx = tile_tx(xy[t]), ty = tile_ty(xy[t]);
            out_xy[ex] = pack_tile((tx + 1) * 8, ty * 8);
            w[ex] = (uint16_t)((uint16_t)(tile_tx(xy[t + 1]) - tx - 1) * 8u);
            tile[ex] = (uint32_t)t;
        }
        const uint32_t r = rf[t] & RF_RASTER;
        if ((rf[t] & RF_ROW) && (t == 0 || (rf[t - 1] & RF_RASTER) != r)) raster_span_off[r] = ex;
        if (t + 1 == dev_count(n_tiles, n_dev)) raster_span_off[n_rasters] = ex + v;
    }
    using takes_all = void;
    template <int N>
    __device__ __forceinline__ void store_all(uint64_t t, uint32_t run, const uint32_t (&v)[N]) const {
        uint32_t f[N];
        load_words(rf + t, f);
#pragma unroll
        for (int k = 0; k < N; k++) {
            // (only a row start may be a raster's first tile; most tiles are neither)
            if (v[k] || (f[k] & RF_ROW) || t + k + 1 == dev_count(n_tiles, n_dev)) (*this)(t + k, run, v[k]);
            run += v[k];
        }
    }
};

// One launch of the coverage kernel with TPW tiles per warp (4 warps per CTA).
// Coverage launch.  With at least ROW_FORM_MIN_ROWS_PER_SM tile rows per SM
// the row form runs (persistent warps taking rows by ticket); otherwise the
// block form, whose look-back chains stay short when rows are few.
constexpr uint32_t ROW_FORM_MIN_ROWS_PER_SM = 64;

template <int TPW>
static void launch_tile_cov(ochre_gpu_ctx* ctx, const TileView& tiles, uint32_t T, uint32_t n_rows, bool want_cov,
                            cudaStream_t s) {
    DevScalars* ds = dev_scalars(ctx);
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    cudaMemsetAsync(&ds->ticket, 0, 4, s);
    float* cov = want_cov ? ctx->out_tile_cov.as<float>() : nullptr;
    // graph replays: T is the capacity and n_rows the planned row count; the
    // kernels read both counts on the device
    const uint32_t* t_dev = ctx->plan ? &ds->n_tiles : nullptr;
    const bool row_form = ctx->tune_chain_coverage_form == 2 ||
                          (ctx->tune_chain_coverage_form == 0 && n_rows >= ROW_FORM_MIN_ROWS_PER_SM * (uint32_t)sms);
    if (row_form) {
        // no more warps than rows, nor than the GPU keeps resident (16 CTAs of 4 warps per SM)
        const uint32_t ctas = (uint32_t)std::min<uint64_t>(((uint64_t)n_rows + 3) / 4, (uint64_t)sms * 16);
        launch_after(k_tile_cov<TPW>, ctas, 128, 0, s,
            ctx->vals.as<uint32_t>(), ctx->bins.as<BinRec>(), ctx->incs.as<float2>(), tiles, T, t_dev,
            &ds->ticket, ctx->out_tile_xy.as<uint32_t>(), ctx->out_tile_alpha.as<uint8_t>(), cov,
            &ds->err, ctx->cov_signed);
    } else {
        const uint32_t blocks = (T + TPW - 1) / TPW;
        cudaMemsetAsync(ctx->tile_state.p, 0, (size_t)blocks * sizeof(TileBlockState), s);
        launch_after(k_tile_cov_blocks<TPW>, (blocks + 3) / 4, 128, 0, s,
            ctx->vals.as<uint32_t>(), ctx->bins.as<BinRec>(), ctx->incs.as<float2>(), tiles, T, t_dev,
            ctx->tile_state.as<TileBlockState>(), &ds->ticket, ctx->out_tile_xy.as<uint32_t>(),
            ctx->out_tile_alpha.as<uint8_t>(), cov, &ds->err, ctx->cov_signed);
    }
}

template <class K>
static int tiles_impl(ochre_gpu_ctx* ctx, const ochre_batch* in, uint64_t E, cudaStream_t s, uint32_t* n_tiles_out,
                      uint32_t* n_spans_out) {
    DevScalars* ds = dev_scalars(ctx);
    const uint32_t R = in->n_rasters;
    // tile metadata: no more tiles than entries
    OCHRE_CUDA_TRY(ctx->tile_head.ensure(E * 4));
    OCHRE_CUDA_TRY(ctx->tile_xy.ensure(E * 4));
    OCHRE_CUDA_TRY(ctx->tile_rf.ensure(E * 4));
    OCHRE_CUDA_TRY(ctx->out_raster_tile_off.ensure((size_t)(R + 1) * 4));
    OCHRE_CUDA_TRY(ctx->out_raster_span_off.ensure((size_t)(R + 1) * 4));
    // graph replays: E and T are capacities, the counts stay on the device
    const GraphPlan* plan = ctx->plan;
    const uint32_t* t_dev = plan ? &ds->n_tiles : nullptr;
    const uint32_t* e_dev = plan ? &ds->n_entries : nullptr;
    const TileView tiles{ctx->tile_head.as<uint32_t>(), ctx->tile_xy.as<uint32_t>(), ctx->tile_rf.as<uint32_t>(),
                         (uint32_t)E, e_dev};
    static_assert(offsetof(DevScalars, head_wind) == offsetof(DevScalars, n_tiles) + 4, "HeadScan layout");
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    const int steps = E < (uint64_t)sms * 2 * HEAD_BLOCK * 16 ? 4 : 16;
    const uint32_t blocks = (uint32_t)((E + HEAD_BLOCK * steps - 1) / (HEAD_BLOCK * steps));
    ScanSpace sp;
    OCHRE_CUDA_TRY(scan_space(ctx, blocks * (sizeof(ScanStatus<HeadScan>) + sizeof(uint64_t)), blocks, 0u, s, &sp));
    const HeadArgs args{ctx->vals.as<uint32_t>(), ctx->bins.as<BinRec>(), ctx->raster_wbase.as<int32_t>(), E, e_dev, R,
                        ctx->tile_head.as<uint32_t>(), ctx->tile_xy.as<uint32_t>(), ctx->tile_rf.as<uint32_t>(),
                        ctx->out_raster_tile_off.as<uint32_t>(), reinterpret_cast<HeadScan*>(&ds->n_tiles),
                        &ds->n_rows};
    auto* status = reinterpret_cast<ScanStatus<HeadScan>*>(sp.status);
    auto* last_head = reinterpret_cast<uint64_t*>(status + blocks);
    if (steps == 4)
        OCHRE_LAUNCH(ctx, "tile_heads", s, launch_after(k_tile_heads<K, 4>, blocks, HEAD_BLOCK, 0, s,
            ctx->keys.as<K>(), args, status, last_head, sp.ticket, sp.ticket_base, sp.tag, &ds->err));
    else
        OCHRE_LAUNCH(ctx, "tile_heads", s, launch_after(k_tile_heads<K, 16>, blocks, HEAD_BLOCK, 0, s,
            ctx->keys.as<K>(), args, status, last_head, sp.ticket, sp.ticket_base, sp.tag, &ds->err));
    OCHRE_CUDA_TRY(cudaGetLastError());
    int st = OCHRE_OK;
    uint32_t T, n_rows;
    if (plan) {
        OCHRE_LAUNCH(ctx, "plan_tiles", s, launch_after(k_plan_tiles, 1, 1, 0, s, ds, plan->tiles));
        OCHRE_CUDA_TRY(cudaGetLastError());
        T = plan->tiles;
        n_rows = plan->rows;
    } else {
        st = read_scalars(ctx, s);
        if (st != OCHRE_OK) return st;
        st = check_device_error(ctx);
        if (st != OCHRE_OK) return st;
        T = host_scalars(ctx)->n_tiles;
        n_rows = host_scalars(ctx)->n_rows;
    }
    *n_tiles_out = T;
    const uint32_t tpw = (uint32_t)ctx->tune_chain_tiles_per_warp;
    OCHRE_CUDA_TRY(ctx->tile_state.ensure((size_t)((T + tpw - 1) / tpw) * sizeof(TileBlockState)));
    OCHRE_CUDA_TRY(ctx->out_tile_xy.ensure((size_t)T * 4));
    OCHRE_CUDA_TRY(ctx->out_tile_alpha.ensure((size_t)T * 64));
    const bool want_cov = (ctx->flags & OCHRE_CTX_WANT_COV) != 0;
    if (want_cov) OCHRE_CUDA_TRY(ctx->out_tile_cov.ensure((size_t)T * 64 * 4));
    // Spans: compact in tile order.  Capacity: at most one span per tile.
    OCHRE_CUDA_TRY(ctx->out_span_xy.ensure((size_t)T * 4));
    OCHRE_CUDA_TRY(ctx->out_span_w.ensure((size_t)T * 2));
    OCHRE_CUDA_TRY(ctx->out_span_tile.ensure((size_t)T * 4));
    OCHRE_LAUNCH(ctx, "span_scan", s,
                 OCHRE_CUDA_TRY(launch_scan<uint32_t>(
                     ctx, T, SpanIn{tiles.xy, tiles.rf, T, t_dev},
                     SpanOut{tiles.xy, tiles.rf, T, R, t_dev, ctx->out_span_xy.as<uint32_t>(),
                             ctx->out_span_w.as<uint16_t>(), ctx->out_span_tile.as<uint32_t>(),
                             ctx->out_raster_span_off.as<uint32_t>()},
                     OpSumU32{}, 0u, &ds->n_spans, s, t_dev)));
    switch (tpw) {
    case 4: OCHRE_LAUNCH(ctx, "tile_coverage", s, launch_tile_cov<4>(ctx, tiles, T, n_rows, want_cov, s)); break;
    case 8: OCHRE_LAUNCH(ctx, "tile_coverage", s, launch_tile_cov<8>(ctx, tiles, T, n_rows, want_cov, s)); break;
    case 16: OCHRE_LAUNCH(ctx, "tile_coverage", s, launch_tile_cov<16>(ctx, tiles, T, n_rows, want_cov, s)); break;
    default: return OCHRE_E_INVALID;
    }
    OCHRE_CUDA_TRY(cudaGetLastError());
    if (plan) {
        *n_spans_out = 0;   // on the device; read after the replay
        return OCHRE_OK;
    }
    st = read_scalars(ctx, s);
    if (st != OCHRE_OK) return st;
    *n_spans_out = host_scalars(ctx)->n_spans;
    ctx->stats.n_bins = E - host_scalars(ctx)->n_cross;
    return check_device_error(ctx);
}

int stage_tiles(ochre_gpu_ctx* ctx, const ochre_batch* in, uint64_t E, cudaStream_t s, uint32_t* n_tiles,
                uint32_t* n_spans) {
    *n_tiles = 0;
    *n_spans = 0;
    if (E == 0) return OCHRE_OK;
    return ctx->keys64 ? tiles_impl<uint64_t>(ctx, in, E, s, n_tiles, n_spans)
                       : tiles_impl<uint32_t>(ctx, in, E, s, n_tiles, n_spans);
}

}  // namespace ochre
