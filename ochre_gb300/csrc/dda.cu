// Stage 2: line segments -> sort entries (pixel DDA binning).
//
// Reference: Rasterizer::line_to (rasterizer.rs:72-140) and the run-length
// binning of finish (rasterizer.rs:185-208).
//
// The count takes a line's row and column recurrences one after the other,
// without its cells.  The emission walks the cells with the reference's exact
// serial recurrence: one thread a line, or a group of lanes a long line, all
// of which run both recurrences alike.  Invariant used to make lines independent: at the start of
// every line_to, tile_y_prev == div_euclid(floor(last.y) as i16, 8) — move_to
// sets it that way (rasterizer.rs:68) and every walk ends by snapping to
// floor(point) and updating tile_y_prev for that cell (rasterizer.rs:118-131).
//
// The emission stores the increment (area, height) of every cell once, line
// by line (the count gives each line its offset), and produces two
// kinds of sort entries:
//   * a *bin* per run of consecutive increment cells in one tile
//     (value = entry index; the BinRec at that index holds the run's first
//     increment, first cell and steps, so the tile kernel finds every cell's
//     increment without walking again);
//   * a *crossing* per tile-row change (rasterizer.rs:123-131)
//     (value = CROSS_TAG | raster << 8 | sign byte).
// Keys order entries by (raster, tile_y, tile_x, kind) inside a compact key
// space: key_base[raster] + ((ty - by0) * w + (tx - bx0)) * 2 + kind, with
// the raster's tile bounding box (bx0, by0)..(bx1, by1) measured in the count
// pass; kind 0 (crossing) sorts before kind 1 (bin) of the same tile.
#include <algorithm>

#include "common.cuh"
#include "internal.h"
#include "scan.cuh"

namespace ochre {

struct BBoxAcc {
    int x0, y0, x1, y1;
};

__device__ __forceinline__ void bbox_add(BBoxAcc& b, int x, int y) {
    const int tx = div8(x), ty = div8(y);
    b.x0 = min(b.x0, tx);
    b.y0 = min(b.y0, ty);
    b.x1 = max(b.x1, tx);
    b.y1 = max(b.y1, ty);
}

// What a line's walk leaves: sort entries (bins and crossings), crossings
// alone, increment cells, the sum of its crossing signs, the tile box of its visited cells.
struct LineCount {
    uint32_t ent, cross, cells;
    int wsum;
    BBoxAcc box;
};

// The same by walking (a line that reaches WALK_CAP).
__device__ __noinline__ LineCount count_by_walking(V2 a, V2 p, uint32_t* err) {
    uint32_t ent = 0, cross = 0, cells = 0;
    int ws = 0, ptx = 0x7fffffff, pty = 0x7fffffff;
    BBoxAcc box{0x7fffffff, 0x7fffffff, (int)0x80000000, (int)0x80000000};
    const bool ok = walk_line(
        a, p,
        [&](const Walk&, const WalkState& s) {
            const int tx = div8(s.x), ty = div8(s.y);
            if (tx != ptx || ty != pty) { ent++; ptx = tx; pty = ty; }
            cells++;
        },
        [&](int, int, int sign) {
            ent++;
            cross++;
            ws += sign;
        },
        [&](int x, int y) { bbox_add(box, x, y); });
    if (!ok) atomicOr(err, ERR_LIMIT);
    return LineCount{ent, cross, cells, ws, box};
}

// Counts of a line without walking it.  The walk takes the row and column
// steps in order of their parameters and ends with the first at 1, so it
// takes every step below 1 of either axis whatever their order, then one
// more: the numbers of row and column steps below 1 (two independent
// recurrences, each two operations a step) give the last cell, and with it
//   * cells: every step below 1 leads to a cell, and there is the first one;
//   * bins: each step moves along one axis, so a new bin opens exactly where
//     a step leaves a tile column or a tile row;
//   * crossings: the tile rows left that way, and the snapped end cell's.
// Cells wrap at the i16 limits, which are tile boundaries too: a step across
// one leaves a tile like any other, in the walk's direction (the sign byte of
// -8191 is +1, of 8191 -1).  Bound by instruction issue: eight instructions
// per step of the longer axis, where walking took about 25 per cell.  20,000
// uneven paths (60 M lines, 689 M cells): 2.55 ms (walked, ordered by length,
// the long lines beside) -> 1.08 ms, the lines in their own order.
__device__ __forceinline__ LineCount count_line(V2 a, V2 p, uint32_t* err) {
    LineCount n{0u, 0u, 0u, 0, {0x7fffffff, 0x7fffffff, (int)0x80000000, (int)0x80000000}};
    if (veq(a, p)) return n;
    Walk w;
    WalkState s;
    walk_setup(a, p, w, s);
    uint32_t rows = 0, cols = 0;
    float rt = s.row_t1, ct = s.col_t1;
    while (rt < 1.0f || ct < 1.0f) {
#pragma unroll
        for (int k = 0; k < 4; k++) {   // (past 1 nothing more is counted)
            if (rt < 1.0f) rows++;
            if (ct < 1.0f) cols++;
            rt = rmin(__fadd_rn(rt, w.y_step), 1.0f);
            ct = rmin(__fadd_rn(ct, w.x_step), 1.0f);
        }
        if (rows + cols >= WALK_CAP) {
            return count_by_walking(a, p, err);
        }
    }
    // the last cell, not wrapped
    const int lx = s.x + w.x_dir * (int)cols, ly = s.y + w.y_dir * (int)rows;
    const int left_x = abs(div8(lx) - div8(s.x)), left_y = abs(div8(ly) - div8(s.y));
    const int end_ty = div8(w.end_y), last_ty = div8(wrap16(ly));
    n.cells = rows + cols + 1u;
    n.cross = (uint32_t)left_y + (end_ty != last_ty ? 1u : 0u);
    n.ent = 1u + (uint32_t)left_x + (uint32_t)left_y + n.cross;
    n.wsum = w.y_dir * left_y + (int)(int8_t)(int16_t)(end_ty - last_ty);
    bbox_add(n.box, s.x, s.y);
    bbox_add(n.box, wrap16(lx), wrap16(ly));
    bbox_add(n.box, w.end_x, w.end_y);
    if (lx != wrap16(lx)) {   // past an i16 limit: every column of the range's ends
        n.box.x0 = min(n.box.x0, -4096);
        n.box.x1 = max(n.box.x1, 4095);
    }
    if (ly != wrap16(ly)) {
        n.box.y0 = min(n.box.y0, -4096);
        n.box.y1 = max(n.box.y1, 4095);
    }
    return n;
}

// Block-local work order by walk length: the items of a block are grouped by
// log2 of their cell count (unstable within a group), so each warp walks
// lines of about the same length and a warp of short lines does not run as
// long as the longest of a random 32.  Not finer: neighbours in a group are
// neighbours in memory, and what their lanes write lies together (groups of
// one cell count, eight an octave from 32 on: 7.45 ms instead of 7.20 for the 60 M
// lines of 20,000 uneven paths).  Returns this thread's place in that order; items without a
// walk (cells 0) come last, from *n_walks on.  Every thread of the block calls
// it.
constexpr int LENGTH_GROUPS = 17;
__device__ __forceinline__ uint32_t order_by_length(uint32_t cells, uint32_t* s_cnt, uint32_t* n_walks) {
    const uint32_t g = cells == 0u ? (uint32_t)LENGTH_GROUPS - 1u : 31u - (uint32_t)__clz(cells);
    if (threadIdx.x < LENGTH_GROUPS) s_cnt[threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t k = atomicAdd(&s_cnt[g], 1u);
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        const uint32_t c = lane < LENGTH_GROUPS ? s_cnt[lane] : 0u;
        uint32_t inc = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += o;
        }
        if (lane < LENGTH_GROUPS) s_cnt[lane] = inc - c;
    }
    __syncthreads();
    *n_walks = s_cnt[LENGTH_GROUPS - 1];
    return s_cnt[g] + k;
}

// The next window of a warp (lane 0 takes the ticket).
__device__ __forceinline__ uint64_t next_window(uint32_t* ticket) {
    uint32_t w = 0;
    if ((threadIdx.x & 31u) == 0u) w = atomicAdd(ticket, 1u);
    return (uint64_t)__shfl_sync(0xffffffffu, w, 0);
}

// A raster's global tile box grows by atomics only where it grows.
__device__ __forceinline__ void box_grow(int4* d, int x0, int y0, int x1, int y1) {
    const int4 cur = ld_words(d);
    if (x0 < cur.x) atomicMin(&d->x, x0);
    if (y0 < cur.y) atomicMin(&d->y, y0);
    if (x1 > cur.z) atomicMax(&d->z, x1);
    if (y1 > cur.w) atomicMax(&d->w, y1);
}

// ---------------------------------------------------------------------
// Long lines: a group of G lanes per line.
//
// Walk lengths run from one cell to thousands (a path's long edges).  One
// thread per line, as the count and emit kernels walk most lines, would give
// a long line's warp one busy lane for thousands of steps, every cell's work
// (two points on the line, area, tile, entry, stores) in one dependent chain.
// The flatten stage queues every line of more than `long_cells` (estimated)
// cells, and the walkers below take G cells of a line per round: only the
// reference's two recurrences are serial (row_t1 and col_t1, one compare, one
// add and one min per step, run alike by every lane of the group), each lane
// keeps the parameter of its own step, and the work of the G cells is then
// done side by side.  Where a cell lies follows from the row steps before it
// (a bit mask of the round).
//
// Against one thread per line with idle lanes refilled: a document of 415
// paths (65,417 lines) 285 -> 42 us, one path of 2,093 lines 54 -> 15 us.
// ---------------------------------------------------------------------
template <int G>
struct GroupLine {
    // the line, the same in every lane of the group
    V2 a, p;
    int x_dir, y_dir, end_x, end_y;
    float x_step, y_step;
    // the walk before the round's first cell
    float row, col;      // row_t1, col_t1
    float t;             // where that cell begins
    int x, y;            // that cell
    bool seen_row, seen_col;   // a row / column step was taken
    uint32_t it;         // cells walked
    bool live;

    __device__ __forceinline__ void begin(V2 from, V2 to) {
        Walk w;
        WalkState s;
        walk_setup(from, to, w, s);
        a = from;
        p = to;
        x_dir = w.x_dir;
        y_dir = w.y_dir;
        end_x = w.end_x;
        end_y = w.end_y;
        x_step = w.x_step;
        y_step = w.y_step;
        row = s.row_t1;
        col = s.col_t1;
        t = 0.0f;
        x = s.x;
        y = s.y;
        seen_row = seen_col = false;
        it = 0;
        live = true;
    }
};
// What a round leaves in each lane (cell c = lane within the group), and its
// totals for the group.
struct GroupCell {
    bool valid;          // the cell exists
    float t0, t1;        // where the line enters and leaves it
    int x, y;            // the cell
    int nx, ny;          // the cell visited next (the snapped end cell after the last one)
    uint32_t row_bits;   // bit k: the step out of cell k went to another row (group)
    uint32_t m;          // cells of the round (group)
    bool fin;            // the walk ends in this round (group)
    bool capped;         // ... because it reached WALK_CAP (group)
};

// The next G cells of every group's line (walk_line's steps, common.cuh; all
// lanes of the warp call it, dead groups get no valid cell).
template <int G>
__device__ __forceinline__ void group_round(GroupLine<G>& L, GroupCell& q) {
    const uint32_t lane = threadIdx.x & 31u, c = lane & (G - 1), gshift = lane & ~(uint32_t)(G - 1);
    constexpr uint32_t ALL = G == 32 ? 0xffffffffu : (1u << G) - 1u;
    float mine = 0.0f;
    uint32_t rows = 0;
#pragma unroll
    for (int k = 0; k < G; k++) {
        const bool r = L.row < L.col;   // ties step x
        const float t = r ? L.row : L.col;
        if (c == (uint32_t)k) mine = t;
        if (r) rows |= 1u << k;
        const float rn = rmin(__fadd_rn(L.row, L.y_step), 1.0f), cn = rmin(__fadd_rn(L.col, L.x_step), 1.0f);
        L.row = r ? rn : L.row;
        L.col = r ? L.col : cn;
    }
    // the walk ends with the first step at t == 1 (steps past it are not used)
    const uint32_t ends = (__ballot_sync(0xffffffffu, mine == 1.0f) >> gshift) & ALL;
    q.m = L.live ? (ends ? (uint32_t)__ffs(ends) : (uint32_t)G) : 0u;
    q.capped = !ends && L.it + q.m >= WALK_CAP;
    q.fin = ends != 0u || q.capped;
    q.valid = c < q.m;
    q.row_bits = rows;
    const uint32_t lt = (1u << c) - 1u;
    const int steps_y = __popc(rows & lt), steps_x = (int)c - steps_y;
    q.x = wrap16(L.x + L.x_dir * steps_x);
    q.y = wrap16(L.y + L.y_dir * steps_y);
    q.t1 = mine;
    const float before = __shfl_up_sync(0xffffffffu, mine, 1, G);
    // max(row_t0, col_t0): the last step's parameter, and 0 for an axis not
    // stepped along yet
    q.t0 = c == 0 ? L.t : before;
    if (!((L.seen_row || (rows & lt)) && (L.seen_col || (~rows & lt)))) q.t0 = rmax(q.t0, 0.0f);
    const bool r = (rows >> c) & 1u;
    q.nx = r ? q.x : wrap16(q.x + L.x_dir);
    q.ny = r ? wrap16(q.y + L.y_dir) : q.y;
    if (mine == 1.0f) {
        q.nx = L.end_x;
        q.ny = L.end_y;
    }
}
// The line after the round.
template <int G>
__device__ __forceinline__ void group_advance(GroupLine<G>& L, const GroupCell& q) {
    const int last = (int)q.m - 1;
    L.t = __shfl_sync(0xffffffffu, q.t1, max(last, 0), G);
    L.x = __shfl_sync(0xffffffffu, q.nx, max(last, 0), G);
    L.y = __shfl_sync(0xffffffffu, q.ny, max(last, 0), G);
    if (q.m) {
        L.seen_row = L.seen_row || q.row_bits != 0u;
        L.seen_col = L.seen_col || q.row_bits != (G == 32 ? 0xffffffffu : (1u << G) - 1u);
    }
    L.it += q.m;
    if (q.fin) L.live = false;
}
// Lanes per line: a line alone in its warp takes the fewest cycles a cell
// (its recurrences plus 1/32 of the cells' work), which is what counts while
// warps are idle; where there are more lines than warps, four share one and
// the warp does less work per cell.
__device__ __forceinline__ bool long_lines_share(uint32_t n_queue) {
    return n_queue > gridDim.x * (blockDim.x >> 5);
}

constexpr int LONG_THREADS = 128;
constexpr uint32_t LONG_BLOCKS_PER_SM = 2;
// The walkers are for few long lines among many.  Where an eighth of all lines
// and more are long, and they are many enough to occupy the GPU by themselves,
// the per-line kernel takes them too: its warps then walk long lines side by
// side, and a lane does less for a cell than a group does.  The call, walkers
// against none: 20,000 rasters of 100 lines (1.36 M of the 2.0 M long, 168 cells on
// average) 8.9 -> 5.8 ms, its replay 15.4 -> 6.8; 50,000 lines of 4,000 cells 7.95 ->
// 6.97 and 12.7 -> 7.0 ms; 40,000 of 160 cells 0.46 -> 0.40 and 0.70 -> 0.43 ms.
bool long_lines_apart(uint64_t n_long, uint64_t n_lines) {
    return n_long * 8 < n_lines || n_long < (1u << 15);
}

// Entry counts per line (written in place of the offsets, then scanned)
// and the raster tile boxes.  Counting is a separate kernel, not folded into
// the offset scan: a count's length varies from no step to thousands, and a
// single-pass scan would hold every later block behind the slowest one.
// Persistent warps take windows of `groups` times 32 consecutive lines by
// ticket (more than one group only where there are lines enough to fill the
// GPU).  Boxes (and the rasters' crossing-sign sums) are reduced before any
// global atomic: lanes of one raster by warp reductions, then the window's
// first BOX_SLOTS rasters (lines of a raster are contiguous) in the warp's
// shared slots; each global box is then updated only where it grows.
constexpr int COUNT_GROUPS_MAX = 8;
constexpr int WALK_BLOCK = 128;
constexpr int BOX_SLOTS = 8;
__global__ void __launch_bounds__(WALK_BLOCK) k_line_count(const float4* lines,
                                                           const uint32_t* line_raster, uint32_t n_cap,
                                                           const uint32_t* n_dev, uint32_t groups, int4* bbox,
                                                           int* raster_wsum, uint32_t* __restrict__ counts,
                                                           uint32_t* __restrict__ inc_counts,
                                                           unsigned long long* inc_total, uint32_t* n_cross,
                                                           uint32_t* ticket, uint32_t* err) {
    dependent_start();
    constexpr int WARPS = WALK_BLOCK / 32;
    __shared__ int4 s_box[WARPS][BOX_SLOTS];
    __shared__ int s_ws[WARPS][BOX_SLOTS];
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint64_t n_lines = dev_count(n_cap, n_dev);
    unsigned long long incs = 0;   // the warp's increments (lane 0)
    uint32_t crosses = 0;          // this lane's crossings
    for (;;) {
        const uint64_t i0 = next_window(ticket) * (32u * groups);
        if (i0 >= n_lines) break;
        if (lane < BOX_SLOTS) {
            s_box[wid][lane] = make_int4(0x7fffffff, 0x7fffffff, (int)0x80000000, (int)0x80000000);
            s_ws[wid][lane] = 0;
        }
        const uint32_t r0 = line_raster[i0];
        __syncwarp();
        for (uint32_t j = 0; j < groups; j++) {
            const uint64_t i = i0 + j * 32u + lane;
            LineCount n{0u, 0u, 0u, 0, {0x7fffffff, 0x7fffffff, (int)0x80000000, (int)0x80000000}};
            uint32_t r = r0;
            if (i < n_lines) {
                const float4 l = lines[i];
                r = line_raster[i];
                n = count_line(v2(l.x, l.y), v2(l.z, l.w), err);
                counts[i] = n.ent;
                inc_counts[i] = n.cells;
            }
            const unsigned grp = __match_any_sync(0xffffffffu, r);
            const int x0 = __reduce_min_sync(grp, n.box.x0), y0 = __reduce_min_sync(grp, n.box.y0);
            const int x1 = __reduce_max_sync(grp, n.box.x1), y1 = __reduce_max_sync(grp, n.box.y1);
            const int wsg = __reduce_add_sync(grp, n.wsum);
            if ((int)lane == __ffs(grp) - 1) {
                if (r - r0 < (uint32_t)BOX_SLOTS) {
                    if (x0 <= x1) {
                        int4* d = &s_box[wid][r - r0];
                        atomicMin(&d->x, x0);
                        atomicMin(&d->y, y0);
                        atomicMax(&d->z, x1);
                        atomicMax(&d->w, y1);
                    }
                    if (wsg) atomicAdd(&s_ws[wid][r - r0], wsg);
                } else {
                    if (x0 <= x1) box_grow(bbox + r, x0, y0, x1, y1);
                    if (wsg) atomicAdd(raster_wsum + r, wsg);
                }
            }
            // (at most 32 capped walks: 32 bits hold it)
            incs += __reduce_add_sync(0xffffffffu, n.cells);
            crosses += n.cross;
        }
        __syncwarp();
        if (lane < BOX_SLOTS) {
            const int4 b = s_box[wid][lane];
            if (b.x <= b.z) box_grow(bbox + r0 + lane, b.x, b.y, b.z, b.w);
            if (s_ws[wid][lane]) atomicAdd(raster_wsum + r0 + lane, s_ws[wid][lane]);
        }
        __syncwarp();
    }
    crosses = __reduce_add_sync(0xffffffffu, crosses);
    if (lane == 0 && incs) atomicAdd(inc_total, incs);
    if (lane == 0 && crosses) atomicAdd(n_cross, crosses);
}
// Entry and increment offsets of every line, one scan of the pair (in place:
// every count is read by the thread that writes its offset).  Bound by memory
// requests: with a thread's 8 items in 16-byte accesses (load_all, store_all) 60
// M lines take 326 us, item by item 686 (14 M lines 84 and 176).
struct LinePair {
    uint32_t ent, inc;
};
struct OpLinePair {
    __device__ __forceinline__ LinePair operator()(LinePair a, LinePair b) const {
        return LinePair{a.ent + b.ent, a.inc + b.inc};
    }
};
struct LinePairIn {
    const uint32_t* ent;
    const uint32_t* inc;
    __device__ __forceinline__ LinePair operator()(uint64_t i) const { return LinePair{ent[i], inc[i]}; }
    using takes_all = void;
    template <int N>
    __device__ __forceinline__ void load_all(uint64_t i, LinePair (&v)[N]) const {
        uint32_t e[N], q[N];
        load_words(ent + i, e);
        load_words(inc + i, q);
#pragma unroll
        for (int k = 0; k < N; k++) v[k] = LinePair{e[k], q[k]};
    }
};
struct LinePairOut {
    uint32_t* ent;
    uint32_t* inc;
    __device__ __forceinline__ void operator()(uint64_t i, LinePair ex, LinePair) const {
        ent[i] = ex.ent;
        inc[i] = ex.inc;
    }
    using takes_all = void;
    template <int N>
    __device__ __forceinline__ void store_all(uint64_t i, LinePair run, const LinePair (&v)[N]) const {
        uint32_t e[N], q[N];
#pragma unroll
        for (int k = 0; k < N; k++) {
            e[k] = run.ent;
            q[k] = run.inc;
            run = OpLinePair{}(run, v[k]);
        }
        store_words(ent + i, e);
        store_words(inc + i, q);
    }
};

__global__ void k_bbox_init(int4* bbox, int* wsum, uint32_t n) {
    dependent_start();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        bbox[i] = make_int4(0x7fffffff, 0x7fffffff, (int)0x80000000, (int)0x80000000);
        wsum[i] = 0;
    }
}

// Per-raster key space: w * h * 2 keys; rasters without increments get a
// 1x1 box at tile (0,0) and one synthetic bin (finish pushes a bin at (0,0)
// even when there are no increments, rasterizer.rs:194-208).
struct RasterScan {
    uint64_t ks;
    uint32_t ne;
    int32_t w;   // crossing signs of the rasters so far
    uint32_t by_size[3];   // rasters sorted by the middle and the large block of stage_sort_local, and by neither
    uint32_t begin, n;     // (of one raster alone) its entries
    uint32_t pad;
};
struct OpRaster {
    __device__ __forceinline__ RasterScan operator()(RasterScan a, RasterScan b) const {
        return RasterScan{a.ks + b.ks, a.ne + b.ne, a.w + b.w,
                          {a.by_size[0] + b.by_size[0], a.by_size[1] + b.by_size[1], a.by_size[2] + b.by_size[2]}, 0u, 0u, 0u};
    }
};
// First entry of raster r's lines (r = n_rasters: their end).
struct RasterEntries {
    const uint32_t* cmd_line_off;
    uint64_t n_cmds;
    const uint32_t* fill_off;
    const uint32_t* raster_off;   // or null: one fill per raster
    const uint32_t* line_ent_off;
    uint32_t n_lines;
    const uint32_t* line_ent_total;
    __device__ __forceinline__ uint32_t operator()(uint32_t r) const {
        const uint32_t c = fill_off[raster_off ? raster_off[r] : r];
        const uint32_t l = c < n_cmds ? cmd_line_off[c] : n_lines;
        return l < n_lines ? line_ent_off[l] : *line_ent_total;
    }
};
struct RasterIn {
    const int4* bbox;
    const int* wsum;
    RasterEntries first;
    bool sizes;   // the rasters are listed by size
    __device__ __forceinline__ RasterScan operator()(uint64_t r) const {
        const int4 b = bbox[r];
        const uint32_t e = sizes ? first((uint32_t)r) : 0u;
        if (b.x > b.z) return RasterScan{2ull, 1u, wsum[r], {0u, 0u, 0u}, e, 0u, 0u};
        const uint64_t w = (uint64_t)(b.z - b.x + 1), h = (uint64_t)(b.w - b.y + 1);
        RasterScan v{w * h * 2ull, 0u, wsum[r], {0u, 0u, 0u}, e, 0u, 0u};
        if (sizes) {
            v.n = first((uint32_t)r + 1u) - e;
            if (v.n > LOCAL_SORT_LARGE || v.ks > (1ull << LOCAL_SORT_KEY_BITS)) v.by_size[2] = 1u;
            else if (v.n > LOCAL_SORT_MIDDLE) v.by_size[1] = 1u;
            else if (v.n > LOCAL_SORT_SMALL) v.by_size[0] = 1u;
        }
        return v;
    }
};
struct RasterOut {
    int4* bbox;
    uint64_t* key_base;
    uint32_t* empty;   // 0: has increments; else 1 + rank among empty rasters
    int* wbase;        // crossing signs of all earlier rasters
    RasterRun* run;    // (or null) small from the front, middle from n_rasters - 1 down, large from n_rasters on
    uint32_t n_rasters;
    __device__ __forceinline__ void operator()(uint64_t r, RasterScan ex, RasterScan v) const {
        key_base[r] = ex.ks;
        wbase[r] = ex.w;
        empty[r] = v.ne ? ex.ne + 1u : 0u;
        if (run != nullptr && !v.by_size[2]) {
            const uint32_t at = v.by_size[0]   ? n_rasters - 1u - ex.by_size[0]
                                : v.by_size[1] ? n_rasters + ex.by_size[1]
                                               : (uint32_t)r - ex.by_size[0] - ex.by_size[1] - ex.by_size[2];
            run[at] = RasterRun{(uint32_t)r, v.begin, v.n, v.begin + ex.ne};
        }
        if (v.ne) bbox[r] = make_int4(0, 0, 0, 0);
    }
};

// Entries and increments of queued lines (see k_line_emit, whose entries in
// the same order these are).
template <int G, class K>
__device__ __forceinline__ void emit_long(const float4* lines, const uint32_t* line_raster,
                                          const uint32_t* ent_off, const uint32_t* inc_off,
                                          const int4* bbox, const uint64_t* key_base,
                                          K* __restrict__ keys, uint32_t* __restrict__ vals, BinRec* __restrict__ bins,
                                          float2* __restrict__ incs, const uint32_t* queue,
                                          uint32_t n_queue, uint32_t* ticket) {
    const uint32_t lane = threadIdx.x & 31u, c = lane & (G - 1), gshift = lane & ~(uint32_t)(G - 1);
    constexpr uint32_t ALL = G == 32 ? 0xffffffffu : (1u << G) - 1u;
    const uint32_t lt = (1u << c) - 1u;
    GroupLine<G> L;
    L.begin(v2(0.0f, 0.0f), v2(1.0f, 1.0f));
    L.live = false;
    bool more = true;
    // the group's line: raster, key of tile (0, 0) and tile columns, next entry, next increment
    uint32_t r = 0, e = 0, inc = 0;
    K key0 = 0, cols = 0;
    // the bin left open by the round before: its entry, first increment, first
    // cell, cells and steps so far (n 0: none; else the next cell is in it)
    uint32_t o_entry = 0, o_inc = 0, o_xy = 0, o_n = 0, o_steps = 0;
    for (;;) {
        if (more && !L.live) {
            more = false;   // until a line is taken
            const uint32_t gmask = ALL << gshift;
            uint32_t k = 0;
            // (lanes of a group agree on more and live)
            if (c == 0) k = atomicAdd(ticket, 1u);
            k = __shfl_sync(gmask, k, 0, G);
            if (k < n_queue) {
                more = true;
                const uint32_t i = queue[k];
                const float4 l = lines[i];
                r = line_raster[i];
                e = ent_off[i];
                inc = inc_off[i];
                const int4 bb = bbox[r];
                cols = (K)(bb.z - bb.x + 1);
                key0 = (K)key_base[r] - (((K)(int64_t)bb.y * cols + (K)(int64_t)bb.x) << 1);
                L.begin(v2(l.x, l.y), v2(l.z, l.w));
                o_n = 0;
            }
        }
        __syncwarp();
        if (__ballot_sync(0xffffffffu, L.live) == 0u) {
            if (__ballot_sync(0xffffffffu, more) == 0u) break;
            continue;
        }
        GroupCell q;
        group_round<G>(L, q);
        if (q.valid) {
            // the cell's increment (rasterizer.rs:98-106)
            const V2 p0 = vlerp(q.t0, L.a, L.p), p1 = vlerp(q.t1, L.a, L.p);
            const float height = __fsub_rn(p1.y, p0.y);
            const float right = (float)wrap16(q.x + 1);
            const float area =
                __fmul_rn(__fmul_rn(0.5f, height), __fadd_rn(__fsub_rn(right, p0.x), __fsub_rn(right, p1.x)));
            incs[inc + c] = make_float2(area, height);
        }
        const int tx = div8(q.x), ty = div8(q.y), nty = div8(q.ny);
        const int tile = (int)(((uint32_t)ty << 16) | ((uint32_t)tx & 0xffffu));
        const int before = __shfl_up_sync(0xffffffffu, tile, 1, G);
        const bool new_bin = q.valid && (c == 0 ? o_n == 0 : tile != before);
        const bool cross = q.valid && nty != ty;
        const uint32_t B = (__ballot_sync(0xffffffffu, new_bin) >> gshift) & ALL;
        const uint32_t X = (__ballot_sync(0xffffffffu, cross) >> gshift) & ALL;
        // a cell's bin opens before its crossing
        const uint32_t mine = e + (uint32_t)__popc(B & lt) + (uint32_t)__popc(X & lt);
        auto key_of = [&](int kx, int ky, K kind) {
            return key0 + (((K)(int64_t)ky * cols + (K)(int64_t)kx) << 1) + kind;
        };
        if (cross) {
            const uint32_t x = mine + (new_bin ? 1u : 0u);
            keys[x] = key_of(div8(q.nx), min(ty, nty), (K)0);
            vals[x] = CROSS_TAG | (r << 8) | ((uint32_t)(nty - ty) & 0xffu);
        }
        // runs: a lane that opens a bin owns it, and lane 0 the one left open
        // by the round before; the round's last run stays open if the walk
        // goes on in its tile
        // (the shuffle is every lane's, ended groups' too)
        const int next_same = __shfl_sync(0xffffffffu, div8(q.nx) == tx && nty == ty ? 1 : 0, (int)max(q.m, 1u) - 1, G);
        const bool goes_on = !q.fin && next_same != 0;
        const uint32_t cells = q.m == 32u ? 0xffffffffu : (1u << q.m) - 1u;
        const uint32_t xsteps = ~q.row_bits & cells;
        const bool carried = c == 0 && o_n != 0;
        const uint32_t after = (B >> c) >> 1;   // bins opened by later cells
        const uint32_t run = after ? (uint32_t)__ffs(after) : q.m - c;
        const bool owner = q.valid && (new_bin || carried);
        const bool stays = owner && !after && goes_on;
        const uint32_t have = carried ? o_n : 0u;
        const uint32_t n = have + run;
        const uint32_t in_run = run >= 32u ? 0xffffffffu : (1u << run) - 1u;
        // steps out of the run's cells; the last one leaves the bin unless it stays open
        const uint32_t steps = (carried ? o_steps : 0u) | (((xsteps >> c) & (stays ? in_run : in_run >> 1)) << have);
        const uint32_t xy = carried ? o_xy : ((uint32_t)(uint16_t)(int16_t)q.x | ((uint32_t)(uint16_t)(int16_t)q.y << 16));
        const uint32_t at = carried ? o_entry : mine, first = carried ? o_inc : inc + c;
        if (owner && !stays) {
            BinRec rec;
            rec.inc = first;
            rec.raster = r;
            rec.x = (int16_t)(xy & 0xffffu);
            rec.y = (int16_t)(xy >> 16);
            rec.steps = (uint16_t)steps;
            rec.n = (uint8_t)n;
            rec.dirs = (uint8_t)((L.x_dir < 0 ? 1u : 0u) | (L.y_dir < 0 ? 2u : 0u));
            *reinterpret_cast<uint4*>(bins + at) = *reinterpret_cast<const uint4*>(&rec);
            keys[at] = key_of(tx, ty, (K)1);   // (the owner's cell lies in the bin's tile)
            vals[at] = at;
        }
        const uint32_t open = (__ballot_sync(0xffffffffu, stays) >> gshift) & ALL;   // at most one
        const int src = open ? __ffs(open) - 1 : 0;
        o_entry = __shfl_sync(0xffffffffu, at, src, G);
        o_inc = __shfl_sync(0xffffffffu, first, src, G);
        o_xy = __shfl_sync(0xffffffffu, xy, src, G);
        o_steps = __shfl_sync(0xffffffffu, steps, src, G);
        o_n = __shfl_sync(0xffffffffu, n, src, G);
        if (!open) o_n = 0;
        e += (uint32_t)__popc(B) + (uint32_t)__popc(X);
        inc += q.m;
        group_advance<G>(L, q);
        __syncwarp();
    }
}

// The queued long lines' entries and increments (see k_line_emit).
template <class K>
__global__ void __launch_bounds__(LONG_THREADS) k_line_emit_long(
    const float4* lines, const uint32_t* line_raster, const uint32_t* ent_off,
    const uint32_t* inc_off, uint64_t n_cap, const uint32_t* n_dev, const int4* bbox,
    const uint64_t* key_base, K* __restrict__ keys, uint32_t* __restrict__ vals,
    BinRec* __restrict__ bins, float2* __restrict__ incs, const uint32_t* queue, const uint32_t* n_queue,
    uint32_t* ticket) {
    dependent_start();
    // (a line count zeroed on the device, after an overflow of a graph's
    // plan, stops these walks too: their offsets were not written)
    if (dev_count(n_cap, n_dev) == 0) return;
    const uint32_t n = *n_queue;
    if (long_lines_share(n))
        emit_long<8, K>(lines, line_raster, ent_off, inc_off, bbox, key_base, keys, vals, bins, incs, queue, n, ticket);
    else
        emit_long<32, K>(lines, line_raster, ent_off, inc_off, bbox, key_base, keys, vals, bins, incs, queue, n, ticket);
}

// Four increments, one aligned 32-byte store (sm_100 and later).
__device__ __forceinline__ void store_increments(float2* o, float2 a, float2 b, float2 c, float2 d) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o), "f"(a.x), "f"(a.y), "f"(b.x),
                 "f"(b.y), "f"(c.x), "f"(c.y), "f"(d.x), "f"(d.y)
                 : "memory");
}

// Every thread walks one line, the lines of a block in order of length
// (order_by_length) so a warp's lanes walk lines of about the same length.
// Lines of more than long_cells cells are left to k_line_emit_long (default
// 96: on 20,000 strokes a call takes 4.93 / 4.84 / 4.79 / 4.79 / 4.84 ms at 48 /
// 64 / 96 / 128 / 192, a document of 415 paths 0.824 .. 0.828 ms up to 96 and
// 0.852 at 192; one path, shapes and the uneven mix do not care).
//
// Bound by its store requests and by issue (77 % of the slots, 13 of 32 lanes
// active): a lane writes its own line's increments, bins and entries, so nearly
// every store is a request of its own (840 M of 4 to 16 bytes for 139 M bins and
// 689 M increments), and more lanes in flight made it slower (20,000 uneven
// paths: 5.9 ms alone with 16 to 32 warps an SM, 7.4 ms with 40, 10.4 ms with 64).
// So increments leave four at a time, a whole 32-byte sector in one store, offsets and lines are read coalesced before the block orders them,
// keys are one multiply-add of the key's own width, a cell starts where the
// one before ended, and a bin, its crossing and the next bin's opening are one
// branch.  20,000 uneven paths (60 M lines; the long lines beside): 7.86 ms -> 6.37 ms; 1,000
// shapes 128 -> 110 us; 128 dense scenes (14 M lines of two cells) 388 -> 364 us.
constexpr int EMIT_BLOCK = 128;
constexpr int EMIT_CARVEOUT = 28;          // percent shared: room for the blocks that fit by registers
template <class K>
__global__ void __launch_bounds__(EMIT_BLOCK) k_line_emit(
    const float4* lines, const uint32_t* line_raster, const uint32_t* ent_off,
    const uint32_t* inc_off, uint64_t n_cap, const uint32_t* n_dev, const int4* bbox,
    const uint64_t* key_base, K* __restrict__ keys, uint32_t* __restrict__ vals,
    BinRec* __restrict__ bins, float2* __restrict__ incs, uint32_t long_cells) {
    dependent_start();
    __shared__ uint32_t s_cnt[LENGTH_GROUPS];
    __shared__ float4 s_line[EMIT_BLOCK];
    __shared__ uint4 s_off[EMIT_BLOCK];   // first entry, first increment, raster, twice the raster's tile columns
    __shared__ K s_key0[EMIT_BLOCK];      // key of tile (0, 0)
    const uint64_t n_lines = dev_count(n_cap, n_dev);
    const uint64_t i0 = blockIdx.x * (uint64_t)EMIT_BLOCK;
    if (i0 >= n_lines) return;
    {
        const uint64_t i = i0 + threadIdx.x;
        uint32_t cells = 0;
        float4 l = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        uint4 off = make_uint4(0u, 0u, 0u, 0u);
        K key0 = 0;
        if (i < n_lines) {
            l = lines[i];
            off = make_uint4(ent_off[i], inc_off[i], line_raster[i], 0u);
            cells = walk_cells(l);
            if ((l.x == l.z && l.y == l.w) || (long_cells && cells > long_cells)) cells = 0;
            if (cells) {
                const int4 bb = bbox[off.z];
                const K cols = (K)(bb.z - bb.x + 1);
                key0 = (K)key_base[off.z] - (((K)(int64_t)bb.y * cols + (K)(int64_t)bb.x) << 1);
                off.w = (uint32_t)cols << 1;
            }
        }
        uint32_t n_walks;
        const uint32_t at = order_by_length(cells, s_cnt, &n_walks);
        s_line[at] = l;
        s_off[at] = off;
        s_key0[at] = key0;
        __syncthreads();
        if (threadIdx.x >= n_walks) return;
    }
    const float4 l = s_line[threadIdx.x];
    const uint4 off = s_off[threadIdx.x];
    const K key0 = s_key0[threadIdx.x];
    const K cols2 = (K)off.w;
    const uint32_t r = off.z;
    Walk w;
    WalkState s;
    walk_setup(v2(l.x, l.y), v2(l.z, l.w), w, s);
    // A cell's start parameter is the larger of the two axes' last steps,
    // which is the step into the cell, so its start point is the end point of
    // the cell before.  Before both axes have stepped 0 takes part, which
    // matters to a step below 0 (cells at the i16 limits).
    const bool below = rmin(s.row_t1, s.col_t1) < 0.0f;
    bool row_moved = false, col_moved = false;
    V2 p0 = w.a;
    uint32_t e = off.x, q = off.y;   // next entry, next increment
    const uint32_t q_cap = q + WALK_CAP;
    // increments leave in fours, a whole 32-byte sector; three wait here
    float2 h0 = make_float2(0.0f, 0.0f), h1 = h0, h2 = h0;
    bool held = false;
    // the open bin: entry, tile, cells, steps and first cell
    uint32_t bin = e++, b_n = 0, b_steps = 0, b_inc = q;
    int btx = div8(s.x), bty = div8(s.y);
    uint32_t b_xy = (uint32_t)(uint16_t)s.x | ((uint32_t)(uint16_t)s.y << 16);
    const uint32_t dirs = (w.x_dir < 0 ? 1u << 24 : 0u) | (w.y_dir < 0 ? 2u << 24 : 0u);
    for (;;) {
        // the cell's increment (rasterizer.rs:98-106)
        const bool row = s.row_t1 < s.col_t1;
        const float t1 = row ? s.row_t1 : s.col_t1;
        const V2 p1 = vlerp(t1, w.a, w.p);
        const float height = __fsub_rn(p1.y, p0.y);
        const float right = (float)wrap16(s.x + 1);
        const float2 v = make_float2(
            __fmul_rn(__fmul_rn(0.5f, height), __fadd_rn(__fsub_rn(right, p0.x), __fsub_rn(right, p1.x))), height);
        if ((q & 3u) == 3u && held) {
            store_increments(incs + (q - 3u), h0, h1, h2, v);
            held = false;
        } else if (held || (q & 3u) == 0u) {
            if ((q & 3u) == 0u) h0 = v;
            if ((q & 3u) == 1u) h1 = v;
            if ((q & 3u) == 2u) h2 = v;
            held = true;
        } else {
            incs[q] = v;   // before the line's first whole sector
        }
        q++;
        b_n++;
        // the step out of it (rasterizer.rs:108-121)
        p0 = p1;
        if (below) {
            if (row) row_moved = true; else col_moved = true;
            if (t1 < 0.0f && !(row_moved && col_moved)) p0 = w.a;
        }
        if (row) {
            s.row_t1 = rmin(__fadd_rn(s.row_t1, w.y_step), 1.0f);
            s.y = wrap16(s.y + w.y_dir);
        } else {
            s.col_t1 = rmin(__fadd_rn(s.col_t1, w.x_step), 1.0f);
            s.x = wrap16(s.x + w.x_dir);
        }
        const bool snap = t1 == 1.0f;
        if (snap) {
            s.x = w.end_x;
            s.y = w.end_y;
        }
        const bool done = snap || q == q_cap;
        const int tx = div8(s.x), ty = div8(s.y);
        if (tx != btx || ty != bty || done) {
            *reinterpret_cast<uint4*>(bins + bin) = make_uint4(b_inc, r, b_xy, b_steps | (b_n << 16) | dirs);
            keys[bin] = key0 + (K)(int64_t)bty * cols2 + ((K)(int64_t)btx << 1) + (K)1;
            vals[bin] = bin;
            if (ty != bty) {
                keys[e] = key0 + (K)(int64_t)min(bty, ty) * cols2 + ((K)(int64_t)tx << 1);
                vals[e] = CROSS_TAG | (r << 8) | ((uint32_t)(ty - bty) & 0xffu);
                e++;
            }
            if (done) break;
            bin = e++;
            btx = tx;
            bty = ty;
            b_n = 0;
            b_steps = 0;
            b_inc = q;
            b_xy = (uint32_t)(uint16_t)s.x | ((uint32_t)(uint16_t)s.y << 16);
        } else if (!row) {
            b_steps |= 1u << (b_n - 1u);   // the step into the next cell moves in x
        }
    }
    if (held) {
        float2* o = incs + (q & ~3u);
        o[0] = h0;
        if ((q & 3u) >= 2u) o[1] = h1;
        if ((q & 3u) == 3u) o[2] = h2;
    }
}

template <class K>
__global__ void k_empty_emit(const uint32_t* empty, uint32_t n_rasters, uint32_t first_entry,
                             const uint32_t* first_dev, const uint32_t* n_ent_dev,
                             const uint64_t* key_base, K* __restrict__ keys,
                             uint32_t* __restrict__ vals, BinRec* __restrict__ bins) {
    dependent_start();
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rasters) return;
    const uint32_t rank = empty[r];
    if (!rank) return;
    // device-held counts (graph replays): entries after the lines' entries,
    // none when the entry count was over capacity (zeroed)
    if (first_dev != nullptr) first_entry = *first_dev;
    const uint32_t e = first_entry + rank - 1u;
    if (n_ent_dev != nullptr && e >= *n_ent_dev) return;
    BinRec rec;
    rec.inc = 0;
    rec.raster = r;
    rec.x = 0;
    rec.y = 0;
    rec.steps = 0;
    rec.n = 0;
    rec.dirs = 0;
    bins[e] = rec;
    keys[e] = (K)(key_base[r] + 1ull);
    vals[e] = e;
}

// The stream the long-line walkers run on: a side stream that waits for
// the run's stream s here (join_walks makes s wait for it in turn), so that
// the walkers, whose time is the longest line's serial walk, overlap the
// per-line kernel.  s itself when the context has no side stream.
static cudaError_t fork_walks(ochre_gpu_ctx* ctx, cudaStream_t s, cudaStream_t* side) {
    *side = s;
    if (ctx->no_side_stream) return cudaSuccess;
    if (!ctx->walk_stream) {
        if (cudaStreamCreateWithFlags(&ctx->walk_stream, cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&ctx->ev_walk_fork, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&ctx->ev_walk_join, cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            ctx->no_side_stream = true;
            return cudaSuccess;
        }
    }
    cudaError_t e = cudaEventRecord(ctx->ev_walk_fork, s);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->walk_stream, ctx->ev_walk_fork, 0);
    if (e == cudaSuccess) *side = ctx->walk_stream;
    return e;
}
static cudaError_t join_walks(ochre_gpu_ctx* ctx, cudaStream_t side, cudaStream_t s) {
    if (side == s) return cudaSuccess;
    cudaError_t e = cudaEventRecord(ctx->ev_walk_join, side);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s, ctx->ev_walk_join, 0);
    return e;
}

// Persistent grid of the count kernel and the 32-line groups of its windows:
// the blocks the GPU keeps resident, with larger windows (fewer updates of
// the rasters' boxes) only where every resident warp still gets one.
static void count_shape(ochre_gpu_ctx* ctx, uint64_t n_lines, unsigned* grid, uint32_t* groups) {
    int sms = 152, occ = 1;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_line_count, WALK_BLOCK, 0) != cudaSuccess || occ < 1) {
        cudaGetLastError();
        occ = 1;
    }
    const uint64_t warps = (uint64_t)sms * (uint64_t)occ * (WALK_BLOCK / 32);
    *groups = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(COUNT_GROUPS_MAX, n_lines / (32 * warps)));
    const uint64_t windows = (n_lines + 32ull * *groups - 1) / (32ull * *groups);
    const uint64_t blocks = (windows + WALK_BLOCK / 32 - 1) / (WALK_BLOCK / 32);
    *grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(blocks, warps / (WALK_BLOCK / 32)));
}

int stage_bin(ochre_gpu_ctx* ctx, const ochre_batch* in, uint32_t n_lines, cudaStream_t s, uint64_t* n_entries,
              uint32_t* key_bits) {
    DevScalars* ds = dev_scalars(ctx);
    const uint32_t R = in->n_rasters;
    *n_entries = 0;
    *key_bits = 0;
    if (R == 0) return OCHRE_OK;
    if (R > MAX_RASTERS) return OCHRE_E_CAPACITY;
    OCHRE_CUDA_TRY(ctx->raster_bbox.ensure((size_t)R * sizeof(int4)));
    OCHRE_CUDA_TRY(ctx->raster_keybase.ensure((size_t)R * 8));
    OCHRE_CUDA_TRY(ctx->raster_empty.ensure((size_t)R * 4));
    OCHRE_CUDA_TRY(ctx->raster_wsum.ensure((size_t)R * 4));
    OCHRE_CUDA_TRY(ctx->raster_wbase.ensure((size_t)R * 4));
    OCHRE_LAUNCH(ctx, "bbox_init", s, launch_after(k_bbox_init, (R + 255) / 256, 256, 0, s, ctx->raster_bbox.as<int4>(),
                                                                                 ctx->raster_wsum.as<int>(), R));
    OCHRE_CUDA_TRY(cudaGetLastError());
    // the line pair's totals, the 64-bit increment count, the long lines' ticket
    // and the crossing count
    static_assert(offsetof(DevScalars, inc_total) == offsetof(DevScalars, line_ent_total) + 8 &&
                      offsetof(DevScalars, walk_ticket) == offsetof(DevScalars, line_ent_total) + 16,
                  "layout");
    OCHRE_CUDA_TRY(cudaMemsetAsync(&ds->line_ent_total, 0, 24, s));
    OCHRE_CUDA_TRY(cudaMemsetAsync(&ds->line_ticket, 0, 4, s));
    const uint32_t long_cells = (uint32_t)ctx->tune_chain_long_cells;
    const uint32_t* queue = long_cells ? ctx->long_lines.as<uint32_t>() : nullptr;
    // graph replays: n_lines is the capacity, the count is on the device
    const GraphPlan* plan = ctx->plan;
    if (n_lines) OCHRE_CUDA_TRY(ctx->line_ent_off.ensure((size_t)n_lines * 4));
    const bool sizes = n_lines != 0 && sort_local_wanted(ctx);
    if (sizes) OCHRE_CUDA_TRY(ctx->raster_run.ensure((size_t)R * 2 * sizeof(RasterRun)));
    static_assert(sizeof(RasterScan) == 40 && offsetof(DevScalars, n_sort) == offsetof(DevScalars, keyspace) + 16,
                  "layout");
    const RasterEntries first{ctx->cmd_line_off.as<uint32_t>(), in->n_cmds, in->fill_cmd_off, in->raster_fill_off,
                              ctx->line_ent_off.as<uint32_t>(), n_lines, &ds->line_ent_total};
    const uint32_t* lines_dev = plan ? &ds->n_lines : nullptr;
    if (n_lines) {
        OCHRE_CUDA_TRY(ctx->line_inc_off.ensure((size_t)n_lines * 4));
        unsigned count_grid = 1;
        uint32_t groups = 1;
        count_shape(ctx, n_lines, &count_grid, &groups);
        OCHRE_LAUNCH(ctx, "dda_count", s, launch_after(k_line_count, count_grid, WALK_BLOCK, 0, s,
            ctx->lines.as<float4>(), ctx->line_raster.as<uint32_t>(), n_lines, lines_dev, groups,
            ctx->raster_bbox.as<int4>(),
            ctx->raster_wsum.as<int>(), ctx->line_ent_off.as<uint32_t>(), ctx->line_inc_off.as<uint32_t>(),
            reinterpret_cast<unsigned long long*>(&ds->inc_total), &ds->n_cross, &ds->line_ticket,
            &ds->err));
        OCHRE_CUDA_TRY(cudaGetLastError());
        // in place: every count is read by the thread that writes its offset
        OCHRE_LAUNCH(ctx, "dda_offset_scan", s, OCHRE_CUDA_TRY(launch_scan<LinePair>(
            ctx, n_lines, LinePairIn{ctx->line_ent_off.as<uint32_t>(), ctx->line_inc_off.as<uint32_t>()},
            LinePairOut{ctx->line_ent_off.as<uint32_t>(), ctx->line_inc_off.as<uint32_t>()}, OpLinePair{},
            LinePair{0u, 0u}, reinterpret_cast<LinePair*>(&ds->line_ent_total), s, lines_dev)));
    }
    OCHRE_LAUNCH(ctx, "raster_key_scan", s, OCHRE_CUDA_TRY(launch_scan<RasterScan>(
        ctx, R, RasterIn{ctx->raster_bbox.as<int4>(), ctx->raster_wsum.as<int>(), first, sizes},
        RasterOut{ctx->raster_bbox.as<int4>(), ctx->raster_keybase.as<uint64_t>(), ctx->raster_empty.as<uint32_t>(),
                  ctx->raster_wbase.as<int>(), sizes ? ctx->raster_run.as<RasterRun>() : nullptr, R},
        OpRaster{}, RasterScan{0, 0, 0, {0, 0, 0}, 0, 0, 0}, reinterpret_cast<RasterScan*>(&ds->keyspace), s)));
    uint64_t E;
    uint32_t bits;
    uint32_t first_entry = 0;
    uint64_t n_incs;
    bool any_empty = true;
    if (plan) {
        // entry total, key space and stored increments checked against the plan on the device
        OCHRE_LAUNCH(ctx, "plan_entries", s, OCHRE_CUDA_TRY(launch_plan_entries(ctx, plan->entries, plan->key_bits,
                                                                                plan->incs, s)));
        E = plan->entries;
        bits = plan->key_bits;
        n_incs = plan->incs;
    } else {
        int st = read_scalars(ctx, s);
        if (st != OCHRE_OK) return st;
        st = check_device_error(ctx);
        if (st != OCHRE_OK) return st;
        const DevScalars* hs = host_scalars(ctx);
        E = (uint64_t)hs->line_ent_total + hs->n_empty;
        n_incs = hs->inc_total;
        if (E > MAX_COUNT || n_incs > MAX_INCS) return OCHRE_E_CAPACITY;
        ctx->stats.n_incs = (uint32_t)n_incs;
        const uint64_t K = hs->keyspace;
        bits = 1;
        while (bits < 64 && (K - 1) >> bits) bits++;
        first_entry = hs->line_ent_total;
        any_empty = hs->n_empty != 0;
    }
    OCHRE_CUDA_TRY(ctx->incs.ensure((size_t)std::max<uint64_t>(n_incs, 1) * sizeof(float2)));
    *key_bits = bits;
    *n_entries = E;
    ctx->keys64 = bits > 32;
    const size_t ksz = ctx->keys64 ? 8 : 4;
    OCHRE_CUDA_TRY(ctx->keys.ensure(E * ksz));
    OCHRE_CUDA_TRY(ctx->vals.ensure(E * 4));
    OCHRE_CUDA_TRY(ctx->keys_alt.ensure(E * ksz));
    OCHRE_CUDA_TRY(ctx->vals_alt.ensure(E * 4));
    OCHRE_CUDA_TRY(ctx->bins.ensure(E * sizeof(BinRec)));
    auto emit_empty = [&](auto key) {
        using K = decltype(key);
        OCHRE_LAUNCH(ctx, "empty_emit", s, launch_after(
            k_empty_emit<K>, (R + 255) / 256, 256, 0, s, ctx->raster_empty.as<uint32_t>(), R, first_entry,
            plan ? &ds->line_ent_total : nullptr, plan ? &ds->n_entries : nullptr, ctx->raster_keybase.as<uint64_t>(),
            ctx->keys.as<K>(), ctx->vals.as<uint32_t>(), ctx->bins.as<BinRec>()));
    };
    // The walkers' blocks have to be placed before the per-line kernel's, whose
    // many would otherwise all go first.  Here the launches' order sees to it;
    // in a captured chain both would be ready at once, the per-line kernel even
    // earlier (early launch), so there it is an ordinary launch after another
    // kernel, the empty rasters' (a replay of 1,000 uneven paths 2.09 -> 1.75 ms,
    // of 20,000 strokes 5.92 -> 5.36).
    if (n_lines) {
        // long-line walkers: persistent, their groups take lines from the queue
        const bool apart = long_cells != 0 &&
                           (plan ? plan->long_apart : long_lines_apart(host_scalars(ctx)->n_long, n_lines));
        uint32_t long_blocks = 0;
        if (apart) {
            int sms = 152;
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
            long_blocks = (uint32_t)sms * LONG_BLOCKS_PER_SM;
        }
        cudaStream_t side = s;
        if (long_blocks) OCHRE_CUDA_TRY(fork_walks(ctx, s, &side));
        auto emit = [&](auto key) {
            using K = decltype(key);
            if (long_blocks)
                OCHRE_LAUNCH(ctx, "dda_emit_long", side, launch_beside(
                    EMIT_CARVEOUT, k_line_emit_long<K>, long_blocks, LONG_THREADS, 0, side,
                    ctx->lines.as<float4>(), ctx->line_raster.as<uint32_t>(), ctx->line_ent_off.as<uint32_t>(),
                    ctx->line_inc_off.as<uint32_t>(), n_lines, lines_dev, ctx->raster_bbox.as<int4>(),
                    ctx->raster_keybase.as<uint64_t>(), ctx->keys.as<K>(), ctx->vals.as<uint32_t>(),
                    ctx->bins.as<BinRec>(), ctx->incs.as<float2>(), queue, &ds->n_long, &ds->walk_ticket));
            if (any_empty) emit_empty(key);
            OCHRE_LAUNCH(ctx, "dda_emit", s, launch_kernel(
                plan == nullptr, k_line_emit<K>, (unsigned)((n_lines + EMIT_BLOCK - 1) / EMIT_BLOCK), EMIT_BLOCK, 0, s,
                ctx->lines.as<float4>(), ctx->line_raster.as<uint32_t>(), ctx->line_ent_off.as<uint32_t>(),
                ctx->line_inc_off.as<uint32_t>(), n_lines, lines_dev, ctx->raster_bbox.as<int4>(),
                ctx->raster_keybase.as<uint64_t>(), ctx->keys.as<K>(), ctx->vals.as<uint32_t>(),
                ctx->bins.as<BinRec>(), ctx->incs.as<float2>(), apart ? long_cells : 0u));
        };
        if (ctx->keys64) emit(uint64_t{}); else emit(uint32_t{});
        OCHRE_CUDA_TRY(cudaGetLastError());
        OCHRE_CUDA_TRY(join_walks(ctx, side, s));
    } else if (any_empty) {
        if (ctx->keys64) emit_empty(uint64_t{}); else emit_empty(uint32_t{});
        OCHRE_CUDA_TRY(cudaGetLastError());
    }
    return OCHRE_OK;
}

}  // namespace ochre
