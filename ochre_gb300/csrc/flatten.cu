// Stage 1: commands -> line segments (flattening).
//
// Reference: Rasterizer::fill / command (rasterizer.rs:145-165),
// PathCmd::transform (path.rs:16-37), PathCmd::flatten (path.rs:41-109),
// and the implicit closing lines of move_to / finish (rasterizer.rs:62-64,
// 181-183).
//
// A raster's line list is the sequence of its line_to calls.  Each command
// contributes, in order:
//   Move   : the closing line last -> first when last != first
//   Line   : last -> point
//   Quad   : n lines from the serial t recurrence (path.rs:52-57)
//   Cubic  : n lines (path.rs:65-73)
//   Conic  : 2 lines per subdivision leaf (path.rs:76-101)
//   Close  : nothing (rasterizer.rs:154 ignores it)
// plus, on the raster's last command, the final closing line of finish.
// `last` for a command is the transformed end point of the most recent
// earlier non-Close command of the raster (or (0,0)), `first` the point of
// the most recent earlier Move (or (0,0)); both come from one scan.
#include "common.cuh"
#include "flatten.cuh"
#include "internal.h"
#include "scan.cuh"

namespace ochre {


// The line finish() adds after a raster's last command, if any
// (rasterizer.rs:181-183: line_to(first) when last != first).
__device__ __forceinline__ bool closing_line(const CmdCtx& k, V2* from, V2* to) {
    if (!k.last_of_raster) return false;
    *from = k.verb == V_CLOSE ? k.last : k.verb == V_CUBIC ? k.pt[2]
          : k.verb == V_MOVE || k.verb == V_LINE ? k.pt[0] : k.pt[1];
    *to = k.verb == V_MOVE ? k.pt[0] : k.first;
    return !veq(*from, *to);
}

// Line count of one command (the count pass never materialises points for
// curves: it only replays the t recurrence).
__device__ uint32_t count_cmd(const CmdCtx& k, bool* capped) {
    uint32_t n = 0;
    switch (k.verb) {
    case V_MOVE: n = veq(k.last, k.first) ? 0u : 1u; break;
    case V_LINE: n = 1; break;
    case V_QUAD: n = flatten_steps(quad_dt(k.last, k.pt[0], k.pt[1]), capped); break;
    case V_CUBIC: n = flatten_steps(cubic_dt(k.last, k.pt[0], k.pt[1], k.pt[2]), capped); break;
    case V_CONIC: conic_flatten(k.last, k.pt[0], k.pt[1], k.w, capped, [&](V2) { n++; }); break;
    default: break;
    }
    V2 from, to;
    if (closing_line(k, &from, &to)) n++;
    return n;
}

struct Load32 {
    const uint32_t* v;
    __device__ __forceinline__ uint32_t operator()(uint64_t i) const { return v[i]; }
    using takes_all = void;
    template <int N>
    __device__ __forceinline__ void load_all(uint64_t i, uint32_t (&w)[N]) const {
        load_words(v + i, w);
    }
};

// Line counts, one thread per command, then a scan of them (a scan that counted
// as it read gave each thread eight serial t loops, one after the other: 161
// against 108 us for the 2.0 M commands of 20,000 uneven paths).
__global__ void __launch_bounds__(128) k_cmd_count(BatchView b, uint32_t* __restrict__ counts, uint32_t* err) {
    dependent_start();
    const uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (c >= b.n_cmds) return;
    const CmdCtx k = load_cmd(b, (uint32_t)c);
    uint32_t n = 0;
    if (!k.ok) {
        atomicOr(err, ERR_INVALID);
    } else {
        bool capped = false;
        n = count_cmd(k, &capped);
        if (capped) atomicOr(err, ERR_LIMIT);
    }
    counts[c] = n;
}

// Lines of a block's commands.  SHARED: a curve's line is one thread's work,
// as the next line of the same curve is the next thread's; the parameter of a
// point is the reference's serial sum, which a thread carries from one of its
// lines to the next, and the line's two points follow from it.  The other
// commands (and a raster's closing line) are written by the thread that read
// them, and without SHARED the curves as well.  A thread that writes a whole
// curve writes line after line, 16 bytes at a time in as many places as there
// are lanes, which is what bounds it with many lines a command: 2.0 M commands,
// 60 M lines 1.15 ms, shared 0.71 ms.  With few lines a command a thread's
// lines lie close together and the sharing costs more than it saves (14 M
// lines of 2.7 M commands 158 us, shared 207), and with few commands the blocks
// have too many lines each (33,000 commands, 1.1 M lines 26 us, shared 76).  So:
// shared from 8 lines a command and 131,072 commands on.  (Blocks of 128
// commands, a conic's stack out of the curves' way: 190 -> 158 us, strokes 174 ->
// 150.)
// Lines of more than long_cells cells (walk_cells) are also queued for the
// long-line emit walk of the DDA stage (long_cells 0: none are).
constexpr int FLAT_BLOCK = 128;
constexpr uint64_t FLAT_SHARED_LINES = 8, FLAT_SHARED_CMDS = 1u << 17;
template <bool SHARED>
__global__ void __launch_bounds__(FLAT_BLOCK) k_cmd_emit(BatchView b, const uint32_t* line_off,
                                                         const uint32_t* n_lines, uint32_t n_lines_cap,
                                                         float4* __restrict__ lines, uint32_t* __restrict__ line_raster,
                                                         uint32_t long_cells, uint32_t* __restrict__ long_lines,
                                                         uint32_t* n_long, uint32_t* err) {
    dependent_start();
    // the curves: last, control points and end; parameter step; 2 or 3 (0: no
    // curve); raster.  And every command's first line.
    constexpr int CMDS = FLAT_BLOCK, S = SHARED ? CMDS : 1;
    __shared__ V2 s_p[4][S];
    __shared__ float s_dt[S];
    __shared__ uint8_t s_degree[S];
    __shared__ uint32_t s_raster[S], s_off[S + 1], s_end[S];
    const uint64_t c0 = blockIdx.x * (uint64_t)CMDS;
    const int n = (int)min((uint64_t)CMDS, b.n_cmds - c0);
    auto put = [&](uint32_t o, V2 a, V2 p, uint32_t raster) {
        if (o < n_lines_cap) {
            const float4 l = make_float4(a.x, a.y, p.x, p.y);
            lines[o] = l;
            line_raster[o] = raster;
            if (long_cells && walk_cells(l) > long_cells) long_lines[atomicAdd(n_long, 1u)] = o;
        } else {
            atomicOr(err, ERR_CAPACITY);
        }
    };
    uint8_t degree = 0;
    if ((int)threadIdx.x < n) {
        const uint64_t c = c0 + threadIdx.x;
        const CmdCtx k = load_cmd(b, (uint32_t)c);
        const uint32_t first = line_off[c];
        uint32_t o = first;
        // (a line count zeroed on the device, after an overflow of a graph's plan, ends no lines)
        uint32_t end = max(o, c + 1 < b.n_cmds ? line_off[c + 1] : *n_lines);
        if (k.ok) {
            V2 from, to;
            const bool closes = closing_line(k, &from, &to);
            if (closes && end > o) put(end - 1u, from, to, k.raster);
            if (closes && end > o) end--;
            switch (k.verb) {
            case V_MOVE:
                if (!veq(k.last, k.first)) put(o, k.last, k.first, k.raster);
                break;
            case V_LINE:
                put(o, k.last, k.pt[0], k.raster);
                break;
            case V_QUAD:
            case V_CUBIC: {
                degree = k.verb == V_QUAD ? 2 : 3;
                const float dt = degree == 2 ? quad_dt(k.last, k.pt[0], k.pt[1]) : cubic_dt(k.last, k.pt[0], k.pt[1], k.pt[2]);
                if (SHARED) {
                    s_dt[threadIdx.x] = dt;
                    break;
                }
                V2 prev = k.last;
                float t = 0.0f;
                for (; o < end; o++) {
                    t = rmin(__fadd_rn(t, dt), 1.0f);
                    const V2 p = degree == 2 ? quad_point(t, k.last, k.pt[0], k.pt[1])
                                             : cubic_point(t, k.last, k.pt[0], k.pt[1], k.pt[2]);
                    put(o, prev, p, k.raster);
                    prev = p;
                }
                break;
            }
            case V_CONIC: {
                bool capped = false;
                V2 prev = k.last;
                conic_flatten(k.last, k.pt[0], k.pt[1], k.w, &capped, [&](V2 p) {
                    put(o++, prev, p, k.raster);
                    prev = p;
                });
                break;
            }
            default:
                break;
            }
            if (SHARED) {
                s_p[0][threadIdx.x] = k.last;
                s_p[1][threadIdx.x] = k.pt[0];
                s_p[2][threadIdx.x] = k.pt[1];
                s_p[3][threadIdx.x] = k.pt[2];
                s_raster[threadIdx.x] = k.raster;
            }
        }
        if (SHARED) {
            s_off[threadIdx.x] = first;
            s_degree[threadIdx.x] = degree;
            s_end[threadIdx.x] = end;   // of the command's own lines
            if ((int)threadIdx.x == n - 1) s_off[n] = end;
        }
    }
    if (!SHARED) return;
    if (!__syncthreads_or(degree != 0)) return;
    int curve = -1;         // the command of the thread's line before this one,
    uint32_t done = 0;      // the steps of its parameter taken
    float t = 0.0f;         // and where they led
    for (uint32_t o = s_off[0] + threadIdx.x; o < s_off[n]; o += FLAT_BLOCK) {
        int j = 0;   // the last command with s_off <= o
#pragma unroll
        for (int step = CMDS / 2; step > 0; step >>= 1)
            if (j + step < n && s_off[j + step] <= o) j += step;
        const int degree = s_degree[j];
        if (degree == 0 || o >= s_end[j]) continue;
        const V2 last = s_p[0][j], p0 = s_p[1][j], p1 = s_p[2][j], p2 = s_p[3][j];
        const float dt = s_dt[j];
        const uint32_t before = o - s_off[j];
        if (j != curve) {
            curve = j;
            done = 0;
            t = 0.0f;
        }
        for (; done < before; done++) t = rmin(__fadd_rn(t, dt), 1.0f);
        const float t1 = rmin(__fadd_rn(t, dt), 1.0f);
        V2 a, p;
        if (degree == 2) {
            a = quad_point(t, last, p0, p1);
            p = quad_point(t1, last, p0, p1);
        } else {
            a = cubic_point(t, last, p0, p1, p2);
            p = cubic_point(t1, last, p0, p1, p2);
        }
        put(o, before ? a : last, p, s_raster[j]);
    }
}

int stage_flatten(ochre_gpu_ctx* ctx, const ochre_batch* in, cudaStream_t s, uint32_t* n_lines) {
    const uint64_t n = in->n_cmds;
    DevScalars* ds = dev_scalars(ctx);
    *n_lines = 0;
    if (n == 0) return OCHRE_OK;
    OCHRE_CUDA_TRY(ctx->cmd_foff.ensure(n * 4));
    OCHRE_CUDA_TRY(ctx->cmd_mv.ensure(n * 4));
    OCHRE_CUDA_TRY(ctx->cmd_ep.ensure(n * 4));
    OCHRE_CUDA_TRY(ctx->cmd_line_off.ensure(n * 4));

    CmdScan total_id{0, 0, 0};
    OCHRE_LAUNCH(ctx, "cmd_scan", s, OCHRE_CUDA_TRY(launch_scan<CmdScan>(ctx, n, CmdIn{in->verbs, &ds->err},
                                        CmdOut{ctx->cmd_foff.as<uint32_t>(), ctx->cmd_mv.as<uint32_t>(),
                                               ctx->cmd_ep.as<uint32_t>()},
                                        OpCmd{}, total_id, reinterpret_cast<CmdScan*>(&ds->n_floats), s)));

    // A command whose points lie beyond the point array is flagged invalid
    // by the kernels that read it (load_cmd), reported at the next read-back.
    const GraphPlan* plan = ctx->plan;
    int st = OCHRE_OK;
    const DevScalars* hs = host_scalars(ctx);

    wait_inputs(ctx, s);   // the counts read points
    BatchView b{in->verbs, in->pts, in->fill_cmd_off, in->fill_xf, in->fill_flags, in->raster_fill_off,
                in->n_fills, in->n_rasters, n, ctx->cmd_foff.as<uint32_t>(), ctx->cmd_mv.as<uint32_t>(),
                ctx->cmd_ep.as<uint32_t>(), in->n_floats};
    // counts first, then the offsets in place
    OCHRE_LAUNCH(ctx, "flatten_count", s, launch_after(k_cmd_count, (unsigned)((n + 127) / 128), 128, 0, s, b,
                                                       ctx->cmd_line_off.as<uint32_t>(), &ds->err));
    OCHRE_CUDA_TRY(cudaGetLastError());
    OCHRE_LAUNCH(ctx, "flatten_count_scan", s, OCHRE_CUDA_TRY(launch_scan<uint32_t>(
        ctx, n, Load32{ctx->cmd_line_off.as<uint32_t>()}, ScanOff{ctx->cmd_line_off.as<uint32_t>()}, OpSumU32{}, 0u,
        &ds->n_lines, s)));
    uint32_t L;
    if (plan) {
        // the line count stays on the device; above the plan it is zeroed
        OCHRE_LAUNCH(ctx, "plan_lines", s, OCHRE_CUDA_TRY(launch_plan_cap(ctx, &ds->n_lines, plan->lines, s)));
        L = plan->lines;
    } else {
        st = read_scalars(ctx, s);
        if (st != OCHRE_OK) return st;
        st = check_device_error(ctx);
        if (st != OCHRE_OK) return st;
        L = hs->n_lines;
    }
    *n_lines = L;
    if (L == 0) return OCHRE_OK;
    if (L > MAX_COUNT) return OCHRE_E_CAPACITY;
    OCHRE_CUDA_TRY(ctx->lines.ensure((size_t)L * sizeof(float4)));
    OCHRE_CUDA_TRY(ctx->line_raster.ensure((size_t)L * 4));
    const uint32_t long_cells = (uint32_t)ctx->tune_chain_long_cells;
    if (long_cells) OCHRE_CUDA_TRY(ctx->long_lines.ensure((size_t)L * 4));
    OCHRE_CUDA_TRY(cudaMemsetAsync(&ds->n_long, 0, 4, s));
    // (planned: L is the plan's capacity)
    const bool shared = L >= FLAT_SHARED_LINES * n && n >= FLAT_SHARED_CMDS;
    OCHRE_LAUNCH(ctx, "flatten_emit", s, launch_after(shared ? k_cmd_emit<true> : k_cmd_emit<false>,
        (unsigned)((n + FLAT_BLOCK - 1) / FLAT_BLOCK), FLAT_BLOCK, 0, s, b, ctx->cmd_line_off.as<uint32_t>(), &ds->n_lines,
        L, ctx->lines.as<float4>(), ctx->line_raster.as<uint32_t>(), long_cells,
        long_cells ? ctx->long_lines.as<uint32_t>() : nullptr, &ds->n_long, &ds->err));
    OCHRE_CUDA_TRY(cudaGetLastError());
    return OCHRE_OK;
}

}  // namespace ochre
