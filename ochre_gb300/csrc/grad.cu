// Differentiable fill: dense coverage images, an L2 loss, and the
// hand-written adjoint back to control points and transforms.
//
// The reference only renders (rasterizer.rs:180-268); this extends its
// forward model.  Coverage of pixel (x, y) of raster r's w x h canvas:
//   c = min(|S|, 1),  S = (sum of heights left of the pixel on its row) + area
// inside boundary tiles (S is the reference's accum + area before
// quantisation, rasterizer.rs:232-239), 1 inside spans, 0 elsewhere.
//
// Backward, with the discrete structure (line counts, visited cells, tiles)
// held fixed: the one the last render_coverage of the same batch left in the
// context while nothing has rewritten it since, else recomputed by running
// the forward chain again:
//   dL/dS   = dL/dc * sign(S) * [|S| < 1] at boundary-tile pixels, else 0;
//   an increment (cell x, y; area a, height h) adds a to S(x, y) and h to
//   S(x', y) for every x' > x, so dL/da = dL/dS(x, y) and dL/dh = the suffix
//   sum of dL/dS to the right of x on row y;
//   a = h * m, h = p1.y - p0.y, m = ((x+1 - p0.x) + (x+1 - p1.x)) / 2 where
//   p0 / p1 are where the line enters / leaves the cell: the line's start or
//   end, or its crossing with a pixel boundary x = X (p.y = A.y + s (B.y - A.y),
//   s = (X - A.x) / (B.x - A.x)) or y = Y (symmetric);
//   line end points q_j = curve(t_j), t_j = min(j * dt, 1) with dt the
//   reference's step (path.rs:50, 60-63), so dq_j/dtheta = basis_j + curve'(t_j)
//   * j * d(dt)/dtheta for unclamped t_j;
//   device-space points p = M v + o, so dv = M^T dp, dM = dp v^T, do = dp.
// Closing lines whose ends coincide are kept as zero-length edges (see
// degenerate_dy).  Conic points are the conic at the subdivision's
// parameters t (held fixed, like the curves' line counts): linear in the
// control points, with a weight derivative (path.rs:75-104).
#include <algorithm>

#include "common.cuh"
#include "flatten.cuh"
#include "internal.h"
#include "tiles.cuh"

namespace ochre {

__device__ __forceinline__ int tile_x_of(uint32_t xy) { return (int)(int16_t)(xy & 0xffffu); }
__device__ __forceinline__ int tile_y_of(uint32_t xy) { return (int)(int16_t)(xy >> 16); }

// ---- forward: tiles and spans onto dense canvases ----
// (t_dev / n_dev / l_dev below: a count held on the device, in CUDA-graph
// replays; the launch-time count is then its capacity, see dev_count)
// A thread owns one pixel row of one tile: the tile's raster and place are
// read once for its eight pixels (from the chain's tile metadata, not by a
// search of the raster offsets per pixel), and the pixels move as two 16-byte
// words where the images' rows keep that alignment.  Of 128 dense scenes (381,634 tiles):
// 140 and 168 us with a thread and a search per pixel, 44 and 59 now.
// First pixel of a tile's row in the images, and how many of its eight lie on
// the canvas (0: none; tiles start at multiples of 8, so none straddles x = 0).
__device__ __forceinline__ int tile_row(const uint32_t* xy, const uint32_t* rf, uint32_t t,
                                        int y8, uint32_t W, uint32_t H, size_t& at) {
    const int x = 8 * tile_tx(xy[t]), y = 8 * tile_ty(xy[t]) + y8;
    if (x < 0 || y < 0 || x >= (int)W || y >= (int)H) return 0;
    at = (size_t)(rf[t] & RF_RASTER) * W * H + (size_t)y * W + (size_t)x;
    return min(8, (int)W - x);
}
__global__ void k_composite_tiles(const uint32_t* xy, const uint32_t* rf,
                                  const float* tile_sum, uint32_t T, const uint32_t* t_dev, uint32_t W,
                                  uint32_t H, bool vec, float* __restrict__ cov) {
    dependent_start();
    const uint64_t idx = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint32_t t = (uint32_t)(idx >> 3), y8 = (uint32_t)(idx & 7u);
    size_t at = 0;
    const int n = t < dev_count(T, t_dev) ? tile_row(xy, rf, t, (int)y8, W, H, at) : 0;
    if (n == 0) return;
    const float4* src = reinterpret_cast<const float4*>(tile_sum + (size_t)t * 64 + 8 * y8);
    const float4 a = src[0], b = src[1];
    const float c[8] = {fminf(fabsf(a.x), 1.0f), fminf(fabsf(a.y), 1.0f), fminf(fabsf(a.z), 1.0f),
                        fminf(fabsf(a.w), 1.0f), fminf(fabsf(b.x), 1.0f), fminf(fabsf(b.y), 1.0f),
                        fminf(fabsf(b.z), 1.0f), fminf(fabsf(b.w), 1.0f)};
    float* o = cov + at;
    if (vec && n == 8) {
        reinterpret_cast<float4*>(o)[0] = make_float4(c[0], c[1], c[2], c[3]);
        reinterpret_cast<float4*>(o)[1] = make_float4(c[4], c[5], c[6], c[7]);
    } else {
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (k < n) o[k] = c[k];
    }
}

__global__ void k_composite_spans(const uint32_t* span_xy, const uint16_t* span_w,
                                  uint32_t N, const uint32_t* n_dev, const uint32_t* raster_span_off,
                                  uint32_t R, uint32_t W, uint32_t H, float* __restrict__ cov) {
    dependent_start();
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= dev_count(N, n_dev)) return;
    const uint32_t s = (uint32_t)warp;
    const uint32_t r = upper_bound_u32(raster_span_off, R + 1, s) - 1u;
    const int x0 = tile_x_of(span_xy[s]), y0 = tile_y_of(span_xy[s]);
    const int w = span_w[s];
    float* img = cov + (size_t)r * W * H;
    for (int i = lane; i < 8 * w; i += 32) {
        const int x = x0 + i % w, y = y0 + i / w;
        if (x >= 0 && y >= 0 && x < (int)W && y < (int)H) img[(size_t)y * W + x] = 1.0f;
    }
}

// ---- L2 loss ----
// Per thread a compensated (Kahan) float sum of (cov - target)^2 (its error
// does not grow with the count: FP64 arithmetic per pixel would bound this
// kernel by the GPU's FP64 rate instead of HBM), one double per thread into
// the block reduction.  16-byte accesses when all three arrays allow.
__global__ void k_l2(const float* cov, const float* target, uint64_t n,
                     double* __restrict__ loss, float* __restrict__ dl) {
    dependent_start();
    float sum = 0.0f, comp = 0.0f;
    auto add = [&](float d) {
        const float y = d * d - comp;
        const float t = sum + y;
        comp = (t - sum) - y;
        sum = t;
    };
    const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    const bool vec = ((reinterpret_cast<uintptr_t>(cov) | reinterpret_cast<uintptr_t>(target) |
                       reinterpret_cast<uintptr_t>(dl)) & 15u) == 0;
    uint64_t done = 0;
    if (vec) {
        const uint64_t n4 = n / 4;
        const float4* c4 = reinterpret_cast<const float4*>(cov);
        const float4* t4 = reinterpret_cast<const float4*>(target);
        float4* d4 = reinterpret_cast<float4*>(dl);
        for (uint64_t i = tid; i < n4; i += stride) {
            const float4 c = c4[i], g = t4[i];
            const float4 d = make_float4(c.x - g.x, c.y - g.y, c.z - g.z, c.w - g.w);
            add(d.x);
            add(d.y);
            add(d.z);
            add(d.w);
            if (dl) d4[i] = make_float4(2.0f * d.x, 2.0f * d.y, 2.0f * d.z, 2.0f * d.w);
        }
        done = n4 * 4;
    }
    for (uint64_t i = done + tid; i < n; i += stride) {
        const float d = cov[i] - target[i];
        add(d);
        if (dl) dl[i] = 2.0f * d;
    }
    double acc = (double)sum - (double)comp;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    __shared__ double s[32];
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += s[k];
        atomicAdd(loss, t);
    }
}

// ---- backward 1: dL/dS at boundary-tile pixels ----
// An image row of W values stands at the front of the row's W pairs, where the
// next kernel leaves (dL/dS, suffix sum): one image of pairs is all the
// backward keeps, 8 bytes a pixel.  A warp clears a row's values (cudaMemset2D
// takes 15 us longer for the 65,536 rows of 128 dense scenes).
__global__ void k_clear_rows(uint64_t rows, uint32_t W, bool vec, float* __restrict__ gsig) {
    dependent_start();
    const uint64_t row = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    if (row >= rows) return;
    float* g = gsig + 2 * row * W;
    if (vec) {
        for (uint32_t i = lane; i < W / 4; i += 32) reinterpret_cast<float4*>(g)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    } else {
        for (uint32_t i = lane; i < W; i += 32) g[i] = 0.0f;
    }
}
__global__ void k_gsigma(const uint32_t* xy, const uint32_t* rf,
                         const float* tile_sum, uint32_t T, const uint32_t* t_dev, uint32_t W, uint32_t H,
                         bool vec, const float* dl_dcov, float* __restrict__ gsig) {
    dependent_start();
    const uint64_t idx = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint32_t t = (uint32_t)(idx >> 3), y8 = (uint32_t)(idx & 7u);
    size_t at = 0;
    const int n = t < dev_count(T, t_dev) ? tile_row(xy, rf, t, (int)y8, W, H, at) : 0;
    if (n == 0) return;
    const float4* src = reinterpret_cast<const float4*>(tile_sum + (size_t)t * 64 + 8 * y8);
    const float4 a = src[0], b = src[1];
    const float s[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    auto dsig = [](float v, float g) { return fabsf(v) < 1.0f ? (v > 0.0f ? g : v < 0.0f ? -g : 0.0f) : 0.0f; };
    const float* d = dl_dcov + at;
    float* o = gsig + (2 * at - (size_t)(8 * tile_tx(xy[t])));
    if (vec && n == 8) {
        const float4 g = reinterpret_cast<const float4*>(d)[0], h = reinterpret_cast<const float4*>(d)[1];
        reinterpret_cast<float4*>(o)[0] = make_float4(dsig(s[0], g.x), dsig(s[1], g.y), dsig(s[2], g.z), dsig(s[3], g.w));
        reinterpret_cast<float4*>(o)[1] = make_float4(dsig(s[4], h.x), dsig(s[5], h.y), dsig(s[6], h.z), dsig(s[7], h.w));
    } else {
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (k < n) o[k] = dsig(s[k], d[k]);
    }
}

// ---- backward 2: exclusive suffix sums of dL/dS along every canvas row ----
// Writes (dL/dS, suffix sum) pairs over the row's values: the adjoint of a cell
// reads both at once.  In place: a step's pairs lie at or past twice its first
// value's place, and every value not yet read lies before that one.
__global__ void k_row_suffix(uint64_t rows, uint32_t W, float2* gG, float* __restrict__ row_total) {
    dependent_start();
    const uint64_t row = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    float2* o = gG + row * W;
    const float* g = reinterpret_cast<const float*>(o);
    float carry = 0.0f;
    int base = (int)((W - 1) / 32) * 32;
    float next = base + lane < (int)W ? g[base + lane] : 0.0f;
    for (; base >= 0; base -= 32) {
        const int i = base + lane;
        const float v = next;
        if (base >= 32) next = g[base - 32 + lane];   // in flight during this step's sum
        float suf = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float u = __shfl_down_sync(0xffffffffu, suf, d);
            if (lane + d < 32) suf += u;
        }
        float ex = __shfl_down_sync(0xffffffffu, suf, 1);
        if (lane == 31) ex = 0.0f;
        if (i < (int)W) o[i] = make_float2(v, ex + carry);
        carry += __shfl_sync(0xffffffffu, suf, 0);
    }
    if (lane == 0) row_total[row] = carry;
}

// ---- backward 3: per line, dL/d(start, end) along the reference's cells ----
struct LineGrad {
    float ax, ay, bx, by;
};

// A zero-length edge at P (a closing line whose ends coincide, or a line_to
// to the current point): moving its end B by d opens a piece of height d.y in
// cell floor(P), so dL/dB = (0, m g + G) with m = x + 1 - P.x, and
// dL/dA = -dL/dB.  The reference draws nothing for it, but the derivative of
// the closed outline needs it.
__device__ __forceinline__ float degenerate_dy(V2 P, uint32_t r, uint32_t W, uint32_t H, const float2* gG,
                                               const float* row_total) {
    const int x = (int)floorf(P.x), y = (int)floorf(P.y);
    if (y < 0 || y >= (int)H) return 0.0f;
    float g = 0.0f, G;
    if (x < 0) {
        G = row_total[(size_t)r * H + y];
    } else if (x < (int)W) {
        const float2 v = gG[(size_t)r * W * H + (size_t)y * W + x];
        g = v.x;
        G = v.y;
    } else {
        return 0.0f;
    }
    return ((float)(x + 1) - P.x) * g + G;
}

// Pixel-cell lookup of dL/dS (g) and its exclusive row suffix sum (G);
// cells left of the canvas see the whole row's sum, cells right of it or
// off its rows see nothing.
__device__ __forceinline__ void cell_grads(int x, int y, uint32_t r, uint32_t W, uint32_t H, const float2* gG,
                                           const float* row_total, float& g, float& G) {
    g = 0.0f;
    G = 0.0f;
    if (y < 0 || y >= (int)H) return;
    if (x < 0) {
        G = row_total[(size_t)r * H + y];
    } else if (x < (int)W) {
        const float2 v = gG[(size_t)r * W * H + (size_t)y * W + x];
        g = v.x;
        G = v.y;
    }
}

// a / b for r = 1 / b rounded to nearest: the product with the reciprocal and
// one residual correction give the rounded quotient (Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990, for
// quotients in the normal range).  Beyond it the division itself: where the
// product is no number below 1e38, as it never is with a reciprocal that does
// not serve (reciprocal_for).
__device__ __forceinline__ float reciprocal_for(float r) {
    return fabsf(r) > 1e30f ? __int_as_float(0x7f800000) : r;
}
__device__ __forceinline__ float div_by(float a, float b, float r) {
    const float q = __fmul_rn(a, r);
    if (!(fabsf(q) < 1e38f)) return a / b;
    return __fmaf_rn(__fmaf_rn(-b, q, a), r, q);
}

// Per line: dL/dA and dL/dB summed over the pieces the reference's walk
// cuts the line into (one per visited cell).  Every piece end is the line's
// start (first cell only), its end (last cell only), or a crossing of the
// pixel boundary the walk stepped across (a row step crosses y = Y, a column
// step x = X).  An end point lying on a pixel boundary belongs to the cell
// floor(point), like the start of the line that follows it: when the walk's
// last cell is not floor(B), the last piece ends on the boundary and a
// zero-length piece in floor(B) carries B.  (The coverage is continuous
// there; taking both sides of a shared point in the same cell keeps the
// suffix-sum terms of consecutive lines cancelling.)
// Bound by instruction issue.  Where a line crosses a boundary between two
// cells, the cell it leaves and the cell it enters share the crossing and all
// that does not depend on their gradients; a cell's first point is the last
// one of the cell before; and a quotient by D or E takes the walk's own
// reciprocal and one correction (div_by).  Adding the two cells' gradients
// before they go to A and B would save more, but the terms of steep and flat
// lines cancel, and single gradients then moved by 0.3 % of their rms; as it
// is every operation rounds as it did.  14.4 M lines (27.9 M cells) of 128
// dense scenes: 567 us with both sides and all divisions on their own, 383 now.
__global__ void __launch_bounds__(128) k_line_grad(const float4* lines,
                                                   const uint32_t* line_raster, uint32_t L,
                                                   const uint32_t* l_dev, uint32_t W, uint32_t H,
                                                   const float2* gG, const float* row_total,
                                                   LineGrad* __restrict__ out) {
    dependent_start();
    const uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= dev_count(L, l_dev)) return;
    const float4 ln = lines[l];
    const V2 A = v2(ln.x, ln.y), B = v2(ln.z, ln.w);
    const uint32_t r = line_raster[l];
    LineGrad d{0.0f, 0.0f, 0.0f, 0.0f};
    if (veq(A, B)) {
        const float dy = degenerate_dy(B, r, W, H, gG, row_total);
        d.ay = -dy;
        d.by = dy;
        out[l] = d;
        return;
    }
    Walk w;
    WalkState s;
    walk_setup(A, B, w, s);
    const float D = B.x - A.x, E = B.y - A.y;
    const float rD = reciprocal_for(w.x_dir < 0 ? -w.x_step : w.x_step);   // 1 / D
    const float rE = reciprocal_for(w.y_dir < 0 ? -w.y_step : w.y_step);   // 1 / E
    // p.y on the vertical pixel boundary x = X, as a function of A and B
    // (dL/d(p.y) from one cell, then from the other)
    auto vertical = [&](float X, float gy, float gy2) {
        const float u = div_by(X - A.x, D, rD);
        const float db = div_by(-E * u, D, rD);
        if (gy != 0.0f) {
            d.ay += gy * (1.0f - u);
            d.by += gy * u;
            d.ax += div_by(gy * E * (u - 1.0f), D, rD);
            d.bx += gy * db;
        }
        if (gy2 != 0.0f) {
            d.ay += gy2 * (1.0f - u);
            d.by += gy2 * u;
            d.ax += div_by(gy2 * E * (u - 1.0f), D, rD);
            d.bx += gy2 * db;
        }
    };
    // p.x on the horizontal pixel boundary y = Y
    auto horizontal = [&](float Y, float gx, float gx2) {
        const float u = div_by(Y - A.y, E, rE);
        const float db = div_by(-D * u, E, rE);
        if (gx != 0.0f) {
            d.ax += gx * (1.0f - u);
            d.bx += gx * u;
            d.ay += div_by(gx * D * (u - 1.0f), E, rE);
            d.by += gx * db;
        }
        if (gx2 != 0.0f) {
            d.ax += gx2 * (1.0f - u);
            d.bx += gx2 * u;
            d.ay += div_by(gx2 * D * (u - 1.0f), E, rE);
            d.by += gx2 * db;
        }
    };
    V2 p0 = A;                       // where the line enters the cell
    float ex = 0.0f, ey = 0.0f;      // dL/d(p0) from the cell before
    bool first = true, row_in = false;   // row_in: the step into the cell went to another row
    for (uint32_t it = 0;; ++it) {
        const int x = s.x, y = s.y;
        const bool row_out = s.row_t1 < s.col_t1;   // the walk's own choice (ties step x)
        const float t1 = rmin(s.row_t1, s.col_t1);
        const bool last = t1 >= 1.0f;
        float g, G;
        cell_grads(x, y, r, W, H, gG, row_total, g, G);
        const V2 p1 = vlerp(t1, A, B);
        const float h = p1.y - p0.y;
        const float right = (float)(x + 1);
        const float m = 0.5f * ((right - p0.x) + (right - p1.x));
        // dL/dp0 = (dx, -dy) and dL/dp1 = (dx, dy) of a = h m and h (nothing
        // where no pixel sees the cell: its h and m may have overflowed)
        const bool seen = g != 0.0f || G != 0.0f;
        const float dx = seen ? -0.5f * h * g : 0.0f, dy = seen ? m * g + G : 0.0f;
        if (first) {
            d.ax += dx;
            d.ay -= dy;
        } else if (row_in) {
            if (ex != 0.0f || dx != 0.0f) horizontal((float)(w.y_dir > 0 ? y : y + 1), ex, dx);
        } else {
            if (ey != 0.0f || dy != 0.0f) vertical((float)(w.x_dir > 0 ? x : x + 1), ey, -dy);
        }
        if (last) {
            if (x == w.end_x && y == w.end_y) {
                d.bx += dx;
                d.by += dy;
            } else {
                // the boundary the last step goes to, then zero-length pieces from
                // there into floor(B), the column first (the walk's tie rule); each
                // holds the height term of its cell: dL/dp0 = (0, -q), dL/dp1 = (0, q)
                int cx = x, cy = y;
                bool row = row_out;
                float bnd = row ? (float)(w.y_dir > 0 ? y + 1 : y) : (float)(w.x_dir > 0 ? x + 1 : x);
                if (row) {
                    if (dx != 0.0f) horizontal(bnd, dx, 0.0f);
                    cy = w.y_dir > 0 ? cy + 1 : cy - 1;
                } else {
                    if (dy != 0.0f) vertical(bnd, dy, 0.0f);
                    cx = w.x_dir > 0 ? cx + 1 : cx - 1;
                }
                for (int k = 0; k < 4; k++) {
                    float gz, Gz;
                    cell_grads(cx, cy, r, W, H, gG, row_total, gz, Gz);
                    const float q = ((float)(cx + 1) - B.x) * gz + Gz;
                    if (!row) vertical(bnd, -q, 0.0f);   // a horizontal entry passes only dL/dp.x = 0
                    if (cx == w.end_x && cy == w.end_y) {
                        d.by += q;
                        break;
                    }
                    row = cx == w.end_x;
                    const int sx = w.end_x > cx ? 1 : -1, sy = w.end_y > cy ? 1 : -1;
                    bnd = row ? (float)(sy > 0 ? cy + 1 : cy) : (float)(sx > 0 ? cx + 1 : cx);
                    if (!row) vertical(bnd, q, 0.0f);
                    if (row) cy += sy; else cx += sx;
                }
            }
        }
        p0 = p1;
        ex = dx;
        ey = dy;
        first = false;
        row_in = row_out;
        if (walk_step(w, s) || it + 1 >= WALK_CAP) break;
    }
    out[l] = d;
}

// ---- backward 4: per command, through the flattening to device-space points ----
__device__ __forceinline__ void add_point(float* gp, const BatchView& b, int64_t cmd, int q, V2 g) {
    if (cmd < 0) return;
    const uint32_t f = b.cmd_foff[cmd] + 2u * (uint32_t)q;
    atomicAdd(gp + f, g.x);
    atomicAdd(gp + f + 1, g.y);
}
__device__ __forceinline__ int endpoint_index(uint8_t v) {
    return v == V_CUBIC ? 2 : (v == V_QUAD || v == V_CONIC) ? 1 : 0;
}
__device__ __forceinline__ V2 add2(V2 a, V2 b) { return v2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ V2 mul2(float s, V2 a) { return v2(s * a.x, s * a.y); }

// (`err`: a planned run's error word; when a count of the run outgrew its
// capacity the lines and offsets are not all there, and nothing is read)
__global__ void k_cmd_grad(BatchView b, const uint32_t* line_off, uint32_t L, const uint32_t* l_dev,
                           const uint32_t* err, const LineGrad* lg, float* __restrict__ gp, uint32_t W,
                           uint32_t H, const float2* gG, const float* row_total) {
    dependent_start();
    const uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (c >= b.n_cmds) return;
    if (err != nullptr && (ld_relaxed(err) & ERR_CAPACITY)) return;
    L = (uint32_t)dev_count(L, l_dev);
    const CmdCtx k = load_cmd(b, (uint32_t)c);
    if (!k.ok) return;
    const uint32_t o0 = line_off[c];
    const uint32_t o1 = c + 1 < b.n_cmds ? line_off[c + 1] : L;
    const int64_t self = (int64_t)c;
    // the final closing line of finish (rasterizer.rs:181-183) is the raster's last line
    const V2 last_end = k.verb == V_CLOSE ? k.last : k.verb == V_CUBIC ? k.pt[2]
                      : k.verb == V_MOVE || k.verb == V_LINE ? k.pt[0] : k.pt[1];
    const V2 first_end = k.verb == V_MOVE ? k.pt[0] : k.first;
    const bool final_close = k.last_of_raster && !veq(last_end, first_end);
    const int n_own = (int)(o1 - o0) - (final_close ? 1 : 0);
    auto add_last = [&](V2 g) {
        if (k.last_ref >= 0) add_point(gp, b, k.last_ref, endpoint_index(b.verbs[k.last_ref]), g);
    };
    auto add_first = [&](V2 g) { add_point(gp, b, k.first_ref, 0, g); };
    switch (k.verb) {
    case V_MOVE:
        if (n_own == 1) {
            const LineGrad g = lg[o0];
            add_last(v2(g.ax, g.ay));
            add_first(v2(g.bx, g.by));
        } else {
            // closing line last -> first of zero length
            const float dy = degenerate_dy(k.first, k.raster, W, H, gG, row_total);
            add_last(v2(0.0f, -dy));
            add_first(v2(0.0f, dy));
        }
        break;
    case V_LINE: {
        const LineGrad g = lg[o0];
        add_last(v2(g.ax, g.ay));
        add_point(gp, b, self, 0, v2(g.bx, g.by));
        break;
    }
    case V_QUAD:
    case V_CUBIC: {
        const bool cubic = k.verb == V_CUBIC;
        const V2 P0 = k.last, P1 = k.pt[0], P2 = k.pt[1], P3 = k.pt[2];
        const float dt = cubic ? cubic_dt(P0, P1, P2, P3) : quad_dt(P0, P1, P2);
        V2 g0 = v2(0, 0), g1 = v2(0, 0), g2 = v2(0, 0), g3 = v2(0, 0);
        float S = 0.0f;   // sum_j j * <curve'(t_j), dL/dq_j> over unclamped t_j
        const LineGrad first_line = lg[o0];
        g0 = v2(first_line.ax, first_line.ay);   // q_0 = last
        float t = 0.0f;
        for (int j = 1; j <= n_own; j++) {
            t = rmin(__fadd_rn(t, dt), 1.0f);
            const LineGrad gj = lg[o0 + j - 1];
            V2 dq = v2(gj.bx, gj.by);
            if (j < n_own) {
                const LineGrad gn = lg[o0 + j];
                dq = add2(dq, v2(gn.ax, gn.ay));
            }
            const float u = 1.0f - t;
            V2 dcurve;
            if (cubic) {
                const float b0 = u * u * u, b1 = 3.0f * u * u * t, b2 = 3.0f * u * t * t, b3 = t * t * t;
                g0 = add2(g0, mul2(b0, dq));
                g1 = add2(g1, mul2(b1, dq));
                g2 = add2(g2, mul2(b2, dq));
                g3 = add2(g3, mul2(b3, dq));
                dcurve = add2(add2(mul2(3.0f * u * u, vsub(P1, P0)), mul2(6.0f * u * t, vsub(P2, P1))),
                              mul2(3.0f * t * t, vsub(P3, P2)));
            } else {
                const float b0 = u * u, b1 = 2.0f * u * t, b2 = t * t;
                g0 = add2(g0, mul2(b0, dq));
                g1 = add2(g1, mul2(b1, dq));
                g2 = add2(g2, mul2(b2, dq));
                dcurve = add2(mul2(2.0f * u, vsub(P1, P0)), mul2(2.0f * t, vsub(P2, P1)));
            }
            if (t < 1.0f) S += (float)j * (dcurve.x * dq.x + dcurve.y * dq.y);
        }
        if (S != 0.0f && isfinite(dt)) {
            if (cubic) {
                // conc = max(|b|, |a + b|), b = 3(P0 - 2P1 + P2), a + b = 2P0 - 3P1 + P3
                const V2 bv = vscale(3.0f, vadd(vsub(P0, vscale(2.0f, P1)), P2));
                const V2 ab = v2(2.0f * P0.x - 3.0f * P1.x + P3.x, 2.0f * P0.y - 3.0f * P1.y + P3.y);
                const float lb = vlength(bv), lab = vlength(ab);
                const float conc = rmax(lb, lab);
                const float k1 = S * (-0.5f * dt / conc);   // dL/dconc
                if (lb >= lab && lb > 0.0f) {
                    const V2 u1 = mul2(k1 / lb, bv);
                    g0 = add2(g0, mul2(3.0f, u1));
                    g1 = add2(g1, mul2(-6.0f, u1));
                    g2 = add2(g2, mul2(3.0f, u1));
                } else if (lab > 0.0f) {
                    const V2 u1 = mul2(k1 / lab, ab);
                    g0 = add2(g0, mul2(2.0f, u1));
                    g1 = add2(g1, mul2(-3.0f, u1));
                    g3 = add2(g3, u1);
                }
            } else {
                const V2 vv = vadd(vsub(P0, vscale(2.0f, P1)), P2);
                const float len2 = vv.x * vv.x + vv.y * vv.y;
                if (len2 > 0.0f) {
                    const V2 u1 = mul2(S * (-0.5f * dt / len2), vv);   // dL/dv
                    g0 = add2(g0, u1);
                    g1 = add2(g1, mul2(-2.0f, u1));
                    g2 = add2(g2, u1);
                }
            }
        }
        add_last(g0);
        add_point(gp, b, self, 0, g1);
        add_point(gp, b, self, 1, g2);
        if (cubic) add_point(gp, b, self, 2, g3);
        break;
    }
    case V_CONIC: {
        // path.rs:75-104: every emitted point is the conic at a subdivision
        // parameter t, q = ((1-t)^2 P0 + 2t(1-t) w P1 + t^2 P2) / D, D =
        // (1-t)^2 + 2t(1-t) w + t^2; the subdivision (which t) is held fixed,
        // so q is linear in the control points, and dq/dw = 2t(1-t)(P1 - q)/D.
        const V2 P0 = k.last, P1 = k.pt[0], P2 = k.pt[1];
        const float w = k.w;
        const LineGrad first_line = lg[o0];
        V2 g0 = v2(first_line.ax, first_line.ay), g1 = v2(0, 0), g2 = v2(0, 0);
        float gw = 0.0f;
        int j = 0;
        bool capped = false;
        conic_flatten_t(P0, P1, P2, w, &capped, [&](V2 q, float t) {
            j++;
            if (j > n_own) return;
            const LineGrad gj = lg[o0 + j - 1];
            V2 dq = v2(gj.bx, gj.by);
            if (j < n_own) {
                const LineGrad gn = lg[o0 + j];
                dq = add2(dq, v2(gn.ax, gn.ay));
            }
            const float u = 1.0f - t;
            const float D = u * u + 2.0f * t * u * w + t * t;
            const float A = u * u / D, B = 2.0f * t * u * w / D, C = t * t / D;
            g0 = add2(g0, mul2(A, dq));
            g1 = add2(g1, mul2(B, dq));
            g2 = add2(g2, mul2(C, dq));
            const float dw = 2.0f * t * u / D;
            gw += dw * ((P1.x - q.x) * dq.x + (P1.y - q.y) * dq.y);
        });
        add_last(g0);
        add_point(gp, b, self, 0, g1);
        add_point(gp, b, self, 1, g2);
        atomicAdd(gp + b.cmd_foff[c] + 4, gw);   // the weight (not transformed)
        break;
    }
    default:
        break;
    }
    if (k.last_of_raster) {
        V2 ga, gb;
        if (final_close) {
            const LineGrad g = lg[o1 - 1];
            ga = v2(g.ax, g.ay);
            gb = v2(g.bx, g.by);
        } else {
            // zero-length final closing line (the contour ends where it began)
            const float dy = degenerate_dy(first_end, k.raster, W, H, gG, row_total);
            ga = v2(0.0f, -dy);
            gb = v2(0.0f, dy);
        }
        if (k.verb == V_CLOSE) add_last(ga);
        else add_point(gp, b, self, endpoint_index(k.verb), ga);
        if (k.verb == V_MOVE) add_point(gp, b, self, 0, gb);
        else add_first(gb);
    }
}

// ---- backward 5: device-space point gradients -> input points and transforms ----
__global__ void k_fill_grad(BatchView b, const float* gp, float* __restrict__ dl_dpts,
                            float* __restrict__ dl_dxf) {
    dependent_start();
    const uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool valid = c < b.n_cmds;
    float acc[6] = {0, 0, 0, 0, 0, 0};
    uint32_t f = 0xffffffffu;
    if (valid) {
        f = fill_of(b, (uint32_t)c);
        const uint8_t v = b.verbs[c];
        const uint32_t fo = b.cmd_foff[c];
        const int np = v == V_MOVE || v == V_LINE ? 1 : v == V_QUAD || v == V_CONIC ? 2 : v == V_CUBIC ? 3 : 0;
        const bool raw = b.fill_flags != nullptr && (b.fill_flags[f] & OCHRE_FILL_RAW);
        const float* m = b.fill_xf + 6 * (size_t)f;
        for (int q = 0; q < np; q++) {
            const float gx = gp[fo + 2 * q], gy = gp[fo + 2 * q + 1];
            if (raw) {
                dl_dpts[fo + 2 * q] = gx;
                dl_dpts[fo + 2 * q + 1] = gy;
            } else {
                const float vx = b.pts[fo + 2 * q], vy = b.pts[fo + 2 * q + 1];
                dl_dpts[fo + 2 * q] = m[0] * gx + m[2] * gy;
                dl_dpts[fo + 2 * q + 1] = m[1] * gx + m[3] * gy;
                acc[0] += gx * vx;
                acc[1] += gx * vy;
                acc[2] += gy * vx;
                acc[3] += gy * vy;
                acc[4] += gx;
                acc[5] += gy;
            }
        }
        if (v == V_CONIC) dl_dpts[fo + 4] = gp[fo + 4];   // the weight's gradient, as accumulated
    }
    // commands of a fill are contiguous: segmented reduction over the warp
    const uint32_t fprev = __shfl_up_sync(0xffffffffu, f, 1);
    const bool head = lane == 0 || fprev != f;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t fo = __shfl_down_sync(0xffffffffu, f, d);
#pragma unroll
        for (int i = 0; i < 6; i++) {
            const float o = __shfl_down_sync(0xffffffffu, acc[i], d);
            if (lane + d < 32 && fo == f) acc[i] += o;
        }
    }
    // a lane's sum may include lanes past its segment only if f matched all the way, which the
    // contiguity of fills guarantees; heads hold their segment's total
    if (valid && head) {
        for (int i = 0; i < 6; i++)
            if (acc[i] != 0.0f) atomicAdd(dl_dxf + 6 * (size_t)f + i, acc[i]);
    }
}

// Runs the forward chain with signed tile coverage (the backward's
// recomputation and the coverage render share it).
static int run_signed_chain(ochre_gpu_ctx* ctx, const ochre_batch* in, cudaStream_t s, ochre_result* res) {
    const uint32_t saved = ctx->flags;
    ctx->flags = (saved | OCHRE_CTX_WANT_COV | OCHRE_CTX_CHAIN_ONLY);
    ctx->cov_signed = true;
    const int st = run_device(ctx, in, res, s);
    ctx->flags = saved;
    ctx->cov_signed = false;
    return st;
}

static BatchView view_of(ochre_gpu_ctx* ctx, const ochre_batch* in) {
    return BatchView{in->verbs, in->pts, in->fill_cmd_off, in->fill_xf, in->fill_flags, in->raster_fill_off,
                     in->n_fills, in->n_rasters, in->n_cmds, ctx->cmd_foff.as<uint32_t>(),
                     ctx->cmd_mv.as<uint32_t>(), ctx->cmd_ep.as<uint32_t>(), in->n_floats};
}

// Pixel rows of an image pair may move as 16-byte words.
static bool rows_aligned(const void* a, const void* b, uint32_t w) {
    return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15u) == 0 && w % 4 == 0;
}

// Counts of a forward: launch-time values, or capacities with the counts on
// the device (graph replays).
struct ForwardCounts {
    uint32_t tiles, spans, lines;
    const uint32_t *tiles_dev, *spans_dev, *lines_dev;
    const uint32_t* err_dev;   // graph replays: the run's error word, else null
};

// Dense coverage of the chain's tiles and spans.
static int launch_render(ochre_gpu_ctx* ctx, const ForwardCounts& n, uint32_t R, uint32_t w, uint32_t h, float* cov,
                         cudaStream_t s) {
    const size_t npx = (size_t)R * w * h;
    if (npx) OCHRE_CUDA_TRY(cudaMemsetAsync(cov, 0, npx * sizeof(float), s));
    if (npx && n.tiles)
        OCHRE_LAUNCH(ctx, "composite_tiles", s, launch_after(
            k_composite_tiles, (unsigned)(((uint64_t)n.tiles * 8 + 255) / 256), 256, 0, s,
            ctx->tile_xy.as<uint32_t>(), ctx->tile_rf.as<uint32_t>(), ctx->out_tile_cov.as<float>(), n.tiles,
            n.tiles_dev, w, h, rows_aligned(cov, cov, w), cov));
    if (npx && n.spans)
        OCHRE_LAUNCH(ctx, "composite_spans", s, launch_after(
            k_composite_spans, (unsigned)(((uint64_t)n.spans * 32 + 255) / 256), 256, 0, s,
            ctx->out_span_xy.as<uint32_t>(), ctx->out_span_w.as<uint16_t>(), n.spans, n.spans_dev,
            ctx->out_raster_span_off.as<uint32_t>(), R, w, h, cov));
    OCHRE_CUDA_TRY(cudaGetLastError());
    return OCHRE_OK;
}

// Loss and dL/d(coverage).
static int launch_loss(ochre_gpu_ctx* ctx, const float* cov, const float* target, uint64_t n, double* loss,
                       float* dl_dcov, cudaStream_t s) {
    OCHRE_CUDA_TRY(cudaMemsetAsync(loss, 0, sizeof(double), s));
    if (n == 0) return OCHRE_OK;
    const int blocks = (int)std::min<uint64_t>((n + 255) / 256, 152u * 16u);
    OCHRE_LAUNCH(ctx, "l2_loss", s, launch_after(k_l2, blocks, 256, 0, s, cov, target, n, loss, dl_dcov));
    OCHRE_CUDA_TRY(cudaGetLastError());
    return OCHRE_OK;
}

// The backward on the lines and tiles the chain left in the context.
static int launch_backward(ochre_gpu_ctx* ctx, const ochre_batch* in, const ForwardCounts& n, uint32_t w, uint32_t h,
                           const float* dl_dcov, float* dl_dpts, float* dl_dxf, cudaStream_t s) {
    const uint32_t R = in->n_rasters;
    const size_t npx = (size_t)R * w * h;
    if (in->n_floats) OCHRE_CUDA_TRY(cudaMemsetAsync(dl_dpts, 0, in->n_floats * sizeof(float), s));
    if (in->n_fills) OCHRE_CUDA_TRY(cudaMemsetAsync(dl_dxf, 0, (size_t)in->n_fills * 6 * sizeof(float), s));
    if (R == 0 || in->n_cmds == 0 || n.lines == 0 || npx == 0) return OCHRE_OK;
    OCHRE_CUDA_TRY(ctx->grad_gs.ensure(npx * sizeof(float2)));
    OCHRE_CUDA_TRY(ctx->grad_left.ensure((size_t)R * h * 4));
    OCHRE_CUDA_TRY(ctx->grad_line.ensure((size_t)n.lines * sizeof(LineGrad)));
    OCHRE_CUDA_TRY(ctx->grad_pts.ensure(in->n_floats * 4));
    float2* gG = ctx->grad_gs.as<float2>();
    float* gsig = ctx->grad_gs.as<float>();   // (a row's values at the front of its pairs)
    float* row_total = ctx->grad_left.as<float>();
    LineGrad* lg = ctx->grad_line.as<LineGrad>();
    float* gp = ctx->grad_pts.as<float>();
    OCHRE_CUDA_TRY(cudaMemsetAsync(gp, 0, in->n_floats * 4, s));
    const uint64_t rows = (uint64_t)R * h;
    const unsigned row_warps = (unsigned)((rows * 32 + 255) / 256);
    OCHRE_LAUNCH(ctx, "grad_clear", s, launch_after(k_clear_rows, row_warps, 256, 0, s, rows, w,
                                                    rows_aligned(gsig, gsig, w), gsig));
    if (n.tiles)
        OCHRE_LAUNCH(ctx, "grad_sigma", s, launch_after(
            k_gsigma, (unsigned)(((uint64_t)n.tiles * 8 + 255) / 256), 256, 0, s, ctx->tile_xy.as<uint32_t>(),
            ctx->tile_rf.as<uint32_t>(), ctx->out_tile_cov.as<float>(), n.tiles, n.tiles_dev, w, h,
            rows_aligned(dl_dcov, gsig, w), dl_dcov, gsig));
    OCHRE_LAUNCH(ctx, "grad_row_suffix", s, launch_after(k_row_suffix, row_warps, 256, 0, s, rows, w, gG, row_total));
    OCHRE_LAUNCH(ctx, "grad_lines", s, launch_after(
        k_line_grad, (n.lines + 127) / 128, 128, 0, s, ctx->lines.as<float4>(), ctx->line_raster.as<uint32_t>(),
        n.lines, n.lines_dev, w, h, gG, row_total, lg));
    const BatchView b = view_of(ctx, in);
    const unsigned cb = (unsigned)((in->n_cmds + 127) / 128);
    OCHRE_LAUNCH(ctx, "grad_commands", s, launch_after(
        k_cmd_grad, cb, 128, 0, s, b, ctx->cmd_line_off.as<uint32_t>(), n.lines, n.lines_dev, n.err_dev, lg, gp, w, h,
        gG, row_total));
    OCHRE_LAUNCH(ctx, "grad_fills", s, launch_after(k_fill_grad, cb, 128, 0, s, b, gp, dl_dpts, dl_dxf));
    OCHRE_CUDA_TRY(cudaGetLastError());
    return OCHRE_OK;
}

int stage_diff_tail(ochre_gpu_ctx* ctx, const ochre_batch* in, const DiffStep& d, cudaStream_t s) {
    DevScalars* ds = dev_scalars(ctx);
    const GraphPlan* plan = ctx->plan;
    // capacities; the counts stay on the device (span capacity = tile capacity)
    const ForwardCounts n{plan->tiles, plan->tiles, plan->lines, &ds->n_tiles, &ds->n_spans, &ds->n_lines, &ds->err};
    int st = launch_render(ctx, n, in->n_rasters, d.w, d.h, d.cov, s);
    if (st != OCHRE_OK) return st;
    st = launch_loss(ctx, d.cov, d.target, (uint64_t)in->n_rasters * d.w * d.h, d.loss, d.dl_dcov, s);
    if (st != OCHRE_OK) return st;
    return launch_backward(ctx, in, n, d.w, d.h, d.dl_dcov, d.dl_dpts, d.dl_dxf, s);
}

}  // namespace ochre

using namespace ochre;

extern "C" {

int ochre_gpu_render_coverage(ochre_gpu_ctx* ctx, const ochre_batch* in, uint32_t w, uint32_t h, float* cov,
                              void* stream) {
    if (!ctx || !in || (!cov && in->n_rasters && w && h) || w > MAX_CANVAS || h > MAX_CANVAS) return OCHRE_E_INVALID;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return OCHRE_E_CUDA;
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : ctx->own_stream;
    ctx->saved.valid = false;
    ochre_result res;
    int st = run_signed_chain(ctx, in, s, &res);
    if (st != OCHRE_OK) return st;
    if (!in->fill_width)
        ctx->saved = ochre_gpu_ctx::SavedForward{true, ctx->epoch, *in, res, (uint32_t)ctx->stats.n_lines};
    const ForwardCounts n{res.n_tiles, res.n_spans, 0u, nullptr, nullptr, nullptr, nullptr};
    st = launch_render(ctx, n, in->n_rasters, w, h, cov, s);
    if (st != OCHRE_OK) return st;
    ctx->stats.n_launches = ctx->launches;
    collect_timings(ctx, s);
    return OCHRE_OK;
}

int ochre_gpu_l2_loss(ochre_gpu_ctx* ctx, const float* cov, const float* target, uint64_t n, double* loss,
                      float* dl_dcov, void* stream) {
    if (!ctx || !cov || !target || !loss) return OCHRE_E_INVALID;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return OCHRE_E_CUDA;
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : ctx->own_stream;
    ctx->prof_used = 0;
    ctx->launches = 0;
    const int st = launch_loss(ctx, cov, target, n, loss, dl_dcov, s);
    if (st != OCHRE_OK) return st;
    if (n) collect_timings(ctx, s);
    return OCHRE_OK;
}

int ochre_gpu_fill_backward(ochre_gpu_ctx* ctx, const ochre_batch* in, uint32_t w, uint32_t h,
                            const float* dl_dcov, float* dl_dpts, float* dl_dxf, void* stream) {
    if (!ctx || !in || (in->n_rasters && w && h && !dl_dcov) || (in->n_floats && !dl_dpts) ||
        (in->n_fills && !dl_dxf) || w > MAX_CANVAS || h > MAX_CANVAS)
        return OCHRE_E_INVALID;
    if (in->fill_width) return OCHRE_E_INVALID;   // stroked fills are not differentiated
    if (cudaSetDevice(ctx->device) != cudaSuccess) return OCHRE_E_CUDA;
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : ctx->own_stream;
    // the forward structure (lines, cells, tiles) and signed coverage: the
    // one the last render_coverage of this batch left, else recomputed
    ochre_result res;
    uint32_t L;
    if (ctx->saved.valid && ctx->saved.epoch == ctx->epoch && same_batch(ctx->saved.in, *in)) {
        res = ctx->saved.res;
        L = ctx->saved.n_lines;
        ctx->prof_used = 0;
        ctx->launches = 0;
    } else {
        const int st = run_signed_chain(ctx, in, s, &res);
        if (st != OCHRE_OK) return st;
        L = (uint32_t)ctx->stats.n_lines;
    }
    const ForwardCounts n{res.n_tiles, res.n_spans, L, nullptr, nullptr, nullptr, nullptr};
    const int st = launch_backward(ctx, in, n, w, h, dl_dcov, dl_dpts, dl_dxf, s);
    if (st != OCHRE_OK) return st;
    ctx->stats.n_launches = ctx->launches;
    collect_timings(ctx, s);
    return OCHRE_OK;
}

}  // extern "C"
