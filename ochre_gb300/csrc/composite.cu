// Headless compositing of rasterization results into an RGBA8 canvas: the
// reference example's GL path (examples/svg.rs) restated on the device.
//   * every tile is an 8x8 quad textured with its alpha mask, every span an
//     n x 8 quad with mask 1 (atlas texel (0,0) = 255, :33-38, 85-87);
//   * fragment = raster colour * (1, 1, 1, mask) (:341-353);
//   * blend SRC_ALPHA, ONE_MINUS_SRC_ALPHA on all four channels (:173-174)
//     into an RGBA8 target, quantised after every quad: f -> floor(f*255 + 0.5);
//   * rasters are drawn in order (:139-165); within one raster no two quads
//     overlap, so only the raster order matters per pixel.
// The GL pipeline itself is unavailable on this machine; this kernel and the
// oracle restate its arithmetic.
//
// Device form: every quad is cut into the 8x8 screen tiles it covers (tile
// and span positions are multiples of 8).  The pieces are emitted in raster
// order (a raster's tiles, then its spans) with the key (screen tile, raster)
// and sorted by the screen tile alone: the sort is stable, so a screen tile's
// pieces keep their raster order, and half the key's digits need no pass.  One
// warp per screen tile then blends its pieces in order, two pixels per lane,
// with the canvas in registers.
#include "common.cuh"
#include "internal.h"
#include "scan.cuh"

namespace ochre {

// The result's tiles and spans in raster order: item i of raster r's range
// [tile_off[r] + span_off[r], tile_off[r + 1] + span_off[r + 1]) is one of its
// tiles, then one of its spans.
struct PieceItems {
    const int16_t* tile_xy;
    const int16_t* span_xy;
    const uint16_t* span_w;
    const uint32_t* raster_tile_off;
    const uint32_t* raster_span_off;
    uint32_t T, N, R;
    int w, h, w8;

    struct Item {
        uint32_t raster, value;   // value: tile index, or T + span index
        int x0, x1, y;            // the screen tiles' left edges are x0, x0 + 8, .. < x1
    };
    __device__ __forceinline__ Item operator()(uint32_t i) const {
        Item it{0u, 0u, 0, 0, 0};
        uint32_t lo = 0, hi = R + 1;   // first raster whose range starts after i
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (raster_tile_off[mid] + raster_span_off[mid] <= i) lo = mid + 1; else hi = mid;
        }
        const uint32_t r = lo - 1u;
        if (lo == 0u || r >= R) return it;   // a raster past the caller's count: not drawn
        const uint32_t t0 = raster_tile_off[r], s0 = raster_span_off[r];
        const uint32_t nt = raster_tile_off[r + 1] - t0, k = i - t0 - s0;
        it.raster = r;
        if (k < nt) {
            const uint32_t t = t0 + k;
            const int x = tile_xy[2 * (size_t)t], y = tile_xy[2 * (size_t)t + 1];
            it.value = t;
            if (x >= 0 && y >= 0 && x < w && y < h) {
                it.x0 = x;
                it.x1 = x + 8;
                it.y = y;
            }
            return it;
        }
        const uint32_t s = s0 + (k - nt);
        const int x = span_xy[2 * (size_t)s], y = span_xy[2 * (size_t)s + 1];
        it.value = T + s;
        if (y >= 0 && y < h) {
            it.x0 = max(x, 0);
            it.x1 = max(it.x0, min(x + (int)span_w[s], 8 * w8));
            it.y = y;
        }
        return it;
    }
};
struct PieceCount {
    PieceItems items;
    __device__ __forceinline__ uint32_t operator()(uint64_t i) const {
        const PieceItems::Item it = items((uint32_t)i);
        return (uint32_t)((it.x1 - it.x0) >> 3);
    }
};
struct PieceOff {
    uint32_t* off;
    __device__ __forceinline__ void operator()(uint64_t i, uint32_t ex, uint32_t) const { off[i] = ex; }
};

template <class K>
__global__ void k_piece_emit(PieceItems items, uint32_t rbits, const uint32_t* off, K* __restrict__ keys,
                             uint32_t* __restrict__ vals) {
    dependent_start();
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= (uint64_t)items.T + items.N) return;
    const PieceItems::Item it = items((uint32_t)i);
    uint32_t o = off[i];
    for (int x = it.x0; x < it.x1; x += 8) {
        const K st = (K)(it.y >> 3) * (K)items.w8 + (K)(x >> 3);
        keys[o] = (st << rbits) | (K)it.raster;
        vals[o] = it.value;
        o++;
    }
}

// First sorted piece of every screen tile that has one (the others keep
// NO_PIECE): one pass over the keys instead of two searches of the sorted keys
// per screen tile.
constexpr uint32_t NO_PIECE = 0xffffffffu;
template <class K>
__global__ void k_piece_heads(const K* keys, uint32_t E, uint32_t rbits, uint32_t n_tiles,
                              uint32_t* __restrict__ head, const uint32_t* err, uint32_t* late_err) {
    dependent_start();
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    if (run_aborted(err)) {   // a wait of the sort gave up: the sorted pieces are not valid
        if (e == 0) atomicOr(late_err, ERR_TIMEOUT);   // (the call will have returned)
        return;
    }
    const K st = keys[e] >> rbits;
    if ((e == 0 || (keys[e - 1] >> rbits) != st) && st < (K)n_tiles) head[st] = e;
}

// ---- two pixels at a time: packed f32 pairs (every operation rounds each
// half as the scalar one does) ----
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    return (f32x2)__float_as_uint(a) | ((f32x2)__float_as_uint(b) << 32);
}
__device__ __forceinline__ float lo2(f32x2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi2(f32x2 v) { return __uint_as_float((uint32_t)(v >> 32)); }
// The product alone, rounded: a fused multiply-add of -0 (x + -0 = x), with
// the -0 handed in at run time.  Written as a packed mul (or with a literal
// -0) it was fused with the add that follows into one rounding, and one pixel
// in half a million differed from the reference's two roundings.
__device__ __forceinline__ f32x2 mul2x(f32x2 a, f32x2 b, f32x2 neg_zero) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(neg_zero));
    return r;
}
__device__ __forceinline__ f32x2 add2x(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2x_down(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2x(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
constexpr float RCP_255 = 0x1.010102p-8f;   // 1 / 255 to the nearest f32
constexpr float TWO_23 = 8388608.0f;
// x / 255 rounded to nearest for integers 0 .. 255: the product with 1/255 and
// one residual correction give the correctly rounded quotient for all 256 of
// them (tests/test_composite_pieces.py).
__device__ __forceinline__ float div255(float x) {
    const float q = __fmul_rn(x, RCP_255);
    return __fmaf_rn(__fmaf_rn(-255.0f, q, x), RCP_255, q);
}
__device__ __forceinline__ f32x2 div255x2(f32x2 x, f32x2 neg_zero) {
    const f32x2 rcp = pack2(RCP_255, RCP_255);
    const f32x2 q = mul2x(x, rcp, neg_zero);
    return fma2x(fma2x(pack2(-255.0f, -255.0f), q, x), rcp, q);
}
// floor(f * 255 + 0.5) for 0 <= f (f * 255 + 0.5 < 2^23): adding 2^23 rounded
// down leaves the floor, exactly.  (f is s a + d (1 - a) with s, a, d in
// [0, 1], which rounds to at most 1 + 2^-23, so the result never exceeds 255.)
__device__ __forceinline__ f32x2 unorm8x2(f32x2 f, f32x2 neg_zero) {
    const f32x2 y = add2x(mul2x(f, pack2(255.0f, 255.0f), neg_zero), pack2(0.5f, 0.5f));
    return add2x(add2x_down(y, pack2(TWO_23, TWO_23)), pack2(-TWO_23, -TWO_23));
}
// Bytes 0 and 1 of v as floats: 2^23 + byte, minus 2^23.
__device__ __forceinline__ f32x2 bytes2(uint32_t v) {
    const f32x2 m = pack2(__uint_as_float(0x4b000000u | (v & 0xffu)), __uint_as_float(0x4b000000u | ((v >> 8) & 0xffu)));
    return add2x(m, pack2(-TWO_23, -TWO_23));
}

// One warp per screen tile.  Bound by instruction issue (about 60 per piece
// and warp): a lane holds two neighbouring pixels, so every step of the blend
// is one packed operation for both, the divisions by 255 take three, and 32
// pieces' keys, values and colours (already divided) are loaded by the 32
// lanes at once and handed round by shuffles; the masks of BLEND_AHEAD pieces
// are in flight before the first is blended.  20,000 glyphs on a 2048 x 2048
// canvas: 250 us with one scalar pixel at a time, IEEE divisions and the
// pieces' loads one after the other, 72 us now; the sort by screen tile alone
// 28 us where (screen tile, raster) took 58.
constexpr int BLEND_AHEAD = 4;
template <class K>
__global__ void __launch_bounds__(128) k_composite(const K* keys, const uint32_t* vals,
                                                   uint32_t E, const uint32_t* head, uint32_t rbits,
                                                   uint32_t T, const uint8_t* tile_alpha,
                                                   const uint32_t* colors, uint32_t n_rasters, uint32_t w,
                                                   uint32_t h, uint32_t w8, uint32_t h8, uint32_t* canvas,
                                                   float neg_zero, const uint32_t* err) {
    dependent_start();
    const uint32_t st = (uint32_t)((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5);
    const uint32_t lane = threadIdx.x & 31u;
    // a wait of the sort gave up: the sorted pieces are not valid
    if (st >= w8 * h8 || run_aborted(err)) return;
    uint32_t e0 = head[st];
    if (e0 == NO_PIECE) return;
    const uint32_t tx = st % w8, ty = st / w8;
    const K rmask = (K)(((K)1 << rbits) - 1);
    const bool alpha16 = (reinterpret_cast<uintptr_t>(tile_alpha) & 1u) == 0;   // a caller's copy may sit anywhere
    const uint32_t x = 8 * tx + ((2 * lane) & 7u), y = 8 * ty + (lane >> 2);
    const bool in0 = x < w && y < h, in1 = x + 1 < w && y < h;
    uint32_t* px = canvas + (size_t)y * w + x;
    const uint32_t p0 = in0 ? px[0] : 0u, p1 = in1 ? px[1] : 0u;
    f32x2 d[4];   // channel values 0 .. 255 of the two pixels
#pragma unroll
    for (int c = 0; c < 4; c++) d[c] = bytes2(((p0 >> (8 * c)) & 0xffu) | (((p1 >> (8 * c)) & 0xffu) << 8));
    const f32x2 one = pack2(1.0f, 1.0f), minus = pack2(-1.0f, -1.0f), nz = pack2(neg_zero, neg_zero);
    for (;;) {
        const uint32_t e = e0 + lane;
        bool mine = false;
        uint32_t val = 0;
        float col[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (e < E) {
            const K key = keys[e];
            const uint32_t r = (uint32_t)(key & rmask);
            mine = (key >> rbits) == (K)st && r < n_rasters;
            if (mine) {
                val = vals[e];
                const uint32_t c32 = colors[r];
#pragma unroll
                for (int c = 0; c < 4; c++) col[c] = div255((float)((c32 >> (8 * c)) & 0xffu));
            }
        }
        const int n = __popc(__ballot_sync(0xffffffffu, mine));   // the first n lanes
        for (int k0 = 0; k0 < n; k0 += BLEND_AHEAD) {
            uint32_t mask[BLEND_AHEAD];
#pragma unroll
            for (int u = 0; u < BLEND_AHEAD; u++) {
                const uint32_t v = __shfl_sync(0xffffffffu, val, (k0 + u) & 31);
                mask[u] = 0xffffu;
                if (k0 + u < n && v < T) {
                    const uint8_t* m = tile_alpha + (size_t)v * 64 + 2 * lane;
                    mask[u] = alpha16 ? *reinterpret_cast<const uint16_t*>(m) : (uint32_t)m[0] | ((uint32_t)m[1] << 8);
                }
            }
#pragma unroll
            for (int u = 0; u < BLEND_AHEAD; u++) {
                const int k = k0 + u;
                if (k >= n) break;
                const float ca = __shfl_sync(0xffffffffu, col[3], k);
                const f32x2 a = mul2x(pack2(ca, ca), div255x2(bytes2(mask[u]), nz), nz);
                const f32x2 ia = fma2x(a, minus, one);   // 1 - a, rounded once
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const float s = __shfl_sync(0xffffffffu, col[c], k);
                    d[c] = unorm8x2(add2x(mul2x(pack2(s, s), a, nz), mul2x(div255x2(d[c], nz), ia, nz)), nz);
                }
                d[3] = unorm8x2(add2x(mul2x(a, a, nz), mul2x(div255x2(d[3], nz), ia, nz)), nz);
            }
        }
        if (n < 32) break;
        e0 += 32;
    }
    uint32_t o0 = 0, o1 = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        o0 |= (uint32_t)lo2(d[c]) << (8 * c);
        o1 |= (uint32_t)hi2(d[c]) << (8 * c);
    }
    if (in0) px[0] = o0;
    if (in1) px[1] = o1;
}

// Pieces, sort by screen tile, heads, blend; K holds (screen tile, raster).
template <class K>
static int composite_pieces(ochre_gpu_ctx* ctx, const PieceItems& items, uint32_t E, uint32_t sbits, uint32_t rbits,
                            const uint8_t* tile_alpha, const uint8_t* colors, uint8_t* canvas, cudaStream_t s) {
    DevScalars* ds = dev_scalars(ctx);
    const uint64_t S = (uint64_t)items.T + items.N;
    const uint32_t w8 = (uint32_t)items.w8, h8 = (uint32_t)(items.h + 7) / 8, screen = w8 * h8;
    ctx->keys64 = sizeof(K) == 8;
    OCHRE_CUDA_TRY(ctx->keys.ensure((size_t)E * sizeof(K)));
    OCHRE_CUDA_TRY(ctx->vals.ensure((size_t)E * 4));
    OCHRE_CUDA_TRY(ctx->keys_alt.ensure((size_t)E * sizeof(K)));
    OCHRE_CUDA_TRY(ctx->vals_alt.ensure((size_t)E * 4));
    OCHRE_CUDA_TRY(ctx->tile_head.ensure((size_t)screen * 4));
    OCHRE_LAUNCH(ctx, "composite_pieces", s, launch_after(k_piece_emit<K>, (unsigned)((S + 255) / 256), 256, 0, s,
        items, rbits, ctx->line_ent_off.as<uint32_t>(), ctx->keys.as<K>(), ctx->vals.as<uint32_t>()));
    OCHRE_CUDA_TRY(cudaGetLastError());
    uint32_t passes = 0;
    const int st = stage_sort(ctx, E, sbits, s, &passes, rbits);
    if (st != OCHRE_OK) return st;
    uint32_t* head = ctx->tile_head.as<uint32_t>();
    OCHRE_CUDA_TRY(cudaMemsetAsync(head, 0xff, (size_t)screen * 4, s));
    OCHRE_LAUNCH(ctx, "composite_heads", s, launch_after(k_piece_heads<K>, (E + 255) / 256, 256, 0, s,
        ctx->keys.as<K>(), E, rbits, screen, head, &ds->err, &ds->late_err));
    OCHRE_CUDA_TRY(cudaGetLastError());
    OCHRE_LAUNCH(ctx, "composite", s, launch_after(k_composite<K>, (unsigned)(((uint64_t)screen * 32 + 127) / 128), 128, 0, s,
        ctx->keys.as<K>(), ctx->vals.as<uint32_t>(), E, head, rbits, items.T, tile_alpha,
        reinterpret_cast<const uint32_t*>(colors), items.R, (uint32_t)items.w, (uint32_t)items.h, w8, h8,
        reinterpret_cast<uint32_t*>(canvas), -0.0f, &ds->err));
    OCHRE_CUDA_TRY(cudaGetLastError());
    return OCHRE_OK;
}

static int composite(ochre_gpu_ctx* ctx, const ochre_result* res, uint32_t n_rasters, const uint8_t* colors, uint32_t w,
                     uint32_t h, uint8_t* canvas, cudaStream_t s) {
    const uint32_t T = res->n_tiles, N = res->n_spans;
    const uint32_t w8 = (w + 7) / 8, h8 = (h + 7) / 8;
    uint32_t rbits = 1;
    while (rbits < 32 && ((n_rasters - 1) >> rbits)) rbits++;
    uint32_t sbits = 1;
    while (sbits < 40 && (((uint64_t)w8 * h8 - 1) >> sbits)) sbits++;
    DevScalars* ds = dev_scalars(ctx);
    const uint64_t S = (uint64_t)T + N;
    const PieceItems items{res->tile_xy, res->span_xy, res->span_width, res->raster_tile_off, res->raster_span_off,
                           T, N, n_rasters, (int)w, (int)h, (int)w8};
    OCHRE_CUDA_TRY(ctx->line_ent_off.ensure(S * 4));
    OCHRE_CUDA_TRY(reset_scalars(ctx, s));
    OCHRE_LAUNCH(ctx, "composite_count", s, OCHRE_CUDA_TRY(launch_scan<uint32_t>(
        ctx, S, PieceCount{items}, PieceOff{ctx->line_ent_off.as<uint32_t>()}, OpSumU32{}, 0u, &ds->n_line_ent, s)));
    int st = read_scalars(ctx, s);
    if (st != OCHRE_OK) return st;
    st = check_device_error(ctx);
    if (st != OCHRE_OK) return st;
    const uint64_t E = host_scalars(ctx)->n_line_ent;
    if (E == 0) return OCHRE_OK;
    if (E > MAX_COUNT) return OCHRE_E_CAPACITY;
    st = sbits + rbits <= 32
             ? composite_pieces<uint32_t>(ctx, items, (uint32_t)E, sbits, rbits, res->tile_alpha, colors, canvas, s)
             : composite_pieces<uint64_t>(ctx, items, (uint32_t)E, sbits, rbits, res->tile_alpha, colors, canvas, s);
    if (st != OCHRE_OK) return st;
    ctx->stats.n_launches = ctx->launches;
    collect_timings(ctx, s);
    return OCHRE_OK;
}

}  // namespace ochre

using namespace ochre;

extern "C" int ochre_gpu_composite(ochre_gpu_ctx* ctx, const ochre_result* res, uint32_t n_rasters,
                                   const uint8_t* colors, uint32_t w, uint32_t h, uint8_t* canvas, void* stream) {
    if (!ctx || !res || (n_rasters && !colors) || (w && h && !canvas)) return OCHRE_E_INVALID;
    if (w > 32768 || h > 32768 || n_rasters > MAX_RASTERS) return OCHRE_E_INVALID;
    if ((reinterpret_cast<uintptr_t>(canvas) & 3) || (reinterpret_cast<uintptr_t>(colors) & 3)) return OCHRE_E_INVALID;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return OCHRE_E_CUDA;
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : ctx->own_stream;
    const bool nothing = w == 0 || h == 0 || n_rasters == 0 || (uint64_t)res->n_tiles + res->n_spans == 0;
    if (!nothing && stream_captures(s)) return OCHRE_E_CUDA;
    ctx->epoch++;   // the sort reuses the chain's buffers
    ctx->prof_used = 0;
    ctx->launches = 0;
    if (nothing) return OCHRE_OK;
    const int st = composite(ctx, res, n_rasters, colors, w, h, canvas, s);
    ctx->test_spin_log2 = 0;   // (this call's)
    if (st != OCHRE_OK) ctx->scan_dirty = true;   // a scan may be counted that never ran
    return st;
}
