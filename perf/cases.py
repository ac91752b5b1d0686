"""The work a program asks of ochre_gb300, as measurable cases.

Every case goes through the package's public entry points on a context the
program keeps for all its batches (buffers grow once and are reused), with
another batch in hand from pass to pass, and on one stream.  Batches come from
the package's own seeded workload generators.  A result belongs to the context
only until its next call, so a program that keeps tiles on the device copies
them into arrays of its own; what it reads on the host it reads in place.
Kinds:

* ``glyphs``   text: many small rasters, from device buffers or, end to end,
  from host buffers to host results;
* ``path``     one vector path of a given number of segments, host to host:
  what a program that follows the reference's one-rasterizer-per-path API does;
* ``boxes``    closed paths of 16 cubics, about a thousand lines each;
* ``mix``      a map-like batch of paths of very uneven length on an 8192 px canvas;
* ``strokes``  stroked outlines;
* ``frame``    a drawing: rasterize a batch, then draw it onto an RGBA8 canvas
  (a page of text, or fills, text and strokes mixed);
* ``union``    one optimisation step on many overlapping shapes in one raster:
  coverage render, L2 loss, backward; by the eager calls or a captured graph;
* ``scenes``   the same step on a set of dense scenes.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from ochre_gb300 import Batch, DeviceBatch, GpuContext, concat, workloads

DEV = "cuda:0"


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a label: a word or two laid out and drawn at once; latency counts
        {"name": "label_host", "kind": "glyphs", "n": 33, "host": True, "pinned": False},
        # all text of a large map view or document, outlines kept on the device
        {"name": "glyphs_device", "kind": "glyphs", "n": 100_000, "host": False, "pinned": False},
        # the same volume handed over from pinned host memory, results read on the host
        {"name": "glyphs_host", "kind": "glyphs", "n": 50_000, "host": True, "pinned": True},
        # one path at a time, as the reference's API is used
        {"name": "path_host", "kind": "path", "segments": 61, "canvas": 1024},
        # a set of mid-sized shapes (icons, charts)
        {"name": "boxes_device", "kind": "boxes", "n": 1000},
        # a whole map layer: segment counts from 4 to 20,000
        {"name": "mix_device", "kind": "mix", "n": 20_000},
        # outlines, roads, rules
        {"name": "strokes_device", "kind": "strokes", "n": 20_000},
        # a page of a document viewer: shapes, text and strokes, composited
        {"name": "document_frame", "kind": "frame", "boxes": 24, "glyphs": 301, "strokes": 90, "canvas": 1024},
        # a screen of text, composited
        {"name": "text_frame", "kind": "frame", "boxes": 0, "glyphs": 20_000, "strokes": 0, "canvas": 2048},
        # one step of fitting a picture with overlapping shapes, eager calls
        {"name": "union_step", "kind": "union", "n": 256, "canvas": 1024, "graph": False},
        # the same step replayed from a captured graph, as a long fit does it
        {"name": "union_graph", "kind": "union", "n": 256, "canvas": 1024, "graph": True},
        # a training step over a set of dense scenes
        {"name": "scenes_step", "kind": "scenes", "n": 128, "canvas": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["glyphs", "glyphs", "path", "boxes", "mix", "strokes", "frame", "union", "scenes"])
    if kind == "glyphs":
        host = rng.random() < 0.5
        return {"kind": kind, "n": _log_int(rng, 20, 100_000), "host": host, "pinned": host and rng.random() < 0.5}
    if kind == "path":
        return {"kind": kind, "segments": _log_int(rng, 4, 2000), "canvas": rng.randrange(200, 4096)}
    if kind == "boxes":
        return {"kind": kind, "n": _log_int(rng, 10, 1000)}
    if kind == "mix":
        return {"kind": kind, "n": _log_int(rng, 100, 10_000)}
    if kind == "strokes":
        return {"kind": kind, "n": _log_int(rng, 50, 20_000)}
    if kind == "frame":
        text = rng.random() < 0.5
        return {"kind": kind, "boxes": 0 if text else _log_int(rng, 4, 60),
                "glyphs": _log_int(rng, 100, 20_000) if text else _log_int(rng, 50, 2000),
                "strokes": 0 if text else _log_int(rng, 10, 400), "canvas": rng.randrange(300, 2500)}
    if kind == "union":
        return {"kind": kind, "n": _log_int(rng, 8, 400), "canvas": rng.randrange(200, 1100),
                "graph": rng.random() < 0.5}
    return {"kind": kind, "n": _log_int(rng, 2, 128), "canvas": rng.randrange(130, 513)}


# Per raster of each generator, from the exact counts of its default
# configuration: input bytes (1 per verb, 4 per float, 24 per transform),
# tiles, spans, pixel cells crossed.
_GLYPH = (456.0, 21.2, 2.54, 276.0)
_BOX = (434.0, 874.0, 170.0, 10_086.0)
_MIX = (2_120.0, 3_518.0, 899.0, 34_578.0)
_STROKE = (236.0, 291.0, 4.1, 3_801.0)
_UNION = (851.0, 33.7, 3.9, 1_134.0)       # per shape of the union
_SCENE = (372_000.0, 3_008.0, 192.0, 221_373.0)
# One segment of an uneven path crosses about 345 pixel cells and touches 35 tiles.
_SEGMENT = (21.0, 35.0, 9.0, 345.0)
PER_RASTER = {"glyphs": _GLYPH, "boxes": _BOX, "mix": _MIX, "strokes": _STROKE, "path": _SEGMENT, "union": _UNION,
              "scenes": _SCENE}


# ---------------------------------------------------------------------------
# what a program has in hand
# ---------------------------------------------------------------------------
_contexts: dict = {}


def _context() -> GpuContext:
    """The program's context, kept for all its batches."""
    if "ctx" not in _contexts:
        _contexts["ctx"] = GpuContext(0)
    return _contexts["ctx"]


def _reordered(b: Batch, rng) -> Batch:
    """The batch's rasters in another order."""
    def gather(off, order):   # the ranges off[o] .. off[o + 1] - 1 of every o in order, one after the other
        n = np.diff(off)[order]
        new = np.concatenate([[0], np.cumsum(n)])
        return np.repeat(off[order] - new[:-1], n) + np.arange(new[-1]), new

    rasters = rng.permutation(b.n_rasters)
    fills, roff = (rasters, None) if b.raster_fill_off is None else gather(b.raster_fill_off.astype(np.int64), rasters)
    coff = b.fill_cmd_off.astype(np.int64)
    foff = np.concatenate([[0], np.cumsum(np.array([2, 2, 4, 6, 5, 0])[b.verbs])])[coff]
    cmds, new_coff = gather(coff, fills)
    floats, _ = gather(foff, fills)
    return Batch(b.verbs[cmds], b.pts[floats], new_coff.astype(np.uint32), b.fill_xf[fills], None,
                 None if roff is None else roff.astype(np.uint32), b.n_rasters)


def _batch(case, seed) -> Batch:
    """The case's input batch, from the case and the seed alone."""
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "glyphs":
        if case["host"]:   # one set of glyphs, laid out in the seed's order
            return _reordered(workloads.glyph_run(n_paths=case["n"]), rng)
        return workloads.glyph_run(n_paths=case["n"], seed=seed)
    if kind == "path":
        return workloads.uneven_mix(n_paths=1, seed=seed, canvas=float(case["canvas"]), median=float(case["segments"]),
                                    sigma=0.0)
    if kind == "boxes":
        return workloads.cubic_boxes(n_paths=case["n"], seed=seed)
    if kind == "mix":
        return workloads.uneven_mix(n_paths=case["n"], seed=seed)
    if kind == "strokes":
        return workloads.stroke_run(n_paths=case["n"], seed=seed)
    if kind == "frame":
        size = float(case["canvas"])
        parts = []
        if case["boxes"]:
            parts.append(workloads.cubic_boxes(n_paths=case["boxes"], seed=seed, canvas=size, box=size / 4, n_cubics=8))
        parts.append(workloads.glyph_run(n_paths=case["glyphs"], seed=seed, canvas=size))
        if case["strokes"]:
            parts.append(workloads.stroke_run(n_paths=case["strokes"], seed=seed, canvas=size))
        return concat(parts) if len(parts) > 1 else parts[0]
    if kind == "union":
        return workloads.diff_union(n_paths=case["n"], seed=seed, canvas=float(case["canvas"]))
    # one set of scenes, in the seed's order and shifted by the seed
    b = _reordered(workloads.diff_scenes(n_scenes=case["n"], size=float(case["canvas"])), rng)
    shift = rng.uniform(-4.0, 4.0, size=(b.n_rasters, 2)).astype(np.float32)
    b.fill_xf[:, 4:6] += np.repeat(shift, np.diff(b.raster_fill_off), axis=0)
    return b


def _target(n, size, seed):
    """Soft pictures to fit, [n, size, size] in [0, 1]."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    low = torch.rand((n, 1, 12, 12), generator=g, device=DEV)
    return torch.nn.functional.interpolate(low, size=(size, size), mode="bilinear", align_corners=False)[:, 0].contiguous()


def _pinned(batch: Batch) -> Batch:
    def pin(a):
        return None if a is None else torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()

    return Batch(pin(batch.verbs), pin(batch.pts), pin(batch.fill_cmd_off), pin(batch.fill_xf), pin(batch.fill_flags),
                 pin(batch.raster_fill_off), batch.n_rasters, pin(batch.fill_width))


def prepare(case, seed):
    kind = case["kind"]
    batch = _batch(case, seed)
    s = {"case": case, "ctx": _context(), "n_rasters": batch.n_rasters}
    if kind == "path":   # drawn path by path into the program's own tile list
        s["batch"] = batch
        t = 64 + 200 * case["segments"]
        s["own"] = {"tile_xy": np.zeros((t, 2), np.int16), "tile_alpha": np.zeros((t, 64), np.uint8),
                    "span_xy": np.zeros((t, 2), np.int16), "span_width": np.zeros(t, np.uint16),
                    "span_tile": np.zeros(t, np.uint32)}
        return s
    if kind == "glyphs" and case["host"]:
        s["batch"] = _pinned(batch) if case["pinned"] else batch
        return s
    s["dbatch"] = DeviceBatch(batch, 0)
    if kind == "frame":
        g = torch.Generator(device=DEV).manual_seed(seed)
        s["colors"] = torch.randint(0, 256, (batch.n_rasters, 4), generator=g, device=DEV, dtype=torch.uint8)
        s["canvas"] = torch.empty((case["canvas"], case["canvas"], 4), device=DEV, dtype=torch.uint8)
    elif kind in ("union", "scenes"):
        size = case["canvas"]
        target = _target(batch.n_rasters, size, seed)
        if case.get("graph"):
            s["graph"] = s["ctx"].graph_diff(s["dbatch"], size, size, target)
        else:
            s["target"] = target
            s["cov"] = torch.empty_like(target)
            s["dl_dcov"] = torch.empty_like(target)
    else:
        # the program's own tile list; uneven paths vary the most
        room = (1.2 + (40.0 if kind == "mix" else 8.0) / math.sqrt(case["n"])) * case["n"]
        t, n = (64 + int(room * c) for c in PER_RASTER[kind][1:3])
        z = dict(device=DEV)
        s["own"] = {"tile_xy": torch.zeros((t, 2), dtype=torch.int16, **z),
                    "tile_alpha": torch.zeros((t, 64), dtype=torch.uint8, **z),
                    "span_xy": torch.zeros((n, 2), dtype=torch.int16, **z),
                    "span_width": torch.zeros(n, dtype=torch.int16, **z),
                    "span_tile": torch.zeros(n, dtype=torch.int32, **z)}
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
class _DeviceArray:
    """A device pointer of a result as a tensor's storage."""

    def __init__(self, ptr, typestr, shape):
        self.__cuda_array_interface__ = {"data": (ptr, False), "typestr": typestr, "shape": shape, "strides": None,
                                         "version": 2}


def _tensor(ptr, typestr, *shape):
    return torch.as_tensor(_DeviceArray(ptr, typestr, shape), device=DEV)


def _copy_out(r, n_rasters, own):
    """A device result, its tiles and spans copied into the program's arrays."""
    t, n = r.n_tiles, r.n_spans
    own["tile_xy"][:t] = _tensor(r.tile_xy, "<i2", t, 2)
    own["tile_alpha"][:t] = _tensor(r.tile_alpha, "|u1", t, 64)
    if n:
        own["span_xy"][:n] = _tensor(r.span_xy, "<i2", n, 2)
        own["span_width"][:n] = _tensor(r.span_width, "<i2", n)
        own["span_tile"][:n] = _tensor(r.span_tile, "<i4", n)
    return {**own, "raster_tile_off": _tensor(r.raster_tile_off, "<i4", n_rasters + 1),
            "raster_span_off": _tensor(r.raster_span_off, "<i4", n_rasters + 1)}


def _array(ptr, dtype, *shape):
    count = int(np.prod(shape))
    if count == 0:
        return np.zeros(shape, dtype)
    raw = (ctypes.c_char * (count * np.dtype(dtype).itemsize)).from_address(ptr)
    return np.frombuffer(raw, dtype=dtype).reshape(shape)


def _host_result(r, n_rasters):
    t, n = r.n_tiles, r.n_spans
    return {"tile_xy": _array(r.tile_xy, np.int16, t, 2), "tile_alpha": _array(r.tile_alpha, np.uint8, t, 64),
            "span_xy": _array(r.span_xy, np.int16, n, 2), "span_width": _array(r.span_width, np.uint16, n),
            "span_tile": _array(r.span_tile, np.uint32, n),
            "raster_tile_off": _array(r.raster_tile_off, np.uint32, n_rasters + 1),
            "raster_span_off": _array(r.raster_span_off, np.uint32, n_rasters + 1)}


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind, n = case["kind"], state["n_rasters"]
    if "batch" in state:   # host buffers in, the context's host buffers out
        res = _host_result(ctx.rasterize_raw(state["batch"]), n)
        if "own" in state:
            for k, a in state["own"].items():
                a[:len(res[k])] = res[k]
            res.update(state["own"])
        return res
    db, stream = state["dbatch"], torch.cuda.current_stream().cuda_stream
    if kind == "frame":
        canvas = state["canvas"]
        canvas.fill_(255)
        r = ctx.rasterize_device(db, stream)
        return ctx.composite(r, n, state["colors"], canvas)
    if kind in ("union", "scenes"):
        if "graph" in state:
            g = state["graph"]
            g.launch(stream)
            return {"cov": g.cov, "loss": g.loss, "dl_dcov": g.dl_dcov, "dl_dpts": g.dl_dpts, "dl_dxf": g.dl_dxf}
        size = case["canvas"]
        cov = ctx.render_coverage(db, size, size, out=state["cov"])
        loss, dl_dcov = ctx.l2_loss(cov, state["target"], state["dl_dcov"])
        dl_dpts, dl_dxf = ctx.fill_backward(db, size, size, dl_dcov)
        return {"cov": cov, "loss": loss, "dl_dcov": dl_dcov, "dl_dpts": dl_dpts, "dl_dxf": dl_dxf}
    return _copy_out(ctx.rasterize_device(db, stream), n, state["own"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
CELL_FLOPS = 20.0   # one step of the walk and its area and height


def work(case):
    kind = case["kind"]
    if kind == "frame":
        # the tiles are an intermediate: inputs read, canvas written
        k = [(case["glyphs"], _GLYPH), (case["boxes"], _BOX), (case["strokes"], _STROKE)]
        return {"bytes": sum(n * c[0] for n, c in k) + 4.0 * case["canvas"] ** 2,
                "flops": CELL_FLOPS * sum(n * c[3] for n, c in k)}
    n, c = case["segments"] if kind == "path" else case["n"], PER_RASTER[kind]
    if kind in ("union", "scenes"):
        # inputs read, their gradients written; target read, coverage and dL/dcov written
        px = case["canvas"] ** 2 * (1 if kind == "union" else n)
        return {"bytes": 2.0 * n * c[0] + 12.0 * px, "flops": 3.0 * CELL_FLOPS * n * c[3]}
    return {"bytes": n * (c[0] + 68.0 * c[1] + 6.0 * c[2]), "flops": CELL_FLOPS * n * c[3]}


# ---------------------------------------------------------------------------
# the differentiable step in 64 bits
# ---------------------------------------------------------------------------
_TOL = np.float32(0.1)   # flattening tolerance, device pixels


def _line_counts(p, cubic):
    """Lines of every curve: the f32 step of the flattening rule and its
    serial f32 recurrence (t = min(t + dt, 1) until 1).  p: [n, 4, 2] f32."""
    f = np.float32

    def length(v):
        return np.sqrt(v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1])

    with np.errstate(all="ignore"):
        quad = np.sqrt((f(4.0) * _TOL) / length((p[:, 0] - f(2.0) * p[:, 1]) + p[:, 2]))
        a = (f(-1.0) * p[:, 0] + f(3.0) * p[:, 1]) - f(3.0) * p[:, 2] + p[:, 3]
        b = f(3.0) * ((p[:, 0] - f(2.0) * p[:, 1]) + p[:, 2])
        cub = np.sqrt((np.sqrt(f(8.0)) * _TOL) / np.maximum(length(b), length(a + b)))
    dt = np.where(cubic, cub, quad).astype(f)
    t = np.zeros_like(dt)
    n = np.zeros(len(dt), np.int64)
    while True:
        live = t < f(1.0)
        if not live.any():
            return n
        t = np.where(live, np.minimum(t + dt, f(1.0)), t)
        n += live


def exact(case, seed):
    """The differentiable step in 64-bit torch: curves to lines with the
    reference rule's line counts, exact area coverage of the lines, autograd
    back to points and transforms.  The other kinds give whole numbers."""
    if case["kind"] not in ("union", "scenes"):
        return None
    b = _batch(case, seed)
    W = H = case["canvas"]
    R = b.n_rasters
    target = _target(R, W, seed).double()
    D = dict(dtype=torch.float64, device=DEV)
    pts = torch.tensor(b.pts, **D, requires_grad=True)
    xf = torch.tensor(b.fill_xf, **D, requires_grad=True)
    # commands: every contour is Move, curves, Close
    nf = np.array([2, 2, 4, 6, 5, 0])[b.verbs]
    foff = np.concatenate([[0], np.cumsum(nf)])[:-1]
    cmd = np.arange(len(b.verbs))
    fill_of = np.searchsorted(b.fill_cmd_off, cmd, side="right") - 1
    raster_of_fill = np.searchsorted(b.raster_fill_off, np.arange(b.n_fills), side="right") - 1
    is_curve = (b.verbs == 2) | (b.verbs == 3)
    move = np.maximum.accumulate(np.where(b.verbs == 0, cmd, -1))
    cur = cmd[is_curve]
    cubic = b.verbs[cur] == 3
    end_off = foff + np.where(b.verbs == 3, 4, np.where(b.verbs == 2, 2, 0))
    # float offsets of a curve's points: start (end of the command before), controls, end
    at = np.stack([end_off[cur - 1], foff[cur], foff[cur] + 2, foff[cur] + np.where(cubic, 4, 2)], axis=1)
    # device-space f32 points for the line counts, in the transform's operation order
    p32 = np.stack([b.pts[at], b.pts[at + 1]], axis=2)
    m = b.fill_xf[fill_of[cur]][:, None, :]
    d32 = np.stack([(m[..., 0] * p32[..., 0] + m[..., 1] * p32[..., 1]) + m[..., 4],
                    (m[..., 2] * p32[..., 0] + m[..., 3] * p32[..., 1]) + m[..., 5]], axis=2)
    n = _line_counts(d32, cubic)

    def idx(a):
        return torch.as_tensor(np.ascontiguousarray(a), device=DEV)

    def device(a, fills):   # device-space points at float offsets a
        x, y, q = pts[a], pts[a + 1], xf[fills]
        return torch.stack([q[..., 0] * x + q[..., 1] * y + q[..., 4], q[..., 2] * x + q[..., 3] * y + q[..., 5]], -1)

    P = device(idx(at), idx(fill_of[cur])[:, None].expand(-1, 4))
    isc = idx(cubic)

    def length(v):
        return (v * v).sum(-1).sqrt()

    dq = P[:, 0] - 2 * P[:, 1] + P[:, 2]
    lq = length(torch.where(isc[:, None], torch.ones_like(dq), dq))
    lc = torch.maximum(length(3 * dq), length(2 * P[:, 0] - 3 * P[:, 1] + P[:, 3]))
    lc = torch.where(isc, lc, torch.ones_like(lc))
    dt = torch.where(isc, (math.sqrt(8.0) * 0.1 / lc).sqrt(), (0.4 / lq).sqrt())
    # line end points q_j = curve(min(j dt, 1)), the last one at 1
    cnt = idx(n)
    of = torch.repeat_interleave(torch.arange(len(n), device=DEV), cnt)
    first = torch.cumsum(cnt, 0) - cnt
    j = torch.arange(len(of), device=DEV) - first[of] + 1
    t = torch.where(j == cnt[of], torch.ones((), **D), torch.clamp(j * dt[of], max=1.0))[:, None]
    u = 1 - t
    C = P[of]
    q = torch.where(isc[of][:, None],
                    u ** 3 * C[:, 0] + 3 * u * u * t * C[:, 1] + 3 * u * t * t * C[:, 2] + t ** 3 * C[:, 3],
                    u * u * C[:, 0] + 2 * u * t * C[:, 1] + t * t * C[:, 2])
    start = torch.where((j == 1)[:, None], C[:, 0], torch.cat([q[:1], q[:-1]]))
    # the closing line of every contour, from its last end to its Move
    last_cmd = np.concatenate([cur[1:] != cur[:-1] + 1, [True]])
    lc_cmd = cur[last_cmd]
    mf = idx(fill_of[lc_cmd])
    A = torch.cat([start, device(idx(end_off[lc_cmd]), mf)])
    B = torch.cat([q, device(idx(foff[move[lc_cmd]]), mf)])
    ras = torch.cat([idx(raster_of_fill[fill_of[cur]])[of], idx(raster_of_fill[fill_of[lc_cmd]])])
    # cut every line at the pixel boundaries it crosses
    with torch.no_grad():
        lines = torch.arange(len(A), device=DEV)
        lo, hi = torch.minimum(A, B), torch.maximum(A, B)
        k0, k1 = torch.floor(lo).long() + 1, torch.ceil(hi).long() - 1
        cx, cy = [(k1[:, a] - k0[:, a] + 1).clamp(min=0) for a in (0, 1)]
        lx, ly = torch.repeat_interleave(lines, cx), torch.repeat_interleave(lines, cy)
        X = k0[lx, 0] + torch.arange(len(lx), device=DEV) - (torch.cumsum(cx, 0) - cx)[lx]
        Y = k0[ly, 1] + torch.arange(len(ly), device=DEV) - (torch.cumsum(cy, 0) - cy)[ly]
    sx = (X - A[lx, 0]) / (B[lx, 0] - A[lx, 0])
    sy = (Y - A[ly, 1]) / (B[ly, 1] - A[ly, 1])
    line = torch.cat([lines, lx, ly, lines])
    s = torch.cat([torch.zeros(len(A), **D), sx, sy, torch.ones(len(A), **D)])
    with torch.no_grad():
        rank = torch.cat([torch.zeros(len(A), **D), 0.25 + 0.5 * sx, 0.25 + 0.5 * sy, 0.9 * torch.ones(len(A), **D)])
        order = torch.argsort(line.double() + rank)
    line, s = line[order], s[order]
    pt = A[line] + s[:, None] * (B - A)[line]
    keep = line[1:] == line[:-1]
    p0, p1, rr = pt[:-1][keep], pt[1:][keep], ras[line[:-1][keep]]
    with torch.no_grad():
        cell = torch.floor(0.5 * (p0 + p1)).long()
        x, y = cell[:, 0], cell[:, 1]
        inside = (y >= 0) & (y < H) & (x < W)
    p0, p1, rr, x, y = p0[inside], p1[inside], rr[inside], x[inside], y[inside]
    h = p1[:, 1] - p0[:, 1]
    area = h * (x + 1 - 0.5 * (p0[:, 0] + p1[:, 0]))
    row = (rr * H + y) * (W + 1)
    hsum = torch.zeros(R * H * (W + 1), **D).index_add(0, row + x.clamp(min=-1) + 1, h)
    on = x >= 0
    asum = torch.zeros(R * H * (W + 1), **D).index_add(0, (row + x)[on], area[on])
    S = torch.cumsum(hsum.view(R, H, W + 1), 2)[..., :W] + asum.view(R, H, W + 1)[..., :W]
    mag = S.abs()
    soft = (mag < 1 - 1e-9) & (mag > 1e-9)
    cov = torch.where(soft, mag, mag.detach().clamp(max=1.0))
    diff = cov - target
    loss = (diff * diff).sum()
    loss.backward()
    return {"cov": cov.detach(), "loss": loss.detach().reshape(1), "dl_dcov": 2 * diff.detach(), "dl_dpts": pts.grad,
            "dl_dxf": xf.grad}
