"""The work that programs on this framework have it do, as timed cases.

Every case goes through a public entry point of skity_gb300.canvas: the
canvas a program draws on and flushes, draw streams rendered in one call,
batches kept on the device, the serving loop, and single paths drawn onto a
canvas that already lives in device memory.  Path counts, verb mixes, sizes
and paints are those of the repository's workloads (skity_gb300.scene:
config1 .. config4, the serving pool of bench.py, the imported picture) and
the shapes that pages and illustrations are made of; the contents are drawn
from the seed.

The outputs are RGBA8 pixels, whole numbers, so no tolerance applies to them.
"""
import math

import numpy as np
import torch

from skity_gb300 import canvas as C
from skity_gb300 import scene as S

WHITE = 0xFFFFFFFF
_STATE = {}


def _context():
    """The context a program keeps for all of its rendering."""
    if "ctx" not in _STATE:
        _STATE["ctx"] = C.Context(0)
    return _STATE["ctx"]


def _server():
    """The serving loop a program keeps running."""
    if "server" not in _STATE:
        _STATE["server"] = C.Server(0)
    return _STATE["server"]


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # an immediate-mode caller that puts one path onto a device-resident frame
        {"name": "device_path", "kind": "device", "width": 256, "height": 256, "paths": 1,
         "verbs": 24},
        # an icon redrawn on its own small canvas: latency and launches
        {"name": "icon_canvas", "kind": "page", "width": 48, "height": 48, "draws": 6},
        # a phone page: cards, text outlines, ovals, gradients, shadows, clip rects
        {"name": "page_canvas", "kind": "page", "width": 412, "height": 915, "draws": 160},
        # one canvas of random fills (config1)
        {"name": "fills_512", "kind": "fills", "canvases": 1, "side_lo": 512, "side_hi": 512,
         "paths_lo": 1000, "paths_hi": 1000, "verbs": 32, "resident": False},
        # an illustration: few long smooth outlines, half of them stroked, under a scale
        {"name": "picture", "kind": "picture", "width": 2560, "height": 1920, "draws": 305,
         "nodes": 240},
        # every gradient kind, blend modes, colour filters, image shaders and layers
        {"name": "effects", "kind": "effects", "width": 1204, "height": 803, "draws": 400},
        # draws under nested path clips
        {"name": "path_clips", "kind": "clips", "width": 901, "height": 703, "draws": 240,
         "states": 24},
        # a glyph-dense sheet, a tenth of the outlines blurred (config4)
        {"name": "glyphs_4096", "kind": "glyphs", "width": 4096, "height": 4096,
         "draws": 100000},
        # one large scene of fills, strokes and gradients (config2)
        {"name": "scene_2048", "kind": "scene", "width": 2048, "height": 2048, "draws": 20000,
         "verbs": 64},
        # many uneven canvases kept on the device and rendered again (config3)
        {"name": "batch_256", "kind": "fills", "canvases": 256, "side_lo": 64, "side_hi": 1024,
         "paths_lo": 50, "paths_hi": 2000, "verbs": 32, "resident": True},
        # uneven canvases from host streams to host pixels in one call
        {"name": "streams_61", "kind": "fills", "canvases": 61, "side_lo": 64, "side_hi": 1024,
         "paths_lo": 50, "paths_hi": 2000, "verbs": 32, "resident": False},
        # a burst of requests to the serving loop
        {"name": "serve_24", "kind": "serve", "canvases": 24, "side_lo": 128, "side_hi": 2048,
         "paths_lo": 10, "paths_hi": 5000, "verbs": 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    # canvases with gradients are a multiple of 4 px wide
    kind = rng.choice(["device", "page", "page", "fills", "fills", "fills", "picture", "effects",
                       "clips", "glyphs", "scene", "scene", "serve"])
    if kind == "device":
        return {"kind": kind, "width": _log(rng, 32, 2048), "height": _log(rng, 32, 2048),
                "paths": _log(rng, 1, 16), "verbs": _log(rng, 3, 64)}
    if kind == "page":
        return {"kind": kind, "width": 4 * _log(rng, 6, 360), "height": _log(rng, 24, 1440),
                "draws": _log(rng, 2, 600)}
    if kind == "fills":
        n = _log(rng, 1, 128)
        lo = _log(rng, 64, 512)
        return {"kind": kind, "canvases": n, "side_lo": lo, "side_hi": lo + _log(rng, 1, 512),
                "paths_lo": 50, "paths_hi": _log(rng, 100, 2000), "verbs": rng.randint(6, 32),
                "resident": rng.random() < 0.5}
    if kind == "picture":
        return {"kind": kind, "width": _log(rng, 300, 2560), "height": _log(rng, 300, 2560),
                "draws": _log(rng, 20, 600), "nodes": _log(rng, 12, 300)}
    if kind == "effects":
        return {"kind": kind, "width": 4 * _log(rng, 25, 350), "height": _log(rng, 100, 1400),
                "draws": _log(rng, 20, 500)}
    if kind == "clips":
        return {"kind": kind, "width": _log(rng, 100, 1400), "height": _log(rng, 100, 1400),
                "draws": _log(rng, 20, 400), "states": rng.randint(1, 32)}
    if kind == "glyphs":
        return {"kind": kind, "width": _log(rng, 256, 4096), "height": _log(rng, 256, 4096),
                "draws": _log(rng, 100, 60000)}
    if kind == "scene":
        return {"kind": kind, "width": 4 * _log(rng, 64, 512), "height": _log(rng, 256, 2048),
                "draws": _log(rng, 50, 6000), "verbs": rng.randint(8, 64)}
    return {"kind": kind, "canvases": _log(rng, 1, 24), "side_lo": 128,
            "side_hi": _log(rng, 256, 2048), "paths_lo": 10, "paths_hi": _log(rng, 100, 5000),
            "verbs": 32}


# ---------------------------------------------------------------------------
# scenes, built a whole array at a time
# ---------------------------------------------------------------------------
def _scene(width, height, verbs, points, nverb, npoint, paints, **more):
    offs = lambda n: np.concatenate([[0], np.cumsum(n)]).astype(np.uint32)  # noqa: E731
    return S.Scene(width, height, (1.0, 1.0, 1.0, 1.0), verbs, points.astype(np.float32),
                   np.zeros(0, np.float32), offs(nverb), offs(npoint),
                   np.zeros(len(paints) + 1, np.uint32), paints, **more)


def _paints(n, rng):
    p = np.zeros(n, S.PAINT_DTYPE)
    p[:] = S.default_paint()
    c = np.concatenate([rng.integers(0, 256, (n, 3)).astype(np.float32) / np.float32(255.0),
                        rng.uniform(0.3, 1.0, (n, 1)).astype(np.float32)], 1)
    p["fill_color"] = c
    p["stroke_color"] = c
    return p


def _random_paths(rng, width, height, n, verbs_hi, margin=0.0):
    """Closed paths of 3 .. verbs_hi verbs (half lines, a quarter each quads
    and cubics), control points uniform over the canvas and its margin."""
    count = rng.integers(3, max(verbs_hi, 3) + 1, n)
    nverb = count + 2
    end = np.cumsum(nverb)
    total = int(end[-1])
    r = rng.random(total)
    verbs = np.where(r < 0.5, S.LINE, np.where(r < 0.75, S.QUAD, S.CUBIC)).astype(np.uint8)
    verbs[end - nverb] = S.MOVE
    verbs[end - 1] = S.CLOSE
    per = np.array([S.VERB_POINTS[v] for v in range(6)])[verbs]
    npoint = np.add.reduceat(per, end - nverb)
    points = rng.uniform((-margin, -margin), (width + margin, height + margin),
                         (int(per.sum()), 2))
    return verbs, points.astype(np.float32), nverb, npoint


def fills_scene(seed, width, height, n, verbs_hi):
    """config1 at any size: nonzero fills in solid colours."""
    rng = np.random.default_rng(seed)
    verbs, points, nverb, npoint = _random_paths(rng, width, height, n, verbs_hi)
    return _scene(width, height, verbs, points, nverb, npoint, _paints(n, rng))


def _gradients(rng, kinds, boxes):
    """One gradient record per draw of `kinds` that is not 0, its geometry in
    the draw's box, 2 to 8 stops with offsets."""
    at = np.nonzero(kinds)[0]
    g = np.zeros(len(at), S.GRADIENT_DTYPE)
    stops = rng.integers(2, 9, len(at))
    start = np.concatenate([[0], np.cumsum(stops)])
    lo, hi = boxes[at, 0:2], boxes[at, 2:4]
    g["type"], g["stop_count"], g["stop_start"], g["has_offsets"] = kinds[at], stops, start[:-1], 1
    g["p0"] = lo + rng.random((len(at), 2)) * (hi - lo)
    g["p1"] = lo + rng.random((len(at), 2)) * (hi - lo)
    half = 0.5 * np.hypot(*(hi - lo).T)
    radial = g["type"] == S.GRAD_RADIAL
    g["radius"][:, 0] = np.where(radial, rng.uniform(0.25, 1.0, len(at)) * half, 0)
    g["p1"][radial] = 0
    colors = np.round(rng.uniform(0, 255, (int(start[-1]), 4))).astype(np.float32) / np.float32(255)
    offsets = np.zeros(int(start[-1]), np.float32)
    for i in range(len(at)):
        o = np.sort(rng.random(int(stops[i])).astype(np.float32))
        o[0], o[-1] = 0.0, 1.0
        offsets[start[i]:start[i + 1]] = o
    index = np.full(len(kinds), -1, np.int32)
    index[at] = np.arange(len(at))
    return index, g, colors, offsets


def paths_scene(seed, width, height, n, verbs_hi):
    """config2 at any size: 30% even-odd, half solid, a quarter each linear
    and radial gradients, a fifth stroked 1 to 8 px wide."""
    rng = np.random.default_rng(seed)
    verbs, points, nverb, npoint = _random_paths(rng, width, height, n, verbs_hi, 64.0)
    p = _paints(n, rng)
    p["fill_type"] = rng.random(n) < 0.3
    stroked = rng.random(n) < 0.2
    p["style"][stroked] = S.STROKE
    p["stroke_width"] = np.where(stroked, rng.uniform(1, 8, n), 1)
    p["cap"] = np.where(stroked, rng.integers(0, 3, n), 0)
    p["join"] = np.where(stroked, rng.integers(0, 3, n), 0)
    first = np.concatenate([[0], np.cumsum(npoint)[:-1]])
    boxes = np.concatenate([np.minimum.reduceat(points, first), np.maximum.reduceat(points, first)], 1)
    r = rng.random(n)
    kinds = np.where(r < 0.5, 0, np.where(r < 0.75, S.GRAD_LINEAR, S.GRAD_RADIAL))
    p["gradient"], g, colors, offsets = _gradients(rng, kinds, boxes)
    return _scene(width, height, verbs, points, nverb, npoint, p, gradients=g, stop_colors=colors,
                  stop_offsets=offsets)


def glyphs_scene(seed, width, height, n):
    """config4 at any size: closed cubic outlines of 8 to 40 verbs in 1 to 3
    contours in boxes of 8 to 48 px, even-odd, a tenth of them blurred with a
    sigma of 2 to 20 px."""
    rng = np.random.default_rng(seed)
    contours = rng.integers(1, 4, n)
    per = np.maximum(3, rng.integers(8, 41, n) // contours)
    box = rng.uniform(8, 48, n)
    cx, cy = rng.random(n) * (width - box) + box / 2, rng.random(n) * (height - box) + box / 2
    # one entry per contour
    glyph = np.repeat(np.arange(n), contours)
    level = np.concatenate([np.arange(k) for k in (1, 2, 3)])
    level = level[np.repeat(np.array([0, 1, 3])[contours - 1], contours) +
                  (np.arange(len(glyph)) - np.repeat(np.cumsum(contours) - contours, contours))]
    segs = per[glyph]
    # one entry per node: `segs` nodes in each contour, the first one again at the end
    cont = np.repeat(np.arange(len(glyph)), segs)
    k = np.arange(len(cont)) - np.repeat(np.cumsum(segs) - segs, segs)
    last = k == segs[cont] - 1
    step = np.where(level[cont] == 0, 1.0, -1.0) * 2 * np.pi / segs[cont]
    rad = box[glyph[cont]] * 0.5 * np.array([1.0, 0.55, 0.3])[level[cont]]
    rr = rng.uniform(0.75, 1.0, len(cont))
    nxt = np.arange(len(cont)) + 1
    nxt[last] = np.repeat(np.cumsum(segs) - segs, 1)
    a0, a1 = step * k, step * np.where(last, 0, k + 1)
    ox, oy = cx[glyph[cont]], cy[glyph[cont]]
    r0, r1 = rad * rr, rad * rr[nxt]
    k1 = rad * rng.uniform(0.85, 1.15, len(cont)) * (2 * rr + rr[nxt]) / 3
    k2 = rad * rng.uniform(0.85, 1.15, len(cont)) * (rr + 2 * rr[nxt]) / 3
    t1, t2 = step * (k + 1 / 3), step * (k + 2 / 3)
    start = np.stack([ox + r0 * np.cos(a0), oy + r0 * np.sin(a0)], 1)
    cubic = np.stack([ox + k1 * np.cos(t1), oy + k1 * np.sin(t1), ox + k2 * np.cos(t2),
                      oy + k2 * np.sin(t2), ox + r1 * np.cos(a1), oy + r1 * np.sin(a1)],
                     1).reshape(-1, 3, 2)
    # contour c: MOVE, its cubics, CLOSE
    vstart = np.cumsum(segs + 2) - (segs + 2)
    verbs = np.full(int((segs + 2).sum()), S.CUBIC, np.uint8)
    verbs[vstart] = S.MOVE
    verbs[vstart + segs + 1] = S.CLOSE
    pstart = np.cumsum(3 * segs + 1) - (3 * segs + 1)
    points = np.empty((int((3 * segs + 1).sum()), 2))
    points[pstart] = start[k == 0]
    at = pstart[cont] + 1 + 3 * k
    for j in range(3):
        points[at + j] = cubic[:, j]
    p = _paints(n, rng)
    p["fill_type"] = S.EVEN_ODD
    blurred = rng.random(n) < 0.1
    p["blur_style"] = blurred
    p["blur_radius"] = np.where(blurred, (rng.uniform(2, 20, n) - 0.5) / 0.57735, 0)
    by_glyph = lambda v: np.add.reduceat(v, np.cumsum(contours) - contours)  # noqa: E731
    return _scene(width, height, verbs, points, by_glyph(segs + 2), by_glyph(3 * segs + 1), p)


def picture_scene(seed, width, height, n, nodes_hi):
    """An illustration: smooth closed outlines (Catmull-Rom through a wobbly
    ring of 4 .. nodes_hi nodes), big and small, half filled and half stroked
    0.5 to 6 px wide, drawn in a 2/3 size and scaled up by the canvas."""
    rng = np.random.default_rng(seed)
    scale = 1.5
    w, h = width / scale, height / scale
    verbs, points = [], []
    for _ in range(n):
        m = int(round(math.exp(rng.uniform(math.log(4), math.log(max(nodes_hi, 4))))))
        a = np.arange(m) * (2 * np.pi / m)
        size = math.exp(rng.uniform(math.log(4.0), math.log(0.45 * min(w, h))))
        r = size * rng.uniform(0.6, 1.0, m)
        q = np.stack([r * np.cos(a), r * rng.uniform(0.3, 1.0) * np.sin(a)], 1)
        q += rng.uniform((0, 0), (w, h))
        tan = (np.roll(q, -1, 0) - np.roll(q, 1, 0)) / 6
        seg = np.stack([q + tan, np.roll(q - tan, -1, 0), np.roll(q, -1, 0)], 1).reshape(-1, 2)
        points.append(np.concatenate([q[:1], seg]))
        verbs.append(np.concatenate([[S.MOVE], np.full(m, S.CUBIC), [S.CLOSE]]).astype(np.uint8))
    p = _paints(n, rng)
    stroked = rng.random(n) < 0.5
    p["style"][stroked] = S.STROKE
    p["stroke_width"] = np.where(stroked, rng.uniform(0.5, 6, n), 1)
    p["cap"] = np.where(stroked, rng.integers(0, 3, n), 0)
    p["join"] = np.where(stroked, rng.integers(0, 3, n), 0)
    matrix = np.tile(np.array([scale, 0, 0, 0, scale, 0], np.float32), (n, 1))
    return _scene(width, height, np.concatenate(verbs), np.concatenate(points),
                  [len(v) for v in verbs], [len(q) for q in points], p, matrices=matrix)


def _blob(rng, width, height, verbs_hi=12):
    """One random closed path around a point of the canvas."""
    n = int(rng.integers(3, verbs_hi + 1))
    kinds = rng.choice([S.LINE, S.QUAD, S.CUBIC], n)
    m = 1 + int(sum(S.VERB_POINTS[int(v)] for v in kinds))
    reach = rng.uniform(0.05, 0.5) * min(width, height)
    pts = rng.uniform((0, 0), (width, height)) + rng.uniform(-reach, reach, (m, 2))
    return [S.MOVE] + [int(v) for v in kinds] + [S.CLOSE], pts.astype(np.float32)


def effects_scene(seed, width, height, n):
    """Paints past solid and gradient fills: sweep and two-point conical
    gradients, every blend mode, colour filters, image shaders; a run of the
    draws inside a layer."""
    rng = np.random.default_rng(seed)
    b = S.SceneBuilder(width, height)
    images = [b.add_image(rng.integers(0, 256, (int(rng.integers(4, 65)), int(rng.integers(4, 65)), 4),
                                       dtype=np.uint8), S.ALPHA_UNPREMUL) for _ in range(4)]
    first, last = n // 3, n // 2
    clip = None
    for i in range(n):
        if i == first:
            clip = b.save_layer((0.1 * width, 0.1 * height, 0.8 * width, 0.9 * height), 0.7)
        if i == last and clip is not None:
            b.restore_layer()
            clip = None
        verbs, pts = _blob(rng, width, height)
        p = _paints(1, rng)[0]
        p["fill_type"] = int(rng.random() < 0.3)
        if rng.random() < 0.2:
            p["style"], p["stroke_width"] = S.STROKE, rng.uniform(1, 8)
        kind, shader, cf = rng.integers(0, 6), None, None
        cols = rng.uniform(0, 1, (int(rng.integers(2, 6)), 4)).astype(np.float32)
        q0, q1 = (tuple(float(v) for v in rng.uniform((0, 0), (width, height))) for _ in range(2))
        tile = int(rng.integers(0, 4))
        sh = None
        if kind == 1:
            a = float(rng.uniform(-180, 180))
            sh = C.Shader.MakeSweep(q0[0], q0[1], a, a + float(rng.uniform(90, 400)), cols, None,
                                    len(cols), tile)
        elif kind == 2:
            sh = C.Shader.MakeTwoPointConical(q0, float(rng.uniform(5, 30)), q1,
                                              float(rng.uniform(40, 200)), cols, None, len(cols), tile)
        elif kind == 3:
            p["blend"] = int(rng.integers(0, 29))
        elif kind == 4:
            cf = S.filter_record(S.FILTER_MATRIX, matrix=rng.uniform(-0.6, 1.2, 20))
        elif kind == 5:
            z = float(rng.uniform(0.5, 6))
            shader = S.image_shader(images[int(rng.integers(0, 4))], int(rng.integers(0, 2)), tile, tile,
                                    (z, 0.0, q0[0], 0.0, z, q0[1]))
        if sh is not None:
            p["gradient"] = b.add_gradient(sh.kind, sh.p0, sh.p1, sh.radius, sh.colors, sh.pos, sh.tile)
        b.draw_path(verbs, pts, p, clip=clip, color_filter=cf, image_shader=shader)
    return b.build()


def clips_scene(seed, width, height, n, states):
    """Draws under path clips: clips set one inside another in groups of up
    to three under a Save, with draws between them."""
    rng = np.random.default_rng(seed)
    b = S.SceneBuilder(width, height)
    every, depth = max(1, n // max(states, 1)), 0
    bounds = S.NO_CLIP
    for i in range(n):
        if i % every == 0:
            if depth == 3 or depth == 0:
                if depth:
                    b.restore()
                b.save()
                depth, bounds = 0, S.NO_CLIP
            reach = np.array([width, height]) * rng.uniform(0.2, 0.6)
            at = rng.uniform((0, 0), (width, height))
            a = np.sort(rng.uniform(0, 2 * np.pi, 9))
            pts = (at + reach * np.stack([np.cos(a), np.sin(a)], 1)).astype(np.float32)
            verbs = [S.MOVE] + [S.QUAD] * 4 + [S.CLOSE]
            op = S.CLIP_INTERSECT if depth == 0 or rng.random() < 0.5 else S.CLIP_DIFFERENCE
            b.clip_path(verbs, pts, op, bounds=bounds)
            if op == S.CLIP_INTERSECT:
                bounds = S.map_clip(bounds, (*pts.min(0), *pts.max(0)))
            depth += 1
        verbs, pts = _blob(rng, width, height)
        p = _paints(1, rng)[0]
        if rng.random() < 0.2:
            p["style"], p["stroke_width"] = S.STROKE, rng.uniform(1, 8)
        b.draw_path(verbs, pts, p, clip=bounds)
    return b.build()


# ---------------------------------------------------------------------------
# pages: calls on a canvas
# ---------------------------------------------------------------------------
def _round_rect(l, t, r, b, rad):
    w = 0.70710677
    return (C.Path().MoveTo(l + rad, t).LineTo(r - rad, t).ConicTo(r, t, r, t + rad, w)
            .LineTo(r, b - rad).ConicTo(r, b, r - rad, b, w).LineTo(l + rad, b)
            .ConicTo(l, b, l, b - rad, w).LineTo(l, t + rad).ConicTo(l, t, l + rad, t, w).Close())


def _glyph(rng, x, y, size):
    """An outline with a counter, 4 cubics each way."""
    p = C.Path().SetFillType(C.PathFillType.kEvenOdd)
    for s in (0.5, 0.27):
        a = np.arange(5) * (np.pi / 2) * (1 if s == 0.5 else -1)
        r = size * s * rng.uniform(0.8, 1.0, 5)
        r[4] = r[0]
        q = np.stack([x + r * np.cos(a), y + r * np.sin(a)], 1)
        d = np.stack([-np.sin(a), np.cos(a)], 1) * (r * 0.55)[:, None] * (1 if s == 0.5 else -1)
        p.MoveTo(*q[0])
        for i in range(4):
            p.CubicTo(*(q[i] + d[i]), *(q[i + 1] - d[i + 1]), *q[i + 1])
        p.Close()
    return p


def _page_calls(seed, width, height, n):
    """(clip rect or None, translation, path, paint) per draw."""
    rng = np.random.default_rng(seed)
    small = min(width, height)
    calls = []
    for i in range(n):
        x, y = rng.uniform(0, width), rng.uniform(0, height)
        e = rng.uniform(0.1, 0.5) * small
        kind = rng.random()
        paint = C.Paint().SetColor(C.ColorSetARGB(int(rng.integers(80, 256)), *(int(v) for v in rng.integers(0, 256, 3))))
        if kind < 0.5:
            path = _glyph(rng, x, y, max(4.0, 0.04 * small))
        elif kind < 0.65:
            path = _round_rect(x - e, y - e / 2, x + e, y + e / 2, e / 6)
        elif kind < 0.75:
            path = C.Path().AddRect(x - e, y - 0.5, x + e, y + 0.5)
        elif kind < 0.85:
            path = C.Path().AddOvalRRect(x - e / 3, y - e / 3, x + e / 3, y + e / 3)
        elif kind < 0.95:
            path = C.Path().MoveTo(x, y).CubicTo(x + e, y - e, x - e, y + e, x + e, y + e)
            paint.SetStyle(C.Style.kStroke_Style).SetStrokeWidth(float(rng.uniform(0.5, 4)))
        else:
            path = _round_rect(x - e, y - e / 2, x + e, y + e / 2, e / 8)
            paint.SetMaskFilter(C.MaskFilter.MakeBlur(C.BlurStyle.kNormal, float(rng.uniform(1, 12))))
        if 0.5 <= kind < 0.65 and rng.random() < 0.4:
            cols = rng.uniform(0, 1, (3, 4)).astype(np.float32)
            paint.SetShader(C.Shader.MakeLinear([(x - e, y), (x + e, y)], cols, [0.0, 0.4, 1.0], 3))
        clip = None
        if kind < 0.95 and rng.random() < 0.15:
            clip = (0.1 * width, 0.1 * height, 0.9 * width, 0.9 * height)
        calls.append((clip, (float(int(rng.integers(-3, 4))), 0.0), path, paint))
    return calls


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def _spread(case):
    """(width, height, paths) of each canvas of a case: log-uniform over its
    ranges by a low-discrepancy sequence, the same for every seed."""
    def pick(i, a, lo, hi):
        f = (0.5 + (i + 1) * a) % 1.0 if case["canvases"] > 1 else 0.5
        return max(1, int(round(math.exp(math.log(lo) + f * (math.log(hi) - math.log(lo))))))
    return [(pick(i, 0.8191725134, case["side_lo"], case["side_hi"]),
             pick(i, 0.6710436067, case["side_lo"], case["side_hi"]),
             pick(i, 0.5497004779, case["paths_lo"], case["paths_hi"]))
            for i in range(case["canvases"])]


def _outputs(sizes):
    """Page-locked pixels of all canvases, and each canvas's rows in them."""
    flat = torch.empty(sum(w * h * 4 for w, h in sizes), dtype=torch.uint8, pin_memory=True)
    a, rows, at = flat.numpy(), [], 0
    for w, h in sizes:
        rows.append(a[at:at + w * h * 4].reshape(h, w, 4))
        at += w * h * 4
    return flat, rows


def prepare(case, seed):
    kind = case["kind"]
    seed = int(seed) * 1000003 + 17
    if kind == "device":
        sc = fills_scene(seed, case["width"], case["height"], case["paths"], case["verbs"])
        pixels = torch.zeros((case["height"], case["width"], 4), dtype=torch.uint8, device="cuda")
        canvas = C.DeviceCanvas(pixels.data_ptr(), case["width"], case["height"],
                                stream=torch.cuda.current_stream().cuda_stream)
        return {"kind": kind, "scene": sc, "pixels": pixels, "canvas": canvas}
    if kind == "page":
        bitmap = np.zeros((case["height"], case["width"], 4), np.uint8)
        return {"kind": kind, "bitmap": bitmap, "canvas": C.Canvas.MakeCUDACanvas(_context(), bitmap),
                "calls": _page_calls(seed, case["width"], case["height"], case["draws"])}
    if kind in ("fills", "serve"):
        scenes = [fills_scene(seed + 7919 * i, w, h, n, case["verbs"])
                  for i, (w, h, n) in enumerate(_spread(case))]
        if kind == "serve":
            return {"kind": kind, "server": _server(), "scenes": scenes}
    else:
        w, h, n = case["width"], case["height"], case["draws"]
        scenes = [glyphs_scene(seed, w, h, n) if kind == "glyphs" else
                  paths_scene(seed, w, h, n, case["verbs"]) if kind == "scene" else
                  picture_scene(seed, w, h, n, case["nodes"]) if kind == "picture" else
                  effects_scene(seed, w, h, n) if kind == "effects" else
                  clips_scene(seed, w, h, n, case["states"])]
    flat, rows = _outputs([(s.width, s.height) for s in scenes])
    if case.get("resident"):
        return {"kind": "batch", "batch": C.Batch(_context(), scenes), "flat": flat, "rows": rows}
    return {"kind": "streams", "ctx": _context(), "scenes": scenes, "flat": flat, "rows": rows}


def run(state):
    kind = state["kind"]
    if kind == "streams":
        state["ctx"].render_streams(state["scenes"], out=state["rows"])
        return state["flat"]
    if kind == "batch":
        state["batch"].render()
        for i, rows in enumerate(state["rows"]):
            state["batch"].read(i, rows)
        return state["flat"]
    if kind == "serve":
        tickets = [state["server"].submit(scene=s) for s in state["scenes"]]
        return [state["server"].wait(t, 600000)[0] for t in tickets]
    if kind == "device":
        state["pixels"].fill_(255)
        state["canvas"].draw_scene(state["scene"])
        return state["pixels"]
    canvas = state["canvas"]
    canvas.Clear(WHITE)
    for clip, move, path, paint in state["calls"]:
        canvas.Save()
        canvas.Translate(*move)
        if clip is not None:
            canvas.ClipRect(*clip)
        canvas.DrawPath(path, paint)
        canvas.Restore()
    canvas.Flush()
    return state["bitmap"]


def work(case):
    """Bytes of the draws (verbs, points, paints) read once and of the pixels
    written once.  The blending's arithmetic depends on the coverage, which
    the sizes alone do not give, so it is not counted."""
    kind = case["kind"]
    record = 80 + 12  # paint and offsets
    if kind in ("fills", "serve"):
        spread = _spread(case)
        mean = (3 + max(case["verbs"], 3)) / 2  # 1 byte and 1.75 points of 8 bytes a verb
        return {"bytes": sum(4 * w * h + n * (record + 10 + 15 * mean) for w, h, n in spread), "flops": 0}
    n = case["paths"] if kind == "device" else case["draws"]
    points = {"device": 1.75 * (3 + max(case.get("verbs", 3), 3)) / 2, "page": 18, "glyphs": 72,
              "scene": 1.75 * (3 + case.get("verbs", 3)) / 2,
              "picture": 3 * (max(case.get("nodes", 4), 5) - 4) / math.log(max(case.get("nodes", 4), 5) / 4),
              "effects": 15, "clips": 15}[kind]
    return {"bytes": 4 * case["width"] * case["height"] + n * (record + 10 + 8.5 * points), "flops": 0}


def exact(case, seed):
    """Pixels are whole numbers, compared for equality: no value in 64 bits."""
    return None
