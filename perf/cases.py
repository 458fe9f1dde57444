"""Performance cases: the calls a program makes of this library, through its public API.

Each case is one pass over images that live on the GPU (torch tensors behind
``Image.wrap``, as a program that shares pixels with PyTorch holds them, and
the library's own images for work layers).  The kinds:

fill    one fillPath call, blocking, as pixie's own callers make it: an icon
        (the heart of pixie's tests) up to a poster-sized path of many cubics
stroke  one strokePath call: a chart line, a signature, dashed or not
scene   a retained scene (recorded once, as a UI or an SVG viewer keeps it)
        redrawn on a cleared canvas
serve   a handful of render jobs through the batching server, canvases
        downloaded: a thumbnail service
glyphs  a text run: ``whole`` builds the mask batch from outlines each pass
        (a label that changes), otherwise the batch is kept, re-rendered and
        composited (a page of text)
stack   artboards of layers composited with every blend and mask mode,
        enqueued without waiting (the library's non-blocking mode)
layers  frosted-glass panels and drop shadows: a source copied to a work
        layer, blurred or turned into a shadow, composited onto a canvas
canvas  a gradient background, a shape with a gradient paint, and rotated,
        scaled sprites: draw with a Mat3

Every output is bytes: the same calls on the same inputs give the same bytes.
"""
import math

import numpy as np
import torch

import pixie_gb300 as px
from pixie_gb300 import workloads as wl

PLAIN_MODES = [m for m in range(20) if m not in (16, 17, 18, 19)]


def listed():
    return [
        # the smallest call: one icon (pixie's test heart at its own size)
        {"name": "fill_icon", "kind": "fill", "w": 100, "h": 100, "cubics": 0, "blend": 0, "evenodd": False,
         "alpha": 1.0},
        # the benchmark's plain fill: one 512 x 512 image, one closed path of 64 cubics
        {"name": "fill_512", "kind": "fill", "w": 512, "h": 512, "cubics": 64, "blend": 0, "evenodd": False,
         "alpha": 1.0},
        # a chart line: 300 points, round caps and joins, half transparent, odd canvas
        {"name": "stroke_chart", "kind": "stroke", "w": 1021, "h": 767, "points": 300, "width": 3.0, "dash": False},
        # an illustration of 240 local shapes (the size of an SVG document) on an odd canvas
        {"name": "scene_svg", "kind": "scene", "w": 901, "h": 701, "paths": 240, "local": True},
        # the benchmark's dense scene: 2000 mixed fills and strokes over the whole canvas
        {"name": "scene_dense", "kind": "scene", "w": 1024, "h": 1024, "paths": 2000, "local": False},
        # a thumbnail service: eight jobs in flight, a third of them blurred
        {"name": "serve_mix", "kind": "serve", "jobs": 8, "side": 480, "paths": 120},
        # a label: 240 glyphs built, rendered and composited in one pass
        {"name": "glyphs_label", "kind": "glyphs", "w": 1000, "h": 600, "count": 240, "size": 24.0, "mode": 0,
         "whole": True},
        # the benchmark's page: 4096 glyphs of 8..256 px on 4096 x 4096
        {"name": "glyphs_page", "kind": "glyphs", "w": 4096, "h": 4096, "count": 4096, "size": 0.0, "mode": 0,
         "whole": False},
        # the benchmark's 20 modes at 2048 x 2048 as 5 artboards of 4 layers
        {"name": "stack_2048", "kind": "stack", "w": 2048, "h": 2048, "boards": 5, "layers": 4, "offset": False},
        # a card with a frosted panel and a shadow: odd sides, radii as UI toolkits use them
        {"name": "layers_ui", "kind": "layers", "w": 1237, "h": 1001, "r0": 12, "r1": 3, "spread": 4, "shadow": 12,
         "r2": 0, "r3": 0},
        # the benchmark's four blurs at 4096 x 4096
        {"name": "layers_4096", "kind": "layers", "w": 4096, "h": 4096, "r0": 1, "r1": 4, "r2": 16, "r3": 64,
         "spread": 0, "shadow": 0},
        # gradients and sprites on an odd canvas
        {"name": "canvas_sprites", "kind": "canvas", "w": 1601, "h": 1203, "sprite": 640, "sprites": 4, "angular": False},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["fill", "fill", "stroke", "scene", "scene", "serve", "glyphs", "glyphs", "stack", "layers",
                       "layers", "canvas"])
    if kind == "fill":
        w = _log(rng, 24, 2500)
        h = max(24, min(2500, int(w * rng.uniform(0.5, 2.0))))
        return {"kind": kind, "w": w, "h": h, "cubics": rng.choice([0, _log(rng, 2, 300)]),
                "blend": rng.choice([0, 0, rng.choice(PLAIN_MODES)]), "evenodd": rng.random() < 0.3,
                "alpha": rng.choice([1.0, 0.5])}
    if kind == "stroke":
        w = _log(rng, 64, 2500)
        return {"kind": kind, "w": w, "h": max(48, int(w * rng.uniform(0.4, 1.2))), "points": _log(rng, 8, 3000),
                "width": round(math.exp(rng.uniform(math.log(0.6), math.log(12.0))), 2), "dash": rng.random() < 0.3}
    if kind == "scene":
        local = rng.random() < 0.6
        w = _log(rng, 120, 2000 if local else 1024)
        h = max(96, min(2000 if local else 1024, int(w * rng.uniform(0.6, 1.6))))
        most = max(20, min(2000, int((1500 if local else 800) * 1024 * 1024 / (w * h))))
        return {"kind": kind, "w": w, "h": h, "paths": _log(rng, 12, most), "local": local}
    if kind == "serve":
        return {"kind": kind, "jobs": rng.randint(1, 12), "side": _log(rng, 96, 640), "paths": _log(rng, 10, 200)}
    if kind == "glyphs":
        whole = rng.random() < 0.4
        w = _log(rng, 200, 1600 if whole else 4096)
        return {"kind": kind, "w": w, "h": max(64, int(w * rng.uniform(0.3, 1.0))),
                "count": _log(rng, 4, 600 if whole else 4096), "size": round(rng.uniform(9.0, 96.0), 1),
                "mode": rng.choice([0, 0, 10]), "whole": whole}
    if kind == "stack":
        w = _log(rng, 64, 2048)
        return {"kind": kind, "w": w, "h": max(33, min(2048, int(w * rng.uniform(0.5, 1.8)))),
                "boards": rng.randint(1, 5), "layers": rng.randint(2, 4), "offset": rng.random() < 0.5}
    if kind == "layers":
        w = _log(rng, 96, 4096)
        r = [_log(rng, 1, 100) for _ in range(4)]
        shadow = rng.choice([0, _log(rng, 2, 24)])
        return {"kind": kind, "w": w, "h": max(64, min(4096, int(w * rng.uniform(0.5, 1.6)))), "r0": r[0], "r1": r[1],
                "r2": rng.choice([0, r[2]]), "r3": rng.choice([0, r[3]]), "spread": rng.randint(0, 8) if shadow else 0,
                "shadow": shadow}
    w = _log(rng, 128, 2400)
    return {"kind": "canvas", "w": w, "h": max(96, int(w * rng.uniform(0.5, 1.5))), "sprite": _log(rng, 32, 1024),
            "sprites": rng.randint(1, 6), "angular": rng.random() < 0.3}


# -- inputs -----------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _pixels(w, h, g):
    """A premultiplied RGBX image of soft shapes with grain: about a third of it
    transparent, a third opaque, edges between, as drawn layers have."""
    low = torch.rand((1, 4, h // 48 + 3, w // 48 + 3), generator=g, device="cuda")
    f = torch.nn.functional.interpolate(low, size=(h, w), mode="bilinear")[0].permute(1, 2, 0)
    f = f + (torch.rand((h, w, 4), generator=g, device="cuda") - 0.5) * 0.06
    a = ((f[..., 3:4] - 0.42) * 6.0).clamp(0, 1)
    c = f[..., :3].clamp(0, 1) * a
    return (torch.cat([c, a], dim=2) * 255.0 + 0.5).to(torch.uint8).contiguous()


def _wrapped(t):
    return px.Image.wrap(t.data_ptr(), t.shape[1], t.shape[0])


def _blank(w, h):
    return torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")


def _items(seed, n, w, h, local):
    """Paths over a w x h canvas: dense_scene's mix, over the whole canvas or as
    local shapes placed across it."""
    if not local:
        items = wl.dense_scene(seed % 100003 + 1, n_paths=n, size=float(max(w, h)))
        return items
    size = max(24.0, min(w, h) / 6.0)
    items = wl.dense_scene(seed % 100003 + 1, n_paths=n, size=size)
    u = np.random.RandomState(seed % (1 << 31)).rand(n, 3)
    for i, it in enumerate(items):
        s = 0.4 + 1.2 * u[i, 2]
        it["transform"] = [s, 0, 0, 0, s, 0, u[i, 0] * (w - 0.5 * size), u[i, 1] * (h - 0.5 * size), 1]
        it["blend"] = it["blend"] if i % 4 == 0 else 0  # most shapes of a document are drawn Normal
    return items


def _scene(seed, n, w, h, local):
    sc = px.Scene()
    sc.record_batch(_items(seed, n, w, h, local))
    return sc


def _outlines(seed, count, size):
    """Glyph-like outlines, an alphabet of 200 repeated over the run: (path, width, height, winding)."""
    alphabet = []
    for k in range(min(count, 200)):
        cmds, w, h, wind = wl.glyph((seed % 100003) * 211 + k)
        if size:  # one type size: the outline scaled to it
            s = np.float32(size / max(w, h))
            cmds = _stretched(cmds, s, s)
            w, h = max(1, int(w * s)), max(1, int(h * s))
        alphabet.append((cmds, w, h, wind))
    return [alphabet[i % len(alphabet)] for i in range(count)]


_PARAMS = {0: 0, 1: 2, 2: 2, 5: 6, 7: 4}  # values after a close, move, line, cubic, quadratic


def _stretched(cmds, sx, sy):
    """Moves, lines, curves and closes with their points scaled."""
    out, i = cmds.copy(), 0
    while i < len(out):
        n = _PARAMS[int(out[i])]
        out[i + 1:i + 1 + n:2] *= np.float32(sx)
        out[i + 2:i + 1 + n:2] *= np.float32(sy)
        i += 1 + n
    return out


def prepare(case, seed):
    kind = case["kind"]
    px.set_blocking(kind not in ("stack", "layers"))
    rs = np.random.RandomState((seed * 7919 + 13) % (1 << 31))
    g = _gen(seed * 31 + 7)
    st = {"case": case}
    if kind in ("fill", "stroke"):
        w, h = case["w"], case["h"]
        st["pixels"] = _pixels(w, h, g)
        st["image"] = _wrapped(st["pixels"])
        if kind == "fill" and case["cubics"]:
            cmds = wl.plain_path(seed % 100003 + 1, n_cubics=case["cubics"], size=1.0)
            cmds = _stretched(cmds, w, h)
        elif kind == "fill":
            cmds = wl.heart_commands(min(w, h) / 100.0 * (0.8 + 0.2 * rs.rand()))
        else:
            n = case["points"]
            x = np.linspace(0.02 * w, 0.98 * w, n)
            y = h * (0.5 + 0.35 * np.sin(np.cumsum(rs.randn(n)) * 0.6) + 0.1 * rs.randn(n))
            p = px.Path()
            p.move_to(float(x[0]), float(y[0]))
            for k in range(1, n):
                if k % 3 == 2:
                    p.quadratic_curve_to(float(x[k] - 0.4 * w / n), float(y[k - 1]), float(x[k]), float(y[k]))
                else:
                    p.line_to(float(x[k]), float(y[k]))
            cmds = p.array()
        st["path"] = np.ascontiguousarray(cmds, np.float32)
        st["paint"] = px.Paint(color=[float(v) for v in rs.rand(3)] + [float(case.get("alpha", 0.5))],
                               blend_mode=px.BlendMode(case.get("blend", 0)))
    elif kind == "scene":
        st["pixels"] = _blank(case["w"], case["h"])
        st["image"] = _wrapped(st["pixels"])
        st["scene"] = _scene(seed, case["paths"], case["w"], case["h"], case["local"])
    elif kind == "serve":
        st["server"] = px.Server()
        st["jobs"] = []
        for k in range(case["jobs"]):
            side = max(64, int(case["side"] * (0.6 + 0.8 * ((k * 5 + 3) % 8) / 7)))
            n = max(4, int(case["paths"] * (0.5 + ((k * 3 + 1) % 8) / 7)))
            st["jobs"].append((_scene(seed * 17 + k, n, side, side, k % 2 == 0), side, 2 + 6 * k if k % 3 == 2 else 0))
    elif kind == "glyphs":
        w, h = case["w"], case["h"]
        st["pixels"] = _blank(w, h)
        st["image"] = _wrapped(st["pixels"])
        st["outlines"] = _outlines(seed, case["count"], case["size"])
        st["at"] = np.stack([rs.randint(0, w, case["count"]), rs.randint(0, h, case["count"])], 1).astype(np.int64)
        if not case["whole"]:
            st["masks"] = px.Masks()
            st["masks"].add_paths(st["outlines"])
    elif kind == "stack":
        w, h = case["w"], case["h"]
        st["pixels"] = [_blank(w, h) for _ in range(case["boards"])]
        st["boards"] = [_wrapped(t) for t in st["pixels"]]
        st["sources"] = [_pixels(w, h, g) for _ in range(case["boards"] * case["layers"])]
        st["layers"] = [_wrapped(t) for t in st["sources"]]
        # the modes in turn over the boards; a board's first layer is never lost under a later Overwrite
        order = [17, 0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 18, 16, 19]
        k = len(st["layers"])
        st["modes"] = [order[(i * 20 // k) % 20] for i in range(k)]
        st["offsets"] = [(int(rs.randint(-w // 8, w // 8 + 1)), int(rs.randint(-h // 8, h // 8 + 1)))
                         if case["offset"] else (0, 0) for _ in range(k)]
        st["back"] = [float(v) for v in rs.rand(3)] + [1.0]
    elif kind == "layers":
        w, h = case["w"], case["h"]
        st["source"] = _pixels(w, h, g)
        st["layer"] = _wrapped(st["source"])
        st["pixels"] = _blank(w, h)
        st["image"] = _wrapped(st["pixels"])
        st["work"] = px.Image(w, h)
        st["radii"] = [case[k] for k in ("r0", "r1", "r2", "r3") if case[k]]
        if case["shadow"]:
            st["dropped"] = px.Image(w, h)
        st["back"] = [float(v) for v in rs.rand(3)] + [1.0]
    else:
        w, h, s = case["w"], case["h"], case["sprite"]
        st["pixels"] = _blank(w, h)
        st["image"] = _wrapped(st["pixels"])
        st["source"] = _pixels(s, s, g)
        st["sprite"] = _wrapped(st["source"])
        c = [[float(v) for v in rs.rand(3)] + [1.0] for _ in range(4)]
        st["back"] = px.Paint(kind=px.PaintKind.LinearGradientPaint, handles=[(0.1 * w, 0.2 * h), (0.9 * w, 0.7 * h)],
                              stops=[(c[0], 0.0), (c[1], 0.6), (c[2], 1.0)])
        shape = px.PaintKind.AngularGradientPaint if case["angular"] else px.PaintKind.RadialGradientPaint
        st["paint"] = px.Paint(kind=shape, opacity=0.8,
                               handles=[(0.5 * w, 0.5 * h), (0.8 * w, 0.5 * h), (0.5 * w, 0.8 * h)],
                               stops=[(c[2], 0.0), (c[3], 0.5), (c[0][:3] + [0.4], 1.0)])
        st["path"] = wl.heart_commands(min(w, h) / 100.0)
        st["places"] = []
        for k in range(case["sprites"]):
            a, z = 2 * math.pi * rs.rand(), [0.35, 1.0, 1.3, 0.8][k % 4] * (0.9 + 0.2 * rs.rand())
            sa, ca = math.sin(a) * z, math.cos(a) * z
            tx, ty = rs.rand() * 0.7 * w, rs.rand() * 0.7 * h
            if k % 4 == 1:  # moved by a part of a pixel only
                st["places"].append(np.array([1, 0, 0, 0, 1, 0, tx, ty, 1], np.float32))
            else:
                st["places"].append(np.array([ca, sa, 0, -sa, ca, 0, tx, ty, 1], np.float32))
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "fill":
        state["image"].fill_path(state["path"], state["paint"], None,
                                 px.WindingRule.EvenOdd if case["evenodd"] else px.WindingRule.NonZero)
        return state["pixels"]
    if kind == "stroke":
        state["image"].stroke_path(state["path"], state["paint"], None, case["width"], px.LineCap.RoundCap,
                                   px.LineJoin.RoundJoin, dashes=(9.0, 4.0) if case["dash"] else ())
        return state["pixels"]
    if kind == "scene":
        state["image"].fill((1, 1, 1, 1))
        state["image"].draw_scene(state["scene"])
        return state["pixels"]
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(sc, side, side, blur) for sc, side, blur in state["jobs"]]
        while server.pending():
            server.step()
        server.poll()
        return [server.take(i)[0] for i in ids]
    if kind == "glyphs":
        masks = state.get("masks")
        if masks is None:
            masks = px.Masks()
            masks.add_paths(state["outlines"])
        masks.render()
        state["image"].fill((1, 1, 1, 1) if case["mode"] else (0, 0, 0, 0))
        state["image"].draw_masks(masks, state["at"], px.BlendMode(case["mode"]))
        return state["pixels"]
    if kind == "stack":
        for board in state["boards"]:
            board.fill(state["back"])
        n = len(state["boards"])
        for i, layer in enumerate(state["layers"]):
            state["boards"][i % n].draw(layer, state["offsets"][i], state["modes"][i])
        return state["pixels"]
    if kind == "layers":
        image, work = state["image"], state["work"]
        image.fill(state["back"])
        if case["shadow"]:
            state["layer"].shadow_into(state["dropped"], (6, 9), case["spread"], case["shadow"], (0, 0, 0, 0.6))
            image.draw(state["dropped"])
        for r in state["radii"]:
            work.draw(state["layer"], (0, 0), px.BlendMode.OverwriteBlend)
            work.blur(r)
            image.draw(work)
        return state["pixels"]
    state["image"].fill(state["back"])
    state["image"].fill_path(state["path"], state["paint"])
    for m in state["places"]:
        state["image"].draw_transform(state["sprite"], m)
    return state["pixels"]


def work(case):
    """Bytes: images read once and written once, outlines read once.  Operations:
    the blend of a covered pixel as 24 integer operations, a blur tap as 8."""
    kind = case["kind"]
    if kind == "serve":
        side, n = case["side"], case["jobs"]
        return {"bytes": n * (8.0 * side * side + 400.0 * case["paths"]),
                "flops": 24.0 * 0.2 * n * case["paths"] * side * side}
    w, h = case["w"], case["h"]
    p = float(w * h)
    if kind == "fill":
        return {"bytes": 8.0 * p * 0.6 + 28.0 * max(4, case["cubics"]), "flops": 24.0 * 0.6 * p}
    if kind == "stroke":
        covered = min(p, 1.5 * case["points"] * case["width"] * max(2.0, 0.2 * h))
        return {"bytes": 8.0 * covered + 12.0 * case["points"], "flops": 24.0 * covered}
    if kind == "scene":
        covered = case["paths"] * (min(w, h) ** 2 / 50.0 if case["local"] else 0.38 * p)
        return {"bytes": 8.0 * p + 700.0 * case["paths"], "flops": 24.0 * covered}
    if kind == "glyphs":
        side = case["size"] or 72.0
        covered = case["count"] * side * side
        return {"bytes": 4.0 * p + min(p, covered) * 4.0 + covered + 1200.0 * case["count"], "flops": 24.0 * covered}
    if kind == "stack":
        n = case["boards"] * case["layers"]
        return {"bytes": 4.0 * p * (n + case["boards"]), "flops": 40.0 * n * p}
    if kind == "layers":
        radii = [case[k] for k in ("r0", "r1", "r2", "r3") if case[k]]
        taps = sum(2 * (2 * r + 1) for r in radii) + 4.0 * case["shadow"]
        return {"bytes": 8.0 * p, "flops": 8.0 * taps * p + 24.0 * (len(radii) + 1) * p}
    return {"bytes": 4.0 * p + 4.0 * case["sprite"] ** 2,
            "flops": 60.0 * p + 60.0 * case["sprites"] * min(p, float(case["sprite"] ** 2))}
