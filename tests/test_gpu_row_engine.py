"""The row engine of the fill kernels at the edges of its instances: numbers of
crossings around each instance's limit, images around its tile widths and its
widest image, trapezoid rows in one and several tiles, rows without
anti-aliasing, and canvases whose bytes are not premultiplied -- drawn path by
path, recorded as a scene, and as masks, byte for byte against the oracle."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _init():
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)


def poly(points):
    cmds = []
    for i, (x, y) in enumerate(points):
        cmds += [1.0 if i == 0 else 2.0, float(x), float(y)]
    return np.asarray(cmds + [0.0], np.float32)


def zigzag(n, w, h, seed):
    """n crossings a row: edges up and down across the image's height."""
    rs = np.random.RandomState(seed)
    xs = np.sort(rs.uniform(0.5, w - 0.5, n)) if seed % 2 else rs.uniform(-3, w + 3, n)
    return poly([(x, 0.3 if k % 2 else h - 0.4) for k, x in enumerate(xs)])


def joined(paths):
    return np.concatenate(paths).astype(np.float32)


def rects(n, w, h, frac, seed):
    """n rectangles in one path, on whole pixels or not."""
    rs = np.random.RandomState(seed)
    out = []
    for _ in range(n):
        x, y = rs.randint(0, w - 2), rs.randint(0, h - 2)
        u, v = x + rs.randint(1, max(2, w // 3)), y + rs.randint(1, max(2, h // 2))
        f = rs.rand() * frac
        out.append(poly([(x + f, y), (u + f, y), (u + f, v), (x + f, v)]))
    return joined(out)


def overlapping(n, w, seed):
    """n triangles sharing vertices and edges: many crossings at one position."""
    rs = np.random.RandomState(seed)
    c = [(w * k / 7.0, 2.0 + 5 * (k % 3)) for k in range(8)]
    return joined([poly([c[i] for i in rs.choice(8, 3, replace=False)]) for _ in range(n)])


def canvas(w, h, seed):
    return np.random.RandomState(seed).randint(0, 256, (h, w, 4)).astype(np.uint8)


def check(paths, w, h, seed, blends=(0,), windings=(0, 1), color=(0.8, 0.3, 0.1, 0.7)):
    back = canvas(w, h, seed)
    for cmds in paths:
        for blend in blends:
            for winding in windings:
                ref = back.copy()
                pxo.fill_path(ref, cmds, list(color), 1.0, blend, None, winding)
                img = px.Image.from_numpy(back)
                img.fill_path(cmds, px.Paint(color=color, blend_mode=blend), None, winding)
                assert np.array_equal(img.to_numpy(), ref), f"{w}x{h} blend {blend} winding {winding}"
                sc = px.Scene()
                sc.fill_path(cmds, px.Paint(color=color, blend_mode=blend), None, winding)
                img = px.Image.from_numpy(back)
                img.draw_scene(sc)
                assert np.array_equal(img.to_numpy(), ref), f"scene {w}x{h} blend {blend} winding {winding}"


@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 15, 16, 17, 18, 31, 32, 33, 63, 64, 65, 66, 127, 128, 129, 130, 255, 256, 257, 258, 511, 512,
                               513, 514, 1100, 2047, 2048])
def test_crossings_per_row(n):
    check([zigzag(n, 700, 9, 2 * n), zigzag(n, 700, 9, 2 * n + 1)], 700, 9, n)


@pytest.mark.parametrize("w", [1, 3, 15, 16, 17, 127, 255, 257, 1007, 1008, 1009, 1023, 1024, 1025, 1040, 2047, 2049,
                               3001])
def test_widths(w):
    paths = [zigzag(12, w, 7, 3), poly([(-2, -1), (w + 2, 1.5), (w * 0.7, 6.2), (w * 0.1, 6.9)])]
    if w > 3:
        paths.append(rects(6, w, 7, 1.0, w))
    check(paths, w, 7, w)


@pytest.mark.parametrize("w", [8191, 8192, 16383, 16384, 32767, 32768])
def test_widest_images(w):
    far = poly([(w - 40.5, 0.2), (w + 30, 2.7), (w - 90.25, 4.6), (10.3, 4.9), (33.1, 0.6)])
    check([far, zigzag(140, w, 5, 4), zigzag(300, w, 5, 6)], w, 5, 1, windings=(0,))


@pytest.mark.parametrize("blend", range(20))
def test_trapezoid_rows_every_mode(blend):
    w, h = 1100, 14
    shallow = poly([(-3.5, 0.1), (w - 20, 9.0), (w + 4, 13.3), (200.4, 12.2)])
    bars = joined([poly([(20 * k + 0.3, -2), (20 * k + 9.6, -2), (20 * k + 9.9, 20), (20 * k + 0.31, 20)])
                   for k in range(40)])
    check([shallow, bars], w, h, blend, blends=(blend,), windings=(0,))


@pytest.mark.parametrize("blend", [0, 2, 17])
def test_rows_without_antialiasing(blend):
    check([rects(k, 90, 24, 0.0, k) for k in (1, 2, 5, 30)], 90, 24, 3, blends=(blend,))


@pytest.mark.parametrize("n", [2, 3, 5, 9, 40])
def test_crossings_at_one_position(n):
    check([overlapping(n, 61, s) for s in range(4)], 61, 19, n)


@pytest.mark.parametrize("variant", [0, 1])
def test_masks(variant):
    shapes = [(zigzag(n, w, h, n), w, h, n % 2) for n, w, h in
              [(2, 5, 5), (7, 33, 9), (64, 250, 6), (65, 251, 7), (66, 255, 5), (140, 257, 8), (300, 600, 5),
               (9, 1021, 6), (10, 1030, 5)]] + [(rects(5, 50, 20, 0.0, 1), 50, 20, 0), (rects(4, 51, 20, 1.0, 2), 51, 20, 0)]
    m = px.Masks()
    for cmds, w, h, wind in shapes:
        m.add_path(cmds, w, h, None, wind)
    m.render_config(variant, 3)
    for i, (cmds, w, h, wind) in enumerate(shapes):
        ref = pxo.new_image(w, h)
        pxo.fill_path(ref, cmds, [1, 1, 1, 1], 1.0, 0, None, wind)
        assert np.array_equal(m.mask(i), ref[..., 3]), f"mask {i}"


@pytest.mark.parametrize("lines", [600, 2200])
@pytest.mark.parametrize("n,w", [(2, 60), (16, 700), (17, 700), (18, 700), (40, 1100), (64, 700), (65, 700), (66, 700),
                                 (128, 300), (255, 700), (256, 1100), (257, 700), (600, 1100)])
def test_paths_of_many_lines(n, w, lines):
    """A path of so many lines that each row takes a CTA (the lines are
    horizontal, so the crossings are the zigzag's)."""
    flat = poly([(10 + k % 7, 3.0) for k in range(lines)])
    check([joined([zigzag(n, w, 9, 2 * n + 1), flat]), joined([flat, rects(n // 2 + 1, w, 9, 1.0, n)])], w, 9, n)
