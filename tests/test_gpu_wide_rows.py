"""Rows wider than the row engine's difference array: gone through in tiles,
with the sample lines' spans kept from the first tile where they fit (up to 102
crossings a row on one warp; always with a warp per line) and the trapezoids
tried out first.  Numbers of crossings around the groups' 16, that limit and the
kernels' 64 and 256, widths around one and several tiles, by warps and by CTAs
per row, into images and masks, byte for byte against the oracle."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo

pytestmark = pytest.mark.gpu
H = 24
COLOR = [0.1, 0.7, 0.4, 0.8]


@pytest.fixture(scope="module", autouse=True)
def _init():
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)


def comb(n, w, seed, work=0):
    """A closed zigzag of about n edges over the width, crossing itself here and
    there; `work` adds short lines above the image."""
    rs = np.random.RandomState(seed)
    n = max(2, n // 2 * 2)
    x = (np.arange(n) + 0.5) * w / n + (rs.rand(n) - 0.5) * w / n * 2.2
    y = np.where(np.arange(n) & 1, H * (0.6 + 0.38 * rs.rand(n)), H * (0.02 + 0.38 * rs.rand(n)))
    cmds = [1.0, x[0], y[0]]
    for k in range(1, n):
        cmds += [2.0, x[k], y[k]]
    cmds += [0.0]
    if work:
        cmds += [1.0, 5.0, -20.0]
        for k in range(work):
            cmds += [2.0, 5.0 + k % 7, -21.0 - k % 5]
        cmds += [0.0]
    return np.asarray(cmds, np.float32)


def check(cmds, w, winding, masks=False):
    ref = pxo.new_image(w, H)
    pxo.fill_path(ref, cmds, COLOR, 1.0, 0, None, winding)
    paint = px.Paint(color=COLOR)
    img = px.Image(w, H)
    img.fill_path(cmds, paint, None, winding)
    assert np.array_equal(img.to_numpy(), ref)
    sc = px.Scene()
    sc.fill_path(cmds, paint, None, winding)
    img = px.Image(w, H)
    img.draw_scene(sc)
    assert np.array_equal(img.to_numpy(), ref)
    if masks:
        ref = pxo.new_image(w, H)
        pxo.fill_path(ref, cmds, [1, 1, 1, 1], 1.0, 0, None, winding)
        m = px.Masks()
        m.add_path(cmds, w, H, None, winding)
        for variant in (0, 1):
            m.render_config(variant, 1)
            assert np.array_equal(m.mask(0), ref[..., 3])


@pytest.mark.parametrize("n", [2, 8, 16, 18, 64, 100, 102, 104, 130, 254, 258, 400])
@pytest.mark.parametrize("w", [1025, 2500, 4100])
@pytest.mark.parametrize("work", [0, 600])
def test_tiled_rows(n, w, work):
    check(comb(n, w, n + w, work), w, (n // 2) % 2, masks=work == 0)


@pytest.mark.parametrize("n", [4, 30, 200])
def test_very_wide_rows(n):
    check(comb(n, 20011, n), 20011, 0, masks=True)
    check(comb(n, 40000, n), 40000, 1)


def test_wide_trapezoids_and_spans():
    """Rows of trapezoids, simple and not, and of whole pixels, over many tiles."""
    w = 9001
    for slant in (0.0, 0.3, 700.0):
        cmds = []
        for a, b in ((10.0, 2000.0), (2000.0 + slant, 5100.0), (5100.0 + 2 * slant, 8000.0)):
            cmds += [1.0, a, 0.0, 2.0, b, 0.0, 2.0, b + slant, float(H), 2.0, a + slant, float(H), 0.0]
        check(np.asarray(cmds, np.float32), w, 0, masks=True)


def test_wide_strokes():
    w, h = 6000, 50
    rs = np.random.RandomState(3)
    x, y = np.linspace(20, w - 20, 60), h * (0.2 + 0.6 * rs.rand(60))
    cmds = [1.0, x[0], y[0]]
    for k in range(1, 60):
        cmds += [2.0, x[k], y[k]]
    cmds = np.asarray(cmds, np.float32)
    ref = pxo.new_image(w, h)
    pxo.stroke_path(ref, cmds, COLOR, 1.0, 0, None, 3.0, 1, 1)
    img = px.Image(w, h)
    img.stroke_path(cmds, px.Paint(color=COLOR), None, 3.0, 1, 1)
    assert np.array_equal(img.to_numpy(), ref)


@pytest.mark.parametrize("curves", [0, 90])  # with 90 short curves above the image the paths count as heavy
def test_many_crossings_at_mixed_widths(curves):
    """Rows of more than 256 crossings of images that the kernel for them takes and
    of wider ones, in one launch and alone."""
    ws = [4200, 900, 5000, 4095, 4096]
    above = [1.0, 5.0, -20.0] + [5.0, 6.0, -20.5, 7.0, -21.0, 5.0, -20.0 - 0.01] * curves + [0.0]
    cmds = [np.concatenate([comb(n, w, n), np.asarray(above, np.float32)]) for n, w in zip((400, 500, 20, 300, 700), ws)]
    refs = []
    for c, w in zip(cmds, ws):
        refs.append(pxo.new_image(w, H))
        pxo.fill_path(refs[-1], c, COLOR, 1.0, 0, None, 0)
    for pick in ([0, 1, 2, 3, 4], [0], [2], [0, 4], [1, 3]):
        imgs = [px.Image(ws[k], H) for k in pick]
        assert not px.fill_paths_batch(imgs, [cmds[k] for k in pick], [COLOR] * len(pick)).any()
        for im, k in zip(imgs, pick):
            assert np.array_equal(im.to_numpy(), refs[k])
