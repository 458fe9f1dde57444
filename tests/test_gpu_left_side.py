"""Trapezoid rows whose edges cross the image's left side between pixels -1 and
0: pixel 0 has an area above 1 there, a multiplier that a byte of coverage does
not hold.  The row kernels draw such pixels themselves -- no row is handed on --
in images of one and of several tiles, by warps and by a CTA per row, in
masks and scenes, byte for byte as the oracle."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _init():
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)


def wedge(w, h, n):
    """A shape whose left side crosses x = 0 once a row, between -0.95 and 0.45,
    with its corners on the rows' edges, so that rows are trapezoids; n > 0: its
    right side broken n times, where they are not."""
    u = np.random.RandomState(h).rand(h + 5)
    pts = [(0.8 * w, -2.0)]
    for k in range(n):
        pts.append(((0.55 + 0.2 * (k % 2)) * w, h * (0.1 + 0.3 * (k + 1) / (n + 1))))
    pts.append((0.7 * w, h + 2.0))
    for y in range(h + 2, -3, -1):
        pts.append((-0.5 - 0.45 * u[y] if y % 2 else 0.05 + 0.4 * u[y], y))
    cmds = [1.0, *pts[0]]
    for p in pts[1:]:
        cmds += [2.0, *p]
    return np.asarray(cmds + [0.0], np.float32)


@pytest.mark.parametrize("w,h", [(11, 53), (64, 97), (1021, 30), (1500, 41), (4096, 19), (7, 3000)])
def test_left_side(w, h):
    rs = np.random.RandomState(w)
    for n in (0, 3, 600):
        cmds = wedge(w, h, n)
        for mode, alpha in ((0, 1.0), (0, 0.6), (13, 0.6), (17, 0.5), (18, 0.5)):
            color = [0.2, 0.6, 0.9, alpha]
            back = (rs.rand(h, w, 1) * rs.rand(h, w, 4) * 255).astype(np.uint8)
            back[..., 3] = back.max(2)
            ref = back.copy()
            pxo.fill_path(ref, cmds, color, 1.0, mode, None, 0)
            img = px.Image.from_numpy(back)
            img.fill_path(cmds, px.Paint(color=color, blend_mode=px.BlendMode(mode)))
            assert np.array_equal(img.to_numpy(), ref)
            assert px.last_fill_stats()["wide_rows"] == 0
        ref = pxo.new_image(w, h)
        pxo.fill_path(ref, cmds, [1, 1, 1, 1], 1.0, 0, None, 0)
        m = px.Masks()
        m.add_path(cmds, w, h)
        for variant in (0, 1):
            m.render_config(variant, 1)
            assert np.array_equal(m.mask(0), ref[..., 3])
            if n < 600:  # (else rows of more than the 64 crossings of variant 1)
                assert px.last_fill_stats()["wide_rows"] == 0


@pytest.mark.parametrize("w,h", [(11, 53), (300, 64), (1500, 41), (4096, 19)])
def test_left_side_of_scenes(w, h):
    rs = np.random.RandomState(w)
    back = (rs.rand(h, w, 1) * rs.rand(h, w, 4) * 255).astype(np.uint8)
    back[..., 3] = back.max(2)
    for opaque in (False, True):
        if opaque:
            back[..., 3] = 255
        sc, ref = px.Scene(), back.copy()
        for k, mode in enumerate((0, 13, 0, 1, 10, 18, 0, 5, 19)):
            cmds = wedge(w * (0.4 + 0.07 * k), h, 3 * (k % 2))
            color = [0.2 + 0.05 * k, 0.6, 0.9 - 0.07 * k, 1.0 if k == 2 else 0.6]
            pxo.fill_path(ref, cmds, color, 1.0, mode, None, 0)
            sc.fill_path(cmds, px.Paint(color=color, blend_mode=px.BlendMode(mode)))
        img = px.Image.from_numpy(back)
        img.draw_scene(sc)
        assert np.array_equal(img.to_numpy(), ref)
        assert px.last_fill_stats()["wide_rows"] == 0
