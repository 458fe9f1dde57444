"""Mask composites around the numbers of masks at which they are binned and
tested in chunks, at offsets on and off the page, byte for byte against the
oracle's draws one after another."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,w,h", [(1, 33, 31), (511, 65, 64), (512, 64, 65), (513, 333, 217), (700, 130, 33),
                                   (4095, 40, 40), (4096, 31, 70), (4097, 63, 32), (8200, 40, 20)])
@pytest.mark.parametrize("mode", [0, 10, 17])
def test_ordered_composite(n, w, h, mode):
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)
    rs = np.random.RandomState(n + mode)
    masks = px.Masks()
    shapes = []
    for k in range(min(n, 40)):
        u, v = rs.randint(1, 24, 2)
        pts = rs.rand(4, 2) * (u, v)
        cmds = np.asarray([1.0, *pts[0], 2.0, *pts[1], 7.0, *pts[2], *pts[3], 0.0], np.float32)
        ref = pxo.new_image(int(u), int(v))
        pxo.fill_path(ref, cmds, [1, 1, 1, 1])
        shapes.append((cmds, int(u), int(v), 0, ref))
    pick = [shapes[int(i)] for i in rs.randint(0, len(shapes), n)]
    masks.add_paths([s[:4] for s in pick])
    masks.render()
    at = np.stack([rs.randint(-30, w + 8, n), rs.randint(-30, h + 8, n)], 1).astype(np.int64)
    at[0] = (1 << 40, -(1 << 40))  # far off the page
    page = np.random.RandomState(5).randint(0, 256, (h, w, 4)).astype(np.uint8)
    img = px.Image.from_numpy(page)
    img.draw_masks(masks, at, mode)
    ref = page.copy()
    for (x, y), s in zip(at[1:], pick[1:]):
        pxo.draw(ref, s[4], int(x), int(y), mode)
    assert np.array_equal(img.to_numpy(), ref)


def test_batches_rendered_again():
    """The first rendering is issued as launches, later ones replay a graph."""
    m = px.Masks()
    paths = []
    for step in range(3):
        w, h = 20 + 13 * step, 31 - 5 * step
        cmds = np.asarray([1, 1.3, 2, 2, w - 2.6, 3.1, 2, w * 0.5, h - 1.4, 0], np.float32)
        paths.append((cmds, w, h))
        m.add_path(cmds, w, h)
        for _ in range(3):
            m.render()
            for i, (c, cw, ch) in enumerate(paths):
                ref = pxo.new_image(cw, ch)
                pxo.fill_path(ref, c, [1, 1, 1, 1], 1.0, 0, None, 0)
                assert np.array_equal(m.mask(i), ref[..., 3])
