"""Every tile shape of the mask composite, below and above the number of masks
from which they are binned by rows of tiles, byte for byte against the oracle's
draws one after another."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [0, 1, 2])
@pytest.mark.parametrize("n,w,h", [(3, 31, 33), (512, 65, 63), (513, 129, 130), (4100, 63, 65)])
@pytest.mark.parametrize("mode", [0, 12, 17])
def test_tile_shapes(tile, n, w, h, mode):
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)
    rs = np.random.RandomState(n + mode)
    shapes = []
    for _ in range(min(n, 30)):
        u, v = rs.randint(1, 40, 2)
        pts = rs.rand(4, 2) * (u, v)
        cmds = np.asarray([1.0, *pts[0], 2.0, *pts[1], 7.0, *pts[2], *pts[3], 0.0], np.float32)
        ref = pxo.new_image(int(u), int(v))
        pxo.fill_path(ref, cmds, [1, 1, 1, 1])
        shapes.append((cmds, int(u), int(v), 0, ref))
    pick = [shapes[int(i)] for i in rs.randint(0, len(shapes), n)]
    masks = px.Masks()
    masks.add_paths([s[:4] for s in pick])
    masks.render()
    at = np.stack([rs.randint(-40, w + 8, n), rs.randint(-40, h + 8, n)], 1).astype(np.int64)
    page = np.random.RandomState(5).randint(0, 256, (h, w, 4)).astype(np.uint8)
    img = px.Image.from_numpy(page)
    px.draw_masks(img, masks, at, mode, tile)
    ref = page.copy()
    for (x, y), s in zip(at, pick):
        pxo.draw(ref, s[4], int(x), int(y), mode)
    assert np.array_equal(img.to_numpy(), ref)


def test_shapes_there_are():
    m = px.Masks()
    m.add_path([1, 1, 1, 2, 5, 1, 2, 3, 6, 0], 8, 8)
    m.render()
    img = px.Image(20, 20)
    for tile in (-1, 3):
        with pytest.raises(px.PixieError, match="Invalid configuration"):
            px.draw_masks(img, m, [(1, 1)], 0, tile)
