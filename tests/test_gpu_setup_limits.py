"""The setup kernel at the limits of its arithmetic: paths whose rows lie outside
what the image, 32 bits or 64 bits hold, and segments whose band range is empty
because a coordinate wraps in the reference's 32-bit conversion, byte for byte
against the oracle."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _init():
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)


def zigzag(n, w, y0, y1):
    """n lines between the heights y0 and y1, closed."""
    x = np.linspace(0.3, w - 0.4, n + 1)
    cmds = [1.0, x[0], y0]
    for k in range(1, n + 1):
        cmds += [2.0, x[k], y1 if k & 1 else y0]
    return np.asarray(cmds + [0.0], np.float32)


def check(cmds, w, h, modes=(0,)):
    """A fill, with the modes of a fill path and of a clearing mask, and a scene."""
    for mode in modes:
        back = np.random.RandomState(7).randint(0, 256, (h, w, 4)).astype(np.uint8)
        back[..., :3] = np.minimum(back[..., :3], back[..., 3:])
        ref = back.copy()
        pxo.fill_path(ref, cmds, [0.1, 0.7, 0.4, 0.8], 1.0, mode, None, 0)
        paint = px.Paint(color=(0.1, 0.7, 0.4, 0.8), blend_mode=px.BlendMode(mode))
        img = px.Image.from_numpy(back)
        img.fill_path(cmds, paint)
        assert np.array_equal(img.to_numpy(), ref)
        sc = px.Scene()
        sc.fill_path(cmds, paint)
        img = px.Image.from_numpy(back)
        img.draw_scene(sc)
        assert np.array_equal(img.to_numpy(), ref)


# the path's last row is past 2^63, its first one in the image; or all rows are far below or above it
@pytest.mark.parametrize("y0,y1", [(240.0, 1.0e19), (0.0, 3.0e38), (394.75, 3.0e38), (4294967296.0, 4294970000.0),
                                   (4294967396.0, 9.0e9), (-4294967296.0, -4294967000.0), (-9.0e9, -4294967000.0),
                                   (-3.0e38, -1.0e19), (400.0, 500.0), (-9.0, 0.0), (1.0e19, 1.0e20)])
@pytest.mark.parametrize("n", [2, 40, 301, 3000])
def test_rows_out_of_range(n, y0, y1):
    check(zigzag(n, 37, y0, y1), 37, 400, (0, 16))


# 2^32 and above wrap to small bands; from 2^63 on the conversion yields its minimum
@pytest.mark.parametrize("far", [4294967296.0, 4294967296.0 + 1024, 3.0e10, 9.0e18, 1.0e19, 3.0e38])
@pytest.mark.parametrize("n,h", [(2, 400), (40, 400), (301, 400), (3000, 333), (300, 5000)])
def test_segments_in_no_band(n, h, far):
    w = 37
    rs = np.random.RandomState(n + h)
    for near in (h * 0.6, h - 5.25):
        cmds = zigzag(n, w, near, far)[:-1]
        # and a shape of ordinary segments besides
        pts = rs.rand(6, 2) * (w, h)
        cmds = np.concatenate([cmds, [0.0, 1.0, *pts[0]], *[[2.0, *p] for p in pts[1:]], [0.0]]).astype(np.float32)
        try:
            check(cmds, w, h)
        except px.PixieError as e:  # the library's limit of 2048 crossings a row
            assert n > 2048 and "Path too complex" in str(e)


def tall(n, w, h, seed, far=0):
    """n short lines, quadratics and cubics wandering over a tall image, six edges
    through all of it, and edges that end `far` beyond 32 bits."""
    rs = np.random.RandomState(seed)
    at = np.array([0.5 * w, 0.02 * h])
    cmds = [1.0, *at]
    for k in range(n):
        kind = [0, 0, 1, 2, 0][k % 5]
        pts = []
        for _ in range(kind + 1):
            at = np.clip(at + (rs.rand(2) - 0.5) * (w, 60.0) + (0, 0.9 * h / n / (kind + 1)), 0, (w, h - 0.25))
            pts += [at[0], at[1]]
        cmds += [[2.0, 7.0, 5.0][kind]] + pts
    cmds += [0.0, 1.0, 0.1 * w, 0.0]
    for k in range(6):
        cmds += [2.0, (0.15 + 0.12 * k) * w, h if k % 2 == 0 else 0.0]
    for k in range(far):
        cmds += [0.0, 1.0, 0.2 * w, h * (0.3 + 0.1 * k), 2.0, 0.7 * w, 4294967296.0, 2.0, 0.8 * w, h * 0.9]
    return np.asarray(cmds + [0.0], np.float32)


# images around one, two and three windows of 1024 bands, with segments enough for a band every 4 rows
@pytest.mark.parametrize("h", [4092, 4096, 4100, 8192, 8200, 12300])
@pytest.mark.parametrize("n,far", [(700, 0), (2300, 0), (2300, 3)])
def test_windows_of_bands(h, n, far):
    check(tall(n, 11, h, h + n, far), 11, h)


def test_windows_of_bands_in_batches():
    """Masks and images of several heights in one launch, and strokes."""
    hs = [37, 4100, 8300, 700, 9000]
    cmds = [tall(1500, 11, h, h) for h in hs]
    refs = []
    for c, h in zip(cmds, hs):
        refs.append(pxo.new_image(11, h))
        pxo.fill_path(refs[-1], c, [1, 1, 1, 1], 1.0, 0, None, 0)
    m = px.Masks()
    m.add_paths([(c, 11, h, 0) for c, h in zip(cmds, hs)])
    m.render()
    imgs = [px.Image(11, h) for h in hs]
    assert not px.fill_paths_batch(imgs, cmds, [(1, 1, 1, 1)] * len(hs)).any()
    for k, ref in enumerate(refs):
        assert np.array_equal(m.mask(k), ref[..., 3])
        assert np.array_equal(imgs[k].to_numpy(), ref)
    line = tall(150, 40, 8300, 5)
    ref = pxo.new_image(40, 8300)
    pxo.stroke_path(ref, line, [0.1, 0.7, 0.4, 0.8], 1.0, 0, None, 3.0, 1, 1)
    img = px.Image(40, 8300)
    img.stroke_path(line, px.Paint(color=(0.1, 0.7, 0.4, 0.8)), None, 3.0, 1, 1)
    assert np.array_equal(img.to_numpy(), ref)


def test_more_band_entries_than_32_bits():
    """262,200 edges through all 8191 bands of a 32,767-row image are 2^31 + 196,552
    entries: the call fails, leaves the image alone, and the next calls are whole."""
    w, h, n = 9, 32767, 262200
    cmds = np.empty((n, 3), np.float32)
    cmds[:, 0] = 2.0
    cmds[0, 0] = 1.0
    cmds[:, 1] = np.linspace(0.5, w - 0.5, n)
    cmds[:, 2] = np.where(np.arange(n) & 1, h, 0.0)
    cmds = np.concatenate([cmds.ravel(), [0.0]]).astype(np.float32)
    paint = px.Paint(color=(0.1, 0.7, 0.4, 0.8))
    small = np.asarray([1, 1.3, 2, 2, 7.6, 9.1, 2, 4.5, 90.25, 0], np.float32)
    ref = pxo.new_image(w, h)
    pxo.fill_path(ref, small, [0.1, 0.7, 0.4, 0.8], 1.0, 0, None, 0)
    img = px.Image(w, h)
    with pytest.raises(px.PixieError, match="Out of workspace memory"):
        img.fill_path(cmds, paint)
    assert not img.to_numpy().any()
    img.fill_path(small, paint)
    assert np.array_equal(img.to_numpy(), ref)
    sc = px.Scene()
    sc.fill_path(small, paint)
    sc.fill_path(cmds, paint)
    sc.fill_path(small, paint)
    img = px.Image(w, h)
    with pytest.raises(px.PixieError, match="Out of workspace memory"):
        img.draw_scene(sc)
    assert np.array_equal(img.to_numpy(), ref)  # the path before it is drawn, as by calls one by one
