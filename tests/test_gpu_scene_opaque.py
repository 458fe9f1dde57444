"""Scenes over opaque backdrops, whose colour modes have a composite of their
own: every backdrop byte in two channels against each source, opaque, all but
transparent and at the modes' branches, whole pixels and part-covered ones, and
canvases opaque only in part -- byte for byte against the oracle."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _init():
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)


def backdrop(part):
    b = np.random.RandomState(5).randint(0, 256, (256, 256, 4)).astype(np.uint8)
    b[..., 0] = np.arange(256)[None, :]
    b[..., 1] = np.arange(256)[:, None]
    b[..., 3] = 255
    if part:  # a third of the canvas of lower alphas (premultiplied)
        b[:, 100:190, 3] = np.random.RandomState(6).randint(0, 256, (256, 90))
        b[..., :3] = np.minimum(b[..., :3], b[..., 3:])
    return b


SHAPES = [[1, -2, -2, 2, 300, -2, 2, 300, 300, 2, -2, 300, 0],          # the whole canvas
          [1, 3.3, 1.7, 2, 250.2, 90.4, 2, 128.6, 254.1, 2, 10.9, 99.5, 0]]  # edges of every coverage
COLORS = [(0, 0, 0, 1), (1, 1, 1, 1), (0.5, 0.498, 0.502, 1), (0.2, 0.9, 0.6, 1), (0.7, 0.1, 0.4, 0.996),
          (0.3, 0.6, 1, 0.5), (1, 0, 0.25, 0.251), (0.9, 0.8, 0.1, 0.004), (0.4, 0.4, 0.4, 0.0)]


@pytest.mark.parametrize("part", [False, True])
@pytest.mark.parametrize("blend", range(20))
def test_scene_modes(blend, part):
    back = backdrop(part)
    for color in COLORS:
        for w in (256, 77):  # many rows, and a width that is no multiple of 32
            ref = np.ascontiguousarray(back[:, 60:60 + w] if w < 256 else back)
            img = px.Image.from_numpy(ref.copy())
            sc = px.Scene()
            for shape in SHAPES:
                cmds = np.asarray(shape, np.float32)
                pxo.fill_path(ref, cmds, list(color), 1.0, blend, None, 0)
                sc.fill_path(cmds, px.Paint(color=color, blend_mode=blend), None, 0)
            img.draw_scene(sc)
            assert np.array_equal(img.to_numpy(), ref), f"color {color} width {w}"


@pytest.mark.parametrize("blend", [0, 1, 9, 12])
def test_scene_any_bytes(blend):
    """Canvases of any bytes (colour under alpha 0, not premultiplied), with sources down to nothing."""
    rs = np.random.RandomState(8)
    back = rs.randint(0, 256, (90, 151, 4)).astype(np.uint8)
    back[..., 3] = rs.choice([0, 0, 1, 128, 254, 255, 255], (90, 151))
    for color in [(0.9, 0.8, 0.1, 0.004), (0.4, 0.4, 0.4, 0.0), (0.2, 0.9, 0.6, 1), (1, 0, 0.25, 0.5)]:
        ref = back.copy()
        img = px.Image.from_numpy(back)
        sc = px.Scene()
        for shape in SHAPES:
            cmds = np.asarray(shape, np.float32)
            pxo.fill_path(ref, cmds, list(color), 1.0, blend, None, 0)
            sc.fill_path(cmds, px.Paint(color=color, blend_mode=blend), None, 0)
        img.draw_scene(sc)
        assert np.array_equal(img.to_numpy(), ref), f"color {color}"


@pytest.mark.parametrize("slice_w", [0, 36, 64])
def test_scene_mixed_modes(slice_w):
    """Mask modes among the colour modes: what they leave is not opaque."""
    back = backdrop(False)[:60]
    ref, img, sc = back.copy(), px.Image.from_numpy(back), px.Scene()
    for i in range(70):
        mode = 16 + i % 4 if i in (21, 22, 40, 65) else (i * 7) % 16
        x, y = (i * 37) % 200, (i * 11) % 40
        cmds = np.asarray([1, x + 0.3, y - 3, 2, x + 60.6, y + 2.2, 2, x + 20, y + 30.7, 0], np.float32)
        color = ((i * 5 % 11) / 10, (i * 3 % 7) / 6, (i % 5) / 4, 1.0 if i % 3 else 0.6)
        pxo.fill_path(ref, cmds, list(color), 1.0, mode, None, 0)
        sc.fill_path(cmds, px.Paint(color=color, blend_mode=mode), None, 0)
    px.scene_config(slice_w)
    try:
        img.draw_scene(sc)
    finally:
        px.scene_config(0)
    assert np.array_equal(img.to_numpy(), ref)
