"""Which passes a blur ran on: the ring passes by tensor maps where the image's
rows are whole 16-byte units and begin at one, by plain copies where not, and
where they are not taken at all; radii 6 to 8 on both sides of the sizes from
which the ring takes them."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo
from pixie_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _init():
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)
    px.blur_config(3)
    yield
    px.blur_config(3)


def blurred(w, h, r, want):
    img = wl.premultiplied_image(w * 3 + h + r, w, h)
    g = px.Image.from_numpy(img)
    g.blur(r, (0.2, 0.5, 0.9, 0.6))
    ref = img.copy()
    pxo.blur(ref, r, pxo.color_to_rgbx((0.2, 0.5, 0.9, 0.6)))
    assert np.array_equal(g.to_numpy(), ref)
    assert px.last_blur_ring() == want, (w, h, r)


@pytest.mark.parametrize("w,h,r,want", [
    (64, 64, 9, 1), (64, 61, 9, 1), (128, 70, 16, 1),                     # rows of whole 16-byte units, any height
    (61, 64, 9, 2), (37, 29, 9, 2), (129, 72, 16, 2), (5, 300, 64, 2),    # other rows
    (3, 64, 9, 0), (64, 3, 9, 0), (64, 64, 129, 0),                       # a side below 4, a radius above 128
    (64, 64, 5, 0), (61, 64, 8, 0)])
def test_passes_by_image(w, h, r, want):
    blurred(w, h, r, want)


# r * w * h from 29,000,000 on with tensor maps (r >= 6), from 38,000,000 without (r >= 7)
@pytest.mark.parametrize("w,h,r,want", [
    (2200, 2197, 6, 1), (2200, 2196, 6, 0), (2400, 2400, 5, 0), (1904, 1904, 8, 1), (1904, 1903, 8, 0),
    (2331, 2329, 7, 2), (2331, 2328, 7, 0), (2701, 2700, 6, 0), (2181, 2178, 8, 2), (2181, 2177, 8, 0)])
def test_small_radii(w, h, r, want):
    assert (r * w * h >= (29000000 if w % 4 == 0 else 38000000) and r >= (6 if w % 4 == 0 else 7)) == (want > 0)
    blurred(w, h, r, want)


def test_other_modes_are_told_apart():
    img = wl.premultiplied_image(3, 129, 72)
    for mode in (1, 0):
        px.blur_config(mode)
        g = px.Image.from_numpy(img)
        g.blur(16)
        assert px.last_blur_ring() == 0 and px.last_blur_kernel() == mode
        px.blur_config(3)
        h = px.Image.from_numpy(img)
        h.blur(16)
        assert px.last_blur_ring() == 2
        assert np.array_equal(g.to_numpy(), h.to_numpy())
