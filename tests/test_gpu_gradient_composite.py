"""A path filled with a gradient: the colours go through the mask and onto the
image in one kernel under NormalBlend, through a masked paint image under the
others.  Image sizes around groups of four pixels and rows, numbers of stops on
both sides of the inline limit, opacities down to 0 of 255, backdrops that are
not premultiplied (a transparent pixel with colour) -- bytes equal to the
oracle's (no tolerance: the same operations)."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo
from pixie_gb300.paths import parse_path

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (2, 1), (3, 5), (5, 3), (4, 4), (31, 33), (127, 130), (600, 411)]


@pytest.mark.parametrize("kind", [3, 4, 5])
@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("blend,nstops,opacity", [(0, 1, 1.0), (0, 16, 0.5), (0, 17, 0.004), (0, 3, 0.0015), (17, 2, 0.7),
                                                  (10, 16, 1.0), (12, 17, 0.3), (18, 4, 0.9)])
def test_gradient_composite(kind, w, h, blend, nstops, opacity):
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)
    rng = np.random.default_rng(kind * 1000 + w * 31 + h + nstops)
    f = lambda v: float(np.float32(v))
    dst = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    dst[rng.random((h, w)) < 0.3, 3] = 0
    stops = [(tuple(f(v) for v in rng.uniform(0, 1, 4)), f(p)) for p in np.sort(rng.uniform(-0.1, 1.1, nstops))]
    handles = [(f(rng.uniform(-2, w + 2)), f(rng.uniform(-2, h + 2))) for _ in range(2 if kind == 3 else 3)]
    corners = [(0.2 * w, 0.1 * h), (0.95 * w, 0.2 * h), (0.8 * w, 0.9 * h), (0.1 * w, 0.7 * h)]
    path = parse_path("M " + " L ".join(f"{x} {y}" for x, y in corners) + " Z").array()
    paint = dict(kind=kind, handles=handles, stops=stops, opacity=f(opacity), blend=blend)
    ref = dst.copy()
    pxo.fill_path_paint(ref, path, paint, None, 0)
    img = px.Image.from_numpy(dst)
    img.fill_path(path, px.Paint((0, 0, 0, 0), f(opacity), blend, kind=kind, handles=handles, stops=stops))
    assert np.array_equal(img.to_numpy(), ref)
