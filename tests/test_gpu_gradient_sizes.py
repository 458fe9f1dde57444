"""Gradients on images around the size from which a thread takes four pixels
(4096 pixels per SM: 622,592 on 152 SMs), whole images and paths, ragged widths,
byte for byte against the oracle."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo
from pixie_gb300.paths import parse_path

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [3, 4, 5])
@pytest.mark.parametrize("w,h", [(622592, 1), (789, 789), (790, 789), (1301, 503), (1024, 609)])
@pytest.mark.parametrize("blend,nstops", [(0, 3), (0, 20), (12, 5)])
def test_gradient_sizes(kind, w, h, blend, nstops):
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)
    rng = np.random.default_rng(kind * 100 + w + nstops)
    f = lambda v: float(np.float32(v))
    dst = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    dst[rng.random((h, w)) < 0.3, 3] = 0
    stops = [(tuple(f(v) for v in rng.uniform(0, 1, 4)), f(p)) for p in np.sort(rng.uniform(-0.1, 1.1, nstops))]
    handles = [(f(rng.uniform(-2, w + 2)), f(rng.uniform(-2, h + 2))) for _ in range(2 if kind == 3 else 3)]
    corners = [(0.2 * w, 0.1 * h), (0.95 * w, 0.2 * h), (0.8 * w, 0.9 * h), (0.1 * w, 0.7 * h)]
    path = parse_path("M " + " L ".join(f"{x} {y}" for x, y in corners) + " Z").array()
    paint = dict(kind=kind, handles=handles, stops=stops, opacity=f(0.7), blend=blend)
    ref = dst.copy()
    pxo.fill_path_paint(ref, path, paint, None, 0)
    img = px.Image.from_numpy(dst)
    img.fill_path(path, px.Paint((0, 0, 0, 0), f(0.7), blend, kind=kind, handles=handles, stops=stops))
    assert np.array_equal(img.to_numpy(), ref)
