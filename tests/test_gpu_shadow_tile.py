"""The one-pass shadow kernel at every radius and spread it takes: each radius
residue mod 4 (the weights' place in the staged words), each spread on both
sides of a word, |spread| + radius at the limit, and tiles that end inside a
word, on random alpha -- bytes equal to the oracle's (integer sums: no
tolerance)."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo
from pixie_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

CASES = [(sp, r) for r in range(0, 33) for sp in ((32 - r), -(32 - r), (r * 5 + 1) % (33 - r))]


@pytest.mark.parametrize("sp,r", CASES)
def test_every_radius_and_spread(sp, r):
    px.lib().pxg_init(0)
    w, h = 61 + (r * 7 + sp) % 9, 127 + (r + sp * 3) % 5
    img = wl.premultiplied_image(r * 100 + sp, w, h)
    off = (r % 5 - 2, sp % 7 - 3)
    col = [0.3, 0.8, 0.5, 0.9]
    ref = pxo.shadow(img, off[0], off[1], sp, r, col)
    out = px.Image.from_numpy(img).shadow(off, sp, r, col)
    assert np.array_equal(out.to_numpy(), ref)
