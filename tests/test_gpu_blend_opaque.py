"""Every blend mode over opaque backdrops, from opaque sources and from all
alphas in between (the composites that need no division), and over backdrops
of every alpha beside them, byte for byte against the oracle."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo

pytestmark = pytest.mark.gpu


def pixels(n, alpha, seed):
    rs = np.random.RandomState(seed)
    a = np.full(n, alpha) if alpha is not None else rs.randint(0, 256, n)
    rgb = (rs.randint(0, 256, (n, 3)) * a[:, None] + 127) // 255
    return np.concatenate([rgb, a[:, None]], 1).astype(np.uint8).reshape(256, -1, 4)


@pytest.mark.parametrize("mode", range(20))
def test_opaque_backdrops_and_sources(mode):
    px.lib().pxg_init(0)
    n = 256 * 96
    for back, src in [(255, None), (255, 255), (None, 255), (254, None), (255, 1), (255, 0), (0, None)]:
        b, s = pixels(n, back, 11 + mode), pixels(n, src, 77 + mode)
        ref = b.copy()
        pxo.draw(ref, s, 0, 0, mode)
        img = px.Image.from_numpy(b)
        img.draw(px.Image.from_numpy(s), (0, 0), mode)
        assert np.array_equal(img.to_numpy(), ref), f"mode {mode} backdrop alpha {back} source alpha {src}"
