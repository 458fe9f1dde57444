"""The setup kernel at the edges of its split: numbers of curves and lines
around the lanes, groups and CTAs they are shared out over, curves whose steps
stay, double, halve far or end early, images above 4096 rows, and paths that
fail, byte for byte against the oracle."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _init():
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)


def path(kinds, w, h, seed, spread=1.0):
    """A move, then lines (0), quadratics (1) and cubics (2) between random points, closed."""
    rs = np.random.RandomState(seed)
    at = rs.rand(2) * (w, h)
    cmds = [1.0, at[0], at[1]]
    for k in kinds:
        pts = []
        for _ in range(k + 1):
            at = np.clip(at + (rs.rand(2) - 0.5) * 2 * spread * np.array((w, h)), 0, (w, h))
            pts += [at[0], at[1]]
        cmds += [[2.0, 7.0, 5.0][k]] + pts
    return np.asarray(cmds + [0.0], np.float32)


def check(cmds, w, h, transform=None, winding=0, scene=True):
    ref = pxo.new_image(w, h)
    pxo.fill_path(ref, cmds, [0.1, 0.7, 0.4, 0.8], 1.0, 0, transform, winding)
    paint = px.Paint(color=(0.1, 0.7, 0.4, 0.8))
    img = px.Image(w, h)
    img.fill_path(cmds, paint, transform, winding)
    assert np.array_equal(img.to_numpy(), ref)
    if scene:
        sc = px.Scene()
        sc.fill_path(cmds, paint, transform, winding)
        img = px.Image(w, h)
        img.draw_scene(sc)
        assert np.array_equal(img.to_numpy(), ref)


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 600,
                               2100])
@pytest.mark.parametrize("kind", [1, 2, 3])
def test_numbers_of_curves(n, kind):
    kinds = [kind] * n if kind < 3 else [(k * 7 + n) % 3 for k in range(n)]
    check(path(kinds, 300, 120, n, 1.0 if n < 300 else 0.05), 300, 120, winding=n % 2)


@pytest.mark.parametrize("lines,curves", [(300, 1), (1000, 4), (5000, 0), (5000, 9), (20000, 40), (63, 0), (257, 2)])
def test_many_lines_few_curves(lines, curves):
    kinds = [0] * lines
    for k in range(curves):
        kinds[(k * 7919) % lines] = 2
    check(path(kinds, 400, 333, lines, 0.03), 400, 333, scene=lines < 6000)


@pytest.mark.parametrize("size", [3, 40, 700, 2500])
def test_step_patterns(size):
    s = float(size)
    cubics = [
        [0, 0, s, 0, s, s],                    # an arc-like curve
        [s * 3, 0, -s * 2, s * 0.5, s, s],     # a loop
        [s, 0, s, 0, s, s],                    # a cusp's control points together
        [0, s * 1e-3, s * 1e-3, 0, s, s * 1e-3],
        [s * 0.3, s * 0.3, s * 0.6, s * 0.6, s * 0.9, s * 0.9],  # a straight one
        [s * 5, s * 5, -s * 4, s * 5, s * 0.1, s],
    ]
    cmds = [1.0, s * 0.1, s * 0.1]
    for c in cubics:
        cmds += [5.0] + c
    for q in ([0, s, s, s * 0.5], [s, s, s * 0.2, s * 0.1], [s * 9, -s * 3, s * 0.5, s * 0.9]):
        cmds += [7.0] + q
    cmds = np.asarray(cmds + [0.0], np.float32)
    w = min(size, 900)
    check(cmds, w, w)
    check(cmds, w, w, [0.7, 0.2, 0, -0.3, 1.4, 0, 4.25, -3.5, 1], 1)


@pytest.mark.parametrize("h", [4091, 4092, 4093, 4100, 9000])
def test_tall_images(h):
    check(path([2, 0, 1, 2, 0, 2, 2, 1, 0, 0], 9, h, h), 9, h)
    check(path([k % 3 for k in range(90)], 9, h, h, 0.2), 9, h)


@pytest.mark.parametrize("at", [0, 5, 400])
def test_failing_curves(at):
    """A curve that cannot be discretised fails the call whatever CTA meets it, and draws nothing."""
    cmds = path([2] * 420, 300, 300, 4, 0.2)
    bad = cmds.copy()
    bad[3 + at * 7 + 1:3 + at * 7 + 5] = [1e7, -1e7, -1e7, 1e7]
    ref = pxo.new_image(300, 300)
    with pytest.raises(pxo.OracleError) as want:
        pxo.fill_path(ref, bad, [0, 0, 0, 1])
    img = px.Image(300, 300)
    with pytest.raises(px.PixieError) as got:
        img.fill_path(bad, px.Paint(color=(0, 0, 0, 1)))
    assert str(got.value) == str(want.value)
    assert not img.to_numpy().any()
    img.fill_path(cmds, px.Paint(color=(0, 0, 0, 1)))  # and the next call is whole
    pxo.fill_path(ref, cmds, [0, 0, 0, 1])
    assert np.array_equal(img.to_numpy(), ref)
