"""Scenes whose coverage would not fit its arena are drawn in chunks of paths:
the same bytes as the calls one by one."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo
from pixie_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("paths", [64, 65, 79, 300])
def test_chunks_of_paths(paths):
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)
    items = [it for it in wl.dense_scene(11, n_paths=paths, size=64.0)]
    ref, sc, n = pxo.new_image(64, 64), px.Scene(), 0
    for it in items:
        if it["kind"] != "fill":
            continue
        paint = px.Paint(color=it["color"], blend_mode=it["blend"])
        for _ in range(2):
            try:
                pxo.fill_path(ref, it["cmds"], it["color"], 1.0, it["blend"], None, it["winding"])
            except Exception:
                continue
            sc.fill_path(it["cmds"], paint, None, it["winding"])
            n += 1
    px.scene_config(0, 400000)  # 78 canvases of 80 x 64
    try:
        img = px.Image(64, 64)
        img.draw_scene(sc)
        assert px.last_fill_stats()["paths"] == n
        assert np.array_equal(img.to_numpy(), ref)
    finally:
        px.scene_config(0, 4 << 30)
