"""Scenes of many small paths on a tall canvas: the workspace is bounded by the
paths' rows, so they are drawn in several launches although their coverage would
fit one; servers whose coverage arena holds none of their jobs' paths."""
import numpy as np
import pytest

import pixie_gb300 as px
from oracle import pxo
from pixie_gb300 import workloads as wl

pytestmark = pytest.mark.gpu
KERNELS = 6  # of a chunk: setup, recording, rows of many crossings (two and the rest), drawing


@pytest.fixture(scope="module", autouse=True)
def _init():
    px.lib().pxg_init(0)
    pxo.set_golden_mode(False)


def test_many_small_paths_on_many_rows():
    w, h, n = 8, 4000, 20000  # 80 million path rows
    rs = np.random.RandomState(1)
    ref = pxo.new_image(w, h)
    items = []
    for k in range(n):
        x, y = rs.rand() * 6, rs.rand() * (h - 4)
        cmds = np.asarray([1, x, y, 2, x + 2.3, y + 0.4, 2, x + 1.1, y + 3.2, 0], np.float32)
        color = [float(v) for v in rs.rand(4).astype(np.float32)]
        items.append({"kind": "fill", "cmds": cmds, "color": color, "blend": k % 3, "winding": 0})
        pxo.fill_path(ref, cmds, color, 1.0, k % 3, None, 0)
    sc = px.Scene()
    sc.record_batch(items)
    assert len(sc) == n
    img = px.Image(w, h)
    before = px.launch_count()
    img.draw_scene(sc)
    assert px.launch_count() - before >= 3 * KERNELS  # 32 million rows a chunk at most
    assert px.last_fill_stats()["paths"] == n
    assert np.array_equal(img.to_numpy(), ref)


def test_jobs_larger_than_the_coverage_arena():
    """Jobs none of which the arena holds go together, as they did before there were chunks."""
    side, jobs = 200, 6
    scenes, refs = [], []
    for k in range(jobs):
        sc, ref = px.Scene(), pxo.new_image(side, side)
        for it in wl.dense_scene(k + 1, n_paths=40, size=float(side)):
            if it["kind"] != "fill":
                continue
            try:
                pxo.fill_path(ref, it["cmds"], it["color"], 1.0, it["blend"], None, it["winding"])
            except Exception:
                continue
            sc.fill_path(it["cmds"], px.Paint(color=it["color"], blend_mode=it["blend"]), None, it["winding"])
        scenes.append(sc)
        refs.append(ref)
    px.scene_config(0, 4096)
    try:
        server = px.Server()
        before = px.launch_count()
        ids = [server.submit(s, side, side, 0) for s in scenes]
        while server.pending():
            server.step()
        server.poll()
        for i, ref in zip(ids, refs):
            assert np.array_equal(server.take(i)[0], ref)
        assert px.launch_count() - before < 2 * KERNELS + 4 * jobs
    finally:
        px.scene_config(0, 4 << 30)
