"""Outlines of a mask batch built on as many host threads as their pace asks for:
whatever the number, the batch is the one that adding them one by one makes,
and the first failing outline is the one reported.  Runs on the host only."""
import numpy as np
import pytest

import pixie_gb300 as px


def outline(n, seed):
    rs = np.random.RandomState(seed)
    pts = rs.rand(n, 2).astype(np.float32) * 90
    cmds = np.empty((n, 3), np.float32)
    cmds[:, 0] = 2.0
    cmds[0, 0] = 1.0
    cmds[:, 1:] = pts
    return np.concatenate([cmds.ravel(), [0.0]]).astype(np.float32)


BATCHES = [[3], [3] * 5, [2000] * 2, [2000] * 60, [5] * 240, [5] * 200 + [4000] * 40, [4000] * 40 + [5] * 200]


@pytest.mark.parametrize("lines", BATCHES, ids=lambda b: f"{len(b)}x{b[0]}-{b[-1]}")
@pytest.mark.parametrize("threads", [0, 1, 3])
def test_batches_are_whole(lines, threads):
    paths = [(outline(n, k), 90 + k % 3, 90, k % 2) for k, n in enumerate(lines)]
    m = px.Masks()
    m.add_paths(paths, threads)
    assert len(m) == len(lines)
    m.add_paths(paths[:1], threads)
    assert len(m) == len(lines) + 1


@pytest.mark.parametrize("at", [0, 3, 30, 59])
def test_first_failure_is_reported(at):
    paths = [(outline(1500, k), 90, 90, 0) for k in range(60)]
    paths[at] = (np.asarray([1, 2, np.inf, 0], np.float32), 90, 90, 0)
    if at < 59:
        paths[59] = (paths[59][0], 0, 90, 0)
    m = px.Masks()
    with pytest.raises(px.PixieError, match="non-finite"):
        m.add_paths(paths)
    assert len(m) == 0
