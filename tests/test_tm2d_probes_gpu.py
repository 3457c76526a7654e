"""Blocks of probes: a run's time loop is no slower than on the tile kernels.

The time-domain gradient records every design cell. A rectangle that holds a
block reads it off by register; where one would hold thousands, the run takes
the tile kernels. Scattered probes, and probes that name a cell twice, go entry by
entry. Records are the same bits either way.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cells(n, kind):
    if kind == "twice":
        c = np.random.default_rng(n).integers(0, n, (3000, 2))
        return np.concatenate([c, c[:700]])
    a = n // 2 - kind // 2
    return np.stack(np.meshgrid(np.arange(a, a + kind), np.arange(a, a + kind), indexing="ij"),
                    -1).reshape(-1, 2)


@pytest.mark.parametrize("n,kind,dtype", [
    (640, 40, torch.float32), (1024, 40, torch.float32), (640, 200, torch.float32),
    (1024, 200, torch.float32), (280, 104, torch.float64), (200, "twice", torch.float32),
    (700, "twice", torch.float32)])
def test_blocks_of_probes(n, kind, dtype, monkeypatch):
    import gradenna_b200 as gb
    from gradenna_b200 import _native

    steps, cells = 300, _cells(n, kind)
    wave = np.sin(0.1 * np.arange(steps))

    def best():
        t = []
        for _ in range(6):
            torch.cuda.synchronize()
            _native.tm_loop_stats(reset=True)
            r = gb.simulate_tm(gb.Grid2D(n, n, 1e-3, 1e-3), dtype=dtype, cpml=gb.CPMLSpec(10),
                               source_ij=[(n // 2, n // 2)], source_current=wave[:, None],
                               probe_ij=cells)
            t.append(_native.tm_loop_stats(reset=True)[0])
        return min(t), r.probe_ez

    for _ in range(3):  # another process on the host can disturb a try
        mine, got = best()
        with monkeypatch.context() as m:
            m.setenv("GDN_TM_KERNEL", "tile")
            tile, want = best()
        assert torch.equal(want, got)
        if mine <= 1.05 * tile:  # the same kernels where a rectangle is crowded
            return
    assert mine <= 1.05 * tile
