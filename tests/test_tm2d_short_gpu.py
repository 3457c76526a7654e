"""Runs of a few steps with scattered points: no slower than on the tile kernels.

Such a call is mostly set-up: tables of points, their upload, and the launches.
Whole calls, the best of many; results are the same bits.
"""

import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,points,dtype", [(1024, 2000, torch.float32), (480, 2000, torch.float64),
                                            (280, 300, torch.float32), (640, 20000, torch.float32)])
def test_few_steps_with_scattered_points(n, points, dtype, monkeypatch):
    import gradenna_b200 as gb

    rng = np.random.default_rng(n)
    c = rng.permutation((n - 4) ** 2)[:2 * points]
    cells = np.stack([c // (n - 4) + 2, c % (n - 4) + 2], 1)
    steps = 6
    cur = torch.as_tensor(rng.normal(size=(steps, points)), dtype=dtype, device="cuda")

    def call():
        return gb.simulate_tm(gb.Grid2D(n, n, 1e-3, 1e-3), dtype=dtype, cpml=gb.CPMLSpec(10),
                              source_ij=cells[:points], source_current=cur, probe_ij=cells[points:])

    def best():
        t = []
        for _ in range(20):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            r = call()
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        return min(t), [r.ez, r.hx, r.hy, r.probe_ez]

    for _ in range(3):  # another process on the host can disturb a try
        mine, got = best()
        with monkeypatch.context() as m:
            m.setenv("GDN_TM_KERNEL", "tile")
            tile, want = best()
        for a, b in zip(want, got):
            assert torch.equal(a, b)
        if mine <= 1.15 * tile:
            return
    assert mine <= 1.15 * tile
