"""Many small monitors in a rectangle: same bits as the tile kernels, no slower.

Up to 32, up to 544 and more monitor parts in one rectangle of the resident
kernels take three ways to the threads that hold the cells.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

F32, F64 = torch.float32, torch.float64


def _call(n, dtype, steps, count, size, across=20):
    import gradenna_b200 as gb

    rng = np.random.default_rng(n)
    step = size + 1
    mons = [(q % 3, 80 + q // across * step, 80 + q % across * step,
             80 + q // across * step + size, 80 + q % across * step + size) for q in range(count)]
    wave = torch.as_tensor(rng.normal(size=(steps, 1)), dtype=dtype, device="cuda")
    return lambda: gb.simulate_tm(gb.Grid2D(n, n, 1e-3, 1e-3), dtype=dtype, cpml=gb.CPMLSpec(10),
                                  source_ij=[(90, 90)], source_current=wave, dft_freqs=(2e9, 3e9),
                                  dft_monitors=mons)


def _loop(call):
    from gradenna_b200 import _native

    t = []
    for _ in range(5):
        torch.cuda.synchronize()
        _native.tm_loop_stats(reset=True)
        r = call()
        t.append(_native.tm_loop_stats(reset=True)[0])
    return min(t), [r.ez, r.hx, r.hy, *r.monitors]


@pytest.mark.parametrize("n,dtype,count,size", [
    (1024, F32, 200, 3), (640, F32, 100, 3), (640, F32, 200, 1), (640, F32, 200, 3),
    (420, F32, 200, 3), (420, F64, 200, 3), (420, F64, 200, 1)])
def test_no_slower_than_the_tile_kernels(n, dtype, count, size, monkeypatch):
    call = _call(n, dtype, 160, count, size)
    for _ in range(3):  # another process on the host can disturb a try
        mine, got = _loop(call)
        with monkeypatch.context() as m:
            m.setenv("GDN_TM_KERNEL", "tile")
            tile, want = _loop(call)
        for a, b in zip(want, got):
            assert torch.equal(a, b)
        if mine <= tile:
            return
    assert mine <= tile


@pytest.mark.parametrize("n,dtype,count,size,across", [
    (640, F32, 33, 1, 20), (640, F32, 800, 1, 40), (880, F32, 640, 2, 30), (420, F64, 600, 1, 24),
    (150, F32, 300, 1, 20)])
def test_bits(n, dtype, count, size, across, monkeypatch):
    call = _call(n, dtype, 37, count, size, across)
    got = call()
    monkeypatch.setenv("GDN_TM_KERNEL", "tile")
    want = call()
    assert torch.equal(want.ez, got.ez)
    for a, b in zip(want.monitors, got.monitors):
        assert torch.equal(a, b)
