"""Runs where the memory left does not hold the faster kernels' scratch.

The process' share of the device is cut to the memory of a full run less part of
what that run takes beyond the least scratch. The run then takes the least
scratch and returns the same bits.
"""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(kind):
    import gradenna_b200 as gb
    from gradenna_b200.fdtd3d import simulate_3d

    steps = 20
    wave = np.sin(0.2 * np.arange(steps))
    if kind == "2d":
        g = gb.Grid2D(1024, 1024, 1e-3, 1e-3)
        r = gb.simulate_tm(g, dtype=torch.float32, cpml=gb.CPMLSpec(12), source_ij=[(500, 400)],
                           source_current=wave[:, None], probe_ij=[(510, 400)], dft_freqs=(3e9,),
                           dft_monitors=[(0, 450, 350, 550, 450)])
        return [r.ez, r.hx, r.hy, r.probe_ez, *r.monitors]
    g = gb.Grid3D(220, 210, 160, 1e-3, 1e-3, 1e-3)
    r = simulate_3d(g, dtype=torch.float32, cpml=gb.CPMLSpec(8), source_current=wave,
                    source_ijk=(100, 100, 80), probe_ijk=((104, 100, 80),))
    return [r.ex, r.ey, r.ez, r.hx, r.hy, r.hz, r.probe_ez]


@pytest.mark.parametrize("kind", ["2d", "3d"])
def test_short_of_memory(kind, monkeypatch):
    from gradenna_b200 import _native

    want = [x.cpu() for x in _call(kind)]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    # Peak of a full run, and its scratch.
    asked = []
    scratch = _native.scratch

    def watch(size, least, *a):
        for fn in (size, least):
            n = ctypes.c_size_t()
            _native.check(fn(ctypes.byref(a[0]), ctypes.byref(a[1]), int(a[2]), ctypes.byref(n)))
            asked.append(n.value)
        t = scratch(size, least, *a)
        asked.append(t.numel())
        return t

    monkeypatch.setattr(_native, "scratch", watch)
    torch.cuda.reset_peak_memory_stats()
    _call(kind)
    torch.cuda.synchronize()
    size, least, got = asked
    assert got == size > least + (32 << 20)
    peak = torch.cuda.max_memory_reserved()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    asked.clear()
    try:
        torch.cuda.set_per_process_memory_fraction((peak - (size - least) / 2) / total)
        out = [x.cpu() for x in _call(kind)]
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert asked[2] == least
    for a, b in zip(want, out):
        assert torch.equal(a, b)
