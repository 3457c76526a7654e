"""A 2D run whose wait between two rectangles runs out returns NaN everywhere.

The library's hook keeps one rectangle's words of a block back, with waits of a
few milliseconds: its neighbours give up and every rectangle leaves. Nothing of
such a run may look like a result: fields, phasors, and the probe and port
records (whose steps past the failure nothing wrote) are NaN, the run is
counted, and the next run on the same stream is right. The block lies in the
first or in the second segment of 1024 steps.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("block", [2, 300])
def test_run_out_wait_voids_every_output(block, dtype):
    import gradenna_b200 as gb
    from gradenna_b200 import _native

    grid = gb.Grid2D(96, 90, 1e-3, 1e-3)
    wave = np.sin(2 * np.pi * 4e9 * (np.arange(1500) + 0.5) * grid.dt)

    def run():
        r = gb.simulate_tm(grid, dtype=dtype, cpml=gb.CPMLSpec(8), dft_freqs=(3e9, 4e9),
                           source_ij=[(40, 40)], source_current=wave[:, None],
                           ports=(gb.Port((50, 30), 50.0, wave),), probe_ij=[(30, 60), (70, 20)],
                           dft_monitors=[(0, 10, 10, 60, 60), (1, 5, 5, 80, 6)])
        return [r.ez, r.hx, r.hy, r.probe_ez, r.port_v, r.port_i, *r.monitors]

    want = run()
    _native.tm_timeouts()
    try:
        _native.check(_native.load().gdn_tm_inject_timeout(block))
        bad = run()
    finally:
        _native.check(_native.load().gdn_tm_inject_timeout(-1))
    good = run()
    assert _native.tm_timeouts() == 1
    for a, b, c in zip(want, bad, good):
        assert bool(torch.isnan(torch.view_as_real(b) if b.is_complex() else b).all())
        assert torch.equal(a, c)
    assert _native.tm_timeouts() == 0
