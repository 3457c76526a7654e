"""Full-grid phasors: a run's time loop is no slower than on the tile kernels.

Tones and types at both ends of what the DFT's sums are compiled for (up to 4, 8
and 16 tones; sums in float32 and float64), on grids whose monitor ring holds
many steps and few. The results of both are the same bits.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [(517, 4, torch.float32, np.complex64), (517, 8, torch.float32, np.complex64),
         (400, 16, torch.float32, np.complex128), (1024, 16, torch.float32, np.complex128),
         (400, 9, torch.float64, np.complex64), (400, 16, torch.float64, np.complex128),
         (280, 5, torch.float64, np.complex128), (140, 16, torch.float32, np.complex64),
         (640, 1, torch.float32, np.complex64), (1024, 4, torch.float32, np.complex64)]


@pytest.mark.parametrize("n,tones,dtype,cdtype", CASES)
def test_full_grid_phasors(n, tones, dtype, cdtype, monkeypatch):
    import gradenna_b200 as gb
    from gradenna_b200 import _native

    steps = 480
    wave = np.sin(0.1 * np.arange(steps))

    def call():
        return gb.simulate_tm(gb.Grid2D(n, n, 1e-3, 1e-3), dtype=dtype, cpml=gb.CPMLSpec(10),
                              source_ij=[(n // 2, n // 2)], source_current=wave[:, None],
                              dft_freqs=tuple(np.linspace(1e9, 3e9, tones)), dft_dtype=cdtype)

    def best():
        t = []
        for _ in range(5):
            torch.cuda.synchronize()
            _native.tm_loop_stats(reset=True)
            r = call()
            t.append(_native.tm_loop_stats(reset=True)[0])
        return min(t), [r.ez, r.dft_ez, r.dft_hx, r.dft_hy]

    for _ in range(3):  # another process on the host can disturb a try
        mine, got = best()
        with monkeypatch.context() as m:
            m.setenv("GDN_TM_KERNEL", "tile")
            tile, want = best()
        for a, b in zip(want, got):
            assert torch.equal(a, b)
        if mine <= tile:
            return
    assert mine <= tile
