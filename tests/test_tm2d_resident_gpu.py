"""GPU check of the register-resident 2D kernels.

Runs that fit the chip take them; the tile kernels, which any setting of
GDN_TM_KERNEL other than 'resident' selects, do the same arithmetic in the same
order. So both give the same bits (tolerance zero): fields, probe and port
records, running DFT and monitors. The sizes cover every kind of launch (one to
many rectangles, general shapes alone, the largest kind), no CPML, grids
smaller than a tile, odd extents, step counts that end inside a block of four
steps, inside a partial DFT sum of 32 and in a second segment; points lie
anywhere, on each other, in the corners and in the slabs, and monitor boxes
overlap. Where one list names a cell twice the second current is zero: the tile
kernels add such entries in any order.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [  # nx, ny, npml, steps
    (33, 30, 0, 37), (32, 29, 10, 50), (70, 53, 8, 1061), (64, 1000, 9, 70),
    (200, 300, 16, 335), (517, 384, 12, 130), (1024, 1024, 16, 66), (1300, 1111, 16, 34),
]


def _run(nx, ny, npml, steps, dtype, layout):
    import gradenna_b200 as gb

    rng = np.random.default_rng(nx + 7 * ny + steps)
    grid = gb.Grid2D(nx, ny, 1e-3, 1.1e-3)

    def cells(n):
        c = np.unique(np.stack([rng.integers(1, nx - 2, n), rng.integers(1, ny - 2, n)], 1), axis=0)
        return np.concatenate([c, c[: n // 4]])  # some twice

    def drive(ij, scale):
        x = rng.normal(size=(steps, len(ij))) * scale
        x[:, len(np.unique(ij, axis=0)):] = 0
        return torch.as_tensor(x, dtype=dtype, device="cuda")

    src, mx, my = cells(60), cells(40), cells(40)
    t = (np.arange(steps) + 0.5) * grid.dt
    wave = np.sin(2 * np.pi * 4e9 * t)
    kw = dict(
        dtype=dtype, cpml=gb.CPMLSpec(npml),
        eps_r=1.0 + 3.0 * rng.random((nx, ny)), sigma=0.1 * rng.random((nx, ny)),
        source_ij=src, source_current=drive(src, 1.0),
        mx_ij=mx, mx_current=drive(mx, 1e-3), my_ij=my, my_current=drive(my, 1e-3),
        probe_ij=np.concatenate([cells(50), [[0, 0], [nx - 1, ny - 1]]]),
        ports=tuple(gb.Port((int(i), int(j)), 30.0 + k, wave if k < 2 else None)
                    for k, (i, j) in enumerate(np.unique(np.concatenate([cells(5), src[:2]]), axis=0))),
        dft_freqs=(2e9, 4e9, 5e9))
    if layout == "boxes":
        kw["dft_monitors"] = [(0, 3, 5, nx - 2, ny - 7), (1, 1, 2, 4, ny - 2), (2, 0, 1, nx - 2, 3),
                              (0, nx // 2, ny // 2, nx // 2 + 1, ny // 2 + 1), (1, 5, 6, 9, 9)]
    elif layout == "many":
        kw["dft_monitors"] = [(k % 3, k % 7, 1 + k % 5, nx - 2 - k % 3, 6 + k % 11) for k in range(40)]
    r = gb.simulate_tm(grid, **kw)
    out = [r.probe_ez, r.ez, r.hx, r.hy, r.port_v, r.port_i, r.dft_ez, r.dft_hx, r.dft_hy]
    return [x for x in out + list(r.monitors or []) if x is not None]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_resident_kernels_match_the_tile_kernels(size, dtype, monkeypatch):
    for layout in ("full", "boxes", "many"):
        monkeypatch.setenv("GDN_TM_KERNEL", "tile")
        want = _run(*size, dtype, layout)
        monkeypatch.delenv("GDN_TM_KERNEL")
        got = _run(*size, dtype, layout)
        assert len(want) == len(got)
        for a, b in zip(want, got):
            assert torch.isfinite(torch.view_as_real(b) if b.is_complex() else b).all()
            assert torch.equal(a, b)
