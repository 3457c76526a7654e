"""2D runs whose rectangles hold many injections: an adjoint run's flux contour,
and a block of sources.

Injected values of a block are staged on the chip, as many as fit. The cases
have a few hundred in some rectangles (a contour of Jz, Mx and My), and more
than fit (a filled block). Results are those of the tile kernels, bit for bit
(the same arithmetic in the same order; no list names a cell twice), and the
contour run's time loop is no slower than theirs.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _contour(n, b):
    """Cells of the adjoint sources of the flux through the box (b, n - b - 1)."""
    lo, hi = b, n - b - 1
    s = np.arange(lo + 1, hi + 1)
    at = lambda i, j: np.stack(np.broadcast_arrays(i, j), 1)  # noqa: E731
    ez = [at(lo, s), at(lo + 1, s), at(hi, s), at(hi + 1, s),
          at(s, lo), at(s, lo + 1), at(s, hi), at(s, hi + 1)]
    return (np.unique(np.concatenate(ez), axis=0), np.concatenate([at(s, lo), at(s, hi)]),
            np.concatenate([at(lo, s), at(hi, s)]))


def _run(n, npml, steps, dtype, cells):
    import gradenna_b200 as gb

    rng = np.random.default_rng(n)
    ez, hx, hy = cells
    kw = {}
    for k, ij in (("source", ez), ("mx", hx), ("my", hy)):
        if len(ij):
            kw[f"{k}_ij"] = ij
            kw[f"{k}_current"] = torch.as_tensor(rng.normal(size=(steps, len(ij))), dtype=dtype,
                                                 device="cuda")
    r = gb.simulate_tm(gb.Grid2D(n, n, 1e-3, 1e-3), dtype=dtype, cpml=gb.CPMLSpec(npml),
                       dft_freqs=(2e9, 3e9), dft_monitors=[(0, n // 4, n // 4, n // 2, n // 2)],
                       sigma=0.1 * rng.random((n, n)), **kw)
    return [r.ez, r.hx, r.hy, *r.monitors]


@pytest.mark.parametrize("case", ["f32", "f64", "block"])
def test_many_injections_match_the_tile_kernels(case, monkeypatch):
    n, npml, dtype = (420, 12, torch.float64) if case == "f64" else (1024, 16, torch.float32)
    cells = _contour(n, 60 if case == "f64" else 150)
    if case == "block":
        i = np.stack(np.meshgrid(np.arange(300, 500), np.arange(300, 500), indexing="ij"), -1)
        cells = (i.reshape(-1, 2), cells[1], cells[2])
    monkeypatch.setenv("GDN_TM_KERNEL", "tile")
    want = _run(n, npml, 37, dtype, cells)
    monkeypatch.delenv("GDN_TM_KERNEL")
    got = _run(n, npml, 37, dtype, cells)
    for a, b in zip(want, got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
def test_contour_run_is_no_slower_than_the_tile_kernels(dtype, monkeypatch):
    from gradenna_b200 import _native

    n, npml, b = (1024, 16, 150) if dtype == torch.float32 else (420, 12, 60)
    cells = _contour(n, b)

    def best():
        t = []
        for _ in range(5):
            torch.cuda.synchronize()
            _native.tm_loop_stats(reset=True)
            _run(n, npml, 800, dtype, cells)
            t.append(_native.tm_loop_stats(reset=True)[0])
        return min(t)

    for _ in range(3):  # another process on the host can disturb a try
        mine = best()
        with monkeypatch.context() as m:
            m.setenv("GDN_TM_KERNEL", "tile")
            tile = best()
        if mine <= tile:
            return
    assert mine <= tile
