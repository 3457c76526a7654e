"""The memory estimate against the library's own layouts (no device needed).

estimate.py counts what a run needs at least: gdn_*_workspace_least. The 2D
figures follow the layout's padding (points and tables aside: 1 MiB); the 3D
ones count unpadded cells, so they lie up to 12 % lower.
"""

import ctypes

import pytest


def _sizes(size, least, p, pts, f64):
    from gradenna_b200 import _native

    out = []
    for fn in (size, least):
        n = ctypes.c_size_t()
        _native.check(fn(ctypes.byref(p), ctypes.byref(pts), f64, ctypes.byref(n)))
        out.append(n.value)
    return out


@pytest.mark.parametrize("nx,ny,f64,freqs", [(1024, 1024, 0, 4), (1024, 900, 0, 0), (280, 280, 1, 1),
                                             (100, 130, 0, 2), (1024, 1024, 1, 2)])
def test_least_2d_scratch_is_the_estimate(nx, ny, f64, freqs):
    import gradenna_b200 as gb
    from gradenna_b200 import _native
    from gradenna_b200.estimate import fdtd2d_memory_estimate

    lib = _native.load()
    p = _native.TmParams()
    p.nx, p.ny, p.npml, p.n_steps, p.n_freq = nx, ny, 10, 4000, freqs
    size, least = _sizes(lib.gdn_tm_workspace_size, lib.gdn_tm_workspace_least, p,
                         _native.TmPoints(), f64)
    est = fdtd2d_memory_estimate(gb.Grid2D(nx, ny, 1e-3, 1e-3), 4000, n_dft_freqs=freqs,
                                 dtype="float64" if f64 else "float32")
    want = (est["b200_planes_gb"] + est["b200_ring_gb"]) * 2**30
    assert least <= size
    assert abs(least - want) <= 2**20


@pytest.mark.parametrize("n,f64", [((160, 160, 64), 0), ((97, 83, 61), 1), ((300, 300, 300), 0)])
def test_least_3d_scratch_is_the_estimate(n, f64):
    import gradenna_b200 as gb
    from gradenna_b200 import _native, fdtd3d
    from gradenna_b200.estimate import fdtd3d_memory_estimate

    lib = _native.load()
    p = fdtd3d.YeeParams()
    p.nx, p.ny, p.nz, p.npml, p.n_steps = *n, 8, 100
    size, least = _sizes(lib.gdn_yee_workspace_size, lib.gdn_yee_workspace_least, p,
                         fdtd3d.YeePoints(), f64)
    b = 8 if f64 else 4
    vol = (n[0] + 2) * (n[1] + 2) * ((n[2] + 2 + 3) // 4 * 4)
    assert abs(size - least - 2 * vol * b) <= 512  # the padded ca and cb
    est = fdtd3d_memory_estimate(gb.Grid3D(*n, 1e-3, 1e-3, 1e-3), 100,
                                 dtype="float64" if f64 else "float32")
    want = est["b200_forward_gb"] * 2**30 - 3 * n[0] * n[1] * n[2] * b  # without the caller's arrays
    assert 0.88 * least <= want <= least
