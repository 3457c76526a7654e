"""GPU check of the 3D step kernels at the edges of their vectors and classes.

A thread owns 16 bytes of cells of a row, and boxes within reach of a CPML slab
round differently from the others. The sizes below end rows at every remainder
of a vector, give rows of a few vectors and of many, and mix both classes along
every axis; points, the port and probes lie on first and last cells. Each run
is held to the numpy oracle, and a run whose scratch has no room for the padded
coefficients to the same run with it, bit for bit. Tolerances are those of the
other 3D parity tests (float64 1e-10; float32 1e-5 on records, 2e-3 on fields).
"""

import ctypes

import numpy as np
import pytest
import torch

from oracle import fdtd2d_np as o2
from oracle import fdtd3d_np as ref

pytestmark = pytest.mark.gpu

SIZES = [(9, 11, 7, 1), (8, 9, 10, 2), (12, 8, 9, 2), (10, 13, 8, 0), (11, 10, 33, 3),
         (30, 34, 99, 2), (7, 40, 66, 1)]
COMPS = ("ex", "ey", "ez", "hx", "hy", "hz")


def _np(x):
    return x.detach().cpu().numpy() if isinstance(x, torch.Tensor) else np.asarray(x)


def _rel(a, b):
    a, b = _np(a), _np(b)
    return float(np.max(np.abs(a - b)) / (np.max(np.abs(b)) + 1e-300))


class _SmallScratch:
    """The library, reporting the scratch size without padded coefficients."""

    def __init__(self, lib, saved):
        self._lib, self._saved = lib, saved

    def __getattr__(self, name):
        return getattr(self._lib, name)

    def gdn_yee_workspace_size(self, p, pts, f64, out):
        st = self._lib.gdn_yee_workspace_size(p, pts, f64, out)
        size = ctypes.cast(out, ctypes.POINTER(ctypes.c_size_t)).contents
        size.value -= self._saved // 256 * 256
        return st


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_vector_edges(size, dtype, monkeypatch):
    import gradenna_b200 as gb
    from gradenna_b200 import _native
    from gradenna_b200.fdtd3d import simulate_3d

    nx, ny, nz, npml = size
    steps = 40
    rng = np.random.default_rng(nx + 10 * ny + 100 * nz)
    g, og = (m.Grid3D(nx, ny, nz, 1e-3, 1.1e-3, 0.9e-3) for m in (gb, ref))
    t = (np.arange(steps) + 0.5) * og.dt
    base = np.asarray(o2.gaussian_derivative(t, 10 * og.dt, 4 * og.dt), dtype)
    kw = dict(eps_r=1 + 3 * rng.random((nx, ny, nz)), sigma=0.05 * rng.random((nx, ny, nz)),
              source_ijk=(nx // 2, ny // 2, nz - 2), source_current=base,
              source_x_ijk=(nx - 2, ny // 2, nz // 2), source_x_current=(0.7 * base).astype(dtype),
              source_y_ijk=(nx // 2, ny - 2, 1), source_y_current=(0.4 * base).astype(dtype),
              mx_ijk=(1, ny // 2, 0), mx_current=(3 * base).astype(dtype),
              mz_ijk=(nx // 2, 0, nz - 1), mz_current=(2 * base).astype(dtype),
              port_ijk=(nx // 2, ny // 2, min(nz - 2, 31)), port_voltage=(0.5 * base).astype(dtype),
              probe_ijk=((1, 1, 0), (nx - 2, ny - 2, nz - 2), (nx // 2, ny // 2, min(nz - 2, 32))),
              dft_freqs=(3e9,))
    # A source on the port's edge enters the port's update, which the oracle does
    # not model: it is compared without that source.
    common = dict(kw)
    if kw["source_ijk"] == kw["port_ijk"]:
        del common["source_ijk"], common["source_current"]
    r = simulate_3d(g, cpml=gb.CPMLSpec(npml), dtype=dtype, **common)
    o = ref.simulate_3d(og, cpml=o2.CPMLSpec(npml), dtype=dtype, **common)
    rec, fld = (1e-10, 1e-10) if dtype == np.float64 else (1e-5, 2e-3)
    for nm in ("probe_ez", "port_v", "port_i"):
        assert _rel(getattr(r, nm), getattr(o, nm)) <= rec, nm
    for nm in COMPS:
        assert _rel(getattr(r, nm), getattr(o, nm)) <= fld, nm

    r = simulate_3d(g, cpml=gb.CPMLSpec(npml), dtype=dtype, return_state=True, **kw)
    vol = (nx + 2) * (ny + 2) * ((nz + 2 + 3) // 4 * 4)
    lib = _SmallScratch(_native.load(), 2 * vol * np.dtype(dtype).itemsize)
    monkeypatch.setattr(_native, "load", lambda: lib)
    s = simulate_3d(g, cpml=gb.CPMLSpec(npml), dtype=dtype, return_state=True, **kw)
    assert torch.equal(r.state, s.state)
    for nm in ("probe_ez", "port_v", "port_i"):
        assert torch.equal(getattr(r, nm), getattr(s, nm)), nm
