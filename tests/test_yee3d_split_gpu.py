"""GPU check of the 3D step kernels' split: planes a CTA, and runs without CPML.

Sizes whose CTAs take 3 to 8 planes on 148 SMs, with last CTAs that hold fewer, and
grids without CPML, which have kernels of their own. Sources, the port and probes
lie on several planes of a CTA. Held to the numpy oracle with the tolerances of the
other 3D parity tests (float64 1e-10; float32 1e-5 on records, 2e-3 on fields).
"""

import numpy as np
import pytest

from oracle import fdtd2d_np as o2
from oracle import fdtd3d_np as ref

pytestmark = pytest.mark.gpu

COMPS = ("ex", "ey", "ez", "hx", "hy", "hz")
F32, F64 = np.float32, np.float64


def _rel(a, b):
    a, b = np.asarray(a.detach().cpu()), np.asarray(b)
    return float(np.max(np.abs(a - b)) / (np.max(np.abs(b)) + 1e-300))


@pytest.mark.parametrize("size,dtype", [
    ((64, 64, 64, 6, 8), F64), ((64, 64, 64, 0, 8), F64), ((101, 99, 98, 6, 5), F32),
    ((200, 30, 120, 6, 5), F64), ((30, 200, 120, 4, 5), F64), ((30, 200, 120, 0, 5), F32),
    ((97, 83, 61, 0, 6), F64), ((97, 83, 61, 0, 6), F32), ((17, 6, 5, 0, 20), F64),
    ((6, 17, 5, 0, 20), F32), ((5, 6, 37, 1, 20), F32)],
    ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else v.__name__)
def test_split(size, dtype):
    import gradenna_b200 as gb
    from gradenna_b200.fdtd3d import simulate_3d

    nx, ny, nz, npml, steps = size
    rng = np.random.default_rng(nx + nz)
    g, og = (m.Grid3D(nx, ny, nz, 1e-3, 1.1e-3, 0.9e-3) for m in (gb, ref))
    base = np.asarray(np.sin(0.5 * (np.arange(steps) + 0.5)), dtype)
    i, j, k = nx // 2, ny // 2, nz // 2
    kw = dict(eps_r=1 + 3 * rng.random((nx, ny, nz)), sigma=0.05 * rng.random((nx, ny, nz)),
              source_ijk=(i + 1, j, k), source_current=base,
              source_x_ijk=(i, j, k), source_x_current=(0.7 * base).astype(dtype),
              my_ijk=(i - 1, j, 1), my_current=(3 * base).astype(dtype),
              port_ijk=(i, j - 1, k), port_voltage=(0.5 * base).astype(dtype),
              probe_ijk=tuple((min(i + q, nx - 2), j, k) for q in range(-1, 8)))
    r = simulate_3d(g, cpml=gb.CPMLSpec(npml), dtype=dtype, **kw)
    o = ref.simulate_3d(og, cpml=o2.CPMLSpec(npml), dtype=dtype, **kw)
    rec, fld = (1e-10, 1e-10) if dtype == F64 else (1e-5, 2e-3)
    for nm in ("probe_ez", "port_v", "port_i"):
        assert _rel(getattr(r, nm), getattr(o, nm)) <= rec, nm
    for nm in COMPS:
        assert _rel(getattr(r, nm), getattr(o, nm)) <= fld, nm
