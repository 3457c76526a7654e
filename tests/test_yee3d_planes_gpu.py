"""GPU check of the 3D step kernels' planes per CTA.

Grids with more CTAs than fit on the chip take two planes a CTA (61 x 83 x 61:
671 and 1281 CTAs for one plane each): the values carried from plane to plane,
an odd last plane, and points and the port on a CTA's second plane. Grids with
more planes than a launch has second indices for take more of them. Held to the
numpy oracle with the tolerances of the other 3D parity tests (float64 1e-10;
float32 1e-5 on records, 2e-3 on fields).
"""

import numpy as np
import pytest

from oracle import fdtd2d_np as o2
from oracle import fdtd3d_np as ref

pytestmark = pytest.mark.gpu

COMPS = ("ex", "ey", "ez", "hx", "hy", "hz")


def _rel(a, b):
    a, b = np.asarray(a.detach().cpu()), np.asarray(b)
    return float(np.max(np.abs(a - b)) / (np.max(np.abs(b)) + 1e-300))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("size", [(61, 83, 61, 6, 30), (131075, 7, 6, 1, 6)],
                         ids=lambda s: "x".join(map(str, s[:3])))
def test_planes_per_cta(size, dtype):
    import gradenna_b200 as gb
    from gradenna_b200.fdtd3d import simulate_3d

    nx, ny, nz, npml, steps = size
    rng = np.random.default_rng(nx)
    g, og = (m.Grid3D(nx, ny, nz, 1e-3, 1.1e-3, 0.9e-3) for m in (gb, ref))
    base = np.asarray(np.sin(0.5 * (np.arange(steps) + 0.5)), dtype)
    i = nx // 2 | 1  # odd: the second plane of a pair
    last = nx - npml - 3 | 1
    j, k = ny // 2, nz // 2
    kw = dict(eps_r=1 + 3 * rng.random((nx, ny, nz)), sigma=0.05 * rng.random((nx, ny, nz)),
              source_ijk=(last, j, k), source_current=base,
              source_x_ijk=(i, j, k), source_x_current=(0.7 * base).astype(dtype),
              mx_ijk=(i + 2, j, 1), mx_current=(3 * base).astype(dtype),
              port_ijk=(i + 4, j - 1, k), port_voltage=(0.5 * base).astype(dtype),
              probe_ijk=((last - 1, j, k), (i, j, k), (i + 2, j + 1, k), (nx - 2, j, k)))
    r = simulate_3d(g, cpml=gb.CPMLSpec(npml), dtype=dtype, **kw)
    o = ref.simulate_3d(og, cpml=o2.CPMLSpec(npml), dtype=dtype, **kw)
    rec, fld = (1e-10, 1e-10) if dtype == np.float64 else (1e-5, 2e-3)
    for nm in ("probe_ez", "port_v", "port_i"):
        assert _rel(getattr(r, nm), getattr(o, nm)) <= rec, nm
    for nm in COMPS:
        assert _rel(getattr(r, nm), getattr(o, nm)) <= fld, nm
