"""Every kind of resident 2D launch, with the path that was taken asserted.

The sizes give the kinds (rectangle shapes) A, B, C, D, E of float32 and A, B, C of
float64 on a device of 148 SMs, with odd extents, and leave some SMs over so
that a device with a few less takes them too. Fields, records, phasors and
monitors are those of the tile kernels, bit for bit; a resident run launches
some kernels a segment, the tile kernels two a block of four steps.
"""

import pytest
import torch

from tests.test_tm2d_resident_gpu import _run

pytestmark = pytest.mark.gpu

F32, F64 = torch.float32, torch.float64
SIZES = [(150, 131, 9, 77, F32), (281, 251, 10, 70, F32), (421, 380, 10, 66, F32),
         (640, 701, 16, 101, F32), (880, 901, 16, 90, F32),
         (140, 131, 9, 75, F64), (280, 271, 10, 62, F64), (400, 411, 10, 70, F64)]


@pytest.mark.parametrize("layout", ["full", "boxes", "many"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: f"{s[0]}x{s[1]}-{'f32' if s[4] == F32 else 'f64'}")
def test_kind(size, layout, monkeypatch):
    from gradenna_b200 import _native

    *shape, dtype = size
    blocks = (shape[3] + 3) // 4

    def launches(f):
        n = _native.kernel_launches()
        r = f()
        return r, _native.kernel_launches() - n

    got, mine = launches(lambda: _run(*shape, dtype, layout))
    monkeypatch.setenv("GDN_TM_KERNEL", "tile")
    want, tile = launches(lambda: _run(*shape, dtype, layout))
    assert tile >= 2 * blocks and mine <= tile - 2 * blocks + 16
    assert len(want) == len(got)
    for a, b in zip(want, got):
        assert torch.isfinite(torch.view_as_real(b) if b.is_complex() else b).all()
        assert torch.equal(a, b)
