"""2D scratch off a 16-byte boundary, and scratch for the tile kernels only.

Every kernel moves 16 bytes at a time. A caller's scratch that starts elsewhere
is left alone and the library takes its own; scratch of the least size runs the
tile kernels in it. Both return the bits of an ordinary run, single or batched.
"""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("n,offset", [(150, 4), (150, 8), (150, 0), (1100, 4)])
@pytest.mark.parametrize("batch", [False, True], ids=["single", "batch"])
def test_scratch_off_a_boundary_or_small(n, offset, dtype, batch):
    import gradenna_b200 as gb
    from gradenna_b200 import _native, fdtd2d
    from gradenna_b200.batch import TmProblem

    if batch and dtype == torch.float64:
        pytest.skip("batched runs are float32")
    lib = _native.load()
    steps = 50
    grid = gb.Grid2D(n, n - 13, 1e-3, 1e-3)
    kw = dict(dtype=dtype, cpml=gb.CPMLSpec(9), source_ij=[(n // 2, n // 2)],
              source_current=np.sin(0.3 * np.arange(steps))[:, None], probe_ij=[(n // 3, n // 2)],
              dft_freqs=(3e9,), dft_monitors=[(0, 20, 20, 60, 63)])
    want = gb.simulate_tm(grid, **kw)
    p = fdtd2d._prepare_tm(grid, **kw)
    size = ctypes.c_size_t()
    fn = lib.gdn_tm_workspace_size if offset else lib.gdn_tm_workspace_least
    _native.check(fn(ctypes.byref(p.params), ctypes.byref(p.pts), int(p.f64), ctypes.byref(size)))
    ws = torch.full((size.value + 32,), 0xA5, dtype=torch.uint8, device="cuda")
    assert ws.data_ptr() % 16 == 0
    p.bufs.workspace, p.bufs.workspace_bytes = ws.data_ptr() + offset, size.value
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if batch:
        one = (TmProblem * 1)()
        one[0].params, one[0].points = ctypes.pointer(p.params), ctypes.pointer(p.pts)
        one[0].buffers = ctypes.pointer(p.bufs)
        _native.check(lib.gdn_tm_run_batch_f32(one, 1, -1, stream))
    else:
        run = lib.gdn_tm_run_f64 if p.f64 else lib.gdn_tm_run_f32
        _native.check(run(ctypes.byref(p.params), ctypes.byref(p.pts), ctypes.byref(p.bufs), stream))
    torch.cuda.synchronize()
    if offset:
        assert bool((ws == 0xA5).all())  # untouched
    r = p.result
    for a, b in zip((want.ez, want.hx, want.hy, want.probe_ez, *want.monitors),
                    (r.ez, r.hx, r.hy, r.probe_ez, *r.monitors)):
        assert torch.equal(a, b)
