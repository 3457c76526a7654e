"""Runs started by several host threads at once, each on a stream of its own.

2D runs on the resident and on the tile kernels and 3D runs share the library's
private streams for graph captures and its book of resident runs. Every thread
gets, run after run, what the same call returns alone, bit for bit.
"""

import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _calls(kind):
    import gradenna_b200 as gb
    from gradenna_b200.fdtd3d import simulate_3d

    def tm(n, steps):
        g = gb.Grid2D(n, n + 11, 1e-3, 1e-3)
        w = np.sin(2 * np.pi * 4e9 * (np.arange(steps) + 0.5) * g.dt)

        def call():
            r = gb.simulate_tm(g, dtype=torch.float32, cpml=gb.CPMLSpec(8), dft_freqs=(3e9,),
                               source_ij=[(n // 2, n // 3)], source_current=w[:, None],
                               probe_ij=[(n // 3, n // 2)])
            return [r.ez, r.hx, r.hy, r.probe_ez, r.dft_ez]
        return call

    def yee(n, steps):
        g = gb.Grid3D(n, n + 3, n - 2, 1e-3, 1e-3, 1e-3)
        w = np.sin(2 * np.pi * 9e9 * (np.arange(steps) + 0.5) * g.dt)

        def call():
            r = simulate_3d(g, dtype=torch.float32, cpml=gb.CPMLSpec(4), source_current=w,
                            source_ijk=(n // 2, n // 2, n // 2), probe_ijk=((n // 3,) * 3,))
            return [r.ex, r.ez, r.hy, r.probe_ez]
        return call

    if kind == "3d":
        return [yee(n, 150) for n in (24, 27, 30, 35)]
    # Resident: alone each fits the chip; the last two do not fit beside each other.
    return [tm(n, s) for n, s in ((70, 400), (140, 300), (500, 200), (900, 150))]


@pytest.mark.parametrize("kind", ["resident", "tile", "3d"])
def test_threads_get_the_results_of_single_runs(kind, monkeypatch):
    if kind == "tile":
        monkeypatch.setenv("GDN_TM_KERNEL", "tile")
    calls = _calls(kind)
    want = [f() for f in calls]
    torch.cuda.synchronize()
    got, errors = [[] for _ in calls], []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(6):
                    got[k].append(calls[k]())
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors[0]
    for w, runs in zip(want, got):
        assert len(runs) == 6
        for r in runs:
            assert all(torch.equal(a, b) for a, b in zip(w, r))
