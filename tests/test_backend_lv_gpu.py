"""The two-factor local-vol backend kernel at the edges of its tiles.

rg_lv_terminal_spots walks paths in warps of 32, steps in tiles of 8 and stages grids of up to 192
points in shared memory (16-byte copies where a row is a multiple of four).  A path's result depends
on its own normals only, so any split of the paths over calls — which moves every path to another
lane, warp and tile row — gives the same bits, and so does a longer run's prefix of steps for the
knock-outs that fall in it.
"""
from __future__ import annotations

import numpy as np
import pytest

from riga_gb300 import gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("paths,steps", [(2, 1), (33, 7), (64, 8), (129, 9), (1000, 64), (4097, 33)])
@pytest.mark.parametrize("gx", [2, 3, 40, 97, 192, 193, 300])
def test_results_do_not_depend_on_the_split(paths, steps, gx):
    rng = np.random.default_rng(paths * 1000 + gx)
    z = rng.standard_normal((paths, steps, 2)).astype(np.float32)
    axis = np.concatenate([np.linspace(3.6, 5.4, gx), np.linspace(2.9, 4.9, gx)]).astype(np.float32)
    rows = rng.uniform(0.1, 0.6, (2, steps, gx)).astype(np.float32)
    s0, refs, q = np.float32([100.0, 50.0]), np.float32([100.0, 51.0]), np.float32([0.01, 0.02])

    def run(z, rows, bar):
        return gpu.lv_terminal_spots(z.ravel(), rows.ravel(), axis, s0, refs, bar, z.shape[0], z.shape[1], 1 / 52, 0.03, q)

    for bar in (1.001, 1.1, 1e30, -1.0):
        out, ko = run(z, rows, bar)
        cut = paths // 2 + 1 if paths > 2 else 1
        parts = [run(z[:cut], rows, bar), run(z[cut:], rows, bar)]
        assert np.array_equal(np.concatenate([p[0] for p in parts]).view(np.uint32), out.view(np.uint32))
        assert np.array_equal(np.concatenate([p[1] for p in parts]), ko)
        if steps > 1:
            half = steps // 2
            _, early = run(z[:, :half].copy(), rows[:, :half].copy(), bar)
            assert np.array_equal(early, np.where((ko >= 0) & (ko < half), ko, -1))
        assert (ko == 0).all() if bar < 0 else True
        assert (ko == -1).all() if bar > 1e20 else True


@pytest.mark.parametrize("bar,ref", [(1e-44, 1e30), (1e-10, 1e-34), (1e-20, 1e-24), (1.1754944e-38, 1.0), (1.0, 1.1754944e-38),
                                     (0.7, 3.0), (1e30, 1e8)])
def test_knock_out_at_the_rounding_of_tiny_barriers(bar, ref):
    """Without drift and volatility a path stays at its spot, and it knocks out at once exactly where the ratio
    of the returned spot, rounded in FP32, reaches the barrier: also where the ratio or the barrier's spot is
    subnormal and rounds by percents, far below what separates log-spots from the barrier's."""
    bar, ref = np.float32(bar), np.float32(ref)
    axis = np.concatenate([np.linspace(-110.0, 89.0, 4)] * 2).astype(np.float32)
    rows, z, q = np.zeros((2, 3, 4), np.float32), np.zeros(6, np.float32), np.zeros(2, np.float32)
    seen = set()
    for k in np.linspace(0.9, 1.1, 401):
        s0 = np.float32(np.float64(bar) * np.float64(ref) * k)
        out, ko = gpu.lv_terminal_spots(z, rows.ravel(), axis, np.float32([s0, s0]), np.float32([ref, ref]), float(bar), 1, 3, 1 / 52, 0.0, q)
        want = 0 if out[0] / ref >= bar else -1
        assert ko[0] == want, (k, out[0], out[0] / ref, bar)
        seen.add(want)
    assert seen == {0, -1}
