"""The 2D Brusselator's residual at the edges of its row chunks, and its norm over them.

The residual kernel's warps cover 31 columns and its threads a number of rows chosen by size: sizes
with one, two and an odd number of column groups, row chunks of one row and chunks that leave a
remainder, against the CPU restatement bit for bit.  The norm a solve starts from (its res0) sums
2 n^2 squares of those values in blocks: within 1e-12 of the host's sum (n^2 rounding errors of 2^-53
cannot exceed 3e-11, and pairwise block sums stay far below).
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PRM = dict(A=1.0, B=3.4, Du=0.002, Dv=0.002, dt=0.01)


@pytest.mark.parametrize("n", [4, 30, 31, 62, 94, 257, 500])
def test_residual_and_norm_over_row_chunks(gpu, oracle, n):
    import numa_gpu as G

    N = 2 * n * n
    op = G.Brusselator2D(gpu, n, G.brusselator_params())
    prev = G.brusselator2d_initial(n, 1.0, 3.4, 11)
    w = prev + 0.02 * np.sin(0.37 * np.arange(N))
    op.set_previous(gpu.from_numpy(prev))
    out = gpu.vec(N)
    op.eval(gpu.from_numpy(w), out)
    f = oracle.bruss2d_eval(n, PRM, prev, w)
    assert np.array_equal(out.numpy(), f)
    r = G.solve(op, gpu.from_numpy(w), "nk", G.default_params(max_nl=1, gmres_restart=4, gmres_max_iters=4),
                G.Provider.create(gpu, "none", op))
    assert abs(r["res0"] - np.sqrt(np.sum(f * f))) <= 1e-12 * r["res0"]


@pytest.mark.parametrize("n", [8, 20, 24, 40, 72, 136, 200, 264, 512, 1000])
@pytest.mark.parametrize("pre,post", [(2, 2), (1, 3), (3, 1), (4, 1)])
def test_vcycle_tiles(gpu, oracle, n, pre, post):
    """Levels whose coarse rows end in remainders (31 coarse columns a warp) or are narrower than one,
    hierarchies ending in a large coarsest level, other sweep counts: FP64 bit for bit; FP32 within 2e-5, the
    bound of the FP32 V-cycle's other tests.  FP32 levels of 16 < n <= 256 run in tiles (up to three sweeps)."""
    import numa_gpu as G

    N = 2 * n * n
    w = G.brusselator2d_initial(n, 1.0, 3.4, 5)
    r = np.sin(0.13 * np.arange(N) + 0.3)
    zo = oracle.bmg2d_apply(n, PRM, w, r, pre, post)
    for precision in (G.FP64, G.FP32):
        mg = G.BrussMG2D(gpu, n, G.brusselator_params(), precision, pre, post)
        z = gpu.vec(N)
        for state in (0.5 * w, w):  # a second state and a second cycle see nothing of the first
            mg.set_state(gpu.from_numpy(state))
            mg.apply(gpu.from_numpy(r), z)
        if precision == G.FP64:
            assert np.array_equal(z.numpy(), zo)
        else:
            assert np.max(np.abs(z.numpy() - zo)) / np.max(np.abs(zo)) < 2e-5
