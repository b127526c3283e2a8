"""GMRES with modified Gram-Schmidt across the edges of its compact WY form: bases that end inside and at a group of
eight vectors, at and past the 32 vectors it holds, on vectors shorter and longer than a block, against the oracle's
chain of inner products and updates."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 8, 17, 40])
@pytest.mark.parametrize("restart", [1, 7, 8, 9, 31, 32, 33, 45])
def test_mgs_against_oracle(gpu, oracle, n, restart):
    import numa_gpu as G
    N, rtol = n ** 3, 1e-8
    rng = np.random.default_rng(n)
    u, b = 0.1 * rng.standard_normal(N), rng.standard_normal(N)
    op = G.Bratu3D(gpu, n, 2.0)
    x = gpu.vec(N)
    g = G.gmres_bratu3d(op, gpu.from_numpy(u), gpu.from_numpy(b), x, rtol, restart, 120)
    want, r = oracle.gmres_bratu3d(n, 2.0, u, b, rtol, restart, 120)
    assert bool(g["converged"]) == bool(r["converged"])
    assert abs(g["iters"] - r["iters"]) <= 1
    # the same iterate up to rounding, amplified by at most the condition number (2 (n + 1) / pi)^2 < 700
    if g["iters"] == r["iters"]:
        assert np.linalg.norm(x.numpy() - want) <= 1e-10 * np.linalg.norm(want)
