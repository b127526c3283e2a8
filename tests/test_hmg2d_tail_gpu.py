"""HelmholtzMG2D around the one-CTA tail (levels of n <= 31) and the two-field cycle of the Burgers preconditioner:
bit for bit the oracle's, in place and out of place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 9, 14, 20, 29, 30, 31, 32, 33, 39, 47, 62, 95])
@pytest.mark.parametrize("pre,post", [(2, 2), (0, 1), (1, 0)])
def test_vcycle_bit_exact(gpu, oracle, n, pre, post):
    import numa_gpu as G
    alpha, nu = 25.0, 0.02
    r = np.random.default_rng(n).standard_normal(n * n)
    mg = G.HelmholtzMG2D(gpu, n, alpha, nu, pre, post)
    want = oracle.hmg2d_apply(n, alpha, nu, r, pre, post)
    rv, z = gpu.from_numpy(r), gpu.vec(n * n)
    for _ in range(2):  # the second application replays the captured levels
        mg(rv, z)
        assert np.array_equal(z.numpy(), want)
    mg(rv, rv)
    assert np.array_equal(rv.numpy(), want)


@pytest.mark.parametrize("n", [1, 16, 31, 33, 95])
def test_two_fields(gpu, oracle, n):
    import numa_gpu as G
    nu, dt = 0.05, 0.04
    r = np.random.default_rng(n).standard_normal(2 * n * n)
    pc = G.Provider.burgers_mg(gpu, n, nu, dt)
    z = gpu.vec(r.size)
    pc.apply(gpu.from_numpy(r), z)
    want = np.concatenate([oracle.hmg2d_apply(n, 1.0 / dt, nu, h) for h in (r[: n * n], r[n * n:])])
    assert np.array_equal(z.numpy(), want)


@pytest.mark.parametrize("n", [17, 19, 23, 31, 39, 63, 79, 111, 127, 129])
@pytest.mark.parametrize("pre,post", [(1, 1), (3, 2), (2, 3), (1, 4)])
def test_tiled_levels_bit_exact(gpu, oracle, n, pre, post):
    """Levels run in tiles (15 < n <= 127, up to three sweeps): tiles that end in remainders or on the last row, a
    level above them, more sweeps than they take."""
    import numa_gpu as G
    alpha, nu = 25.0, 0.02
    r = np.random.default_rng(n).standard_normal(n * n)
    mg = G.HelmholtzMG2D(gpu, n, alpha, nu, pre, post)
    want = oracle.hmg2d_apply(n, alpha, nu, r, pre, post)
    rv, z = gpu.from_numpy(r), gpu.vec(n * n)
    for _ in range(2):
        mg(rv, z)
        assert np.array_equal(z.numpy(), want)
    mg(rv, rv)
    assert np.array_equal(rv.numpy(), want)
