"""GMRES's modified Gram-Schmidt on both sides of the limits between its chain and its compact WY form, and the property
that the compact form has to share with the chain: the loss of orthogonality stays proportional to the condition number
of the vectors orthogonalised."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("n", [50, 51, 101, 102])  # below and above 2^17 and 2^20 points
def test_against_oracle(gpu, oracle, n):
    import numa_gpu as G
    N, m = n ** 3, 12
    rng = np.random.default_rng(n)
    u, b = 0.1 * rng.standard_normal(N), rng.standard_normal(N)
    x = gpu.vec(N)
    op = G.Bratu3D(gpu, n, 2.0)
    g = G.gmres_bratu3d(op, gpu.from_numpy(u), gpu.from_numpy(b), x, 1e-14, m, m)
    want, r = oracle.gmres_bratu3d(n, 2.0, u, b, 1e-14, m, m)
    assert g["iters"] == r["iters"] == m
    # twelve steps from a random vector: the least-squares matrix has a condition number below 100, which enters squared
    assert abs(g["rel_res"] - r["rel_res"]) <= 1e-10 * r["rel_res"]
    assert np.linalg.norm(x.numpy() - want) <= 1e-10 * np.linalg.norm(want)


@pytest.mark.parametrize("N,spread", [(300, 6), (4000, 10), (140000, 8)])
def test_loss_of_orthogonality(gpu, N, spread):
    """A diagonal operator with 14 clusters of eigenvalues, each 10^-spread wide, so that the vectors orthogonalised
    become dependent (condition numbers up to 1e13); the callback sees every basis vector.  After k steps ||I - V^T V|| <= 10 k^1.5 u kappa, kappa the condition number of [b, A v_0, ..., A v_{k-1}] with columns of
    unit norm (Bjorck's bound, the constant of order one in place of the worst case)."""
    import numa_gpu as G
    rng = np.random.default_rng(N)
    d = np.logspace(0, -2, 14)[rng.integers(0, 14, N)] * (1 + 10.0 ** -spread * rng.standard_normal(N))
    b = rng.standard_normal(N)
    basis = []

    def apply(v, out):
        h = v.numpy()
        basis.append(h)
        out.upload(d * h)

    x = gpu.vec(N)
    G.gmres(gpu, apply, gpu.from_numpy(b), x, 1e-16, 28, 28)
    V = np.array(basis[:28]).T
    assert V.shape[1] >= 20
    for k in range(2, V.shape[1]):
        Q = V[:, :k + 1]
        W = np.column_stack([b, d[:, None] * V[:, :k]])
        s = np.linalg.svd(W / np.linalg.norm(W, axis=0), compute_uv=False)
        loss = np.linalg.norm(np.eye(k + 1) - Q.T @ Q, 2)
        assert loss <= min(2.0 * (k + 1), 10 * k ** 1.5 * U * s[0] / s[-1]), (k, loss, s[0] / s[-1])
