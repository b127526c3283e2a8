"""The FP32 V-cycle through the chain of coarse levels, Poisson's and the Jacobian-aware one (levels n <= 15 of
-Lap_h - c), bit for bit a float32 restatement: right-hand sides of ordinary size, and of a size whose quotients leave
the range in which a correction by the reciprocal is exact (the Jacobian-aware levels and the last point then divide)."""
import numpy as np
import pytest

from test_mixed_gpu import F, colour_mask, shifted

pytestmark = pytest.mark.gpu


def _fma(a, b, c):
    return (a.astype(np.longdouble) * b + c).astype(F)  # exact product, one rounding but for the longdouble's


def _div6(s):
    q = s * F(0.16666667)
    return _fma(_fma(-q, F(6), s), F(0.16666667), q)


def _weight(r, nc):
    w = np.array([0.25, 0.5, 0.25], F)
    acc = np.zeros((nc,) * 3, F)
    for a in range(3):
        for b in range(3):
            for c in range(3):
                acc = _fma(r[a:a + 2 * nc:2, b:b + 2 * nc:2, c:c + 2 * nc:2], w[a] * w[b] * w[c], acc)
    return acc


def _interp(x):
    """Trilinear, each point's terms in the order of its coarse neighbours (an absent one adds a zero)."""
    n = 2 * x.shape[0] + 1
    X = np.pad(x, 1)
    f = np.arange(n)
    acc = np.zeros((n,) * 3, F)
    terms = [(((f + 1) >> 1) + t, np.where(f % 2 == 1, F(1 - t), F(0.5)).astype(F)) for t in (0, 1)]
    for ii, wi in terms:
        for jj, wj in terms:
            for kk, wk in terms:
                acc = _fma(X[np.ix_(ii, jj, kk)], wi[:, None, None] * wj[None, :, None] * wk[None, None, :], acc)
    return acc


def vcycle32_jacobian(r, n, c, pre, post):
    """c None: no level is shifted."""
    poisson = c is None
    coef, m = [np.zeros((n,) * 3, F) if poisson else c.reshape(n, n, n).astype(F)], n
    while m > 1:
        m = (m - 1) // 2
        coef.append(_weight(coef[-1], m))

    def cycle(l, b):
        m = coef[l].shape[0]
        h2 = (m + 1.0) ** 2
        shift = not poisson and l > 0 and m <= 15
        if m == 1:
            return b / (F(6 * h2) - coef[l])
        cs, bs, mask = coef[l] * F(1 / h2), b * F(1 / h2), colour_mask(m)

        def sweep(x, order):
            for colour in (order, 1 - order):
                acc = bs
                for axis in (0, 1, 2):
                    acc = acc + shifted(x, axis, -1)
                    acc = acc + shifted(x, axis, +1)
                x = np.where(mask == colour, acc / (F(6) - cs) if shift else _div6(acc), x)
            return x

        x = np.zeros((m,) * 3, F)
        for _ in range(pre):
            x = sweep(x, 0)
        s = F(6) * x
        for axis in (0, 1, 2):
            s = s - shifted(x, axis, -1)
            s = s - shifted(x, axis, +1)
        if shift:
            s = s - cs * x
        xc = cycle(l + 1, _weight(b - F(h2) * s, (m - 1) // 2))
        x = x + np.where(mask == 0, _interp(xc), F(0))
        for _ in range(post):
            x = sweep(x, 1)
        return x

    return cycle(0, r.reshape(n, n, n).astype(F)).astype(np.float64).ravel()


@pytest.mark.parametrize("n,pre,post", [(31, 2, 2), (31, 1, 3), (63, 2, 2)])
@pytest.mark.parametrize("size", [1.0, 1e-36])
def test_jacobian_vcycle_bit_exact(gpu, n, pre, post, size):
    import numa_gpu as G
    rng = np.random.default_rng(n + pre)
    k = rng.integers(-2, 3, n ** 3)
    u = k * np.log(2.0)  # lambda e^u = 6 2^k to FP64 rounding, so exactly that in FP32
    pc = G.Provider.jacobian_mg(gpu, n, pre, post)
    # a solve of one Newton step leaves the coefficients of its start with the preconditioner
    G.newton_krylov(G.Bratu3D(gpu, n, 6.0), gpu.from_numpy(u),
                    G.default_params(max_nl=1, gmres_restart=2, gmres_max_iters=1, flexible=1, jvp_precision=G.FP32,
                                     orth=G.CGS1), pc)
    r = size * rng.standard_normal(n ** 3)
    z = gpu.vec(n ** 3)
    pc.apply(gpu.from_numpy(r), z)
    assert np.array_equal(z.numpy(), vcycle32_jacobian(r, n, 6.0 * 2.0 ** k, pre, post))


@pytest.mark.parametrize("n,pre,post", [(31, 2, 2), (63, 1, 2)])
@pytest.mark.parametrize("size", [1.0, 1e-37])
def test_poisson_vcycle_bit_exact(gpu, n, pre, post, size):
    import numa_gpu as G
    r = size * np.random.default_rng(n).standard_normal(n ** 3)
    mg, z = G.PoissonMG(gpu, n, pre, post, precision=G.FP32), gpu.vec(n ** 3)
    mg(gpu.from_numpy(r), z)
    assert np.array_equal(z.numpy(), vcycle32_jacobian(r, n, None, pre, post))
