"""The FP32 V-cycle of the 2D Brusselator multigrid bit for bit a numpy float32 restatement (its kernels contract no
multiply-add, and float32 division is IEEE in both): hierarchies whose levels are launched, run in tiles, in the
one-CTA tail or by its warp, ending in 4, 6, 10, 14 or 18 points a side."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32
PRM = dict(A=1.0, B=3.4, Du=0.002, Dv=0.002, dt=0.01)


def _at(x, di, dj):
    return np.roll(x, (-di, -dj), axis=(0, 1))


def _sum4(x):
    return ((_at(x, 0, -1) + _at(x, 0, 1)) + _at(x, -1, 0)) + _at(x, 1, 0)


def _weight(x):
    """9-point full weighting of a fine array at its even points."""
    edge = (_at(x, 0, -1) + _at(x, 0, 1)) + (_at(x, -1, 0) + _at(x, 1, 0))
    corner = ((_at(x, -1, -1) + _at(x, -1, 1)) + _at(x, 1, -1)) + _at(x, 1, 1)
    return (((F(4) * x + F(2) * edge) + corner) * F(0.0625))[::2, ::2]


def _blocks(w, n):
    u, v = w.astype(F).reshape(2, n, n)
    uv2, uu = (F(2) * u) * v, u * u
    c1, c2 = F(1.0 / PRM["dt"] + (PRM["B"] + 1.0)), F(1.0 / PRM["dt"])
    return [c1 - uv2, -uu, uv2 - F(PRM["B"]), c2 + uu]


def vcycle32(w, r, n, pre, post):
    i, j = np.indices((n, n))

    def cycle(b, K):
        n = b.shape[1]
        s64 = (PRM["Du"] * (float(n) * n), PRM["Dv"] * (float(n) * n))
        (su, sv), (su4, sv4) = map(F, s64), (F(4.0 * s64[0]), F(4.0 * s64[1]))
        colour = (i[:n, :n] + j[:n, :n]) & 1
        m11, m22 = K[0] + su4, K[3] + sv4
        det = m11 * m22 - K[1] * K[2]

        def sweep(x, order):
            for c in (order, 1 - order):
                ru, rv = b[0] + su * _sum4(x[0]), b[1] + sv * _sum4(x[1])
                new = np.stack([(m22 * ru - K[1] * rv) / det, (m11 * rv - K[2] * ru) / det])
                x = np.where(colour == c, new, x)
            return x

        x = np.zeros_like(b)
        if n % 4 != 0 or n // 2 < 4:
            for _ in range(30):
                x = sweep(x, 0)
            return x
        for _ in range(pre):
            x = sweep(x, 0)
        ru = b[0] - ((K[0] * x[0] + K[1] * x[1]) + su * (F(4) * x[0] - _sum4(x[0])))
        rv = b[1] - ((K[2] * x[0] + K[3] * x[1]) + sv * (F(4) * x[1] - _sum4(x[1])))
        xc = cycle(np.stack([_weight(ru), _weight(rv)]), [_weight(k) for k in K])
        x = x.copy()
        for f, c in zip(x, xc):
            f[::2, ::2] = f[::2, ::2] + c
            f[1::2, 1::2] = f[1::2, 1::2] + F(0.25) * (((c + _at(c, 1, 0)) + _at(c, 0, 1)) + _at(c, 1, 1))
        for _ in range(post):
            x = sweep(x, 1)
        return x

    return cycle(r.astype(F).reshape(2, n, n), _blocks(w, n)).astype(np.float64).ravel()


@pytest.mark.parametrize("n", [8, 18, 20, 24, 36, 56, 64, 80, 96, 136, 256, 520])
@pytest.mark.parametrize("pre,post", [(2, 2), (1, 3), (4, 1)])
def test_vcycle_bit_exact(gpu, n, pre, post):
    import numa_gpu as G
    w = G.brusselator2d_initial(n, 1.0, 3.4, 5)
    r = np.random.default_rng(n).standard_normal(2 * n * n)
    mg, z = G.BrussMG2D(gpu, n, G.brusselator_params(), G.FP32, pre, post), gpu.vec(2 * n * n)
    mg.set_state(gpu.from_numpy(w))
    want = vcycle32(w, r, n, pre, post)
    for _ in range(2):
        mg.apply(gpu.from_numpy(r), z)
        assert np.array_equal(z.numpy(), want)
