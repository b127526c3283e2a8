"""The compile-time chain of coarse levels (31, 15, 7, 3, 1): the FP64 V-cycle bit for bit the oracle's, the FP32 one
within FP32 accuracy of it, with the chain as the whole cycle and below launched levels, for several sweep counts.
(The FP32 cycles are compared bit for bit with a float32 restatement in the mixed tests.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 63])
@pytest.mark.parametrize("pre,post", [(2, 2), (1, 1), (3, 1), (1, 2)])
def test_fp32_chain(gpu, oracle, n, pre, post):
    import numa_gpu as G
    r = np.random.default_rng(n).standard_normal(n ** 3)
    mg = G.PoissonMG(gpu, n, pre, post, precision=G.FP32)
    z = gpu.vec(n ** 3)
    mg(gpu.from_numpy(r), z)
    want = oracle.mg_apply(n, r, pre, post)
    # a few dozen FP32 roundings of a contracting iteration: 2^-24 each
    assert np.linalg.norm(z.numpy() - want) <= 64 * 2.0 ** -24 * np.linalg.norm(want)


@pytest.mark.parametrize("n", [15, 31, 63])
@pytest.mark.parametrize("pre,post", [(1, 1), (3, 1), (1, 3)])
def test_fp64_chain_bit_exact(gpu, oracle, n, pre, post):
    import numa_gpu as G
    r = np.random.default_rng(n).standard_normal(n ** 3)
    mg = G.PoissonMG(gpu, n, pre, post)
    rv = gpu.from_numpy(r)
    mg(rv, rv)
    assert np.array_equal(rv.numpy(), oracle.mg_apply(n, r, pre, post))
