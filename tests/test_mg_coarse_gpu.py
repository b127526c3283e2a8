"""The coarse end of the FP64 V-cycle in one cluster kernel: bit for bit the oracle's V-cycle at the edges of its
split (the largest and smallest sizes of one CTA and of the slabs, slabs with a short last plane, hierarchies that
end in an even grid), in place and out of place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6, 8, 9, 10, 11, 12, 13, 14, 15, 17, 19, 23, 27, 29, 31, 39, 47, 95])
@pytest.mark.parametrize("pre,post", [(2, 2), (0, 1), (1, 0)])
def test_vcycle_bit_exact(gpu, oracle, n, pre, post):
    import numa_gpu as G
    r = np.random.default_rng(n).standard_normal(n ** 3)
    mg = G.PoissonMG(gpu, n, pre, post)
    want = oracle.mg_apply(n, r, pre, post)
    rv, z = gpu.from_numpy(r), gpu.vec(n ** 3)
    mg(rv, z)
    assert np.array_equal(z.numpy(), want)
    mg(rv, rv)
    assert np.array_equal(rv.numpy(), want)
