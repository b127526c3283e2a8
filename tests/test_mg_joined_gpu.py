"""The FP32 V-cycle's joined kernels (residual with restriction, prolongation with the first post-smoothing pass): bit
for bit the float32 restatement, for sizes with odd and even coarser levels, rows that end one cell past a warp or a
block, and other sweep counts (post = 0 runs the prolongation by itself)."""
import numpy as np
import pytest

from test_mixed_gpu import vcycle32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,pre,post", [(5, 2, 2), (9, 1, 1), (33, 2, 2), (35, 1, 3), (39, 2, 1), (47, 2, 2),
                                        (63, 1, 1), (63, 2, 3), (65, 2, 2), (69, 1, 2), (95, 2, 2), (129, 1, 1), (193, 1, 1), (259, 1, 1)])
def test_bit_exact(gpu, n, pre, post):
    import numa_gpu as G
    r = np.random.default_rng(n).standard_normal(n ** 3)
    mg = G.PoissonMG(gpu, n, pre, post, precision=G.FP32)
    z = gpu.vec(n ** 3)
    for _ in range(2):  # a second cycle sees nothing of the first
        mg(gpu.from_numpy(r), z)
    assert np.array_equal(z.numpy(), vcycle32(r, n, pre, post))
