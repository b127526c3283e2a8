"""The batched solver's coarse levels on clusters of 8 CTAs (few grids) and of 4 (more grids than clusters of 8 run at
a time): the same instances in batches of either kind take the same Newton steps and agree to rounding.  The
partial sums of the Gram-Schmidt passes are grouped by the batch's size, so the basis differs by FP32 roundings: the
solutions, each converged to 1e-10, within 1e-8 as the batched solver's other tests ask."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jac", [0, 1])
@pytest.mark.parametrize("n,many", [(31, 40), (63, 24)])
def test_cluster_sizes_agree(gpu, n, many, jac):
    import numa_gpu as G
    p = G.default_params(rtol_nl=1e-10, gmres_restart=30, flexible=1, jvp_precision=G.FP32, orth=G.CGS1, jvp_tight=jac,
                         coarse_jacobian=jac)
    inst = [(n, 1.0 + 5.0 * k / many) for k in range(many)]
    big = G.BatchSolver(gpu, inst, p)
    small = G.BatchSolver(gpu, inst[:3], p)
    try:
        rb, _, xb = big.solve(want_x=True)
        rs, _, xs = small.solve(want_x=True)
    finally:
        big.close()
        small.close()
    assert all(r["converged"] == 1 for r in rb)
    for k in range(3):
        assert rb[k]["iters"] == rs[k]["iters"] and rb[k]["n_F"] == rs[k]["n_F"]
        assert np.max(np.abs(xb[k] - xs[k])) <= 1e-8 * np.max(np.abs(xs[k]))
