"""The batched solver's block size is the one that was set, and the one reported."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL = [(31, 6.0), (63, 2.5)]
LARGE = SMALL + [(127, 3.0)] * 3


def _solver(G, gpu, inst):
    return G.BatchSolver(gpu, inst, G.default_params(rtol_nl=1e-10, gmres_restart=30, flexible=1, jvp_precision=G.FP32,
                                                     orth=G.CGS1))


@pytest.mark.parametrize("elems", [1024, 4096, 16384])
def test_set_block_size_is_used(gpu, elems):
    """An instance has the same bits alone, where the default block is small, and in a batch whose default is larger."""
    import numa_gpu as G
    runs = []
    for inst in (SMALL, LARGE):
        bs = _solver(G, gpu, inst)
        try:
            bs.set_tuning(8, elems)
            assert bs.tuning() == {"planes": 8, "elems_per_block": elems}
            r, _, x = bs.solve(want_x=True)
            runs.append(([dict(q, seconds=0) for q in r[:2]], x[:2]))
        finally:
            bs.close()
    (r0, x0), (r1, x1) = runs
    assert all(np.array_equal(a, b) for a, b in zip(x0, x1))
    assert r0 == r1


@pytest.mark.parametrize("inst", [SMALL, LARGE])
def test_default_block_size_is_reported(gpu, inst):
    """The default fills the SMs eight times where the batch is that large; setting it changes no bits."""
    import torch

    import numa_gpu as G
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    bs = _solver(G, gpu, inst)
    try:
        t = bs.tuning()
        assert t["elems_per_block"] == max(2048, min(16384, sum(n ** 3 for n, _ in inst) // (8 * sms) // 1024 * 1024))
        x0 = bs.solve(want_x=True)[2]
        bs.set_tuning(**t)
        x1 = bs.solve(want_x=True)[2]
    finally:
        bs.close()
    assert all(np.array_equal(a, b) for a, b in zip(x0, x1))
