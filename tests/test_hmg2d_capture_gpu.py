"""HelmholtzMG2D and the Burgers preconditioner captured into a caller's CUDA graph on the context's stream, as the
hierarchy's first application and after one: replays on new right-hand sides, bit for bit the oracle's cycle, and calls
outside the capture as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [9, 33, 95, 129])
@pytest.mark.parametrize("warm", [False, True])
def test_captured_application(gpu, oracle, n, warm):
    import torch

    import numa_gpu as G
    nu, dt = 0.05, 0.04
    rng = np.random.default_rng(n)
    stream = torch.cuda.ExternalStream(gpu.stream())
    pc, mg = G.Provider.burgers_mg(gpu, n, nu, dt), G.HelmholtzMG2D(gpu, n, 25.0, nu)
    r, z = gpu.from_numpy(rng.standard_normal(2 * n * n)), gpu.vec(2 * n * n)
    r1, z1 = gpu.from_numpy(rng.standard_normal(n * n)), gpu.vec(n * n)
    if warm:
        pc.apply(r, z)
        mg(r1, z1)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        pc.apply(r, z)
        mg(r1, z1)

    def check():
        h, h1 = r.numpy(), r1.numpy()
        want = np.concatenate([oracle.hmg2d_apply(n, 1.0 / dt, nu, f) for f in (h[: n * n], h[n * n:])])
        assert np.array_equal(z.numpy(), want)
        assert np.array_equal(z1.numpy(), oracle.hmg2d_apply(n, 25.0, nu, h1))

    for _ in range(2):
        r.upload(rng.standard_normal(2 * n * n))
        r1.upload(rng.standard_normal(n * n))
        with torch.cuda.stream(stream):
            graph.replay()
        check()
    r.upload(rng.standard_normal(2 * n * n))
    r1.upload(rng.standard_normal(n * n))
    pc.apply(r, z)
    mg(r1, z1)
    check()
