"""Swarms on a stream of a green context, which has a few of the device's SMs.
The one-launch PSO's blocks wait for one another, so there may be no more of
them than that; a swarm that then does not fit is a launch an iteration.  Both
give the bits of the same call on the whole device, which for these swarms is
one launch: this is also the comparison of the two paths, objective by
objective."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOUNDS = {0: 5.0, 1: 5.12, 2: 32.768, 3: 5.0}


@pytest.fixture(scope="module")
def green():
    """A stream on 8 SMs."""
    import torch

    driver = pytest.importorskip("cuda.bindings.driver")
    torch.zeros(1, device="cuda")

    def ok(r):
        if r[0] != driver.CUresult.CUDA_SUCCESS:
            pytest.skip(f"green contexts: {r[0]}")
        return r[1] if len(r) == 2 else r[1:]

    dev = ok(driver.cuDeviceGet(torch.cuda.current_device()))
    sm = driver.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM
    groups = ok(driver.cuDevSmResourceSplitByCount(1, ok(driver.cuDeviceGetDevResource(dev, sm)),
                                                   0, 8))[0]
    desc = ok(driver.cuDevResourceGenerateDesc(groups[:1], 1))
    ctx = ok(driver.cuGreenCtxCreate(
        desc, dev, driver.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    assert groups[0].sm.smCount <= 16
    h = ok(driver.cuGreenCtxStreamCreate(
        ctx, driver.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield torch.cuda.ExternalStream(int(h))
    torch.cuda.synchronize()
    driver.cuStreamDestroy(h)
    driver.cuGreenCtxDestroy(ctx)


def _objective(zb, kind, dim):
    if kind == 4:
        edges = np.geomspace(0.085, 0.54, 21)
        x = 0.5 * (edges[1:] + edges[:-1])
        lam = 1e4 * (1 - x) ** 10 / x ** 4
        return zb.PoissonNLL(np.random.default_rng(3).poisson(lam).astype(np.int32), x)
    if kind == 3:
        return zb.Gaussian(zb.gaussian_matrix(dim))
    return [zb.Rosenbrock, zb.Rastrigin, zb.Ackley][kind](dim)


def _launches(obj, n, lo, hi, iters, stream):
    """Kernels that a call records."""
    import torch
    from cuda.bindings import runtime

    import zeus_b200 as zb

    gr = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(gr, stream=stream):
        out = zb.pso_device(obj, 6, n, lo, hi, iters)
    raw = runtime.cudaGraph_t(gr.raw_cuda_graph())
    err, _, count = runtime.cudaGraphGetNodes(raw, 0)
    assert err == 0
    err, nodes, _ = runtime.cudaGraphGetNodes(raw, count)
    kinds = [runtime.cudaGraphNodeGetType(k)[1] for k in nodes]
    with torch.cuda.stream(stream):
        gr.replay()
    stream.synchronize()
    return sum(k == runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds), out


# fewer, larger blocks; then swarms past what 8 to 16 blocks hold: a thread, a
# warp and the tensor cores a particle
@pytest.mark.parametrize("prng", ["philox", "sobol"])
@pytest.mark.parametrize("kind,dim,n,one", [
    (0, 10, 3000, True), (1, 2, 3000, True), (3, 8, 1500, True),
    (0, 2, 20000, False), (0, 10, 20000, False), (0, 32, 9000, False), (1, 10, 9000, False),
    (1, 16, 9000, False), (2, 2, 9000, False), (2, 30, 9000, False), (3, 2, 9000, False),
    (3, 32, 9000, False), (4, 4, 9000, False), (0, 64, 3000, False), (0, 128, 2000, False),
    (0, 256, 1000, False), (3, 150, 300, False)])
def test_swarm_on_a_part_of_the_device(green, kind, dim, n, one, prng):
    import torch

    import zeus_b200 as zb

    obj = zb.device.DeviceProblem(_objective(zb, kind, dim))
    lo, hi = (0.5, 10.0) if kind == 4 else (-BOUNDS[kind], BOUNDS[kind])
    whole = zb.pso_device(obj, 6, n, lo, hi, 5, prng=prng)
    torch.cuda.synchronize()
    with torch.cuda.stream(green):
        part = zb.pso_device(obj, 6, n, lo, hi, 5, prng=prng)
    green.synchronize()
    for u, v in zip(part, whole):
        np.testing.assert_array_equal(u.cpu().numpy(), v.cpu().numpy())
    if prng == "philox":
        kernels, out = _launches(obj, n, lo, hi, 5, green)
        assert kernels == (1 if one else 2 + 5)
        for u, v in zip(out, whole):
            np.testing.assert_array_equal(u.cpu().numpy(), v.cpu().numpy())
        kernels, out = _launches(obj, n, lo, hi, 5, torch.cuda.Stream())
        assert kernels == 1
