"""The one-launch PSO at the edges of its split into blocks, against the
oracle's synchronous PSO."""
import numpy as np
import pytest

from tests import _oracle as O

pytestmark = pytest.mark.gpu


def _run(obj, seed, n, lo, hi, iters, stream=False):
    import torch

    import zeus_b200 as zb

    with torch.cuda.stream(torch.cuda.Stream() if stream else torch.cuda.default_stream()):
        out = zb.pso_device(obj, seed, n, lo, hi, iters)
    torch.cuda.synchronize()
    return [t.cpu().numpy() for t in out]


# one block (n D <= 1024), two, many, more particles than threads and SMs
@pytest.mark.parametrize("dim,n", [(2, 1), (2, 512), (2, 513), (2, 30000), (10, 103), (10, 104),
                                   (10, 205), (16, 4097), (32, 65), (32, 20001)])
def test_rosenbrock_swarm_bits_equal_the_oracle(dim, n):
    import zeus_b200 as zb

    x, f, g = _run(zb.Rosenbrock(dim), 9, n, -5.0, 5.0, 4, stream=n % 2 == 0)
    wx, wf, wgx, wgf = O.oracle_pso(0, dim, 9, n, -5.0, 5.0, 4)
    np.testing.assert_array_equal(x, wx)
    np.testing.assert_array_equal(f, wf)
    np.testing.assert_array_equal(g, np.concatenate([[wgf], wgx]))


@pytest.mark.parametrize("dim,n", [(2, 700), (8, 129), (32, 33), (32, 500)])
def test_quadratic_swarm_bits_equal_the_oracle(dim, n):
    import zeus_b200 as zb

    C = zb.gaussian_matrix(dim) + np.triu(np.full((dim, dim), 0.125))
    x, f, g = _run(zb.Gaussian(C), 4, n, -5.0, 5.0, 3)
    wx, wf, wgx, wgf = O.oracle_pso(3, dim, 4, n, -5.0, 5.0, 3, data=C)
    np.testing.assert_array_equal(x, wx)
    np.testing.assert_array_equal(f, wf)
    np.testing.assert_array_equal(g, np.concatenate([[wgf], wgx]))


@pytest.mark.parametrize("n", [1, 8, 9, 1184, 1185])
def test_gaussian150_swarm_values(n):
    """Values of the tensor-core sums at the bests they are reported with
    (1184 particles are the most with C in shared memory)."""
    import zeus_b200 as zb

    C = zb.gaussian_matrix(150)
    x, f, g = _run(zb.Gaussian(C), 4, n, -5.0, 5.0, 2)
    want = 0.5 * np.einsum("ij,jk,ik->i", x, C, x)
    # positive terms dominate: 22 500 products added within a few chains
    np.testing.assert_allclose(f, want, rtol=200 * 2.0 ** -53 * 10)
    k = int(np.argmin(f))
    assert g[0] == f[k]
    np.testing.assert_array_equal(g[1:], x[k])


def test_swarm_with_no_finite_value_keeps_gbest_at_infinity():
    import zeus_b200 as zb

    x, f, g = _run(zb.Rosenbrock(2), 1, 2000, 1e200, 2e200, 2)
    assert not np.isfinite(f).any()
    assert np.isposinf(g[0]) and (g[1:] == 0).all()


def test_swarm_is_captured_into_a_graph():
    import torch

    import zeus_b200 as zb

    obj = zb.device.DeviceProblem(zb.Rastrigin(10))
    want = _run(obj, 5, 3000, -5.12, 5.12, 6)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        zb.pso_device(obj, 5, 3000, -5.12, 5.12, 6)
    torch.cuda.synchronize()
    gr = torch.cuda.CUDAGraph()
    with torch.cuda.graph(gr, stream=s):
        out = zb.pso_device(obj, 5, 3000, -5.12, 5.12, 6)
    for _ in range(3):
        gr.replay()
    torch.cuda.synchronize()
    for u, v in zip(out, want):
        np.testing.assert_array_equal(u.cpu().numpy(), v)
