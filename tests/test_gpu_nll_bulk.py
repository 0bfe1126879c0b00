"""The tile layout's two kernels for a likelihood on 32 lanes, the one for few
runs and the one for many: a run's results do not depend on how many others
there are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gradient", ["adjoint", "dual"])
@pytest.mark.parametrize("nbins", [1, 33, 64, 100])
def test_runs_of_a_large_batch_equal_those_of_a_small_one(cuda, nbins, gradient):
    import torch

    import zeus_b200 as zb

    edges = np.geomspace(0.085, 0.54, nbins + 1)
    x = 0.5 * (edges[1:] + edges[:-1])
    lam = (1 - x) ** 10 / x ** 5
    k = np.random.default_rng(nbins).poisson(lam * (3000.0 / lam.sum())).astype(np.int32)
    obj, max_iter = zb.PoissonNLL(k, x), 40
    n = 4096 + 2 * max_iter  # the last size of the kernel for few
    x0 = zb.starts(11, n + 1, 4, 0.0, 10.0)

    def run(s):
        r = zb.bfgs_device(obj, s, max_iter=max_iter, gradient=gradient, layout=zb.LAYOUT_TILE,
                           tile=32)
        torch.cuda.synchronize()
        return {a: getattr(r, a).cpu().numpy()
                for a in ("fval", "status", "iter", "gnorm", "x", "counters")}

    small, large = run(x0[:n].contiguous()), run(x0)
    for a, u in small.items():
        np.testing.assert_array_equal(u, large[a][:n], err_msg=a)
    # searches past the first sweep took part
    assert (large["counters"][:, 1] - large["counters"][:, 0]).max() > 20
