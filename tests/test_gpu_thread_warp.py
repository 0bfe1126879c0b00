"""The thread layout's two forms: a warp per run (the default for small
batches) gives the bits of a thread per run (which a block size asks for)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOUNDS = {0: 5.0, 1: 5.12, 2: 32.768}
CASES = [(0, 2), (0, 4), (0, 8), (0, 10), (1, 2), (1, 10), (2, 2), (2, 10), (4, 4)]


def _objective(zb, kind, dim):
    if kind == 4:
        edges = np.geomspace(0.085, 0.54, 21)
        x = 0.5 * (edges[1:] + edges[:-1])
        lam = 1e4 * (1 - x) ** 10 / x ** 4
        return zb.PoissonNLL(np.random.default_rng(3).poisson(lam).astype(np.int32), x)
    return [zb.Rosenbrock, zb.Rastrigin, zb.Ackley][kind](dim)


@pytest.mark.parametrize("gradient", ["adjoint", "dual"])
@pytest.mark.parametrize("kind,dim", CASES)
def test_warp_form_equals_thread_form(kind, dim, gradient):
    import torch

    import zeus_b200 as zb

    obj = _objective(zb, kind, dim)
    rng = np.random.default_rng(11 * kind + dim)
    for n in (1, 2, 333):
        lo, hi = (0.0, 10.0) if kind == 4 else (-BOUNDS[kind], BOUNDS[kind])
        x0 = torch.from_numpy(rng.uniform(lo, hi, (n, dim))).cuda()
        runs = [zb.bfgs_device(obj, x0, max_iter=250, gradient=gradient,
                               layout=zb.LAYOUT_THREAD, block=b) for b in (0, 128)]
        torch.cuda.synchronize()
        for a in ("fval", "status", "iter", "gnorm", "x", "counters"):
            u, v = (getattr(r, a).cpu().numpy() for r in runs)
            np.testing.assert_array_equal(u, v, err_msg=f"{a} of {n} runs")


def test_warp_form_stops_early():
    import torch

    import zeus_b200 as zb

    x0 = zb.starts(42, 1024, 2, -5.0, 5.0)
    r = zb.bfgs_device(zb.Rosenbrock(2), x0, required=10, layout=zb.LAYOUT_THREAD)
    torch.cuda.synchronize()
    st = r.status.cpu().numpy()
    assert (st == 1).sum() >= 10
    # the runs still going see the flag (the others ended by themselves)
    assert (st == 2).sum() > 0
    # a flag that is up before the launch stops every run at its start
    r.control[0] = 1
    r.launch(x0, reset_control=False)
    torch.cuda.synchronize()
    assert (r.status == 2).all() and (r.iter == 0).all()
    assert torch.equal(r.x, x0)
