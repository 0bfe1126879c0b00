"""The thread layout on both sides of its lines between a warp and a thread a
run, and with several waves of warps: the bits of a thread a run (which a
block size asks for)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOUNDS = {0: 5.0, 1: 5.12, 2: 32.768}


# kind, dim, gradient, max_iter, the last size that has a warp a run
@pytest.mark.parametrize("kind,dim,gradient,max_iter,line", [
    (0, 2, "adjoint", 20, 3072), (0, 2, "adjoint", 100, 4000), (0, 2, "dual", 100, 3072),
    (0, 8, "adjoint", 20, 1024), (0, 8, "adjoint", 300, 6000), (0, 8, "dual", 300, 4500),
    (1, 2, "adjoint", 5, 6144), (2, 2, "dual", 20, 4800), (2, 10, "adjoint", 300, 4096),
    (4, 4, "adjoint", 8, 12288), (4, 4, "dual", 8, 1024)])
def test_both_sides_of_the_line(cuda, kind, dim, gradient, max_iter, line):
    import torch

    import zeus_b200 as zb

    if kind == 4:
        edges = np.geomspace(0.085, 0.54, 21)
        x = 0.5 * (edges[1:] + edges[:-1])
        lam = 1e4 * (1 - x) ** 10 / x ** 4
        obj = zb.PoissonNLL(np.random.default_rng(3).poisson(lam).astype(np.int32), x)
        lo, hi = 0.0, 10.0
    else:
        obj = [zb.Rosenbrock, zb.Rastrigin, zb.Ackley][kind](dim)
        lo, hi = -BOUNDS[kind], BOUNDS[kind]
    warps = zb.lib().zeus_internal_thread_layout_warps
    grad = {"adjoint": zb.GRAD_ADJOINT, "dual": zb.GRAD_DUAL}[gradient]
    for n in (line, line + 1):
        assert bool(warps(kind, dim, grad, max_iter, n)) == (n == line)
        x0 = zb.starts(5, n, dim, lo, hi)
        runs = [zb.bfgs_device(obj, x0, max_iter=max_iter, gradient=gradient,
                               layout=zb.LAYOUT_THREAD, block=b) for b in (0, 128)]
        torch.cuda.synchronize()
        for a in ("fval", "status", "iter", "gnorm", "x", "counters"):
            u, v = (getattr(r, a).cpu().numpy() for r in runs)
            np.testing.assert_array_equal(u, v, err_msg=f"{a} of {n} runs")
