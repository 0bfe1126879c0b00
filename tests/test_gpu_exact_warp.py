"""Exact mode's warp form (up to D = 32) against the oracle's iterates and,
where the block form serves the same dimension, against it bit for bit."""
import numpy as np
import pytest

from tests import _oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 4, 8, 10, 16])
@pytest.mark.parametrize("n,max_iter", [(1, 40), (7, 0), (65, 60)])
def test_rosenbrock_bits_equal_the_oracle(dim, n, max_iter):
    import torch

    import zeus_b200 as zb

    st = O.oracle_starts(5, n, dim, -5.0, 5.0)
    want = O.oracle_bfgs(0, dim, st, max_iter=max_iter)
    r = zb.bfgs_device(zb.Rosenbrock(dim), torch.from_numpy(st).cuda(), max_iter=max_iter,
                       mode="exact", gradient="dual")
    torch.cuda.synchronize()
    for name in ("status", "fval", "x"):
        np.testing.assert_array_equal(getattr(r, name).cpu().numpy(), want[name], err_msg=name)


@pytest.mark.parametrize("kind,dim", [(0, 32), (2, 30), (3, 32)])
def test_warp_form_equals_block_form(kind, dim):
    """The two forms of the same dimension, picked by the number of runs."""
    import torch

    import zeus_b200 as zb

    obj = {0: zb.Rosenbrock, 2: zb.Ackley}[kind](dim) if kind < 3 else zb.Gaussian(
        zb.gaussian_matrix(dim) + np.triu(np.full((dim, dim), 0.01)))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    few, many = 40, 2 * sms + 1
    rng = np.random.default_rng(dim)
    x0 = torch.from_numpy(rng.uniform(-5, 5, (many, dim))).cuda()
    a = zb.bfgs_device(obj, x0[:few].contiguous(), max_iter=30, mode="exact",
                       gradient="dual", traj=True)
    b = zb.bfgs_device(obj, x0, max_iter=30, mode="exact", gradient="dual", traj=True)
    torch.cuda.synchronize()
    for name in ("fval", "status", "iter", "gnorm", "x", "counters"):
        np.testing.assert_array_equal(getattr(a, name).cpu().numpy(),
                                      getattr(b, name)[:few].cpu().numpy(), err_msg=name)
    for name in ("x", "f", "g", "status"):
        np.testing.assert_array_equal(a.traj[name].cpu().numpy(),
                                      b.traj[name][..., :few].cpu().numpy(), err_msg=name)


def test_workspace_of_many_runs_serves_few():
    """A caller may size one workspace for its largest launch."""
    import ctypes as C

    import zeus_b200 as zb

    cfg = zb.make_config(10, 1 << 30, 1e-8, "exact", "dual")
    for obj in (zb.Rosenbrock(10), zb.Rosenbrock(32), zb.Ackley(30)):
        p = obj.problem(None, None)
        sizes = [zb.lib().zeus_bfgs_workspace_size(C.byref(p), C.byref(cfg), n)
                 for n in (1, 40, 200, 1000, 20000)]
        assert sizes == sorted(sizes) and sizes[0] > 0
