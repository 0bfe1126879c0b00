"""A one-launch swarm whose blocks' wait for one another runs out: the kernel
returns with NaN in what is not the swarm's, and the calls that read it back
report an error.  The limit is set to no read at all, on this thread."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def no_wait():
    import zeus_b200 as zb

    limit = zb.lib().zeus_internal_swarm_wait
    limit.restype = C.POINTER(C.c_int)
    full = limit()[0]
    assert full > 0
    limit()[0] = 0
    yield
    limit()[0] = full


# a thread, a warp and the tensor cores a particle; the blocks of each are many
SWARMS = [("rosenbrock", 10, 3000), ("rosenbrock", 64, 400), ("gaussian", 150, 300)]


def _objective(name, dim):
    import zeus_b200 as zb

    return zb.Gaussian(zb.gaussian_matrix(dim)) if name == "gaussian" else zb.Rosenbrock(dim)


@pytest.mark.parametrize("name,dim,n", SWARMS)
def test_the_kernel_fills_with_nan(cuda, no_wait, name, dim, n):
    import torch

    import zeus_b200 as zb
    from zeus_b200.device import check_swarm

    x, f, g = zb.pso_device(_objective(name, dim), 3, n, -5.0, 5.0, 4)
    torch.cuda.synchronize()
    assert torch.isnan(x).all() and torch.isnan(f).all() and torch.isnan(g[0])
    with pytest.raises(zb.ZeusError, match="incomplete"):
        check_swarm(g)


def test_the_whole_call_reports_it(cuda, no_wait, tmp_path, monkeypatch):
    import zeus_b200 as zb
    from zeus_b200.shard import sharded_optimize

    monkeypatch.chdir(tmp_path)
    obj, n, dim = zb.Rosenbrock(10), 3000, 10
    prob, cfg = obj.problem(None, None), zb.make_config(100, n + 1, 1e-8)
    best, cen, x = zb.CResult(), zb.CCensus(), np.full(dim, 7.0)
    rc = zb.lib().zeus_optimize(C.byref(prob), -5.0, 5.0, n, 100, 4, n + 1, 1e-8, 42,
                                C.byref(cfg), C.byref(best), x.ctypes.data, C.byref(cen), None,
                                None, None)
    assert rc == zb.E_CUDA and "incomplete" in zb.last_error()
    assert best.status == 4 and best.idx == -1 and (x == 7.0).all()
    with pytest.raises(zb.ZeusError, match="incomplete"):
        sharded_optimize(obj, n, -5.0, 5.0, 100, 4, n + 1, 1e-8, 42)
    with pytest.raises(zb.ZeusError, match="incomplete"):
        zb.Zeus(obj, -5.0, 5.0, n, 20, 4, n + 1, "rosenbrock", 1e-8, 42, 0,
                trajectory_file="t.tsv")


def test_the_batch_plan_reports_it(cuda, no_wait):
    import zeus_b200 as zb

    classes = [dict(obj=zb.Rosenbrock(10), n=3000, lower=-5.0, upper=5.0, pso_iter=4, seed=1),
               dict(obj=zb.Rosenbrock(2), n=64, lower=-5.0, upper=5.0, seed=2)]
    plan = zb.BatchPlan(classes, max_iter=50)
    with pytest.raises(zb.ZeusError, match="incomplete"):
        plan.run()
    plan.close()


def test_a_swarm_of_one_block_waits_for_nobody(cuda, no_wait):
    import torch

    import zeus_b200 as zb

    x, f, g = zb.pso_device(zb.Rosenbrock(10), 3, 100, -5.0, 5.0, 4)
    torch.cuda.synchronize()
    assert torch.isfinite(x).all() and torch.isfinite(f).all() and g[0] == f.min()
