"""The autotuner's choice for a standalone launch of few runs, whose thread
layout has a warp a run: it is timed as it runs there."""
import pytest

pytestmark = pytest.mark.gpu


def _ms(f):
    import torch

    f()
    best = 1e30
    for _ in range(3):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        f()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


@pytest.mark.parametrize("kind,dim", [("Rosenbrock", 2), ("Rosenbrock", 4), ("Rosenbrock", 8),
                                      ("Rastrigin", 2), ("Ackley", 2)])
def test_a_tuned_launch_is_no_slower_than_the_thread_layout(cuda, kind, dim):
    import zeus_b200 as zb

    obj = zb.device.DeviceProblem(getattr(zb, kind)(dim))
    x0 = zb.starts(7, 1024, dim, -5.0, 5.0)
    lay, tile, ms = zb.autotune(obj, n_sample=1024, lower=-5.0, upper=5.0)
    assert lay in (zb.LAYOUT_THREAD, zb.LAYOUT_TILE) and ms > 0
    try:
        tuned = _ms(lambda: zb.bfgs_device(obj, x0))
        thread = _ms(lambda: zb.bfgs_device(obj, x0, layout=zb.LAYOUT_THREAD))
    finally:  # the table lasts as long as the process
        zb.lib().zeus_autotune_record(obj.obj.kind, dim, zb.GRAD_ADJOINT, zb.LAYOUT_THREAD, 0)
    # the tuner's estimate is of 200 iterations of one run: a fifth's room
    assert tuned <= 1.2 * thread


def test_a_recorded_choice_serves_both(cuda):
    import torch

    import zeus_b200 as zb

    obj = zb.device.DeviceProblem(zb.Rosenbrock(8))
    x0 = zb.starts(7, 64, 8, -5.0, 5.0)
    try:
        assert zb.lib().zeus_autotune_record(zb.OBJ_ROSENBROCK, 8, zb.GRAD_ADJOINT,
                                             zb.LAYOUT_TILE, 8) == 0
        few, tile = (zb.bfgs_device(obj, x0, max_iter=200, **kw)
                     for kw in ({}, dict(layout=zb.LAYOUT_TILE, tile=8)))
        torch.cuda.synchronize()
        assert torch.equal(few.x, tile.x) and torch.equal(few.counters, tile.counters)
    finally:
        zb.lib().zeus_autotune_record(zb.OBJ_ROSENBROCK, 8, zb.GRAD_ADJOINT, zb.LAYOUT_THREAD, 0)
