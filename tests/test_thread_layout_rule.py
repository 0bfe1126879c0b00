"""The thread layout gives a run a warp only where that measured no slower than
a thread (times on a B200 in zb_fast_thread.cu): the rule's side at sizes
measured on both."""
import ctypes as C

import pytest

import zeus_b200 as zb

ROSENBROCK, RASTRIGIN, ACKLEY, GAUSSIAN, NLL = range(5)
ADJ, DUAL = zb.GRAD_ADJOINT, zb.GRAD_DUAL


def _warps(kind, dim, grad, max_iter, n):
    f = zb.lib().zeus_internal_thread_layout_warps
    f.argtypes = [C.c_int] * 4 + [C.c_int64]
    return bool(f(kind, dim, grad, max_iter, n))


# the thread form was faster by a tenth or more, twenty times at the end
@pytest.mark.parametrize("kind,dim,grad,max_iter,n", [
    (ROSENBROCK, 2, ADJ, 50, 12288), (ROSENBROCK, 2, ADJ, 5, 16384), (ROSENBROCK, 2, DUAL, 1000, 32768),
    (ROSENBROCK, 4, ADJ, 50, 8192), (ROSENBROCK, 4, DUAL, 50, 4096), (ROSENBROCK, 8, ADJ, 5, 3072),
    (ROSENBROCK, 8, ADJ, 50, 2048 + 1024), (ROSENBROCK, 8, ADJ, 200, 6144),
    (ROSENBROCK, 8, ADJ, 1000, 32768), (ROSENBROCK, 8, DUAL, 1000, 16384),
    (ROSENBROCK, 10, ADJ, 1000, 32768), (RASTRIGIN, 2, ADJ, 5, 16384), (RASTRIGIN, 2, DUAL, 20, 16384),
    (RASTRIGIN, 10, ADJ, 20, 8192), (RASTRIGIN, 10, DUAL, 50, 2048), (ACKLEY, 2, DUAL, 20, 8192),
    (ACKLEY, 10, ADJ, 10000, 8192), (ACKLEY, 10, DUAL, 10000, 1536), (NLL, 4, ADJ, 1000, 32768),
    (NLL, 4, DUAL, 200, 1536), (NLL, 4, DUAL, 5, 65536), (GAUSSIAN, 8, ADJ, 10000, 100)])
def test_a_thread_a_run_where_it_is_faster(kind, dim, grad, max_iter, n):
    assert not _warps(kind, dim, grad, max_iter, n)


# the warp form was faster by a tenth or more
@pytest.mark.parametrize("kind,dim,grad,max_iter,n", [
    (ROSENBROCK, 2, ADJ, 10000, 1024), (ROSENBROCK, 2, ADJ, 10000, 16384), (ROSENBROCK, 2, DUAL, 200, 4096),
    (ROSENBROCK, 4, ADJ, 10000, 65536), (ROSENBROCK, 8, ADJ, 10000, 4099), (ROSENBROCK, 8, ADJ, 1000, 12288),
    (ROSENBROCK, 8, ADJ, 10000, 65536), (ROSENBROCK, 8, DUAL, 10000, 32768), (ROSENBROCK, 8, DUAL, 50, 1024),
    (RASTRIGIN, 2, ADJ, 10000, 32768), (RASTRIGIN, 2, DUAL, 200, 32768), (RASTRIGIN, 10, ADJ, 1000, 65536),
    (ACKLEY, 2, ADJ, 10000, 32768), (ACKLEY, 2, DUAL, 1000, 32768), (ACKLEY, 10, ADJ, 10000, 3072),
    (ACKLEY, 10, DUAL, 10000, 1024), (NLL, 4, ADJ, 200, 8192), (NLL, 4, DUAL, 1000, 1024)])
def test_a_warp_a_run_where_it_is_faster(kind, dim, grad, max_iter, n):
    assert _warps(kind, dim, grad, max_iter, n)
