"""The symmetric quadratic form's kernel (C in shared memory, H in registers)
gives the bits of the CTA layout's kernel, which the cycle timers select."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,max_iter,flags", [(1, 10000, 0), (3, 0, 0), (5, 1, 0), (7, 4, 0),
                                              (147, 10000, 0), (149, 10000, 1), (400, 6, 0)])
def test_equals_the_cta_layout(n, max_iter, flags):
    import torch

    import zeus_b200 as zb

    rng = np.random.default_rng(n)
    a = rng.standard_normal((150, 150))
    for C in (zb.gaussian_matrix(150), a @ a.T / 150 + np.eye(150)):
        obj = zb.Gaussian(0.5 * (C + C.T))
        x0 = torch.from_numpy(rng.uniform(-5, 5, (n, 150))).cuda()
        x0[0, :] = 0.0 if n > 1 else x0[0, :]  # a run that starts at the minimum
        r = [zb.bfgs_device(obj, x0, max_iter=max_iter, flags=flags, cycles=c)
             for c in (False, True)]
        torch.cuda.synchronize()
        for name in ("fval", "status", "iter", "gnorm", "x", "counters"):
            u, v = (getattr(q, name).cpu().numpy() for q in r)
            np.testing.assert_array_equal(u, v, err_msg=name)


def test_nonfinite_start_and_raised_stop_flag():
    import torch

    import zeus_b200 as zb

    obj = zb.Gaussian(zb.gaussian_matrix(150))
    x0 = torch.from_numpy(np.random.default_rng(1).uniform(-5, 5, (6, 150))).cuda()
    x0[2, 149] = float("nan")
    x0[4, 0] = 1e200
    r = [zb.bfgs_device(obj, x0, cycles=c) for c in (False, True)]
    torch.cuda.synchronize()
    assert int(r[0].status[2]) == 5
    for name in ("fval", "status", "iter", "gnorm", "x"):
        u, v = (getattr(q, name).cpu().numpy() for q in r)
        np.testing.assert_array_equal(u, v, err_msg=name)
    r[0].control[0] = 1
    r[0].launch(x0, reset_control=False)
    torch.cuda.synchronize()
    assert (r[0].status == 2).all() and (r[0].iter == 0).all()


def test_matrix_that_is_not_16_byte_aligned():
    """C at an odd double: the CTA layout's kernel, whose sums split otherwise."""
    import torch

    import zeus_b200 as zb

    C = zb.gaussian_matrix(150)
    dp = zb.device.DeviceProblem(zb.Gaussian(C))
    buf = torch.zeros(1 + 150 * 150, dtype=torch.float64, device="cuda")
    buf[1:] = dp.data.reshape(-1)
    dp.data = buf[1:]
    assert dp.data.data_ptr() % 16 == 8
    x0 = torch.from_numpy(np.random.default_rng(2).uniform(-5, 5, (20, 150))).cuda()
    r = [zb.bfgs_device(dp, x0, cycles=c) for c in (False, True)]
    torch.cuda.synchronize()
    assert (r[0].status == 1).all()
    for name in ("fval", "status", "iter", "gnorm", "x", "counters"):
        u, v = (getattr(q, name).cpu().numpy() for q in r)
        np.testing.assert_array_equal(u, v, err_msg=name)
