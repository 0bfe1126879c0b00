"""The tile layout's line search on the binned Poisson likelihood evaluates
several trials to a sweep over the bins, the last partial round of bins
shared out over the lanes: whatever trial is taken, the value reported with
it is f at the point reported."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _nll_and_scale(th, x, k, lgk):
    """f(th) and the sum of its terms' magnitudes (what their rounding
    scales with)."""
    lx, l1 = np.log(x), np.log(1 - x)
    ll = np.log(th[0]) + th[1] * l1 - (th[2] + th[3] * lx) * lx
    parts = np.stack([np.exp(ll), -k * ll, lgk])
    mag = np.abs(np.log(th[0])) + np.abs(th[1] * l1) + (abs(th[2]) + np.abs(th[3] * lx)) * np.abs(lx)
    scale = np.exp(ll) * (1 + mag) + k * (1 + mag) + np.abs(lgk)
    return parts.sum(), scale.sum()


@pytest.mark.parametrize("nbins", [1, 5, 31, 32, 33, 39, 64, 100, 131])
def test_reported_value_is_f_at_the_reported_point(nbins):
    import torch
    from scipy.special import gammaln

    import zeus_b200 as zb

    edges = np.geomspace(0.085, 0.54, nbins + 1)
    x = 0.5 * (edges[1:] + edges[:-1])
    rng = np.random.default_rng(nbins)
    lam = 3.0 * (1 - x) ** 10 / x ** 5
    k = rng.poisson(lam).astype(np.int32)
    x0 = rng.uniform([0.5, 5, 2, 0], [6, 12, 6, 0.5], (40, 4))
    r = zb.bfgs_device(zb.PoissonNLL(k, x), torch.from_numpy(x0).cuda(), max_iter=40,
                       layout=zb.LAYOUT_TILE, tile=32)
    torch.cuda.synchronize()
    fv, xs, cnt = r.fval.cpu().numpy(), r.x.cpu().numpy(), r.counters.cpu().numpy()
    ok = np.isfinite(fv) & np.isfinite(xs).all(1) & (xs[:, 0] > 0) & (r.status.cpu().numpy() != 5)
    assert ok.sum() >= 20
    # searches that went past the first trial took part
    assert (cnt[:, 1] > cnt[:, 0] + 1).any()
    lgk = gammaln(k + 1.0)
    for i in np.flatnonzero(ok):
        f, scale = _nll_and_scale(xs[i], x, k, lgk)
        # logarithms, exponentials and lgamma within a few ulp, then at most
        # nbins + 8 additions
        assert abs(fv[i] - f) <= (nbins + 32) * 2.0 ** -52 * scale
