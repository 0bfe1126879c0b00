"""Which line-search trial the tile layout takes on the binned Poisson
likelihood, whose trials it evaluates seven at a time, against the same search
on the host: one iteration from the start, p = -grad f, the first of
alpha = 2^-k, k = 0..19, that decreases f enough, else 2^-20."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _terms(th, lx, l1, k, lgk):
    """Per point of th (m, 4): f's terms (m, bins) and their magnitudes."""
    ll = np.log(th[:, :1]) + th[:, 1:2] * l1 - (th[:, 2:3] + th[:, 3:4] * lx) * lx
    mag = 1 + np.abs(np.log(th[:, :1])) + np.abs(th[:, 1:2] * l1) + (
        np.abs(th[:, 2:3]) + np.abs(th[:, 3:4] * lx)) * np.abs(lx)
    e = np.exp(ll)
    return ll, e, e - k * ll + lgk, (e + k) * mag + np.abs(lgk)


@pytest.mark.parametrize("nbins", [1, 5, 32, 39, 64, 100])
def test_the_first_passing_trial_is_taken(cuda, nbins):
    import torch
    from scipy.special import gammaln

    import zeus_b200 as zb

    edges = np.geomspace(0.085, 0.54, nbins + 1)
    x = 0.5 * (edges[1:] + edges[:-1])
    lx, l1 = np.log(x), np.log(1 - x)
    rng = np.random.default_rng(nbins)
    k = rng.poisson(4.0 * (1 - x) ** 2 / x).astype(np.int32)
    lgk = gammaln(k + 1.0)
    # amplitudes from 0.004 to 400: first steps from large to the last trials
    x0 = np.stack([4.0 * 10.0 ** rng.uniform(-3, 2, 256), rng.uniform(0, 4, 256),
                   rng.uniform(0, 2, 256), rng.uniform(-0.2, 0.2, 256)], 1)
    r = zb.bfgs_device(zb.PoissonNLL(k, x), torch.from_numpy(x0).cuda(), max_iter=1,
                       layout=zb.LAYOUT_TILE, tile=32)
    torch.cuda.synchronize()
    taken = r.counters.cpu().numpy()[:, 1] - 2  # 1 at the start, k + 1 trials
    xs, compared, late = r.x.cpu().numpy(), 0, 0
    for i in range(len(x0)):
        ll, e, t, m = _terms(x0[i:i + 1], lx, l1, k, lgk)
        d = (e - k)[0]
        g = np.array([d.sum() / x0[i, 0], (d * l1).sum(), -(d * lx).sum(), -(d * lx * lx).sum()])
        a = 0.5 ** np.arange(21)
        pts = x0[i] - a[:, None] * g
        with np.errstate(invalid="ignore", over="ignore", divide="ignore"):
            _, _, tk, mk = _terms(pts, lx, l1, k, lgk)
            f, f0 = tk.sum(1), t.sum()
            # logarithms, exponentials, lgamma and the sums within some ulp
            # of the magnitudes, the point itself within some of the gradient's
            err = (nbins + 64) * 2.0 ** -52 * (mk.sum(1) + m.sum())
            bar = np.minimum(f0 - 0.1 * a * (g @ g), np.nextafter(f0, -np.inf))
            ok = f <= bar
            sure = ~(np.abs(f - bar) <= err) | np.isnan(f) | np.isposinf(f)
        first = int(np.argmax(ok[:20])) if ok[:20].any() else 20
        if not sure[:min(first, 19) + 1].all():
            continue  # a trial too close to call
        compared += 1
        late += first > 7
        assert taken[i] == first, (i, taken[i], first)
        if first < 20:
            # within the gradient's error, some ulp of its terms
            w = np.array([np.full(nbins, 1 / x0[i, 0]), np.abs(l1), np.abs(lx), lx * lx])
            tol = 2.0 ** -52 * (a[first] * (nbins + 64) * (w * m).sum(1)
                                + 4 * (np.abs(x0[i]) + np.abs(pts[first])))
            assert (np.abs(xs[i] - pts[first]) <= tol).all(), i
    assert compared >= 128 and late >= 16  # trials of the second and third sweep too
