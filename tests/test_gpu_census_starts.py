"""The census kernel over its block, cluster and group-width splits against
numpy; start points at the edges of their split into items against the
oracle's."""
import numpy as np
import pytest

from tests import _oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [1, 2, 3, 5, 16, 17, 33, 150])
@pytest.mark.parametrize("n", [1, 31, 2048, 2049, 9001])
def test_census_counts_and_argmin(n, dim):
    import torch

    import zeus_b200 as zb

    rng = np.random.default_rng(100 * dim + n)
    f = rng.integers(0, max(2, n // 3), n).astype(np.float64)  # ties: lowest index wins
    f[rng.random(n) < 0.1] = np.nan
    st = rng.choice([0, 1, 1, 2, 5], n).astype(np.int32)
    km = rng.standard_normal(dim)
    # distances spread about the limit of 0.5, none within rounding of it
    x = km + rng.standard_normal((n, dim)) * (0.5 / np.sqrt(dim)) * rng.uniform(0.2, 2, (n, 1))
    dist = np.sqrt(((x - km) ** 2).sum(1))
    assert (np.abs(dist - 0.5) > 1e-12).all()
    got = zb.census_device(*(torch.from_numpy(a).cuda() for a in (f, st, x)), dim, km)
    conv = st == 1
    want = dict(actual=int((conv & (dist < 0.5)).sum()), claimed=int(conv.sum()),
                surrendered=int(((st != 1) & (st != 2)).sum()), stopped=int((st == 2).sum()),
                best_idx=int(np.nanargmin(f)) if np.isfinite(f).any() else got["best_idx"])
    assert got == want


def test_census_without_coordinates():
    import torch

    import zeus_b200 as zb

    st = torch.ones(5000, dtype=torch.int32, device="cuda")
    f = torch.arange(5000, 0, -1, dtype=torch.float64, device="cuda")
    got = zb.census_device(f, st, None, 7)
    assert got == dict(actual=0, claimed=5000, surrendered=0, stopped=0, best_idx=4999)


@pytest.mark.parametrize("dim,n", [(1, 1), (1, 70001), (2, 300000), (3, 9), (7, 40000),
                                   (10, 33333), (255, 1500), (1001, 700)])
def test_philox_starts_bits_equal_the_oracle(dim, n):
    import zeus_b200 as zb

    got = zb.starts_uniform(77, n, dim, -3.0, 4.5).cpu().numpy()
    np.testing.assert_array_equal(got, O.oracle_starts(77, n, dim, -3.0, 4.5))


def test_starts_into_a_buffer_that_is_not_16_byte_aligned():
    import torch

    import zeus_b200 as zb

    buf = torch.zeros(1 + 64 * 10, dtype=torch.float64, device="cuda")
    out = buf[1:]
    zb.check(zb.lib().zeus_starts_uniform(3, 64, 10, -1.0, 1.0, out.data_ptr(), 0))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy().reshape(64, 10),
                                  O.oracle_starts(3, 64, 10, -1.0, 1.0))
    assert float(buf[0]) == 0.0


@pytest.mark.parametrize("dim,n", [(1, 1), (3, 7), (3, 8), (3, 9), (10, 4099), (1024, 130)])
def test_sobol_starts_bits_equal_the_oracle(dim, n):
    import zeus_b200 as zb

    got = zb.starts(5, n, dim, -3.0, 4.5, prng="sobol").cpu().numpy()
    np.testing.assert_array_equal(got, O.oracle_starts(5, n, dim, -3.0, 4.5,
                                                       prng=O.PRNG_SOBOL))
