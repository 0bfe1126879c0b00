"""How soon a run sees that the required number of runs has converged: two runs
in one warp, side by side, one of which converges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,tile", [(8, 4), (10, 8), (16, 16), (32, 16)])
def test_tile_runs_stop_within_five_iterations(cuda, dim, tile):
    import torch

    import zeus_b200 as zb

    rng = np.random.default_rng(1)
    late = []
    for _ in range(24):
        x0 = np.stack([1 + 0.1 * rng.standard_normal(dim), rng.uniform(-5, 5, dim)])
        r = zb.bfgs_device(zb.Rosenbrock(dim), torch.from_numpy(x0).cuda(), required=1,
                           layout=zb.LAYOUT_TILE, tile=tile)
        torch.cuda.synchronize()
        status, it = r.status.tolist(), r.iter.tolist()
        if status == [1, 2]:
            late.append(it[1] - it[0])
    # the flag is read every fourth iteration and tested at the next: raised
    # in iteration i (counted from 0), it is read at the next multiple of four,
    # i + 1 to i + 4, and stops the run one later
    assert len(late) >= 16
    assert 1 <= min(late) and max(late) <= 5
    assert len(set(late)) > 1  # raised at several places between two reads
