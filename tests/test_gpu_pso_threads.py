"""Swarms of several sizes seeded from several host threads, a stream each:
every call is accepted and gives what the same call gives alone."""
import ctypes as C
import threading

import pytest

pytestmark = pytest.mark.gpu

DIM = 10
# shared memory of a block: 95 KB, 72 KB, 152 KB
SIZES = (40000, 30000, 64000)


def test_concurrent_swarms_of_several_sizes(cuda):
    import torch

    import zeus_b200 as zb

    L, prob = zb.lib(), zb.device.DeviceProblem(zb.Rosenbrock(DIM)).c()
    alone = {n: zb.pso_device(zb.Rosenbrock(DIM), 3, n, -5.0, 5.0, 1) for n in SIZES}
    torch.cuda.synchronize()
    errors, results = [], []

    def work(n, stream, x, f, g, ws):
        torch.cuda.set_device(0)
        for _ in range(500):
            rc = L.zeus_pso_device(C.byref(prob), 3, n, -5.0, 5.0, 1, 0.5, 1.2, 1.5, x.data_ptr(),
                                   f.data_ptr(), g.data_ptr(), ws.data_ptr(), ws.numel(),
                                   stream.cuda_stream)
            if rc:
                errors.append((n, rc, zb.last_error()))
        stream.synchronize()
        results.append((n, x, f, g))

    threads = []
    for n in SIZES * 2:
        x, f, g = (torch.empty_like(t) for t in alone[n])
        ws = torch.empty(L.zeus_pso_workspace_size(n, DIM), dtype=torch.uint8, device=cuda)
        threads.append(threading.Thread(target=work, args=(n, torch.cuda.Stream(), x, f, g, ws)))
    torch.cuda.synchronize()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, (len(errors), errors[:3])
    assert len(results) == len(threads)
    for n, *got in results:
        assert all(torch.equal(u, v) for u, v in zip(got, alone[n]))
