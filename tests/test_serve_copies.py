"""The server's budget holds with the copies of the wavefields that whole time
steps take (sfwi_set_copy_limit)."""
import threading
import time

import numpy as np
import pytest

from sfwi_gb300 import serve


@pytest.mark.parametrize("batch", [False, True])
def test_runs_and_their_copies_stay_within_the_budget(monkeypatch, batch):
    reqs = serve.poisson_requests(24, 2000.0, grid=((60, 40), (200, 150)), nt=(60, 120), shots=(1, 4))
    lock, held, most, given = threading.Lock(), [0], [0], []

    def run(group, strip_chunk, copy_limit):
        size = (serve.batch_bytes(group) if batch else serve.request_bytes(group[0])) + copy_limit
        with lock:
            held[0] += size
            most[0] = max(most[0], held[0])
            given.append((copy_limit, serve.copy_bytes(group), serve.copy_bytes(group, 4)))
        time.sleep(0.01)
        with lock:
            held[0] -= size
        z = np.zeros((1, 1))
        return [(0.0, z, z, z) for _ in group]

    monkeypatch.setattr(serve, "run_request", lambda r, sc, limit: run([r], sc, limit)[0])
    monkeypatch.setattr(serve, "run_requests", run)
    budget = 30 * max(serve.request_bytes(r) for r in reqs)
    res = serve.Server(budget, max_active=8, batch=batch, max_batch=3).run(reqs)
    assert len(res) == len(reqs)
    assert most[0] <= budget
    assert all(g[0] in (0,) + g[1:] for g in given) and any(g[0] for g in given)
    # no copies where they do not fit in an eighth of what is left
    del given[:]
    serve.Server(max((serve.batch_bytes([r]) if batch else serve.request_bytes(r)) for r in reqs) + 1000, max_active=8,
                 batch=batch, max_batch=1).run(reqs)
    assert given and not all(g[0] for g in given) and most[0] <= budget


@pytest.mark.gpu
def test_copies_stay_within_their_limit_and_change_nothing():
    from tests.test_gpu_parity import _batch_inputs
    from tests.test_step_ways import engine, enqueue, results
    nx, nz, pml, nt = 401, 331, 13, 30
    _, model, shots = _batch_inputs(1, nshots=20, allnx=nx, allnz=nz, pml=pml, nt=nt)
    X, P = 20 * (nx + 2 * pml), (nz + 2 * pml + 3) // 4 * 4
    fd = engine(1, nx, nz, pml, nt, model)
    out = []
    m, s, cells = "march", "sweeps", 4 * X * P
    for limit, ways in ((None, (m, m)), (44 * cells, (m, m)), (44 * cells - 4, (m, s)), (4 * cells, (m, s)),
                        (4 * cells - 4, (s, s)), (0, (s, s)), (None, (m, m))):
        fd.set_copy_limit(limit)
        fd.imagebuffer_resettozero()
        enqueue(fd, shots, pml)
        out.append(results(fd, shots))
        assert fd.debug_steps() == ways, limit
    fd.close()
    assert all(np.array_equal(a, b) for o in out[1:] for a, b in zip(out[0], o))


@pytest.mark.gpu
def test_requests_give_the_same_without_copies():
    reqs = serve.poisson_requests(4, 50.0, grid=((120, 60), (300, 200)), nt=(60, 120), shots=(1, 3))
    a = [serve.run_request(r) for r in reqs]
    b = [serve.run_request(r, copy_limit=0) for r in reqs]
    c = serve.Server(64 << 30, max_active=2).run(reqs)
    for x, y, z in zip(a, b, c):
        assert x[0] == y[0] == z.misfit
        assert all(np.array_equal(u, v) for u, v in zip(x[1:], y[1:]))
        assert all(np.array_equal(u, v) for u, v in zip(x[1:], (z.grad_pp, z.grad_ps, z.illum)))
