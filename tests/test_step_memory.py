"""The whole steps' optional copy of the fields and the memory of other runs:
what fits without it fits with it.  A limit on the engine's buffers stands in
for a full device."""
import numpy as np
import pytest

from tests.test_gpu_parity import _batch_inputs
from tests.test_step_ways import engine, enqueue

pytestmark = pytest.mark.gpu


def _transport(fd, model):
    fd.set_misfit(1)
    return (fd.run()[1],) + fd.read_gradients_f64()


def _search(fd, model):
    return fd.line_search_parabola(model["dvp"], model["dvs"], 0.5, 1.0)


@pytest.mark.parametrize("run,stage,nx,nz,pml,nt", [
    (lambda fd, m: fd.hessian_vector(m["dvp"], m["dvs"]), 2, 397, 214, 20, 24),
    (lambda fd, m: fd.born_adjoint(), 2, 397, 214, 20, 24),
    (_transport, 1, 230, 41, 8, 7300),  # traces too long for shared memory: global scratch
    (_search, 1, 397, 214, 20, 24),
], ids=["hessian", "adjoint", "transport", "search"])
def test_a_later_run_has_the_copy_given_back(run, stage, nx, nz, pml, nt):
    _, model, shots = _batch_inputs(stage, nshots=1, allnx=nx, allnz=nz, pml=pml, nt=nt)
    limit, out = None, []
    for sweeps in (True, False):
        fd = engine(stage, nx, nz, pml, nt, model, sweeps)
        enqueue(fd, shots, pml)
        fd.run()
        fd.imagebuffer_resettozero()
        if not sweeps:
            assert fd.debug_steps() == ("burst", "burst")
            # all that the two runs need without the copy, and 64 KB for the items
            assert limit < fd.debug_memory_limit() + (need - first)
            fd.debug_memory_limit(limit)
        else:
            first = fd.debug_memory_limit()
        enqueue(fd, shots, pml)
        out.append(run(fd, model))
        if sweeps:
            need = fd.debug_memory_limit()
            limit = need + (64 << 10)
        fd.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))


def test_state_that_was_given_back_is_refused():
    import sfwi_gb300 as sg
    nx, nz, pml, nt = 397, 214, 20, 24
    _, model, shots = _batch_inputs(1, nshots=1, allnx=nx, allnz=nz, pml=pml, nt=nt)
    fd = engine(1, nx, nz, pml, nt, model)
    enqueue(fd, shots, pml)
    fd.run()
    fd.debug_grid()
    # no room for the next allocation (of trial models), nor for its batch once the copy is gone
    fd.debug_memory_limit(0)
    enqueue(fd, shots, pml)
    with pytest.raises(sg.SfwiError, match="sfwi error -3"):
        fd.line_search_parabola(model["dvp"], model["dvs"], 0.5, 1.0)
    with pytest.raises(sg.SfwiError, match="given back"):
        fd.debug_grid()
    with pytest.raises(sg.SfwiError, match="wait timed out"):
        fd.wait_selftest(4096)  # (the sweeps' pipeline)
    assert all(v > 0 for v in fd.time_kernels(4).values())
    fd.debug_memory_limit()
    fd.imagebuffer_resettozero()
    enqueue(fd, shots, pml)
    m, _ = fd.run()
    assert np.isfinite(m) and fd.debug_steps() == ("burst", "burst")
    fd.close()
