"""Failure path of the whole-step kernels' bounded waits, without a GPU fault:
sfwi_wait_selftest launches a step of each direction with waits that give up
at once; the kernel reports it, leaves when its copies have landed, and the
handle gives the same results afterwards."""
import numpy as np
import pytest

from tests.test_gpu_parity import _batch_inputs
from tests.test_step_ways import engine, enqueue, results

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stage,nx,nz,pml,nshots,snap,ways", [
    (1, 230, 41, 8, 1, None, ("burst", "burst")),
    (2, 397, 214, 20, 1, None, ("burst", "burst")),
    (1, 97, 130, 11, 1, (4, "f16"), ("burst", "burst")),
    (1, 299, 151, 20, 3, None, ("march", "sweeps")),
    (2, 399, 331, 13, 20, None, ("march", "march")),
    (1, 150, 83, 11, 8, (4, "f32"), ("sweeps", "march")),
])
def test_step_wait_timeout_is_reported_and_the_handle_stays_usable(stage, nx, nz, pml, nshots, snap, ways):
    import sfwi_gb300 as sg
    nt = 30
    _, model, shots = _batch_inputs(stage, nshots=nshots, allnx=nx, allnz=nz, pml=pml, nt=nt)
    fd = engine(stage, nx, nz, pml, nt, model)
    if snap:
        fd.set_snapshots(*snap)
    enqueue(fd, shots, pml)
    first = results(fd, shots)
    assert fd.debug_steps() == ways
    before = fd.kernel_launches()
    with pytest.raises(sg.SfwiError, match="wait timed out"):
        fd.wait_selftest(4096)
    assert fd.kernel_launches() - before == 1 + sum(w != "sweeps" for w in ways)
    fd.imagebuffer_resettozero()
    enqueue(fd, shots, pml)
    again = results(fd, shots)
    fd.close()
    assert all(np.array_equal(x, y) for x, y in zip(first, again))


def test_step_wait_timeout_of_a_modelling_run():
    import sfwi_gb300 as sg
    nx, nz, pml, nt = 230, 41, 8, 30
    _, model, shots = _batch_inputs(1, nshots=1, allnx=nx, allnz=nz, pml=pml, nt=nt)
    fd = engine(1, nx, nz, pml, nt, model)
    enqueue(fd, shots, pml)
    fd.run_forward()
    assert fd.debug_steps() == ("burst", "sweeps")
    with pytest.raises(sg.SfwiError, match="wait timed out"):
        fd.wait_selftest(4096)
    fd.close()
