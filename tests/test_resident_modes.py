"""Calls on the batch that the last run left on the device, when that run was
of another mode than the handle's: they are refused, or take what is there."""
import pytest

from tests.test_gpu_parity import _batch_inputs
from tests.test_step_ways import engine, enqueue

pytestmark = pytest.mark.gpu


def test_gradient_steps_need_a_run_of_the_present_mode():
    import sfwi_gb300 as sg
    nx, nz, pml, nt = 64, 30, 8, 60
    _, model, shots = _batch_inputs(2, nshots=2, allnx=nx, allnz=nz, pml=pml, nt=nt)
    fd = engine(2, nx, nz, pml, nt, model)
    enqueue(fd, shots, pml)
    fd.born_adjoint()  # snapshots of its own, no edge strips
    for call in (fd.time_kernels, fd.autotune):
        with pytest.raises(sg.SfwiError, match="no gradient state"):
            call()
    fd.set_tile_shape("32x32")  # re-tiles what is there
    enqueue(fd, shots, pml)
    fd.run()
    assert all(v > 0 for v in fd.time_kernels(4).values())
    fd.set_snapshots(2, "f16")  # the resident run kept no snapshots
    with pytest.raises(sg.SfwiError, match="no gradient state"):
        fd.time_kernels()
    fd.set_snapshots(0)
    assert all(v > 0 for v in fd.time_kernels(4).values())
    fd.close()

