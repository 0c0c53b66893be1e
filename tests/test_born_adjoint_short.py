"""The Born adjoint's units (the power of two that its accumulators are kept in) in
runs of a few steps, whose first step has no wave yet, or next to none."""
import numpy as np
import pytest

from tests.test_gpu_parity import _batch_inputs
from tests.test_step_ways import engine, enqueue

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt", [5, 16, 17, 33])
@pytest.mark.parametrize("first", [0.0, 2.0 ** -100])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -88, 2.0 ** 60])
def test_units_of_short_runs(nt, first, scale):
    """A source scaled by a power of two scales the image by it, to the rounding
    of FP32 fields (normal numbers throughout: the velocities are about 1e-8
    of the source, 1e-34 at the smallest scale)."""
    nx, nz, pml = 64, 30, 8
    _, model, shots = _batch_inputs(2, nshots=2, allnx=nx, allnz=nz, pml=pml, nt=nt)
    rng = np.random.default_rng(nt)
    model["sou"] = rng.standard_normal(nt).astype(np.float32)
    model["sou"][0] = first
    for d in shots:
        d["obs_z"], d["obs_x"] = (rng.standard_normal((d["ntr"], nt)).astype(np.float32) for _ in range(2))
    out = []
    for f in (2.0 ** 20, scale):  # (any scale that is far from both ends)
        m = dict(model, sou=(f * model["sou"]).astype(np.float32))
        fd = engine(2, nx, nz, pml, nt, m)
        enqueue(fd, shots, pml)
        out.append(np.concatenate(fd.born_adjoint()) / f)
        fd.close()
    a, b = out
    assert np.abs(a).max() > 0 and np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(a)
