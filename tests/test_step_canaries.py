"""Stray-write checks of the whole-step kernels, as tests/test_canaries.py has them
for the sweeps: the outer four rows and columns of every shot and the
padding below each column start at zero and stay so, in the state arrays, the
accumulators and both copies of the fields that the steps advance.  The state
itself is the sweeps', bit for bit (a copy of the scattered field that the
adjoint took over reads as zeros)."""
import numpy as np
import pytest

from tests.test_gpu_parity import _batch_inputs
from tests.test_step_ways import engine

pytestmark = pytest.mark.gpu
NOP, SC, AD, ACC = 4, 10, 20, 28


def _outer(a, widths, depths):
    row0 = 0
    for w, n in zip(widths, depths):
        g = a[row0:row0 + w]
        assert not (np.any(g[:NOP]) or np.any(g[w - NOP:]) or np.any(g[:, :NOP]) or np.any(g[:, n - NOP:]))
        row0 += w
    assert row0 == a.shape[0]


@pytest.mark.parametrize("stage,nx,nz,pml,nshots,nt,option,ways", [
    (1, 230, 41, 8, 1, 31, "rho", ("burst", "burst")),
    (2, 149, 83, 11, 1, 30, "rho", ("burst", "burst")),
    (2, 203, 97, 11, 1, 31, "vz", ("burst", "burst")),
    (1, 97, 130, 11, 1, 31, "snap4 f16", ("burst", "burst")),
    (2, 120, 90, 31, 1, 30, "snap4 f32", ("burst", "burst")),
    (1, 299, 151, 20, 3, 31, "vz", ("march", "sweeps")),
    (2, 150, 260, 11, 5, 31, "lengths", ("march", "sweeps")),
    (1, 150, 183, 11, 7, 30, "lengths", ("march", "sweeps")),
    (2, 301, 117, 11, 7, 31, "uneven", ("burst", "burst")),
    (2, 201, 187, 11, 6, 33, "snap5 f32", ("march", "march")),
    (1, 150, 208, 20, 54, 30, "rho", ("sweeps", "march")),
    (1, 150, 83, 11, 8, 31, "snap4 f32", ("sweeps", "march")),
    (1, 401, 331, 13, 20, 31, "rho", ("march", "march")),
    (2, 399, 331, 13, 20, 30, "lengths", ("march", "march")),
    (1, 230, 41, 8, 1, 31, "forward", ("burst", "sweeps")),
    (2, 150, 260, 11, 5, 31, "forward", ("march", "sweeps")),
])
def test_no_writes_outside_the_update_region(stage, nx, nz, pml, nshots, nt, option, ways):
    import sfwi_gb300 as sg
    few = min(nshots, (nx - 8) // 10)
    _, model, shots = _batch_inputs(stage, nshots=few, allnx=nx, allnz=nz, pml=pml, nt=nt, uneven=option == "uneven")
    shots = [shots[k % few] for k in range(nshots)]
    widths = [d["nx"] + 2 * pml for d in shots]
    depths = [nz + 2 * pml] * nshots
    state = []
    for sweeps in (False, True):
        fd = engine(stage, nx, nz, pml, nt, model, sweeps)
        if option == "rho":
            fd.set_density_gradient(True)
        elif option == "vz":
            fd.set_source(sg.SOURCE_VZ_FORCE)
        elif option.startswith("snap"):
            fd.set_snapshots(int(option[4]), option[6:])
        # (odd and even lengths: a shot's forward steps end in either copy)
        lens = [nt - 3 * (2 * k >= nshots) if option == "lengths" else nt for k in range(nshots)]
        for n, d in zip(lens, shots):
            fd.enqueue_shot(d["nx"], d["isx"], pml + 2, pml, d["ngx_left"], d["delta_left"], 0, d["gc"],
                            d["obs_z"][:, :n], d["obs_x"][:, :n], nt=n)
        if option == "lengths":
            models = [dict(model, nt=n) for n in (nt, nt - 3)]
            fd.run_models(models, [int(2 * k >= nshots) for k in range(nshots)])
        elif option == "forward":
            fd.run_forward()
        else:
            fd.run()
        grid, nstate = fd.debug_grid()
        state.append(grid[:nstate])
        if not sweeps:
            assert fd.debug_steps() == ways
            copies = fd.debug_copies()
        fd.close()
    got, want = state
    assert np.any(got[0]) and (option == "forward" or np.any(got[ACC]))
    for a in got:
        _outer(a, widths, depths)
    for key, a in copies.items():
        _outer(a, widths, depths)
        assert key[2] > 4 or key[3] or np.any(a), key  # (totals of the first field: the wave has come)
    taken = stage == 2 and ways[0] != "sweeps" and ways[1] != "sweeps" and not option.startswith("snap")
    for k in range(len(want)):
        if taken and SC <= k < AD:
            assert not np.any(got[k])
        else:
            assert np.array_equal(got[k], want[k]), k
