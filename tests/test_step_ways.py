"""Which way a batch takes its time steps (152 SMs), forward and backward, and the
same results as the sweeps bit for bit, also where only one direction
takes whole steps."""
import numpy as np
import pytest

from tests.test_gpu_parity import _batch_inputs

pytestmark = pytest.mark.gpu


def engine(stage, nx, nz, pml, nt, model, sweeps=False):
    import sfwi_gb300 as sg
    fd = sg.FD2DGPU_ELASTIC(model["sou"], 10.0, 10.0, 1e-3, nx + 2 * pml, nz + 2 * pml, nx, nz, 1, pml, nt, 4, 1,
                            stage=stage)
    fd.GPUbufferVPVS(model["vp"], model["vs"], model["rho"] if stage == 1 else None)
    fd.GPUbufferM(model["dvp"], model["dvs"])
    if sweeps:
        fd.set_tile_shape("16x32")
    return fd


def enqueue(fd, shots, pml, **over):
    for d in shots:
        d = dict(d, isz=pml + 2, igz=pml, **over)
        fd.enqueue_shot(d["nx"], d["isx"], d["isz"], d["igz"], d["ngx_left"], d["delta_left"], 0, d["gc"], d["obs_z"],
                        d["obs_x"])


def results(fd, shots):
    _, per = fd.run()
    return [per] + list(fd.read_gradients_f64()) + [v for k, d in enumerate(shots)
                                                    for v in fd.read_records(k, d["ntr"]).values()]


@pytest.mark.parametrize("stage,nx,nz,pml,nshots,snap,ways", [
    (1, 230, 41, 8, 1, None, ("burst", "burst")),
    (2, 397, 214, 20, 1, None, ("burst", "burst")),
    (1, 97, 130, 11, 1, (4, "f16"), ("burst", "burst")),
    (1, 299, 151, 20, 3, None, ("march", "sweeps")),
    (2, 150, 260, 11, 5, None, ("march", "sweeps")),
    (2, 201, 187, 11, 6, (5, "f32"), ("march", "march")),
    (1, 401, 331, 13, 20, None, ("march", "march")),
    (2, 399, 331, 13, 20, None, ("march", "march")),
    # backward alone: from the sweeps' plain fields to pairs, and from the sweeps' snapshots
    (1, 150, 208, 20, 54, None, ("sweeps", "march")),
    (1, 150, 83, 11, 8, (4, "f32"), ("sweeps", "march")),
    (2, 64, 30, 8, 1, None, ("sweeps", "sweeps")),
])
def test_steps_taken_and_their_bits(stage, nx, nz, pml, nshots, snap, ways):
    nt = 45
    few = min(nshots, (nx - 8) // 10)  # (sources 10 nodes apart)
    _, model, shots = _batch_inputs(stage, nshots=few, allnx=nx, allnz=nz, pml=pml, nt=nt)
    shots = [shots[k % few] for k in range(nshots)]
    out = []
    for sweeps in (False, True):
        fd = engine(stage, nx, nz, pml, nt, model, sweeps)
        if snap:
            fd.set_snapshots(*snap)
        enqueue(fd, shots, pml)
        out.append(results(fd, shots))
        assert fd.debug_steps() == (("sweeps", "sweeps") if sweeps else ways)
        fd.close()
    assert all(np.abs(x).max() > 0 for x in out[1][:4])
    assert all(np.array_equal(x, y) for x, y in zip(*out))
