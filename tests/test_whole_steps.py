"""Whole time steps in one launch (csrc/sfwi_march.cu) against the sweeps,
which sfwi_set_tile_shape selects: both take every cell through the same
arithmetic in the same order, so records, misfits, gradients and illumination
agree bit for bit."""
import numpy as np
import pytest

from tests.test_gpu_parity import _batch_inputs

pytestmark = pytest.mark.gpu


def _run(stage, nx, nz, pml, nshots, nt, option, sweeps):
    import sfwi_gb300 as sg
    cfg, model, shots = _batch_inputs(stage, nshots=nshots, allnx=nx, allnz=nz, pml=pml, nt=nt,
                                      uneven=option == "uneven")
    fd = sg.FD2DGPU_ELASTIC(model["sou"], cfg["dx"], cfg["dx"], cfg["dt"], nx + 2 * pml, nz + 2 * pml, nx, nz, 1, pml,
                            nt, 4, shots[0]["ntr"], stage=stage)
    fd.GPUbufferVPVS(model["vp"], model["vs"], model["rho"] if stage == 1 else None)
    fd.GPUbufferM(model["dvp"], model["dvs"])
    if sweeps:
        fd.set_tile_shape("16x32")
    if option == "rho":
        fd.set_density_gradient(True)
    elif option == "host":
        fd.set_cpu_mem(True, 7)
    elif option == "vz":
        fd.set_source(sg.SOURCE_VZ_FORCE)
    elif option and option.startswith("snap"):
        fd.set_snapshots(int(option[4]), option[6:])
        if option.endswith("bf16"):
            fd.set_source(sg.SOURCE_VZ_FORCE)
    lens = [nt - 3 * (k % 2) if option == "lengths" else nt for k in range(nshots)]
    for n, d in zip(lens, shots):
        fd.enqueue_shot(d["nx"], d["isx"], pml + 2, pml, d["ngx_left"], d["delta_left"], 0, d["gc"],
                        d["obs_z"][:, :n], d["obs_x"][:, :n], nt=n)
    before = fd.kernel_launches()
    if option == "lengths":
        models = [dict(vp=model["vp"], vs=model["vs"], rho=model["rho"], nt=n) for n in (nt, nt - 3)]
        per, grads = fd.run_models(models, [k % 2 for k in range(nshots)])
        out = [per] + [g for one in grads for g in one[:3]]
    else:
        m, per = fd.run()
        out = [per] + list(fd.read_gradients_f64())
        out += [v for k, d in enumerate(shots) for v in fd.read_records(k, d["ntr"]).values()]
    if option == "rho":
        out.append(fd.read_density_gradient_f64())
    launches = fd.kernel_launches() - before
    fd.close()
    return out, launches


# one wave of bursts: less than a strip, one column more than a strip, runs of
# 4 and of 16 rows; march forward with backward sweeps: a few shots; march both
# ways: more than 15,000 cells an SM.  Odd heights leave the last column pair
# half outside, widths the last group of rows.
@pytest.mark.parametrize("stage,nx,nz,pml,nshots,nt,option", [
    (1, 230, 41, 8, 1, 61, None),
    (2, 149, 83, 11, 1, 60, "rho"),
    (1, 203, 97, 11, 1, 75, "vz"),
    (2, 397, 214, 20, 1, 60, None),
    (1, 149, 183, 11, 1, 61, "host"),
    (1, 97, 130, 11, 1, 45, "snap4 f16"),
    (2, 120, 90, 31, 1, 60, None),
    (1, 299, 151, 20, 3, 60, "rho"),
    (2, 150, 260, 11, 5, 61, "rho"),
    (1, 151, 213, 12, 6, 61, "host"),
    (1, 151, 213, 12, 5, 61, "vz"),
    (1, 150, 183, 11, 7, 60, "lengths"),
    (2, 301, 117, 11, 7, 60, "uneven"),
    (1, 201, 190, 11, 6, 33, "snap1 f16"),
    (2, 201, 187, 11, 6, 45, "snap5 f32"),
    (1, 333, 140, 11, 4, 45, "snap4 bf16"),
    (1, 401, 331, 13, 20, 61, "rho"),
    (2, 399, 331, 13, 20, 60, "rho"),
    (1, 499, 205, 20, 20, 60, "lengths"),
    (1, 401, 331, 13, 19, 61, "host"),
])
def test_whole_steps_give_the_sweeps_bits(stage, nx, nz, pml, nshots, nt, option):
    a, few = _run(stage, nx, nz, pml, nshots, nt, option, False)
    b, many = _run(stage, nx, nz, pml, nshots, nt, option, True)
    assert few != many  # the batch did run whole steps
    assert len(a) == len(b)
    assert all(np.abs(y).max() > 0 for y in b[:4])  # misfits, both gradients, illumination
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
